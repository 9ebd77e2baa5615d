"""Fixed budgets shorter than the chain of CTAs of the resident sweeps: the
first CTA is done before the last has begun, and every CTA must still run the
whole budget. Repeated, since which CTA is late changes from launch to launch."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import oracle_project, random_fields
from vapor_b200.abi import SOLVER_RED_BLACK_SOR, LinearSolveOptions, ProjectionOptions

pytestmark = pytest.mark.gpu

DT, OMEGA = 0.01, 1.7


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("budget", [1, 2, 3, 7])
@pytest.mark.parametrize("n", [16, 17, 24, 32, 45, 48, 49, 64, 96])
def test_short_fixed_budgets(n, budget):
    opts = LinearSolveOptions.defaults(max_iterations=budget, fixed_iterations=1)
    fields = [np.asarray(a, np.float32) for a in random_fields(n, seed=n + budget)[1:]]
    st, ro, *want = oracle_project(n, 1.0, *[f.copy() for f in fields], DT, OMEGA, 6.0, opts,
                                   solver_kind=SOLVER_RED_BLACK_SOR)
    assert st == 0
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(SOLVER_RED_BLACK_SOR)
    first = None
    for _ in range(40):
        got = [f.copy() for f in fields]
        r, p = stage.project(*got, ProjectionOptions(DT, OMEGA, opts), 6.0, want_pressure=True)
        assert r.linear_solve.iterations == budget
        got.append(p)
        if first is None:
            first = got
        for a, b in zip(got, first):
            assert np.array_equal(_bits(a), _bits(b))
    stage.close()
    # The removed mean is an FP64 sum in another order and may be the next float:
    # the pressure then moves by at most omega / 3 of that per iteration, a face
    # velocity by the difference of two such pressures.
    mean, other = np.float32(r.removed_rhs_mean), np.float32(ro.removed_rhs_mean)
    if mean == other:
        for a, b in zip(first, want):
            assert np.array_equal(_bits(a), _bits(b))
    else:
        moved = budget * OMEGA / 3 * abs(float(mean) - float(other))
        for a, b, scale in zip(first, want, (2 * DT * n,) * 3 + (2,)):
            assert np.abs(a - b).max() <= scale * moved + 4 * np.spacing(np.abs(b).max())


@pytest.mark.parametrize("iterations", [1, 2, 6])
def test_short_budgets_inside_recorded_steps(iterations):
    """The Reflection step halves its budget; scenes of a batch run side by side."""
    def make():
        sims = []
        for k, n in enumerate((32, 64, 45, 48)):
            p = vb.default_params()
            p.reflection, p.project_iterations = 1, iterations
            sim = vb.MacSimulation3D(n, 1.0, p)
            sim.upload(*random_fields(n, seed=9 + k))
            sims.append(sim)
        return sims

    alone, together = make(), make()
    batch = vb.Batch(together)
    for _ in range(20):
        batch.advance(1 / 60)
        for s in alone:
            s.advance(1 / 60)
    batch.synchronize()
    for a, b in zip(alone, together):
        assert a.total_iterations() == b.total_iterations()
        for x, y in zip(a.download(), b.download()):
            assert np.array_equal(_bits(x), _bits(y))
    batch.close()
