"""The bounded waits of the pressure sweeps. With the test hook the first wait
of a launch polls for something that never comes and runs out: the projection
ends at its next decision and reports VAPOR_RUNTIME_ERROR, and the next one on
the same object is right again, bit for bit."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import random_fields, sphere_mask
from vapor_b200 import mac2d
from vapor_b200.abi import (SOLVER_FPCG, SOLVER_MIXED_REFINEMENT, SOLVER_RED_BLACK_SOR, VAPOR_RUNTIME_ERROR,
                            LinearSolveOptions, ProjectionOptions)

pytestmark = pytest.mark.gpu


def _project(stage, n, opts):
    fields = [np.array(a, np.float32, copy=True) for a in random_fields(n, seed=n)[1:]]
    r, p = stage.project(*fields, ProjectionOptions(0.01, 1.8, opts), 6.0, want_pressure=True)
    return r.linear_solve.iterations, fields + [p]


def _runs_out_and_recovers(n, kind, opts, masked=False):
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(kind)
    if masked:
        stage.set_solid(sphere_mask(n, (0.45, 0.55, 0.5), 0.2))
    before = _project(stage, n, opts)
    vb.check(vb.library().vapor_stage_set_wait_probe(stage._h, 64))
    with pytest.raises(vb.VaporError) as error:
        _project(stage, n, opts)
    assert error.value.status == VAPOR_RUNTIME_ERROR and "timed out" in str(error.value)
    vb.check(vb.library().vapor_stage_set_wait_probe(stage._h, 0))
    after = _project(stage, n, opts)
    stage.close()
    assert before[0] == after[0]
    for a, b in zip(before[1], after[1]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("kind", [SOLVER_MIXED_REFINEMENT, SOLVER_FPCG])
def test_passes_over_large_grids(kind):
    opts = LinearSolveOptions.defaults(max_iterations=24, relative_tolerance=1e-6, absolute_tolerance=0.0)
    _runs_out_and_recovers(192, kind, opts)


# one cluster, the whole device
@pytest.mark.parametrize("n", [33, 96])
@pytest.mark.parametrize("kind, fixed, masked", [(SOLVER_RED_BLACK_SOR, 1, False), (SOLVER_RED_BLACK_SOR, 0, False),
                                                 (SOLVER_MIXED_REFINEMENT, 0, False), (SOLVER_MIXED_REFINEMENT, 0, True)])
def test_resident_sweeps(n, kind, fixed, masked):
    opts = LinearSolveOptions.defaults(max_iterations=40, fixed_iterations=fixed, relative_tolerance=1e-6,
                                       absolute_tolerance=0.0)
    _runs_out_and_recovers(n, kind, opts, masked)


@pytest.mark.parametrize("n, kind", [(33, SOLVER_MIXED_REFINEMENT), (96, SOLVER_MIXED_REFINEMENT),
                                     (136, SOLVER_MIXED_REFINEMENT), (192, SOLVER_FPCG)])
def test_a_timeout_ends_the_solve(n, kind):
    """Not the iteration budget: a solve that cannot converge stops within a few launches."""
    opts = LinearSolveOptions.defaults(max_iterations=4000, relative_tolerance=0.0, absolute_tolerance=0.0)
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(kind)
    vb.check(vb.library().vapor_stage_set_wait_probe(stage._h, 64))
    before = vb.kernel_launch_count()
    with pytest.raises(vb.VaporError, match="timed out"):
        _project(stage, n, opts)
    assert vb.kernel_launch_count() - before < 60
    stage.close()


@pytest.mark.parametrize("n", [32, 300])
def test_2d_sweeps(n):
    def frame(sim):
        sim.upload(np.zeros((n, n), np.float32), np.ones((n, n + 1), np.float32), np.zeros((n + 1, n), np.float32))
        sim.advance(1 / 60)
        return sim.download()

    sim = mac2d.ReflectionSimulation2D(n)
    frame(sim)  # the emitter's random state moves on: a second object goes the same way
    twin = mac2d.ReflectionSimulation2D(n)
    frame(twin)
    vb.check(vb.library().vapor_mac2d_refl_set_wait_probe(sim._h, 64))
    with pytest.raises(vb.VaporError, match="timed out"):
        frame(sim)
    frame(twin)
    vb.check(vb.library().vapor_mac2d_refl_set_wait_probe(sim._h, 0))
    for a, b in zip(frame(sim), frame(twin)):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))
    sim.close()
    twin.close()
