"""Two-iteration passes over large grids: the same bits, iteration counts and
residuals as the blocked sweep (itself pinned to the one-colour sweep), at the
sizes where a tile can go wrong (a last tile of one 4-slot group, uneven row
tiles and plane chunks, grids whose rows end in a tile), with budgets and check
intervals that leave one, two or three iterations over, eagerly and inside
captured steps; and the preconditioner's smoothing in passes against the colour
launches that an obstacle mask without obstacles keeps."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import random_fields
from vapor_b200.abi import SOLVER_FPCG, SOLVER_MIXED_REFINEMENT, LinearSolveOptions, ProjectionOptions

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _restore_blocking():
    yield
    vb.tune_sor_blocking(0)


def _project(n, kind, blocking, opts, floor=6.0, mask=None):
    vb.tune_sor_blocking(blocking)
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(kind)
    if mask is not None:
        stage.set_solid(mask)
    fields = [np.array(a, np.float32, copy=True) for a in random_fields(n, seed=70 + n)[1:]]
    r, p = stage.project(*fields, ProjectionOptions(0.01, 1.9, opts), floor, want_pressure=True)
    stage.close()
    return r, fields + [p]


def _same(a, b):
    (ra, fa), (rb, fb) = a, b
    la, lb = ra.linear_solve, rb.linear_solve
    assert la.iterations == lb.iterations and la.converged == lb.converged
    assert la.final_residual == lb.final_residual and ra.divergence_after == rb.divergence_after
    for x, y in zip(fa, fb):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


@pytest.mark.parametrize("floor", [6.0, 0.0])
@pytest.mark.parametrize("n", [136, 144, 168, 200, 264])
def test_mixed_passes_equal_blocked_sweeps(n, floor):
    for interval, budget in ((8, 400), (6, 45), (5, 21), (4, 3), (100, 50)):
        opts = LinearSolveOptions.defaults(max_iterations=budget, residual_check_interval=interval,
                                           relative_tolerance=1e-4, absolute_tolerance=0.0)
        _same(_project(n, SOLVER_MIXED_REFINEMENT, 0, opts, floor), _project(n, SOLVER_MIXED_REFINEMENT, 2, opts, floor))


@pytest.mark.parametrize("budget", [9, 11, 2000])
def test_captured_steps_equal_blocked_sweeps(budget):
    from vapor_b200.plume import scene_params, swirl_fields
    n = 136
    fields = swirl_fields(n, 5)
    outs = []
    for blocking in (0, 2):
        vb.tune_sor_blocking(blocking)
        p = scene_params(vb.default_params(), n, rel=1e-4, max_iterations=budget)
        p.solver_kind = SOLVER_MIXED_REFINEMENT
        sim = vb.MacSimulation3D(n, 1.0, p)
        sim.upload(*fields)
        for _ in range(2):
            sim.advance(0.01)
        outs.append((sim.total_iterations(), sim.download()))
        sim.close()
    assert outs[0][0] == outs[1][0]
    for x, y in zip(outs[0][1], outs[1][1]):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


@pytest.mark.parametrize("n", [192, 200])
def test_smoothing_in_passes_follows_the_colour_launches(n):
    """The sums of the dot products differ in their order, 1e-16 of CG's
    coefficients: the FP32 vectors may round elsewhere, 2^-24 a step over some
    50 steps, 3e-6; 2e-5 of the field is allowed."""
    opts = LinearSolveOptions.defaults(max_iterations=500, relative_tolerance=1e-6, absolute_tolerance=0.0)
    r0, f0 = _project(n, SOLVER_FPCG, 0, opts)
    r1, f1 = _project(n, SOLVER_FPCG, 0, opts, mask=np.zeros((n, n, n), np.uint8))
    assert r0.linear_solve.converged and r1.linear_solve.converged
    assert abs(r0.linear_solve.iterations - r1.linear_solve.iterations) <= 1
    if r0.linear_solve.iterations == r1.linear_solve.iterations:
        for x, y in zip(f0[:3], f1[:3]):
            assert np.abs(x - y).max() <= 2e-5 * np.abs(y).max()
