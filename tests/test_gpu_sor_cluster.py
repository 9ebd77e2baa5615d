"""The resident sweeps of small grids (one cluster) and medium grids (the whole
device) against the oracle, which is pinned to the reference's CPU SOR: bit for
bit, with the same iteration counts and residuals, at the sizes where a split
can go wrong (one plane per CTA, slabs and row blocks of unequal size, padded
and odd rows, the largest grid of each form and the first beyond it), for one
divisor and a divisor per diagonal, and for right-hand sides whose quotients
leave the range of the two-product division."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import oracle_project, random_fields, sphere_mask
from vapor_b200.abi import (SOLVER_MIXED_REFINEMENT, SOLVER_RED_BLACK_SOR, LinearSolveOptions, ProjectionOptions)

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 7, 16, 17, 24, 31, 33, 45, 49, 50, 61, 64, 65, 72, 97, 128, 129]


def _both(n, kind, opts, floor, scale=1.0, mask=None, omega=1.7):
    fields = [np.asarray(a) * np.float32(scale) for a in random_fields(n, seed=40 + n)[1:]]
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(kind)
    if mask is not None:
        stage.set_solid(mask)
    got = [np.array(a, np.float32, copy=True) for a in fields]
    r, p = stage.project(*got, ProjectionOptions(0.01, omega, opts), floor, want_pressure=True)
    stage.close()
    st, ro, *want = oracle_project(n, 1.0, *fields, 0.01, omega, floor, opts, solver_kind=kind, solid=mask)
    assert st == 0
    return r, got + [p], ro, want


def _same(r, got, ro, want):
    a, b = r.linear_solve, ro.linear_solve
    assert a.iterations == b.iterations and a.converged == b.converged
    assert a.initial_residual == b.initial_residual
    # The means are FP64 sums in another order: where the float that is
    # subtracted is another one, the fields differ by its rounding.
    if np.float32(r.removed_rhs_mean) == np.float32(ro.removed_rhs_mean):
        for x, y in zip(got[:3], want[:3]):
            assert np.abs(x - y).max() <= 2e-6 * max(np.abs(y).max(), 1e-37)
    return np.float32(r.removed_rhs_mean) == np.float32(ro.removed_rhs_mean)


def _bits(got, want):
    for x, y in zip(got, want):
        assert np.array_equal(np.ascontiguousarray(x).view(np.uint32), np.ascontiguousarray(y).view(np.uint32))


@pytest.mark.parametrize("floor", [6.0, 0.0, 5.5, 7.25])
@pytest.mark.parametrize("n", SIZES)
def test_fixed_budget(n, floor):
    opts = LinearSolveOptions.defaults(max_iterations=21, fixed_iterations=1)
    r, got, ro, want = _both(n, SOLVER_RED_BLACK_SOR, opts, floor)
    if _same(r, got, ro, want):
        assert r.linear_solve.final_residual == ro.linear_solve.final_residual
        _bits(got, want)


@pytest.mark.parametrize("scale", [1e-30, 1e-33, 1e-36, 1e25])
def test_quotients_outside_the_two_product_range(scale):
    opts = LinearSolveOptions.defaults(max_iterations=30, fixed_iterations=1, absolute_tolerance=0.0)
    for floor in (6.0, 0.0):
        r, got, ro, want = _both(24, SOLVER_RED_BLACK_SOR, opts, floor, scale)
        if _same(r, got, ro, want):
            _bits(got, want)


@pytest.mark.parametrize("n", SIZES)
def test_tolerance_driven(n):
    for interval, floor in ((8, 6.0), (3, 0.0)):
        opts = LinearSolveOptions.defaults(max_iterations=100, residual_check_interval=interval,
                                           relative_tolerance=1e-3, absolute_tolerance=0.0)
        r, got, ro, want = _both(n, SOLVER_RED_BLACK_SOR, opts, floor)
        if _same(r, got, ro, want):
            assert r.linear_solve.final_residual == ro.linear_solve.final_residual
            _bits(got, want)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [n for n in SIZES if n > 3])
def test_mixed_refinement(n, masked):
    """Iteration counts and the FP64 residual are the oracle's; the fields
    agree to FP32 rounding (the FP64 pressure mean is a tree sum here)."""
    mask = sphere_mask(n, (0.45, 0.55, 0.5), 0.2) if masked else None
    for interval in (8, 5):
        opts = LinearSolveOptions.defaults(max_iterations=400, residual_check_interval=interval,
                                           relative_tolerance=1e-5, absolute_tolerance=0.0)
        r, got, ro, want = _both(n, SOLVER_MIXED_REFINEMENT, opts, 6.0, mask=mask)
        if _same(r, got, ro, want):
            assert r.linear_solve.final_residual == pytest.approx(ro.linear_solve.final_residual, rel=1e-9)


@pytest.mark.parametrize("n", [33, 64, 80])
def test_a_graph_step_equals_the_eager_step(n):
    """The recorded step (fixed budget, tolerance and mixed loops) gives the
    bits of the same launches issued one by one."""
    for kind, fixed in ((SOLVER_RED_BLACK_SOR, 1), (SOLVER_RED_BLACK_SOR, 0), (SOLVER_MIXED_REFINEMENT, 0)):
        out = []
        for timing in (False, True):
            p = vb.default_params()
            p.reflection, p.use_solve_options, p.solver_kind = 1, 1, kind
            p.solve = LinearSolveOptions.defaults(max_iterations=60, fixed_iterations=fixed, relative_tolerance=1e-4)
            sim = vb.MacSimulation3D(n, 1.0, p)
            sim.set_timing(timing)  # eager
            for _ in range(3):
                sim.advance(1 / 60)
            out.append(sim.download() + [np.array([sim.total_iterations()], np.float32)])
            sim.close()
        _bits(*out)


def test_scenes_of_one_batch_share_the_device():
    """Cluster and device-wide sweeps of one batch's scenes, on the split for
    scenes that share the device, give each scene the bits of its own steps."""
    sizes = (64, 96, 72, 33, 96)

    def make():
        sims = []
        for k, n in enumerate(sizes):
            p = vb.default_params()
            p.use_solve_options, p.solver_kind = 1, SOLVER_MIXED_REFINEMENT if k % 2 else SOLVER_RED_BLACK_SOR
            p.solve = LinearSolveOptions.defaults(max_iterations=120, fixed_iterations=0, relative_tolerance=1e-5)
            sims.append(vb.MacSimulation3D(n, 1.0, p))
        return sims

    alone, together = make(), make()
    batch = vb.Batch(together)
    for _ in range(3):
        batch.advance(1 / 60)
        for s in alone:
            s.advance(1 / 60)
    batch.synchronize()
    for a, b in zip(alone, together):
        assert a.total_iterations() == b.total_iterations()
        _bits(a.download(), b.download())
    batch.close()
