"""The resident sweeps against one launch per colour, which runs in their place
where the device cannot hold their kernels (a cluster of 16 SMs, or a CTA on
every SM): the same device sums feed both, so counts, residuals and fields agree
bit for bit in every mode, with one divisor and a divisor per diagonal, with an
obstacle, and beyond the range of the two-product division."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import random_fields, sphere_mask
from vapor_b200 import mac2d
from vapor_b200.abi import SOLVER_MIXED_REFINEMENT, SOLVER_RED_BLACK_SOR, LinearSolveOptions, ProjectionOptions, \
    field_shapes_2d

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 7, 16, 17, 31, 33, 43, 45, 48, 49, 50, 52, 61, 64, 65, 72, 97, 99, 104, 128]


def _projections(n, kind, opts, floor, scale=1.0, mask=None):
    """The same projection with the resident sweeps and without, and the launches of each."""
    fields = [np.asarray(a, np.float32) * np.float32(scale) for a in random_fields(n, seed=70 + n)[1:]]
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(kind)
    if mask is not None:
        stage.set_solid(mask)
    out = []
    for enabled in (1, 0):
        vb.check(vb.library().vapor_stage_set_resident_sweeps(stage._h, enabled))
        got = [f.copy() for f in fields]
        before = vb.kernel_launch_count()
        r, p = stage.project(*got, ProjectionOptions(0.01, 1.7, opts), floor, want_pressure=True)
        out.append((r.linear_solve, got + [p], vb.kernel_launch_count() - before))
    stage.close()
    return out


def _same(out, fewer_launches=True):
    (a, x, la), (b, y, lb) = out
    assert la < lb or not fewer_launches
    assert (a.iterations, a.converged, a.initial_residual, a.final_residual) == \
        (b.iterations, b.converged, b.initial_residual, b.final_residual)
    for f, g in zip(x, y):
        assert np.array_equal(f.view(np.uint32), g.view(np.uint32))


@pytest.mark.parametrize("floor", [6.0, 0.0, 5.5])
@pytest.mark.parametrize("n", SIZES)
def test_reference_sweeps(n, floor):
    for fixed, interval, tolerance in ((1, 8, 1e-3), (0, 8, 1e-3), (0, 3, 0.0)):
        opts = LinearSolveOptions.defaults(max_iterations=43, fixed_iterations=fixed, residual_check_interval=interval,
                                           relative_tolerance=tolerance, absolute_tolerance=0.0)
        _same(_projections(n, SOLVER_RED_BLACK_SOR, opts, floor))


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [n for n in SIZES if n > 3])
def test_mixed_refinement(n, masked):
    mask = sphere_mask(n, (0.45, 0.55, 0.5), 0.2) if masked else None
    for interval, floor in ((8, 6.0), (5, 0.0)):
        opts = LinearSolveOptions.defaults(max_iterations=203, residual_check_interval=interval,
                                           relative_tolerance=1e-6, absolute_tolerance=0.0)
        _same(_projections(n, SOLVER_MIXED_REFINEMENT, opts, floor, mask=mask))


@pytest.mark.parametrize("scale", [1e-30, 1e-33, 1e-36, 1e25])
@pytest.mark.parametrize("n", [24, 96])
def test_beyond_the_two_product_range(n, scale):
    opts = LinearSolveOptions.defaults(max_iterations=30, fixed_iterations=1, absolute_tolerance=0.0)
    for floor in (6.0, 0.0):
        _same(_projections(n, SOLVER_RED_BLACK_SOR, opts, floor, scale))


@pytest.mark.parametrize("mc", [0, 1])
@pytest.mark.parametrize("n", [2, 9, 32, 130, 352, 353])
def test_2d_frames(n, mc):
    frames = []
    for enabled in (1, 0):
        sim = mac2d.ReflectionSimulation2D(n, mac2d.reflection_app_params(mc))
        vb.check(vb.library().vapor_mac2d_refl_set_resident_sweeps(sim._h, enabled))
        rng = np.random.default_rng(n)
        sim.upload(*[rng.random(s, dtype=np.float32) for s in field_shapes_2d(n)])
        for _ in range(2):
            sim.advance(1 / 60)
        frames.append([np.array(a) for a in sim.download()])
        sim.close()
    for a, b in zip(*frames):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
