"""The 2D limiter's march beyond the sizes whose cells a Python loop can visit
(up to 16 warps of 32 rows, ragged last warps and chunks), and its ordered path
(taken when a -0 is among the inputs): frames against a restatement of the in-place
limiter along the wavefronts x + 2 y, bit for bit, signs of zeros included."""
import numpy as np
import pytest

import test_gpu_mac2d_frames as frames
from vapor_b200.abi import field_shapes_2d
from vapor_b200.mac2d import ReflectionSimulation2D, reflection_app_params

pytestmark = pytest.mark.gpu
F = np.float32


def _limited(smoke, fwd, back):
    """field[y, x] = clamp(fwd + (field - back) / 2, bounds of fwd and field over
    the 3x3 cells), in raster order and in place, every comparison as a strict
    one against the bound so far (std::min and std::max keep the first)."""
    n = smoke.shape[0]
    field = smoke.copy()
    for t in range(3 * n - 2):
        y = np.arange(max(0, (t - n + 2) // 2), min(n - 1, t // 2) + 1)
        x = t - 2 * y
        y, x = y[(x >= 0) & (x < n)], x[(x >= 0) & (x < n)]
        fw, fd = fwd[y, x], field[y, x]
        c = fw + F(0.5) * (fd - back[y, x])
        lo, hi = np.where(fw < fd, fw, fd), np.where(fd < fw, fw, fd)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                inside = (x + dx >= 0) & (x + dx < n) & (y + dy >= 0) & (y + dy < n)
                b, a = np.clip(y + dy, 0, n - 1), np.clip(x + dx, 0, n - 1)
                for v in (fwd[b, a], field[b, a]):
                    lo = np.where(inside & (v < lo), v, lo)
                    hi = np.where(inside & (hi < v), v, hi)
        field[y, x] = np.where(c < lo, lo, np.where(hi < c, hi, c))
    return field


def _smoke(n, h, dt, u, v, smoke, mc):
    fwd = frames._trace(n, h, dt, u, v, smoke, 0, 0, F(-1))
    if not mc:
        return fwd
    return _limited(smoke, fwd, frames._trace(n, h, dt, u, v, fwd, 0, 0, F(1)))


def _run(n, smoke, monkeypatch, count=2, still=False):
    monkeypatch.setattr(frames, "_smoke", _smoke)
    par = reflection_app_params(1)
    par.source_strength, par.buoyancy, par.smoke_decay, par.project_iterations = 0.0, 0.0, 0.0, 6
    rng = np.random.default_rng(n)
    u, v = [np.zeros(s, F) if still else (rng.random(s, dtype=F) - F(0.3)) for s in field_shapes_2d(n)[1:]]
    sim = ReflectionSimulation2D(n, par)
    sim.upload(smoke, u, v)
    for _ in range(count):
        sim.advance(1 / 60)
        smoke, u, v, _ = frames._frame(n, 1 / 60, smoke, u.copy(), v.copy(), par)
    got = [np.array(a) for a in sim.download()]
    sim.close()
    assert np.array_equal(got[1], u) and np.array_equal(got[2], v)
    return got[0], smoke


@pytest.mark.parametrize("n", [33, 131, 255, 256, 257, 480, 511, 512])
def test_march(n, monkeypatch):
    rng = np.random.default_rng(2 * n)
    got, want = _run(n, rng.random((n, n), dtype=F), monkeypatch)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("n", [2, 31, 65, 160, 512])
def test_negative_zeros(n, monkeypatch):
    """Zeros of both signs are most of a cell's bounds. In a field that stands
    still a trace returns a -0 as +0, so the field's zeros alone keep theirs."""
    rng = np.random.default_rng(3 * n)
    smoke = np.where(rng.random((n, n)) < 0.2, rng.random((n, n), dtype=F), F(0)).astype(F)
    smoke[(smoke == 0) & (rng.random((n, n)) < 0.4)] = F(-0.0)  # no negative density: the buoyancy takes its root
    for still in (False, True):
        got, want = _run(n, smoke, monkeypatch, count=1, still=still)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))

