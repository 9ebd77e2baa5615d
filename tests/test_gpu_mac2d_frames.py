"""Frames of the 2D reflection solver against a NumPy float32 restatement of its
step (no emission, no buoyancy: those draw on the C library's exp and pow),
bit for bit, at the sizes where the limiter's march (warps of 32 rows, chunks of
steps) and the cluster's SOR (slabs of rows, groups of 4 slots, the largest grid
and the first beyond it) can go wrong."""
import numpy as np
import pytest

from vapor_b200.abi import field_shapes_2d
from vapor_b200.mac2d import ReflectionSimulation2D, reflection_app_params

pytestmark = pytest.mark.gpu
F = np.float32


def _axis(p, h, n, staggered):
    g = p / h if staggered else p / h - F(0.5)
    g = np.clip(g, F(0), F(n if staggered else n - 1))
    i0 = np.minimum(g.astype(np.int32), n - 1) if staggered else g.astype(np.int32)
    i1 = i0 + 1 if staggered else np.minimum(i0 + 1, n - 1)
    return i0, i1, g - i0.astype(F)


def _sample(f, n, h, px, py, sx, sy):
    x0, x1, tx = _axis(px, h, n, sx)
    y0, y1, ty = _axis(py, h, n, sy)

    def mix(a, b, t):
        return a + (b - a) * t
    return mix(mix(f[y0, x0], f[y0, x1], tx), mix(f[y1, x0], f[y1, x1], tx), ty)


def _points(n, h, sx, sy):
    x = np.arange(n + sx, dtype=F)
    y = np.arange(n + sy, dtype=F)
    x = x * h if sx else (x + F(0.5)) * h
    y = y * h if sy else (y + F(0.5)) * h
    return np.meshgrid(x, y)


def _trace(n, h, dt, u, v, src, sx, sy, sign):
    px, py = _points(n, h, sx, sy)
    qx = px + sign * (_sample(u, n, h, px, py, 1, 0) * dt)
    qy = py + sign * (_sample(v, n, h, px, py, 0, 1) * dt)
    padx, pady = (F(0) if sx else F(0.5) * h), (F(0) if sy else F(0.5) * h)
    qx = np.clip(qx, padx, F(1) - padx)
    qy = np.clip(qy, pady, F(1) - pady)
    return _sample(src, n, h, qx, qy, sx, sy)


def _smoke(n, h, dt, u, v, smoke, mc):
    fwd = _trace(n, h, dt, u, v, smoke, 0, 0, F(-1))
    if not mc:
        return fwd
    back = _trace(n, h, dt, u, v, fwd, 0, 0, F(1))
    field = smoke.copy()
    for y in range(n):
        ya, yb = max(0, y - 1), min(n, y + 2)
        for x in range(n):
            xa, xb = max(0, x - 1), min(n, x + 2)
            c = fwd[y, x] + F(0.5) * (field[y, x] - back[y, x])
            lo = min(fwd[ya:yb, xa:xb].min(), field[ya:yb, xa:xb].min())
            hi = max(fwd[ya:yb, xa:xb].max(), field[ya:yb, xa:xb].max())
            field[y, x] = lo if c < lo else (hi if hi < c else c)
    return field


def _project(n, h, dt, u, v, omega, iterations):
    u, v = u.copy(), v.copy()
    u[:, 0] = u[:, -1] = 0
    v[0] = v[-1] = 0
    hinv, h2 = F(1) / h, h * h
    div = (u[:, 1:] - u[:, :-1] + v[1:] - v[:-1]) * hinv
    d = div * h2 / dt
    p = np.zeros((n + 2, n + 2), F)
    terms = np.full((n, n), 4, F)
    for edge in (terms[0], terms[-1], terms[:, 0], terms[:, -1]):
        edge -= F(1)
    yy, xx = np.mgrid[0:n, 0:n]
    for _ in range(iterations):
        for parity in (0, 1):
            s = p[1:-1, :-2] + p[1:-1, 2:]
            s = s + p[:-2, 1:-1]
            s = s + p[2:, 1:-1]
            new = (F(1) - omega) * p[1:-1, 1:-1] + omega * (s - d) / np.maximum(terms, F(1))
            p[1:-1, 1:-1] = np.where((xx + yy) % 2 == parity, new, p[1:-1, 1:-1])
    q = p[1:-1, 1:-1]
    u[:, 1:-1] -= dt * (q[:, 1:] - q[:, :-1]) * hinv
    v[1:-1] -= dt * (q[1:] - q[:-1]) * hinv
    u[:, 0] = u[:, -1] = 0
    v[0] = v[-1] = 0
    return u, v, q


def _frame(n, dt, smoke, u, v, par):
    h, dt = F(1) / F(n), F(dt)
    half, its = F(0.5) * dt, max(1, par.project_iterations // 2)
    omega, mc = F(par.sor_omega), par.mac_cormack_smoke
    u[:, 0] = u[:, -1] = 0
    v[0] = v[-1] = 0
    smoke = _smoke(n, h, half, u, v, smoke, mc)
    ut, vt = _trace(n, h, half, u, v, u, 1, 0, F(-1)), _trace(n, h, half, u, v, v, 0, 1, F(-1))
    um, vm, _ = _project(n, h, half, ut, vt, omega, its)
    # the reflection starts from the advected velocity before its walls close
    uh, vh = F(2) * um - ut, F(2) * vm - vt
    smoke = _smoke(n, h, half, um, vm, smoke, mc)
    u, v = _trace(n, h, half, um, vm, uh, 1, 0, F(-1)), _trace(n, h, half, um, vm, vh, 0, 1, F(-1))
    u, v, p = _project(n, h, half, u, v, omega, its)
    return smoke, u, v, p


@pytest.mark.parametrize("mc", [0, 1])
@pytest.mark.parametrize("n", [2, 3, 9, 31, 32, 33, 65, 130, 352, 353])
def test_frames_equal_the_numpy_restatement(n, mc):
    if mc and n > 130:
        pytest.skip("the limiter's restatement is a loop over the cells")
    par = reflection_app_params(mc)
    par.source_strength, par.buoyancy, par.smoke_decay, par.project_iterations = 0.0, 0.0, 0.0, 26
    sim = ReflectionSimulation2D(n, par)
    rng = np.random.default_rng(n)
    smoke, u, v = [(rng.random(s, dtype=F) - F(0.3 * (k > 0))).astype(F) for k, s in enumerate(field_shapes_2d(n))]
    sim.upload(smoke, u, v)
    for _ in range(2):
        sim.advance(1 / 60)
        smoke, u, v, p = _frame(n, 1 / 60, smoke, u.copy(), v.copy(), par)
    for got, want in zip(sim.download(), (smoke, u, v, p)):
        assert np.array_equal(got, want)
    sim.close()
