"""The whole backward pass against a restatement in 64 bits on the CPU, at ragged
sizes, with data for which the device's FP32 sums are exact: small integers,
sparse weights of -1, 0 and 1, so that every stored BF16 value is the rounding of
the same number on both sides, whatever the order of its sum. So the output
head's, bias, pooling and upsampling gradients and the ReLU masks are compared
with something other than themselves."""
import numpy as np
import pytest

import vapor_b200 as vb
from test_gpu_unet import LAYERS, Net

pytestmark = pytest.mark.gpu


def _parameters(rng):
    """Two weights per output channel and layer (one for the centre tap), integer biases."""
    out = []
    for cin, cout in LAYERS:
        w = np.zeros((27, cout, cin), np.float32)
        for co in range(cout):
            w[13, co, rng.integers(cin)] = 1.0
            w[rng.integers(27), co, rng.integers(cin)] = rng.choice([-1.0, 1.0])
        out += [w.reshape(-1), rng.integers(0, 2, cout).astype(np.float32)]
    out += [rng.choice([-1.0, 1.0, 2.0], 16).astype(np.float32), np.ones(1, np.float32)]
    return np.concatenate(out)


def _reference(params, x, g):
    """Gradients in the parameter vector's order, and per block the sum of the
    absolute values of its terms; x (n, n, n, 16), g (n, n, n), both float64."""
    import torch
    import torch.nn.functional as F
    r = lambda t: t.to(torch.bfloat16).to(torch.float64)
    ws, bs, off = [], [], 0
    for cin, cout in LAYERS:
        w = params[off:off + 27 * cout * cin].reshape(27, cout, cin)
        ws.append(torch.tensor(w.transpose(1, 2, 0).reshape(cout, cin, 3, 3, 3).astype(np.float64)))
        off += 27 * cout * cin
        bs.append(torch.tensor(params[off:off + cout].astype(np.float64)))
        off += cout
    head = torch.tensor(params[off:off + 16].astype(np.float64))
    conv = lambda i, t: r(F.relu(F.conv3d(t, ws[i], bs[i], padding=1)))
    up = lambda t: F.interpolate(t, scale_factor=2, mode="nearest")
    spread = lambda t: up(t) / 8
    gather = lambda t: F.avg_pool3d(t, 2) * 8
    e = [None] * 10
    x = torch.tensor(x).permute(3, 0, 1, 2).unsqueeze(0)
    g = torch.tensor(g)[None, None]
    e1a = conv(0, x)
    s1 = conv(1, e1a)
    p1 = r(F.avg_pool3d(s1, 2))
    e2a = conv(2, p1)
    s2 = conv(3, e2a)
    p2 = r(F.avg_pool3d(s2, 2))
    e3a = conv(4, p2)
    e3b = conv(5, e3a)
    dec2 = torch.cat([up(e3b), s2], 1)
    d2a = conv(6, dec2)
    d2b = conv(7, d2a)
    dec1 = torch.cat([up(d2b), s1], 1)
    d1a = conv(8, dec1)
    d1b = conv(9, d1a)
    ins = [x, e1a, p1, e2a, p2, e3a, dec2, d2a, dec1, d1a]
    masked = lambda t, act: torch.where(act > 0, t, torch.zeros_like(t))

    def layer(i, gout, mask=None, need=True):
        cout, cin = ws[i].shape[:2]
        taps = []
        for values, grads in ((ins[i], gout), (ins[i].abs(), gout.abs())):
            padded = F.pad(values, (1,) * 6)[0]
            D, H, W = grads.shape[2:]
            flat = grads[0].reshape(cout, -1)
            taps.append(torch.stack([flat @ padded[:, z:z + D, y:y + H, x0:x0 + W].reshape(cin, -1).T
                                     for z in range(3) for y in range(3) for x0 in range(3)]).reshape(-1).numpy())
        e[i] = (taps[0], gout.sum((0, 2, 3, 4)).numpy(), taps[1], gout.abs().sum((0, 2, 3, 4)).numpy())
        if need:
            dx = r(F.conv_transpose3d(gout, ws[i], padding=1))
            return dx if mask is None else masked(dx, mask)

    g9 = masked(r(g * head.view(1, 16, 1, 1, 1)), d1b)
    gb = layer(9, g9, d1a)
    gdec1 = layer(8, gb)
    gl2b = masked(r(gather(gdec1[:, :32])), d2b)
    gl2 = layer(7, gl2b, d2a)
    gdec2 = layer(6, gl2)
    gl3b = masked(r(gather(gdec2[:, :64])), e3b)
    gl3 = layer(5, gl3b, e3a)
    gs2 = masked(r(gdec2[:, 64:] + spread(layer(4, gl3))), s2)
    gl2 = layer(3, gs2, e2a)
    gs1 = masked(r(gdec1[:, 32:] + spread(layer(2, gl2))), s1)
    ga = layer(1, gs1, e1a)
    layer(0, ga, need=False)
    grads, sizes = [], []
    for w, b, wa, ba in e:
        grads += [w, b]
        sizes += [wa, ba]
    grads += [(d1b * g).sum((0, 2, 3, 4)).numpy(), g.sum().reshape(1).numpy()]
    sizes += [(d1b * g).abs().sum((0, 2, 3, 4)).numpy(), g.abs().sum().reshape(1).numpy()]
    out = (d1b * head.view(1, 16, 1, 1, 1)).sum(1) + float(params[-1])
    return out[0].numpy(), grads, sizes


@pytest.mark.parametrize("n", [8, 12, 20, 36])
def test_backward_pass_equals_64_bits(n):
    """Every term is exact; a sum of N of them in FP32, in any order and tree, is
    off by at most about log2(N) roundings of the sum of their absolute values on
    the tree's paths: 2^-24 x 40 covers 36^3 voxels, whose longest chain here is a
    CTA's stages and one atomic per CTA."""
    import torch
    rng = np.random.default_rng(100 + n)
    net = Net(seed=3)
    params = _parameters(rng)
    assert params.size == net.P
    vb.check(net.lib.vapor_unet_set_parameters(net.h, params.ctypes.data, net.P))
    x = (64.0 * rng.integers(-2, 4, (n, n, n, 16))).astype(np.float32)
    g = (64.0 * rng.integers(-1, 2, (n, n, n))).astype(np.float32)
    xin = torch.tensor(x).to(torch.bfloat16).cuda().contiguous()
    out = torch.zeros(n ** 3, dtype=torch.float32, device="cuda")
    gdev = torch.tensor(g.reshape(-1)).cuda()
    got = np.zeros(net.P, np.float32)
    vb.check(net.lib.vapor_unet_forward_features(net.h, n, xin.data_ptr(), out.data_ptr()))
    vb.check(net.lib.vapor_unet_backward(net.h, n, gdev.data_ptr(), got.ctypes.data))
    want_out, want, sizes = _reference(params, x.astype(np.float64), g.astype(np.float64))
    assert np.array_equal(out.cpu().numpy(), want_out.reshape(-1).astype(np.float32))
    off = 0
    for k, (w, size) in enumerate(zip(want, sizes)):
        have = got[off:off + w.size].astype(np.float64)
        off += w.size
        assert np.abs(w).max() > 0, k
        assert (np.abs(have - w) <= 40 * 2.0 ** -24 * size).all(), (k, np.abs(have - w).max())
    assert off == net.P
