"""The backward pass' kernels at ragged sizes: weight gradients whose last
voxel stage is partly empty, and input gradients on the TMA-fed plane-window
convolution with the ReLU mask in its epilogue, against the CUDA-core weight
gradient and the block-synchronous convolution on the same forward pass."""
import numpy as np
import pytest

import vapor_b200 as vb
from test_gpu_unet import LAYERS, Net, features

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 12, 20, 36, 64])
def test_backward_kernels_agree_at_ragged_sizes(n):
    """Both sides add FP32 products of the same BF16 values (the one-chunk
    input gradients in the same order, so the BF16 gradients are the same);
    sums of a few thousand terms per CTA in another order differ by about
    2^-24 sqrt(4096) = 4e-6 of the sum, and by 2e-5 at the most."""
    import torch
    net = Net(seed=23)
    xin = torch.tensor(features(n, 31)).to(torch.bfloat16).cuda().contiguous()
    out = torch.zeros(n ** 3, dtype=torch.float32, device="cuda")
    g = torch.tensor(np.random.default_rng(6).standard_normal(n ** 3).astype(np.float32)).cuda()
    vb.check(net.lib.vapor_unet_forward_features(net.h, n, xin.data_ptr(), out.data_ptr()))
    grads = []
    try:
        for conv, wgrad in ((0, 0), (vb.DEFAULT_CONV_KERNEL, 1)):
            vb.tune_conv_kernel(conv)
            vb.tune_wgrad_kernel(wgrad)
            gp = np.zeros(net.P, np.float32)
            vb.check(net.lib.vapor_unet_backward(net.h, n, g.data_ptr(), gp.ctypes.data))
            grads.append(gp)
    finally:
        vb.tune_conv_kernel(vb.DEFAULT_CONV_KERNEL)
        vb.tune_wgrad_kernel(1)
    a, b = grads
    off = 0
    for cin, cout in LAYERS:
        for size in (27 * cout * cin, cout):
            s = slice(off, off + size)
            off += size
            assert np.abs(a[s]).max() > 0
            assert np.abs(a[s] - b[s]).max() <= 2e-5 * float(np.abs(a[s]).max()), (cin, cout, size)
    assert np.abs(a[off:] - b[off:]).max() <= 2e-5 * float(np.abs(a[off:]).max())
