"""What an object costs that is made and not yet used: a kernel's first need for
an attribute loads it to the device, so a workspace that set the attributes of
every sweep variant filled 8 MB and took some 35 ms, also for callers that never
solve. Device memory is what a test can count; each measurement is a process of
its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _megabytes(make):
    code = f"""
import torch
import vapor_b200 as vb
from vapor_b200.mac2d import ReflectionSimulation2D, reflection_app_params
torch.zeros(1, device="cuda")
vb.library()
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
kept = {make}
torch.cuda.synchronize()
print("MB", (before - torch.cuda.mem_get_info()[0]) / 2 ** 20)
kept.close()
"""
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    return float(out.stdout.split("MB")[1].split()[0])


def test_a_workspace_loads_no_sweep_kernels():
    # buffers of 8^3 cells and the streams: at most two granules of 2 MB
    assert _megabytes("vb.StageBackend(8, 1.0)") <= 6.0


def test_2d_limiter_buffers_only_with_the_limiter():
    off, on = [_megabytes(f"ReflectionSimulation2D(512, reflection_app_params({mc}))") for mc in (0, 1)]
    # 20 bytes for each of 16 x 576 x 32 steps of the march: 5.6 MB
    assert on - off >= 4.0


def test_2d_limiter_switched_on_later():
    import numpy as np
    from vapor_b200.mac2d import ReflectionSimulation2D, reflection_app_params
    frames = []
    for first in (1, 0):
        sim = ReflectionSimulation2D(65, reflection_app_params(first))
        if not first:
            sim.params = reflection_app_params(1)
        sim.advance(1 / 60)
        sim.advance(1 / 60)
        frames.append([np.array(a) for a in sim.download()])
        sim.close()
    for a, b in zip(*frames):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
