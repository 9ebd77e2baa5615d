"""A call right after an upload works on all of it. The library's streams do not
wait for the default stream, and a copy from pageable memory returns while its
last part is still on the way: the upload has to be ordered with the stream that
reads it. Many uploads of other fields, each followed at once by a step, against
the same with the device idle in between."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import sphere_mask
from vapor_b200 import mac2d
from vapor_b200.abi import SOLVER_MIXED_REFINEMENT, LinearSolveOptions, ProjectionOptions, field_shapes, field_shapes_2d

pytestmark = pytest.mark.gpu
F = np.float32


def _differences(put, step, inputs):
    import torch
    wrong = 0
    for k, fields in enumerate(inputs):
        other = inputs[(k + 1) % len(inputs)]
        results = []
        for wait in (True, False):
            put(other)
            torch.cuda.synchronize()
            step()
            put(fields)
            if wait:
                torch.cuda.synchronize()
            results.append(step())
        wrong += any(not np.array_equal(a.view(np.uint8), b.view(np.uint8)) for a, b in zip(*results))
    return wrong


def _fields(n, count):
    rng = np.random.default_rng(n)
    return [[rng.random(s, dtype=F) for s in field_shapes_2d(n)] for _ in range(count)]


@pytest.mark.parametrize("n", [353, 512])
def test_2d_reflection_frames(n):
    par = mac2d.reflection_app_params(1)
    par.source_strength, par.project_iterations = 0.0, 2
    sim = mac2d.ReflectionSimulation2D(n, par)

    def step():
        sim.advance(1 / 60)
        return [np.array(a) for a in sim.download()]
    assert _differences(lambda f: sim.upload(*f), step, _fields(n, 40)) == 0
    sim.close()


@pytest.mark.parametrize("n", [256, 1024])
def test_2d_frames(n):
    sim = mac2d.MacSimulation2D(n, 1.0)
    par = sim.params
    par.source_strength = 0.0
    par.project_iterations = 2
    sim.params = par

    def step():
        sim.advance(1 / 60)
        return [np.array(a) for a in sim.download()]
    assert _differences(lambda f: sim.upload(*f), step, _fields(n, 20)) == 0
    sim.close()


def test_masks():
    n = 128
    rng = np.random.default_rng(5)
    velocity = [rng.standard_normal(s).astype(F) for s in field_shapes(n)[1:]]
    masks = [sphere_mask(n, rng.uniform(0.3, 0.7, 3), 0.2) for _ in range(20)]
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(SOLVER_MIXED_REFINEMENT)
    opts = LinearSolveOptions.defaults(max_iterations=8, relative_tolerance=0.0, absolute_tolerance=0.0)

    def step():
        out = [f.copy() for f in velocity]
        stage.project(*out, ProjectionOptions(0.01, 1.7, opts), 6.0)
        return out
    assert _differences(stage.set_solid, step, masks) == 0
    stage.close()
