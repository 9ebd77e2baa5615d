"""The bounded waits of the pressure sweeps. With the test hook the first wait
of a launch polls for something that never comes and runs out: the projection
reports VAPOR_RUNTIME_ERROR, and the next one on the same object is right again,
bit for bit."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import random_fields
from vapor_b200.abi import (SOLVER_FPCG, SOLVER_MIXED_REFINEMENT, VAPOR_RUNTIME_ERROR, LinearSolveOptions,
                            ProjectionOptions)

pytestmark = pytest.mark.gpu


def _project(stage, n, opts):
    fields = [np.array(a, np.float32, copy=True) for a in random_fields(n, seed=n)[1:]]
    r, p = stage.project(*fields, ProjectionOptions(0.01, 1.8, opts), 6.0, want_pressure=True)
    return r.linear_solve.iterations, fields + [p]


def _runs_out_and_recovers(n, kind, opts):
    stage = vb.StageBackend(n, 1.0)
    stage.set_solver_kind(kind)
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
