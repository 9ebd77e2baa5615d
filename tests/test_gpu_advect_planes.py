"""Transport with several planes per thread, cached traced velocities and the
corrected-quotient division against the oracle, bit for bit: grids whose last
chunk of planes or last block is ragged, cell sizes that are and are not powers
of two, and cell sizes and time steps at which the quotients leave the range of
the corrected division."""
import numpy as np
import pytest

import vapor_b200 as vb
from oracle_lib import oracle_advect, random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mc", [0, 1])
@pytest.mark.parametrize("n,box,dt", [(2, 1.0, 0.1), (33, 4.5, 0.2), (84, 1.0, 0.02), (97, 4.5, 0.1), (128, 1.0, 0.01),
                                      (137, 3.3, 0.05), (24, 1e-12, 1e-14), (24, 1e13, 1e12), (33, 1.0, 1e-25)])
def test_planes_and_divisions(n, box, dt, mc):
    d, u, v, w = [np.asarray(a, np.float32) for a in random_fields(n, seed=300 + n, scale=0.8)]
    stage = vb.StageBackend(n, box)
    method = vb.abi.MACCORMACK if mc else vb.abi.SEMI_LAGRANGIAN
    for loc, src in enumerate((d, u, v, w)):
        want = oracle_advect(n, box, loc, dt, 3.0, mc, src, u, v, w)
        for _ in range(2):
            out = np.array(src, np.float32, copy=True) if loc == 0 else np.zeros_like(src)
            if loc == 0:
                stage.advect_scalar(dt, 3.0, method, out, [u, v, w])
            else:
                stage.advect_face(loc - 1, dt, 3.0, method, src, [u, v, w], out)
            assert np.array_equal(out.view(np.uint32), np.asarray(want, np.float32).view(np.uint32)), loc
    stage.close()

