"""FP64 stages whose membrane potential has no finite GHK factor: every cleft's
LCC flux is a product with it, of closed channels too, so every FRU ends with
NaN -- in the launch of few FRUs, the fixed and the packed one as in the
one-lane kernel, whose products are written out."""
import numpy as np
import pytest

from test_gpu_substep import random_set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,packed", [(64, 0), (3100, 0), (64, 3)])
@pytest.mark.parametrize("v", [1e4, -np.inf, np.inf, np.nan])
def test_potential_without_ghk_factor(gw, v, n, packed):
    s = random_set(n, n, (-4.0, -1.5))
    s["ltype"][:, :, 0] = 1 + s["ltype"][:, :, 0] % 5  # closed states 1 .. 5
    d = np.array([v, 3e-4, 0.5])
    got = []
    for lanes in (1, 4):
        cell = gw.Cell(n, fru_lanes=lanes)
        cell.set_stage_packing(packed if lanes == 4 else 0)
        cell.upload(s)
        cell.stage(0.0, 0.02, d, d)
        got.append(cell.download()["frus"])
        cell.close()
    assert np.isnan(got[0]).all()
    np.testing.assert_array_equal(np.isnan(got[1]), np.isnan(got[0]))
