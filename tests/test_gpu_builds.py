"""Every build and shape of the stage kernels gives the same bits, at FRU counts
on either side of the lines between them (152 SMs; FRUs of the wide FP64 launch
up to 3,040, of the roomy one up to 13,376 with single-warp blocks and 9,728 with
larger ones, the dense one beyond): 1, 2, 4 and 8 warps per block, packed, and
one lane per FRU."""
import numpy as np
import pytest

from test_gpu_substep import random_set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [2433, 4001, 9737, 13385])
def test_builds_same_bits(gw, n, prec):
    s = random_set(n, 31 + n, (-4.0, -1.5))
    d0, df = np.array([5.0, 3e-4, 0.5]), np.array([5.4, 3e-4, 0.49])
    shapes = [(4, 1, 0), (4, 2, 0), (4, 4, 0), (4, 8, 0), (4, 1, (n + 15) // 16)]
    if prec == "fp64":
        shapes.append((1, 1, 0))
    ref = None
    for lanes, warps, packed in shapes:
        cell = gw.Cell(n, precision=prec, fru_lanes=lanes, stage_warps=warps)
        cell.set_stage_packing(packed)
        cell.upload(s)
        sums = np.concatenate([np.concatenate(cell.stage(t, t + 0.02, d0, df)) for t in (0.0, 0.02, 0.04)])
        got = cell.download()
        cell.close()
        if ref is None:
            ref = sums, got
        what = "lanes %d warps %d packed %d" % (lanes, warps, packed)
        np.testing.assert_array_equal(sums, ref[0], err_msg=what)
        for k in got:
            np.testing.assert_array_equal(got[k], ref[1][k], err_msg="%s %s" % (k, what))
