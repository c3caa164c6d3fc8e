"""The currents of a launch's totals, formed one per lane, against the plain
expressions of the one-lane kernel: the same bits, also for infinite and
vanishing operands and the sign of a zero."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

INF = np.inf


@pytest.mark.parametrize("v", [-80.0, 20.0, 1e-7, -1e-6, 499.0, 501.0])
@pytest.mark.parametrize("cai,cansr,cass", [(1e-4, 0.5, None), (INF, 0.5, None), (-INF, 0.5, None), (1e-4, INF, None),
                                            (1e-4, 0.5, INF), (1e300, 1e-300, None), (5e-324, 0.0, 0.0)])
@pytest.mark.parametrize("channels", ["closed", "open"])
def test_currents_of_any_operands(gw, v, cai, cansr, cass, channels):
    n = 24
    s = O.rest_set(n, "base", 5489)
    s["ito2"][:] = 2 if channels == "open" else 1
    s["ltype"][:, :, 0] = 6 if channels == "open" else 1
    if cass is not None:
        s["frus"][3, 2] = cass
    got = []
    for lanes, prec in ((1, "fp64"), (4, "fp64"), (4, "mixed")):
        cell = gw.Cell(n, fru_lanes=lanes, precision=prec)
        cell.upload(s)
        got.append(cell.flux(np.array([v, cai, cansr])))
        cell.close()
    one, four, mixed = got
    np.testing.assert_array_equal(one[0], four[0])
    np.testing.assert_array_equal(np.signbit(one[0]), np.signbit(four[0]))
    np.testing.assert_array_equal(one[1], four[1])
    # the mixed unit fuses the products of a difference: one rounding less of
    # operands that cancel by at most a factor of 1,000
    np.testing.assert_allclose(mixed[0], one[0], rtol=1e-12, atol=0)
