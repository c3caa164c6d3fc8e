"""The stage trace measures the launch that the cell runs: with the trace on, a
stage of few FRUs (FP64: sixteen lanes per FRU, mixed: two FRUs per warp) takes
as long as with it off -- the form with eight FRUs per warp takes 14 to 21%
longer -- and the groups' times lie inside the launch."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_traced_launch_is_the_launch(gw, prec):
    n = 250
    rng = np.random.default_rng(5)
    s = O.rest_set(n, "base", 5489)
    s["ltype"][:, :, 0] = rng.integers(1, 7, (n, 4))
    s["ryr"][:] = rng.integers(1, 5, (n, 4, 5))
    s["frus"][:, 1:] = 10 ** rng.uniform(-4.0, -2.0, (n, 4))
    cell = gw.Cell(n, precision=prec)
    cell.upload(s)
    cell.save()
    d0, df = [5.0, 3e-4, 0.5], [5.4, 3e-4, 0.49]
    cell.flux(d0)
    med, num = {}, {}
    for traced in (False, True):
        cell.stage_trace(traced)
        ms = []
        for i in range(21):
            cell.resume()
            cell.profile(True)
            _, num[traced] = cell.stage(0.0, 0.05, d0, df)
            ms.append(cell.profile_read()[0])
        med[traced] = np.median(ms)
    sub, ns = cell.stage_trace_read()
    ns = ns.astype(np.int64)
    print(prec, med)
    assert med[True] < 1.06 * med[False]
    np.testing.assert_array_equal(num[True], num[False])
    assert sub.min() >= 1 and ns.shape == ((n + 7) // 8, 2)
    assert (ns[:, 0] < ns[:, 1]).all()
    assert (ns.max() - ns.min()) * 1e-6 < 1.02 * ms[-1]
