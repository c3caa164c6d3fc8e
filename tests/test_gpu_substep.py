"""The FP64 substep's estimates and exact rates against the oracle: every
channel state and RyR regime, potentials and concentrations inside and outside
the range where the FP32 estimates of the rates decide (|V| < 150 mV, 0 <
CaSS < 16 mM), FRU counts at the edges of a warp, fixed and packed launches.
Channel states and draws are equal; concentrations differ by the last place
of the exponentials (2^-53 relative) through at most a few hundred substeps:
1e-12."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def random_set(n, seed, ca):
    rng = np.random.default_rng(seed)
    s = O.rest_set(n, "base", 5489 + seed)
    s["ltype"][:, :, 0] = rng.integers(1, 13, (n, 4))
    s["ltype"][:, :, 1] = rng.integers(1, 3, (n, 4))
    s["ryr"][:] = rng.integers(1, 9, (n, 4, 5))
    s["ito2"][:] = rng.integers(1, 3, (n, 4))
    s["mti"][:] = rng.integers(0, 625, n)
    s["mt"][:] = rng.integers(0, 1 << 32, (n, 624), dtype=np.uint32)
    lo, hi = ca
    s["frus"][:, 0] = rng.uniform(0.1, 1.0, n)
    s["frus"][:, 1:] = 10.0 ** rng.uniform(lo, hi, (n, 4))
    return s


@pytest.mark.parametrize("packed", [0, 3])
@pytest.mark.parametrize("n,v,dv,ca,ms", [
    (1, -95.0, 0.3, (-4.2, -3.5), 0.1),
    (7, 10.0, -2.0, (-4.0, -1.3), 0.1),
    (257, -30.0, 60.0, (-4.5, -1.0), 0.05),   # V crosses 0
    (200, 1e-7, 0.0, (-4.0, -1.5), 0.05),     # V = 0 form
    (129, 149.9, 0.3, (-3.0, -1.0), 0.02),    # V leaves the estimates' range
    (64, -160.0, 0.0, (-4.0, -2.0), 0.002),
    (64, 300.0, 10.0, (-4.0, -2.0), 0.01),
    (96, 20.0, 1.0, (-40.0, -29.0), 0.01),    # CaSS below the estimates' range
    (96, 20.0, 1.0, (0.5, 1.5), 0.002),       # and above it
])
def test_substep_matches_oracle(gw, n, v, dv, ca, ms, packed):
    s = random_set(n, n, ca)
    cell = gw.Cell(n)
    if packed:
        cell.set_stage_packing(packed)
    cell.upload(s)
    t0 = 3.0
    for a, b in ((0.0, 0.4), (0.4, 1.0)):
        d0, df = np.array([v + a * dv, 2e-4, 0.6]), np.array([v + b * dv, 2.1e-4, 0.59])
        cell.stage(t0 + a * ms, t0 + b * ms, d0, df)
        O.simfru(s, t0 + a * ms, t0 + b * ms, d0, df)
    got = cell.download()
    for k in ("ltype", "ryr", "ito2", "mti", "mt"):
        np.testing.assert_array_equal(got[k], s[k], err_msg=k)
    np.testing.assert_allclose(got["frus"], s["frus"], rtol=1e-12, atol=0)


@pytest.mark.parametrize("n", [3, 9, 1216, 2433, 3039, 3041])
def test_few_frus_per_warp_match_oracle(gw, n):
    """FP64 launches of two FRUs per warp on sixteen lanes each, and of 8 per
    warp above 3,040 FRUs; in the former the group of 8 is summed by the warp
    that completes it.  The sums over n FRUs of values equal to 1e-12 are
    equal to 1e-12."""
    s = random_set(n, 11 + n, (-4.0, -1.5))
    cell = gw.Cell(n)
    cell.upload(s)
    d0, df = np.array([5.0, 3e-4, 0.5]), np.array([5.4, 3e-4, 0.49])
    for t in (0.0, 0.02, 0.04):
        _, num = cell.stage(t, t + 0.02, d0, df)
        O.simfru(s, t, t + 0.02, d0, df)
        np.testing.assert_allclose(num, O.flux_sums(s), rtol=1e-12)
    got = cell.download()
    for k in ("ltype", "ryr", "ito2", "mti", "mt"):
        np.testing.assert_array_equal(got[k], s[k], err_msg=k)
    np.testing.assert_allclose(got["frus"], s["frus"], rtol=1e-12, atol=0)


@pytest.mark.parametrize("n", [5, 1217, 2433])
def test_mixed_few_frus_per_warp_same_bits(gw, n):
    """Mixed launches with 2, 4 and 8 FRUs per warp (by FRU count) against
    packed ones, whose sums come from the fixed layout: the same bits."""
    s = random_set(n, 23 + n, (-4.0, -1.5))
    d0, df = np.array([5.0, 3e-4, 0.5]), np.array([5.4, 3e-4, 0.49])
    res = []
    for packed in (0, 7):
        cell = gw.Cell(n, precision="mixed")
        if packed:
            cell.set_stage_packing(packed)
        cell.upload(s)
        nums = [cell.stage(t, t + 0.02, d0, df)[1] for t in (0.0, 0.02, 0.04)]
        res.append((nums, cell.download()))
    np.testing.assert_array_equal(res[0][0], res[1][0])
    for k in ("frus", "ltype", "ryr", "ito2", "mti", "mt"):
        np.testing.assert_array_equal(res[0][1][k], res[1][1][k], err_msg=k)
