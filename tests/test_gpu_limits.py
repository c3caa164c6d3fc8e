"""The substep limit (2^22 substeps of an FRU in one stage) as an error that
ends with the call: a stage over [0, 1e9) ms, whose substeps are at most 0.01
ms, runs into it.  No fault is involved and the state stays finite.  The call
reports it, cells beside it are not touched, and the next call on the same
cell, from an uploaded state, gives the bits of a fresh cell."""
import numpy as np
import pytest

from test_gpu_batch import _cells

pytestmark = pytest.mark.gpu


def _long(gw):
    return gw.settings(time_step=1e9, step_max=1e9)


def _alone(gw, run, size, first):
    cells, sets, states = _cells(gw, [size], "mixed", first=first)
    t, old = np.zeros(1), np.full(1, 0.1)
    run(cells, sets, t, states, old, 2)
    return states[0], cells[0].download()


def _same(a, b):
    np.testing.assert_array_equal(a[0], b[0])
    for k in b[1]:
        np.testing.assert_array_equal(a[1][k], b[1][k], err_msg=k)


def test_device_runner_runs_again_after_the_limit(gw):
    cells, sets, states = _cells(gw, [2], "mixed")
    s0, st0 = cells[0].download(), states.copy()
    with pytest.raises(gw.GWError, match="substep limit"):
        gw.run_device(cells, [_long(gw)], np.zeros(1), states, np.full(1, 1e9), 1)
    cells[0].upload(s0)
    states[:] = st0
    gw.run_device(cells, sets, np.zeros(1), states, np.full(1, 0.1), 2)
    _same((states[0], cells[0].download()), _alone(gw, gw.run_device, 2, 0))


def test_lockstep_batch_keeps_the_limit_to_its_cell(gw):
    sizes = [2, 40, 25]
    b = gw.Batch("mixed")
    cells, sets, states = _cells(gw, sizes, "mixed")
    s0, st0 = cells[0].download(), states[0].copy()
    t = np.zeros(3)
    with pytest.raises(gw.GWError, match="cell 0.*substep limit"):
        b.run(cells, [_long(gw)] + sets[1:], t, states, np.array([1e9, 0.1, 0.1]), 2)
    assert t[1] == 2 and t[2] == 2
    want = [_alone(gw, gw.Batch("mixed").run, n, i) for i, n in enumerate(sizes)]
    for i in (1, 2):
        _same((states[i], cells[i].download()), want[i])
    cells[0].upload(s0)
    states[0] = st0
    t0, old = np.zeros(1), np.full(1, 0.1)
    b.run(cells[:1], sets[:1], t0, states[:1], old, 2)
    _same((states[0], cells[0].download()), want[0])


@pytest.mark.parametrize("packed", [0, 1])
def test_limit_is_reported_by_its_own_stage(gw, packed):
    """The flag is stored before the launch's number, which ends the wait."""
    dep = np.array([-80.0, 1e-4, 0.5])
    cells, _, _ = _cells(gw, [2, 2], "mixed")
    cells[1].upload(cells[0].download())
    s0 = cells[0].download()
    for c in cells:
        c.set_stage_packing(packed)
    with pytest.raises(gw.GWError, match="substep limit"):
        cells[0].stage(0.0, 1e9, dep, dep)
    cells[0].upload(s0)
    for t in (0.0, 0.02):
        a, b = (c.stage(t, t + 0.02, dep, dep) for c in cells)
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])
    a, b = (c.download() for c in cells)
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def test_stages_after_a_stopped_persistent_run(gw):
    """The tickets of a persistent run that the wait limit ended are reset on
    the cell's own stream, so the next stages sum every group."""
    dep = np.array([-80.0, 1e-4, 0.5])
    cells, sets, _ = _cells(gw, [500, 500], "fp64")
    s0 = cells[1].download()
    assert gw.persist_watchdog(cells[0], sets[0], 0.1) == 3
    for c in cells:
        c.upload(s0)
    for t in (0.0, 0.02):
        a, b = (c.stage(t, t + 0.02, dep, dep) for c in cells)
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])
