"""Builds of the stage kernels by load: blocks of several warps take the roomy
and the wide build only while all their warps are resident (8 per SM, as the
builds' registers allow), single-warp blocks up to the measured lines; launches
that do not advance never share a group."""
import os
import subprocess

import pytest

from conftest import ROOT, TBUILD

SMS = 152


@pytest.fixture(scope="module")
def shape():
    os.makedirs(TBUILD, exist_ok=True)
    exe = os.path.join(TBUILD, "stage_shape_check")
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O2", "-std=c++17",
                           "-I" + os.path.join(ROOT, "greenstein2002_gb300", "csrc"), "-o", exe,
                           os.path.join(ROOT, "tests", "native", "stage_shape_check.cpp")])

    def call(groups, warps, advance=1):
        out = subprocess.check_output([exe, str(groups), str(SMS), str(warps), str(advance)], text=True)
        return tuple(int(x) for x in out.split())
    return call


@pytest.mark.parametrize("warps,roomy,wide", [(1, 11, 10), (2, 8, 8), (4, 8, 8), (8, 8, 8)])
def test_builds_by_load(shape, warps, roomy, wide):
    assert [shape(g, warps)[0] for g in (1, roomy * SMS, roomy * SMS + 1, 10000)] == [0, 0, 1, 1]
    assert [shape(g, warps)[1] for g in (1, wide * SMS // 4, wide * SMS // 4 + 1)] == [1, 1, 0]
    assert [shape(g, warps)[2] for g in (1, SMS, SMS + 1, 2 * SMS, 2 * SMS + 1)] == [2, 2, 4, 4, 8]
    assert shape(1, warps, advance=0) == (0, 0, 8)
