"""The host's wait for a launch's totals: work that has ended without writing
its number is not taken for a launch with results."""
import os
import subprocess

from conftest import ROOT, TBUILD


def test_wait_ends_with_the_number_or_the_work():
    os.makedirs(TBUILD, exist_ok=True)
    exe = os.path.join(TBUILD, "wait_check")
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "greenstein2002_gb300", "csrc"),
                           "-o", exe, os.path.join(ROOT, "tests", "native", "wait_check.cpp")])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60, check=True).stdout
    assert out.splitlines() == ["there 1 0", "while running 1 3", "with the end 1", "never 0",
                                "next 1 8 1"]
