"""The FP64 form's fixed-point transforms on the host, against the same DFTs in
double: a line in block fixed point may be no further from extended precision
than one in double is (2-norm, averaged over 24 lines of each kind)."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "ocelot_gb300", "csrc")


@pytest.fixture(scope="module")
def output(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("needs g++")
    exe = str(tmp_path_factory.mktemp("fx") / "fixed_point_lines")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                    os.path.join(REPO, "tests", "host", "fixed_point_lines.cpp"), "-o", exe], check=True)
    return [line.split(",") for line in subprocess.run([exe], check=True, capture_output=True,
                                                       text=True).stdout.splitlines()]


def test_fixed_point_lines_are_no_further_off_than_double_ones(output):
    rows = [r for r in output if len(r) == 5]
    assert len(rows) == 5 * 6 * 5
    for name, kind, length, double, fixed in rows:
        assert float(fixed) <= float(double), (name, kind, length, double, fixed)


def test_conversions_are_exact(output):
    assert output[-1] == ["conversions", "0"]
