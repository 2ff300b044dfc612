"""Priority of the screened form's side streams (ct_internal.h: side_stream_priority), compiled on the host:
one level above the call's stream, never past the device's greatest, whatever the caller's level."""
import subprocess
from pathlib import Path

import pytest

from covertreex_gb300 import _build

PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "ct_internal.h"
int main(int, char** a) { printf("%d", ct::side_stream_priority(atoi(a[1]), atoi(a[2]))); }
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = tmp_path_factory.mktemp("prio")
    (out / "p.cc").write_text(PROGRAM)
    include = Path(_build.nvcc_path()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", f"-I{_build.CSRC}", f"-I{include}", "p.cc", "-o", "p"], cwd=out, check=True)
    return str(out / "p")


@pytest.mark.parametrize("call,greatest,side", [(0, -5, -1), (-1, -5, -2), (-4, -5, -5), (-5, -5, -5), (0, 0, 0)])
def test_side_streams_are_one_level_above_the_call(program, call, greatest, side):
    got = subprocess.run([program, str(call), str(greatest)], capture_output=True, text=True, check=True)
    assert int(got.stdout) == side
