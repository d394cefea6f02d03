"""Row ranges of a single small call (single_rows): they cover the canvas, none is below eight rows
but the last, and never are there more of them than SMs."""
import ctypes
import os
import shutil
import subprocess

import pytest

from footile_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    (d / "r.cpp").write_text('#include "ft_kernels.cuh"\nextern "C" int rows(int h, int s) { return ftk::single_rows(h, s); }\n')
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.check_call([shutil.which("g++"), "-std=c++17", "-shared", "-fPIC", "-I", cuda, "-I",
                           os.path.join(ROOT, "footile_gb300", "csrc"), str(d / "r.cpp"), "-o", str(d / "r.so")])
    return ctypes.CDLL(str(d / "r.so")).rows


@pytest.mark.parametrize("sms", [0, 1, 2, 132, 152])
@pytest.mark.parametrize("h", [1, 7, 8, 9, 61, 256, 1215, 1216, 1217, 2000, 16000, 1 << 20])
def test_ranges(rows, h, sms):
    r = rows(h, sms)
    n = -(-h // r)
    assert r >= 8 and n * r >= h and n <= max(sms, 1) and (r == 8 or r <= -(-h // max(sms, 1)))
