"""Lanes that walk one row of a segment (item_shift): enough for every cell of the walk that is on
the raster, and no more than twice as many, however flat and long the segment is."""
import ctypes
import os
import shutil
import subprocess

import pytest

from footile_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def shift(tmp_path_factory):
    d = tmp_path_factory.mktemp("items")
    (d / "i.cpp").write_text('#include "ft_kernels.cuh"\nextern "C" int shift(int c, int w) { return ftk::item_shift(c, w); }\n')
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.check_call([shutil.which("g++"), "-std=c++17", "-shared", "-fPIC", "-I", cuda, "-I",
                           os.path.join(ROOT, "footile_gb300", "csrc"), str(d / "i.cpp"), "-o", str(d / "i.so")])
    return ctypes.CDLL(str(d / "i.so")).shift


@pytest.mark.parametrize("W", [1, 2, 4, 5, 16, 63, 64, 65, 256, 512, 4096, 65535])
def test_lanes_cover_the_raster_and_little_more(shift, W):
    for cells in [2, 3, 4, 5, 7, 8, 9, 12, 16, 17, 64, 65, 100, 4097, 65538]:
        lanes, on = 1 << shift(cells, W), min(cells, W)
        assert 4 * lanes >= on
        assert lanes == 1 or 4 * lanes < 2 * on + 4
