"""When the tile rasteriser hands a path over (tile_overflows): as soon as the slots so far foretell
more than its scratch holds, never a path that stays inside at an even rate."""
import ctypes
import os
import shutil
import subprocess

import pytest

from footile_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def overflows(tmp_path_factory):
    d = tmp_path_factory.mktemp("over")
    (d / "o.cpp").write_text('#include "ft_kernels.cuh"\nextern "C" int over(int s, int d, int n, int c) '
                             '{ return ftk::tile_overflows(s, d, n, c); }\n')
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.check_call([shutil.which("g++"), "-std=c++17", "-shared", "-fPIC", "-I", cuda, "-I",
                           os.path.join(ROOT, "footile_gb300", "csrc"), str(d / "o.cpp"), "-o", str(d / "o.so")])
    return ctypes.CDLL(str(d / "o.so")).over


@pytest.mark.parametrize("chunk,cap", [(128, 32768), (512, 65504)])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 512, 513, 3000, 100_000, 2_000_000])
def test_even_paths(overflows, chunk, cap, n):
    for per_op in (1, 4, 16, 33, 200, 4097):
        seen = [(min(c0 + chunk, n), min(c0 + chunk, n) * per_op) for c0 in range(0, n, chunk)]
        first = next((d for d, s in seen if overflows(min(s, 2**31 - 1), d, n, cap)), None)
        # a path that does not fit is handed over with the first ops seen, one that does is not
        assert first == (min(chunk, n) if n * per_op > cap else None), (per_op, first)
