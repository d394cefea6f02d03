"""What a warp of the tile compositor asks for ahead of a call (ct_ahead) stays inside that call's
run of edges: runs of none (a call without edges in the warp's segment) and the last run of a
pool that is full to its last edge."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from footile_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def ahead(tmp_path_factory):
    d = tmp_path_factory.mktemp("ahead")
    src, lib = d / "ahead.cpp", d / "libahead.so"
    src.write_text('#include "ft_kernels.cuh"\nextern "C" int ahead(int n) { return ftk::ct_ahead(n); }\n')
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.check_call([shutil.which("g++"), "-std=c++17", "-shared", "-fPIC", "-I", cuda, "-I",
                           os.path.join(ROOT, "footile_gb300", "csrc"), str(src), "-o", str(lib)])
    return ctypes.CDLL(str(lib)).ahead


@pytest.mark.parametrize("segs", [1, 2, 4])
def test_asks_for_nothing_past_a_run(ahead, segs):
    rng = np.random.default_rng(segs)
    calls = 200
    n = rng.integers(0, 80, (calls, segs))
    n[rng.random((calls, segs)) < 0.4] = 0
    n[-1, -1] = 0  # the pool's last run is empty: it begins where the pool ends
    first = np.cumsum(n).reshape(calls, segs) - n
    cap = int(n.sum())
    for seg in range(segs):
        for i in range(calls):
            k = ahead(int(n[i, seg]))
            last = first[i, seg] + k - 1
            assert k <= 32 and last < first[i, seg] + n[i, seg] and (k == 0 or last < cap)
            assert k == min(n[i, seg], 32)
