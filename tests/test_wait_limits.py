"""The limits of the tile compositor's waits: work that goes on, however slowly, is waited for;
work that has stopped is given up after the limit of polls."""
import ctypes
import os
import shutil
import subprocess

import pytest

from footile_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include "ft_kernels.cuh"
// polls until the wait gives up (-1: it does not) while the word moves every `every` polls, `moves` times
extern "C" long long gives_up(unsigned limit, unsigned every, unsigned moves) {
    ftk::Patience p;
    unsigned word = 0;
    for (long long k = 1; k <= (long long)every * (moves + 1) + limit; k++) {
        if (k % every == 0 && word < moves) word++;
        if (p.ends(word, limit)) return k;
        if (word == moves && moves && k % every == 0) return -1;
    }
    return -1;
}
extern "C" unsigned limit(int tile) { return tile ? ftk::CT_POLLS_TILE : ftk::CT_POLLS_SMEM; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("wait")
    (d / "w.cpp").write_text(SRC)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.check_call([shutil.which("g++"), "-O1", "-std=c++17", "-shared", "-fPIC", "-I", cuda, "-I",
                           os.path.join(ROOT, "footile_gb300", "csrc"), str(d / "w.cpp"), "-o", str(d / "w.so")])
    so = ctypes.CDLL(str(d / "w.so"))
    so.gives_up.restype, so.limit.restype = ctypes.c_longlong, ctypes.c_uint
    return so


@pytest.mark.parametrize("limit", [1, 2, 1000])
def test_slow_work_is_waited_for(lib, limit):
    assert lib.gives_up(limit, limit, 5000) == -1  # thousands of times the limit in all
    assert lib.gives_up(limit, 1, 5000) == -1


@pytest.mark.parametrize("limit", [1, 2, 1000])
def test_stopped_work_is_given_up(lib, limit):
    assert lib.gives_up(limit, 10**6, 0) == limit + 1


def test_limits_are_many_seconds_of_polls(lib):
    # a poll of another CTA's batch sleeps 200 ns and reads L2 twice; a poll of shared memory takes
    # 30 cycles and more of at most 2.1 GHz
    assert lib.limit(1) * 0.5e-6 > 60 and lib.limit(0) * 30 / 2.1e9 > 30
