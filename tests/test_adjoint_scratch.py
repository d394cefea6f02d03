"""Scratch of a fill's coverage adjoint, which every Adjoint holds for some 450 CTAs: what a path of
the most vertices needs and no more (24 bytes a vertex, the binned edges and the bands' offsets)."""
import os
import shutil
import subprocess

from footile_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scratch_per_cta(tmp_path):
    src, exe = tmp_path / "s.cpp", tmp_path / "s"
    src.write_text('#include <cstdio>\n#include "ft_adjoint.cuh"\nusing namespace fta;\n'
                   'int main() { std::printf("%zu %zu %d %d %d\\n", A_SCRATCH_PER_CTA, AS_VNODE, VCAP, PAIR_CAP, NB_CAP); }\n')
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.check_call([shutil.which("g++"), "-std=c++17", "-I", cuda, "-I",
                           os.path.join(ROOT, "footile_gb300", "csrc"), str(src), "-o", str(exe)])
    per_cta, strokes_from, vcap, pairs, bands = (int(v) for v in subprocess.check_output([str(exe)]).split())
    assert per_cta <= 24 * vcap + 4 * pairs + 4 * (bands + 1) + 256 * 6  # arrays start on 256 bytes
    assert strokes_from == per_cta
