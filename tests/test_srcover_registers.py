"""The float SrcOver kernels that take canvases of any size spill nothing: their launch bounds leave the
registers that the loads in flight need.  (The backward's shape of nine CTAs per SM spills; it only
takes canvases that it spares a round.)"""
import os
import re
import subprocess

from footile_gb300 import _build


def test_no_spills(tmp_path):
    cmd = [_build.nvcc()] + _build.GENCODE + _build.NVFLAGS + ["-Xptxas", "-v", "-c", os.path.join(_build.CSRC, "ft_convert.cu"),
                                                              "-o", str(tmp_path / "c.o")]
    out = subprocess.run(cmd, capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    text = out.stdout + out.stderr
    found = re.findall(r"entry function '(\w*k_srcover\w*)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads", text, re.S)
    found = [f for f in found if "Li9E" not in f[0]]
    assert len(found) == 4  # forward by 8 and by 4 layers, backward of some and of all coverage
    assert all(s == "0" and ld == "0" for _, s, ld in found), found
