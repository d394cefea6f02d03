"""Rasters of no columns may have any number of rows: there is nothing to draw, but the pen width
after the call is the path's."""
import ctypes

import pytest

from footile_gb300 import _abi
from footile_gb300.path import PathOp, ops_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stroke", [False, True])
@pytest.mark.parametrize("h", [0, 1, 3000, (1 << 31) - 1, 1 << 31, (1 << 32) - 1])
def test_no_columns(ctx, h, stroke):
    ctx.set_pen_width(1.0)
    ops = ops_array([PathOp.PenWidth(3.5), PathOp.Move(1.0, 1.0), PathOp.Line(5.0, 2.0), PathOp.Line(2.0, 7.0)])
    clr = (ctypes.c_uint8 * 4)(1, 2, 3, 255)
    args = (ops.ctypes.data_as(ctypes.c_void_p), len(ops), _abi.RGBA8P, clr, None, 0, h, 0, _abi.HOST)
    rc = ctx.L.ft_stroke(ctx.h, *args) if stroke else ctx.L.ft_fill(ctx.h, _abi.NONZERO, *args)
    assert rc == 0
    width = ctypes.c_float(0)
    assert ctx.L.ft_get_pen_width(ctx.h, ctypes.byref(width)) == 0 and width.value == 3.5
