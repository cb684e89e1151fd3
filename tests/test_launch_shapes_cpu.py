"""Launch shapes of the element-wise and pooling kernels (host arithmetic only, no GPU)."""
import ctypes as C
import itertools
import re
import subprocess

import pytest

from geeps_b200 import _native
from geeps_b200.ops import _lib as L


def test_average_pooling_blocks_cover_the_rows_and_are_full():
    for Cc, width, rows, group in itertools.product((8, 24, 96, 576, 1024, 2048, 2056), (1, 2, 4, 5, 7, 13, 14, 56, 224, 257, 513),
                                                    (1, 2, 5, 64, 448, 2560), (0, 1)):
        out = (C.c_int * 5)()
        L.lib().geeps_avgpool_blocks(Cc, width, C.c_longlong(rows), group, out)
        gx, gy, bx, by, bz = out
        assert bx == min(Cc // 8, 256) and bx * by * bz <= 256 and 1 <= bz <= (64 if group else 1)
        assert gx * bz >= rows and (gx - 1) * bz < rows              # every row once, no empty block
        assert gy * by >= width and (gy - 1) * by < width            # every pixel once, no empty block
        # threads that have a pixel, of all in the launched warps, where there is work for more than one block
        if rows * width * bx >= 512 and (group or width * bx >= 16):
            launched = gx * gy * -(-bx * by * bz // 32) * 32
            assert rows * width * bx >= 0.5 * launched, (Cc, width, rows, list(out))


def test_average_pooling_of_nothing_and_of_very_wide_rows():
    out = (C.c_int * 5)()
    for Cc, width, rows in ((64, 7, 0), (64, 0, 7), (0, 7, 7)):
        L.lib().geeps_avgpool_blocks(Cc, width, C.c_longlong(rows), 1, out)
        assert (out[0] == 0) == (width * rows == 0)
    L.lib().geeps_avgpool_blocks(2048, 70000, C.c_longlong(3), 1, out)
    assert list(out) == [3, 65535, 256, 1, 1]                        # the second grid dimension has 16 bits


@pytest.mark.parametrize("which,per_sm,floats", [(0, 2, 2), (1, 2, 1), (2, 2, 0), (3, 4, 1)])
def test_channel_blocks_cover_the_matrix_and_spread_few_pixels(which, per_sm, floats):
    """The grids that the passes launch; floats: per channel and pixel row in shared memory."""
    for P, Cc in itertools.product((1, 3, 8, 32, 49, 100, 392, 1568, 20000, 100352, 1000000),
                                   (8, 24, 64, 192, 576, 1000, 1024, 1032, 1288, 1536, 2040, 2048, 2056, 4096, 8192)):
        out = (C.c_int * 4)()
        assert L.lib().geeps_channel_pass_blocks(which, C.c_longlong(P), Cc, out) == 0
        cols, blocks, threads, smem = out
        cv = Cc // 8
        cvb = -(-cv // cols)                          # slots of a block, as the kernels compute them
        rows = threads // cvb
        assert threads % 32 == 0 and threads <= 256 and rows >= 1 and (cols - 1) * cvb < cv
        # sums of the pixel rows, or four constants a channel
        assert smem == (rows * cvb * 8 * floats * 4 if floats else cvb * 8 * 4 * 4) and smem <= 32 * 1024
        assert cols * blocks <= 148 * per_sm
        one = 148 // cols
        assert which == 3 or blocks <= one or blocks >= 2 * one, (P, Cc, list(out))      # no SM with two where others have one
        assert rows * cv >= 0.75 * cols * threads, (P, Cc, list(out))         # threads with a slot
        # few pixels: an eighth of the SMs at least, or a block for every batch of rows
        assert cols * blocks >= min(148 // 8, cols * -(-P // rows)), (P, Cc, list(out))
        if which == 0:
            same = (C.c_int * 4)()
            L.lib().geeps_channel_blocks(C.c_longlong(P), Cc, same)
            assert list(same) == list(out)


def test_channel_blocks_of_an_unknown_pass_are_refused():
    out = (C.c_int * 4)()
    assert L.lib().geeps_channel_pass_blocks(4, C.c_longlong(1), 8, out) != 0 and L.lib().geeps_channel_pass_blocks(-1, C.c_longlong(1), 8, out) != 0


def test_lrn_backward_lanes_fit_the_channels():
    for cv, pixels in itertools.product(range(1, 65), (1, 700, 40000, 200000)):
        lp, nv = C.c_int(), C.c_int()
        L.lib().geeps_lrn_lanes(cv * 8, C.c_longlong(pixels), C.byref(lp), C.byref(nv))
        lp, nv = lp.value, nv.value
        # the splits that the kernel is compiled for
        assert (lp, nv) in ((1, 1), (2, 1), (2, 3), (4, 1), (4, 2), (4, 3), (8, 2), (8, 3), (16, 2), (16, 3), (32, 2))
        assert lp * nv >= cv
        assert pixels < 40000 or 3 * cv >= 2 * lp * nv, (cv, lp, nv)


def test_channel_kernels_keep_to_registers_at_their_launch_bounds():
    """What the compiler printed for the kernels whose blocks per SM are set by launch bounds: no spills."""
    names = ("channel_reduce_kernel|bn_backward_kernel|bn_apply_fused_kernel|lrn_maxpool_forward_kernel|lrn_maxpool_backward_quad_kernel|"
             "avgpool3_kernel")
    found = re.findall(rf"entry function '\w*?({names})(\w*)'.*?(\d+) bytes spill stores", _native.ptxas_report(), re.S)
    if not found:
        pytest.skip("no compiler output here: the library was built elsewhere")
    assert len(found) >= 16 and {f[0] for f in found} == set(names.split("|"))
    assert [f for f in found if f[2] != "0"] == []


def test_exported_calls_keep_their_arguments(tmp_path):
    """A call that gets an option gets a name: programs that hold the C signatures, by the header or by a loaded symbol, go on as
    they are (an argument in front of the stream would take the stream for an option)."""
    src = tmp_path / "calls.cpp"
    src.write_text("""
#include "nn_ops.h"
using P = const void*; using V = void*; using L = long long;
int (*pool)(P x, V y, V argmax, const GeepsPoolGeom* g, V stream) = geeps_maxpool_forward;
int (*relu)(P dy, P y, V dx, float* colsum, L n, int c, L lddy, L ldy, L lddx, V stream) = geeps_relu_backward_colsum;
""")
    r = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", f"-I{_native.CSRC / 'kernels'}", str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
