"""Geometry of the halo-tile convolution kernels over a sweep of layer shapes (host arithmetic only, no GPU): every
plan the kernels would accept keeps its tiles inside shared memory, tensor memory and the MMA's shape limits."""
import ctypes as C
import itertools

import pytest

from geeps_b200.ops import _lib as L

SMEM_LIMIT = 227 * 1024


def _params(mode, B, H, W, cg, og, k, pad, stride=1):
    p = L.ConvTcParams()
    # the planners only look at shapes, pitches and alignment: any 16-byte aligned non-null addresses will do
    p.x, p.y, p.w = 0x10000, 0x20000, 0x30000
    p.bias, p.status = None, None
    OH, OW = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    p.x_pitch, p.y_pitch = cg, og
    p.ldw = (k * k * cg + 7) // 8 * 8
    p.B, p.H, p.W, p.cg, p.OH, p.OW, p.og = B, H, W, cg, OH, OW, og
    p.KH, p.KW, p.pad, p.relu, p.mode, p.split_k, p.stride = k, k, pad, 0, mode, 0, stride
    return p, OH, OW


SHAPES = [(B, H, cg, og, k, pad)
          for B, H, (cg, og), (k, pad) in itertools.product(
              (1, 8, 32, 256), (7, 13, 14, 27, 28, 55, 56, 57, 64, 112),
              ((8, 16), (16, 40), (32, 96), (48, 128), (64, 192), (96, 96), (192, 384), (256, 256)),
              ((2, 0), (3, 0), (3, 1), (5, 2), (7, 3)))
          if H + 2 * pad >= k]


@pytest.mark.parametrize("mode", [0, 1])
def test_forward_and_data_gradient_plans_respect_the_hardware_limits(mode):
    lib = L.lib()
    seen = routed = 0
    for B, H, cg, og, k, pad in SHAPES:
        p, OH, OW = _params(mode, B, H, H, cg, og, k, pad)
        info = L.HaloPlanInfo()
        if not lib.geeps_conv_halo_plan(C.byref(p), C.byref(info)):
            assert info.ok == 0
            continue
        seen += 1
        routed += info.routed
        GW, GH = (OW, OH) if mode == 0 else (H, H)
        nch = og if mode == 0 else cg
        assert info.PW >= GW + k - 1 and info.PW <= 128
        assert info.positions == info.R * info.PW and info.positions % 8 == 0 and 0 < info.positions <= 128
        assert info.ncols2 % 16 == 0 and 2 * info.positions <= info.ncols2 <= 256
        assert info.ncols1 % 16 == 0 and info.positions <= info.ncols1 <= 128
        assert 2 * info.R * info.row_tiles >= GH                     # the tiles cover every output row
        assert 2 * info.R * (info.row_tiles - 1) < GH                # and no tile is entirely outside the image
        assert info.m_tiles == (nch + 127) // 128
        # a tap-shifted MMA of ncols2 rows stays inside one activation stage
        rows_read = (k - 1) * info.PW + (k - 1) + info.ncols2
        assert rows_read * 128 <= info.x_stage_bytes
        assert ((2 * info.R + k - 1) * info.PW) * 128 <= info.x_stage_bytes
        assert info.x_stage_bytes % 1024 == 0
        assert info.stages_w >= 3 and info.stages_x == 2
        assert info.smem_bytes <= SMEM_LIMIT
        assert info.tmem_cols == 512
        assert 0.0 < info.util <= 1.0
    assert seen > 100 and routed > 0


def test_strided_calls_are_not_given_to_the_halo_kernels():
    lib = L.lib()
    for mode in (0, 1, 2):
        p, _, _ = _params(mode, 32, 28, 28, 64, 96, 3, 1, stride=2)
        info = L.HaloPlanInfo()
        fn = lib.geeps_conv_wgrad_halo_plan if mode == 2 else lib.geeps_conv_halo_plan
        assert fn(C.byref(p), C.byref(info)) == 0 and info.ok == 0


def test_weight_gradient_plans_respect_the_hardware_limits():
    lib = L.lib()
    seen = routed = 0
    for B, H, cg, og, k, pad in SHAPES:
        p, OH, OW = _params(2, B, H, H, cg, og, k, pad)
        p.ldw = (k * k * cg + 3) // 4 * 4
        info = L.HaloPlanInfo()
        if not lib.geeps_conv_wgrad_halo_plan(C.byref(p), C.byref(info)):
            continue
        seen += 1
        routed += info.routed
        assert info.PW >= OW + k - 1 and info.PW <= 128
        assert info.positions == info.R * info.PW and info.positions % 16 == 0 and 0 < info.positions <= 128
        assert 1 <= info.TY <= k and info.TY * k * 64 <= 512 and info.passes == -(-k // info.TY)
        assert info.tmem_cols >= info.TY * k * 64 and info.tmem_cols <= 512
        assert info.n_blocks == B * info.row_tiles and info.R * info.row_tiles >= OH
        per = -(-info.n_blocks // info.split)
        assert 1 <= info.split <= info.n_blocks and per * (info.split - 1) < info.n_blocks    # no empty slice
        rows_read = (info.TY - 1) * info.PW + (k - 1) + info.positions
        assert rows_read * 128 <= info.x_stage_bytes
        assert info.stages_x >= 2 and info.smem_bytes <= SMEM_LIMIT
    assert seen > 100 and routed > 0


def test_column_pair_data_gradient_plans_respect_the_hardware_limits():
    lib = L.lib()
    seen = routed = 0
    for B, H, cg, og, k, pad in SHAPES + [(256, H, cg, 96, k, k // 2) for H in (2, 3, 27, 31, 40, 55) for cg in (8, 48, 56, 64)
                                          for k in (2, 3, 4, 5, 6, 7)]:
        p, OH, OW = _params(1, B, H, H, cg, og, k, pad)
        info = L.HaloPlanInfo()
        if not lib.geeps_conv_halo_pair_plan(C.byref(p), C.byref(info)):
            continue
        seen += 1
        routed += info.routed
        assert cg <= 64 and H >= 2 and OW >= 2 and info.m_tiles == 1
        assert info.PW >= (H + 1) // 2 + k // 2 and info.PW <= 128          # no window leaves its row
        assert info.positions == info.R * info.PW and info.positions % 8 == 0 and 0 < info.positions <= 128
        assert info.ncols2 % 16 == 0 and 2 * info.positions <= info.ncols2 <= 256
        assert 2 * info.R * info.row_tiles >= H > 2 * info.R * (info.row_tiles - 1)
        # the last step of a row reads k // 2 columns on, in either parity's tile
        assert ((k - 1) * info.PW + k // 2 + info.ncols2) * 128 <= info.x_stage_bytes // 2
        assert info.x_stage_bytes % 2048 == 0
        # whole filter rows of panels (8192 bytes); a panel in front of them and one behind are read for disabled lanes
        slab = max(8192, (info.positions * 128 + 1023) // 1024 * 1024)
        assert info.stages_w % k == 0 and 5 <= info.stages_w <= 16 and info.stages_x * info.x_stage_bytes >= 8192
        assert info.stages_x * info.x_stage_bytes + info.stages_w * 8192 + 2 * slab < info.smem_bytes <= SMEM_LIMIT
        assert 0.0 < info.util <= 1.0
    assert seen > 100 and routed > 0


def test_weight_gradient_slices_do_not_leave_the_busiest_sm_longer_than_two_slices_per_sm():
    """Position blocks on the busiest of 148 SMs, for layers of 5 to 150 (output block, channel chunk, filter row) items."""
    lib, sms = L.lib(), 148
    seen = set()
    for B, H, cg, og, k in itertools.product((100, 200, 256), (14, 20, 28), range(64, 449, 64), range(128, 641, 128), (5, 7)):
        p, OH, OW = _params(2, B, H, H, cg, og, k, k // 2)
        info = L.HaloPlanInfo()
        if not lib.geeps_conv_wgrad_halo_plan(C.byref(p), C.byref(info)):
            continue
        base = info.m_tiles * (-(-cg // 64)) * info.passes
        assert info.TY == 1 and base == -(-og // 128) * -(-cg // 64) * k

        def path(n):      # blocks walked, and five more for every item that is drained
            waves, per = -(-base * n // sms), -(-info.n_blocks // n)
            return waves * (per + 5)
        # (a slice count that leaves the last slice empty is lowered until none is)
        assert path(info.split) <= min(path(1), path(max(1, sms // base)), path(max(1, 2 * sms // base))), (B, H, cg, og, k)
        seen.add(base)
    assert min(seen) == 5 and len([b for b in seen if 50 <= b <= 148]) > 10


def test_short_forward_tiles_keep_two_pairs_of_store_slabs():
    """3 x 3 layers of at most 48 input channels, wherever three weight stages remain; one pair and more stages elsewhere."""
    lib = L.lib()
    two = one = 0
    for mode, (B, H, cg, og, k, pad) in itertools.product((0, 1), SHAPES):
        p, OH, OW = _params(mode, B, H, H, cg, og, k, pad)
        info = L.HaloPlanInfo()
        if not lib.geeps_conv_halo_plan(C.byref(p), C.byref(info)):
            continue
        rest = info.smem_bytes - info.stages_x * info.x_stage_bytes - info.stages_w * 16384     # slabs and barriers
        pairs = rest // 32768
        assert pairs in (1, 2) and rest - pairs * 32768 < 2048 and info.smem_bytes <= SMEM_LIMIT
        short = mode == 0 and k <= 3 and cg <= 48
        room = 224 * 1024 - info.stages_x * info.x_stage_bytes >= 65536 + 3 * 16384
        assert pairs == (2 if short and room else 1), (mode, B, H, cg, og, k)
        two += pairs == 2
        one += pairs == 1
    assert two > 50 and one > 50


def test_weight_gradients_that_repeat_bit_for_bit_keep_their_kernel():
    """Rows off 128-byte lines, where expected times choose the kernel: a gradient in one slice, or in two on zeros, has the
    same bits in every call, and is not sent to a kernel that adds up more slices."""
    lib = L.lib()

    def plans(B, H, cg, og, k):
        p, _, _ = _params(2, B, H, H, cg, og, k, k // 2)
        info = L.HaloPlanInfo()
        ok = lib.geeps_conv_wgrad_halo_plan(C.byref(p), C.byref(info))
        return ok, info, lib.geeps_conv_box_wgrad_slices(C.byref(p))

    for layer, slices in (((7, 8, 72, 136, 3), 7), ((2, 13, 368, 352, 3), 4), ((1, 19, 80, 288, 3), 5)):
        ok, info, box = plans(*layer)
        assert ok and info.split == slices and box == 1 and not info.routed, layer
    routed = kept = 0
    for B, H, cg, og, k in itertools.product((1, 2, 4, 7, 16, 40, 100, 256), (5, 8, 13, 19, 28, 53), (32, 40, 72, 80, 168, 368),
                                             (40, 88, 136, 208, 352), (3, 5)):
        ok, info, box = plans(B, H, cg, og, k)
        if not ok:
            continue
        routed += info.routed
        tail = cg - (cg + 63) // 64 * 64 + 64
        lines_rule = tail >= 32 and info.util >= 0.6 and info.n_blocks >= 4 * 148 and (k >= 5 or (info.m_tiles == 1 and cg <= 64))
        if box <= 2 < info.split and not lines_rule:
            assert not info.routed, (B, H, cg, og, k)
            kept += 1
        if info.split <= 2 < box and lines_rule:
            assert info.routed, (B, H, cg, og, k)
            kept += 1
    assert routed > 200 and kept > 50


@pytest.mark.parametrize("B,H,cg,og,k,pad,there", [
    # us, filter-row kernel / box kernel
    (1, 12, 344, 400, 5, 0, False),               # 11.5 / 8.2
    (94, 17, 416, 336, 7, 3, False),              # 463 / 349
    (20, 29, 288, 416, 6, 3, False),              # 273 / 213
    (104, 29, 240, 80, 4, 2, False),              # 99 / 80
    (10, 7, 288, 264, 7, 3, False),               # 21.7 / 17.4
    (48, 31, 40, 176, 6, 3, True),                # 66 / 157
    (72, 46, 32, 80, 4, 2, True),                 # 37 / 48
    (68, 53, 40, 208, 3, 1, True),                # 60 / 144
    (45, 15, 264, 344, 7, 3, False),              # the faster one by its sums of 1260 steps instead of 636
    (41, 28, 136, 104, 5, 2, True)])              # 44 / 80
def test_weight_gradients_off_128_byte_lines_go_to_the_faster_kernel(B, H, cg, og, k, pad, there):
    p, _, _ = _params(2, B, H, H, cg, og, k, pad)
    assert bool(L.lib().geeps_conv_wgrad_halo_applicable(C.byref(p))) == there


def test_weight_gradients_of_filters_that_were_not_timed_go_by_the_rule_for_whole_lines():
    p, _, _ = _params(2, 2, 40, 40, 40, 176, 8, 4)         # few blocks: the box kernel's by that rule
    assert not L.lib().geeps_conv_wgrad_halo_applicable(C.byref(p))


def test_weight_gradients_go_to_no_kernel_with_longer_sums():
    """What each step of 16 positions adds is cut off at the partial sum: off 128-byte lines the expected times choose a kernel
    only if its slices have no more steps than those of the rule for whole lines."""
    lib = L.lib()
    lib.geeps_conv_box_wgrad_steps.restype = C.c_longlong
    moved = 0
    for B, H, cg, og, k in itertools.product((1, 3, 12, 45, 68, 200), (8, 15, 28, 41, 53), (32, 40, 80, 104, 264, 344), (40, 112, 208, 344), (3, 4, 5, 7)):
        p, _, _ = _params(2, B, H, H, cg, og, k, k // 2)
        info = L.HaloPlanInfo()
        if not lib.geeps_conv_wgrad_halo_plan(C.byref(p), C.byref(info)):
            continue
        tail = cg - (cg + 63) // 64 * 64 + 64
        rule = tail >= 32 and info.util >= 0.6 and info.n_blocks >= 4 * 148 and (k >= 5 or (info.m_tiles == 1 and cg <= 64))
        here, box = -(-info.n_blocks // info.split) * info.positions // 16, lib.geeps_conv_box_wgrad_steps(C.byref(p))
        if bool(info.routed) != rule:
            assert (here <= box) if info.routed else (box <= here), (B, H, cg, og, k)
            moved += 1
    assert moved > 50
