"""Implicit-GEMM convolution (tcgen05 + 4-D TMA, stride 1) against torch's fp32 convolution."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


CASES = [
    # B, H, W, C_total, c_off, cg, O_total, o_off, og, k, pad
    (8, 13, 13, 64, 0, 64, 96, 0, 96, 3, 1),            # one channel chunk, one N tile
    (4, 27, 27, 96, 48, 48, 256, 128, 128, 5, 2),       # a 48-channel group slice (zero-filled to 64), 5x5
    (16, 13, 13, 192, 0, 192, 384, 0, 384, 3, 1),       # three chunks, two N tiles
    (5, 10, 12, 16, 0, 16, 40, 0, 40, 3, 0),            # no padding: output smaller than input
    (3, 9, 9, 32, 0, 32, 64, 0, 64, 1, 0),              # 1x1
    (2, 32, 32, 96, 0, 96, 32, 0, 32, 3, 1),            # wide image: boxes split the width
]


# three column slabs a tile and four tiles or more per SM: one epilogue group; the last tile of 312 channels has two slabs
LONG_ROWS = [
    (25, 56, 56, 16, 0, 16, 160, 0, 160, 3, 1),
    (47, 30, 30, 24, 8, 16, 320, 0, 312, 3, 1),
]


@pytest.mark.parametrize("case", CASES + LONG_ROWS)
def test_conv_tc_forward_dgrad_wgrad_match_torch(case):
    from geeps_b200.ops import functional as F
    B, H, W, Ct, c_off, cg, Ot, o_off, og, k, pad = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(hash(case) % 1000)
    OH, OW = H + 2 * pad - k + 1, W + 2 * pad - k + 1
    kd = k * k * cg
    ld = (kd + 7) // 8 * 8
    x_full = torch.randn(B, H, W, Ct, device=dev, generator=gen).to(BF)
    w = torch.zeros(og, ld, device=dev, dtype=BF)
    w[:, :kd] = (torch.randn(og, kd, device=dev, generator=gen) / kd ** 0.5).to(BF)
    bias = torch.randn(og, device=dev, generator=gen)
    dy_full = torch.randn(B, OH, OW, Ot, device=dev, generator=gen).to(BF)
    x = x_full[..., c_off:c_off + cg]
    dy = dy_full[..., o_off:o_off + og]
    status = torch.zeros(4, dtype=torch.int32, device=dev)

    # fp32 reference on the bf16-rounded operands
    xr = x.float().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    wr = w[:, :kd].float().view(og, k, k, cg).permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    yr = torch.nn.functional.conv2d(xr, wr, bias, padding=pad)
    yr.backward(dy.float().permute(0, 3, 1, 2))
    y_ref = torch.relu(yr.detach()).permute(0, 2, 3, 1)
    dx_ref = xr.grad.permute(0, 2, 3, 1)
    dw_ref = wr.grad.permute(0, 2, 3, 1).reshape(og, kd)

    y_full = torch.full((B, OH, OW, Ot), 7.0, device=dev, dtype=BF)
    y = y_full[..., o_off:o_off + og]
    assert F.conv_tc_supported(F.conv_tc_params(F.CONV_FWD, x, y, w, k, pad))
    F.conv_tc(F.CONV_FWD, x, y, w, k, pad, bias=bias, relu=True, status=status)
    assert _rel(y, y_ref) < 1e-2
    if Ot != og:      # channels outside the slice are untouched
        rest = torch.cat([y_full[..., :o_off], y_full[..., o_off + og:]], dim=-1)
        assert bool((rest == 7.0).all())

    dx_full = torch.full((B, H, W, Ct), 3.0, device=dev, dtype=BF)
    dx = dx_full[..., c_off:c_off + cg]
    F.conv_tc(F.CONV_DGRAD, dx, dy, w, k, pad, status=status)
    assert _rel(dx, dx_ref) < 1e-2
    if Ct != cg:
        rest = torch.cat([dx_full[..., :c_off], dx_full[..., c_off + cg:]], dim=-1)
        assert bool((rest == 3.0).all())

    for split in (0, 1):
        dw = torch.full((og, ld), 5.0, device=dev)
        F.conv_tc(F.CONV_WGRAD, x, dy, dw, k, pad, split_k=split, status=status)
        assert _rel(dw[:, :kd], dw_ref) < 1e-2, split
        assert bool((dw[:, kd:] == 0).all())
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0


STRIDED = [
    # B, H, W, cg, og, k, pad, stride
    (4, 28, 28, 64, 96, 3, 1, 2),        # Inception down-sampling branch
    (2, 64, 64, 8, 64, 7, 3, 2),         # first layer of the 22K net (3 channels padded to 8), scaled down
    (3, 17, 17, 32, 32, 3, 0, 2),        # no padding, odd size
    (2, 23, 23, 16, 48, 5, 2, 3),        # stride 3: nine classes, three launches of the data gradient
    (20, 32, 32, 80, 80, 3, 1, 2),       # more tiles than SMs over the four classes
    (2, 1, 9, 16, 16, 3, 1, 2),          # one image row: the classes of odd rows are empty
]


@pytest.mark.parametrize("case", STRIDED)
def test_strided_conv_forward_and_gradients_match_torch(case):
    """Strided layers: the activation boxes are loaded with a TMA element stride, the data gradient runs per parity
    class of the input; no patch matrix."""
    from geeps_b200.ops import functional as F
    B, H, W, cg, og, k, pad, st = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(5)
    OH, OW = (H + 2 * pad - k) // st + 1, (W + 2 * pad - k) // st + 1
    kd = k * k * cg
    ld = (kd + 7) // 8 * 8
    x = torch.randn(B, H, W, cg, device=dev, generator=gen).to(BF)
    w = torch.zeros(og, ld, device=dev, dtype=BF)
    w[:, :kd] = (torch.randn(og, kd, device=dev, generator=gen) / kd ** 0.5).to(BF)
    bias = torch.randn(og, device=dev, generator=gen)
    dy = torch.randn(B, OH, OW, og, device=dev, generator=gen).to(BF)
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    xr = x.float().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    wr = w[:, :kd].float().view(og, k, k, cg).permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    yr = torch.nn.functional.conv2d(xr, wr, bias, stride=st, padding=pad)
    yr.backward(dy.float().permute(0, 3, 1, 2))
    y = torch.empty(B, OH, OW, og, device=dev, dtype=BF)
    assert F.conv_tc_supported(F.conv_tc_params(F.CONV_FWD, x, y, w, k, pad, stride=st))
    assert F.conv_tc_supported(F.conv_tc_params(F.CONV_DGRAD, x, y, w, k, pad, stride=st))
    assert not F.conv_tc_supported(F.conv_tc_params(F.CONV_DGRAD, x, y, w[:, :cg], 1, 0, stride=st))
    F.conv_tc(F.CONV_FWD, x, y, w, k, pad, bias=bias, relu=True, status=status, stride=st)
    assert _rel(y, torch.relu(yr.detach()).permute(0, 2, 3, 1)) < 1e-2
    dw_ref = wr.grad.permute(0, 2, 3, 1).reshape(og, kd)
    for split in (0, 1):
        dw = torch.full((og, ld), 5.0, device=dev)
        F.conv_tc(F.CONV_WGRAD, x, dy, dw, k, pad, split_k=split, status=status, stride=st)
        assert _rel(dw[:, :kd], dw_ref) < 1e-2, split
    dx = torch.full((B, H, W, cg), 3.0, device=dev, dtype=BF)
    F.conv_tc(F.CONV_DGRAD, dx, dy, w, k, pad, status=status, stride=st)
    assert _rel(dx, xr.grad.permute(0, 2, 3, 1)) < 1e-2
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0


COLUMN_PAIRS = [
    # B, H, W, C_total, c_off, cg, O_total, o_off, og, k, pad
    (160, 27, 27, 96, 48, 48, 256, 128, 128, 5, 2),     # AlexNet conv2, channel slices on both sides, more tiles than SMs
    (75, 9, 28, 64, 0, 64, 72, 0, 72, 3, 1),            # even width, second chunk of 8 gradient channels, several rows of panels
    (75, 26, 27, 56, 0, 56, 40, 0, 40, 4, 1),           # even filter: halo of 2, the last step reads the even parity
    (40, 17, 40, 8, 0, 8, 64, 0, 64, 7, 0),             # 7 taps, no padding
    (100, 20, 20, 24, 0, 24, 64, 0, 64, 7, 3),
    (75, 13, 28, 16, 0, 16, 24, 0, 24, 2, 0),           # two taps a row, few k
    (1, 5, 2, 8, 0, 8, 8, 0, 8, 3, 1),                  # one pair of columns
    (2, 7, 9, 64, 0, 64, 136, 0, 136, 5, 2),            # three chunks, the last of 8
    (3, 11, 13, 24, 8, 16, 48, 0, 48, 6, 3),
]


@pytest.mark.parametrize("case", COLUMN_PAIRS)
def test_column_pair_data_gradient_matches_torch(case):
    """The even and the odd column of a pair in the two halves of an accumulator, KW + 1 steps per filter row: against 64
    bits, and bitwise against one column per position, which adds the same products in the same order."""
    from geeps_b200.ops import functional as F
    B, H, W, Ct, c_off, cg, Ot, o_off, og, k, pad = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(11)
    OH, OW, kd = H + 2 * pad - k + 1, W + 2 * pad - k + 1, k * k * cg
    ld = (kd + 7) // 8 * 8
    w = torch.zeros(og, ld, device=dev, dtype=BF)
    w[:, :kd] = (torch.randn(og, kd, device=dev, generator=gen) / kd ** 0.5).to(BF)
    dy = torch.randn(B, OH, OW, Ot, device=dev, generator=gen).to(BF)[..., o_off:o_off + og]
    dy[0, OH // 2, OW // 2, 0] = float("inf")           # spoils its own window only
    wr = w[:, :kd].double().view(og, k, k, cg).permute(0, 3, 1, 2)
    ref = torch.nn.functional.conv_transpose2d(dy.double().permute(0, 3, 1, 2), wr, padding=pad).permute(0, 2, 3, 1)
    dx_full = torch.full((B, H, W, Ct), 3.0, device=dev, dtype=BF)
    dx = dx_full[..., c_off:c_off + cg]
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    single = torch.full((B, H, W, Ct), 3.0, device=dev, dtype=BF)
    F.conv_halo(F.CONV_DGRAD, single[..., c_off:c_off + cg], dy, w, k, pad, columns=1, status=status)
    F.conv_halo(F.CONV_DGRAD, dx, dy, w, k, pad, columns=2, status=status)
    torch.cuda.synchronize()
    spoilt = torch.zeros(H, W, dtype=torch.bool, device=dev)
    y0, x0 = OH // 2 - pad, OW // 2 - pad
    spoilt[max(y0, 0):y0 + k, max(x0, 0):x0 + k] = True
    fine = torch.isfinite(dx).all(-1)
    assert bool(fine[1:].all()) and bool((fine[0] == ~spoilt).all())
    # fp32 sums rounded once to bf16: uniform relative rounding errors of up to 2^-9, 2^-9 / sqrt(3) = 1.1e-3 in the 2-norm
    assert _rel(dx[fine], ref[fine]) < 2.5e-3
    finite = torch.isfinite(dx_full)                    # what infinity and NaN are made of may differ
    assert torch.equal(finite, torch.isfinite(single)) and torch.equal(dx_full[finite], single[finite])
    assert bool((dx_full[..., :c_off] == 3.0).all()) and bool((dx_full[..., c_off + cg:] == 3.0).all())
    assert status.tolist()[0] == 0


@pytest.mark.parametrize("case", [(160, 27, 48, 128, 5, 2), (200, 28, 64, 96, 3, 1)])
def test_conv_tc_runs_a_data_gradient_by_column_pairs(case):
    """Layers that conv_tc() sends to the pairs: the result is that of the kernel asked for them."""
    import ctypes
    from geeps_b200.ops import _lib as L
    from geeps_b200.ops import functional as F
    B, H, cg, og, k, pad = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(12)
    w = (torch.randn(og, k * k * cg, device=dev, generator=gen) / (k * k * cg) ** 0.5).to(BF)
    dy = torch.randn(B, H, H, og, device=dev, generator=gen).to(BF)
    out = [torch.zeros(B, H, H, cg, device=dev, dtype=BF) for _ in range(2)]
    p, pairs = F.conv_tc_params(F.CONV_DGRAD, out[0], dy, w, k, pad), L.HaloPlanInfo()
    assert L.lib().geeps_conv_halo_pair_plan(ctypes.byref(p), ctypes.byref(pairs)) and pairs.routed
    F.conv_tc(F.CONV_DGRAD, out[0], dy, w, k, pad)
    F.conv_halo(F.CONV_DGRAD, out[1], dy, w, k, pad, columns=2)
    torch.cuda.synchronize()
    assert torch.equal(*out)
    p.mode, p.columns = F.CONV_FWD, 2                   # no such thing
    assert L.lib().geeps_conv_halo(ctypes.byref(p), L.stream_ptr()) != 0


HALO_CASES = CASES + [
    (3, 57, 57, 48, 0, 48, 96, 0, 96, 3, 0),            # AlexNet conv1 after space-to-depth: 96 channels leave in 32-wide slabs
    (3, 28, 28, 192, 0, 192, 96, 0, 96, 3, 1),          # three chunks, rows split 4 + 4 per tile, last tile short
    (2, 14, 14, 96, 32, 32, 64, 0, 48, 5, 2),           # 5x5 on a small map, channel slices on both sides
    (2, 56, 56, 64, 0, 64, 192, 0, 192, 3, 1),          # two rows per block, two N tiles
]


# several tiles per SM through two pairs of store slabs: a last tile of one block, a channel block with one slab to store
SHORT_TILES = [
    (60, 28, 28, 48, 0, 48, 160, 0, 160, 3, 1),
    (160, 9, 27, 24, 8, 16, 104, 0, 104, 3, 1),
    (90, 28, 28, 8, 0, 8, 96, 0, 96, 2, 0),
]


@pytest.mark.parametrize("case", HALO_CASES + SHORT_TILES)
def test_conv_halo_forward_dgrad_match_torch(case):
    """The halo-tile kernel called directly on every shape it accepts (conv_tc() picks it only where it pays)."""
    from geeps_b200.ops import functional as F
    B, H, W, Ct, c_off, cg, Ot, o_off, og, k, pad = case
    if k * k < 4:
        pytest.skip("single-tap filters have no halo")
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(hash(case) % 1000)
    OH, OW = H + 2 * pad - k + 1, W + 2 * pad - k + 1
    kd = k * k * cg
    ld = (kd + 7) // 8 * 8
    x_full = torch.randn(B, H, W, Ct, device=dev, generator=gen).to(BF)
    w = torch.zeros(og, ld, device=dev, dtype=BF)
    w[:, :kd] = (torch.randn(og, kd, device=dev, generator=gen) / kd ** 0.5).to(BF)
    bias = torch.randn(og, device=dev, generator=gen)
    dy_full = torch.randn(B, OH, OW, Ot, device=dev, generator=gen).to(BF)
    x = x_full[..., c_off:c_off + cg]
    dy = dy_full[..., o_off:o_off + og]
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    xr = x.float().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    wr = w[:, :kd].float().view(og, k, k, cg).permute(0, 3, 1, 2).contiguous()
    yr = torch.nn.functional.conv2d(xr, wr, bias, padding=pad)
    yr.backward(dy.float().permute(0, 3, 1, 2))
    y_ref = torch.relu(yr.detach()).permute(0, 2, 3, 1)
    dx_ref = xr.grad.permute(0, 2, 3, 1)

    y_full = torch.full((B, OH, OW, Ot), 7.0, device=dev, dtype=BF)
    y = y_full[..., o_off:o_off + og]
    F.conv_halo(F.CONV_FWD, x, y, w, k, pad, bias=bias, relu=True, status=status)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0
    assert _rel(y, y_ref) < 1e-2
    if Ot != og:
        rest = torch.cat([y_full[..., :o_off], y_full[..., o_off + og:]], dim=-1)
        assert bool((rest == 7.0).all())
    dx_full = torch.full((B, H, W, Ct), 3.0, device=dev, dtype=BF)
    dx = dx_full[..., c_off:c_off + cg]
    F.conv_halo(F.CONV_DGRAD, dx, dy, w, k, pad, status=status)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0
    assert _rel(dx, dx_ref) < 1e-2
    if Ct != cg:
        rest = torch.cat([dx_full[..., :c_off], dx_full[..., c_off + cg:]], dim=-1)
        assert bool((rest == 3.0).all())


@pytest.mark.parametrize("case", [c for c in HALO_CASES if c[9] > 1 and c[9] <= 8])
def test_conv_wgrad_halo_matches_torch(case):
    """The filter-row weight-gradient kernel (one activation tile serves the taps of a row through overlapping
    N panels) called directly on every shape it accepts."""
    from geeps_b200.ops import functional as F
    B, H, W, Ct, c_off, cg, Ot, o_off, og, k, pad = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(hash(case) % 1000)
    OH, OW = H + 2 * pad - k + 1, W + 2 * pad - k + 1
    kd = k * k * cg
    ld = (kd + 7) // 8 * 8
    x = torch.randn(B, H, W, Ct, device=dev, generator=gen).to(BF)[..., c_off:c_off + cg]
    dy = torch.randn(B, OH, OW, Ot, device=dev, generator=gen).to(BF)[..., o_off:o_off + og]
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    xr = x.float().permute(0, 3, 1, 2).contiguous()
    wr = torch.zeros(og, cg, k, k, device=dev, requires_grad=True)
    torch.nn.functional.conv2d(xr, wr, None, padding=pad).backward(dy.float().permute(0, 3, 1, 2))
    dw_ref = wr.grad.permute(0, 2, 3, 1).reshape(og, kd)
    dw = torch.full((og, ld), 5.0, device=dev)
    F.conv_wgrad_halo(x, dy, dw, k, pad, status=status)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0
    assert _rel(dw[:, :kd], dw_ref) < 1e-2
    assert bool((dw[:, kd:] == 0).all())


@pytest.mark.parametrize("cpad", [None, 64])
def test_space_to_depth_conv_matches_strided_torch_conv(cpad):
    """Input(s2d) + Conv2d(s2d): an 11x11 stride-4 convolution run as a 3-tap stride-1 implicit GEMM; with cpad the
    48-channel space-to-depth pixel is zero-padded to one 128-byte line."""
    from geeps_b200.ops.layers import Conv2d, Input
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(3)
    B, C, H, k, S, cout = 4, 3, 67, 11, 4, 32
    x = torch.randn(B, C, H, H, device=dev, generator=gen)
    inp = Input(s2d=S, s2d_k=k, cpad=cpad)
    conv = Conv2d("c1", cout, k, stride=S, relu=True, need_dx=False, s2d=S, cin_valid=C if cpad else None)
    shape = conv.setup(inp.setup((B, C, H, H), dev), dev)
    OH = (H - k) // S + 1
    assert shape == (B, OH, OH, cout)
    spec = conv.param_specs()[0]
    assert spec.num_valid() == cout * k * k * C
    w32 = spec.initial(torch.Generator().manual_seed(1)).to(dev) * 5
    bias = torch.randn(cout, device=dev, generator=gen)
    conv.p32, conv.p16 = {"weight": w32, "bias": bias}, {"weight": w32.to(BF)}
    conv.g32 = {"weight": torch.full_like(w32, 9.0), "bias": torch.zeros(cout, device=dev)}
    y = conv.forward(inp.forward(x)).view(B, OH, OH, cout)

    # the same weights as a [cout, C, k, k] filter: column (a*T + b)*48 + (dy*S + dx)*C + c -> tap (a*S+dy, b*S+dx)
    T, Cs, Cp = conv.k, S * S * C, conv.in_shape[-1]
    assert Cp == (cpad or Cs)
    wt = w32.to(BF).float()[:, :T * T * Cp].view(cout, T, T, Cp)[..., :Cs].reshape(cout, T, T, S, S, C)   # [o, a, b, dy, dx, c]
    wfull = wt.permute(0, 5, 1, 3, 2, 4).reshape(cout, C, T * S, T * S)[:, :, :k, :k].contiguous().requires_grad_(True)
    xr = x.to(BF).float()
    yr = torch.nn.functional.conv2d(xr, wfull, bias, stride=S)
    assert _rel(y, torch.relu(yr).permute(0, 2, 3, 1)) < 1e-2

    dy = torch.randn(B, OH, OH, cout, device=dev, generator=gen).to(BF)
    conv.backward(dy.view(-1, cout))
    mask = (yr > 0).float()
    yr.backward(dy.float().permute(0, 3, 1, 2) * mask)
    gfull = conv.g32["weight"][:, :T * T * Cp].view(cout, T, T, Cp)
    assert float(gfull[..., Cs:].abs().max()) == 0 if Cp > Cs else True      # padding channels receive no gradient
    gw = gfull[..., :Cs].reshape(cout, T, T, S, S, C).permute(0, 5, 1, 3, 2, 4).reshape(cout, C, T * S, T * S)
    assert _rel(gw[:, :, :k, :k], wfull.grad) < 1e-2
    # taps past the 11 x 11 filter receive no gradient, so they stay zero under SGD
    assert float(gw[:, :, k:, :].abs().max()) == 0 and float(gw[:, :, :, k:].abs().max()) == 0


@pytest.mark.parametrize("layout", ["s2d64", "s2d48", "nhwc8", "s2d2"])
@pytest.mark.parametrize("mode", ["centre", "random"])
def test_uint8_data_transformer_matches_torch(layout, mode):
    """Input on uint8 source images: crop, mirror, mean subtraction and scale on the device give exactly what the
    same arithmetic in torch followed by the fp32 input path gives (both round the same fp32 value to bf16)."""
    from geeps_b200.ops.layers import Input
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(11)
    B, C, Hin, Win, H, W = 5, 3, 80, 90, 67, 71
    mean, scale = (104.0, 117.0, 123.5), 1.0 / 57.0
    kw = {"s2d64": dict(s2d=4, s2d_k=11, cpad=64), "s2d48": dict(s2d=4, s2d_k=11), "nhwc8": dict(cpad=8),
          "s2d2": dict(s2d=2, s2d_k=7, cpad=16)}[layout]
    inp, ref = Input(mean=mean, scale=scale, **kw), Input(**kw)
    shape = inp.setup((B, C, H, W), dev)
    assert ref.setup((B, C, H, W), dev) == shape
    x = torch.randint(0, 256, (B, C, Hin, Win), device=dev, generator=gen, dtype=torch.uint8)
    if mode == "random":
        inp.randomize((Hin, Win), mirror=True, generator=gen)
        aug = inp.aug.cpu()
        assert int(aug[:, 2].max()) == 1 and int(aug[:, 2].min()) == 0      # both orientations are in the batch
    else:
        aug = torch.tensor([[(Hin - H) // 2, (Win - W) // 2, 0]] * B)
    y = inp.forward(x).clone()
    m = torch.tensor(mean, device=dev).view(1, C, 1, 1)
    rows = []
    for b in range(B):
        ho, wo, mir = (int(v) for v in aug[b])
        win = x[b:b + 1, :, ho:ho + H, wo:wo + W].float()
        rows.append(win.flip(-1) if mir else win)
    xr = (torch.cat(rows) - m) * scale
    yr = ref.forward(xr.contiguous())
    assert y.shape == yr.shape == shape
    assert torch.equal(y, yr)
    if mode == "random":
        inp.set_augmentation(None)          # back to the centre crop, through the same buffer
        y2 = inp.forward(x)
        xc = (x[:, :, (Hin - H) // 2:(Hin - H) // 2 + H, (Win - W) // 2:(Win - W) // 2 + W].float() - m) * scale
        assert torch.equal(y2, ref.forward(xc.contiguous()))


@pytest.mark.parametrize("B,H,W,cpad", [(1, 11, 11, 64), (3, 30, 37, 48), (2, 227, 227, 64), (2, 45, 62, 56)])
@pytest.mark.parametrize("mirror", [0, 1])
def test_space_to_depth_of_8_and_16_bit_sources(B, H, W, cpad, mirror):
    """Rows that start on any byte, ragged right and lower edges, pixels of several rows in one warp, and a source whose
    size is not a whole number of words (16-bit: the kernel by elements; 8-bit: first and last words by bytes)."""
    from geeps_b200.ops import functional as F
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(H * W)
    Hs, Ws = -(-H // 4), -(-W // 4)

    def ref(v):                                            # v: [B, 3, H, W] in the output's values
        p = torch.zeros(B, 3, Hs * 4, Ws * 4, device=dev)
        p[:, :, :H, :W] = v
        p = p.view(B, 3, Hs, 4, Ws, 4).permute(0, 2, 4, 3, 5, 1).reshape(B, Hs, Ws, 48)
        return torch.nn.functional.pad(p, (0, cpad - 48)).to(torch.bfloat16)

    y = torch.full((B, Hs, Ws, cpad), 9.0, dtype=torch.bfloat16, device=dev)
    if not mirror:
        x = torch.randn(B, 3, H, W, device=dev, generator=gen).to(torch.bfloat16)
        F.nchw_to_s2d_bf16(x, y, 4)
        assert torch.equal(y, ref(x.float()))
    for ho, wo in ((0, 0), (2, 3), (5, 6)):
        x = torch.randint(0, 256, (B, 3, H + 5, W + 6), device=dev, generator=gen, dtype=torch.uint8)
        aug = torch.tensor([[ho, wo, mirror]] * B, dtype=torch.int32, device=dev)
        mean, scale = (104.0, 117.0, 123.0), 1.0 / 58.0
        F.u8_transform(x, y.fill_(9.0), (H, W), 4, aug, mean, scale)
        v = x[:, :, ho:ho + H, wo:wo + W].float()
        v = (v.flip(3) if mirror else v) - torch.tensor(mean, device=dev).view(3, 1, 1)
        assert torch.equal(y, ref(v * torch.tensor(scale, device=dev)))


@pytest.mark.parametrize("B,H,W", [(1, 4, 4), (2, 3, 2), (1, 5, 7), (2, 11, 13), (2, 6, 9), (3, 227, 227)])
@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_8_bit_sources_on_any_byte(B, H, W, off):
    """A source that starts and ends on any byte, taken whole (the first and the last quad reach the tensor's ends), as
    it is and mirrored; the bytes around it are another buffer's."""
    from geeps_b200.ops import functional as F
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(B * H * W + off)
    n = B * 3 * H * W
    buf = torch.randint(0, 256, (n + 8,), device=dev, generator=gen, dtype=torch.uint8)
    x = buf[off:off + n].view(B, 3, H, W)
    Hs, Ws = -(-H // 4), -(-W // 4)
    for mirror in (0, 1):
        y = torch.full((B, Hs, Ws, 64), 9.0, dtype=torch.bfloat16, device=dev)
        aug = torch.tensor([[0, 0, mirror]] * B, dtype=torch.int32, device=dev)
        F.u8_transform(x, y, (H, W), 4, aug, (104.0, 117.0, 123.0), 1.0 / 58.0)
        v = x.flip(3) if mirror else x
        v = (v.float() - torch.tensor((104.0, 117.0, 123.0), device=dev).view(3, 1, 1)) * torch.tensor(1.0 / 58.0, device=dev)
        p = torch.zeros(B, 3, Hs * 4, Ws * 4, device=dev)
        p[:, :, :H, :W] = v
        p = p.view(B, 3, Hs, 4, Ws, 4).permute(0, 2, 4, 3, 5, 1).reshape(B, Hs, Ws, 48)
        assert torch.equal(y, torch.nn.functional.pad(p, (0, 16)).to(torch.bfloat16))


def test_8_bit_sources_on_any_byte_take_the_fast_kernel():
    """A source off a word boundary costs about what an aligned one does (by elements it cost seven times as much)."""
    from geeps_b200.ops import functional as F
    dev = torch.device("cuda:0")
    B, H = 128, 227
    n = B * 3 * H * H
    buf = torch.zeros(n + 8, dtype=torch.uint8, device=dev)
    y = torch.empty(B, 57, 57, 64, dtype=torch.bfloat16, device=dev)
    aug = torch.zeros(B, 3, dtype=torch.int32, device=dev)

    def ms(off):
        x = buf[off:off + n].view(B, 3, H, H)
        best = 1e9
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                F.u8_transform(x, y, (H, H), 4, aug, (104.0, 117.0, 123.0), 1.0 / 58.0)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best
    aligned = ms(0)
    assert ms(1) < 2.5 * aligned and ms(2) < 2.5 * aligned


@pytest.mark.parametrize("mode,B,H,W,cg,og,k,pad,wide", [
    ("fwd", 3, 7, 6, 152, 80, 5, 2, 0),           # one box and an empty half of a pair
    ("fwd", 4, 5, 5, 368, 40, 5, 2, 8),           # N = 64 in halves of 32, pitched activations
    ("fwd", 37, 17, 5, 144, 280, 3, 1, 0),        # two tiles of 192 columns, the second one ragged
    ("fwd", 39, 28, 17, 72, 80, 3, 1, 16),        # ragged boxes, columns past the last channel
    ("fwd", 19, 18, 6, 328, 360, 2, 1, 0),
    ("dgrad", 26, 30, 23, 80, 136, 2, 1, 0),      # more pairs than fit at once
    ("dgrad", 26, 27, 26, 72, 72, 3, 0, 0), ("dgrad", 11, 29, 27, 72, 208, 3, 1, 16), ("dgrad", 17, 17, 30, 72, 72, 5, 0, 0),
    ("dgrad", 24, 20, 21, 248, 136, 3, 1, 0),     # 256 columns: two panels of the weights in each half
    ("fwd", 32, 17, 17, 384, 256, 5, 2, 0),       # whole 128-byte lines
    ("fwd", 37, 17, 17, 384, 384, 5, 2, 0), ("dgrad", 37, 17, 17, 256, 384, 5, 2, 0)])
def test_box_convolution_on_cta_pairs_gives_the_bits_of_single_ctas(mode, B, H, W, cg, og, k, pad, wide):
    """Two neighbouring pixel boxes by one product of 256 rows: the same terms in the same order, so the same bits as one CTA per
    box; nothing outside the result is written."""
    import ctypes
    from geeps_b200.ops import _lib as L
    from geeps_b200.ops import functional as F
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(B * cg)
    fwd, OH, OW, kd = mode == "fwd", H + 2 * pad - k + 1, W + 2 * pad - k + 1, k * k * cg
    w = (torch.randn(og, (kd + 7) // 8 * 8, device=dev, generator=gen) / kd ** 0.5).to(BF)
    full = [torch.randn(B, h, v, c + wide, device=dev, generator=gen).to(BF) for h, v, c in ((H, W, cg), (OH, OW, og))]
    src, c_out = (full[0], og) if fwd else (full[1], cg)
    bias = torch.randn(og, device=dev, generator=gen) if fwd else None
    got = []
    for split_k in (-1, -2):
        dst = torch.full(full[1 if fwd else 0].shape, 3.0, device=dev, dtype=BF)
        x, y = ((src, dst) if fwd else (dst, src))
        status = torch.zeros(4, dtype=torch.int32, device=dev)
        p = F.conv_tc_params(F.CONV_FWD if fwd else F.CONV_DGRAD, x[..., :cg], y[..., :og], w, k, pad, bias=bias, relu=fwd,
                             split_k=split_k, status=status)
        L.check(L.lib().geeps_conv_tc(ctypes.byref(p), L.stream_ptr()), "conv_tc")
        assert status.tolist()[0] == 0 and (dst[..., c_out:] == 3.0).all()
        got.append(dst)
    assert L.lib().geeps_conv_box_pairs(ctypes.byref(p))
    assert torch.equal(got[0], got[1])
    x64 = full[0][..., :cg].double().permute(0, 3, 1, 2)
    w64 = w[:, :kd].double().view(og, k, k, cg).permute(0, 3, 1, 2)
    ref = (torch.relu(torch.nn.functional.conv2d(x64, w64, bias.double(), padding=pad)) if fwd else
           torch.nn.functional.conv_transpose2d(full[1][..., :og].double().permute(0, 3, 1, 2), w64, padding=pad))
    # fp32 sums rounded once to bf16: 2^-9 / sqrt(3) = 1.1e-3 in the 2-norm
    assert _rel(got[0][..., :c_out], ref.permute(0, 2, 3, 1)) < 2.5e-3


@pytest.mark.parametrize("B,H,cg,og,k", [(25, 48, 56, 272, 5), (37, 30, 56, 96, 3), (20, 47, 40, 88, 5), (30, 27, 136, 80, 5),
                                         (13, 39, 80, 104, 5), (37, 30, 184, 88, 3), (10, 32, 264, 40, 5), (6, 43, 240, 376, 3)])
def test_layers_off_128_byte_lines_agree_on_both_kernels(B, H, cg, og, k):
    """Layers that the expected times send to the halo kernel, as conv_tc() runs them and kept on the box kernel: the same bits
    forward (one chunk of channels, or not sent there), fp32 sums in two orders backward, where a rounding to bf16 differs now
    and then."""
    import ctypes
    from geeps_b200.ops import _lib as L
    from geeps_b200.ops import functional as F
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(H * cg)
    kd = k * k * cg
    x = torch.randn(B, H, H, cg, device=dev, generator=gen).to(BF)
    dy = torch.randn(B, H, H, og, device=dev, generator=gen).to(BF)
    w = (torch.randn(og, (kd + 7) // 8 * 8, device=dev, generator=gen) / kd ** 0.5).to(BF)
    routed = 0
    for mode in (F.CONV_FWD, F.CONV_DGRAD):
        out = [torch.full_like(dy if mode == F.CONV_FWD else x, 3.0) for _ in range(2)]
        for o, split_k in zip(out, (0, -2)):
            a = (x, o) if mode == F.CONV_FWD else (o, dy)
            p = F.conv_tc_params(mode, *a, w, k, k // 2, split_k=split_k)
            routed += split_k == 0 and L.lib().geeps_conv_halo_applicable(ctypes.byref(p))
            L.check(L.lib().geeps_conv_tc(ctypes.byref(p), L.stream_ptr()), "conv_tc")
        if mode == F.CONV_FWD:
            assert torch.equal(out[0], out[1])
        # a term's rounding is 2^-24 of a partial sum of norm about sqrt(kd): few results cross a rounding boundary of bf16
        assert _rel(out[0], out[1].double()) < 5e-4
    assert routed


@pytest.mark.parametrize("B,H,cg,og,k,there", [
    (68, 53, 40, 208, 3, True), (41, 28, 136, 104, 5, True),
    (14, 24, 136, 152, 5, True),               # a last chunk of 8 channels, few blocks
    (9, 11, 200, 280, 5, True),                # ... and half of the positions beside the image
    (21, 41, 80, 296, 7, True),                # a last chunk of 16
    (95, 33, 64, 360, 5, True), (45, 15, 264, 344, 7, False),
    (5, 26, 280, 200, 5, False), (37, 27, 168, 368, 3, False), (20, 47, 104, 112, 5, False), (40, 28, 136, 72, 3, False)])
def test_weight_gradients_off_128_byte_lines_agree_on_both_kernels(B, H, cg, og, k, there):
    """Layers that the expected times send to the filter-row kernel and such that they keep off it, as conv_tc() runs them and on
    both kernels by name: the same products, summed in fp32 in other slices."""
    import ctypes
    from geeps_b200.ops import _lib as L
    from geeps_b200.ops import functional as F
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(H * cg)
    kd, pad = k * k * cg, k // 2
    ld = (kd + 7) // 8 * 8 + 8
    x = torch.randn(B, H, H, cg, device=dev, generator=gen).to(BF)
    dy = torch.randn(B, H, H, og, device=dev, generator=gen).to(BF)
    out = [torch.full((og, ld), 3.0, device=dev) for _ in range(3)]
    p = F.conv_tc_params(F.CONV_WGRAD, x, dy, out[0], k, pad)
    assert bool(L.lib().geeps_conv_wgrad_halo_applicable(ctypes.byref(p))) == there
    F.conv_tc(F.CONV_WGRAD, x, dy, out[0], k, pad)
    F.conv_tc(F.CONV_WGRAD, x, dy, out[1], k, pad, split_k=-1)
    p.w = out[2].data_ptr()
    L.check(L.lib().geeps_conv_wgrad_halo(ctypes.byref(p), L.stream_ptr()), "conv_wgrad_halo")
    x64 = torch.nn.functional.pad(x.double(), (0, 0, pad, pad, pad, pad))
    d64 = dy.double().view(-1, og)
    ref = torch.cat([d64.t() @ x64[:, i:i + H, j:j + H].reshape(-1, cg) for i in range(k) for j in range(k)], 1)
    for o in out:
        assert (o[:, kd:] == 0).all()
        # One slice at most: a step adds 16 of n positions, so the partial sum behind step j of J = n / 16 has a norm of sqrt(j / J) of the
        # result's, and the tensor cores cut off less than 2^-23 of it: 2 / 3 J 2^-23 in all (steps that hold fewer positions of
        # the image, util of them, are as many more).
        assert _rel(o[:, :kd], ref) < 2 / 3 * (B * H * H / 16 / 0.45) * 2.0 ** -23


@pytest.mark.parametrize("B,H,cg,og", [(7, 8, 72, 136), (2, 13, 368, 352), (1, 19, 80, 288)])
def test_small_weight_gradients_off_128_byte_lines_repeat_bit_for_bit(B, H, cg, og):
    """Layers whose gradient is written in one piece: the same bits in every call."""
    from geeps_b200.ops import functional as F
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(cg)
    x = torch.randn(B, H, H, cg, device=dev, generator=gen).to(BF)
    dy = torch.randn(B, H, H, og, device=dev, generator=gen).to(BF)
    out = [torch.full((og, 9 * cg), 3.0, device=dev) for _ in range(30)]
    for o in out:
        F.conv_tc(F.CONV_WGRAD, x, dy, o, 3, 1)
    assert all(torch.equal(o, out[0]) for o in out)


@pytest.mark.parametrize("B,H,cin,cout,k,groups,masked", [(64, 27, 96, 256, 5, 2, False), (64, 27, 96, 256, 5, 2, True), (50, 13, 128, 96, 3, 2, False),
                                                          (20, 13, 64, 200, 3, 1, False), (1, 7, 32, 48, 3, 2, True), (2, 8, 16, 8, 1, 1, False)])
def test_layer_gradient_is_cleared_once(B, H, cin, cout, k, groups, masked):
    """Weight gradients whose zeros come with the ReLU mask or from one launch for all groups, and such that need none (summed
    in one piece, 1 x 1): two backward passes over a gradient that held other values; whole numbers, so every sum is exact."""
    from geeps_b200.ops import functional as F
    from geeps_b200.ops.layers import Conv2d
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(B + cout)
    rnd = lambda *s: torch.randint(-1, 2, s, device=dev, generator=gen).to(BF)      # noqa: E731
    layer = Conv2d("c", cout, k, pad=k // 2, groups=groups, relu=True)
    layer.setup((B, H, H, cin), dev)
    shapes = {s.name.split(".")[-1]: s.shape for s in layer.param_specs()}
    (wname, wshape), (bname, bshape) = shapes.items()
    layer.p16["weight"], layer.p32["bias"] = rnd(*wshape), torch.zeros(bshape, device=dev)
    layer.g32["weight"], layer.g32["bias"] = torch.full(wshape, 5.0, device=dev), torch.full(bshape, 5.0, device=dev)
    x, dy = rnd(B, H, H, cin), rnd(B * H * H, cout)
    y = layer.forward(x).view(B * H * H, cout)
    dz = dy if masked else torch.where(y > 0, dy, torch.zeros_like(dy))
    if masked:
        layer.dy_is_masked, layer.bias_grad_src = True, dz.float().sum(0)
    ref = torch.full(wshape, 3.0, device=dev)
    cg, og = cin // groups, cout // groups
    for g in range(groups):
        if k == 1:
            ref[:, :cin] = dz.float().t() @ x.float().view(-1, cin)
        else:
            F.conv_tc(F.CONV_WGRAD, x[..., g * cg:(g + 1) * cg], dz.view(B, H, H, cout)[..., g * og:(g + 1) * og], ref[g * og:(g + 1) * og], k, k // 2)
    for _ in range(2):
        layer.backward(dy)
        assert torch.equal(layer.g32["weight"], ref) and torch.equal(layer.g32["bias"], dz.float().sum(0))
