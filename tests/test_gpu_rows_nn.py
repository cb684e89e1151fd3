"""Row ops and training-op kernels vs plain PyTorch fp32 references."""
import ctypes

import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu

from geeps_b200.ops import functional as F
from geeps_b200.ops import _lib as L

DEV = "cuda:0"
BF = torch.bfloat16


def test_row_gather_scatter_add():
    torch.manual_seed(0)
    cache = torch.randn(1000, 128, device=DEV)
    n = 333
    id1 = torch.randperm(1000, device=DEV)[:n]
    index = torch.stack([torch.arange(n, device=DEV), id1], dim=1).contiguous()
    buf = torch.full((n, 128), -7.0, device=DEV)
    st = L.new_status(DEV)
    limit = (n - 1) * 128 + 37  # last row only partly inside the value limit
    F.row_gather(buf, cache, index, num_vals_limit=limit, status=st)
    ref = cache[id1].clone()
    ref.view(-1)[limit:] = -7.0
    assert torch.equal(buf, ref)
    # scatter-add back twice the gathered rows
    oplog = torch.zeros_like(cache)
    F.row_scatter_add(oplog, buf, index, status=st)
    F.row_scatter_add(oplog, buf, index, status=st)
    ref2 = torch.zeros_like(cache)
    ref2[id1] = 2 * buf
    assert torch.allclose(oplog, ref2)
    dst = torch.zeros_like(cache)
    F.row_scatter(dst, buf, index, status=st)
    ref3 = torch.zeros_like(cache)
    ref3[id1] = buf
    assert torch.equal(dst, ref3)
    assert L.read_status(st)["code"] == 0


def test_row_op_bounds_are_reported_not_faulted():
    cache = torch.zeros(10, 128, device=DEV)
    buf = torch.ones(4, 128, device=DEV)
    index = torch.tensor([[0, 1], [1, 99], [2, 3], [3, -5]], device=DEV, dtype=torch.int64)
    st = L.new_status(DEV)
    F.row_scatter_add(cache, buf, index, status=st)
    torch.cuda.synchronize()
    s = L.read_status(st)
    assert s["name"] == "bounds"
    assert cache[1].sum().item() == 128 and cache[3].sum().item() == 128 and cache.sum().item() == 256


def test_axpy_and_convert():
    x = torch.randn(100003, device=DEV)
    y = torch.randn(100003, device=DEV)
    ref = y + 0.25 * x
    F.axpy(y, x, 0.25)
    assert torch.allclose(y, ref)
    h = torch.empty(100003, dtype=BF, device=DEV)
    F.f32_to_bf16(x, h)
    assert torch.equal(h, x.to(BF))


@pytest.mark.parametrize("cfg", [
    dict(B=3, H=13, W=13, C=16, groups=1, Cout=24, k=3, s=1, p=1),
    dict(B=2, H=27, W=27, C=32, groups=2, Cout=48, k=5, s=1, p=2),
    dict(B=2, H=35, W=35, C=3, groups=1, Cout=16, k=11, s=4, p=0),
    dict(B=2, H=16, W=16, C=24, groups=1, Cout=40, k=3, s=2, p=0),
])
def test_conv_via_im2col_gemm(cfg):
    torch.manual_seed(1)
    B, H, W, Cc, G, Cout, k, s, p = (cfg[n] for n in ("B", "H", "W", "C", "groups", "Cout", "k", "s", "p"))
    x = torch.randn(B, Cc, H, W, device=DEV)
    w = torch.randn(Cout, Cc // G, k, k, device=DEV) * 0.1
    xh = F.nchw_to_nhwc_bf16(x)
    assert torch.equal(xh, x.permute(0, 2, 3, 1).to(BF))
    Cg, Og = Cc // G, Cout // G
    kd = k * k * Cg
    ld = (kd + 7) // 8 * 8
    g0 = F.conv_geom(xh.shape, 0, Cg, k, k, s, p, ld)
    OH, OW = g0.OH, g0.OW
    y = torch.empty(B * OH * OW, Cout, dtype=BF, device=DEV)
    ref = TF.conv2d(xh.float().permute(0, 3, 1, 2), w.to(BF).float(), stride=s, padding=p, groups=G)
    dy = torch.randn_like(ref)
    dyh = dy.permute(0, 2, 3, 1).reshape(-1, Cout).to(BF).contiguous()
    dx = torch.empty_like(xh)
    dw = torch.empty(Cout, ld, device=DEV)
    for gi in range(G):
        g = F.conv_geom(xh.shape, gi * Cg, Cg, k, k, s, p, ld)
        col = torch.empty(B * OH * OW, ld, dtype=BF, device=DEV)
        F.im2col(xh, col, g)
        wg = torch.zeros(Og, ld, dtype=BF, device=DEV)
        wg[:, :kd] = w[gi * Og:(gi + 1) * Og].permute(0, 2, 3, 1).reshape(Og, kd).to(BF)
        F.gemm(col, wg, y[:, gi * Og:(gi + 1) * Og])
        # data gradient: dcol = dy_g @ W_g ; weight gradient: dW_g = dy_g^T @ col
        dcol = torch.empty_like(col)
        F.gemm(dyh[:, gi * Og:(gi + 1) * Og], wg, dcol, b_mn=True)
        F.col2im(dcol, dx, g)
        F.gemm(dyh[:, gi * Og:(gi + 1) * Og], col, dw[gi * Og:(gi + 1) * Og], a_mn=True, b_mn=True, split_k=0)
    torch.cuda.synchronize()
    got = y.view(B, OH, OW, Cout).permute(0, 3, 1, 2).float()
    assert torch.allclose(got, ref, atol=5e-2, rtol=2e-2)
    xr = xh.float().permute(0, 3, 1, 2).requires_grad_(True)
    wr = w.to(BF).float().requires_grad_(True)
    TF.conv2d(xr, wr, stride=s, padding=p, groups=G).backward(dyh.float().view(B, OH, OW, Cout).permute(0, 3, 1, 2))
    assert torch.allclose(dx.float().permute(0, 3, 1, 2), xr.grad, atol=8e-2, rtol=3e-2)
    dw_ref = wr.grad.permute(0, 2, 3, 1).reshape(Cout, kd)
    assert torch.allclose(dw[:, :kd], dw_ref, atol=1e-1, rtol=2e-2), (dw[:, :kd] - dw_ref).abs().max()


@pytest.mark.parametrize("relu", [False, True])
def test_batchnorm_forward_backward(relu):
    torch.manual_seed(2)
    P, Cc = 3000, 48
    x = (torch.randn(P, Cc, device=DEV) * 2 + 1).to(BF)
    gamma = torch.rand(Cc, device=DEV) + 0.5
    beta = torch.randn(Cc, device=DEV) * 0.1
    y = torch.empty_like(x)
    sums = torch.empty(2 * Cc, device=DEV)
    mr = torch.empty(2 * Cc, device=DEV)
    rm, rv = torch.zeros(Cc, device=DEV), torch.ones(Cc, device=DEV)
    F.bn_forward(x, y, gamma, beta, sums, mr, rm, rv, eps=1e-5, momentum=0.1, relu=relu)
    xr = x.float().requires_grad_(True)
    gr, br = gamma.clone().requires_grad_(True), beta.clone().requires_grad_(True)
    yr = TF.batch_norm(xr, None, None, gr, br, training=True, eps=1e-5)
    if relu:
        yr = torch.relu(yr)
    assert torch.allclose(y.float(), yr, atol=3e-2, rtol=2e-2)
    dy = torch.randn(P, Cc, device=DEV).to(BF)
    dx = torch.empty_like(x)
    dg, db = torch.empty(Cc, device=DEV), torch.empty(Cc, device=DEV)
    F.bn_backward(x, dy, y, dx, mr, gamma, sums, dg, db, relu=relu)
    # reference masks with its own fp32 y; use the kernel's bf16 y mask for an exact match
    yr2 = TF.batch_norm(xr, None, None, gr, br, training=True, eps=1e-5)
    if relu:
        yr2 = yr2 * (y.float() > 0)
    yr2.backward(dy.float())
    assert torch.allclose(dx.float(), xr.grad, atol=3e-2, rtol=3e-2)
    assert torch.allclose(dg, gr.grad, atol=0.5, rtol=2e-2)
    assert torch.allclose(db, br.grad, atol=0.5, rtol=2e-2)


@pytest.mark.parametrize("relu", [False, True])
def test_batchnorm_layer_alternating_and_repeated_passes(relu):
    """The BatchNorm layer's training-loop form (two launches per direction, each zeroing the other direction's
    scratch) over forward / backward / forward / forward / backward: every result matches torch."""
    from geeps_b200.ops import layers as GL
    torch.manual_seed(4)
    P, Cc = 2048, 64
    bn = GL.BatchNorm("bn", relu=relu)
    bn.setup((P, Cc), torch.device(DEV))
    gamma = torch.rand(Cc, device=DEV) + 0.5
    beta = torch.randn(Cc, device=DEV) * 0.1
    bn.p32 = {"gamma": gamma, "beta": beta}
    bn.g32 = {"gamma": torch.empty(Cc, device=DEV), "beta": torch.empty(Cc, device=DEV)}

    def check(x, dy):
        xr = x.float().requires_grad_(True)
        gr, br = gamma.clone().requires_grad_(True), beta.clone().requires_grad_(True)
        yr = TF.batch_norm(xr, None, None, gr, br, training=True, eps=bn.eps)
        y = bn.forward(x)
        assert torch.allclose(y.float(), torch.relu(yr) if relu else yr, atol=3e-2, rtol=2e-2)
        if dy is None:
            return
        dx = bn.backward(dy)
        (yr * (y.float() > 0) if relu else yr).backward(dy.float())
        assert torch.allclose(dx.float(), xr.grad, atol=3e-2, rtol=3e-2)
        assert torch.allclose(bn.g32["gamma"], gr.grad, atol=0.5, rtol=2e-2)
        assert torch.allclose(bn.g32["beta"], br.grad, atol=0.5, rtol=2e-2)

    mk = lambda: (torch.randn(P, Cc, device=DEV) * 2 + 1).to(BF)
    check(mk(), torch.randn(P, Cc, device=DEV).to(BF))
    check(mk(), None)                      # forward only ...
    check(mk(), None)                      # ... twice in a row: the scratch was not zeroed by a backward pass
    check(mk(), torch.randn(P, Cc, device=DEV).to(BF))
    check(mk(), torch.randn(P, Cc, device=DEV).to(BF))
    torch.cuda.synchronize()


def test_lrn_forward_backward():
    torch.manual_seed(3)
    P, Cc = 500, 96
    x = (torch.randn(P, Cc, device=DEV) * 3).to(BF)
    y = torch.empty_like(x)
    scale = torch.empty(P, Cc, dtype=BF, device=DEV)      # receives 1 / scale in bf16
    F.lrn_forward(x, y, scale, size=5, alpha=1e-2, beta=0.75, k=1.0)
    xr = x.float().requires_grad_(True)
    yr = TF.local_response_norm(xr.view(P, Cc, 1, 1), 5, alpha=1e-2, beta=0.75, k=1.0).view(P, Cc)
    assert torch.allclose(y.float(), yr, atol=3e-2, rtol=2e-2)
    dy = torch.randn(P, Cc, device=DEV).to(BF)
    dx = torch.empty_like(x)
    F.lrn_backward(x, y, scale, dy, dx, size=5, alpha=1e-2, beta=0.75)
    yr.backward(dy.float())
    assert torch.allclose(dx.float(), xr.grad, atol=3e-2, rtol=3e-2)
    # with the producer's ReLU backward folded in: no gradient where the input is not positive
    dxm = torch.empty_like(x)
    F.lrn_backward(x, y, scale, dy, dxm, size=5, alpha=1e-2, beta=0.75, relu_mask=True)
    assert torch.equal(dxm, torch.where(x > 0, dx, torch.zeros_like(dx)))
    # ... and the per-channel sums of that gradient (the producer's bias gradient) from the same pass
    cs = torch.full((Cc,), 5.0, device=DEV)
    dxs = torch.empty_like(x)
    F.lrn_backward(x, y, scale, dy, dxs, size=5, alpha=1e-2, beta=0.75, relu_mask=True, colsum=cs)
    assert torch.equal(dxs, dxm)
    assert torch.allclose(cs, dxm.float().sum(0), atol=1e-2, rtol=1e-4)


def test_relu_backward_with_column_sums_in_one_pass():
    torch.manual_seed(12)
    P, Cc = 3000, 384
    wide_dy = torch.randn(P, Cc + 16, device=DEV).to(BF)
    dy = wide_dy[:, 8:8 + Cc]                                # a channel slice of a wider tensor
    y = torch.relu(torch.randn(P, Cc, device=DEV)).to(BF)
    dx = torch.empty(P, Cc, dtype=BF, device=DEV)
    cs = torch.full((Cc,), 3.0, device=DEV)
    F.relu_backward_colsum(dy, y, dx, cs)
    ref = torch.where(y > 0, dy, torch.zeros_like(dy))
    assert torch.equal(dx, ref)
    assert torch.allclose(cs, ref.float().sum(0), atol=1e-2, rtol=1e-4)


@pytest.mark.parametrize("H,Cc,k,s,p,size", [(13, 96, 3, 2, 0, 5), (27, 256, 3, 2, 0, 5), (16, 24, 3, 2, 0, 3),
                                              (9, 40, 3, 1, 1, 5), (8, 8, 2, 2, 0, 7)])
def test_fused_lrn_maxpool_matches_fp32_reference_and_the_unfused_kernels(H, Cc, k, s, p, size):
    """maxpool(LRN(x)) in one kernel per direction against torch in fp32 (LRN + max_pool2d + autograd) and against
    this library's separate LRN and pooling kernels; with the ReLU mask and the per-channel sums of dx."""
    torch.manual_seed(11)
    B = 3
    alpha, beta, kk = 1e-2, 0.75, 1.0
    x = torch.relu(torch.randn(B, H, H, Cc, device=DEV) * 3).to(BF)        # a ReLU output, as in the network
    g = F.pool_geom(x.shape, k, s, p, Cc, Cc)
    assert F.lrn_maxpool_supported(g, size)
    pooled = torch.empty(B, g.OH, g.OW, Cc, dtype=BF, device=DEV)
    arg = torch.empty(B, g.OH, g.OW, Cc, dtype=torch.uint8, device=DEV)
    F.lrn_maxpool_forward(x, pooled, arg, g, size, alpha, beta, kk)
    # unfused kernels of this library
    y = torch.empty_like(x)
    scale = torch.empty_like(x)
    F.lrn_forward(x.view(-1, Cc), y.view(-1, Cc), scale.view(-1, Cc), size, alpha, beta, kk)
    pooled_u = torch.empty_like(pooled)
    arg_u = torch.empty_like(arg)
    F.maxpool_forward(y, pooled_u, arg_u, g)
    # same values up to the last bf16 digit (the fused kernel evaluates the power as a polynomial), same window choice
    # except where two candidates are that close
    assert torch.allclose(pooled.float(), pooled_u.float(), atol=1e-2, rtol=1e-2)
    assert (arg != arg_u).float().mean().item() < 2e-2
    # fp32 reference
    xr = x.float().permute(0, 3, 1, 2).requires_grad_(True)
    yr = TF.max_pool2d(TF.local_response_norm(xr, size, alpha=alpha, beta=beta, k=kk), k, s, p, ceil_mode=True)
    assert yr.shape[2] == g.OH
    assert torch.allclose(pooled.float().permute(0, 3, 1, 2), yr, atol=3e-2, rtol=2e-2)
    dp = torch.randn_like(pooled)
    yr.backward(dp.float().permute(0, 3, 1, 2))
    ref = xr.grad.permute(0, 2, 3, 1)
    dx = torch.empty_like(x)
    cs = torch.full((Cc,), 7.0, device=DEV)
    F.lrn_maxpool_backward(x, dp, arg, dx, g, size, alpha, beta, kk, relu_mask=True, colsum=cs)
    ref_masked = torch.where(x > 0, ref, torch.zeros_like(ref))
    bad = ((dx.float() - ref_masked).abs() > 3e-2 + 3e-2 * ref_masked.abs()).float().mean().item()
    assert bad < 5e-3, bad       # the window maximum is taken on bf16-rounded values: rare near-ties pick another element
    # the sums are taken before dx is rounded to bf16
    assert torch.allclose(cs, dx.float().sum((0, 1, 2)), atol=8e-2, rtol=5e-3)
    # unfused backward of this library (pool backward, then LRN backward with the mask)
    dy_u = torch.empty_like(x)
    F.maxpool_backward(dp, arg, dy_u, g)
    dx_u = torch.empty_like(x)
    F.lrn_backward(x.view(-1, Cc), y.view(-1, Cc), scale.view(-1, Cc), dy_u.view(-1, Cc), dx_u.view(-1, Cc), size, alpha,
                   beta, relu_mask=True)
    assert torch.allclose(dx.float(), dx_u.float(), atol=4e-2, rtol=4e-2)
    # without the mask and the sums
    dx2 = torch.empty_like(x)
    F.lrn_maxpool_backward(x, dp, arg, dx2, g, size, alpha, beta, kk)
    assert torch.equal(torch.where(x > 0, dx2, torch.zeros_like(dx2)), dx)


@pytest.mark.parametrize("k,s,p,H", [(3, 2, 0, 13), (3, 2, 0, 16), (3, 1, 1, 9), (2, 2, 0, 8)])
def test_maxpool_avgpool(k, s, p, H):
    torch.manual_seed(4)
    B, Cc = 2, 24
    x = torch.randn(B, H, H, Cc, device=DEV).to(BF)
    g = F.pool_geom(x.shape, k, s, p, Cc, Cc + 8)
    wide = torch.zeros(B, g.OH, g.OW, Cc + 8, dtype=BF, device=DEV)
    y = wide[..., :Cc]
    arg = torch.empty(B, g.OH, g.OW, Cc, dtype=torch.uint8, device=DEV)
    F.maxpool_forward(x, y, arg, g)
    xr = x.float().permute(0, 3, 1, 2).requires_grad_(True)
    yr = TF.max_pool2d(xr, k, s, p, ceil_mode=True)
    assert yr.shape[2] == g.OH
    assert torch.equal(y.float().permute(0, 3, 1, 2), yr)
    dyw = torch.zeros_like(wide)
    dyw[..., :Cc] = torch.randn(B, g.OH, g.OW, Cc, device=DEV).to(BF)
    dx = torch.empty_like(x)
    F.maxpool_backward(dyw, arg, dx, g)
    yr.backward(dyw[..., :Cc].float().permute(0, 3, 1, 2))
    assert torch.allclose(dx.float().permute(0, 3, 1, 2), xr.grad, atol=2e-2, rtol=2e-2)
    # average pooling (floor mode shapes for the reference)
    ga = F.pool_geom(x.shape, k, s, p, Cc, Cc, ceil_mode=False)
    ya = torch.empty(B, ga.OH, ga.OW, Cc, dtype=BF, device=DEV)
    F.avgpool_forward(x, ya, ga)
    xa = x.float().permute(0, 3, 1, 2).contiguous().requires_grad_(True)  # NCHW-contiguous reference
    yar = TF.avg_pool2d(xa, k, s, p, ceil_mode=False, count_include_pad=True)
    assert torch.allclose(ya.float().permute(0, 3, 1, 2), yar, atol=2e-2, rtol=2e-2)
    dya = torch.randn_like(ya)
    dxa = torch.empty_like(x)
    F.avgpool_backward(dya, dxa, ga)
    yar.backward(dya.float().permute(0, 3, 1, 2).contiguous())
    assert torch.allclose(dxa.float().permute(0, 3, 1, 2), xa.grad, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("Cc", [10, 1000, 21841])
def test_softmax_cross_entropy(Cc):
    torch.manual_seed(5)
    B = 32
    logits = torch.randn(B, Cc, device=DEV) * 3
    labels = torch.randint(0, Cc, (B,), device=DEV)
    loss = torch.empty(1, device=DEV)
    ldd = (Cc + 7) // 8 * 8
    dl = torch.zeros(B, ldd, dtype=BF, device=DEV)
    F.softmax_ce(logits, labels, loss, dl[:, :Cc], loss_scale=1.0 / B, grad_scale=1.0 / B)
    lr = logits.clone().requires_grad_(True)
    ref = TF.cross_entropy(lr, labels)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 1e-3 * max(1, abs(ref.item()))
    assert torch.allclose(dl[:, :Cc].float(), lr.grad, atol=2e-3, rtol=2e-2)


def test_colsum_relu_backward_dropout():
    torch.manual_seed(6)
    x = torch.randn(777, 64, device=DEV).to(BF)
    out = torch.empty(64, device=DEV)
    F.colsum(x, out, scale=0.5)
    assert torch.allclose(out, 0.5 * x.float().sum(0), atol=5e-2, rtol=1e-2)
    x2 = torch.randn(32, 1001, device=DEV).to(BF)
    out2 = torch.empty(1001, device=DEV)
    F.colsum(x2, out2)
    assert torch.allclose(out2, x2.float().sum(0), atol=5e-2, rtol=1e-2)
    y = torch.randn(1000, 8, device=DEV).to(BF)
    dy = torch.randn(1000, 8, device=DEV).to(BF)
    dx = torch.empty_like(dy)
    F.relu_backward(dy, y, dx)
    assert torch.equal(dx, torch.where(y.float() > 0, dy, torch.zeros_like(dy)))
    big = torch.ones(1 << 20, dtype=BF, device=DEV)
    o1, o2 = torch.empty_like(big), torch.empty_like(big)
    F.dropout(big, o1, 0.5, seed=42)
    F.dropout(big, o2, 0.5, seed=42)
    assert torch.equal(o1, o2)
    keep = (o1 > 0).float().mean().item()
    assert abs(keep - 0.5) < 0.01 and o1.max().item() == 2.0


@pytest.mark.parametrize("relu,fp32_out", [(True, False), (False, False), (False, True)])
def test_linear_with_the_k_range_split_over_the_sms_matches_fp32(relu, fp32_out, monkeypatch):
    """Batch-sized M: split-K GEMM into an fp32 workspace plus the converting pass, forward and data gradient,
    against torch in fp32 on the bf16-rounded operands."""
    from geeps_b200.ops import layers as GL
    monkeypatch.setattr(GL, "SPLIT_K_LINEAR", True)
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(11)
    B, K, N = 64, 1024, 264
    lin = GL.Linear("fc", N, relu=relu, fp32_out=fp32_out)
    lin.setup((B, K), dev)
    w = (torch.randn(N, K, device=dev, generator=gen) * 0.05).to(BF)
    bias = torch.randn(N, device=dev, generator=gen)
    lin.p16, lin.p32 = {"weight": w}, {"bias": bias}
    lin.g32 = {"weight": torch.zeros(N, K, device=dev), "bias": torch.zeros(N, device=dev)}
    x = torch.randn(B, K, device=dev, generator=gen).to(BF)
    y = lin.forward(x)
    ref = x.float() @ w.float().t() + bias
    if relu:
        ref = torch.relu(ref)
    assert y.dtype == (torch.float32 if fp32_out else BF)
    assert ((y.float() - ref).norm() / ref.norm()).item() < 1e-2
    dy = torch.randn(B, N, device=dev, generator=gen).to(torch.float32 if fp32_out else BF)
    dyb = dy.to(BF)
    dx = lin.backward(dyb)
    mask = (ref > 0).float() if relu else torch.ones_like(ref)
    dx_ref = (dyb.float() * mask) @ w.float()
    assert ((dx.float() - dx_ref).norm() / dx_ref.norm()).item() < 1e-2
    torch.cuda.synchronize()


@pytest.mark.parametrize("P,Cc", [(1, 8), (3, 24), (777, 64), (129, 104), (1000, 1600), (37, 2056), (6, 4096),
                                  (1, 1032), (90, 1024), (9, 1032), (50, 2048), (2500, 1288)])
def test_channel_kernels_at_the_edges_of_their_thread_map(P, Cc):
    """One row to more rows than a batch of loads, slots that do not divide a block, C split over several block columns."""
    torch.manual_seed(P + Cc)
    x, dy = torch.randn(P, Cc, device=DEV).to(BF), torch.randn(P, Cc, device=DEV).to(BF)
    x64, dy64 = x.double(), dy.double()
    eps = 2.0 ** -8                                 # half an ulp of bf16, doubled
    total = torch.empty(Cc, device=DEV)
    F.colsum(x, total, scale=0.5)
    assert torch.allclose(total.double(), 0.5 * x64.sum(0), atol=1e-5 * P ** 0.5 * 4, rtol=1e-5)
    dx = torch.empty_like(dy)
    F.relu_backward_colsum(dy, x, dx, total)
    ref = torch.where(x64 > 0, dy64, torch.zeros_like(dy64))
    assert torch.equal(dx.double(), ref)
    assert torch.allclose(total.double(), ref.sum(0), atol=1e-5 * P ** 0.5 * 4, rtol=1e-5)
    if P < 3:
        return
    g, b = torch.rand(Cc, device=DEV) + 0.5, torch.randn(Cc, device=DEV)
    sums, sums_b, stat = torch.zeros(2 * Cc, device=DEV), torch.ones(2 * Cc, device=DEV), torch.empty(2 * Cc, device=DEV)
    rm, rv = torch.zeros(Cc, device=DEV), torch.ones(Cc, device=DEV)
    y = torch.empty_like(x)
    F.bn_forward_fused(x, y, g, b, sums, stat, rm, rv, zero_after=sums_b, relu=True)
    xr, gr, br = (t.double().requires_grad_(True) for t in (x, g, b))
    yr = torch.relu(TF.batch_norm(xr, None, None, gr, br, training=True, eps=1e-5))
    # E[x^2] - mean^2 in fp32: a few 1e-7 of the variance, before bf16 rounding
    assert torch.allclose(y.double(), yr, atol=1e-4, rtol=eps)
    assert torch.allclose(rm.double(), 0.1 * x64.mean(0), atol=1e-6) and sums_b.abs().max().item() == 0
    yr.backward(torch.where(y.double() > 0, dy64, torch.zeros_like(dy64)))
    dg, db = torch.empty(Cc, device=DEV), torch.empty(Cc, device=DEV)
    F.bn_backward_fused(x, dy, y, dx, stat, g, sums_b, dg, db, zero_after=sums, relu=True)
    scale = xr.grad.abs().max().item()
    assert torch.allclose(dx.double(), xr.grad, atol=1e-4 * scale, rtol=eps)
    assert torch.allclose(dg.double(), gr.grad, atol=1e-4 * P ** 0.5, rtol=1e-4)
    assert torch.allclose(db.double(), br.grad, atol=1e-5 * P ** 0.5 * 4, rtol=1e-5) and sums.abs().max().item() == 0


@pytest.mark.parametrize("Cc,pad", [(1, 7), (127, 1), (1000, 0), (1001, 7), (8199, 0), (24576, 0), (30001, 7),
                                    (4095, 1), (4095, 0), (4096, 0), (4096, 1), (4097, 7), (4097, 0), (6000, 0), (6001, 2),
                                    (24577, 7), (24577, 0), (30001, 2)])
def test_softmax_rows_in_registers_and_past_them(Cc, pad):
    """Aligned rows (pitch a multiple of 8) and unaligned ones, on both sides of 4096 classes (fewer: the narrow kernel),
    blocks of fewer than 1024 threads, rows that are read again (more than 24576 classes)."""
    torch.manual_seed(Cc)
    B = 5
    logits = (torch.randn(B, Cc + pad, device=DEV) * 4)[:, :Cc]
    labels = torch.randint(0, Cc, (B,), device=DEV)
    wide = torch.full((B, Cc + pad), 3.0, dtype=BF, device=DEV)
    loss = torch.empty(1, device=DEV)
    F.softmax_ce(logits, labels, loss, wide[:, :Cc], loss_scale=1.0 / B, grad_scale=1.0 / B)
    lr = logits.double().clone().requires_grad_(True)
    ref = TF.cross_entropy(lr, labels)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 1e-5 * max(1, abs(ref.item()))
    assert torch.allclose(wide[:, :Cc].double(), lr.grad, atol=1e-7, rtol=2.0 ** -7)
    assert pad == 0 or (wide[:, Cc:] == 3.0).all()


@pytest.mark.parametrize("H,Cc,pad", [(3, 8, 0), (14, 32, 1), (7, 64, 0), (18, 72, 0), (9, 104, 1), (8, 144, 0), (11, 232, 0),
                                      (6, 264, 1), (5, 512, 0), (5, 520, 0),
                                      (17, 16, 0), (10, 24, 1), (12, 48, 0), (70, 8, 1), (5, 384, 0), (5, 392, 0),
                                      (68, 16, 0), (61, 40, 1), (60, 272, 0)])
@pytest.mark.parametrize("alpha", [1e-4, 0.5])
def test_lrn_maxpool_backward_over_channel_counts(H, Cc, pad, alpha):
    """Every lane / vector split of the register kernel (520 channels take the general one), odd and even sizes with
    and without padding; alpha 0.5 leaves the range of the polynomials."""
    torch.manual_seed(H * Cc)
    B, size, beta, kk = 2 if H < 60 else 9, 5, 0.75, 1.0
    x = torch.relu(torch.randn(B, H, H, Cc, device=DEV) * 3).to(BF)
    g = F.pool_geom(x.shape, 3, 2, pad, Cc, Cc)
    p = torch.empty(B, g.OH, g.OW, Cc, dtype=BF, device=DEV)
    arg = torch.empty(B, g.OH, g.OW, Cc, dtype=torch.uint8, device=DEV)
    F.lrn_maxpool_forward(x, p, arg, g, size, alpha, beta, kk)
    dp = torch.randn_like(p)
    dx, cs = torch.empty_like(x), torch.empty(Cc, device=DEV)
    F.lrn_maxpool_backward(x, dp, arg, dx, g, size, alpha, beta, kk, relu_mask=True, colsum=cs)
    # the pooling gradient by the kernel's own window codes, then autograd through the normalisation
    n = torch.arange(g.OH, device=DEV) * 2 - pad
    rows = n.view(1, -1, 1, 1) + arg.long() // 3
    cols = n.view(1, 1, -1, 1) + arg.long() % 3
    flat = ((torch.arange(B, device=DEV).view(-1, 1, 1, 1) * H + rows) * H + cols) * Cc + torch.arange(Cc, device=DEV)
    dy = torch.zeros(x.numel(), dtype=torch.float64, device=DEV).scatter_add_(0, flat.view(-1), dp.double().view(-1))
    xr = x.double().permute(0, 3, 1, 2).requires_grad_(True)
    TF.local_response_norm(xr, size, alpha=alpha, beta=beta, k=kk).backward(dy.view(B, H, H, Cc).permute(0, 3, 1, 2))
    ref = torch.where(x > 0, xr.grad.permute(0, 2, 3, 1), torch.zeros((), dtype=torch.float64, device=DEV))
    # bf16 result of two bf16-rounded terms (a and the ratios, five of which meet in a window)
    err = (dx.double() - ref).norm() / ref.norm()
    assert err.item() < 3 * 2.0 ** -9, err.item()
    assert torch.allclose(cs.double(), ref.sum((0, 1, 2)), atol=0.02 * (B * H * H) ** 0.5, rtol=1e-2)


@pytest.mark.parametrize("n", [1, 2, 3])
def test_branch_gradients_are_added_in_one_pass(n):
    torch.manual_seed(n)
    dst = torch.randn(333, 88, device=DEV).to(BF)
    srcs = [torch.randn(333, 96 + 8 * i, device=DEV).to(BF)[:, 8:96] for i in range(n)]
    ref = dst.double() + sum(t.double() for t in srcs)
    F.add_2d(dst, srcs[0]) if n == 1 else F.add_2d_n(dst, srcs)
    # one rounding to bf16 of an fp32 sum
    assert torch.allclose(dst.double(), ref, atol=1e-6, rtol=2.0 ** -8)


@pytest.mark.parametrize("P,Cc", [(5, 8), (777, 104), (64, 2056)])
def test_batchnorm_backward_from_mask_bits_equals_the_one_from_the_output(P, Cc):
    torch.manual_seed(P)
    x, dy = torch.randn(P, Cc, device=DEV).to(BF), torch.randn(P, Cc, device=DEV).to(BF)
    g, b = torch.rand(Cc, device=DEV) + 0.5, torch.randn(Cc, device=DEV)
    y, stat = torch.empty_like(x), torch.empty(2 * Cc, device=DEV)
    bits = torch.full((P, Cc // 8), 0xa5, dtype=torch.uint8, device=DEV)
    rm, rv = torch.zeros(Cc, device=DEV), torch.ones(Cc, device=DEV)
    F.bn_forward_fused(x, y, g, b, torch.zeros(2 * Cc, device=DEV), stat, rm, rv, relu=True, bits=bits)
    want = (y.view(P, Cc // 8, 8) > 0).long() << torch.arange(8, device=DEV)
    assert torch.equal(bits.long(), want.sum(2))
    got = []
    for m in (None, bits):
        dx, dg, db = torch.empty_like(x), torch.empty(Cc, device=DEV), torch.empty(Cc, device=DEV)
        F.bn_backward_fused(x, dy, y, dx, stat, g, torch.zeros(2 * Cc, device=DEV), dg, db, relu=True, bits=m)
        got.append((dx, dg, db))
    # the sums of the blocks meet in any order: last digits of fp32, and the bf16 rounding they may tip
    assert torch.allclose(got[0][0].float(), got[1][0].float(), atol=1e-5, rtol=2.0 ** -7)
    assert torch.allclose(got[0][1], got[1][1], atol=1e-4, rtol=1e-4) and torch.allclose(got[0][2], got[1][2], atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("B,H,W,Cc,k,stride,pad", [(40, 5, 5, 24, 3, 1, 1), (3, 1, 1, 8, 1, 1, 0), (5, 4, 4, 8, 2, 2, 0),
                                                   (2, 9, 257, 8, 3, 2, 1), (2, 3, 130, 16, 3, 1, 1), (1, 5, 3, 2056, 3, 1, 1), (3, 9, 9, 16, 5, 1, 2),
                                                   (2, 7, 7, 1024, 7, 1, 0), (4, 8, 8, 40, 5, 2, 2)])
def test_average_pooling_over_launch_shapes(B, H, W, Cc, k, stride, pad):
    """Several rows in a block (with a ragged last block), rows in even shares over two blocks, more vectors than threads;
    windows of up to three taps per direction and more."""
    torch.manual_seed(H * W + Cc)
    x = torch.randn(B, H, W, Cc, device=DEV).to(BF)
    g = F.pool_geom(x.shape, k, stride, pad, Cc, Cc, ceil_mode=False)
    y = torch.empty(B, g.OH, g.OW, Cc, dtype=BF, device=DEV)
    F.avgpool_forward(x, y, g)
    dy = torch.randn_like(y)
    dx = torch.empty_like(x)
    F.avgpool_backward(dy, dx, g)
    xr = x.double().permute(0, 3, 1, 2).contiguous().requires_grad_(True)      # NCHW-contiguous reference
    ref = TF.avg_pool2d(xr, k, stride, pad)
    ref.backward(dy.double().permute(0, 3, 1, 2).contiguous())
    # one rounding to bf16 of fp32 sums of at most 9 terms
    assert torch.allclose(y.double(), ref.detach().permute(0, 2, 3, 1), atol=1e-5, rtol=2.0 ** -8)
    assert torch.allclose(dx.double(), xr.grad.permute(0, 2, 3, 1), atol=1e-5, rtol=2.0 ** -8)


def test_average_pooling_of_an_empty_batch_and_of_very_wide_rows():
    x = torch.empty(0, 6, 6, 16, dtype=BF, device=DEV)
    g = F.pool_geom(x.shape, 3, 1, 1, 16, 16)
    y = torch.empty(0, g.OH, g.OW, 16, dtype=BF, device=DEV)
    F.avgpool_forward(x, y, g)
    F.avgpool_backward(y, x, g)
    W = 65540                                                        # more pixels in a row than the grid's second dimension
    x = torch.randn(1, 1, W, 2048, device=DEV).to(BF)
    g = F.pool_geom(x.shape, 1, 1, 0, 2048, 2048)
    y, dx = torch.empty_like(x), torch.empty_like(x)
    F.avgpool_forward(x, y, g)
    F.avgpool_backward(y, dx, g)
    assert torch.equal(y, x) and torch.equal(dx, x)


@pytest.mark.parametrize("P,Cc", [(1, 8), (5, 24), (300, 1032), (2000, 2056)])
@pytest.mark.parametrize("pitched", [(False, False), (True, False), (False, True), (True, True)])
def test_sums_of_dense_and_pitched_matrices(P, Cc, pitched):
    torch.manual_seed(P)
    full = [torch.randn(P, Cc + (16 if p else 0), device=DEV).to(BF) for p in (*pitched, False)]
    dst, s0, s1 = (t[:, 8:8 + Cc] if t.shape[1] > Cc else t for t in full)
    edges = full[0].clone()
    ref = (dst.double() + s0.double() + s1.double()).to(BF).double()
    F.add_2d_n(dst, [s0, s1])
    assert torch.allclose(dst.double(), ref, atol=0, rtol=2.0 ** -7)      # fp32 sum: at most the other neighbour
    if pitched[0]:
        assert torch.equal(full[0][:, :8], edges[:, :8]) and torch.equal(full[0][:, 8 + Cc:], edges[:, 8 + Cc:])


_COOP = """
import torch
from geeps_b200.ops import functional as F
BF, dev = torch.bfloat16, torch.device("cuda:0")
for P, C in ((5, 8), (777, 104), (64, 2056), (3000, 192)):
    torch.manual_seed(P)
    x, dy = torch.randn(P, C, device=dev).to(BF), torch.randn(P, C, device=dev).to(BF)
    g, b = torch.rand(C, device=dev) + 0.5, torch.randn(C, device=dev)
    z = lambda: torch.zeros(2 * C, device=dev)
    got = []
    for bar in (torch.zeros(8, dtype=torch.int32, device=dev), None):
        y, stat, rm, rv = torch.empty_like(x), z(), torch.zeros(C, device=dev), torch.ones(C, device=dev)
        bits = torch.full((P, C // 8), 0xa5, dtype=torch.uint8, device=dev)
        dx, dg, db = torch.empty_like(x), torch.empty(C, device=dev), torch.empty(C, device=dev)
        F.bn_forward_fused(x, y, g, b, z(), stat, rm, rv, barrier=bar[:4] if bar is not None else None, relu=True, bits=bits)
        want = ((y.view(P, C // 8, 8) > 0).long() << torch.arange(8, device=dev)).sum(2)
        assert torch.equal(bits.long(), want), (P, C, bar is None)
        F.bn_backward_fused(x, dy, torch.ones_like(y), dx, stat, g, z(), dg, db, barrier=bar[4:] if bar is not None else None,
                            relu=True, bits=bits)
        got.append((y, stat, dx, dg, db))
    for u, v in zip(*got):      # sums of blocks meet in any order
        assert torch.allclose(u.float(), v.float(), atol=1e-4, rtol=2.0 ** -7), (P, C)
print("ok")
"""


def test_batchnorm_in_one_launch_keeps_and_reads_the_mask_bits():
    """GEEPS_BN_COOP=1 (read once per process): one cooperative launch per direction writes the same mask, and its backward
    pass reads it in the place of y."""
    import os
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-c", _COOP], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, GEEPS_BN_COOP="1"), cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]


@pytest.mark.parametrize("dtype", [torch.float32, torch.uint8])
def test_recorded_step_keeps_the_input_layers_output(dtype):
    """A plain NHWC input layer makes its output anew; the address that a recording names must not be given away."""
    from geeps_b200.ops.layers import Input
    inp = Input(cpad=8)
    inp.setup((4, 3, 24, 24), DEV)
    x = torch.zeros(4, 3, 24, 24, device=DEV).to(dtype)
    stream = torch.cuda.Stream(device=DEV)
    with torch.cuda.stream(stream):
        inp.forward(x)
        L.start_recording()
        address = inp.forward(x).data_ptr()           # dropped at once
        tape = L.stop_recording()
        graph = L.StepGraph(tape, stream)
        del tape
        others = [torch.empty(4, 24, 24, 8, device=DEV, dtype=BF) for _ in range(8)]
        assert address not in [t.data_ptr() for t in others]
        graph.launch()
    torch.cuda.synchronize()
    graph.close()


@pytest.mark.parametrize("off", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 1023, 4099, 2_000_003])
def test_clear_covers_exactly_its_range(off, n):
    """Heads and tails around 16-byte boundaries; more vectors than threads at the largest."""
    buf = torch.full((n + 16,), 2.0, device=DEV)
    L.check(L.lib().geeps_clear_f32(ctypes.c_void_p(buf.data_ptr() + 4 * (4 + off)), ctypes.c_longlong(n), L.stream_ptr()), "clear")
    assert (buf[4 + off:4 + off + n] == 0).all()
    assert (buf[:4 + off] == 2).all() and (buf[4 + off + n:] == 2).all()


@pytest.mark.parametrize("B,H,W,C,pad,extra", [(1, 3, 4, 8, 0, 0), (2, 4, 3, 8, 0, 8), (3, 13, 13, 256, 0, 0), (2, 14, 9, 24, 1, 16), (2, 5, 12, 40, 2, 0),
                                               (1, 3, 3, 8, 1, 0), (5, 57, 30, 136, 0, 8)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_maxpool_backward_by_quads(B, H, W, C, pad, extra, accumulate):
    """3 x 3 windows at stride 2, even and odd sizes and pads, pitched tensors: the sums of bf16 in the order of the windows."""
    torch.manual_seed(H * C)
    x = torch.randn(B, H, W, C + extra, device=DEV).to(BF)[..., :C]
    g = F.pool_geom((B, H, W, C), 3, 2, pad, C + extra, C + extra)
    y = torch.empty(B, g.OH, g.OW, C + extra, dtype=BF, device=DEV)[..., :C]
    arg = torch.empty(B, g.OH, g.OW, C, dtype=torch.uint8, device=DEV)
    F.maxpool_forward(x, y, arg, g)
    dy = torch.randn(B, g.OH, g.OW, C + extra, device=DEV).to(BF)[..., :C]
    wide = torch.randn(B, H, W, C + extra, device=DEV).to(BF)
    before = wide.clone()
    F.maxpool_backward(dy, arg, wide[..., :C], g, accumulate=accumulate)
    acc = torch.zeros(B, H + 2 * pad + 4, W + 2 * pad + 4, C, dtype=BF, device=DEV)       # padded image; windows may end past it
    for kh in (2, 1, 0):
        for kw in (2, 1, 0):
            view = acc[:, kh:kh + 2 * g.OH:2, kw:kw + 2 * g.OW:2]
            view += torch.where(arg == kh * 3 + kw, dy, torch.zeros_like(dy))
    want = acc[:, pad:pad + H, pad:pad + W]
    assert torch.equal(wide[..., :C], want + before[..., :C] if accumulate else want)
    assert torch.equal(wide[..., C:], before[..., C:])


@pytest.mark.parametrize("K,stride,pad", [(3, 2, 0), (3, 2, 1), (2, 2, 0), (3, 1, 1), (15, 7, 0)])
def test_maxpool_applies_the_mask_of_a_relu(K, stride, pad):
    """Windows that are all zeros or negative hand their gradient to nobody: the masked gradient of the plain passes, bit for bit."""
    torch.manual_seed(K)
    B, H, C = 3, 29, 40
    x = torch.relu(torch.randn(B, H, H, C, device=DEV) - 1.2).to(BF)
    x[0, :20, :20] = 0
    x[1, 3, 4] = -1.0                                                # not from a ReLU: masked by sign all the same
    g = F.pool_geom((B, H, H, C), K, stride, pad, C, C)
    y, ym, dy = (torch.randn(B, g.OH, g.OW, C, device=DEV).to(BF) for _ in range(3))
    arg, argm = (torch.empty(B, g.OH, g.OW, C, dtype=torch.uint8, device=DEV) for _ in range(2))
    dx, dxm = torch.empty_like(x), torch.empty_like(x)
    F.maxpool_forward(x, y, arg, g)
    F.maxpool_backward(dy, arg, dx, g)
    F.maxpool_forward(x, ym, argm, g, relu_mask=True)
    F.maxpool_backward(dy, argm, dxm, g)
    assert torch.equal(y, ym) and (argm == 255).any() and torch.equal(argm[argm != 255], arg[argm != 255])
    assert torch.equal(dxm, torch.where(x > 0, dx, torch.zeros_like(dx)))


@pytest.mark.parametrize("P,C", [(81920, 64), (81921, 64), (30000, 200)])
def test_batchnorm_passes_one_after_the_other(P, C):
    """Tensors on both sides of the size from which a pass lets the next one in only at its end: three forward and backward
    passes back to back, the last one's results against the formulas in fp32."""
    torch.manual_seed(P)
    x, dy = (torch.randn(P, C, device=DEV).to(BF) for _ in range(2))
    y, dx, bits = torch.empty_like(x), torch.empty_like(x), torch.empty(P, C // 8, dtype=torch.uint8, device=DEV)
    g, b = 1 + 0.1 * torch.randn(C, device=DEV), 0.1 * torch.randn(C, device=DEV)
    s, sb, mr = torch.zeros(2 * C, device=DEV), torch.zeros(2 * C, device=DEV), torch.empty(2 * C, device=DEV)
    rm, rv, dg, db = torch.zeros(C, device=DEV), torch.ones(C, device=DEV), torch.empty(C, device=DEV), torch.empty(C, device=DEV)
    bar = torch.zeros(8, dtype=torch.int32, device=DEV)
    for _ in range(3):
        F.bn_forward_fused(x, y, g, b, s, mr, rm, rv, zero_after=sb, barrier=bar[0:4], eps=1e-5, momentum=0.1, relu=True, bits=bits)
        F.bn_backward_fused(x, dy, y, dx, mr, g, sb, dg, db, zero_after=s, barrier=bar[4:8], relu=True, bits=bits)
    xf = x.float()
    mean, rstd = xf.mean(0), (xf.var(0, unbiased=False) + 1e-5).rsqrt()
    xh = (xf - mean) * rstd
    dz = torch.where(y > 0, dy.float(), torch.zeros((), device=DEV))
    # results are rounded to bf16 once: 2^-8 of a value, of which half is the bound
    assert ((y.float() - torch.relu(xh * g + b)).norm() / y.float().norm()).item() < 2.0 ** -8
    want = g * rstd * (dz - dz.mean(0) - xh * (dz * xh).mean(0))
    assert ((dx.float() - want).norm() / want.norm()).item() < 2.0 ** -8
    # sums of P terms of fp32 in some order: sqrt(P) 2^-24 of the terms' norm each way
    assert (dg - (dz * xh).sum(0)).abs().max().item() < 1e-4 * P ** 0.5 and (db - dz.sum(0)).abs().max().item() < 1e-4 * P ** 0.5


@pytest.mark.parametrize("off,n", [(0, 1), (1, 2), (3, 4), (2, 1023), (0, 614400), (1, 5_000_001)])
@pytest.mark.parametrize("P,C", [(3, 8), (5000, 384), (11000, 384)])
def test_relu_backward_clears_a_range_on_the_way(off, n, P, C):
    """Fewer and more values than the launch has threads, off 16-byte boundaries, and a pass that leaves them to a launch of their
    own: the range, nothing beside it, and the results of
    a call without one."""
    dy, y = torch.randn(P, C, device=DEV).to(BF), torch.randn(P, C, device=DEV).to(BF)
    buf = torch.full((n + 16,), 2.0, device=DEV)
    dx, cs = [torch.empty_like(y) for _ in range(2)], [torch.empty(C, device=DEV) for _ in range(2)]
    F.relu_backward_colsum(dy, y, dx[0], cs[0])
    F.relu_backward_colsum(dy, y, dx[1], cs[1], clear=buf[4 + off:4 + off + n])
    assert torch.equal(dx[0], dx[1]) and torch.allclose(cs[0], cs[1], atol=1e-3 * P ** 0.5, rtol=0)
    assert (buf[4 + off:4 + off + n] == 0).all() and (buf[:4 + off] == 2).all() and (buf[4 + off + n:] == 2).all()


@pytest.mark.parametrize("B,H,Cc,pad,ldy", [(64, 29, 8, 0, 8), (61, 31, 8, 1, 8), (40, 13, 120, 0, 136), (9, 61, 40, 1, 40),
                                            (3, 27, 240, 0, 240), (2, 28, 312, 0, 312), (100, 14, 88, 1, 88),
                                            (260, 27, 32, 0, 32), (40, 24, 296, 0, 296), (36, 15, 520, 0, 520)])
@pytest.mark.parametrize("alpha", [1e-4, 0.01, 0.5])
def test_lrn_maxpool_backward_by_quads_matches_small_batches(B, H, Cc, pad, ldy, alpha):
    """A batch large enough for the quad kernel (one step a warp and several, ends of rows and images inside a warp,
    one vector a pixel, vector counts without a common factor with 30) against single images, which the other kernels take:
    the same bits, in the range of the polynomials, beyond it, and on the vectors between whose largest window is inside while
    the sum of all their squares is not."""
    torch.manual_seed(B * Cc)
    size, beta, kk = 5, 0.75, 1.0
    x = (torch.randn(B, H, H, Cc, device=DEV) * 3).clamp_min(-0.5).to(BF)        # some negative inputs: masked by sign
    g = F.pool_geom(x.shape, 3, 2, pad, Cc, ldy)
    vectors, line = ((H + pad + 1) // 2) ** 2 * Cc // 8, 96 * torch.cuda.get_device_properties(0).multi_processor_count
    assert B * vectors >= line > vectors
    arg = torch.randint(0, 9, (B, g.OH, g.OW, Cc), device=DEV, dtype=torch.uint8)
    dp = torch.randn(B, g.OH, g.OW, ldy, device=DEV).to(BF)
    dx, cs = torch.empty_like(x), torch.empty(Cc, device=DEV)
    F.lrn_maxpool_backward(x, dp, arg, dx, g, size, alpha, beta, kk, relu_mask=True, colsum=cs)
    one = F.pool_geom(x[:1].shape, 3, 2, pad, Cc, ldy)
    ref, part, total = torch.empty_like(x[:1]), torch.empty(Cc, device=DEV), torch.zeros(Cc, dtype=torch.float64, device=DEV)
    for b in range(B):
        F.lrn_maxpool_backward(x[b:b + 1], dp[b:b + 1], arg[b:b + 1], ref, one, size, alpha, beta, kk, relu_mask=True, colsum=part)
        total += part
        assert torch.equal(dx[b:b + 1], ref), b
    # n additions, each rounded by at most 2^-24 of the sum of magnitudes, with random signs: four deviations
    mag = dx.double().abs().sum((0, 1, 2))
    bound = 4 * 2.0 ** -24 * (B * H * H) ** 0.5 * mag
    assert ((cs.double() - total).abs() <= bound).all()


def test_lrn_maxpool_backward_by_quads_with_infinities_and_nans():
    """What an infinity or a NaN spoils by quads and in single images: the same places, and the same bits beside an infinity."""
    torch.manual_seed(3)
    B, H, Cc = 40, 13, 120
    x = torch.randn(B, H, H, Cc, device=DEV).to(BF)
    flat = x.view(-1)
    at = torch.randperm(flat.numel(), device=DEV)[:3000]
    flat[at[:1500]] = float("inf")
    g = F.pool_geom(x.shape, 3, 2, 0, Cc, Cc)
    one = F.pool_geom(x[:1].shape, 3, 2, 0, Cc, Cc)
    arg = torch.randint(0, 9, (B, g.OH, g.OW, Cc), device=DEV, dtype=torch.uint8)
    arg[:, ::2] = 4                                    # rows of pixels that no window points at
    dp = torch.randn(B, g.OH, g.OW, Cc, device=DEV).to(BF)
    dx, ref = torch.empty_like(x), torch.empty_like(x)
    for nans in (False, True):
        if nans:
            flat[at[1500:]] = float("nan")
        F.lrn_maxpool_backward(x, dp, arg, dx, g, 5, 1e-4, 0.75, 1.0)
        for b in range(B):
            F.lrn_maxpool_backward(x[b:b + 1], dp[b:b + 1], arg[b:b + 1], ref[b:b + 1], one, 5, 1e-4, 0.75, 1.0)
        bad = ref.isnan()
        assert bad.any() and not bad.all() and torch.equal(dx.isnan(), bad)
        if nans:      # a vector with a NaN takes the exact power by quads, the polynomial (4e-4) otherwise; two roundings to bf16
            assert torch.allclose(dx[~bad].float(), ref[~bad].float(), rtol=2.0 ** -7, atol=1e-3)
        else:
            assert torch.equal(dx[~bad], ref[~bad])


@pytest.mark.parametrize("B,H,W,Cc,pad,ldx,ldy", [(33, 15, 14, 96, 1, 96, 112), (40, 8, 9, 256, 0, 272, 256), (65, 5, 7, 304, 2, 304, 304),
                                                  (30, 3, 3, 2312, 1, 2312, 2320), (2, 1, 9, 8, 1, 8, 8), (3, 4, 5, 16, 2, 24, 32)])
def test_average_pooling_3x3_stride_1(B, H, W, Cc, pad, ldx, ldy):
    """Four rows a thread and one, rows that are no multiple of four, images of one row, pitched input and output, and the
    backward pass added to what is there."""
    torch.manual_seed(H * W + Cc)
    x = torch.randn(B, H, W, ldx, device=DEV).to(BF)
    g = F.pool_geom((B, H, W, Cc), 3, 1, pad, ldx, ldy, ceil_mode=False)
    y = torch.full((B, g.OH, g.OW, ldy), 7.0, dtype=BF, device=DEV)
    F.avgpool_forward(x, y, g)
    dy = torch.randn_like(y)
    xr = x[..., :Cc].double().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    ref = TF.avg_pool2d(TF.pad(xr, (pad, pad, pad, pad)), 3, 1)
    ref.backward(dy[..., :Cc].double().permute(0, 3, 1, 2).contiguous())
    want, grad = ref.detach().permute(0, 2, 3, 1), xr.grad.permute(0, 2, 3, 1)
    # one rounding to bf16 of fp32 sums of at most ten terms
    assert torch.allclose(y[..., :Cc].double(), want, atol=1e-5, rtol=2.0 ** -8)
    assert (y[..., Cc:] == 7).all()
    dx = torch.randn(B, H, W, ldx, device=DEV).to(BF)
    old = dx.clone()
    for accumulate in (1, 0):
        dx.copy_(old)
        L.check(L.lib().geeps_avgpool_backward(L.ptr(dy), L.ptr(dx), ctypes.byref(g), accumulate, L.stream_ptr()), "avgpool_backward")
        assert torch.allclose(dx[..., :Cc].double(), grad + (old[..., :Cc].double() if accumulate else 0.0), atol=1e-5, rtol=2.0 ** -8)
        assert torch.equal(dx[..., Cc:], old[..., Cc:])
