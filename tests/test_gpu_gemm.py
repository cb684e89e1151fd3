"""tcgen05 GEMM vs a plain PyTorch fp32 reference of the same product."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from geeps_b200.ops import functional as F
from geeps_b200.ops import _lib as L


def _ref(a, b, a_mn, b_mn):
    A = a.float().t() if a_mn else a.float()
    Bm = b.float().t() if b_mn else b.float()
    return A @ Bm.t()


def _mk(rows, k, mn, dev, pad=0):
    shape = (k, rows + pad) if mn else (rows, k + pad)
    t = (torch.randn(shape, device=dev) * 0.5).to(torch.bfloat16)
    return t[:, :rows] if mn else t[:, :k]


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 512, 1024), (200, 136, 328), (64, 1000, 4096), (384, 96, 72)])
def test_gemm_tc_matches_fp32(M, N, K, a_mn, b_mn):
    dev = torch.device("cuda:0")
    torch.manual_seed(M * 7 + N * 3 + K)
    a = _mk(M, K, a_mn, dev, pad=8)
    b = _mk(N, K, b_mn, dev, pad=16)
    out = torch.empty((M, N), dtype=torch.float32, device=dev)
    st = L.new_status(dev)
    F.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, status=st, impl="tc")
    torch.cuda.synchronize()
    assert L.read_status(st)["code"] == 0, L.read_status(st)
    ref = _ref(a, b, a_mn, b_mn)
    assert torch.allclose(out, ref, atol=1e-2, rtol=1e-2), (out - ref).abs().max().item()


@pytest.mark.parametrize("bn", [64, 128, 256])
def test_gemm_tc_block_n_and_epilogue(bn):
    dev = torch.device("cuda:0")
    torch.manual_seed(bn)
    M, N, K = 300, 520, 448
    a = (torch.randn(M, K, device=dev) * 0.3).to(torch.bfloat16)
    b = (torch.randn(N, K, device=dev) * 0.3).to(torch.bfloat16)
    bias = torch.randn(N, device=dev)
    wide = torch.zeros((M, N + 24), dtype=torch.bfloat16, device=dev)
    out = wide[:, 8:8 + N]  # column slice of a wider matrix: exercises ldc and unaligned stores
    st = L.new_status(dev)
    F.gemm(a, b, out, bias=bias, relu=True, alpha=0.5, block_n=bn, status=st, impl="tc")
    torch.cuda.synchronize()
    assert L.read_status(st)["code"] == 0
    ref = torch.relu(0.5 * (a.float() @ b.float().t()) + bias)
    assert torch.allclose(out.float(), ref, atol=6e-2, rtol=2e-2)
    assert wide[:, :8].abs().max().item() == 0 and wide[:, 8 + N:].abs().max().item() == 0


def test_gemm_tc_beta_and_bias_m():
    dev = torch.device("cuda:0")
    torch.manual_seed(5)
    M, N, K = 160, 264, 200
    a = (torch.randn(M, K, device=dev) * 0.3).to(torch.bfloat16)
    b = (torch.randn(N, K, device=dev) * 0.3).to(torch.bfloat16)
    bias = torch.randn(M, device=dev)
    c0 = torch.randn(M, N, device=dev)
    out = c0.clone()
    F.gemm(a, b, out, bias=bias, bias_mode=2, beta=0.75, impl="tc")
    ref = a.float() @ b.float().t() + 0.75 * c0 + bias[:, None]
    torch.cuda.synchronize()
    assert torch.allclose(out, ref, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("split", [0, 4])
def test_gemm_tc_split_k(split):
    dev = torch.device("cuda:0")
    torch.manual_seed(11)
    M, N, K = 96, 368, 8192  # weight-gradient shape: tiny output, very long K
    a = (torch.randn(K, M, device=dev) * 0.1).to(torch.bfloat16)   # stored [K, M]
    b = (torch.randn(K, N, device=dev) * 0.1).to(torch.bfloat16)   # stored [K, N]
    out = torch.full((M, N), 3.0, device=dev)
    F.gemm(a, b, out, a_mn=True, b_mn=True, beta=0.0, split_k=split, impl="tc")
    torch.cuda.synchronize()
    ref = a.float().t() @ b.float()
    assert torch.allclose(out, ref, atol=3e-2, rtol=1e-2)


def test_gemm_simt_matches_tc():
    dev = torch.device("cuda:0")
    torch.manual_seed(3)
    M, N, K = 130, 77, 90
    a = (torch.randn(M, K, device=dev) * 0.3).to(torch.bfloat16)
    b = (torch.randn(N, K, device=dev) * 0.3).to(torch.bfloat16)
    out = torch.empty((M, N), dtype=torch.float32, device=dev)
    F.gemm(a, b, out, impl="auto")  # K=90 is not a multiple of 8: takes the SIMT path
    torch.cuda.synchronize()
    assert torch.allclose(out, a.float() @ b.float().t(), atol=1e-2, rtol=1e-2)


@pytest.mark.parametrize("M,N,K,bn,fp32", [(512, 64, 256, 64, False), (512, 256, 256, 256, False),
                                           (1000, 384, 520, 0, False), (4096, 1000, 1024, 0, True)])
def test_gemm_cta_pair_matches_fp32(M, N, K, bn, fp32):
    """CTA-pair kernel (tcgen05 cta_group::2, 256-row tiles): bias + ReLU epilogue, ragged M / N / K edges."""
    dev = torch.device("cuda:0")
    torch.manual_seed(M + N + K)
    a = _mk(M, K, False, dev, pad=8)
    b = _mk(N, K, False, dev, pad=16)
    bias = torch.randn(N, device=dev)
    out = torch.full((M, N + 8), 7.0, dtype=torch.float32 if fp32 else torch.bfloat16, device=dev)[:, :N]
    st = L.new_status(dev)
    F.gemm(a, b, out, bias=bias, relu=True, block_n=bn, status=st, impl="pair")
    torch.cuda.synchronize()
    assert L.read_status(st)["code"] == 0, L.read_status(st)
    ref = torch.relu(_ref(a, b, False, False) + bias)
    assert ((out.float() - ref).norm() / ref.norm()).item() < (1e-5 if fp32 else 5e-3)


def test_gemm_auto_dispatch_uses_pairs_for_large_products():
    dev = torch.device("cuda:0")
    torch.manual_seed(5)
    M, N, K = 20000, 512, 192
    a, b = _mk(M, K, False, dev), _mk(N, K, False, dev)
    out = torch.empty((M, N), dtype=torch.bfloat16, device=dev)
    F.gemm(a, b, out)
    ref = _ref(a, b, False, False)
    assert ((out.float() - ref).norm() / ref.norm()).item() < 5e-3


@pytest.mark.parametrize("M,N,K,b_mn,fp32,cluster", [(256, 512, 8200, False, False, True), (5, 1000, 8264, False, True, True),
                                                     (32, 1024, 21841, True, False, True), (129, 200, 8328, True, True, True),
                                                     (256, 1000, 4096, False, False, False), (100, 72, 16392, False, True, True),
                                                     (1, 200, 8192, False, False, True), (257, 330, 8129, False, False, True)])
def test_gemm_cluster_split_k(M, N, K, b_mn, fp32, cluster):
    """Few output tiles, long K: slices of one tile on the CTAs of a cluster (uneven last slice, ragged M and N, column
    slices that end on odd widths), bias and ReLU applied once; the same bits on every run.  One product takes narrow tiles
    without a cluster."""
    dev = torch.device("cuda:0")
    torch.manual_seed(M + N + K)
    kp = (K + 7) // 8 * 8
    a = _mk(M, kp, False, dev)[:, :K]
    b = _mk(N, K, b_mn, dev, pad=8 if b_mn else kp - K)
    bias = torch.randn(N, device=dev)
    wide = torch.zeros((M, N + 16), dtype=torch.float32 if fp32 else torch.bfloat16, device=dev)
    out = wide[:, 8:8 + N]
    st = L.new_status(dev)
    p, plan = L.GemmParams(), L.GemmPlan()
    p.A, p.B, p.C, p.bias, p.bias_mode = a.data_ptr(), b.data_ptr(), out.data_ptr(), bias.data_ptr(), 1
    p.M, p.N, p.K, p.lda, p.ldb, p.ldc = M, N, K, a.stride(0), b.stride(0), out.stride(0)
    p.alpha, p.b_mn_major, p.out_fp32, p.relu, p.split_k = 0.5, int(b_mn), int(fp32), 1, 1
    assert L.lib().geeps_gemm_plan(ctypes.byref(p), ctypes.byref(plan)) == 1 and (plan.cluster > 1) == cluster
    F.gemm(a, b, out, b_mn=b_mn, bias=bias, relu=True, alpha=0.5, status=st, impl="tc")
    torch.cuda.synchronize()
    assert L.read_status(st)["code"] == 0
    A, B = a.double(), (b.double().t() if b_mn else b.double())
    ref = torch.relu(0.5 * (A @ B.t()) + bias)
    # fp32 sums of K products of size 1/4: K^0.5 * 2^-24 * a few, then the rounding of the output type
    assert torch.allclose(out.double(), ref, atol=2e-6 * K ** 0.5 * 4, rtol=2.0 ** -8 if not fp32 else 1e-5)
    assert wide[:, :8].abs().max().item() == 0 and wide[:, 8 + N:].abs().max().item() == 0
    again = torch.empty_like(wide)[:, 8:8 + N]
    F.gemm(a, b, again, b_mn=b_mn, bias=bias, relu=True, alpha=0.5, impl="tc")
    assert torch.equal(out, again)


@pytest.mark.parametrize("captured", [False, True])
def test_dependent_launches_keep_reads_and_writes_in_order(captured):
    """A product may come up while its predecessor runs.  Each here overwrites what the one before reads, or reads what it
    writes, in one stream, across an event and around a copy; results are those of one call at a time, bitwise."""
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(5)
    n, deep = 256, 4096
    rnd = lambda *s: (torch.randn(*s, device=dev, generator=gen) * 0.05).to(torch.bfloat16)      # noqa: E731
    first, w, u, v, other = rnd(n, deep), rnd(n, deep), rnd(n, n), rnd(deep, n), rnd(n, deep)
    main, side = torch.cuda.Stream(device=dev), torch.cuda.Stream(device=dev)
    torch.cuda.synchronize()

    def run(a, outs, pause):
        event = iter(events)
        with torch.cuda.stream(main):
            a.copy_(first); pause()
            F.gemm(a, w, outs[0]); pause()             # long K: the successor's blocks are there before it ends
            F.gemm(u, v, a); pause()                   # overwrites the operand of the one before
            F.gemm(a, w, outs[1]); pause()             # reads what was just written
            a.copy_(other); pause()                    # a copy behind a product and in front of one
            F.gemm(a, w, outs[2]); pause()
            F.stream_order(main, side, next(event))
        with torch.cuda.stream(side):
            F.gemm(a, w, outs[3]); pause()             # beside the main stream
            F.colsum(a, outs[5]); pause()
        F.stream_order(side, main, next(event))
        with torch.cuda.stream(main):
            F.gemm(u, v, a); pause()                   # overwrites what the other stream reads
            F.gemm(a, w, outs[4]); pause()

    def buffers():
        return rnd(n, deep), [torch.zeros(n, n, device=dev, dtype=torch.bfloat16) for _ in range(5)] + [torch.zeros(deep, device=dev)]

    events = [F.new_event() for _ in range(2)]
    a, ref = buffers()
    run(a, ref, torch.cuda.synchronize)
    a, got = buffers()
    torch.cuda.synchronize()
    if captured:
        graph, nodes = ctypes.c_void_p(), ctypes.c_longlong(0)
        assert L.lib().geeps_graph_begin(ctypes.c_void_p(main.cuda_stream)) == 0
        run(a, got, lambda: None)
        assert L.lib().geeps_graph_end(ctypes.c_void_p(main.cuda_stream), ctypes.byref(graph), ctypes.byref(nodes)) == 0
        for _ in range(20):
            assert L.lib().geeps_graph_launch(graph, ctypes.c_void_p(main.cuda_stream)) == 0
        torch.cuda.synchronize()
        L.lib().geeps_graph_destroy(graph)
    else:
        for _ in range(20):
            run(a, got, lambda: None)
        torch.cuda.synchronize()
    for r, g in zip(ref[:5], got[:5]):
        assert torch.equal(r, g)
    assert torch.allclose(ref[5], got[5], atol=1e-4)   # block sums meet in atomics
