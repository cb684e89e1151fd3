"""How the tcgen05 GEMM cuts a product (host arithmetic only, no GPU: the planner then assumes the 148 SMs of a B200)."""
import ctypes as C
import itertools

import pytest
import torch

from geeps_b200.ops import _lib as L

SMS = 148
pytestmark = pytest.mark.skipif(torch.cuda.is_available() and torch.cuda.get_device_properties(0).multi_processor_count != SMS,
                                reason="the sweep states its bounds for 148 SMs")


def plan(M, N, K, *, fp32=False, split_k=1, relu=False, a_mn=False, b_mn=False, beta=0.0, block_n=0):
    p = L.GemmParams()
    p.A, p.B, p.C, p.bias, p.status = 0x10000, 0x20000, 0x30000, None, None
    p.M, p.N, p.K = M, N, K
    p.lda, p.ldb, p.ldc = ((v + 7) // 8 * 8 for v in (M if a_mn else K, N if b_mn else K, N))
    p.alpha, p.beta = 1.0, beta
    p.a_mn_major, p.b_mn_major, p.out_fp32, p.bias_mode, p.relu = int(a_mn), int(b_mn), int(fp32), 0, int(relu)
    p.split_k, p.block_n = split_k, block_n
    out = L.GemmPlan()
    assert L.lib().geeps_gemm_plan(C.byref(p), C.byref(out)) == 1
    return out


SIZES = list(itertools.product((1, 32, 100, 128, 129, 256, 512, 1000, 1152, 4096), (8, 64, 72, 200, 1000, 1024, 4096, 9216),
                               (8, 64, 512, 520, 960, 1024, 2048, 9216, 21841)))


@pytest.mark.parametrize("fp32,split_k,relu", [(False, 1, True), (True, 1, False), (True, 0, False), (False, 0, False),
                                               (True, 0, True), (True, 4, False)])
@pytest.mark.parametrize("mn", [(False, False), (False, True), (True, True)])
def test_plans_cover_the_product(fp32, split_k, relu, mn):
    for M, N, K in SIZES:
        g = plan(M, N, K, fp32=fp32, split_k=split_k, relu=relu, a_mn=mn[0], b_mn=mn[1])
        kt = (K + 63) // 64
        assert g.block_n % (64 if mn[1] else 32) == 0 and 32 <= g.block_n <= 256
        assert g.tiles == (M + 127) // 128 * ((N + g.block_n - 1) // g.block_n)
        per = -(-kt // g.split_k)
        assert 1 <= g.split_k <= kt and (g.split_k - 1) * per < kt           # no empty K slice
        assert g.cluster in (1, g.split_k) and g.cluster <= 8
        if not fp32 or relu:
            assert g.split_k == g.cluster                                    # no atomics on a bf16 or ReLU output
        if split_k == 1 and g.cluster == 1:
            assert g.split_k == 1


@pytest.mark.parametrize("M,N", [(1000, 4096), (1152, 2048), (512, 4096), (4096, 512)])
@pytest.mark.parametrize("K", [512, 520, 960])
def test_short_k_is_spread_by_narrow_tiles_before_it_is_split(M, N, K):
    """fp32 weight gradients whose K (the batch) is 8 to 15 k tiles: narrow tiles that occupy every SM leave K whole."""
    g = plan(M, N, K, fp32=True, split_k=0, a_mn=True, b_mn=True)
    assert g.split_k == 1 or g.block_n == 64, (g.block_n, g.split_k, g.tiles)
    if M * N >= SMS * 128 * 64 * 2:
        assert g.split_k == 1 and g.tiles >= SMS * 0.8, (g.block_n, g.split_k, g.tiles)
