// bf16 GEMM on the 5th-generation tensor cores: TMA -> swizzled SMEM ring ->
// tcgen05.mma (one issuing thread) -> fp32 accumulators in TMEM -> tcgen05.ld epilogue.
//
//   C[M,N] = alpha * A[M,K] * B[N,K]^T + beta * C + bias, optional ReLU, bf16 or fp32 out.
//
// Both operands may be K-major (row-major [rows][K]) or MN-major (stored [K][rows]), so
// forward (X W^T), data-gradient (dY W) and weight-gradient (dY^T X) products of FC and
// im2col-conv layers all run here without materialising a transpose.
//
// Persistent CTAs (one per SM) of 10 warps: warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, two groups of four
// epilogue warps (one TMEM lane quarter each), which take alternate column slabs: a product with a short K is bound by its
// epilogue (fp32 gradients: 21841 x 1024, K = 32: 22.5 us with one group, 18.2 with two; 4096 x 4096, K = 256: 20.0, 18.4).  Two accumulators live in TMEM, so the epilogue
// of a tile overlaps the main loop of the next one.  Tile 128 x BN x 64 with BN any multiple of 32
// up to 256 (chosen per problem so that narrow outputs do not pad the MMA); partial tiles are
// handled by TMA zero fill on loads and bounds checks on stores, so any M, N, K work as
// long as the leading dimensions are multiples of 8 elements (16 bytes).
// Every mbarrier wait is bounded; on expiry the CTA records TIMEOUT in `status`, stops
// issuing work, frees its TMEM and returns.
//
// Outputs with too few tiles for the machine (batch-sized M) split K over the CTAs of a thread-block cluster: every CTA
// accumulates one K slice of the same tile, leaves it in its shared memory as fp32, and each CTA of the cluster then
// sums its share of the rows over distributed shared memory in slice order (no workspace, no atomics, bit-reproducible).
//
// The reference has no GEMM kernel of its own: it only carries cuBLAS wrappers
// (src/common/gpu-util/math_functions_cuda.cu:14-60) that the parameter server never calls.
#include <cuda.h>
#include <mutex>
#include <stdio.h>

#include "kernels.h"
#include "tc05.cuh"

namespace {

constexpr int BM = 128;
constexpr int BK = 64;              // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;   // 16 KB
constexpr int MAX_STAGES = 8;
constexpr uint64_t WAIT_BUDGET_NS = 2000000000ull;  // 2 s
constexpr int C_SLAB_BYTES = BM * 128;       // epilogue staging slab: 128 rows x 128 bytes, two per epilogue group
constexpr int epi_groups(bool cl) { return cl ? 1 : 2; }
constexpr int gemm_threads(bool cl) { return 64 + 128 * epi_groups(cl); }

struct GemmDev {
  void* C; const float* bias; int* status;
  long long M, N, K, ldc;
  float alpha, beta;
  int out_fp32, bias_mode, relu, split_k, kt_total, stages;
  int bn;           // tile width: multiple of 32 (64 for an MN-major B), <= 256
  int tmem_cols;    // power of two >= 2 * bn: two accumulators, so the epilogue of a tile overlaps the next main loop
  int m_tiles, n_tiles;
  int cluster;      // > 1: K slices of one tile per cluster of this many CTAs (split_k is then the same number)
  int slabs;        // staging slabs: two per epilogue group that has one to fill
  int tma_store;    // 1: epilogue stages 128-byte-wide slabs in swizzled smem and stores them with TMA
};

struct SmemCtl {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem_addr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// byte offset of the 16-byte piece `q` of row `r` in a [128][bn] fp32 tile; the XOR keeps a column of rows (how the
// accumulator comes out of TMEM, one row per lane) off a single bank
__device__ __forceinline__ uint32_t part_off(int r, int q, int bn) { return (uint32_t)(r * bn * 4 + ((q ^ (r & 7)) << 4)); }

// Persistent kernel: one CTA per SM walks the tile list t = blockIdx.x, blockIdx.x + gridDim.x, ...
// Consecutive CTAs take consecutive M tiles of the same N tile, so the B tile they share stays in L2.
// CL: a cluster of d.cluster CTAs per tile, one K slice each.
template <bool A_MN, bool B_MN, bool CL>
__global__ void __launch_bounds__(gemm_threads(CL), 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmC, const GemmDev d) {
  extern __shared__ uint8_t smem_raw[];
  const int BN = d.bn;
  const int B_STAGE_BYTES = BN * BK * 2;
  const int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* cslab = tiles + (size_t)d.stages * STAGE_BYTES;          // the slabs, 1024-byte aligned
  SmemCtl* ctl = (SmemCtl*)(cslab + (CL ? 0 : d.slabs * C_SLAB_BYTES));   // a cluster stages its tile in the operand ring

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = d.stages;
  const int kt_per = (d.kt_total + d.split_k - 1) / d.split_k;
  const int tiles_mn = d.m_tiles * d.n_tiles;
  const int num_tiles = tiles_mn * d.split_k;
  const int acc_stride = d.tmem_cols >> 1;
  // work items t, t + t_step, ...; a cluster CTA has one: K slice (rank) of tile blockIdx.x / cluster
  const int t_first = CL ? (int)(blockIdx.x % d.cluster) * tiles_mn + (int)(blockIdx.x / d.cluster) : (int)blockIdx.x;
  const int t_step = CL ? num_tiles : (int)gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { tc05::mbar_init(&ctl->full[s], 1); tc05::mbar_init(&ctl->empty[s], 1); }
    for (int a = 0; a < 2; ++a) { tc05::mbar_init(&ctl->tmem_full[a], 1); tc05::mbar_init(&ctl->tmem_empty[a], 4 * epi_groups(CL)); }
    ctl->abort_flag = 0;
    tc05::mbar_fence_init();
  }
  if (warp == 1) {
    tc05::tmem_alloc(&ctl->tmem_base, (uint32_t)d.tmem_cols);
    tc05::tmem_relinquish();
  }
  tc05::fence_before_sync();
  __syncthreads();
  tc05::fence_after_sync();
  const uint32_t tmem = ctl->tmem_base;
  geeps_pdl_wait();          // everything above touches this CTA's own memory only
  volatile int* abort_flag = &ctl->abort_flag;
  const uint32_t tiles_u = tc05::smem_u32(tiles), empty_u = tc05::smem_u32(ctl->empty);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    // the loop runs with the whole warp converged; the elected lane issues the copies
    {
      const bool leader = tc05::elect_one();
      if (leader) { tc05::tma_prefetch_desc(&tmA); tc05::tma_prefetch_desc(&tmB); }
      // ring slot and phase advance incrementally: a division per k-tile in this single thread would cost
      // more than issuing the loads
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = t_first; t < num_tiles && ok; t += t_step) {
        const int mn = t % tiles_mn, z = t / tiles_mn;
        const int m0 = (mn % d.m_tiles) * BM, n0 = (mn / d.m_tiles) * BN;
        const int kt_begin = z * kt_per, kt_end = min(d.kt_total, kt_begin + kt_per);
        for (int kt = kt_begin; kt < kt_end; ++kt) {
          if (!tc05::mbar_wait_warp(&ctl->empty[s], ph ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          uint8_t* sa = tiles + (size_t)s * STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE_BYTES;
          const int k0 = kt * BK;
          if (leader) {
          tc05::mbar_expect_tx(&ctl->full[s], STAGE_BYTES);
          if (A_MN) {
#pragma unroll
            for (int h = 0; h < BM / 64; ++h)
              tc05::tma_load_2d(sa + h * (64 * BK * 2), &tmA, &ctl->full[s], m0 + 64 * h, k0);
          } else {
            tc05::tma_load_2d(sa, &tmA, &ctl->full[s], k0, m0);
          }
          if (B_MN) {
            for (int h = 0; h < BN / 64; ++h)
              tc05::tma_load_2d(sb + h * (64 * BK * 2), &tmB, &ctl->full[s], n0 + 64 * h, k0);
          } else {
            tc05::tma_load_2d(sb, &tmB, &ctl->full[s], k0, n0);
          }
          }
          if (++s == S) { s = 0; ph ^= 1u; }
        }
      }
    }
    geeps_pdl_trigger();       // every operand is on its way: the rest of this CTA is its last products and stores
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      const bool leader = tc05::elect_one();
      const uint32_t idesc = tc05::make_idesc_bf16(BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      uint32_t tile_i = 0, ph = 0;
      int s = 0;
      bool ok = true;
      for (int t = t_first; t < num_tiles && ok; t += t_step, ++tile_i) {
        const int z = t / tiles_mn;
        const int kt_begin = z * kt_per, kt_end = min(d.kt_total, kt_begin + kt_per);
        const uint32_t acc = tile_i & 1u, acc_ph = (tile_i >> 1) & 1u;
        // the epilogue must have drained this accumulator (two tiles ago)
        if (!tc05::mbar_wait_warp(&ctl->tmem_empty[acc], acc_ph ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
        tc05::fence_after_sync();
        const uint32_t tacc = tmem + acc * (uint32_t)acc_stride;
        for (int kt = kt_begin; kt < kt_end; ++kt) {
          if (!tc05::mbar_wait_warp(&ctl->full[s], ph, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          tc05::fence_after_sync();
          const uint32_t sa = tiles_u + (uint32_t)(s * STAGE_BYTES), sb = sa + A_STAGE_BYTES;
          // descriptors as 32-bit halves: moving the start is an add.
          // K-major: 16 k-elements = 32 bytes inside the 128-byte swizzle row (2 units of 16 bytes);
          // MN-major: 16 k-rows of 128 bytes = two 8-row groups of 1024 bytes (128 units).
          const uint32_t a_lo = tc05::desc_lo(sa, A_MN ? 64 * BK * 2 : 16), b_lo = tc05::desc_lo(sb, B_MN ? 64 * BK * 2 : 16);
          tc05::mma_ktile_warp<A_MN ? 128 : 2, B_MN ? 128 : 2>(tacc, a_lo, b_lo, tc05::desc_hi(1024), idesc,
                                                               kt > kt_begin ? 1u : 0u, empty_u + 8u * (uint32_t)s);
          if (++s == S) { s = 0; ph ^= 1u; }
        }
        if (ok && leader) tc05::mma_commit(&ctl->tmem_full[acc]);
      }
    }
  } else {
    // ---------------- epilogue: TMEM -> registers -> global ----------------
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    constexpr int G = epi_groups(CL);
    const int grp = (warp - 2) >> 2;
    uint32_t tile_i = 0, slab_i = 0;
    for (int t = t_first; t < num_tiles; t += t_step, ++tile_i) {
      const int mn = t % tiles_mn, z = t / tiles_mn;
      const int m0 = (mn % d.m_tiles) * BM, n0 = (mn / d.m_tiles) * BN;
      const int kt_begin = z * kt_per, kt_end = min(d.kt_total, kt_begin + kt_per);
      const uint32_t acc = tile_i & 1u, acc_ph = (tile_i >> 1) & 1u;
      if (!tc05::mbar_wait(&ctl->tmem_full[acc], acc_ph, abort_flag, WAIT_BUDGET_NS)) break;
      tc05::fence_after_sync();
      const uint32_t tacc = tmem + acc * (uint32_t)acc_stride + ((uint32_t)(q * 32) << 16);
      const long long row = (long long)m0 + q * 32 + lane;
      const float bias_m = (d.bias_mode == 2 && row < d.M) ? d.bias[row] : 0.f;
      const bool add_bias = (d.split_k == 1) || (z == 0);
      const bool has_k = kt_end > kt_begin;
      if (CL) {
        // the commit behind tmem_full covers every MMA of the slice: the operand stages are free to hold the partial tile
        const int r = q * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t v[32];
          tc05::tmem_ld_32x32(tacc + (uint32_t)c, v);
          tc05::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(tiles + part_off(r, (c >> 2) + j, BN)) =
                make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
      } else if (d.tma_store) {
        // 128-byte-wide slabs (64 bf16 or 32 fp32 columns) go through swizzled smem and leave with one
        // TMA store (or reduce-add for split-K) each: coalesced, asynchronous, clipped at the matrix edge
        const int cols_per_slab = d.out_fp32 ? 32 : 64;
        const bool issuer = threadIdx.x == 64 + 128 * grp;
        const int rloc = q * 32 + lane;          // row inside the tile = TMEM lane
        const uint32_t row_off = (uint32_t)rloc * 128u, rsw = (uint32_t)(rloc & 7);
        // everything that does not depend on the column is hoisted out of the slab loop
        const int bmode = add_bias ? d.bias_mode : 0;
        const float alpha = has_k ? d.alpha : 0.f;
        const float bias_row = bmode == 2 ? bias_m : 0.f;
        const bool relu = d.relu != 0;
        const int n_lim = (int)d.N;
#pragma unroll 1
        for (int c = grp * cols_per_slab; c < BN; c += G * cols_per_slab) {
          if ((long long)n0 + c >= d.N) break;
          uint8_t* slab = cslab + (size_t)(2 * grp + (slab_i & 1u)) * C_SLAB_BYTES;
          if (issuer) tc05::bulk_wait_read<1>();   // the slab this group stored two slabs ago has been read out
          tc05::named_bar_sync(1 + grp, 128);
          for (int h = 0; h < cols_per_slab; h += 32) {
            uint32_t r[32];
            tc05::tmem_ld_32x32(tacc + (uint32_t)(c + h), r);
            tc05::tmem_ld_wait();
            const int col0 = n0 + c + h;
            float v[32];
            if (bmode == 1) {
              // per-column bias: the same 32 values for every row of the slab (broadcast loads)
              if (col0 + 32 <= n_lim) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = fmaf(alpha, __uint_as_float(r[j]), __ldg(d.bias + col0 + j));
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  v[j] = fmaf(alpha, __uint_as_float(r[j]), col0 + j < n_lim ? __ldg(d.bias + col0 + j) : 0.f);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = fmaf(alpha, __uint_as_float(r[j]), bias_row);
            }
            if (relu) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
            }
            if (d.out_fp32) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {   // 8 chunks of 4 floats
                const uint32_t off = row_off + (uint32_t)((j ^ rsw) << 4);
                *reinterpret_cast<float4*>(slab + off) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j) {   // 4 chunks of 8 bf16 per 32 columns
                const uint32_t off = row_off + (uint32_t)((((h >> 3) + j) ^ rsw) << 4);
                *reinterpret_cast<uint4*>(slab + off) =
                    make_uint4(pack_bf16x2(v[8 * j], v[8 * j + 1]), pack_bf16x2(v[8 * j + 2], v[8 * j + 3]),
                               pack_bf16x2(v[8 * j + 4], v[8 * j + 5]), pack_bf16x2(v[8 * j + 6], v[8 * j + 7]));
              }
            }
          }
          tc05::fence_proxy_async_smem();
          tc05::named_bar_sync(1 + grp, 128);
          if (issuer) {
            if (d.split_k > 1) tc05::tma_reduce_add_2d(&tmC, slab, n0 + c, m0);
            else tc05::tma_store_2d(&tmC, slab, n0 + c, m0);
            tc05::bulk_commit();
          }
          ++slab_i;
        }
      } else {
  #pragma unroll 1
        for (int c = grp * 32; c < BN; c += G * 32) {
          uint32_t r[32];
          tc05::tmem_ld_32x32(tacc + (uint32_t)c, r);
          tc05::tmem_ld_wait();
          const long long col0 = (long long)n0 + c;
          if (row < d.M && col0 < d.N && has_k) {
            const int ncols = (int)min((long long)32, d.N - col0);
            float v[32];
  #pragma unroll
            for (int j = 0; j < 32; ++j) {
              float x = d.alpha * __uint_as_float(r[j]);
              if (add_bias) {
                if (d.bias_mode == 1 && j < ncols) x += d.bias[col0 + j];
                else if (d.bias_mode == 2) x += bias_m;
              }
              v[j] = x;
            }
            if (d.split_k > 1) {
              float* out = (float*)d.C + row * d.ldc + col0;
              for (int j = 0; j < ncols; ++j) atomicAdd(out + j, v[j]);
            } else if (d.out_fp32) {
              float* out = (float*)d.C + row * d.ldc + col0;
              const bool vec = (ncols == 32) && ((((uintptr_t)out) & 15) == 0);
              if (vec) {
  #pragma unroll
                for (int j = 0; j < 32; j += 4) {
                  float4 o = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                  if (d.beta != 0.f) {
                    float4 old = ld_f4(out + j);
                    o.x += d.beta * old.x; o.y += d.beta * old.y; o.z += d.beta * old.z; o.w += d.beta * old.w;
                  }
                  if (d.relu) { o.x = fmaxf(o.x, 0.f); o.y = fmaxf(o.y, 0.f); o.z = fmaxf(o.z, 0.f); o.w = fmaxf(o.w, 0.f); }
                  st_f4(out + j, o);
                }
              } else {
                for (int j = 0; j < ncols; ++j) {
                  float o = v[j];
                  if (d.beta != 0.f) o += d.beta * out[j];
                  if (d.relu) o = fmaxf(o, 0.f);
                  out[j] = o;
                }
              }
            } else {
              __nv_bfloat16* out = (__nv_bfloat16*)d.C + row * d.ldc + col0;
              const bool vec = (ncols == 32) && ((((uintptr_t)out) & 15) == 0);
              if (vec) {
  #pragma unroll
                for (int j = 0; j < 32; j += 8) {
                  float o[8];
  #pragma unroll
                  for (int e = 0; e < 8; ++e) o[e] = v[j + e];
                  if (d.beta != 0.f) {
                    uint4 oldv = *reinterpret_cast<const uint4*>(out + j);
                    const __nv_bfloat16* ob = reinterpret_cast<const __nv_bfloat16*>(&oldv);
  #pragma unroll
                    for (int e = 0; e < 8; ++e) o[e] += d.beta * __bfloat162float(ob[e]);
                  }
                  if (d.relu) {
  #pragma unroll
                    for (int e = 0; e < 8; ++e) o[e] = fmaxf(o[e], 0.f);
                  }
                  uint4 pk = make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]),
                                        pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
                  *reinterpret_cast<uint4*>(out + j) = pk;
                }
              } else {
                for (int j = 0; j < ncols; ++j) {
                  float o = v[j];
                  if (d.beta != 0.f) o += d.beta * __bfloat162float(out[j]);
                  if (d.relu) o = fmaxf(o, 0.f);
                  out[j] = __float2bfloat16(o);
                }
              }
            }
          }
        }
      }
      // this warp is done reading the accumulator: hand it back to the MMA warp
      tc05::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&ctl->tmem_empty[acc]);
    }
  }

  if (CL) {
    __syncwarp();
    cluster_sync_all();
    // this CTA finishes 128 / cluster rows of the tile, eight columns per thread and step
    const int rank = (int)(blockIdx.x % d.cluster), mn = (int)(blockIdx.x / d.cluster);
    const int m0 = (mn % d.m_tiles) * BM, n0 = (mn / d.m_tiles) * BN;
    const int rows = BM / d.cluster, oct = BN >> 3;
    const uint32_t part = tc05::smem_u32(tiles);
    // a CTA that gave up left no partial tile: nobody stores (the status word names it), as without a cluster
    const uint32_t gave_up = ld_cluster_u32(cluster_addr(tc05::smem_u32(&ctl->abort_flag), lane % d.cluster));
    const int todo = __any_sync(0xffffffffu, gave_up != 0u) ? 0 : rows * oct;
    for (int i = threadIdx.x; i < todo; i += blockDim.x) {
      const int rr = i / oct, o = i - rr * oct;
      const int r = rank * rows + rr;
      const long long row = (long long)m0 + r, col0 = (long long)n0 + o * 8;
      if (row >= d.M || col0 >= d.N) continue;
      const uint32_t o0 = part_off(r, 2 * o, BN), o1 = part_off(r, 2 * o + 1, BN);
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = 0.f;
      for (int z = 0; z < d.cluster; ++z) {
        const uint32_t base = cluster_addr(part, z);
        const float4 a = ld_cluster_f4(base + o0), b = ld_cluster_f4(base + o1);
        v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
        v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
      }
      const int nc = (int)min((long long)8, d.N - col0);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        float x = d.alpha * v[e];
        if (d.bias_mode == 1 && e < nc) x += __ldg(d.bias + col0 + e);
        else if (d.bias_mode == 2) x += __ldg(d.bias + row);
        v[e] = d.relu ? fmaxf(x, 0.f) : x;
      }
      if (d.out_fp32) {
        float* out = (float*)d.C + row * d.ldc + col0;
        if (nc == 8 && (((uintptr_t)out) & 15) == 0) {
          st_f4(out, make_float4(v[0], v[1], v[2], v[3]));
          st_f4(out + 4, make_float4(v[4], v[5], v[6], v[7]));
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) if (e < nc) out[e] = v[e];
        }
      } else {
        __nv_bfloat16* out = (__nv_bfloat16*)d.C + row * d.ldc + col0;
        if (nc == 8 && (((uintptr_t)out) & 15) == 0) {
          *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                                                      pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) if (e < nc) out[e] = __float2bfloat16(v[e]);
        }
      }
    }
    __syncwarp();
    cluster_sync_all();      // nobody leaves while a peer still reads its partial tile
  }
  if (!CL && d.tma_store && (threadIdx.x == 64 || threadIdx.x == 192)) tc05::bulk_wait<0>();   // all TMA stores of this CTA have landed
  tc05::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && ctl->abort_flag)
    geeps_report(d.status, GEEPS_ERR_TIMEOUT, KID_GEMM_TC, (int)blockIdx.x, 0);
  if (warp == 1) {
    tc05::fence_after_sync();
    tc05::tmem_dealloc(tmem, (uint32_t)d.tmem_cols);
  }
}

// ---------------- host side ----------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}

// 2-D bf16 tensor map: `inner` contiguous elements per line, `outer` lines of `ld` elements.
bool make_map(CUtensorMap* map, const void* base, long long inner, long long outer, long long ld,
              int box_inner, int box_outer, bool fp32 = false) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  cuuint64_t strides[1] = {(cuuint64_t)ld * (fp32 ? 4 : 2)};
  cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <bool A_MN, bool B_MN, bool CL>
int launch_kernel(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmDev& d, int grid,
                  cudaStream_t st) {
  const int stage_bytes = A_STAGE_BYTES + d.bn * BK * 2;
  const size_t smem = (size_t)d.stages * stage_bytes + (CL ? 0 : d.slabs * C_SLAB_BYTES) + sizeof(SmemCtl) + 1024;
  static bool attr_set = false;  // per instantiation
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<A_MN, B_MN, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         227 * 1024);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  if (!CL) {
    geeps_launch(gemm_tc_kernel<A_MN, B_MN, CL>, grid, gemm_threads(CL), smem, st, ta, tb, tc, d);
    return (int)cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(gemm_threads(CL));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)d.cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return (int)cudaLaunchKernelEx(&cfg, gemm_tc_kernel<A_MN, B_MN, CL>, ta, tb, tc, d);
}
template <bool A_MN, bool B_MN>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmDev& d, int grid,
           cudaStream_t st) {
  return d.cluster > 1 ? launch_kernel<A_MN, B_MN, true>(ta, tb, tc, d, grid, st)
                       : launch_kernel<A_MN, B_MN, false>(ta, tb, tc, d, grid, st);
}

int round_up(long long v, int m) { return (int)((v + m - 1) / m * m); }

// Tile width and K slices (cluster size) for an output that 256-wide tiles would not spread over every SM: the choice with
// the least operand traffic on the busiest SM, rounds x k tiles per CTA x (A rows + B rows) x 128 bytes, plus kTileOver per
// round (fill, drain) and, for a cluster, the exchange of its partial tile.  Narrow tiles spread an output but re-read A
// once per tile; a cluster keeps the tile wide and cuts K instead.  The traffic is not the bound (the issue of the MMAs
// alone took 256 x 4096, K = 9216 from 38.9 to 32.8 us, L2 flushed), but it ranks the widths as they are now (64, 128, 192, 256; us
// in a captured chain): 256 x 4096, K = 9216 27.0, 35.2, 48.9, 64.4; 256 x 9216, K = 4096 29.5, 20.1, 25.4, 30.0; 256 x 4096,
// K = 4096 13.9, 13.7, 17.5, 22.6; 256 x 1000, K = 4096 13.3, 13.5, 17.5, 22.5; 100 x 512, K = 2048 7.9, 8.4, 10.6, 13.0.
// Clusters: see plan_gemm.
struct TileChoice { int bn, cluster; };
TileChoice choose_tiles(const GeepsGemmParams* p, int unit, int kt, int sms, bool cluster_ok) {
  constexpr double kTileOver = 150e3, kClusterOver = 150e3;
  const long long m_tiles = (p->M + BM - 1) / BM;
  const double a_rows = p->M < BM ? (double)p->M : (double)BM;
  TileChoice best = {unit > 64 ? unit : 64, 1};
  double best_cost = 1e300;
  for (int bn = 64; bn <= 256; bn += unit) {
    const long long tiles = m_tiles * ((p->N + bn - 1) / bn);
    for (int cs = 1; cs <= (cluster_ok ? 8 : 1); cs *= 2) {
      const int per = (kt + cs - 1) / cs;
      if (cs > 1 && (per < 4 || (long long)(cs - 1) * per >= kt)) continue;    // every slice needs k tiles
      // SMs that whole clusters find in GPCs of different sizes: 33 clusters of four and 15 of eight are resident on 148 SMs
      const long long slots = cs <= 2 ? sms : cs == 4 ? sms * 9 / 10 / 4 * 4 : sms * 5 / 6 / 8 * 8;
      const long long rounds = (tiles * cs + slots - 1) / slots;
      // a k step of a slice has its price even for a few rows (4 x 1024, K = 21841: 21.5 us on 64 x 4, 16 on 128 x 8)
      double cost = rounds * (per * ((cs > 1 && a_rows < 32 ? 32.0 : a_rows) + bn) * 128.0 + kTileOver);
      if (cs > 1) cost += rounds * (kClusterOver + a_rows * bn * 8.0);
      if (cost < best_cost * 0.98) { best_cost = cost; best = {bn, cs}; }
    }
  }
  return best;
}

// TMA-store epilogue: C 16-byte aligned with a 16-byte-multiple pitch, no read-modify-write of C
bool tma_c_ok(const GeepsGemmParams* p) {
  return (((uintptr_t)p->C & 15) == 0) && ((p->ldc * (p->out_fp32 ? 4 : 2)) % 16 == 0) && p->beta == 0.f;
}

// How a product is cut: tile width, K slices, and whether the slices of a tile share a cluster.
struct GemmPlan { int bn, split_k, cluster; };
// Calls that may cut K into slices which meet in fp32 atomics (split_k 0, plain fp32 output).
bool auto_split(const GeepsGemmParams* p, int kt) { return p->split_k == 0 && p->out_fp32 && !p->relu && kt >= 8; }
GemmPlan plan_gemm(const GeepsGemmParams* p, int sms) {
  const long long m_tiles = (p->M + BM - 1) / BM;
  const int unit = p->b_mn_major ? 64 : 32;
  const int kt = (int)((p->K + BK - 1) / BK);
  const bool tma_c = tma_c_ok(p);
  GemmPlan g = {p->block_n, 1, 1};
  if (g.bn <= 0 || g.bn > 256 || g.bn % unit) {
    // as few N tiles as possible with little padding ...
    const long long nt = (p->N + 255) / 256;
    g.bn = round_up((p->N + nt - 1) / nt, unit);
    // ... but enough tiles to occupy every SM when the problem allows it
    auto tiles = [&] { return m_tiles * ((p->N + g.bn - 1) / g.bn); };
    if (auto_split(p, kt)) {
      // A long K is split below and keeps its wide tiles.  A short one (K < 1024) is spread by narrow tiles first: every
      // K slice costs a clearing pass and a read-modify-write of the output, so the cost of choose_tiles, which knows
      // only operand bytes, does not hold here (1000 x 4096, K = 512: two slices 20.2 us, narrow tiles 10.9 us;
      // 439 x 4162, K = 632: 15.0 and 10.9 us).
      while (kt < 16 && g.bn > 64 && tiles() < sms) {
        const int narrow = round_up(g.bn / 2, unit);
        if (narrow >= g.bn) break;
        g.bn = narrow;
      }
    } else if (tiles() < sms && p->N > 64) {
      // a bf16 slab is 64 columns wide (see below): several tiles have widths that are multiples of it
      const int step = tma_c && !p->out_fp32 ? 64 : unit;
      // Clusters only for K above 8128 over at most sms / 8 narrow tiles: the data gradient of a wide classifier, 32 x 1024,
      // K = 21841, 16 tiles (tile width x cluster, us in a captured chain): 70 without a cluster, 27.3 on 64 x 8 (16 clusters,
      // of which 15 are resident at once: picked before the cost knew), 22.1 on 64 x 4, 17.0 on 128 x 8, which the cost picks;
      // K = 12000 19.5 on 64 x 8, 12.5, K = 8200 16.7, 11.0.  The line is drawn by the order of the
      // sums, not by speed: a cluster adds its K slices in another order than one running sum, and in a deep network with
      // near-ties in its pooling windows that changes which element a later step's maximum picks, so ordinary layers
      // keep one sum.  What that leaves: 256 x 4096, K = 9216: 27.0 on 64 x 1, 25.1 on 128 x 2; 32 rows: 25.6 on 64 x 1, 13.9
      // on 128 x 4; 256 x 1000, K = 4096: 13.3 on 64 x 1, 9.4 on 64 x 4.
      const bool cluster_ok = p->split_k <= 1 && p->beta == 0.f && kt >= 128 &&
                              m_tiles * ((p->N + 63) / 64) <= sms / 8;
      const TileChoice c = choose_tiles(p, step, kt, sms, cluster_ok);
      if (c.cluster > 1 || c.bn < g.bn) { g.bn = c.bn; g.cluster = c.cluster; }
    }
  }
  if (g.bn > 256) g.bn = 256;
  // a bf16 slab is 64 columns wide: with several N tiles the tile width must be a multiple of it
  if (tma_c && !p->out_fp32 && (g.bn % 64) && (p->N + g.bn - 1) / g.bn > 1) g.bn = round_up(g.bn, 64);
  if (g.cluster > 1) { g.split_k = g.cluster; return g; }
  int split = p->split_k;
  if (split == 0) {  // auto: occupy the SMs about twice over when the output has few tiles
    split = 1;
    const long long tiles = m_tiles * ((p->N + g.bn - 1) / g.bn);
    if (auto_split(p, kt) && tiles < sms) {
      const long long want = (2 * sms) / tiles;   // at most two full waves: one work item more would add a third round
      const long long cap = kt / 4;
      split = (int)(want < cap ? want : cap);
    }
  }
  g.split_k = split < 1 ? 1 : (split > kt ? kt : split);
  if (g.split_k > 1) {
    // every k-slice must be non-empty, otherwise its tile would never be completed by an MMA commit
    const int per = (kt + g.split_k - 1) / g.split_k;
    g.split_k = (kt + per - 1) / per;
  }
  return g;
}
// large K-major products go to CTA pairs (half the B traffic per SM) when 256-row tiles can fill the machine
bool takes_pairs(const GeepsGemmParams* p, int sms) {
  return p->block_n == 0 && p->split_k <= 1 && geeps_gemm_pair_supported(p) &&
         ((p->M + 255) / 256) * ((p->N + 255) / 256) >= sms / 2;
}

}  // namespace

extern "C" {

int geeps_gemm_tc_supported(const GeepsGemmParams* p) {
  if (p->M <= 0 || p->N <= 0 || p->K <= 0) return 0;
  if (((uintptr_t)p->A & 15) || ((uintptr_t)p->B & 15)) return 0;
  if ((p->lda & 7) || (p->ldb & 7)) return 0;
  if (p->split_k > 1 && (!p->out_fp32 || p->relu)) return 0;
  if (p->M > 0x7fffffffLL || p->N > 0x7fffffffLL || p->K > 0x7fffffffLL) return 0;
  return 1;
}

int geeps_gemm_plan(const GeepsGemmParams* p, GeepsGemmPlan* out) {
  if (!geeps_gemm_tc_supported(p)) return 0;
  const int sms = geeps_sm_count();
  const GemmPlan g = plan_gemm(p, sms);
  out->pair = takes_pairs(p, sms) ? 1 : 0;
  out->block_n = g.bn;
  out->split_k = g.split_k;
  out->cluster = g.cluster;
  out->tiles = (p->M + BM - 1) / BM * ((p->N + g.bn - 1) / g.bn);
  return 1;
}

int geeps_gemm_bf16(const GeepsGemmParams* p, void* stream) {
  if (!geeps_gemm_tc_supported(p)) return (int)cudaErrorInvalidValue;
  const int kSMs = geeps_sm_count();
  if (takes_pairs(p, kSMs)) return geeps_gemm_bf16_pair(p, stream);
  const GemmPlan plan = plan_gemm(p, kSMs);
  const int bn = plan.bn, cluster = plan.cluster;
  const int m_tiles = (int)((p->M + BM - 1) / BM);
  const int kt_total = (int)((p->K + BK - 1) / BK);
  const bool tma_c = tma_c_ok(p);
  const long long n_tiles = (p->N + bn - 1) / bn;
  CUtensorMap ta, tb;
  bool ok = p->a_mn_major ? make_map(&ta, p->A, p->M, p->K, p->lda, 64, BK)
                          : make_map(&ta, p->A, p->K, p->M, p->lda, BK, BM);
  ok = ok && (p->b_mn_major ? make_map(&tb, p->B, p->N, p->K, p->ldb, 64, BK)
                            : make_map(&tb, p->B, p->K, p->N, p->ldb, BK, bn));
  if (!ok) return (int)cudaErrorInvalidValue;
  GemmDev d;
  d.C = p->C; d.bias = p->bias; d.status = p->status;
  d.M = p->M; d.N = p->N; d.K = p->K; d.ldc = p->ldc;
  d.alpha = p->alpha; d.beta = p->beta;
  d.out_fp32 = p->out_fp32; d.bias_mode = p->bias ? p->bias_mode : 0; d.relu = p->relu;
  d.kt_total = kt_total;
  d.bn = bn;
  d.m_tiles = m_tiles;
  d.n_tiles = (int)n_tiles;
  int tmem_cols = 32;
  while (tmem_cols < 2 * bn) tmem_cols <<= 1;
  d.tmem_cols = tmem_cols;
  d.split_k = plan.split_k;
  d.cluster = cluster;
  if (d.split_k > 1 && cluster == 1) {
    // partial sums are accumulated with atomics: bring C to beta*C (or zero) first
    int e = geeps_scale_matrix_f32((float*)p->C, p->M, p->N, p->ldc, p->beta, stream);
    if (e) return e;
    d.beta = 0.f;
  }
  d.tma_store = tma_c && cluster == 1 ? 1 : 0;
  CUtensorMap tc;
  if (d.tma_store) {
    if (!make_map(&tc, p->C, p->N, p->M, p->ldc, p->out_fp32 ? 32 : 64, BM, p->out_fp32 != 0)) d.tma_store = 0;
  }
  if (!d.tma_store) tc = ta;   // unused by the kernel
  const int stage_bytes = A_STAGE_BYTES + bn * BK * 2;
  d.slabs = bn > (p->out_fp32 ? 32 : 64) ? 4 : 2;
  d.stages = (cluster > 1 ? 200 * 1024 : 224 * 1024 - d.slabs * C_SLAB_BYTES) / stage_bytes;
  if (d.stages > MAX_STAGES) d.stages = MAX_STAGES;
  if (d.stages < 2) d.stages = 2;
  const long long num_tiles = (long long)m_tiles * n_tiles * d.split_k;
  const int grid = (int)(num_tiles < kSMs || cluster > 1 ? num_tiles : kSMs);
  cudaStream_t st = (cudaStream_t)stream;
  if (!p->a_mn_major && !p->b_mn_major) return launch<false, false>(ta, tb, tc, d, grid, st);
  if (p->a_mn_major && !p->b_mn_major) return launch<true, false>(ta, tb, tc, d, grid, st);
  if (!p->a_mn_major && p->b_mn_major) return launch<false, true>(ta, tb, tc, d, grid, st);
  return launch<true, true>(ta, tb, tc, d, grid, st);
}

}  // extern "C"
