// Implicit-GEMM convolution (stride 1) on the 5th-generation tensor cores: no patch matrix is ever
// written.  The activation operand of every k-tile is fetched straight from the NHWC tensor by one tiled
// 4-D TMA load whose (w, h) start is shifted by the filter tap; pixels that fall into the padding are
// outside the tensor's extent and arrive as zeros.  Three products share one persistent kernel:
//
//   forward        Y[pix, co]  = sum_{tap, ci} X[pix + tap, ci] * W[co, tap, ci]   (+ bias, ReLU)
//   data gradient  dX[pix, ci] = sum_{tap, co} dY[pix - tap, co] * W[co, tap, ci]
//   weight grad.   dW[co, tap, ci] = sum_{pix} dY[pix, co] * X[pix + tap, ci]      (fp32, split over pixels)
//
// The 128 accumulator rows of a tile are a box of bw x bh x bn output pixels (chosen per layer so that the
// box wastes few rows), so the same box shape serves the 4-D load and the 4-D store of the result, and
// ragged edges are clipped by TMA.  The weight matrix [co][tap][ci] is a 3-D tensor for TMA, so channel
// counts that are not multiples of 64 (48-channel groups) are zero-filled instead of reading the next tap.
// For the weight gradient the reduction runs over pixel boxes of 64, both operands are MN-major panels of
// [64 pixels x 64 channels], and one tile's N covers up to four (tap, channel-chunk) panels.
//
// Roles, pipeline, TMEM double buffering, bounded waits and the swizzled-slab TMA-store epilogue are those
// of the plain GEMM in gemm_tc.cu.
//
// The reference has no convolution of its own (its layers lived in a Caffe fork that is not in its tree);
// this replaces the im2col + GEMM + col2im formulation for stride-1 layers.
#include <cuda.h>
#include <mutex>
#include <stdio.h>
#include <string.h>

#include "kernels.h"
#include "tc05.cuh"

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;
constexpr int PANEL_BYTES = 64 * BK * 2;     // one MN-major panel: 64 k-rows x 128 bytes
constexpr int MAX_STAGES = 8;
constexpr uint64_t WAIT_BUDGET_NS = 2000000000ull;
constexpr int C_SLAB_BYTES = BM * 128;
constexpr int kGroups = 2;                   // epilogue groups of four warps, which take alternate column slabs
constexpr int kThreads = 64 + 128 * kGroups;

enum { MODE_FWD = 0, MODE_DGRAD = 1, MODE_WGRAD = 2 };

// One parity class of a data gradient (see geeps_conv_tc): pixels (s i + a, s j + b) of dX with the sub-filter of the
// taps that reach them.  A stride-1 layer is one class.
struct DgradDev {
  int t0;                         // first tile of the class
  int wt, ht, m_tiles;            // pixel boxes along W, along H, in all
  int m_units;                    // boxes or, on CTA pairs, pairs of neighbouring boxes
  int KW, kt_total;               // taps per row of the sub-filter; its taps x channel chunks
  int pad_w, pad_h, tap0;         // dY offset of sub-filter tap (0, 0) and its place in the whole filter
};
constexpr int MAX_CLS = 4;        // classes per launch: all of a stride-2 layer

struct ConvDev {
  const float* bias; int* status;
  int taps, KW, pad, cchunks;     // k-tile (fwd, dgrad) or N panel (wgrad) = (tap, 64-channel chunk)
  int bw, bh, bnb, wt, ht;        // pixel box and number of boxes along W and H (batch boxes follow)
  int rows;                       // bw * bh * bnb
  int bn, n_valid;                // tile width; valid output columns (fwd: Og, dgrad: Cg, wgrad: panels * 64)
  int m_tiles, m_units, n_tiles, kt_total, split_k, stages, tmem_cols;
  int groups;                     // epilogue groups that have columns to take
  int slabs;                      // staging slabs: two per epilogue group that has one to fill
  int relu, zero_fill_c;          // wgrad: a channel coordinate outside X, for panels past the last one
  int ch_valid;                   // wgrad: channels per tap (cg)
  int narrow;                     // fwd / dgrad: result leaves in 32-channel (64-byte) slabs, see the host code
  int stride;                     // fwd / wgrad: pixel stride of the layer (the X boxes are loaded with this element stride)
  int n_cls, tap_dw, tap_dh;      // dgrad: weight tap of loop position (kh, kw) = tap0 + kh * tap_dh + kw * tap_dw
  DgradDev cls[MAX_CLS];          // dgrad: tiles are ordered by class
};

struct OutMaps { CUtensorMap m[MAX_CLS]; };     // dgrad: the view of each class; else m[0]

__device__ __forceinline__ int dgrad_class(const ConvDev& d, int t) {
  int c = 0;
  while (c + 1 < d.n_cls && t >= d.cls[c + 1].t0) ++c;
  return c;
}

struct SmemCtl {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

struct Box { int w0, h0, b0; };
__device__ __forceinline__ Box decode_box(const ConvDev& d, int i, int wt, int ht) {
  Box b;
  const int wi = i % wt;
  const int r = i / wt;
  b.w0 = wi * d.bw;
  b.h0 = (r % ht) * d.bh;
  b.b0 = (r / ht) * d.bnb;
  return b;
}

// tmA: activations of the M side (fwd: X, dgrad: dY, wgrad: dY); tmB: fwd/dgrad: W as (ci, tap, co),
// wgrad: X; tmC: fwd: Y, dgrad: dX (4-D bf16), wgrad: dW as (ci, tap, co) fp32.
//
// PAIR (forward and data gradient): the two CTAs of a cluster compute the tiles of two neighbouring pixel boxes with one
// MMA of 256 rows (cta_group::2).  Each loads its own box and half of the weight tile, so an SM takes 28 KB instead of 40
// from L2 for a k-tile of 192 columns, and that (some 64 bytes a clock) is what bounds the main loop.  The even CTA issues
// the products for both; its barriers count the bytes of both.
template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
conv_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ OutMaps tmC, const ConvDev d) {
  constexpr bool A_MN = MODE == MODE_WGRAD;
  constexpr bool B_MN = MODE != MODE_FWD;
  extern __shared__ uint8_t smem_raw[];
  const int BN = d.bn;
  const int BNC = PAIR ? BN / 2 : BN;                   // columns of the weight tile that this CTA loads
  const int B_STAGE_BYTES = BNC * BK * 2;
  const int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* cslab = tiles + (size_t)d.stages * STAGE_BYTES;
  SmemCtl* ctl = (SmemCtl*)(cslab + d.slabs * C_SLAB_BYTES);
  const int rank = PAIR ? (int)tc05::cluster_ctarank() : 0;
  const int unit0 = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, units = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = d.stages;
  const int kt_per = (d.kt_total + d.split_k - 1) / d.split_k;
  const int tiles_mn = d.m_units * d.n_tiles;
  const int num_tiles = tiles_mn * d.split_k;
  const int acc_stride = d.tmem_cols >> 1;

  if (MODE == MODE_WGRAD && d.rows < 64) {
    // a pixel box with fewer than 64 pixels leaves the tail of every panel untouched: it must read as zero
    uint4* z = reinterpret_cast<uint4*>(tiles);
    const int n16 = d.stages * STAGE_BYTES / 16;
    for (int i = threadIdx.x; i < n16; i += blockDim.x) z[i] = make_uint4(0, 0, 0, 0);
    tc05::fence_proxy_async_smem();
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { tc05::mbar_init(&ctl->full[s], 1); tc05::mbar_init(&ctl->empty[s], 1); }
    for (int a = 0; a < 2; ++a) { tc05::mbar_init(&ctl->tmem_full[a], 1); tc05::mbar_init(&ctl->tmem_empty[a], (PAIR ? 2 : 1) * 4 * kGroups); }
    ctl->abort_flag = 0;
    tc05::mbar_fence_init();
  }
  if (warp == 1) {
    if (PAIR) { tc05::tmem_alloc_pair(&ctl->tmem_base, (uint32_t)d.tmem_cols); tc05::tmem_relinquish_pair(); }
    else { tc05::tmem_alloc(&ctl->tmem_base, (uint32_t)d.tmem_cols); tc05::tmem_relinquish(); }
  }
  tc05::fence_before_sync();
  __syncthreads();
  if (PAIR) tc05::cluster_sync();      // the peer's barriers are initialised before anything signals them
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
      // every index below advances incrementally: this one thread's latency is the producer's throughput,
      // and an integer division costs more than the TMA issue itself
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      const uint32_t tx_bytes = MODE == MODE_WGRAD ? (uint32_t)((2 + BN / 64) * d.rows * 128)
                                                   : (uint32_t)((PAIR ? 2 : 1) * (d.rows * 128 + BNC * 128));
      for (int t = unit0; t < num_tiles && ok; t += units) {
        const DgradDev& q = d.cls[MODE == MODE_DGRAD ? dgrad_class(d, t) : 0];
        const int tq = MODE == MODE_DGRAD ? t - q.t0 : t;
        const int mn = MODE == MODE_DGRAD ? tq : tq % tiles_mn, z = MODE == MODE_DGRAD ? 0 : tq / tiles_mn;
        const int mts = MODE == MODE_DGRAD ? q.m_units : d.m_units;
        const int ni = mn / mts, mi = PAIR ? (mn - ni * mts) * 2 + rank : mn - ni * mts;    // a second box past the last is all zeros
        const int kt_begin = z * kt_per, kt_end = MODE == MODE_DGRAD ? q.kt_total : min(d.kt_total, kt_begin + kt_per);
        const int KW = MODE == MODE_DGRAD ? q.KW : d.KW;
        Box mb = {0, 0, 0};
        if (MODE == MODE_FWD) mb = decode_box(d, mi, d.wt, d.ht);
        if (MODE == MODE_DGRAD) {      // of dY: where tap (0, 0) reads
          mb = decode_box(d, mi, q.wt, q.ht);
          mb.w0 += q.pad_w; mb.h0 += q.pad_h;
        }
        // fwd / dgrad: k-tile = (kh, kw, channel chunk), starting at 0 (no split)
        int kh = 0, kw = 0, cc = 0, tap = 0, wtap = MODE == MODE_DGRAD ? q.tap0 : 0;
        // wgrad: k-tile = pixel box; the N panels of this tile are fixed
        Box kb = {0, 0, 0};
        int pc[4] = {0, 0, 0, 0}, pdw[4] = {0, 0, 0, 0}, pdh[4] = {0, 0, 0, 0};
        if (MODE == MODE_WGRAD) {
          kb = decode_box(d, kt_begin, d.wt, d.ht);
          for (int j = 0; j < BN / 64; ++j) {
            const int panel = ni * (BN / 64) + j;
            const bool valid = panel * 64 < d.n_valid;
            const int ptap = valid ? panel / d.cchunks : 0;
            const int pkh = ptap / d.KW;
            pc[j] = valid ? (panel - ptap * d.cchunks) * 64 : d.zero_fill_c;
            pdw[j] = ptap - pkh * d.KW - d.pad;
            pdh[j] = pkh - d.pad;
          }
        }
        for (int kt = kt_begin; kt < kt_end; ++kt) {
          if (!tc05::mbar_wait_warp(&ctl->empty[s], ph ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          uint8_t* sa = tiles + (size_t)s * STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE_BYTES;
          uint64_t* bar = &ctl->full[s];
          if (leader) {
          if (!PAIR || rank == 0) tc05::mbar_expect_tx(bar, tx_bytes);
          if (PAIR) {
            const uint32_t both = tc05::map_to_cta(tc05::smem_u32(bar), 0);
            const int n = ni * BN + rank * BNC;
            if (MODE == MODE_FWD) {
              tc05::tma_load_4d_pair(sa, &tmA, both, cc * 64, mb.w0 * d.stride + kw - d.pad, mb.h0 * d.stride + kh - d.pad, mb.b0);
              tc05::tma_load_3d_pair(sb, &tmB, both, cc * 64, tap, n);
            } else {
              tc05::tma_load_4d_pair(sa, &tmA, both, cc * 64, mb.w0 - kw, mb.h0 - kh, mb.b0);
              for (int h = 0; h < BNC / 64; ++h)
                tc05::tma_load_3d_pair(sb + h * PANEL_BYTES, &tmB, both, n + 64 * h, wtap, cc * 64);
            }
          } else if (MODE == MODE_FWD) {
            tc05::tma_load_4d(sa, &tmA, bar, cc * 64, mb.w0 * d.stride + kw - d.pad, mb.h0 * d.stride + kh - d.pad, mb.b0);
            tc05::tma_load_3d(sb, &tmB, bar, cc * 64, tap, ni * BN);
          } else if (MODE == MODE_DGRAD) {
            tc05::tma_load_4d(sa, &tmA, bar, cc * 64, mb.w0 - kw, mb.h0 - kh, mb.b0);
            for (int h = 0; h < BN / 64; ++h)
              tc05::tma_load_3d(sb + h * PANEL_BYTES, &tmB, bar, ni * BN + 64 * h, wtap, cc * 64);
          } else {
            for (int h = 0; h < 2; ++h)
              tc05::tma_load_4d(sa + h * PANEL_BYTES, &tmA, bar, mi * BM + 64 * h, kb.w0, kb.h0, kb.b0);
            for (int j = 0; j < BN / 64; ++j)
              tc05::tma_load_4d(sb + j * PANEL_BYTES, &tmB, bar, pc[j], kb.w0 * d.stride + pdw[j], kb.h0 * d.stride + pdh[j], kb.b0);
          }
          }
          if (MODE == MODE_WGRAD) {
            kb.w0 += d.bw;
            if (kb.w0 >= d.wt * d.bw) {
              kb.w0 = 0; kb.h0 += d.bh;
              if (kb.h0 >= d.ht * d.bh) { kb.h0 = 0; kb.b0 += d.bnb; }
            }
          } else if (++cc == d.cchunks) {
            cc = 0; ++tap; wtap += d.tap_dw;
            if (++kw == KW) { kw = 0; ++kh; wtap += d.tap_dh - KW * d.tap_dw; }
          }
          if (++s == S) { s = 0; ph ^= 1u; }
        }
      }
    }
    geeps_pdl_trigger();       // every operand is on its way: the rest of this CTA is its last products and stores
  } else if (warp == 1) {
    // ---------------- MMA issuer (of a pair: the even CTA's) ----------------
    if (!PAIR || rank == 0) {
      const bool leader = tc05::elect_one();
      const uint32_t idesc = tc05::make_idesc_bf16(PAIR ? 2 * BM : BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      uint32_t tile_i = 0, ph = 0;
      int s = 0;
      bool ok = true;
      for (int t = unit0; t < num_tiles && ok; t += units, ++tile_i) {
        const int z = MODE == MODE_DGRAD ? 0 : t / tiles_mn;
        const int kt_begin = z * kt_per;
        const int kt_end = MODE == MODE_DGRAD ? d.cls[dgrad_class(d, t)].kt_total : min(d.kt_total, kt_begin + kt_per);
        const uint32_t acc = tile_i & 1u, acc_ph = (tile_i >> 1) & 1u;
        if (!tc05::mbar_wait_warp(&ctl->tmem_empty[acc], acc_ph ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
        tc05::fence_after_sync();
        const uint32_t tacc = tmem + acc * (uint32_t)acc_stride;
        for (int kt = kt_begin; kt < kt_end; ++kt) {
          if (!tc05::mbar_wait_warp(&ctl->full[s], ph, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          tc05::fence_after_sync();
          const uint32_t sa = tiles_u + (uint32_t)(s * STAGE_BYTES), sb = sa + A_STAGE_BYTES;
          const uint32_t a_lo = tc05::desc_lo(sa, A_MN ? PANEL_BYTES : 16), b_lo = tc05::desc_lo(sb, B_MN ? PANEL_BYTES : 16);
          if (PAIR)
            tc05::mma_ktile_warp_pair<A_MN ? 128 : 2, B_MN ? 128 : 2>(tacc, a_lo, b_lo, tc05::desc_hi(1024), idesc,
                                                                      kt > kt_begin ? 1u : 0u, empty_u + 8u * (uint32_t)s);
          else
            tc05::mma_ktile_warp<A_MN ? 128 : 2, B_MN ? 128 : 2>(tacc, a_lo, b_lo, tc05::desc_hi(1024), idesc,
                                                                 kt > kt_begin ? 1u : 0u, empty_u + 8u * (uint32_t)s);
          if (++s == S) { s = 0; ph ^= 1u; }
        }
        if (ok && leader) {
          if (PAIR) tc05::mma_commit_pair(&ctl->tmem_full[acc], 3);
          else tc05::mma_commit(&ctl->tmem_full[acc]);
        }
      }
    }
  } else {
    // ---------------- epilogue: TMEM -> registers -> swizzled slab -> TMA store ----------------
    const int q = warp & 3, grp = (warp - 2) >> 2;
    uint32_t tile_i = 0, slab_i = 0;
    const int cols_per_slab = (MODE == MODE_WGRAD || d.narrow) ? 32 : 64;
    const bool issuer = threadIdx.x == 64 + 128 * grp;
    const int rloc = q * 32 + lane;
    // wide slab: 128-byte rows, 128-byte swizzle (16-byte chunk ^ row % 8); narrow slab: 64-byte rows, 64-byte
    // swizzle (chunk ^ (row / 2) % 4)
    const bool narrow = MODE != MODE_WGRAD && d.narrow;
    const uint32_t row_off = (uint32_t)rloc * (narrow ? 64u : 128u);
    const uint32_t rsw = narrow ? (uint32_t)((rloc >> 1) & 3) : (uint32_t)(rloc & 7);
    const bool relu = d.relu != 0;
    for (int t = unit0; t < num_tiles; t += units, ++tile_i) {
      const int cl = MODE == MODE_DGRAD ? dgrad_class(d, t) : 0;
      const DgradDev& cq = d.cls[cl];
      const int mn = MODE == MODE_DGRAD ? t - cq.t0 : t % tiles_mn;
      const int mts = MODE == MODE_DGRAD ? cq.m_units : d.m_units;
      const int ni = mn / mts, mi = PAIR ? (mn - ni * mts) * 2 + rank : mn - ni * mts;
      const bool there = !PAIR || mi < (MODE == MODE_DGRAD ? cq.m_tiles : d.m_tiles);
      const int n0 = ni * BN;
      const uint32_t acc = tile_i & 1u, acc_ph = (tile_i >> 1) & 1u;
      if (!tc05::mbar_wait(&ctl->tmem_full[acc], acc_ph, abort_flag, WAIT_BUDGET_NS)) break;
      tc05::fence_after_sync();
      const uint32_t tacc = tmem + acc * (uint32_t)acc_stride + ((uint32_t)(q * 32) << 16);
      Box mb = {0, 0, 0};
      if (MODE == MODE_FWD) mb = decode_box(d, mi, d.wt, d.ht);
      if (MODE == MODE_DGRAD) mb = decode_box(d, mi, cq.wt, cq.ht);
#pragma unroll 1
      for (int c = grp < d.groups && there ? grp * cols_per_slab : BN; c < BN; c += d.groups * cols_per_slab) {
        if (n0 + c >= d.n_valid) break;
        uint8_t* slab = cslab + (size_t)(2 * grp + (slab_i & 1u)) * C_SLAB_BYTES;
        if (issuer) tc05::bulk_wait_read<1>();
        tc05::named_bar_sync(1 + grp, 128);
        for (int h = 0; h < cols_per_slab; h += 32) {
          if (n0 + c + h >= d.n_valid) break;      // columns past the tensor's extent are clipped by the store anyway
          uint32_t r[32];
          tc05::tmem_ld_32x32(tacc + (uint32_t)(c + h), r);
          tc05::tmem_ld_wait();
          if (MODE == MODE_WGRAD) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t off = row_off + (uint32_t)((j ^ rsw) << 4);
              *reinterpret_cast<uint4*>(slab + off) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            }
          } else {
            float v[32];
            const int col0 = n0 + c + h;
            if (MODE == MODE_FWD && d.bias != nullptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                v[j] = __uint_as_float(r[j]) + (col0 + j < d.n_valid ? __ldg(d.bias + col0 + j) : 0.f);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            }
            if (relu) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
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
          if (MODE == MODE_WGRAD) {
            const int panel = (n0 + c) >> 6;
            const int tap = panel / d.cchunks, cc = panel - tap * d.cchunks;
            const int x = cc * 64 + (c & 32);
            if (x < d.ch_valid) {       // never start a store past the extent
              if (d.split_k > 1) tc05::tma_reduce_add_3d(&tmC.m[0], slab, x, tap, mi * BM);
              else tc05::tma_store_3d(&tmC.m[0], slab, x, tap, mi * BM);
            }
          } else {
            tc05::tma_store_4d(&tmC.m[cl], slab, n0 + c, mb.w0, mb.h0, mb.b0);
          }
          tc05::bulk_commit();
        }
        ++slab_i;
      }
      tc05::fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) tc05::mbar_arrive_cluster(tc05::map_to_cta(tc05::smem_u32(&ctl->tmem_empty[acc]), 0));
        else tc05::mbar_arrive(&ctl->tmem_empty[acc]);
      }
    }
  }

  if (threadIdx.x == 64 || threadIdx.x == 192) tc05::bulk_wait<0>();
  tc05::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && ctl->abort_flag)
    geeps_report(d.status, GEEPS_ERR_TIMEOUT, KID_CONV_TC, (int)blockIdx.x, 0);
  // neither CTA of a pair may release TMEM or leave while the other can still signal its barriers or use the pair's TMEM
  if (PAIR) tc05::cluster_sync();
  if (warp == 1) {
    tc05::fence_after_sync();
    if (PAIR) tc05::tmem_dealloc_pair(tmem, (uint32_t)d.tmem_cols);
    else tc05::tmem_dealloc(tmem, (uint32_t)d.tmem_cols);
  }
}

// ---------------- host side ----------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
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

// rank-N map (128-byte swizzle unless told otherwise); dims / box innermost first, strides (bytes) for dims 1..rank-1
bool make_map(CUtensorMap* map, const void* base, int rank, const long long* dims, const long long* strides_bytes,
              const int* box, bool fp32, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B,
              const int* elem_strides = nullptr) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t gd[4], gs[3];
  cuuint32_t bx[4], es[4];
  for (int i = 0; i < rank; ++i) {
    gd[i] = (cuuint64_t)dims[i]; bx[i] = (cuuint32_t)box[i];
    es[i] = elem_strides ? (cuuint32_t)elem_strides[i] : 1;
  }
  for (int i = 0; i + 1 < rank; ++i) gs[i] = (cuuint64_t)strides_bytes[i];
  return fn(map, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank,
            const_cast<void*>(base), gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// NHWC activation tensor as (channels, W, H, B) with a pixel pitch of `pitch` channels.  stride > 1: a box of
// bw x bh pixels takes every stride-th pixel (TMA element strides; the box extent is given in traversed elements,
// of which ceil(extent / stride) are loaded).
bool make_act_map(CUtensorMap* map, const void* base, int ch, int W, int H, int B, long long pitch, int bw, int bh,
                  int bnb, bool narrow = false, int stride = 1) {
  const long long dims[4] = {ch, W, H, B};
  const long long st[3] = {pitch * 2, pitch * 2 * W, pitch * 2 * W * H};
  const int box[4] = {narrow ? 32 : 64, bw * stride, bh * stride, bnb};
  const int es[4] = {1, stride, stride, 1};
  return make_map(map, base, 4, dims, st, box, false, narrow ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                  es);
}

// A parity class of an NHWC tensor: pixels (s * i + a, s * j + b) as a dense (channels, W2, H2, B) tensor
bool make_act_view(CUtensorMap* map, const void* base, int ch, int W, int H, int B, long long pitch, int s, int a,
                   int b, int W2, int H2, int bw, int bh, int bnb, bool narrow) {
  const long long dims[4] = {ch, W2, H2, B};
  const long long st[3] = {pitch * 2 * s, pitch * 2 * W * s, pitch * 2 * W * H};
  const int box[4] = {narrow ? 32 : 64, bw, bh, bnb};
  const char* origin = (const char*)base + ((long long)a * W + b) * pitch * 2;
  return make_map(map, origin, 4, dims, st, box, false, narrow ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B);
}

// Pick the pixel box (bw, bh, bnb) with at most `cap` pixels that covers the W x H x B grid with the fewest
// boxes; ties go to the wider box (longer contiguous runs).  A call asks twice (which kernel, how it is cut): the last answer is
// kept for the thread.
void pick_box(int W, int H, int B, int cap, int* bw, int* bh, int* bnb) {
  thread_local int last[7] = {0, 0, 0, 0, 0, 0, 0};
  if (last[0] == W && last[1] == H && last[2] == B && last[3] == cap) { *bw = last[4]; *bh = last[5]; *bnb = last[6]; return; }
  long long best = -1;
  *bw = 1; *bh = 1; *bnb = 1;
  for (int w = 1; w <= W && w <= cap; ++w) {
    for (int h = 1; h <= H && w * h <= cap; ++h) {
      int n = cap / (w * h);
      if (n > B) n = B;
      if (n > 256 || w > 256 || h > 256) continue;
      const long long boxes = (long long)((W + w - 1) / w) * ((H + h - 1) / h) * ((B + n - 1) / n);
      if (best < 0 || boxes < best || (boxes == best && w > *bw)) { best = boxes; *bw = w; *bh = h; *bnb = n; }
    }
  }
  const int now[7] = {W, H, B, cap, *bw, *bh, *bnb};
  memcpy(last, now, sizeof(last));
}

int round_up(long long v, int m) { return (int)((v + m - 1) / m * m); }

// A result tensor whose pixel pitch is not a multiple of 128 bytes and whose channel count ends in a half
// slab (96 channels: 192-byte pixels) stores badly in 128-byte rows - they straddle lines and the last slab is
// clipped (the 96-channel conv1 output took 218 us where 64 / 128 channels took 144 / 182 us).  Such tensors
// leave in 32-channel slabs: 64-byte rows that never straddle a 128-byte line and are never clipped.
int narrow_store(int channels, long long pitch) {
  return (channels % 64 == 32 && (pitch * 2) % 128 != 0) ? 1 : 0;
}

// How a forward or data-gradient product is cut into tiles, and what its two kernels take.
// (the parity classes of a strided data gradient share one box, which the largest class is cut into)
struct BoxPlan {
  int bw, bh, bnb;                // pixel box
  long long m_tiles;              // boxes: of the whole problem, or of the largest class
  int bn, n_tiles, kt;            // tile width, tiles along the channels, k-tiles (whole filter)
  double one, pair;               // us on single CTAs and on pairs; pair < 0: no pairs
};
// Times (us, captured chain) of 364 forward and 364 data-gradient products with 7 x 7 to 56 x 56 pixels, 32 to 384 channels,
// 3 x 3 and 5 x 5 taps, as launch + waves * (tile + k-tiles * (k-tile + width * per column)); half of the fits lie within
// 13 % of the measurement.  Rows of activations or weights that do not begin on 128-byte lines cost a k-tile more, above all
// where one CTA loads the whole weight tile.  us, single CTAs / pairs: 34 x 23 x 23, 248 -> 256, data gradient 44.3 / 29.0; 9 x 38 x 38, 376 ->
// 256 39.4 / 27.7; 62 x 34 x 34, 216 -> 144, 5 x 5 236 / 172.  Sixty drawn layers that the rule sends to pairs: off the lines 0.84 of the
// time on single CTAs (0.65 to 1.04), on them 0.985 (0.83 to 1.04), nearly all 5 x 5; AlexNet's conv3 - conv5 and the Inception layers
// stay on single CTAs.
struct KernelCost { double launch, tile, tile_col, kt, kt_col, kt_mis, kt_mis_col; };
constexpr KernelCost kFwdOne = {4.09, 1.52, 0.146, 0.143, 0.028, 0., 0.062}, kFwdPair = {4.98, 1.19, 0.326, 0.152, 0.021, 0.012, 0.028},
                     kDgradOne = {3.47, 1.73, 0., 0.182, 0.033, 0., 0.044}, kDgradPair = {5.22, 0., 0.603, 0.208, 0.019, 0.023, 0.008};
double tiles_us(const KernelCost& c, long long waves, int kt, int bn, bool mis) {
  const double cols = bn / 64.0;
  return c.launch + waves * (c.tile + cols * c.tile_col + kt * (c.kt + cols * c.kt_col + (mis ? c.kt_mis + cols * c.kt_mis_col : 0.)));
}

// s, n_cls: stride and classes of this launch of a strided data gradient
BoxPlan plan_box(const GeepsConvTcParams* p, int s, int n_cls, int sms) {
  const bool fwd = p->mode == MODE_FWD;
  BoxPlan b;
  // rows of the tile: pixels of the output (fwd) or of the input gradient (dgrad)
  const int GW = fwd ? p->OW : (p->W + s - 1) / s, GH = fwd ? p->OH : (p->H + s - 1) / s;
  pick_box(GW, GH, p->B, BM, &b.bw, &b.bh, &b.bnb);
  b.m_tiles = (long long)((GW + b.bw - 1) / b.bw) * ((GH + b.bh - 1) / b.bh) * ((p->B + b.bnb - 1) / b.bnb);
  const int kch = fwd ? p->cg : p->og, nch = fwd ? p->og : p->cg;          // reduced and produced channels
  b.kt = p->KH * p->KW * ((kch + 63) / 64);
  const int nt = (nch + 255) / 256;
  b.bn = round_up((nch + nt - 1) / nt, (fwd && nt == 1) ? 32 : 64);
  if (b.bn > 256) b.bn = 256;
  // too few tiles for the machine: narrower ones, while the operand rows (the bound here) of the busiest SM go down:
  // 32 x 14 x 14 pixels, 160 channels: 3 x 3 forward 14.7 -> 12.2 us (160 in), 11.5 -> 9.7 us (128 in)
  const long long all = b.m_tiles * n_cls;
  if (all * ((nch + b.bn - 1) / b.bn) < sms) {
    auto cost = [&](int w) { return (all * ((nch + w - 1) / w) + sms - 1) / sms * (BM + w); };
    for (int w = 64, top = b.bn; w < top; w += 64)
      if (cost(w) < cost(b.bn)) b.bn = w;
  }
  b.n_tiles = (nch + b.bn - 1) / b.bn;
  const void* act = fwd ? p->x : p->y;
  const bool mis = ((fwd ? p->x_pitch : p->y_pitch) % 64) != 0 || p->cg % 64 != 0 || ((uintptr_t)act & 127) != 0;
  b.one = tiles_us(fwd ? kFwdOne : kDgradOne, (b.m_tiles * b.n_tiles + sms - 1) / sms, b.kt, b.bn, mis);
  // Not below the channels that the fits know.  Pairs need whole 64-column panels of a transposed weight tile in each half.  Where the lines are aligned and the
  // k-tiles few the epilogue is the bound (32 x 56 x 56, 64 -> 192: 23.4 us on single CTAs, 26.8 on pairs).
  b.pair = -1;
  if (p->stride <= 1 && s == 1 && b.bn % (fwd ? 32 : 128) == 0 && (mis || b.kt >= 18) && kch >= 32 && nch >= 32)
    b.pair = tiles_us(fwd ? kFwdPair : kDgradPair, ((b.m_tiles + 1) / 2 * b.n_tiles + sms / 2 - 1) / (sms / 2), b.kt, b.bn, mis);
  return b;
}
// How a weight gradient is cut.  us: as tiles_us, fitted to 1300 products of both kernels (here half of them within 9 %).
struct WgradPlan { int bw, bh, bnb, kt, m_tiles, per, n_tiles, split; double us; };      // per: panels (tap, chunk) per tile
WgradPlan plan_wgrad_box(const GeepsConvTcParams* p, int sms) {
  WgradPlan g;
  // reduction over output pixels in boxes of up to 64
  pick_box(p->OW, p->OH, p->B, 64, &g.bw, &g.bh, &g.bnb);
  g.kt = ((p->OW + g.bw - 1) / g.bw) * ((p->OH + g.bh - 1) / g.bh) * ((p->B + g.bnb - 1) / g.bnb);
  g.m_tiles = (p->og + BM - 1) / BM;
  const int panels = p->KH * p->KW * ((p->cg + 63) / 64);
  // panels per tile: fewest panel loads per pixel box over the whole product (2 dY panels + `per` patch panels
  // for each of ceil(panels / per) tiles); ties go to the wider tile
  g.per = 1;
  long long best_cost = -1;
  for (int c = 1; c <= 4 && c <= panels; ++c) {
    const long long cost = (long long)((panels + c - 1) / c) * (2 + c);
    if (best_cost < 0 || cost <= best_cost) { best_cost = cost; g.per = c; }
  }
  g.n_tiles = (panels + g.per - 1) / g.per;
  int split = p->split_k;
  const long long tiles = (long long)g.m_tiles * g.n_tiles;
  if (split <= 0) {
    split = 1;
    if (tiles < sms && g.kt >= 8) {
      // the busiest SM walks `waves` slices, and each costs about eight k-tiles of time beside its own: filling the
      // pipeline, and a read-modify-write of its part of the gradient.  That prefers one wave of longer slices where
      // it fills the machine.  One wave against two, us: 256 x 13 x 13, 256 -> 384: 64.0, 66.6; 192 -> 128: 24.6, 27.7;
      // 32 x 14 x 14, 128 -> 160: 13.3, 17.9; 100 x 32 x 32 stride 2, 80 -> 80: 16.4, 18.4
      auto cost = [&](long long n) { return (tiles * n + sms - 1) / sms * ((g.kt + n - 1) / n + 8); };
      const long long most = (2 * sms) / tiles < g.kt / 4 ? (2 * sms) / tiles : g.kt / 4;
      for (long long n = 2; n <= most; ++n)
        if (cost(n) < cost(split)) split = (int)n;
    }
  }
  if (split > g.kt) split = g.kt;
  if (split > 1) {
    const int per_k = (g.kt + split - 1) / split;
    split = (g.kt + per_k - 1) / per_k;      // every k-slice non-empty
  }
  g.split = split;
  // rows off 16-, 32- and 64-channel boundaries (32-byte sectors, half lines, lines)
  auto off = [](long long v, double by16, double by32, double by64) { return v % 16 ? by16 : v % 32 ? by32 : v % 64 ? by64 : 0.0; };
  const double waves = (double)((tiles * split + sms - 1) / sms), kt = (g.kt + split - 1) / split;
  g.us = 5.95 + waves * (0.43 * g.per + kt * (0.28 + off(p->y_pitch | p->og, 0.119, 0.053, 0.031) +
                                              g.per * (0.009 + off(p->x_pitch | p->cg, 0.061, 0.021, 0.011))));
  return g;
}
bool takes_pairs(const BoxPlan& b) { return b.pair >= 0 && b.pair < 0.97 * b.one; }

template <int MODE, bool PAIR>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const OutMaps& tc, const ConvDev& d, int units, cudaStream_t st) {
  const int stage_bytes = A_STAGE_BYTES + (PAIR ? d.bn / 2 : d.bn) * BK * 2;
  const size_t smem = (size_t)d.stages * stage_bytes + d.slabs * C_SLAB_BYTES + sizeof(SmemCtl) + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(conv_tc_kernel<MODE, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  if (!PAIR) {
    geeps_launch(conv_tc_kernel<MODE, PAIR>, units, kThreads, smem, st, ta, tb, tc, d);
    return (int)cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * units));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, conv_tc_kernel<MODE, PAIR>, ta, tb, tc, d);
  return e == cudaSuccess ? (int)cudaGetLastError() : (int)e;
}

}  // namespace

extern "C" {

int geeps_conv_tc_supported(const GeepsConvTcParams* p) {
  if (p->B <= 0 || p->H <= 0 || p->W <= 0 || p->cg <= 0 || p->og <= 0 || p->KH <= 0 || p->KW <= 0) return 0;
  const int s = p->stride > 1 ? p->stride : 1;
  // a strided data gradient is a problem for each parity class of dX; a class without taps (filter narrower than the stride)
  // would have to be zeroed instead and is left to the caller
  if (s > 8 || (s > 1 && p->mode == MODE_DGRAD && (p->KH < s || p->KW < s))) return 0;
  if (p->OH != (p->H + 2 * p->pad - p->KH) / s + 1 || p->OW != (p->W + 2 * p->pad - p->KW) / s + 1) return 0;
  if (p->OH <= 0 || p->OW <= 0) return 0;
  if (((uintptr_t)p->x & 15) || ((uintptr_t)p->y & 15) || ((uintptr_t)p->w & 15)) return 0;
  if ((p->x_pitch & 7) || (p->y_pitch & 7) || (p->cg & 7) || (p->og & 7)) return 0;
  if (p->mode == MODE_WGRAD ? (p->ldw & 3) : (p->ldw & 7)) return 0;
  if (p->ldw < (long long)p->KH * p->KW * p->cg) return 0;
  if (p->mode < 0 || p->mode > 2) return 0;
  return 1;
}

}  // extern "C"

extern "C" {

// us that the better of the box kernels is expected to take for a stride-1 forward or data-gradient product
double geeps_conv_box_us(const GeepsConvTcParams* p) {
  const BoxPlan b = plan_box(p, 1, 1, geeps_sm_count());
  return takes_pairs(b) ? b.pair : b.one;
}
double geeps_conv_box_wgrad_us(const GeepsConvTcParams* p) { return plan_wgrad_box(p, geeps_sm_count()).us; }
int geeps_conv_box_wgrad_slices(const GeepsConvTcParams* p) { return plan_wgrad_box(p, geeps_sm_count()).split; }
long long geeps_conv_box_wgrad_steps(const GeepsConvTcParams* p) {
  const WgradPlan g = plan_wgrad_box(p, geeps_sm_count());
  return (long long)((g.kt + g.split - 1) / g.split) * ((g.bw * g.bh * g.bnb + 15) / 16);
}
int geeps_conv_box_pairs(const GeepsConvTcParams* p) {
  return p->mode != MODE_WGRAD && p->stride <= 1 && geeps_conv_tc_supported(p) && takes_pairs(plan_box(p, 1, 1, geeps_sm_count())) ? 1 : 0;
}

}  // extern "C"

namespace {
// parity classes (a, b) that one launch of a data gradient covers; s = 1: the whole problem, one class
struct DgradClasses { int s, n, a[MAX_CLS], b[MAX_CLS]; };
int conv_tc_run(const GeepsConvTcParams* p, const DgradClasses& cls, void* stream);
}  // namespace

extern "C" {

int geeps_conv_wgrad_adds(const GeepsConvTcParams* p) {
  if (p->mode != MODE_WGRAD || !geeps_conv_tc_supported(p)) return 0;
  return (p->split_k >= 0 && geeps_conv_wgrad_halo_applicable(p)) || plan_wgrad_box(p, geeps_sm_count()).split > 1;
}
int geeps_conv_tc(const GeepsConvTcParams* p, void* stream) {
  if (!geeps_conv_tc_supported(p)) return (int)cudaErrorInvalidValue;
  if (p->mode != MODE_WGRAD && p->split_k >= 0 && geeps_conv_halo_applicable(p)) return geeps_conv_halo(p, stream);
  if (p->mode == MODE_WGRAD && p->split_k >= 0 && geeps_conv_wgrad_halo_applicable(p))
    return geeps_conv_wgrad_halo(p, stream);
  if (p->mode == MODE_DGRAD && p->stride > 1) {
    // dX[s i + a, s j + b] = sum over u, v of dY[i + oh0 - u, j + ow0 - v] * W[kh0 + s u, kw0 + s v]: s * s
    // stride-1 problems over dense views of dX, each with its sub-filter
    // (100 x 32 x 32 pixels, 80 -> 80 channels, stride 2: four launches of 8 - 12 us one after the other 32.3 us, one launch
    // 19.5).  Classes with more taps come first: few large tiles left over at the end would wait for one another
    const int sd = p->stride;
    DgradClasses all{sd, 0, {}, {}};
    auto taps = [&](int a, int b) {
      const int kh0 = (a + p->pad) % sd, kw0 = (b + p->pad) % sd;
      return ((p->KH - kh0 + sd - 1) / sd) * ((p->KW - kw0 + sd - 1) / sd);
    };
    int order[64], n = 0;
    for (int a = 0; a < sd && a < p->H; ++a)
      for (int b = 0; b < sd && b < p->W; ++b) order[n++] = a * sd + b;
    for (int i = 1; i < n; ++i)       // insertion sort, stable: at most 8 x 8 classes
      for (int j = i; j > 0 && taps(order[j] / sd, order[j] % sd) > taps(order[j - 1] / sd, order[j - 1] % sd); --j) {
        const int o = order[j]; order[j] = order[j - 1]; order[j - 1] = o;
      }
    for (int i = 0; i < n; ++i) {
      all.a[all.n] = order[i] / sd; all.b[all.n] = order[i] % sd;
      if (++all.n == MAX_CLS || i + 1 == n) {
        const int e = conv_tc_run(p, all, stream);
        if (e) return e;
        all.n = 0;
      }
    }
    return 0;
  }
  return conv_tc_run(p, DgradClasses{1, 1, {0}, {0}}, stream);
}

}  // extern "C"

namespace {

int conv_tc_run(const GeepsConvTcParams* p, const DgradClasses& cls, void* stream) {
  const int kSMs = geeps_sm_count();
  cudaStream_t st = (cudaStream_t)stream;
  ConvDev d;
  d.bias = p->mode == MODE_FWD ? p->bias : nullptr;
  d.status = p->status;
  d.taps = p->KH * p->KW; d.KW = p->KW; d.pad = p->pad;
  d.relu = p->mode == MODE_FWD ? p->relu : 0;
  d.split_k = 1;
  d.zero_fill_c = 0;
  d.ch_valid = p->cg;
  d.narrow = 0;
  d.stride = p->stride > 1 ? p->stride : 1;
  d.n_cls = cls.n;
  d.tap_dw = cls.s; d.tap_dh = cls.s * p->KW;
  memset(d.cls, 0, sizeof(d.cls));
  CUtensorMap ta, tb;
  OutMaps tc;
  memset(&tc, 0, sizeof(tc));
  bool ok = true, pair = false;
  const long long wdims[3] = {p->cg, d.taps, p->og};
  if (p->mode == MODE_FWD || p->mode == MODE_DGRAD) {
    const bool fwd = p->mode == MODE_FWD;
    const int GW = fwd ? p->OW : (p->W + cls.s - 1) / cls.s, GH = fwd ? p->OH : (p->H + cls.s - 1) / cls.s;
    if (!fwd) d.stride = 1;
    const BoxPlan plan = plan_box(p, cls.s, cls.n, kSMs);
    d.bw = plan.bw; d.bh = plan.bh; d.bnb = plan.bnb;
    d.rows = d.bw * d.bh * d.bnb;
    d.wt = (GW + d.bw - 1) / d.bw; d.ht = (GH + d.bh - 1) / d.bh;
    const int bt = (p->B + d.bnb - 1) / d.bnb;
    d.m_tiles = d.wt * d.ht * bt;
    int CW[MAX_CLS], CH[MAX_CLS];
    if (!fwd) {
      d.m_tiles = 0;
      for (int i = 0; i < cls.n; ++i) {
        DgradDev& q = d.cls[i];
        const int kh0 = (cls.a[i] + p->pad) % cls.s, kw0 = (cls.b[i] + p->pad) % cls.s;
        const int khs = (p->KH - kh0 + cls.s - 1) / cls.s, kws = (p->KW - kw0 + cls.s - 1) / cls.s;   // >= 1: KH, KW >= s
        CW[i] = (p->W - cls.b[i] + cls.s - 1) / cls.s; CH[i] = (p->H - cls.a[i] + cls.s - 1) / cls.s;
        q.wt = (CW[i] + d.bw - 1) / d.bw; q.ht = (CH[i] + d.bh - 1) / d.bh;
        q.m_tiles = q.wt * q.ht * bt;
        q.pad_h = (cls.a[i] + p->pad - kh0) / cls.s; q.pad_w = (cls.b[i] + p->pad - kw0) / cls.s;
        q.tap0 = kh0 * p->KW + kw0;
        q.KW = kws; q.kt_total = khs * kws;            // times the channel chunks, below
        d.m_tiles += q.m_tiles;
      }
    }
    const int kch = fwd ? p->cg : p->og;          // reduced channels
    const int nch = fwd ? p->og : p->cg;          // produced channels
    d.cchunks = (kch + 63) / 64;
    d.kt_total = d.taps * d.cchunks;
    d.n_valid = nch;
    d.bn = plan.bn;
    d.n_tiles = plan.n_tiles;
    pair = p->split_k != -2 && takes_pairs(plan);
    d.m_units = pair ? (d.m_tiles + 1) / 2 : d.m_tiles;
    if (!fwd) d.m_units = 0;
    for (int i = 0, t0 = 0; !fwd && i < cls.n; ++i) {
      DgradDev& q = d.cls[i];
      q.kt_total *= d.cchunks;
      q.m_units = pair ? (q.m_tiles + 1) / 2 : q.m_tiles;
      d.m_units += q.m_units;
      q.t0 = t0;
      t0 += q.m_units * d.n_tiles;
    }
    const long long wst[2] = {(long long)p->cg * 2, p->ldw * 2};
    if (fwd) {
      ok = make_act_map(&ta, p->x, p->cg, p->W, p->H, p->B, p->x_pitch, d.bw, d.bh, d.bnb, false, d.stride);
      const int wbox[3] = {64, 1, pair ? d.bn / 2 : d.bn};
      ok = ok && make_map(&tb, p->w, 3, wdims, wst, wbox, false);
      d.narrow = narrow_store(p->og, p->y_pitch);
      ok = ok && make_act_map(&tc.m[0], p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, d.bw, d.bh, d.bnb, d.narrow != 0);
    } else {
      ok = make_act_map(&ta, p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, d.bw, d.bh, d.bnb);
      const int wbox[3] = {64, 1, 64};
      ok = ok && make_map(&tb, p->w, 3, wdims, wst, wbox, false);
      d.narrow = narrow_store(p->cg, p->x_pitch);
      for (int i = 0; i < cls.n; ++i)
        ok = ok && make_act_view(&tc.m[i], p->x, p->cg, p->W, p->H, p->B, p->x_pitch, cls.s, cls.a[i], cls.b[i], CW[i], CH[i],
                                 d.bw, d.bh, d.bnb, d.narrow != 0);
    }
  } else {
    const WgradPlan plan = plan_wgrad_box(p, kSMs);
    d.bw = plan.bw; d.bh = plan.bh; d.bnb = plan.bnb;
    d.rows = d.bw * d.bh * d.bnb;
    d.wt = (p->OW + d.bw - 1) / d.bw; d.ht = (p->OH + d.bh - 1) / d.bh;
    d.kt_total = plan.kt;
    d.m_tiles = d.m_units = plan.m_tiles;
    d.cchunks = (p->cg + 63) / 64;
    d.n_valid = d.taps * d.cchunks * 64;
    d.bn = plan.per * 64;
    d.n_tiles = plan.n_tiles;
    d.zero_fill_c = d.cchunks * 64;
    ok = make_act_map(&ta, p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, d.bw, d.bh, d.bnb);
    ok = ok && make_act_map(&tb, p->x, p->cg, p->W, p->H, p->B, p->x_pitch, d.bw, d.bh, d.bnb, false, d.stride);
    const long long wst[2] = {(long long)p->cg * 4, p->ldw * 4};
    const int wbox[3] = {32, 1, BM};
    ok = ok && make_map(&tc.m[0], p->w, 3, wdims, wst, wbox, true);
    const int split = plan.split;
    d.split_k = split;
    const long long kd = (long long)d.taps * p->cg;
    if (split > 1) {
      // partial sums are reduce-added: the whole [og][ldw] block starts at zero
      int e = p->cleared ? 0 : geeps_scale_matrix_f32((float*)p->w, p->og, p->ldw, p->ldw, 0.f, stream);
      if (e) return e;
    } else if (p->ldw > kd) {
      // the pad columns past the last tap are never stored: keep them at zero
      int e = geeps_scale_matrix_f32((float*)p->w + kd, p->og, p->ldw - kd, p->ldw, 0.f, stream);
      if (e) return e;
    }
  }
  if (!ok) return (int)cudaErrorInvalidValue;
  int tmem_cols = 32;
  while (tmem_cols < 2 * d.bn) tmem_cols <<= 1;
  d.tmem_cols = tmem_cols;
  const int stage_bytes = A_STAGE_BYTES + (pair ? d.bn / 2 : d.bn) * BK * 2;
  const long long num_tiles = (long long)d.m_tiles * d.n_tiles * d.split_k;
  // Two groups share a tile of three slabs unevenly, and where many tiles follow one another the epilogue is covered anyway:
  // one group takes them.  3 x 3 forward, us before there were two groups / with two / so: 47 x 52 x 52, 64 -> 312 48.9 / 50.8 /
  // 49.1; 128 x 28 x 28, 64 -> 320 37.7 / 39.1 / 37.0; 32 x 56 x 56, 64 -> 192 (5.3 tiles an SM) 22.0 / 22.2 / 21.3.  Few
  // tiles are faster with two: 64 x 28 x 28, 64 -> 160 (2.6) 12.7 / 11.9 / 12.1; 128 -> 192 at batch 32 14.8 / 13.7 / 13.9.
  const int slab_cols = p->mode == MODE_WGRAD || d.narrow ? 32 : 64;
  d.groups = p->mode == MODE_FWD && !d.narrow && (d.bn + 63) / 64 == 3 && num_tiles >= 4LL * kSMs ? 1 : kGroups;
  d.slabs = d.groups == 2 && d.bn > slab_cols ? 4 : 2;
  d.stages = (224 * 1024 - d.slabs * C_SLAB_BYTES) / stage_bytes;
  if (d.stages > MAX_STAGES) d.stages = MAX_STAGES;
  if (d.stages < 2) d.stages = 2;
  const long long work = (long long)d.m_units * d.n_tiles * d.split_k, room = pair ? kSMs / 2 : kSMs;
  const int units = (int)(work < room ? work : room);
  if (p->mode == MODE_FWD) return pair ? launch<MODE_FWD, true>(ta, tb, tc, d, units, st) : launch<MODE_FWD, false>(ta, tb, tc, d, units, st);
  if (p->mode == MODE_DGRAD)
    return pair ? launch<MODE_DGRAD, true>(ta, tb, tc, d, units, st) : launch<MODE_DGRAD, false>(ta, tb, tc, d, units, st);
  return launch<MODE_WGRAD, false>(ta, tb, tc, d, units, st);
}

}  // namespace
