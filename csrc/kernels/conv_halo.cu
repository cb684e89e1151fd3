// Implicit-GEMM convolution (stride 1, forward and data gradient) that fetches every activation ONCE per
// 64-channel chunk instead of once per filter tap, and issues the widest MMA the tensor core has.
//
// conv_tc.cu loads, for each (tap, chunk) k-step, the 128-pixel activation box shifted by the tap: a 5 x 5 filter
// reads the same activations 25 times out of L2.  Here a tile is up to 256 CONSECUTIVE positions of the zero-padded
// image flattened with pitch PW = out_width + KW - 1:
//
//     out_flat[m] = sum over taps (ty, tx) and channels of  in_flat[m + ty * PW + tx] * W[tap]
//
// (positions whose column is >= out_width are computed and dropped).  One TMA box load brings the halo tile -
// [rows + KH - 1][PW][64 channels], zero-filled outside the image - into shared memory as exactly that flat array,
// 128 bytes per position with the 128-byte swizzle.  The operand of tap (ty, tx) is then the SAME tile read through
// an MMA descriptor whose start address is advanced by (ty * PW + tx) whole 128-byte rows.  Such a start is no longer
// 1024-byte aligned, and that is fine: the 128-byte swizzle is a function of the absolute shared-memory address bits
// (chunk bits 4..6 xor row bits 7..9), for the TMA write and for the MMA read alike, so the descriptor's base-offset
// field stays 0 (measured: with (address >> 7) & 7 in that field the products are wrong, with 0 they match the fp32
// reference).  Only the weights stream per tap.
//
// The product is computed transposed: D[channel, position] = W[channel, k] * X[position, k]^T, weights as the M = 128
// operand (128 output channels per tile; input channels for the data gradient), positions as N <= 256.  One thread
// issues every MMA and spends a few hundred cycles of instructions per pipeline stage (measured: the issue loop, not
// the tensor pipe or L2, bounded the first version of this kernel, which had positions as M = 128 and 48 .. 128
// channels as N), so every MMA must carry as much work as the instruction allows: 128 x 256 x 16.  The roles run
// their loops with the whole warp converged and elect one lane for the TMA / MMA / commit instructions.
//
// The accumulator therefore holds channels in TMEM lanes and positions in columns.  Each epilogue thread owns one
// channel: it adds that channel's bias (one register), applies ReLU and writes bf16 into a [position][64 channels]
// slab with the 128-byte swizzle - the 32 lanes of a warp write 64 contiguous bytes of one position per store - and
// a 4-D TMA store (64 channels, PW, rows, 1) writes the slab to the NHWC tensor, clipping the dropped columns, the
// rows past the image and the channels past the layer's extent.  A tile is two store blocks of Rb image rows; the
// pitch PW is padded until a block has a multiple of 8 positions, which makes the swizzled chunk offsets of a
// thread's channel constants; eight epilogue warps (two per TMEM lane quarter, alternate column groups) share the
// conversion.  Blocks leave through one pair of slabs, one after the other, where the main loop is long: the epilogue has
// the time to wait for a slab to be read, the main loop none to wait for its weights (16 KB per tap and chunk out of L2), and
// the 32 KB of a second pair are two more weight stages: conv2 forward per group with 3 stages 66.6 us, with 5 60.4; conv1
// with 4 99, with 6 96.  Two pairs in turn where it is short (two_slab_pairs).
//
// conv_tc() routes a forward / data-gradient call here when the geometry wastes little (see
// geeps_conv_halo_applicable); GEEPS_HALO_CONV=0 keeps every call on the box kernel.  Bounded waits and TMEM
// double buffering as in conv_tc.cu.
#include <cuda.h>
#include <cuda_bf16.h>
#include <mutex>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "kernels.h"
#include "tc05.cuh"

namespace {

constexpr int BM = 128;                       // channels per tile (TMEM lanes)
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int PANEL_BYTES = 64 * BK * 2;
constexpr int W_STAGE_BYTES = BM * BK * 2;    // 128 channels x 64 k (forward) or two [64 k][64 channels] panels (dgrad)
constexpr int MAX_X_STAGES = 2;
constexpr int MAX_W_STAGES = 16;             // of one panel; 8 of two
constexpr uint64_t WAIT_BUDGET_NS = 2000000000ull;
constexpr int C_SLAB_BYTES = 128 * 128;       // 128 positions x 64 channels bf16
constexpr int ACC_COLS = 256;
constexpr int SMEM_BUDGET = 224 * 1024;       // tiles, weights and slabs
constexpr int kEpilogueWarps = 8;             // two per TMEM lane quarter: they take alternate column groups
constexpr int kThreads = 64 + 32 * kEpilogueWarps;

// MODE_DGRAD2: a data gradient with at most 64 channels, whose 128 accumulator rows hold them twice: once for the even and
// once for the odd column of a pair, a position being a pair.  Both read the same activations one column apart, so a filter
// row of KW taps takes KW + 1 steps - the even column has no tap in the last, the odd one none in the first - of half
// the positions: (KW + 1) / 2 KW of the products that MODE_DGRAD spends with half its rows empty.  The activations are
// loaded by column parity (two maps with twice the pixel pitch) and step s reads parity s % 2 from column s / 2 on; the two
// halves leave through the maps of dX's even and odd columns.  Step s multiplies taps s (even column) and s - 1 (odd): a tap
// is loaded once for both, as two steps read it from neighbouring panels - with a load for each the weights' rows (96 bytes
// of every 2400 for 48 channels and 5 x 5) were the bound, 109 us below.  A half without a tap is left out of the step's
// products (disabled lanes), so every output adds the same products in the same order as in MODE_DGRAD and nothing else.
// 256 x 27 x 27, 128 -> 48, 5 x 5: 114 us in MODE_DGRAD, 85.5 here.
enum { MODE_FWD = 0, MODE_DGRAD = 1, MODE_DGRAD2 = 2 };

struct HaloDev {
  const float* bias; int* status;
  int KH, KW, taps, cchunks, k_last;   // k_last: MMA k-substeps (of 16) in the last chunk (zero channels are skipped)
  int PW, Rb, px, py;                  // padded pitch, image rows per store block (two blocks per tile), halo left / top
  int KWs;                             // steps per filter row: KW, or KW + 1 (MODE_DGRAD2)
  int w_bytes, slab_bytes, slab_pairs; // all weight stages; one store slab; slabs per 64 channels
  int x0, x1, x_tile_bytes;            // MODE_DGRAD2: first column of the two parity maps; bytes of a parity's halo tile
  int split, ncols2, ncols1;           // positions per block (Rb * PW); MMA N for a tile of two blocks / one block
  int GH;                              // output rows of the image
  int row_tiles, m_tiles, n_images;    // tiles = m_tiles * n_images * row_tiles
  int n_valid;                         // channels produced
  int x_stage_bytes, stages_x, stages_w;
  int relu;
};

struct SmemCtl {
  uint64_t full_x[MAX_X_STAGES], empty_x[MAX_X_STAGES];
  uint64_t full_w[MAX_W_STAGES], empty_w[MAX_W_STAGES];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

struct Tile { int b, y0, nb, mi; };
__device__ __forceinline__ Tile decode_tile(const HaloDev& d, int t) {
  Tile q;
  const int per_m = d.n_images * d.row_tiles;
  q.mi = t / per_m;
  const int r = t - q.mi * per_m;
  q.b = r / d.row_tiles;
  q.y0 = (r - q.b * d.row_tiles) * (2 * d.Rb);
  q.nb = d.GH - q.y0 > d.Rb ? 2 : 1;
  return q;
}

// tmX: the source activations (fwd: X, dgrad: dY) as (c, w, h, b) with box (64, PW, 2 Rb + KH - 1, 1);
// tmW: weights (ci, tap, co): fwd box (64 ci, 1, 128 co) K-major, dgrad box (64 ci, 1, 64 co) = one MN-major panel;
// tmC: the result (fwd: Y, dgrad: dX) with box (64, PW, Rb, 1); tmX1, tmC1: MODE_DGRAD2's second parity.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
conv_halo_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmX1,
                 const __grid_constant__ CUtensorMap tmC1, const HaloDev d) {
  constexpr bool W_MN = MODE != MODE_FWD;
  constexpr bool PAIR = MODE == MODE_DGRAD2;
  constexpr int CH = PAIR ? 64 : BM;            // channels per tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles_x = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles_w = tiles_x + (size_t)d.stages_x * d.x_stage_bytes;
  uint8_t* cslab = tiles_w + d.w_bytes;
  SmemCtl* ctl = (SmemCtl*)(cslab + 2 * d.slab_pairs * d.slab_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_tiles = d.m_tiles * d.n_images * d.row_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < d.stages_x; ++s) { tc05::mbar_init(&ctl->full_x[s], 1); tc05::mbar_init(&ctl->empty_x[s], 1); }
    for (int s = 0; s < d.stages_w; ++s) { tc05::mbar_init(&ctl->full_w[s], 1); tc05::mbar_init(&ctl->empty_w[s], 1); }
    for (int a = 0; a < 2; ++a) { tc05::mbar_init(&ctl->tmem_full[a], 1); tc05::mbar_init(&ctl->tmem_empty[a], kEpilogueWarps); }
    ctl->abort_flag = 0;
    tc05::mbar_fence_init();
  }
  {
    // an MMA reads N rows from a shifted start: the few rows past the halo tile feed dropped columns only, but
    // they must not hold NaN patterns left by an earlier kernel
    uint4* z = reinterpret_cast<uint4*>(tiles_x);
    const int n16 = d.stages_x * d.x_stage_bytes / 16;
    for (int i = threadIdx.x; i < n16; i += blockDim.x) z[i] = make_uint4(0, 0, 0, 0);
    tc05::fence_proxy_async_smem();
  }
  if (warp == 1) {
    tc05::tmem_alloc(&ctl->tmem_base, 2 * ACC_COLS);
    tc05::tmem_relinquish();
  }
  tc05::fence_before_sync();
  __syncthreads();
  tc05::fence_after_sync();
  const uint32_t tmem = ctl->tmem_base;
  geeps_pdl_wait();          // everything above touches this CTA's own memory only
  volatile int* abort_flag = &ctl->abort_flag;
  const int NR = 2 * d.Rb + d.KH - 1;
  const uint32_t x_tx = (uint32_t)(NR * d.PW * 128) * (PAIR ? 2u : 1u);

  if (warp == 0) {
    // ---------------- TMA producer: one halo tile per chunk, one weight tile per (tap, chunk) ----------------
    const bool leader = tc05::elect_one();
    if (leader) { tc05::tma_prefetch_desc(&tmX); tc05::tma_prefetch_desc(&tmW); }
    int sx = 0, sw = 0, wrow = 0;
    uint32_t phx = 0, phw = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const Tile q = decode_tile(d, t);
      for (int cc = 0; cc < d.cchunks && ok; ++cc) {
        if (!tc05::mbar_wait_warp(&ctl->empty_x[sx], phx ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
        if (leader) {
          tc05::mbar_expect_tx(&ctl->full_x[sx], x_tx);
          uint8_t* xt = tiles_x + (size_t)sx * d.x_stage_bytes;
          tc05::tma_load_4d(xt, &tmX, &ctl->full_x[sx], cc * 64, PAIR ? d.x0 : -d.px, q.y0 - d.py, q.b);
          if (PAIR) tc05::tma_load_4d(xt + d.x_tile_bytes, &tmX1, &ctl->full_x[sx], cc * 64, d.x1, q.y0 - d.py, q.b);
        }
        if (++sx == d.stages_x) { sx = 0; phx ^= 1u; }
        const int loads = d.KH * d.KW;
        int panel = d.KW - 1;                        // MODE_DGRAD2: where in its row's panels (from wrow on) the tap goes
        for (int tap = 0; tap < loads; ++tap) {
          if (!tc05::mbar_wait_warp(&ctl->empty_w[sw], phw ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          if (leader) {
            uint8_t* dst = tiles_w + (PAIR ? (size_t)(wrow + panel) * PANEL_BYTES : (size_t)sw * W_STAGE_BYTES);
            tc05::mbar_expect_tx(&ctl->full_w[sw], PAIR ? PANEL_BYTES : W_STAGE_BYTES);
            if (MODE == MODE_FWD) {
              tc05::tma_load_3d(dst, &tmW, &ctl->full_w[sw], cc * 64, tap, q.mi * BM);
            } else if (PAIR) {
              tc05::tma_load_3d(dst, &tmW, &ctl->full_w[sw], q.mi * CH, loads - 1 - tap, cc * 64);
            } else {
              // data gradient: the filter is applied mirrored; rows of the product are input channels
              const int wtap = loads - 1 - tap;
              tc05::tma_load_3d(dst, &tmW, &ctl->full_w[sw], q.mi * BM, wtap, cc * 64);
              tc05::tma_load_3d(dst + PANEL_BYTES, &tmW, &ctl->full_w[sw], q.mi * BM + 64, wtap, cc * 64);
            }
          }
          if (++sw == d.stages_w) { sw = 0; phw ^= 1u; }
          if (PAIR && --panel < 0) {
            panel = d.KW - 1;
            wrow = sw;
          }
        }
      }
    }
    geeps_pdl_trigger();       // every operand is on its way: the rest of this CTA is its last products and stores
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const bool leader = tc05::elect_one();
    const uint32_t idesc2 = tc05::make_idesc_bf16(BM, d.ncols2, W_MN ? 1 : 0, 0);
    const uint32_t idesc1 = tc05::make_idesc_bf16(BM, d.ncols1, W_MN ? 1 : 0, 0);
    constexpr uint32_t d_hi = tc05::desc_hi(1024);
    constexpr uint32_t w_kstep = W_MN ? 128u : 2u;      // 16 k: two 8-row groups of 1024 bytes, or 32 bytes in the row
    const uint32_t row_wrap8 = (uint32_t)(d.PW - d.KW + 1) * 8u;
    // MODE_DGRAD2: from a step to the next alternately to the other parity's tile, and back and one column on
    const uint32_t other = (uint32_t)d.x_tile_bytes >> 4;
    const uint32_t pair_wrap = (uint32_t)d.PW * 8u - (uint32_t)(d.KW >> 1) * 8u - ((d.KW & 1) ? other : 0u);
    uint32_t tile_i = 0;
    int sx = 0, sw = 0, wrow = 0;
    uint32_t phx = 0, phw = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++tile_i) {
      const Tile q = decode_tile(d, t);
      const uint32_t idesc = q.nb == 2 ? idesc2 : idesc1;
      const uint32_t acc = tile_i & 1u, acc_ph = (tile_i >> 1) & 1u;
      if (!tc05::mbar_wait_warp(&ctl->tmem_empty[acc], acc_ph ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
      tc05::fence_after_sync();
      const uint32_t tacc = tmem + acc * (uint32_t)ACC_COLS;
      uint32_t accumulate = 0;                          // the very first MMA of a tile overwrites the accumulator
      for (int cc = 0; cc < d.cchunks && ok; ++cc) {
        if (!tc05::mbar_wait_warp(&ctl->full_x[sx], phx, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
        // tap (ty, tx) reads the halo tile from row ty * PW + tx on: 8 descriptor units (128 bytes) per row
        uint32_t x_lo = tc05::desc_lo(tc05::smem_u32(tiles_x + (size_t)sx * d.x_stage_bytes), 16);
        const bool full_k = cc + 1 < d.cchunks || d.k_last == BK / UMMA_K;
        int tx = 0;
        for (int tap = 0; tap < d.taps; ++tap) {
          // MODE_DGRAD2: the last step of a row has no tap of its own
          if ((!PAIR || tx < d.KW) && !tc05::mbar_wait_warp(&ctl->full_w[sw], phw, abort_flag, WAIT_BUDGET_NS)) {
            ok = false;
            break;
          }
          tc05::fence_after_sync();
          if (leader) {
            const uint8_t* wt = tiles_w + (PAIR ? (ptrdiff_t)(wrow + d.KW - 1 - tx) * PANEL_BYTES : (ptrdiff_t)sw * W_STAGE_BYTES);
            const uint32_t w_lo = tc05::desc_lo(tc05::smem_u32(wt), W_MN ? PANEL_BYTES : 16);
            if (PAIR) {
              // no product in the half whose column has no tap in this step; the odd column's first overwrites
              const uint32_t no_even = tx == d.KW ? ~0u : 0u, no_odd = tx == 0 ? ~0u : 0u;
              const int ks = full_k ? BK / UMMA_K : d.k_last;
              if (cc == 0 && tap == 1) {
                tc05::mma_bf16_ss_halves(tacc, w_lo, d_hi, x_lo, d_hi, idesc, 1u, no_even, ~0u);
                tc05::mma_bf16_ss_halves(tacc, w_lo, d_hi, x_lo, d_hi, idesc, 0u, ~0u, 0u);
              } else {
                tc05::mma_bf16_ss_halves(tacc, w_lo, d_hi, x_lo, d_hi, idesc, accumulate, no_even, no_odd);
              }
#pragma unroll
              for (int j = 1; j < BK / UMMA_K; ++j)
                if (j < ks) tc05::mma_bf16_ss_halves(tacc, w_lo + j * w_kstep, d_hi, x_lo + 2 * j, d_hi, idesc, 1u, no_even, no_odd);
            } else if (full_k) {
              tc05::mma_bf16_ss_lohi(tacc, w_lo, d_hi, x_lo, d_hi, idesc, accumulate);
              tc05::mma_bf16_ss_lohi(tacc, w_lo + w_kstep, d_hi, x_lo + 2, d_hi, idesc, 1u);
              tc05::mma_bf16_ss_lohi(tacc, w_lo + 2 * w_kstep, d_hi, x_lo + 4, d_hi, idesc, 1u);
              tc05::mma_bf16_ss_lohi(tacc, w_lo + 3 * w_kstep, d_hi, x_lo + 6, d_hi, idesc, 1u);
            } else {
              tc05::mma_bf16_ss_lohi(tacc, w_lo, d_hi, x_lo, d_hi, idesc, accumulate);
              if (d.k_last > 1) tc05::mma_bf16_ss_lohi(tacc, w_lo + w_kstep, d_hi, x_lo + 2, d_hi, idesc, 1u);
              if (d.k_last > 2) tc05::mma_bf16_ss_lohi(tacc, w_lo + 2 * w_kstep, d_hi, x_lo + 4, d_hi, idesc, 1u);
            }
            // MODE_DGRAD2: the tap of the step before is used up; it is the one in front of sw, or of 0 behind a turn
            if (!PAIR) tc05::mma_commit(&ctl->empty_w[sw]);
            else if (tx > 0) tc05::mma_commit(&ctl->empty_w[sw == 0 ? d.stages_w - 1 : sw - 1]);
          }
          accumulate = 1u;
          if (!PAIR || tx < d.KW) {
            if (++sw == d.stages_w) { sw = 0; phw ^= 1u; }
          }
          if (PAIR) {
            // step tx read parity tx % 2 at column tx / 2
            if (tx == d.KW) { tx = 0; x_lo += pair_wrap; wrow = sw; }
            else { x_lo += (tx & 1) ? 8u - other : other; ++tx; }
          } else if (++tx == d.KW) { tx = 0; x_lo += row_wrap8; } else { x_lo += 8u; }
        }
        if (ok && leader) tc05::mma_commit(&ctl->empty_x[sx]);
        if (++sx == d.stages_x) { sx = 0; phx ^= 1u; }
      }
      if (ok && leader) tc05::mma_commit(&ctl->tmem_full[acc]);
    }
  } else {
    // ---------------- epilogue: TMEM (channel lanes) -> bf16 [position][channel] slab -> TMA store ----------------
    const int q4 = warp & 3;                       // TMEM lane quarter this warp may access
    const int sub = (warp - 2) >> 2;               // which of the quarter's two warps
    const int half = q4 >> 1;                      // which 64-channel slab
    const int chin = (q4 & 1) * 32 + lane;         // channel inside the slab
    const uint32_t chunk = (uint32_t)(chin >> 3), within = (uint32_t)((chin & 7) * 2);
    // Slab rows are positions (128 bytes, 128-byte swizzle: 16-byte chunk ^ row % 8).  A block has a multiple of
    // 8 positions and a column group starts at a multiple of 32, so the row of element e of a group is congruent
    // to e mod 8: the eight swizzled chunk offsets of this thread's channel are constants of the thread.
    uint32_t cb[8];
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) cb[jj] = ((chunk ^ (uint32_t)jj) << 4) + within;
    const uint32_t slab_base = tc05::smem_u32(cslab) + (uint32_t)(half * d.slab_bytes);
    const uint32_t next_pair = d.slab_pairs == 2 ? (uint32_t)(2 * d.slab_bytes) : 0u;
    uint32_t slab_off = 0;                         // 0 and next_pair in turn: the slab of the next block stored
    const bool storer = lane == 0 && (q4 & 1) == 0 && sub == 0;          // one thread per slab issues its stores
    const float floor_v = d.relu ? 0.f : -INFINITY;
    uint32_t tile_i = 0;
    int bias_mi = -1;
    float bias_v = 0.f;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++tile_i) {
      const Tile q = decode_tile(d, t);
      if (q.mi != bias_mi) {                       // tiles are ordered by channel block: this happens m_tiles times
        const int ch = q.mi * BM + q4 * 32 + lane;
        bias_v = (MODE == MODE_FWD && d.bias != nullptr && ch < d.n_valid) ? __ldg(d.bias + ch) : 0.f;
        bias_mi = q.mi;
      }
      const bool slab_valid = PAIR || q.mi * BM + half * 64 < d.n_valid;   // same for every thread of the slab
      const uint32_t acc = tile_i & 1u, acc_ph = (tile_i >> 1) & 1u;
      if (!tc05::mbar_wait(&ctl->tmem_full[acc], acc_ph, abort_flag, WAIT_BUDGET_NS)) break;
      tc05::fence_after_sync();
      const uint32_t tacc = tmem + acc * (uint32_t)ACC_COLS + ((uint32_t)(q4 * 32) << 16);
      for (int p = 0; p < q.nb; ++p) {
        // the store out of this slab, the latest or (two pairs) the one before it, must have read it
        if (storer) { if (next_pair) tc05::bulk_wait_read<1>(); else tc05::bulk_wait_read<0>(); }
        tc05::named_bar_sync(1, 32 * kEpilogueWarps);
        if (slab_valid) {
          const int c_begin = p * d.split, c_end = c_begin + d.split;
#pragma unroll 1
          for (int g = (c_begin & ~31) + 32 * sub; g < c_end; g += 64) {
            uint32_t r[32];
            tc05::tmem_ld_32x32(tacc + (uint32_t)g, r);
            tc05::tmem_ld_wait();
            const int row0 = g - c_begin;              // slab row of element 0: a multiple of 8, negative for a first
            const uint32_t rbase = slab_base + slab_off + (uint32_t)(row0 * 128);     // group that starts in the previous block
            if (row0 >= 0 && row0 + 32 <= d.split) {
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                const float v = fmaxf(__uint_as_float(r[e]) + bias_v, floor_v);
                tc05::st_shared_bf16(rbase + cb[e & 7] + (uint32_t)(e * 128), v);
              }
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                const int row = row0 + e;
                if (row >= 0 && row < d.split) {
                  const float v = fmaxf(__uint_as_float(r[e]) + bias_v, floor_v);
                  tc05::st_shared_bf16(rbase + cb[e & 7] + (uint32_t)(e * 128), v);
                }
              }
            }
          }
        }
        tc05::fence_proxy_async_smem();
        tc05::named_bar_sync(1, 32 * kEpilogueWarps);
        if (storer && slab_valid) {
          // box (64 channels, PW, Rb, 1): columns past the image width, rows past its height and channels past
          // the extent are clipped by TMA
          tc05::tma_store_4d_addr(PAIR && half ? &tmC1 : &tmC, slab_base + slab_off, PAIR ? q.mi * CH : q.mi * BM + half * 64, 0,
                                  q.y0 + p * d.Rb, q.b);
          tc05::bulk_commit();
        }
        if (slab_valid) slab_off ^= next_pair;
      }
      tc05::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&ctl->tmem_empty[acc]);
    }
    if (storer) tc05::bulk_wait<0>();
  }

  tc05::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && ctl->abort_flag)
    geeps_report(d.status, GEEPS_ERR_TIMEOUT, KID_CONV_TC, (int)blockIdx.x, 1);
  if (warp == 1) {
    tc05::fence_after_sync();
    tc05::tmem_dealloc(tmem, 2 * ACC_COLS);
  }
}

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
bool make_map(CUtensorMap* map, const void* base, int rank, const long long* dims, const long long* strides_bytes,
              const int* box) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t gd[4], gs[3];
  cuuint32_t bx[4], es[4];
  for (int i = 0; i < rank; ++i) { gd[i] = (cuuint64_t)dims[i]; bx[i] = (cuuint32_t)box[i]; es[i] = 1; }
  for (int i = 0; i + 1 < rank; ++i) gs[i] = (cuuint64_t)strides_bytes[i];
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gd, gs, bx, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_act_map(CUtensorMap* map, const void* base, int ch, int W, int H, int B, long long pitch, int bw, int bh) {
  const long long dims[4] = {ch, W, H, B};
  const long long st[3] = {pitch * 2, pitch * 2 * W, pitch * 2 * W * H};
  const int box[4] = {64, bw, bh, 1};
  return make_map(map, base, 4, dims, st, box);
}
// the columns of parity b of an NHWC tensor
bool make_parity_map(CUtensorMap* map, const void* base, int ch, int W, int H, int B, long long pitch, int b, int bw, int bh) {
  const long long dims[4] = {ch, (W - b + 1) / 2, H, B};
  const long long st[3] = {pitch * 4, pitch * 2 * W, pitch * 2 * W * H};
  const int box[4] = {64, bw, bh, 1};
  return make_map(map, (const char*)base + pitch * 2 * b, 4, dims, st, box);
}
int round_up(long long v, int m) { return (int)((v + m - 1) / m * m); }

template <int MODE>
int launch(const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& tc, const CUtensorMap& tx1,
           const CUtensorMap& tc1, const HaloDev& d, int grid, size_t smem, cudaStream_t st) {
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(conv_halo_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  geeps_launch(conv_halo_kernel<MODE>, grid, kThreads, smem, st, tx, tw, tc, tx1, tc1, d);
  return (int)cudaGetLastError();
}

// geometry shared by the applicability check and the launch
struct HaloPlan { HaloDev d; size_t smem; double util, cost; bool ok; };      // cost: clocks of the steps on the busiest SM

// MODE_DGRAD2's weights: whole filter rows of KW panels of 64 channels, the taps of a row in descending order, so the 128
// rows of a step's weights are two neighbouring panels and each tap is loaded once for both columns.  (The panel in front of
// a row's last tap and the one behind its first belong to disabled lanes; at the ends they are a halo tile and a store slab.)
// At least five panels: a tap is loaded again some KW steps after its last use.
int pair_rows(int KW) { return (5 + KW - 1) / KW; }
int pair_slab(int positions) { return round_up(positions > 64 ? positions * 128LL : PANEL_BYTES, 1024); }

// a step of four 128 x n x 16 products takes 2 n clocks, but the tap's rows out of L2 and its issue some 520
int step_clocks(int n) { return 2 * n > 520 ? 2 * n : 520; }

// A second pair of store slabs instead of two weight stages: where a tile has few products its epilogue is the bound.  3 x 3
// forward, us with one pair and with two: 256 x 28 x 28, 8 -> 96 77.3, 74.9; 32 -> 128 29.2, 27.5; 256 x 27 x 27, 48 -> 128
// 41.8, 39.8.  One pair from a whole chunk or 5 x 5 taps on: 96 x 57 x 57, 64 -> 96 39.6, 41.3; 96 x 56 x 56, 96 -> 128 66.6,
// 69.3; 256 x 27 x 27, 48 -> 128, 5 x 5 59.2, 65.7; and in the data gradient, whose taps are loaded in two panels: 96 x 56 x
// 56, 16 channels of dY 62.6, 70.1.
bool two_slab_pairs(const GeepsConvTcParams* p, const HaloDev& d) {
  return p->mode == MODE_FWD && d.cchunks == 1 && d.k_last <= 3 && d.taps <= 9;
}

// pair: MODE_DGRAD2
HaloPlan plan_halo(const GeepsConvTcParams* p, bool pair = false) {
  HaloPlan hp;
  hp.ok = false;
  hp.smem = 0;
  hp.util = hp.cost = 0;
  HaloDev& d = hp.d;
  memset(&d, 0, sizeof(d));
  if ((p->mode != MODE_FWD && p->mode != MODE_DGRAD) || p->stride > 1) return hp;
  const bool fwd = p->mode == MODE_FWD;
  if (pair && (fwd || p->cg > 64 || p->W < 2 || p->OW < 2)) return hp;
  const int GW = fwd ? p->OW : (pair ? (p->W + 1) / 2 : p->W), GH = fwd ? p->OH : p->H;
  d.KH = p->KH; d.KW = p->KW; d.KWs = pair ? p->KW + 1 : p->KW; d.taps = p->KH * d.KWs;
  const int span = pair ? p->KW / 2 : p->KW - 1;       // columns that a window reaches past its first
  d.px = fwd ? p->pad : p->KW - 1 - p->pad;
  d.py = fwd ? p->pad : p->KH - 1 - p->pad;
  if (d.px < 0 || d.py < 0 || d.taps < 2) return hp;
  d.GH = GH;
  // Two store blocks of Rb image rows per tile, at most 128 positions each; the rows are spread evenly over the
  // tiles so that the last tile is not mostly padding.  The pitch is the smallest one >= out_width + KW - 1 that
  // makes a block a multiple of 8 positions (the epilogue's constant swizzle offsets rely on it).
  // MODE_DGRAD2 holds two halo tiles per stage, so its rows are also limited by shared memory, and of the pitches and rows
  // that fit the cheapest is taken.
  bool found = false;
  const int sms = geeps_sm_count();
  for (int pw = GW + span; pw <= GW + span + 7 && pw <= 128 && (pair || !found); ++pw) {
    for (int rb_max = 128 / pw; rb_max >= 1; --rb_max) {
      const int row_tiles = (GH + 2 * rb_max - 1) / (2 * rb_max);
      const int rb = (GH + 2 * row_tiles - 1) / (2 * row_tiles);
      if ((rb * pw) % 8 == 0) {
        const int ncols = round_up(2 * rb * pw, 16);
        const long long x_bytes = round_up(((2LL * rb + p->KH - 1) * pw + ncols - 2 * rb * pw + p->KW) * 128, 1024);
        const double cost = (double)(((long long)p->B * row_tiles + sms - 1) / sms) * step_clocks(ncols);
        const bool fits = !pair || 4 * x_bytes + (long long)pair_rows(p->KW) * p->KW * PANEL_BYTES +
                                       2 * pair_slab(rb * pw) <= SMEM_BUDGET;
        if (fits && (!found || cost < hp.cost)) {
          d.PW = pw; d.row_tiles = row_tiles; d.Rb = rb;
          hp.cost = cost;
          found = true;
        }
      }
      if (!pair) break;
    }
  }
  if (!found) return hp;
  d.split = d.Rb * d.PW;
  d.ncols2 = round_up(2 * d.split, 16);
  d.ncols1 = round_up(d.split, 16);
  const int kch = fwd ? p->cg : p->og, nch = fwd ? p->og : p->cg;
  d.cchunks = (kch + 63) / 64;
  const int tail = kch - (d.cchunks - 1) * 64;
  d.k_last = (tail + UMMA_K - 1) / UMMA_K;
  d.n_valid = nch;
  d.m_tiles = pair ? 1 : (nch + BM - 1) / BM;
  d.n_images = p->B;
  const int NR = 2 * d.Rb + p->KH - 1;
  const int over = d.ncols2 - 2 * d.split + p->KW;     // rows an MMA may read past the halo tile
  d.x_tile_bytes = round_up((long long)(NR * d.PW + over) * 128, 1024);
  d.x_stage_bytes = (pair ? 2 : 1) * d.x_tile_bytes;
  d.stages_x = 2;
  d.slab_bytes = pair ? pair_slab(d.split) : C_SLAB_BYTES;
  d.slab_pairs = 1;
  long long budget = SMEM_BUDGET - 2 * d.slab_bytes - (long long)d.stages_x * d.x_stage_bytes;
  if (pair) {
    int rows = pair_rows(p->KW);
    while ((rows + 1) * p->KW <= MAX_W_STAGES && (long long)(rows + 1) * p->KW * PANEL_BYTES <= budget) ++rows;
    d.stages_w = rows * p->KW;
    d.w_bytes = d.stages_w * PANEL_BYTES;
    if (d.stages_w > MAX_W_STAGES || d.w_bytes > budget) return hp;
  } else {
    if (two_slab_pairs(p, d) && budget >= 2 * d.slab_bytes + 3LL * W_STAGE_BYTES) {
      d.slab_pairs = 2;
      budget -= 2 * d.slab_bytes;
    }
    d.stages_w = (int)(budget / W_STAGE_BYTES);
    if (d.stages_w > MAX_W_STAGES / 2) d.stages_w = MAX_W_STAGES / 2;
    if (d.stages_w < 3) return hp;
    d.w_bytes = d.stages_w * W_STAGE_BYTES;
  }
  hp.smem = (size_t)d.stages_x * d.x_stage_bytes + d.w_bytes + 2 * d.slab_pairs * d.slab_bytes + sizeof(SmemCtl) + 1024;
  hp.cost *= (double)d.m_tiles * d.taps * d.cchunks;
  // share of the issued MMA work that lands in real outputs: positions x channels
  const double pos = (double)GH * GW / ((double)d.row_tiles * d.ncols2);
  const double chn = (double)nch / ((double)d.m_tiles * (pair ? 64 : BM)) * d.KW / d.KWs;
  hp.util = pos * chn;
  hp.ok = true;
  return hp;
}

// A data gradient with few channels goes by column pairs where the steps of its busiest SM then take fewer clocks.  Measured
// (us, MODE_DGRAD and pairs): 64 x 28 x 28, 96 -> 64, 3 x 3: 18.4, 15.4; 300 x 14 x 14, 64 -> 32, 5 x 5: 52.2, 35.8; 128 x 20
// x 20, 96 -> 48, 5 x 5: 32.8, 26.6; 64 x 27 x 27, 40 -> 48, 5 x 5: 24.6, 17.4; 256 x 28 x 28, 384 -> 64, 3 x 3: 120, 102.
// Tiles of few rows look cheap by columns alone and are not: a step's weights take some 520 clocks (conv2 in tiles of two
// image rows: 470 us).  Through conv_tc() only 64 channels or 5 x 5 taps and more come here; the rule for those is older than
// the pairs, and fewer channels at 3 x 3 or 4 x 4 are on the box kernel.
bool takes_pairs(const HaloPlan& plain, const HaloPlan& pairs) {
  return plain.ok && pairs.ok && pairs.cost < plain.cost;
}

int halo_mode() {
  static int m = -1;
  if (m < 0) { const char* e = getenv("GEEPS_HALO_CONV"); m = e ? atoi(e) : 1; }
  return m;
}

}  // namespace

extern "C" {

// 1 when conv_tc() should route this call here.  The activations must be re-read often enough by the box kernel (>= 9 taps).
//
// Activations whose rows are whole 128-byte lines (64 channels): the 128-channel row blocks must be mostly real channels, and
// there must be two tiles an SM (a layer of one channel block still wins from 1.7: AlexNet conv5 per group, 256 tiles); a
// 5 x 5 data gradient, which the box kernel runs with narrow products, always comes here.  Fitted to AlexNet and Inception layers.
//
// Other rows straddle lines, and the box kernel fetches them once per tap, this one once per chunk.  There, in the data gradient
// and in a forward pass of one chunk, the expected times decide, each a fit to measured ones (geeps_conv_box_us says how; here half of the fits lie within 5 % of the measurement):
// launch + waves * (tile + chunks * (its activations + taps * step)), and within a tenth of one another, or below the 32
// channels that the fits know, the rule above.  us, halo / box: data gradient 48 x 48, 288 -> 360 at batch 48 204 / 317, 40 x 40,
// 280 -> 120 at batch 81 110 / 162; forward 48 x 48, 56 -> 272, 5 x 5 at batch 25 63 / 105, but 29 x 29, 56 -> 32 at batch 26
// 11.4 / 9.9 (a block of 32 real rows is better than its fit).
// The rule for whole lines loses up to a fifth too (13 x 13, 256 -> 384 at batch 256, data gradient: 70 / 59) and stays, as it does
// for a forward pass of several chunks (27 x 27, 136 -> 80, 5 x 5 at batch 30 29.5 / 60): the kernels add their terms in different
// orders (taps of a chunk, chunks of a tap; one chunk gives the same bits).  In a deep network with near-ties in its pooling
// windows another order changes which element a later step's maximum picks, and behind a ReLU whether an output next to zero
// is one, and with it the gradients under it.
int geeps_conv_halo_applicable(const GeepsConvTcParams* p) {
  if (!halo_mode()) return 0;
  if (!geeps_conv_tc_supported(p)) return 0;
  const HaloPlan hp = plan_halo(p);
  if (!hp.ok || hp.d.taps < 9) return 0;
  const HaloDev& d = hp.d;
  const bool fwd = p->mode == MODE_FWD;
  const double pos = (double)d.GH * (fwd ? p->OW : p->W) / ((double)d.row_tiles * d.ncols2);
  if (pos < 0.6) return 0;
  const int sms = geeps_sm_count();
  const long long tiles = (long long)d.m_tiles * d.n_images * d.row_tiles;
  const double chn = (double)d.n_valid / ((double)d.m_tiles * BM);
  const bool shares = tiles * 10 >= (d.m_tiles == 1 ? 17LL : 20LL) * sms &&
                      (fwd ? (d.m_tiles == 1 && d.n_valid >= 96) || (chn >= 0.85 && pos >= 0.8)
                           : d.taps >= 25 || (d.n_valid >= 64 && (d.n_valid <= 128 || chn >= 0.85)));
  const bool lines = (fwd ? p->x_pitch : p->y_pitch) % 64 == 0 && (fwd ? p->cg : p->og) % 64 == 0;
  if (lines || (fwd && d.cchunks > 1) || p->cg < 32 || p->og < 32) return shares ? 1 : 0;
  const double waves = (double)((tiles + sms - 1) / sms), cols = d.ncols2 / 100.0;
  const double us = fwd ? 4.28 + waves * (1.44 + 0.364 * cols + d.cchunks * (0.035 * cols + d.taps * (0.214 + 0.023 * cols)))
                        : 5.14 + waves * (0.65 + 0.107 * cols + d.cchunks * (0.142 * cols + d.taps * (0.214 + 0.025 * cols)));
  // (column pairs make a 5 x 5 data gradient of few channels better than its fit: 14 x 14, 40 -> 184 at batch 181 65 / 77)
  return us < (shares ? (d.taps >= 25 ? 1.25 : 1.11) : d.n_valid > 32 ? 0.9 : 0.75) * geeps_conv_box_us(p) ? 1 : 0;
}

static int fill_plan(const HaloPlan& hp, int routed, GeepsHaloPlanInfo* out) {
  if (!hp.ok) return 0;
  const HaloDev& d = hp.d;
  out->ok = 1;
  out->routed = routed;
  out->PW = d.PW; out->R = d.Rb; out->row_tiles = d.row_tiles; out->m_tiles = d.m_tiles;
  out->positions = d.split; out->ncols2 = d.ncols2; out->ncols1 = d.ncols1;
  out->stages_x = d.stages_x; out->stages_w = d.stages_w; out->x_stage_bytes = d.x_stage_bytes;
  out->tmem_cols = 2 * ACC_COLS;
  out->smem_bytes = (long long)hp.smem;
  out->util = hp.util;
  return 1;
}
int geeps_conv_halo_plan(const GeepsConvTcParams* p, GeepsHaloPlanInfo* out) {
  memset(out, 0, sizeof(*out));
  if (!geeps_conv_tc_supported(p)) return 0;
  return fill_plan(plan_halo(p), geeps_conv_halo_applicable(p), out);
}
int geeps_conv_halo_pair_plan(const GeepsConvTcParams* p, GeepsHaloPlanInfo* out) {
  memset(out, 0, sizeof(*out));
  if (!geeps_conv_tc_supported(p)) return 0;
  const HaloPlan pairs = plan_halo(p, true);
  return fill_plan(pairs, geeps_conv_halo_applicable(p) && takes_pairs(plan_halo(p), pairs), out);
}

int geeps_conv_halo(const GeepsConvTcParams* p, void* stream) {
  if (!geeps_conv_tc_supported(p)) return (int)cudaErrorInvalidValue;
  HaloPlan hp = plan_halo(p);
  if (!hp.ok) return (int)cudaErrorInvalidValue;
  const HaloPlan pairs = plan_halo(p, true);
  const bool pair = p->columns == 0 ? takes_pairs(hp, pairs) : p->columns == 2;
  if (pair && !pairs.ok) return (int)cudaErrorInvalidValue;
  if (pair) hp = pairs;
  HaloDev& d = hp.d;
  const bool fwd = p->mode == MODE_FWD;
  d.bias = fwd ? p->bias : nullptr;
  d.status = p->status;
  d.relu = fwd ? p->relu : 0;
  const int NR = 2 * d.Rb + p->KH - 1;
  CUtensorMap tx, tw, tc, tx1, tc1;
  bool ok;
  const long long wdims[3] = {p->cg, d.KH * d.KW, p->og};
  const long long wst[2] = {(long long)p->cg * 2, p->ldw * 2};
  if (fwd) {
    ok = make_act_map(&tx, p->x, p->cg, p->W, p->H, p->B, p->x_pitch, d.PW, NR);
    const int wbox[3] = {64, 1, BM};
    ok = ok && make_map(&tw, p->w, 3, wdims, wst, wbox);
    ok = ok && make_act_map(&tc, p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, d.PW, d.Rb);
  } else {
    const int wbox[3] = {64, 1, 64};
    ok = make_map(&tw, p->w, 3, wdims, wst, wbox);
    if (pair) {
      // padded column 2 c + h is image column 2 c + h - px: column x0 (x1) + c of the image's columns of parity b
      const int b0 = d.px & 1, b1 = (d.px + 1) & 1;
      d.x0 = (-d.px - b0) / 2;
      d.x1 = (1 - d.px - b1) / 2;
      ok = ok && make_parity_map(&tx, p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, b0, d.PW, NR) &&
           make_parity_map(&tx1, p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, b1, d.PW, NR) &&
           make_parity_map(&tc, p->x, p->cg, p->W, p->H, p->B, p->x_pitch, 0, d.PW, d.Rb) &&
           make_parity_map(&tc1, p->x, p->cg, p->W, p->H, p->B, p->x_pitch, 1, d.PW, d.Rb);
    } else {
      ok = ok && make_act_map(&tx, p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, d.PW, NR) &&
           make_act_map(&tc, p->x, p->cg, p->W, p->H, p->B, p->x_pitch, d.PW, d.Rb);
    }
  }
  if (!pair) { tx1 = tx; tc1 = tc; }      // unused by the kernel
  if (!ok) return (int)cudaErrorInvalidValue;
  const long long num_tiles = (long long)d.m_tiles * d.n_images * d.row_tiles;
  const int sms = geeps_sm_count();
  const int grid = (int)(num_tiles < sms ? num_tiles : sms);
  if (fwd) return launch<MODE_FWD>(tx, tw, tc, tx1, tc1, d, grid, hp.smem, (cudaStream_t)stream);
  if (pair) return launch<MODE_DGRAD2>(tx, tw, tc, tx1, tc1, d, grid, hp.smem, (cudaStream_t)stream);
  return launch<MODE_DGRAD>(tx, tw, tc, tx1, tc1, d, grid, hp.smem, (cudaStream_t)stream);
}

}  // extern "C"
