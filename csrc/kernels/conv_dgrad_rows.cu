// Data gradient of a stride-1 convolution with few input channels per group, one filter ROW per MMA.
//
//     dX[m, ci] = sum over (ty, tx, co) of  dY[m + ty * PW + tx, co] * W[co, KH-1-ty, KW-1-tx, ci]
//
// with the positions of the zero-padded image flattened at pitch PW, as in conv_halo.cu.  A layer such as AlexNet's conv2
// has 48 input channels per group: as the rows of an MMA (conv_halo.cu) they fill 48 of 128, as its columns (conv_tc.cu)
// 48 of 256, and either way the tensor cores spend two thirds of their time on padding.  The weight matrix stores the taps
// of a filter row next to one another, so the columns here are (tap of the row, input channel) - 5 x 48 = 240 of 256:
//
//     D[p, (tx, ci)] = sum over (ty, co) of dY[p + ty * PW, co] * W[co, KH-1-ty, KW-1-tx, ci]
//     dX[m, ci]      = sum over tx of       D[m + tx, (tx, ci)]
//
// The first line is KH * co / 64 k-steps of 128 x 256 x 64 whose activation operand is one halo tile in shared memory read
// from row ty * PW on; the second is the epilogue's: a position is a TMEM lane, so a sum over tx moves one lane per tap,
// KW - 1 warp shuffles per channel.  PW is 16 or 32, so that the KW - 1 columns an image row is padded by are in the warp
// of that row and no window crosses a warp.
//
// A tile is two blocks of 128 positions that share every weight stage (32 KB per k-step: for one block alone the weights
// would have to arrive at 64 bytes per clock and SM, which L2 does not deliver); their accumulators fill TMEM, and two
// groups of four epilogue warps drain them side by side.  Tiles of one block (odd block counts) come last.
// One group of conv2 (256 x 27 x 27, 128 -> 48 channels, 5 x 5): 120 us in conv_halo.cu (25,600 tensor cycles per 256
// positions), 63.5 here (10,240); bound by the operands' way from L2 (41 bytes per clock and SM at full tensor rate) and by
// the part of the epilogue that no other tile's MMAs cover.
//
// conv_tc() routes a data-gradient call here when geeps_conv_dgrad_rows_applicable() says so; GEEPS_HALO_CONV=0 keeps every
// call on the box kernel.  Roles and bounded waits as in conv_halo.cu.
#include <cuda.h>
#include <mutex>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "kernels.h"
#include "tc05.cuh"

namespace {

constexpr int BM = 128;                       // positions per block (TMEM lanes)
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int PANEL_BYTES = 64 * BK * 2;      // weights: 64 output channels (k) x 64 columns
constexpr int MAX_X_STAGES = 2;
constexpr int MAX_W_STAGES = 4;
constexpr uint64_t WAIT_BUDGET_NS = 2000000000ull;
constexpr int C_SLAB_BYTES = BM * 128;        // 128 positions x 64 channels bf16, one per block
constexpr int ACC_COLS = 256;
constexpr int kThreads = 64 + 2 * 128;        // producer, issuer, four epilogue warps per block

struct RowsDev {
  int* status;
  int KH, KW, cchunks, k_last;         // k_last: MMA k-substeps (of 16) in the last chunk of output channels
  int PW, R, px, py, GH;               // pitch, image rows per block, halo left / top, image rows
  int pairs, single, n_images;         // per image: tiles of two blocks, and whether one block is left over
  int cg, n_cols;                      // channels produced; KW * cg rounded up to whole 64-column panels
  int x_stage_bytes, w_stage_bytes, stages_x, stages_w;
};

struct SmemCtl {
  uint64_t full_x[MAX_X_STAGES], empty_x[MAX_X_STAGES];
  uint64_t full_w[MAX_W_STAGES], empty_w[MAX_W_STAGES];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

struct Tile { int b, y0, nb; };
__device__ __forceinline__ Tile decode_tile(const RowsDev& d, int t) {
  Tile q;
  const int n_pairs = d.pairs * d.n_images;
  if (t < n_pairs) {
    q.b = t / d.pairs;
    q.y0 = (t - q.b * d.pairs) * 2 * d.R;
    q.nb = 2;
  } else {
    q.b = t - n_pairs;
    q.y0 = d.pairs * 2 * d.R;
    q.nb = 1;
  }
  return q;
}

// tmX: dY as (co, w, h, b) with box (64, PW, 2 R + KH - 1, 1); tmW: weights as (tap * cg + ci, co) with box (64, 64), one
// MN-major panel; tmC: dX with box (64, PW, R, 1).
__global__ void __launch_bounds__(kThreads, 1)
conv_dgrad_rows_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                       const __grid_constant__ CUtensorMap tmC, const RowsDev d) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles_x = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles_w = tiles_x + (size_t)d.stages_x * d.x_stage_bytes;
  uint8_t* cslab = tiles_w + (size_t)d.stages_w * d.w_stage_bytes;
  SmemCtl* ctl = (SmemCtl*)(cslab + 2 * C_SLAB_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_tiles = d.n_images * (d.pairs + d.single);

  if (threadIdx.x == 0) {
    for (int s = 0; s < d.stages_x; ++s) { tc05::mbar_init(&ctl->full_x[s], 1); tc05::mbar_init(&ctl->empty_x[s], 1); }
    for (int s = 0; s < d.stages_w; ++s) { tc05::mbar_init(&ctl->full_w[s], 1); tc05::mbar_init(&ctl->empty_w[s], 1); }
    for (int a = 0; a < 2; ++a) { tc05::mbar_init(&ctl->tmem_full[a], 1); tc05::mbar_init(&ctl->tmem_empty[a], 4); }
    ctl->abort_flag = 0;
    tc05::mbar_fence_init();
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

  if (warp == 0) {
    // ---------------- TMA producer: one halo tile per chunk, one filter row of weights per k-step ----------------
    const bool leader = tc05::elect_one();
    if (leader) { tc05::tma_prefetch_desc(&tmX); tc05::tma_prefetch_desc(&tmW); }
    const int panels = d.n_cols / 64, row_cols = d.KW * d.cg;
    int sx = 0, sw = 0;
    uint32_t phx = 0, phw = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const Tile q = decode_tile(d, t);
      for (int cc = 0; cc < d.cchunks && ok; ++cc) {
        if (!tc05::mbar_wait_warp(&ctl->empty_x[sx], phx ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
        if (leader) {
          tc05::mbar_expect_tx(&ctl->full_x[sx], (uint32_t)d.x_stage_bytes);
          tc05::tma_load_4d(tiles_x + (size_t)sx * d.x_stage_bytes, &tmX, &ctl->full_x[sx], cc * 64, -d.px, q.y0 - d.py, q.b);
        }
        if (++sx == d.stages_x) { sx = 0; phx ^= 1u; }
        for (int ty = 0; ty < d.KH; ++ty) {
          if (!tc05::mbar_wait_warp(&ctl->empty_w[sw], phw ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          if (leader) {
            uint8_t* dst = tiles_w + (size_t)sw * d.w_stage_bytes;
            const int col = (d.KH - 1 - ty) * row_cols;             // the filter is applied mirrored
            tc05::mbar_expect_tx(&ctl->full_w[sw], (uint32_t)d.w_stage_bytes);
            for (int h = 0; h < panels; ++h)
              tc05::tma_load_2d(dst + h * PANEL_BYTES, &tmW, &ctl->full_w[sw], col + 64 * h, cc * 64);
          }
          if (++sw == d.stages_w) { sw = 0; phw ^= 1u; }
        }
      }
    }
    geeps_pdl_trigger();       // every operand is on its way: the rest of this CTA is its last products and stores
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const bool leader = tc05::elect_one();
    const uint32_t idesc = tc05::make_idesc_bf16(BM, d.n_cols, 0, 1);
    constexpr uint32_t d_hi = tc05::desc_hi(1024);
    const uint32_t row_units = (uint32_t)d.PW * 8u;                // descriptor units (16 bytes) per image row
    const uint32_t block_units = (uint32_t)d.R * row_units;
    uint32_t ph_acc0 = 0, ph_acc1 = 0;                             // uses of each accumulator so far, mod 2
    int sx = 0, sw = 0;
    uint32_t phx = 0, phw = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const int nb = decode_tile(d, t).nb;
      uint32_t accumulate = 0;                                     // the very first MMA of a block overwrites
      for (int cc = 0; cc < d.cchunks && ok; ++cc) {
        if (!tc05::mbar_wait_warp(&ctl->full_x[sx], phx, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
        uint32_t x_lo = tc05::desc_lo(tc05::smem_u32(tiles_x + (size_t)sx * d.x_stage_bytes), 16);
        const int ksteps = cc + 1 < d.cchunks ? BK / UMMA_K : d.k_last;
        for (int ty = 0; ty < d.KH; ++ty) {
          const bool first = cc == 0 && ty == 0, last = cc + 1 == d.cchunks && ty + 1 == d.KH;
          if (!tc05::mbar_wait_warp(&ctl->full_w[sw], phw, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          // the epilogue must have drained an accumulator before its first MMA
          if (first && !tc05::mbar_wait_warp(&ctl->tmem_empty[0], ph_acc0 ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
          tc05::fence_after_sync();
          const uint32_t w_lo = tc05::desc_lo(tc05::smem_u32(tiles_w + (size_t)sw * d.w_stage_bytes), PANEL_BYTES);
          if (leader) {
            for (int k = 0; k < ksteps; ++k)
              tc05::mma_bf16_ss_lohi(tmem, x_lo + 2 * k, d_hi, w_lo + 128 * k, d_hi, idesc, k ? 1u : accumulate);
            if (last) tc05::mma_commit(&ctl->tmem_full[0]);
          }
          if (nb == 2) {
            if (first && !tc05::mbar_wait_warp(&ctl->tmem_empty[1], ph_acc1 ^ 1u, abort_flag, WAIT_BUDGET_NS)) { ok = false; break; }
            tc05::fence_after_sync();
            if (leader) {
              for (int k = 0; k < ksteps; ++k)
                tc05::mma_bf16_ss_lohi(tmem + ACC_COLS, x_lo + block_units + 2 * k, d_hi, w_lo + 128 * k, d_hi, idesc,
                                       k ? 1u : accumulate);
              if (last) tc05::mma_commit(&ctl->tmem_full[1]);
            }
          }
          if (leader) tc05::mma_commit(&ctl->empty_w[sw]);
          accumulate = 1u;
          x_lo += row_units;
          if (++sw == d.stages_w) { sw = 0; phw ^= 1u; }
        }
        if (ok && leader) tc05::mma_commit(&ctl->empty_x[sx]);
        if (++sx == d.stages_x) { sx = 0; phx ^= 1u; }
      }
      ph_acc0 ^= 1u;
      if (nb == 2) ph_acc1 ^= 1u;
    }
  } else {
    // ---------------- epilogue: sum over the row's taps by lane shifts -> bf16 slab -> TMA store ----------------
    const int q4 = warp & 3;                       // TMEM lane quarter this warp may access
    const int g = (warp - 2) >> 2;                 // block of the tile
    const bool issuer = q4 == 2 && lane == 0;      // (warps 2 and 6)
    const int row = q4 * 32 + lane;
    uint8_t* slab = cslab + (size_t)g * C_SLAB_BYTES + (size_t)row * 128;
    const uint32_t rsw = (uint32_t)(row & 7);
    const uint32_t tacc = tmem + (uint32_t)(g * ACC_COLS) + ((uint32_t)(q4 * 32) << 16);
    uint32_t ph = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const Tile q = decode_tile(d, t);
      if (g >= q.nb) continue;
      if (!tc05::mbar_wait(&ctl->tmem_full[g], ph, abort_flag, WAIT_BUDGET_NS)) break;
      ph ^= 1u;
      tc05::fence_after_sync();
      if (issuer) tc05::bulk_wait_read<0>();       // the last store out of this slab has read it
      tc05::named_bar_sync(1 + g, 128);
#pragma unroll 1
      for (int c = 0; c < d.cg; c += 16) {
        // columns of tap kw of the row: kw * cg + channel; kw = KW - 1 - tx, and what tap tx adds to position m lies tx
        // lanes further on.  The last lanes take in values of the next image row, into columns that the store clips.
        float a[16];
#pragma unroll 1
        for (int kw = 0; kw < d.KW; ++kw) {
          uint32_t r[16];
          tc05::tmem_ld_32x16(tacc + (uint32_t)(kw * d.cg + c), r);
          tc05::tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float v = __uint_as_float(r[e]);
            a[e] = kw ? __shfl_down_sync(0xffffffffu, a[e], 1) + v : v;
          }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
          *reinterpret_cast<uint4*>(slab + (((uint32_t)(c >> 3) + j) ^ rsw) * 16u) =
              make_uint4(pack_bf16x2(a[8 * j], a[8 * j + 1]), pack_bf16x2(a[8 * j + 2], a[8 * j + 3]),
                         pack_bf16x2(a[8 * j + 4], a[8 * j + 5]), pack_bf16x2(a[8 * j + 6], a[8 * j + 7]));
      }
      tc05::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&ctl->tmem_empty[g]);
      tc05::fence_proxy_async_smem();
      tc05::named_bar_sync(1 + g, 128);
      if (issuer) {
        // box (64 channels, PW, R, 1): columns past the image, rows past its height and channels past cg are clipped
        tc05::tma_store_4d(&tmC, cslab + (size_t)g * C_SLAB_BYTES, 0, 0, q.y0 + g * d.R, q.b);
        tc05::bulk_commit();
      }
    }
    if (issuer) tc05::bulk_wait<0>();
  }

  tc05::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && ctl->abort_flag)
    geeps_report(d.status, GEEPS_ERR_TIMEOUT, KID_CONV_TC, (int)blockIdx.x, 3);
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

struct RowsPlan { RowsDev d; size_t smem; double util; bool ok; };

RowsPlan plan_rows(const GeepsConvTcParams* p) {
  RowsPlan rp;
  rp.ok = false;
  rp.smem = 0;
  rp.util = 0;
  RowsDev& d = rp.d;
  memset(&d, 0, sizeof(d));
  if (p->mode != 1 || p->stride > 1 || p->KW < 2 || p->KW > 7 || p->KH < 2 || p->KH > 7) return rp;
  d.KH = p->KH; d.KW = p->KW; d.cg = p->cg; d.GH = p->H;
  d.px = p->KW - 1 - p->pad; d.py = p->KH - 1 - p->pad;
  if (d.px < 0 || d.py < 0) return rp;
  d.n_cols = (p->KW * p->cg + 63) / 64 * 64;
  // one slab of channels, in whole groups of 16 (the epilogue's TMEM loads); one accumulator of columns
  if (p->cg > 64 || p->cg % 16 || d.n_cols > ACC_COLS) return rp;
  d.PW = p->W + p->KW - 1 <= 16 ? 16 : 32;
  if (p->W + p->KW - 1 > d.PW) return rp;
  d.R = BM / d.PW;
  const int blocks = (p->H + d.R - 1) / d.R;
  d.pairs = blocks / 2; d.single = blocks & 1; d.n_images = p->B;
  d.cchunks = (p->og + BK - 1) / BK;
  d.k_last = (p->og - (d.cchunks - 1) * BK + UMMA_K - 1) / UMMA_K;
  d.x_stage_bytes = (2 * d.R + p->KH - 1) * d.PW * 128;    // a multiple of 2048
  d.w_stage_bytes = d.n_cols / 64 * PANEL_BYTES;
  d.stages_x = MAX_X_STAGES;
  d.stages_w = (int)((224 * 1024 - 2 * C_SLAB_BYTES - (long long)d.stages_x * d.x_stage_bytes) / d.w_stage_bytes);
  if (d.stages_w > MAX_W_STAGES) d.stages_w = MAX_W_STAGES;
  if (d.stages_w < 2) return rp;
  rp.smem = (size_t)d.stages_x * d.x_stage_bytes + (size_t)d.stages_w * d.w_stage_bytes + 2 * C_SLAB_BYTES + sizeof(SmemCtl) + 1024;
  // share of the issued MMA work that lands in real gradients: positions x columns
  rp.util = (double)p->H * p->W / ((double)blocks * BM) * (p->KW * p->cg) / d.n_cols;
  rp.ok = true;
  return rp;
}

int halo_mode() {
  static int m = -1;
  if (m < 0) { const char* e = getenv("GEEPS_HALO_CONV"); m = e ? atoi(e) : 1; }
  return m;
}

}  // namespace

extern "C" {

// 1 when conv_tc() should route this data gradient here: wherever the shape fits.  us, L2 evicted, other kernels -> here:
// 256 x 27 x 27 x 48, 5 x 5: 120 -> 63.5; 16 images of it: 18.4 -> 13.8; 100 x 28 x 28 x 32, 5 x 5: 54 -> 27;
// 32 x 28 x 28 x 64, 3 x 3: 14.8 -> 10.2; 128 x 20 x 20 x 48, 5 x 5: 34.8 -> 26.6; 256 x 10 x 10 x 64, 3 x 3: 12.8 -> 11.7.
int geeps_conv_dgrad_rows_applicable(const GeepsConvTcParams* p) {
  if (!halo_mode()) return 0;
  if (!geeps_conv_tc_supported(p)) return 0;
  return plan_rows(p).ok ? 1 : 0;
}

int geeps_conv_dgrad_rows_plan(const GeepsConvTcParams* p, GeepsHaloPlanInfo* out) {
  memset(out, 0, sizeof(*out));
  if (!geeps_conv_tc_supported(p)) return 0;
  const RowsPlan rp = plan_rows(p);
  if (!rp.ok) return 0;
  const RowsDev& d = rp.d;
  out->ok = 1;
  out->routed = geeps_conv_dgrad_rows_applicable(p);
  out->PW = d.PW; out->R = d.R; out->row_tiles = d.pairs + d.single; out->m_tiles = 1;
  out->positions = BM; out->ncols2 = out->ncols1 = d.n_cols;
  out->n_blocks = 2 * d.pairs + d.single;
  out->stages_x = d.stages_x; out->stages_w = d.stages_w; out->x_stage_bytes = d.x_stage_bytes;
  out->tmem_cols = 2 * ACC_COLS;
  out->smem_bytes = (long long)rp.smem;
  out->util = rp.util;
  return 1;
}

int geeps_conv_dgrad_rows(const GeepsConvTcParams* p, void* stream) {
  if (!geeps_conv_tc_supported(p)) return (int)cudaErrorInvalidValue;
  RowsPlan rp = plan_rows(p);
  if (!rp.ok) return (int)cudaErrorInvalidValue;
  RowsDev& d = rp.d;
  d.status = p->status;
  CUtensorMap tx, tw, tc;
  bool ok = make_act_map(&tx, p->y, p->og, p->OW, p->OH, p->B, p->y_pitch, d.PW, 2 * d.R + d.KH - 1);
  const long long wdims[2] = {(long long)d.KH * d.KW * p->cg, p->og};
  const long long wst[1] = {p->ldw * 2};
  const int wbox[2] = {64, BK};
  ok = ok && make_map(&tw, p->w, 2, wdims, wst, wbox);
  ok = ok && make_act_map(&tc, p->x, p->cg, p->W, p->H, p->B, p->x_pitch, d.PW, d.R);
  if (!ok) return (int)cudaErrorInvalidValue;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(conv_dgrad_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const long long num_tiles = (long long)d.n_images * (d.pairs + d.single);
  const int sms = geeps_sm_count();
  const int grid = (int)(num_tiles < sms ? num_tiles : sms);
  geeps_launch(conv_dgrad_rows_kernel, grid, kThreads, rp.smem, (cudaStream_t)stream, tx, tw, tc, d);
  return (int)cudaGetLastError();
}

}  // extern "C"
