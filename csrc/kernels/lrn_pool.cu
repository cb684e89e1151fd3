// Local response normalisation across channels fused with the max pooling that follows it (AlexNet pairs
// them after conv1 and conv2), forward and backward, on NHWC bf16 activations.
//
// Unfused, the pair moves the full-resolution tensor five times per direction: LRN forward writes y and
// 1/scale, pooling reads y; pooling backward writes the full-resolution gradient, LRN backward reads it together
// with x, y and 1/scale.  Here the normalised tensor and its gradient never reach global memory:
//
//   forward   one CTA per output row: the K input rows go to shared memory, LRN is evaluated there once per
//             element, the pooled row and the window codes leave.          traffic: x in, pooled + codes out
//   backward  one CTA per block of input rows: x rows, the covering pooled-gradient rows and their codes go to
//             shared memory; the pooling gradient, scale = k + alpha/n * window sum of x^2, scale^-beta and the
//             cross-channel term are recomputed from them; dx leaves with the ReLU mask of the producing
//             convolution applied and its per-channel sums (that convolution's bias gradient) accumulated.
//                                                                          traffic: x, pooled gradient, codes in, dx out
//
// Nothing of the forward pass is kept for the backward pass except the window codes (one byte per pooled
// element).  The reference has no layer kernels of its own (they lived in its Caffe application).
#include <math.h>
#include <stdlib.h>

#include "common.cuh"
#include "kernels.h"
#include "nn_ops.h"

namespace {

typedef __nv_bfloat16 bf16;

// ---- arithmetic of the normalisation ----
// scale = k + alpha/n * w = k * (1 + eps), w = window sum of x^2, eps = alpha / (n k) * w.  The two powers the
// kernels need are scale^-beta = k^-beta (1+eps)^-beta and scale^-(beta+1).  For eps <= kPolyEps both are
// evaluated as cubic Taylor polynomials, written directly in w (the coefficients carry the powers of alpha/(n k)),
// with a relative error below 4e-4 at the bound - far below the bf16 rounding of the results; only a vector with a
// larger eps takes the special-function path.  These kernels are bound by instruction issue, not by memory: the
// special-function unit runs at a quarter of the FMA rate and every avoided instruction per element counts.
constexpr float kPolyEps = 0.1f;
struct LrnCoef {
  float w_max;              // window sums up to this take the polynomial
  float p0, p1, p2, p3;     // scale^-beta     ~ p0 + w (p1 + w (p2 + w p3))
  float q0, q1, q2, q3;     // scale^-(beta+1) ~ q0 + w (q1 + w (q2 + w q3))
  float es, beta, k;        // exact path: scale = k * (1 + es * w)
};
__device__ __forceinline__ float max8(const float (&w)[8]) {
  return fmaxf(fmaxf(fmaxf(w[0], w[1]), fmaxf(w[2], w[3])), fmaxf(fmaxf(w[4], w[5]), fmaxf(w[6], w[7])));
}

__device__ __forceinline__ float max4(const float2 (&w)[4]) {
  return fmaxf(fmaxf(fmaxf(w[0].x, w[0].y), fmaxf(w[1].x, w[1].y)), fmaxf(fmaxf(w[2].x, w[2].y), fmaxf(w[3].x, w[3].y)));
}
// NaN where a window is
__device__ __forceinline__ float max4_nan(const float2 (&w)[4]) {
  auto larger = [](float a, float b) {
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(a) : "f"(b));
    return a;
  };
  return larger(larger(larger(w[0].x, w[0].y), larger(w[1].x, w[1].y)), larger(larger(w[2].x, w[2].y), larger(w[3].x, w[3].y)));
}
// The sum of all twelve squares under the windows of eight channels (w: windows of 5, edge: the last two squares), two
// additions away, bounds every window; only where it is too large for the polynomials does the largest have to be found.
__device__ __forceinline__ float squares12(const float2 (&w)[4], float2 edge) { return (w[0].x + w[2].y) + (edge.x + edge.y); }

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// The channels [c-4, c+12) of one pixel as floats (zero outside [0, C)): one 16-byte and two 8-byte loads.
// Works on global and shared pointers alike; c is a multiple of 8.
__device__ __forceinline__ void load16(const bf16* px, int c, int C, float (&v)[16]) {
  uint2 lo = make_uint2(0u, 0u), hi = make_uint2(0u, 0u);
  if (c > 0) lo = *reinterpret_cast<const uint2*>(px + c - 4);
  const uint4 mid = *reinterpret_cast<const uint4*>(px + c);
  if (c + 8 < C) hi = *reinterpret_cast<const uint2*>(px + c + 8);
  v[0] = bf_lo(lo.x); v[1] = bf_hi(lo.x); v[2] = bf_lo(lo.y); v[3] = bf_hi(lo.y);
  v[4] = bf_lo(mid.x); v[5] = bf_hi(mid.x); v[6] = bf_lo(mid.y); v[7] = bf_hi(mid.y);
  v[8] = bf_lo(mid.z); v[9] = bf_hi(mid.z); v[10] = bf_lo(mid.w); v[11] = bf_hi(mid.w);
  v[12] = bf_lo(hi.x); v[13] = bf_hi(hi.x); v[14] = bf_lo(hi.y); v[15] = bf_hi(hi.y);
}
// window sums of 2*HALF+1 consecutive entries around index 4+e, e = 0..7 (sliding)
template <int HALF>
__device__ __forceinline__ void window8(const float (&t)[16], float (&w)[8]) {
  float acc = 0.f;
#pragma unroll
  for (int j = 4 - HALF; j <= 4 + HALF; ++j) acc += t[j];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    w[e] = acc;
    if (e < 7) acc += t[4 + e + HALF + 1] - t[4 + e - HALF];
  }
}
__device__ __forceinline__ uint4 pack8(const float (&o)[8]) {
  return make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
}

// Walks the items (row, pixel, channel vector) of a [rows][W][cv] block in row-major order, `nt` items at a time,
// without a division per item.
struct ItemWalk {
  int r, w, cvi, dq, dc;
  __device__ __forceinline__ ItemWalk(int first, int nt, int W, int cv) {
    cvi = first % cv;
    const int t = first / cv;
    w = t % W;
    r = t / W;
    dq = nt / cv;
    dc = nt - dq * cv;
  }
  __device__ __forceinline__ void next(int W, int cv) {
    cvi += dc;
    w += dq;
    if (cvi >= cv) { cvi -= cv; ++w; }
    while (w >= W) { w -= W; ++r; }
  }
};

// ---- fp32 on register pairs (one instruction for two products or sums) ----
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
        "l"(reinterpret_cast<unsigned long long&>(c)));
  return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 unpack2(uint32_t w) { return make_float2(bf_lo(w), bf_hi(w)); }
// sums over five neighbouring entries: t holds entries c-2 .. c+9 as pairs, w the sums around c .. c+7 (sliding, the
// same operations as window8: both kernels of a direction give the same bits)
__device__ __forceinline__ void window5(const float2 (&t)[6], float2 (&w)[4]) {
  const float v[12] = {t[0].x, t[0].y, t[1].x, t[1].y, t[2].x, t[2].y, t[3].x, t[3].y, t[4].x, t[4].y, t[5].x, t[5].y};
  float acc = v[0];
#pragma unroll
  for (int i = 1; i < 5; ++i) acc += v[i];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    w[k].x = acc;
    acc += v[2 * k + 5] - v[2 * k];
    w[k].y = acc;
    if (k < 3) acc += v[2 * k + 6] - v[2 * k + 1];
  }
}

// ---------------- forward ----------------
// grid = B * ceil(OH / RO); one CTA produces RO pooled rows from the (RO-1)*stride + K input rows under them.
// The input is read from global memory (one 16-byte load per 8 outputs and two of 4 bytes for the neighbours, 8 bytes for
// a window of 3 or 7 channels), normalised once per element into shared memory ([n_in][W][C] bf16), and pooled from there.
// K3S2: 3 x 3 windows with stride 2 (window size and stride are then constants of the pooling loops)
template <int HALF, bool K3S2>
__global__ void __launch_bounds__(512, 2)
lrn_maxpool_forward_kernel(const bf16* __restrict__ x, bf16* __restrict__ p, uint8_t* __restrict__ argmax,
                           const GeepsPoolGeom g, const LrnCoef cf, int RO) {
  geeps_pdl_enter();
  extern __shared__ __align__(16) uint8_t lp_smem[];
  const int C = g.C, cv = C >> 3, W = g.W;
  const int PK = K3S2 ? 3 : g.K, PS = K3S2 ? 2 : g.stride;
  const int row_elems = W * C;
  bf16* ys = reinterpret_cast<bf16*>(lp_smem);
  const int oh_blocks = (g.OH + RO - 1) / RO;
  const int b = blockIdx.x / oh_blocks, oh0 = (blockIdx.x - b * oh_blocks) * RO;
  const int n_out = min(RO, g.OH - oh0);
  const int ih_base = oh0 * PS - g.pad;                    // input row of shared-memory row 0 (may be < 0)
  const int r_lo = max(0, -ih_base);
  const int r_hi = min((n_out - 1) * PS + PK, g.H - ih_base);   // rows [r_lo, r_hi) exist
  const int tid = threadIdx.x, nt = blockDim.x;
  {
    const bf16* xbase = x + ((long long)b * g.H + ih_base + r_lo) * row_elems;
    bf16* ybase = ys + (size_t)r_lo * row_elems;
    const int nrows = r_hi - r_lo;
    if constexpr (HALF == 2) {
      // Pairs of channels: half the fp32 instructions, and a halo of one word per side instead of two.  Three items are
      // loaded before the first is computed: with one, half of the time went on waiting for it (256 x 55 x 55 x 96: 94 us,
      // three 79).  Polynomial or exact power in a branch each: the polynomial first and the exact power over it spills at the
      // 64 registers of two blocks per SM and takes 80 us, 103 instead of 94 where half of the vectors are beyond the range.
      constexpr int U = 3;
      for (ItemWalk it(tid, nt, W, cv); it.r < nrows;) {
        uint32_t before[U], after[U];
        uint4 xv[U];
        int at[U];                                            // offsets inside a block of a few rows: 32 bits
#pragma unroll
        for (int u = 0; u < U; ++u) {
          at[u] = -1;
          if (it.r < nrows) {
            const int c = it.cvi * 8;
            at[u] = it.r * row_elems + it.w * C + c;
            const bf16* px = xbase + at[u];
            before[u] = c > 0 ? *reinterpret_cast<const uint32_t*>(px - 2) : 0u;
            xv[u] = *reinterpret_cast<const uint4*>(px);
            after[u] = c + 8 < C ? *reinterpret_cast<const uint32_t*>(px + 8) : 0u;
            it.next(W, cv);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (at[u] < 0) break;
          const float2 v[6] = {unpack2(before[u]), unpack2(xv[u].x), unpack2(xv[u].y), unpack2(xv[u].z), unpack2(xv[u].w),
                               unpack2(after[u])};
          float2 t[6], ws[4], o[4];
#pragma unroll
          for (int k = 0; k < 6; ++k) t[k] = mul2(v[k], v[k]);
          window5(t, ws);
          if (squares12(ws, t[5]) <= cf.w_max || max4(ws) <= cf.w_max) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              o[k] = mul2(v[k + 1], fma2(ws[k], fma2(ws[k], fma2(ws[k], both(cf.p3), both(cf.p2)), both(cf.p1)), both(cf.p0)));
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              o[k] = make_float2(v[k + 1].x * __powf(cf.k * fmaf(cf.es, ws[k].x, 1.f), -cf.beta),
                                 v[k + 1].y * __powf(cf.k * fmaf(cf.es, ws[k].y, 1.f), -cf.beta));
          }
          *reinterpret_cast<uint4*>(ybase + at[u]) =
              make_uint4(pack_bf16x2(o[0].x, o[0].y), pack_bf16x2(o[1].x, o[1].y), pack_bf16x2(o[2].x, o[2].y),
                         pack_bf16x2(o[3].x, o[3].y));
        }
      }
    } else {
      for (ItemWalk it(tid, nt, W, cv); it.r < nrows; it.next(W, cv)) {
        const int c = it.cvi * 8;
        const int pix = it.r * row_elems + it.w * C;
        float v[16], t[16], ws[8], o[8];
        load16(xbase + pix, c, C, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) t[j] = v[j] * v[j];
        window8<HALF>(t, ws);
        if (max8(ws) <= cf.w_max) {
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = v[4 + e] * fmaf(ws[e], fmaf(ws[e], fmaf(ws[e], cf.p3, cf.p2), cf.p1), cf.p0);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = v[4 + e] * __powf(cf.k * fmaf(cf.es, ws[e], 1.f), -cf.beta);
        }
        *reinterpret_cast<uint4*>(ybase + pix + c) = pack8(o);
      }
    }
  }
  __syncthreads();
  for (ItemWalk it(tid, nt, g.OW, cv); it.r < n_out; it.next(g.OW, cv)) {
    const int oh = oh0 + it.r, ow = it.w, c = it.cvi * 8;
    const int ih0 = oh * PS - g.pad;
    const int kh_lo = max(0, -ih0), kh_hi = min(PK, g.H - ih0);
    const int iw0 = ow * PS - g.pad;
    const int kw_lo = max(0, -iw0), kw_hi = min(PK, W - iw0);
    // packed: best value and window code per 16-bit lane; strict > keeps the first maximum
    const uint32_t neg = 0xff7fff7fu;                 // two bf16 lowest finite values
    __nv_bfloat162 best[4];
    uint32_t arg[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { best[j] = *reinterpret_cast<const __nv_bfloat162*>(&neg); arg[j] = 0x00ff00ffu; }
    auto visit = [&](const bf16* yv, uint32_t code1) {
      const uint4 v = *reinterpret_cast<const uint4*>(yv);
      const uint32_t vv[4] = {v.x, v.y, v.z, v.w};
      const uint32_t code = code1 | (code1 << 16);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 x2 = *reinterpret_cast<const __nv_bfloat162*>(&vv[j]);
        const uint32_t gt = __hgt2_mask(x2, best[j]);
        best[j] = __hmax2(best[j], x2);
        arg[j] = (arg[j] & ~gt) | (code & gt);
      }
    };
    const bf16* y0 = ys + (ih0 - ih_base) * row_elems + iw0 * C + c;
    if (K3S2 && kh_hi - kh_lo == 3 && kw_hi - kw_lo == 3) {      // a whole 3 x 3 window: no loop counters, constant codes
#pragma unroll
      for (int t = 0; t < 9; ++t) visit(y0 + (t / 3) * row_elems + (t % 3) * C, (uint32_t)t);
    } else {
      for (int kh = kh_lo; kh < kh_hi; ++kh)
        for (int kw = kw_lo; kw < kw_hi; ++kw) visit(y0 + kh * row_elems + kw * C, (uint32_t)(kh * PK + kw));
    }
    const long long opix = ((long long)b * g.OH + oh) * g.OW + ow;
    *reinterpret_cast<uint4*>(p + opix * g.ldy + c) =
        make_uint4(*reinterpret_cast<const uint32_t*>(&best[0]), *reinterpret_cast<const uint32_t*>(&best[1]),
                   *reinterpret_cast<const uint32_t*>(&best[2]), *reinterpret_cast<const uint32_t*>(&best[3]));
    uint2 pk;      // 16-bit lanes -> bytes
    pk.x = __byte_perm(arg[0], arg[1], 0x6420);
    pk.y = __byte_perm(arg[2], arg[3], 0x6420);
    *reinterpret_cast<uint2*>(argmax + opix * C + c) = pk;
  }
}

// ---------------- backward, 3 x 3 windows with stride 2, window of 5 channels ----------------
// The general kernel below spends 79 instructions per element: three passes over shared memory, the halo channels of
// every 8-channel vector unpacked and squared again, window loops whose trip counts differ inside a warp.  Here LP lanes
// share one pixel and a lane holds NV vectors of 8 channels (vector lane + LP * j, so loads stay coalesced); x, the
// scaled gradient and the ratio stay in registers, a halo channel pair comes from the neighbouring lane by shuffle, and
// nothing goes through shared memory.  A warp takes pixels of one column parity at a time, so all its lanes visit the
// same number of windows (1 or 2 per direction).  fp32 arithmetic runs on register pairs (fma.rn.f32x2).
// 256 x 55 x 55 x 96: 245 -> 173 us; still bound by instruction issue.
// The 32-bit word (two channels) before / after vector j of this lane: the neighbouring lane's, or across the wrap of
// the vector order the last (first) lane's vector j - 1 (j + 1); zero outside the pixel.
template <int LP, int NV>
__device__ __forceinline__ uint32_t word_before(const uint4 (&v)[NV], int j, int lane) {
  const int l = lane & (LP - 1);
  const uint32_t wrap = j > 0 ? v[j > 0 ? j - 1 : 0].w : 0u;
  return __shfl_sync(0xffffffffu, l == LP - 1 ? wrap : v[j].w, (lane & ~(LP - 1)) | ((l - 1) & (LP - 1)));
}
template <int LP, int NV>
__device__ __forceinline__ uint32_t word_after(const uint4 (&v)[NV], int j, int lane) {
  const int l = lane & (LP - 1);
  const uint32_t wrap = j + 1 < NV ? v[j + 1 < NV ? j + 1 : j].x : 0u;
  return __shfl_sync(0xffffffffu, l == 0 ? wrap : v[j].x, (lane & ~(LP - 1)) | ((l + 1) & (LP - 1)));
}

template <int LP, int NV>
__global__ void __launch_bounds__(256, 2)
lrn_maxpool_backward_lanes_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dp,
                                  const uint8_t* __restrict__ argmax, bf16* __restrict__ dx, const GeepsPoolGeom g,
                                  const LrnCoef cf, float coef, int relu_mask, float* __restrict__ colsum) {
  geeps_pdl_enter();
  extern __shared__ __align__(16) uint8_t lp_smem[];
  float* cs_sh = reinterpret_cast<float*>(lp_smem);      // [C]
  constexpr int PPW = 32 / LP;                           // pixels of a warp
  const int C = g.C, cv = C >> 3, W = g.W, OW = g.OW;
  const int lane = threadIdx.x & 31, l = lane & (LP - 1), pix = lane / LP;
  const int strips = ((W + 1) / 2 + PPW - 1) / PPW;      // strips of PPW columns of one parity
  const int per_row = 2 * strips;
  const int items = g.B * g.H * per_row;
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  float2 cs[NV][4];
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) cs[j][k] = both(0.f);
  if (colsum != nullptr) {
    for (int i = threadIdx.x; i < C; i += blockDim.x) cs_sh[i] = 0.f;
    __syncthreads();
  }
  for (int item = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); item < items; item += nwarps) {
    const int row = item / per_row, s = item - row * per_row;
    const int b = row / g.H, h = row - b * g.H;
    const int w = 2 * ((s >> 1) * PPW + pix) + (s & 1);
    const bool in = w < W;
    const long long px = ((long long)row * W + w) * C + l * 8;
    uint4 xv[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j)
      xv[j] = in && l + LP * j < cv ? *reinterpret_cast<const uint4*>(x + px + LP * 8 * j) : make_uint4(0u, 0u, 0u, 0u);
    // pooling gradient at these elements
    float2 dy[NV][4];
    uint32_t hit[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      hit[j] = 0u;
#pragma unroll
      for (int k = 0; k < 4; ++k) dy[j][k] = both(0.f);
    }
    const int th = h + g.pad, tw = w + g.pad;
    const int oh_lo = max(0, (th - 1) >> 1), oh_hi = min(g.OH - 1, th >> 1);
    const int ow_lo = max(0, (tw - 1) >> 1), ow_hi = in ? min(OW - 1, tw >> 1) : -1;
    for (int oh = oh_lo; oh <= oh_hi; ++oh) {
      for (int ow = ow_lo; ow <= ow_hi; ++ow) {
        const uint32_t c4 = (uint32_t)((th - 2 * oh) * 3 + tw - 2 * ow) * 0x01010101u;
        const long long opix = ((long long)b * g.OH + oh) * OW + ow;
        const uint8_t* ap = argmax + opix * C + l * 8;
        const bf16* gp = dp + opix * g.ldy + l * 8;
        uint2 pk[NV];
        uint4 d[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const bool on = l + LP * j < cv;
          pk[j] = on ? *reinterpret_cast<const uint2*>(ap + LP * 8 * j) : make_uint2(0xffffffffu, 0xffffffffu);
          d[j] = on ? *reinterpret_cast<const uint4*>(gp + LP * 8 * j) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const uint32_t m0 = __vcmpeq4(pk[j].x, c4), m1 = __vcmpeq4(pk[j].y, c4);      // 0xff per matching channel
          hit[j] |= m0 | m1;
          // byte mask -> 16-bit lane mask
          dy[j][0] = add2(dy[j][0], unpack2(d[j].x & __byte_perm(m0, 0, 0x1100)));
          dy[j][1] = add2(dy[j][1], unpack2(d[j].y & __byte_perm(m0, 0, 0x3322)));
          dy[j][2] = add2(dy[j][2], unpack2(d[j].z & __byte_perm(m1, 0, 0x1100)));
          dy[j][3] = add2(dy[j][3], unpack2(d[j].w & __byte_perm(m1, 0, 0x3322)));
        }
      }
    }
    // a = dy * scale^-beta, rt = dy * x * scale^-(beta+1), both rounded to bf16 as the general kernel stores them
    uint4 av[NV], rv[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const uint32_t before = word_before<LP, NV>(xv, j, lane), after = word_after<LP, NV>(xv, j, lane);
      const float2 v[4] = {unpack2(xv[j].x), unpack2(xv[j].y), unpack2(xv[j].z), unpack2(xv[j].w)};
      float2 t[6], ws[4], a[4], rt[4];
      t[0] = unpack2(before); t[5] = unpack2(after);
      t[0] = mul2(t[0], t[0]); t[5] = mul2(t[5], t[5]);
#pragma unroll
      for (int k = 0; k < 4; ++k) t[k + 1] = mul2(v[k], v[k]);
      window5(t, ws);
      av[j] = make_uint4(0u, 0u, 0u, 0u);
      rv[j] = make_uint4(0u, 0u, 0u, 0u);
      if (hit[j] != 0u) {
        if (max4(ws) <= cf.w_max) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            a[k] = mul2(dy[j][k], fma2(ws[k], fma2(ws[k], fma2(ws[k], both(cf.p3), both(cf.p2)), both(cf.p1)), both(cf.p0)));
            rt[k] = mul2(mul2(dy[j][k], v[k]),
                         fma2(ws[k], fma2(ws[k], fma2(ws[k], both(cf.q3), both(cf.q2)), both(cf.q1)), both(cf.q0)));
          }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float s0 = cf.k * fmaf(cf.es, ws[k].x, 1.f), s1 = cf.k * fmaf(cf.es, ws[k].y, 1.f);
            a[k] = make_float2(dy[j][k].x * __powf(s0, -cf.beta), dy[j][k].y * __powf(s1, -cf.beta));
            rt[k] = make_float2(a[k].x * v[k].x * __frcp_rn(s0), a[k].y * v[k].y * __frcp_rn(s1));
          }
        }
        av[j] = make_uint4(pack_bf16x2(a[0].x, a[0].y), pack_bf16x2(a[1].x, a[1].y), pack_bf16x2(a[2].x, a[2].y),
                           pack_bf16x2(a[3].x, a[3].y));
        rv[j] = make_uint4(pack_bf16x2(rt[0].x, rt[0].y), pack_bf16x2(rt[1].x, rt[1].y), pack_bf16x2(rt[2].x, rt[2].y),
                           pack_bf16x2(rt[3].x, rt[3].y));
      }
    }
    // dx = a - coef * x * (window sum of rt), ReLU mask, per-channel sums
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const uint32_t before = word_before<LP, NV>(rv, j, lane), after = word_after<LP, NV>(rv, j, lane);
      const float2 t[6] = {unpack2(before), unpack2(rv[j].x), unpack2(rv[j].y), unpack2(rv[j].z), unpack2(rv[j].w),
                           unpack2(after)};
      float2 ws[4], o[4];
      window5(t, ws);
      const uint32_t xw[4] = {xv[j].x, xv[j].y, xv[j].z, xv[j].w}, aw[4] = {av[j].x, av[j].y, av[j].z, av[j].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 v = unpack2(xw[k]);
        o[k] = fma2(mul2(both(-coef), v), ws[k], unpack2(aw[k]));
        if (relu_mask && v.x <= 0.f) o[k].x = 0.f;
        if (relu_mask && v.y <= 0.f) o[k].y = 0.f;
      }
      if (in && l + LP * j < cv) {
        *reinterpret_cast<uint4*>(dx + px + LP * 8 * j) =
            make_uint4(pack_bf16x2(o[0].x, o[0].y), pack_bf16x2(o[1].x, o[1].y), pack_bf16x2(o[2].x, o[2].y),
                       pack_bf16x2(o[3].x, o[3].y));
#pragma unroll
        for (int k = 0; k < 4; ++k) cs[j][k] = add2(cs[j][k], o[k]);
      }
    }
  }
  if (colsum != nullptr) {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int m = LP; m < 32; m <<= 1) {
          cs[j][k].x += __shfl_xor_sync(0xffffffffu, cs[j][k].x, m);
          cs[j][k].y += __shfl_xor_sync(0xffffffffu, cs[j][k].y, m);
        }
        const int c = (l + LP * j) * 8 + 2 * k;
        if (pix == 0 && c < C) { atomicAdd(&cs_sh[c], cs[j][k].x); atomicAdd(&cs_sh[c + 1], cs[j][k].y); }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < C; i += blockDim.x) atomicAdd(colsum + i, cs_sh[i]);
  }
}

// ---------------- backward, 3 x 3 windows with stride 2, window of 5 channels, many pixels ----------------
// The 2 x 2 input pixels between two window rows and two window columns (a quad) lie under the same four windows, so a
// lane takes the four pixels of a quad in one vector of 8 channels: four window loads instead of nine, all of a lane's
// loads in flight at once, and which windows cover a pixel is known when the kernel is compiled.  Neighbouring lanes
// hold neighbouring vectors of the flat (image, quad row, quad, vector) index; the first and the last lane of a warp repeat
// a vector of their neighbours for the halo channels and store nothing, so 30 of 32 lanes work at every channel count.
// The window codes are spread to 16-bit numbers between 0.5 and 2; one packed comparison then is a mask.  The polynomials
// are evaluated without a branch around them (a pixel beyond their range is done again, exactly), so the arithmetic of
// neighbouring pixels overlaps.  Sums over windows and channels, and the choice between polynomial and exact power, are those
// of the lanes kernel above, in its order: the results have the same bits (but for vectors with a NaN, which take the exact
// path here).
// Bound by instruction issue (64 % of the slots, half-rate integer pipe 62 %) at 16 warps per SM: 256 x 55 x 55 x 96
// 170 us (lanes kernel) -> 132, 256 x 27 x 27 x 256 109 -> 90, 64 x 55 x 55 x 264 150 -> 98; with all vectors beyond the range
// 240 -> 228, 150 -> 154, with half of them 205 -> 195, 133 -> 132 (the exact path by the sum of the squares alone, not the largest window:
// 237, 159; in a branch of its own beside the polynomials: 216, 146 and 204, 137).  Three blocks per SM spill: 165 us; two pixels at a
// time spill too: 147; fp32 without the register pairs: 151; without the last four of the savings named at the lines below
// (codes expanded at use, packed sign test, merged halo words, match test only beyond the range): 153.

// c + the two bf16 of w (a mixed-precision sum needs no conversion in front of it)
__device__ __forceinline__ float2 add_bf16(float2 c, uint32_t w) {
  asm("{.reg .b16 l, h; mov.b32 {l, h}, %2; add.f32.bf16 %0, l, %0; add.f32.bf16 %1, h, %1;}" : "+f"(c.x), "+f"(c.y) : "r"(w));
  return c;
}
// o, 0 where x <= lim (never for a NaN)
__device__ __forceinline__ float2 zero_where_le(float2 o, uint32_t x, uint32_t lim) {
  asm("{.reg .pred p, q; setp.le.bf16x2 p|q, %2, %3; selp.f32 %0, 0f00000000, %0, p; selp.f32 %1, 0f00000000, %1, q;}"
      : "+f"(o.x), "+f"(o.y) : "r"(x), "r"(lim));
  return o;
}
// A walk over the mixed-radix index (image, quad row, quad) in steps of a constant.
struct QuadWalk {
  int b, h, w;
  int db, dh, dw;
  __device__ __forceinline__ QuadWalk(int first, int step, int QH, int QW) {
    const int r = first / QW, t = step / QW;
    w = first - r * QW;
    b = r / QH;
    h = r - b * QH;
    dw = step - t * QW;
    db = t / QH;
    dh = t - db * QH;
  }
  __device__ __forceinline__ void next(int QH, int QW) {
    w += dw;
    h += dh;
    b += db;
    if (w >= QW) { w -= QW; ++h; }
    if (h >= QH) { h -= QH; ++b; }
  }
};

// total: vectors of all quads.  warps: those that work, each at vectors 30 warp, 30 (warp + warps), ...; 30 warps is a
// multiple of cv unless every warp takes one step.
__global__ void __launch_bounds__(256, 2)
lrn_maxpool_backward_quad_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dp,
                                 const uint8_t* __restrict__ argmax, bf16* __restrict__ dx, const GeepsPoolGeom g,
                                 const LrnCoef cf, float coef, int relu_mask, float* __restrict__ colsum, int QH, int QW,
                                 int total, int warps) {
  geeps_pdl_enter();
  __shared__ float cs_sh[8][30 * 8 + 1];        // by channel of the vector: the block's 8 x 30 working lanes
  const int C = g.C, cv = C >> 3, W = g.W, OW = g.OW;
  const int lane = threadIdx.x & 31;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int step = warps * 30;
  // the lane before vector 0 has no quad; the values that it hands on are not used
  int f = warp * 30 + lane - 1;
  const int f0 = f < 0 ? 0 : f;
  const int vec = f0 % cv;
  float2 cs[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) cs[k] = both(0.f);
  QuadWalk q(f0 / cv, step / cv, QH, QW);
  // the channels beside a vector: none at the ends of a pixel, loaded at the ends of a warp, else the neighbour's
  const bool first_vec = vec == 0, last_vec = vec == cv - 1;
  const uint32_t keep_b = lane == 0 || first_vec ? 0u : 0xffffffffu, keep_a = lane == 31 || last_vec ? 0u : 0xffffffffu;
  const bool stores = lane != 0 && lane != 31;
  const uint32_t lim = relu_mask ? 0u : 0x7fc07fc0u;
  const int q0 = g.pad >> 1;                     // quad rows and columns begin on a window's first row and column
  for (int it0 = warp * 30; warp < warps && it0 < total; it0 += step, f += step, q.next(QH, QW)) {
    const bool on = f >= 0 && f < total;
    const int h0 = 2 * (q.h + q0) - g.pad, w0 = 2 * (q.w + q0) - g.pad;
    const long long px = (((long long)q.b * g.H + h0) * W + w0) * C + vec * 8;
    uint4 xq[4];
    uint32_t edge[4];
    bool in[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      in[i] = on && (unsigned)(h0 + (i >> 1)) < (unsigned)g.H && (unsigned)(w0 + (i & 1)) < (unsigned)W;
      const bf16* xp = x + px + ((i >> 1) * W + (i & 1)) * C;
      xq[i] = in[i] ? *reinterpret_cast<const uint4*>(xp) : make_uint4(0u, 0u, 0u, 0u);
      edge[i] = 0u;
      if (in[i] && ((lane == 0 && !first_vec) || (lane == 31 && !last_vec)))
        edge[i] = *reinterpret_cast<const uint32_t*>(xp + (lane == 0 ? -2 : 8));
    }
    // windows (row before, column before), (row before, column), (row, column before), (row, column)
    uint32_t d[4][4];
    uint2 raw[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int oh = q.h + q0 - 1 + (i >> 1), ow = q.w + q0 - 1 + (i & 1);
      const bool there = on && (unsigned)oh < (unsigned)g.OH && (unsigned)ow < (unsigned)OW;
      const long long opix = ((long long)q.b * g.OH + oh) * OW + ow;
      raw[i] = there ? *reinterpret_cast<const uint2*>(argmax + opix * C + vec * 8) : make_uint2(0xffffffffu, 0xffffffffu);
      const uint4 dv = there ? *reinterpret_cast<const uint4*>(dp + opix * g.ldy + vec * 8) : make_uint4(0u, 0u, 0u, 0u);
      d[i][0] = dv.x; d[i][1] = dv.y; d[i][2] = dv.z; d[i][3] = dv.w;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (!__any_sync(0xffffffffu, in[2 * r] || in[2 * r + 1])) continue;       // beyond the last row
      uint32_t code[4][4];
#pragma unroll
      for (int j = 2 * r; j < 4; ++j) {
        code[j][0] = __byte_perm(raw[j].x, 0x3f3f3f3fu, 0x4140); code[j][1] = __byte_perm(raw[j].x, 0x3f3f3f3fu, 0x4342);
        code[j][2] = __byte_perm(raw[j].y, 0x3f3f3f3fu, 0x4140); code[j][3] = __byte_perm(raw[j].y, 0x3f3f3f3fu, 0x4342);
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int i = 2 * r + c;
        // pooling gradient: window j covers the pixel unless it begins in the row (column) before and the pixel is in
        // the quad's second row (column)
        float2 dy[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) dy[k] = both(0.f);
#pragma unroll
        for (int j = 2 * r; j < 4; ++j) {
          if ((j & 1) == 0 && c == 1) continue;
          const int kh = j < 2 ? 2 : r, kw = (j & 1) == 0 ? 2 : c;
          const uint32_t want = 0x3f003f00u | (uint32_t)((kh * 3 + kw) * 0x00010001u);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            dy[k] = add_bf16(dy[k], d[j][k] & __heq2_mask(reinterpret_cast<const __nv_bfloat162&>(code[j][k]),
                                                          reinterpret_cast<const __nv_bfloat162&>(want)));
        }
        // a = dy * scale^-beta, rt = dy * x * scale^-(beta+1), both rounded to bf16
        uint32_t before = __shfl_up_sync(0xffffffffu, xq[i].w, 1), after = __shfl_down_sync(0xffffffffu, xq[i].x, 1);
        before = (before & keep_b) | (lane == 0 ? edge[i] : 0u);
        after = (after & keep_a) | (lane == 31 ? edge[i] : 0u);
        const float2 v[4] = {unpack2(xq[i].x), unpack2(xq[i].y), unpack2(xq[i].z), unpack2(xq[i].w)};
        float2 t[6], ws[4], a[4], rt[4];
        t[0] = unpack2(before); t[5] = unpack2(after);
        t[0] = mul2(t[0], t[0]); t[5] = mul2(t[5], t[5]);
#pragma unroll
        for (int k = 0; k < 4; ++k) t[k + 1] = mul2(v[k], v[k]);
        window5(t, ws);
        const bool beyond = !(squares12(ws, t[5]) <= cf.w_max) && !(max4_nan(ws) <= cf.w_max);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          a[k] = mul2(dy[k], fma2(ws[k], fma2(ws[k], fma2(ws[k], both(cf.p3), both(cf.p2)), both(cf.p1)), both(cf.p0)));
          rt[k] = mul2(mul2(dy[k], v[k]),
                       fma2(ws[k], fma2(ws[k], fma2(ws[k], both(cf.q3), both(cf.q2)), both(cf.q1)), both(cf.q0)));
        }
        if (beyond) {
          uint32_t hit = 0u;                      // a vector without a gradient has none here either (no 0 x inf, no 0 x NaN)
#pragma unroll
          for (int j = 2 * r; j < 4; ++j) {
            if ((j & 1) == 0 && c == 1) continue;
            const uint32_t c4 = (uint32_t)((j < 2 ? 2 : r) * 3 + ((j & 1) == 0 ? 2 : c)) * 0x01010101u;
            hit |= __vcmpeq4(raw[j].x, c4) | __vcmpeq4(raw[j].y, c4);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float s0 = cf.k * fmaf(cf.es, ws[k].x, 1.f), s1 = cf.k * fmaf(cf.es, ws[k].y, 1.f);
            a[k] = make_float2(dy[k].x * __powf(s0, -cf.beta), dy[k].y * __powf(s1, -cf.beta));
            rt[k] = make_float2(a[k].x * v[k].x * __frcp_rn(s0), a[k].y * v[k].y * __frcp_rn(s1));
            if (hit == 0u) { a[k] = both(0.f); rt[k] = both(0.f); }
          }
        }
        const uint32_t aw[4] = {pack_bf16x2(a[0].x, a[0].y), pack_bf16x2(a[1].x, a[1].y), pack_bf16x2(a[2].x, a[2].y),
                                pack_bf16x2(a[3].x, a[3].y)};
        const uint4 rv = make_uint4(pack_bf16x2(rt[0].x, rt[0].y), pack_bf16x2(rt[1].x, rt[1].y),
                                    pack_bf16x2(rt[2].x, rt[2].y), pack_bf16x2(rt[3].x, rt[3].y));
        // dx = a - coef * x * (window sum of rt), ReLU mask, per-channel sums
        before = __shfl_up_sync(0xffffffffu, rv.w, 1);
        after = __shfl_down_sync(0xffffffffu, rv.x, 1);
        if (first_vec) before = 0u;
        if (last_vec) after = 0u;
        const float2 u[6] = {unpack2(before), unpack2(rv.x), unpack2(rv.y), unpack2(rv.z), unpack2(rv.w), unpack2(after)};
        window5(u, ws);
        const uint32_t xw[4] = {xq[i].x, xq[i].y, xq[i].z, xq[i].w};
        float2 o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          o[k] = zero_where_le(fma2(mul2(both(-coef), v[k]), ws[k], unpack2(aw[k])), xw[k], lim);
        if (in[i] && stores) {
          *reinterpret_cast<uint4*>(dx + px + (r * W + c) * C) =
              make_uint4(pack_bf16x2(o[0].x, o[0].y), pack_bf16x2(o[1].x, o[1].y), pack_bf16x2(o[2].x, o[2].y),
                         pack_bf16x2(o[3].x, o[3].y));
#pragma unroll
          for (int k = 0; k < 4; ++k) cs[k] = add2(cs[k], o[k]);
        }
      }
    }
  }
  if (colsum != nullptr) {
    // the working lanes of a block hold consecutive vectors, each for all of its steps
    if (stores) {
      const int at = (threadIdx.x >> 5) * 30 + lane - 1;
#pragma unroll
      for (int k = 0; k < 4; ++k) { cs_sh[2 * k][at] = cs[k].x; cs_sh[2 * k + 1][at] = cs[k].y; }
    }
    __syncthreads();
    const int base = (int)(blockIdx.x * 240u % (unsigned)cv);
    // several threads a channel where there are few channels, their sums met in the places of the first ones' vectors
    const int parts = C < 256 ? 256 / C : 1;
    for (int i = threadIdx.x; i < C * parts; i += blockDim.x) {
      const int c = i % C, part = i / C;
      int at = (c >> 3) - base;
      if (at < 0) at += cv;
      at += part * cv;
      const int first = at;
      float sum = 0.f;
      for (; at < 240; at += parts * cv) sum += cs_sh[c & 7][at];
      if (parts == 1) { if (first < 240) atomicAdd(colsum + c, sum); }
      else if (first < 240) cs_sh[c & 7][first] = sum;
    }
    if (parts > 1) {
      __syncthreads();
      const int c = threadIdx.x;
      if (c < C) {
        int at = (c >> 3) - base;
        if (at < 0) at += cv;
        float sum = 0.f;
        for (int part = 0; part < parts && at < 240; ++part, at += cv) sum += cs_sh[c & 7][at];
        atomicAdd(colsum + c, sum);
      }
    }
  }
}

// ---------------- backward, any window ----------------
// Persistent: CTA i handles row blocks i, i + gridDim, ... (a row block = R input rows of one image).
// Shared memory: as, rs [R][W][C] bf16, dps [max_oh][OW][C] bf16, args [max_oh][OW][C] u8, cs [C] float.
//   as = dy * scale^-beta          rs = dy * x * scale^-(beta+1)       (dy = pooling gradient at the element)
//   dx = as - 2 alpha beta / n * x * (window sum of rs)
// The host picks blockDim as a multiple of C/8, so a thread keeps its channel vector for every item it visits and
// sums the bias gradient in registers.
// K3S2: the pooling window is 3 x 3 with stride 2 (AlexNet): window size and stride become constants, so the four
// divisions per pixel vector that find the windows covering it are shifts.
template <int HALF, bool K3S2>
__global__ void __launch_bounds__(512, 2)
lrn_maxpool_backward_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dp, const uint8_t* __restrict__ argmax,
                            bf16* __restrict__ dx, const GeepsPoolGeom g, int R, int max_oh, const LrnCoef cf, float coef,
                            int relu_mask, float* __restrict__ colsum) {
  geeps_pdl_enter();
  extern __shared__ __align__(16) uint8_t lp_smem[];
  const int C = g.C, cv = C >> 3, W = g.W, OW = g.OW;
  const int PK = K3S2 ? 3 : g.K, PS = K3S2 ? 2 : g.stride;
  const int row_elems = W * C, orow_elems = OW * C;
  bf16* as = reinterpret_cast<bf16*>(lp_smem);
  bf16* rs = as + (size_t)R * row_elems;
  bf16* dps = rs + (size_t)R * row_elems;
  uint8_t* args = reinterpret_cast<uint8_t*>(dps + (size_t)max_oh * orow_elems);
  float* cs_sh = reinterpret_cast<float*>(args + (((size_t)max_oh * orow_elems + 15) & ~(size_t)15));
  const int tid = threadIdx.x, nt = blockDim.x;
  const int row_blocks = (g.H + R - 1) / R;
  const int total_blocks = g.B * row_blocks;
  const bool fixed_channel = nt % cv == 0;
  float cs[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) cs[e] = 0.f;
  if (colsum != nullptr) for (int j = tid; j < C; j += nt) cs_sh[j] = 0.f;

  for (int blk = blockIdx.x; blk < total_blocks; blk += gridDim.x) {
    const int b = blk / row_blocks, h0 = (blk - b * row_blocks) * R;
    const int nr = min(R, g.H - h0);
    const int oh_lo = max(0, (h0 + g.pad - PK + PS) / PS);
    const int oh_hi = min(g.OH - 1, (h0 + nr - 1 + g.pad) / PS);
    __syncthreads();                                   // the previous block's readers are done with the buffers
    {
      const long long opix0 = ((long long)b * g.OH + oh_lo) * OW;
      uint4* dd = reinterpret_cast<uint4*>(dps);
      uint2* da = reinterpret_cast<uint2*>(args);
      int i = tid;
      for (ItemWalk it(tid, nt, OW, cv); it.r <= oh_hi - oh_lo; it.next(OW, cv), i += nt) {
        const long long opix = opix0 + (long long)it.r * OW + it.w;
        dd[i] = *reinterpret_cast<const uint4*>(dp + opix * g.ldy + it.cvi * 8);
        da[i] = *reinterpret_cast<const uint2*>(argmax + opix * C + it.cvi * 8);
      }
    }
    __syncthreads();
    const bf16* xblk = x + ((long long)b * g.H + h0) * row_elems;
    // phase 2: pooling gradient; where it is non-zero, the two powers of the scale
    for (ItemWalk it(tid, nt, W, cv); it.r < nr; it.next(W, cv)) {
      const int c = it.cvi * 8;
      const int th = h0 + it.r + g.pad, tw = it.w + g.pad;
      const int roh_lo = max(oh_lo, (th - PK + PS) / PS), roh_hi = min(oh_hi, th / PS);
      const int ow_lo = max(0, (tw - PK + PS) / PS), ow_hi = min(OW - 1, tw / PS);
      float dy[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) dy[e] = 0.f;
      bool any = false;
      for (int oh = roh_lo; oh <= roh_hi; ++oh) {
        const uint32_t code_h = (uint32_t)((th - oh * PS) * PK + tw);
        for (int ow = ow_lo; ow <= ow_hi; ++ow) {
          const uint32_t code = code_h - (uint32_t)(ow * PS);
          const int o = (oh - oh_lo) * orow_elems + ow * C + c;
          const uint2 pk = *reinterpret_cast<const uint2*>(args + o);
          const uint32_t c4 = code * 0x01010101u;
          const uint32_t m0 = __vcmpeq4(pk.x, c4), m1 = __vcmpeq4(pk.y, c4);      // 0xff per matching channel
          if ((m0 | m1) == 0) continue;
          any = true;
          const uint4 d = *reinterpret_cast<const uint4*>(dps + o);
          // keep the gradients of the matching channels: byte mask -> 16-bit lane mask
          const uint32_t k0 = d.x & __byte_perm(m0, 0, 0x1100), k1 = d.y & __byte_perm(m0, 0, 0x3322);
          const uint32_t k2 = d.z & __byte_perm(m1, 0, 0x1100), k3 = d.w & __byte_perm(m1, 0, 0x3322);
          dy[0] += bf_lo(k0); dy[1] += bf_hi(k0); dy[2] += bf_lo(k1); dy[3] += bf_hi(k1);
          dy[4] += bf_lo(k2); dy[5] += bf_hi(k2); dy[6] += bf_lo(k3); dy[7] += bf_hi(k3);
        }
      }
      const int pix = it.r * row_elems + it.w * C;          // offsets inside a block of a few rows: 32 bits
      uint4 oa = make_uint4(0u, 0u, 0u, 0u), orat = make_uint4(0u, 0u, 0u, 0u);
      if (any) {
        float v[16], t[16], ws[8], a[8], rt[8];
        load16(xblk + pix, c, C, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) t[j] = v[j] * v[j];
        window8<HALF>(t, ws);
        if (max8(ws) <= cf.w_max) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            a[e] = dy[e] * fmaf(ws[e], fmaf(ws[e], fmaf(ws[e], cf.p3, cf.p2), cf.p1), cf.p0);
            rt[e] = dy[e] * v[4 + e] * fmaf(ws[e], fmaf(ws[e], fmaf(ws[e], cf.q3, cf.q2), cf.q1), cf.q0);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float sc = cf.k * fmaf(cf.es, ws[e], 1.f);
            a[e] = dy[e] * __powf(sc, -cf.beta);
            rt[e] = a[e] * v[4 + e] * __frcp_rn(sc);
          }
        }
        oa = pack8(a);
        orat = pack8(rt);
      }
      *reinterpret_cast<uint4*>(as + pix + c) = oa;
      *reinterpret_cast<uint4*>(rs + pix + c) = orat;
    }
    __syncthreads();
    // phase 3: dx = a - coef * x * (window sum of ratio), ReLU mask, per-channel sums
    bf16* dblk = dx + ((long long)b * g.H + h0) * row_elems;
    for (ItemWalk it(tid, nt, W, cv); it.r < nr; it.next(W, cv)) {
      const int c = it.cvi * 8;
      const int pix = it.r * row_elems + it.w * C;          // offsets inside a block of a few rows: 32 bits
      float rt[16], ws[8], o[8];
      load16(rs + pix, c, C, rt);
      window8<HALF>(rt, ws);
      const uint4 xv = *reinterpret_cast<const uint4*>(xblk + pix + c);
      const uint4 av = *reinterpret_cast<const uint4*>(as + pix + c);
      const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w}, aw[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float x0 = bf_lo(xw[j]), x1 = bf_hi(xw[j]);
        const float d0 = fmaf(-coef * x0, ws[2 * j], bf_lo(aw[j])), d1 = fmaf(-coef * x1, ws[2 * j + 1], bf_hi(aw[j]));
        o[2 * j] = (relu_mask && x0 <= 0.f) ? 0.f : d0;
        o[2 * j + 1] = (relu_mask && x1 <= 0.f) ? 0.f : d1;
      }
      *reinterpret_cast<uint4*>(dblk + pix + c) = pack8(o);
      if (colsum != nullptr) {
        if (fixed_channel) {
#pragma unroll
          for (int e = 0; e < 8; ++e) cs[e] += o[e];
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) atomicAdd(&cs_sh[c + e], o[e]);
        }
      }
    }
  }
  if (colsum != nullptr) {
    __syncthreads();
    if (fixed_channel) {
      const int c = (tid % cv) * 8;
#pragma unroll
      for (int e = 0; e < 8; ++e) atomicAdd(&cs_sh[c + e], cs[e]);
    }
    __syncthreads();
    for (int j = tid; j < C; j += nt) atomicAdd(colsum + j, cs_sh[j]);
  }
}

LrnCoef make_coef(int size, float alpha, float beta, float k) {
  LrnCoef cf;
  cf.beta = beta; cf.k = k;
  const double es = (double)alpha / ((double)size * k);
  cf.es = (float)es;
  cf.w_max = (float)(kPolyEps / es);
  const double b0 = beta, b1 = beta + 1.0;
  const double p0 = pow((double)k, -b0), q0 = pow((double)k, -b1);
  cf.p0 = (float)p0;
  cf.p1 = (float)(p0 * -b0 * es);
  cf.p2 = (float)(p0 * b0 * (b0 + 1) / 2 * es * es);
  cf.p3 = (float)(p0 * -b0 * (b0 + 1) * (b0 + 2) / 6 * es * es * es);
  cf.q0 = (float)q0;
  cf.q1 = (float)(q0 * -b1 * es);
  cf.q2 = (float)(q0 * b1 * (b1 + 1) / 2 * es * es);
  cf.q3 = (float)(q0 * -b1 * (b1 + 1) * (b1 + 2) / 6 * es * es * es);
  return cf;
}

// 1-D blocks whose size is a multiple of the channel-vector count where that is possible
int lp_threads(int cv, int max_threads) {
  if (cv >= max_threads) return max_threads;
  return max_threads / cv * cv;
}


bool lp_shape_ok(const GeepsPoolGeom* g, int size) {
  return g->C % 8 == 0 && g->ldx == g->C && g->ldy % 8 == 0 && g->K * g->K <= 255 && g->K >= 1 && g->stride >= 1 &&
         (size == 3 || size == 5 || size == 7);
}
// pooled rows per forward CTA: as many as fit three CTAs per SM (74 KB each), at most 4
constexpr size_t kLpMaxSmem = 200 * 1024;
constexpr size_t kLpTwoPerSm = 112 * 1024;    // two CTAs of this size share one SM's shared memory

// Lanes per pixel and 8-channel vectors per lane of the register kernel.  Two thirds of the vector slots are used at every
// channel count (64 x 55 x 55 x 264, 33 vectors: 206 us on 32 x 2 slots, 150 on 16 x 3; x 8, one vector, without column
// sums: 19.7 us on 4 x 1, 6.4 on 1 x 1; x 40: 31 us on 4 x 2, 21.5 on 2 x 3; the general kernel takes 177, 14.0 and 30),
// but where that leaves an SM fewer than eight warps more lanes share a pixel (2 x 27 x 27 x 40: 9.8 us on 2 x 3, 8.3 on 4 x 2).
struct LrnLanes { int lp, nv; };
LrnLanes lrn_lanes(int cv, long long pixels) {
  int lp = cv <= 1 ? 1 : cv == 2 || cv == 5 || cv == 6 ? 2 : cv <= 12 ? 4 : cv <= 24 ? 8 : cv <= 48 ? 16 : 32;
  if (pixels * lp / 32 < 8LL * geeps_sm_count()) lp = cv <= 12 ? 4 : cv <= 24 ? 8 : cv <= 32 ? 16 : 32;
  return {lp, (cv + lp - 1) / lp};
}

int lp_env(const char* name, int dflt) {
  const char* e = getenv(name);
  return e ? atoi(e) : dflt;
}
int lp_fwd_rows(const GeepsPoolGeom* g) {
  static const int forced = lp_env("GEEPS_LP_FWD_RO", 0);
  if (forced > 0) return forced;
  int ro = 3;     // measured: 3 rows with 512 threads (two CTAs per SM) is the fastest of rows 2..4 x threads 256 / 512
  while (ro > 1 && (size_t)((ro - 1) * g->stride + g->K) * g->W * g->C * 2 > kLpTwoPerSm) --ro;
  return ro;
}
size_t lp_fwd_smem(const GeepsPoolGeom* g) { return (size_t)((lp_fwd_rows(g) - 1) * g->stride + g->K) * g->W * g->C * 2; }
int lp_bwd_rows(const GeepsPoolGeom* g) { return g->stride > 1 ? 2 * g->stride : 2; }
int lp_bwd_max_oh(const GeepsPoolGeom* g, int R) { return (R + g->K - 2) / g->stride + 1; }
size_t lp_bwd_smem(const GeepsPoolGeom* g, int R, int max_oh) {
  const size_t out = (size_t)max_oh * g->OW * g->C;
  return (size_t)2 * R * g->W * g->C * 2 + out * 2 + ((out + 15) & ~(size_t)15) + (size_t)g->C * 4;
}

}  // namespace

extern "C" {

int geeps_lrn_maxpool_supported(const GeepsPoolGeom* g, int size) {
  if (!lp_shape_ok(g, size)) return 0;
  int R = lp_bwd_rows(g);
  if (lp_fwd_smem(g) > kLpMaxSmem) return 0;
  while (R > 1 && lp_bwd_smem(g, R, lp_bwd_max_oh(g, R)) > kLpTwoPerSm) R >>= 1;
  return lp_bwd_smem(g, R, lp_bwd_max_oh(g, R)) <= kLpMaxSmem ? 1 : 0;
}

int geeps_lrn_lanes(int C, long long pixels, int* lanes, int* vectors) {
  const LrnLanes l = lrn_lanes(C / 8, pixels);
  *lanes = l.lp;
  *vectors = l.nv;
  return 0;
}

int geeps_lrn_maxpool_forward(const void* x, void* p, void* argmax, const GeepsPoolGeom* g, int size, float alpha,
                              float beta, float k, void* stream) {
  if (!geeps_lrn_maxpool_supported(g, size)) return (int)cudaErrorInvalidValue;
  const size_t smem = lp_fwd_smem(g);
  static const int fwd_threads = lp_env("GEEPS_LP_FWD_THREADS", 512);
  const int block = lp_threads(g->C / 8, fwd_threads);
  const LrnCoef cf = make_coef(size, alpha, beta, k);
  const int RO = lp_fwd_rows(g);
  const int grid = g->B * ((g->OH + RO - 1) / RO);
  cudaStream_t st = (cudaStream_t)stream;
#define LP_FWD(HALF, K3S2)                                                                                         \
  do {                                                                                                             \
    static bool attr_set = false;                                                                                  \
    if (!attr_set) {                                                                                               \
      cudaError_t e = cudaFuncSetAttribute(lrn_maxpool_forward_kernel<HALF, K3S2>,                                 \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLpMaxSmem);          \
      if (e != cudaSuccess) return (int)e;                                                                         \
      attr_set = true;                                                                                             \
    }                                                                                                              \
    geeps_launch_plain(lrn_maxpool_forward_kernel<HALF, K3S2>, grid, block, smem, st, (const bf16*)x, (bf16*)p, (uint8_t*)argmax,   \
                                                                       *g, cf, RO);                                \
  } while (0)
  const bool k3s2 = g->K == 3 && g->stride == 2;
  if (size == 3) { if (k3s2) LP_FWD(1, true); else LP_FWD(1, false); }
  else if (size == 5) { if (k3s2) LP_FWD(2, true); else LP_FWD(2, false); }
  else { if (k3s2) LP_FWD(3, true); else LP_FWD(3, false); }
#undef LP_FWD
  return (int)cudaGetLastError();
}

int geeps_lrn_maxpool_backward(const void* x, const void* dp, const void* argmax, void* dx, const GeepsPoolGeom* g,
                               int size, float alpha, float beta, float k, int relu_mask, float* colsum, void* stream) {
  if (!geeps_lrn_maxpool_supported(g, size)) return (int)cudaErrorInvalidValue;
  int R = lp_bwd_rows(g);
  while (R > 1 && lp_bwd_smem(g, R, lp_bwd_max_oh(g, R)) > kLpTwoPerSm) R >>= 1;   // two CTAs per SM where possible
  const int max_oh = lp_bwd_max_oh(g, R);
  const size_t smem = lp_bwd_smem(g, R, max_oh);
  const int block = lp_threads(g->C / 8, 512);
  const LrnCoef cf = make_coef(size, alpha, beta, k);
  const float coef = 2.f * alpha * beta / (float)size;
  cudaStream_t st = (cudaStream_t)stream;
  const int row_blocks = (g->H + R - 1) / R;
  const long long total = (long long)g->B * row_blocks;
  const int per_sm = smem <= kLpTwoPerSm ? 2 : 1;
  int grid = geeps_sm_count() * per_sm;
  if (grid > total) grid = (int)total;
  if (colsum != nullptr) geeps_clear_f32(colsum, g->C, st);
  const bool k3s2 = g->K == 3 && g->stride == 2;
  // the register kernel covers the usual pair (5 channels, 3 x 3 stride 2) up to 512 channels; its item count is 32 bits
  const int cv = g->C / 8;
  const int q0 = g->pad >> 1, QH = ((g->H - 1 + g->pad) >> 1) - q0 + 1, QW = ((g->W - 1 + g->pad) >> 1) - q0 + 1;
  const long long vectors = (long long)g->B * QH * QW * cv;
  // Below some 100 vectors an SM the lanes kernel has more warps at work (captured chains of 16, lanes / quads, us: 13 x 13 x 32
  // 2.5 / 3.6, 8 x 27 x 27 x 64 3.2 / 3.8, 3 x 33 x 33 x 88 3.7 / 3.8; above, 16 x 27 x 27 x 64 4.0 / 3.8, 64 x 13 x 13 x 40
  // 4.2 / 3.8, 2 x 55 x 55 x 96 3.9 / 3.8, 64 x 27 x 27 x 104 16.2 / 10.5); the quad kernel counts vectors in 32 bits.
  if (k3s2 && size == 5 && vectors >= 96LL * geeps_sm_count() && vectors < (1LL << 30)) {
    // a warp of several steps keeps its channels: then the warps' vectors are a multiple of a pixel's
    long long warps = (vectors + 29) / 30;
    const long long cap = (long long)geeps_sm_count() * 16;
    if (warps > cap) {
      int a = cv, b = 30;
      while (b) { const int t = a % b; a = b; b = t; }
      const int m = cv / a;                                   // 30 m vectors are whole pixels
      warps = m <= cap ? cap / m * m : m;
    }
    geeps_launch_plain(lrn_maxpool_backward_quad_kernel, (int)((warps + 7) / 8), 256, 0, st, (const bf16*)x, (const bf16*)dp,
                       (const uint8_t*)argmax, (bf16*)dx, *g, cf, coef, relu_mask, colsum, QH, QW, (int)vectors, (int)warps);
    return (int)cudaGetLastError();
  }
  if (k3s2 && size == 5 && cv <= 64 && (long long)g->B * g->H * (g->W + 64) < 0x7fffffffLL) {
    const LrnLanes ln = lrn_lanes(cv, (long long)g->B * g->H * g->W);
    const int lp = ln.lp, nv = ln.nv;
    const int ppw = 32 / lp, strips = ((g->W + 1) / 2 + ppw - 1) / ppw;
    long long blocks = ((long long)g->B * g->H * 2 * strips + 7) / 8;
    const long long cap = (long long)geeps_sm_count() * 2;
    if (blocks > cap) blocks = cap;
#define LP_LANES(LP, NV)                                                                                           \
  geeps_launch_plain(lrn_maxpool_backward_lanes_kernel<LP, NV>, (int)blocks, 256, sizeof(float) * g->C, st,                          \
      (const bf16*)x, (const bf16*)dp, (const uint8_t*)argmax, (bf16*)dx, *g, cf, coef, relu_mask, colsum)
    if (lp == 1) LP_LANES(1, 1);
    else if (lp == 2) { if (nv == 1) LP_LANES(2, 1); else LP_LANES(2, 3); }
    else if (lp == 4) { if (nv == 1) LP_LANES(4, 1); else if (nv == 2) LP_LANES(4, 2); else LP_LANES(4, 3); }
    else if (lp == 8) { if (nv == 2) LP_LANES(8, 2); else LP_LANES(8, 3); }
    else if (lp == 16) { if (nv == 2) LP_LANES(16, 2); else LP_LANES(16, 3); }
    else LP_LANES(32, 2);
#undef LP_LANES
    return (int)cudaGetLastError();
  }
#define LP_BWD(HALF, K3S2)                                                                                         \
  do {                                                                                                             \
    static bool attr_set = false;                                                                                  \
    if (!attr_set) {                                                                                               \
      cudaError_t e = cudaFuncSetAttribute(lrn_maxpool_backward_kernel<HALF, K3S2>,                                \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLpMaxSmem);          \
      if (e != cudaSuccess) return (int)e;                                                                         \
      attr_set = true;                                                                                             \
    }                                                                                                              \
    geeps_launch_plain(lrn_maxpool_backward_kernel<HALF, K3S2>, grid, block, smem, st, (const bf16*)x, (const bf16*)dp,             \
                                                                 (const uint8_t*)argmax, (bf16*)dx, *g, R, max_oh,  \
                                                                 cf, coef, relu_mask, colsum);                     \
  } while (0)
  if (size == 3) { if (k3s2) LP_BWD(1, true); else LP_BWD(1, false); }
  else if (size == 5) { if (k3s2) LP_BWD(2, true); else LP_BWD(2, false); }
  else { if (k3s2) LP_BWD(3, true); else LP_BWD(3, false); }
#undef LP_BWD
  return (int)cudaGetLastError();
}

}  // extern "C"
