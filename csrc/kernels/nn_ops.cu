// Training ops around the tensor-core GEMM, all on NHWC bf16 activations with fp32
// arithmetic: layout conversion, im2col / col2im (conv forward, data- and weight-gradient
// run as GEMMs on the patch matrix), BatchNorm, ReLU, LRN, max / average pooling,
// softmax cross-entropy, column sums (bias gradients) and dropout.
//
// The reference ships none of these (its Caffe application is an un-fetched submodule,
// .gitmodules:1-4 of the reference); layer maths follows the usual Caffe definitions so that
// the AlexNet / Inception-BN configurations behave as the originals did.
#include "common.cuh"
#include "kernels.h"
#include "nn_ops.h"

namespace {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float bf(const bf16 v) { return __bfloat162float(v); }

struct alignas(16) Bf8 { bf16 v[8]; };
__device__ __forceinline__ Bf8 ld8(const bf16* p) { Bf8 r; *reinterpret_cast<uint4*>(&r) = *reinterpret_cast<const uint4*>(p); return r; }
__device__ __forceinline__ Bf8 zero8() { Bf8 r; *reinterpret_cast<uint4*>(&r) = make_uint4(0u, 0u, 0u, 0u); return r; }
__device__ __forceinline__ void st8(bf16* p, const Bf8& r) { *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&r); }

// t = q * stride exactly?  Strides 1 and 2 (every layer of the supported nets but conv1) avoid the divider.
__device__ __forceinline__ bool div_exact(int t, int stride, int& q) {
  if (stride == 1) { q = t; return true; }
  if (stride == 2) { q = t >> 1; return (t & 1) == 0; }
  q = t / stride;
  return q * stride == t;
}

// 256 threads as (8-channel vectors of a pixel) x (pixels of a row)
inline dim3 pool_block(int cv) {
  int bx = cv < 1 ? 1 : (cv > 256 ? 256 : cv);
  int by = 256 / bx;
  return dim3(bx, by < 1 ? 1 : by, 1);
}

// Average pooling: up to 256 threads as (8-channel vectors of a pixel) x (pixels of a row, in even shares where it takes
// several blocks) x (rows, where two or more fit and `group` allows it).
// No rows or no pixels: an empty grid, nothing to launch.
struct PoolGrid { dim3 grid, block; };
inline PoolGrid avgpool_grid(int cv, int width, long long rows, bool group) {
  if (rows <= 0 || width <= 0) return {dim3(0, 0, 0), dim3(0, 0, 0)};
  const int bx = cv < 1 ? 1 : (cv > 256 ? 256 : cv), room = 256 / bx;
  const int parts = (width + room - 1) / room;
  const int by = (width + parts - 1) / parts;
  long long bz = group ? 256 / (bx * by) : 1;
  bz = bz > 64 ? 64 : (bz > rows ? rows : bz);
  if (bz < 1) bz = 1;
  PoolGrid g;
  g.block = dim3((unsigned)bx, (unsigned)by, (unsigned)bz);
  g.grid = dim3((unsigned)((rows + bz - 1) / bz), (unsigned)(parts > 65535 ? 65535 : parts), 1);   // the kernels stride over y
  return g;
}

inline int grid_1d(long long n, int block = 256, int cap = 0) {
  if (cap <= 0) cap = geeps_sm_count() * 16;
  long long b = (n + block - 1) / block;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

// ---------------- layout conversion ----------------
// The NCHW input batch is fp32 or bf16 (a host pipeline that ships bf16 halves the host-to-device bytes).
__device__ __forceinline__ float in_val(const float* p) { return __ldg(p); }
__device__ __forceinline__ float in_val(const bf16* p) { return __bfloat162float(*p); }

template <typename T>
__global__ void __launch_bounds__(256)
nchw_f32_to_nhwc_bf16_kernel(const T* __restrict__ x, bf16* __restrict__ y, int B, int C, int H, int W, int Cpad) {
  geeps_pdl_enter();
  const long long total = (long long)B * H * W * Cpad;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % Cpad);
    long long p = i / Cpad;
    const int w = (int)(p % W); p /= W;
    const int h = (int)(p % H);
    const int b = (int)(p / H);
    y[i] = __float2bfloat16(c < C ? in_val(x + (((long long)b * C + c) * H + h) * W + w) : 0.f);
  }
}

// ---------------- im2col / col2im (NHWC, one channel group) ----------------
// col[(b,oh,ow)][(kh,kw,c)] = x[b][oh*s-p+kh][ow*s-p+kw][c0+c]; row pitch ldcol >= KH*KW*Cg.
// One warp builds one row of the patch matrix at a time: the pixel coordinates are decoded once per row
// and the lanes sweep the row's vectors, so the address arithmetic is two 32-bit divisions per vector.
template <int VEC>
__global__ void __launch_bounds__(256)
im2col_kernel(const bf16* __restrict__ x, bf16* __restrict__ col, const GeepsConvGeom g) {
  geeps_pdl_enter();
  const int cv = g.Cg / VEC;
  const int per_kh = g.KW * cv;
  const int per_row = g.KH * per_kh;
  const long long rows = (long long)g.B * g.OH * g.OW;
  const int lane = threadIdx.x & 31;
  const long long warp0 = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long row = warp0; row < rows; row += nwarps) {
    const int ow = (int)(row % g.OW);
    const long long t = row / g.OW;
    const int oh = (int)(t % g.OH);
    const int b = (int)(t / g.OH);
    const int ih0 = oh * g.stride - g.pad, iw0 = ow * g.stride - g.pad;
    bf16* drow = col + row * g.ldcol;
    const bf16* xb = x + (long long)b * g.H * g.W * g.C + g.c0;
    for (int v = lane; v < per_row; v += 32) {
      const int kh = v / per_kh;
      const int rem = v - kh * per_kh;
      const int kw = rem / cv;
      const int c = (rem - kw * cv) * VEC;
      const int ih = ih0 + kh, iw = iw0 + kw;
      const bool in = ih >= 0 && ih < g.H && iw >= 0 && iw < g.W;
      bf16* dst = drow + (kh * g.KW + kw) * g.Cg + c;
      const bf16* src = xb + ((long long)ih * g.W + iw) * g.C + c;
      if (VEC == 8) {
        *reinterpret_cast<uint4*>(dst) = in ? *reinterpret_cast<const uint4*>(src) : make_uint4(0, 0, 0, 0);
      } else if (VEC == 4) {
        *reinterpret_cast<uint2*>(dst) = in ? *reinterpret_cast<const uint2*>(src) : make_uint2(0, 0);
      } else {
        *dst = in ? *src : __float2bfloat16(0.f);
      }
    }
  }
}

// Zero the pad columns [Kd, ldcol) of the patch matrix once (TMA reads them as K).
__global__ void zero_col_pad_kernel(bf16* col, long long rows, int kd, int ldcol) {
  geeps_pdl_enter();
  const int padw = ldcol - kd;
  const long long total = rows * padw;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride)
    col[(i / padw) * ldcol + kd + (i % padw)] = __float2bfloat16(0.f);
}

// dx[b][ih][iw][c0+c] (+)= sum over (kh,kw) windows covering (ih,iw) of dcol[(b,oh,ow)][(kh,kw,c)]
// Gather form: no atomics, deterministic.
template <int VEC>
__global__ void __launch_bounds__(256)
col2im_kernel(const bf16* __restrict__ dcol, bf16* __restrict__ dx, const GeepsConvGeom g, int accumulate) {
  geeps_pdl_enter();
  const int cv = g.Cg / VEC;
  const long long total = (long long)g.B * g.H * g.W * cv;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % cv) * VEC;
    long long p = i / cv;
    const int iw = (int)(p % g.W); p /= g.W;
    const int ih = (int)(p % g.H);
    const int b = (int)(p / g.H);
    float acc[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
    for (int kh = 0; kh < g.KH; ++kh) {
      const int th = ih + g.pad - kh;
      int oh, ow;
      if (th < 0 || !div_exact(th, g.stride, oh) || oh >= g.OH) continue;
      for (int kw = 0; kw < g.KW; ++kw) {
        const int tw = iw + g.pad - kw;
        if (tw < 0 || !div_exact(tw, g.stride, ow) || ow >= g.OW) continue;
        const bf16* src = dcol + (((long long)b * g.OH + oh) * g.OW + ow) * g.ldcol +
                          (long long)(kh * g.KW + kw) * g.Cg + c;
        if (VEC == 8) {
          Bf8 v = ld8(src);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += bf(v.v[e]);
        } else {
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[e] += bf(src[e]);
        }
      }
    }
    bf16* dst = dx + (((long long)b * g.H + ih) * g.W + iw) * g.C + g.c0 + c;
    if (VEC == 8) {
      Bf8 o;
      if (accumulate) { Bf8 old = ld8(dst);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += bf(old.v[e]); }
#pragma unroll
      for (int e = 0; e < 8; ++e) o.v[e] = __float2bfloat16(acc[e]);
      st8(dst, o);
    } else {
#pragma unroll
      for (int e = 0; e < VEC; ++e) dst[e] = __float2bfloat16(acc[e] + (accumulate ? bf(dst[e]) : 0.f));
    }
  }
}

// ---------------- per-channel work on a [P][C] (pitch ld) bf16 matrix ----------------
// How a block's threads cover the matrix: thread = (pixel row r, 8-channel slot), so a thread keeps its slot for every
// pixel it visits: per-channel constants are loaded once, sums stay in registers, and no item costs an integer
// division (bn_apply spent most of its 77 us on a 32 x 56 x 56 x 192 tensor there and on reloading its six
// constants per channel).
// A row of threads reads whole contiguous pixels.  Above 1024 channels the blocks of gridDim.x share the channels, 512 or
// fewer each, neighbouring blocks the same pixels.
struct SlotMap {
  int cvb, rows, row, slot, c;     // slots per block, pixel rows per block, this thread's row / slot / first channel
  bool on;
  long long p0, step;              // first pixel, pixels between two of this thread
  __device__ __forceinline__ explicit SlotMap(int C) {
    const int cv = C >> 3;
    cvb = (cv + (int)gridDim.x - 1) / (int)gridDim.x;
    rows = (int)blockDim.x / cvb;
    row = (int)threadIdx.x / cvb;
    slot = (int)threadIdx.x - row * cvb;
    const int gslot = (int)blockIdx.x * cvb + slot;
    c = gslot * 8;
    on = row < rows && gslot < cv;
    p0 = (long long)blockIdx.y * rows + row;
    step = (long long)gridDim.y * rows;
  }
};
struct SlotGrid { dim3 grid; int threads; size_t smem; };
// Launch shape: 256-ish threads as rows x slots, about `per_thread` pixels a thread (one batch of loads in flight), one
// pixel where more would leave seven SMs in eight without a block, at most `per_sm` blocks per SM.  smem: the block's
// partial sums, nq floats per channel and pixel row.
// At most 64 slots a block above 128: a block then has four rows or more, whose sums meet before they go to memory, and
// nearly all of its threads a slot (one row of 161 slots leaves 31 of 192 idle).  Against one row of up to 256 slots:
// column sums of 100352 x 1032 55 -> 39 us, ReLU mask + sums of 20000 x 1288 42 -> 32 us, BatchNorm backward of 32 x 4096
// 12.5 -> 6.1 us, of 3000 x 2056 35 -> 22 us; up to 128 slots a block lie between the two.  (Mask + sums of
// 100352 x 1032 109 -> 114 us, bound by DRAM.)
inline SlotGrid slot_grid(long long P, int C, int per_thread, int per_sm, int nq) {
  const int cv = C / 8 < 1 ? 1 : C / 8;
  SlotGrid g;
  const int chunks = cv <= 128 ? 1 : (cv + 63) / 64;                // block columns
  const int cvb = (cv + chunks - 1) / chunks;
  const int rows = 256 / cvb;
  g.threads = (rows * cvb + 31) / 32 * 32;
  const int rows_used = g.threads / cvb;        // as SlotMap computes it
  const long long one_each = (P + rows_used - 1) / rows_used;      // blocks at one pixel a thread
  const long long fill = geeps_sm_count() / chunks;
  long long want = (one_each + per_thread - 1) / per_thread;
  if (want * 8 < fill) want = one_each < fill ? one_each : fill;
  const long long cap = (long long)geeps_sm_count() * per_sm / chunks;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  g.grid = dim3((unsigned)chunks, (unsigned)want, 1);
  g.smem = (size_t)rows_used * cvb * 8 * nq * sizeof(float);
  return g;
}
// Sum the threads' partial sums over the block's pixel rows and add them to out[channel] (+ out[C + channel]).  The
// rows meet in shared memory as plain stores: float atomics on shared memory are compare-and-swap loops, and 16 of
// them per thread were most of the 12 us a reduction of a 6272 x 160 matrix took.
template <int NQ>
__device__ __forceinline__ void slot_sums(const SlotMap& m, const float (&a0)[8], const float (&a1)[8], float* out, int C,
                                          float scale, float* part) {
  const int width = m.cvb * 8;
  if (m.row < m.rows) {
    float* d = part + (size_t)m.row * width * NQ + m.slot * 8;
    *reinterpret_cast<float4*>(d) = make_float4(a0[0], a0[1], a0[2], a0[3]);
    *reinterpret_cast<float4*>(d + 4) = make_float4(a0[4], a0[5], a0[6], a0[7]);
    if (NQ == 2) {
      *reinterpret_cast<float4*>(d + width) = make_float4(a1[0], a1[1], a1[2], a1[3]);
      *reinterpret_cast<float4*>(d + width + 4) = make_float4(a1[4], a1[5], a1[6], a1[7]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < width * NQ; i += blockDim.x) {
    float v = 0.f;
    for (int r = 0; r < m.rows; ++r) v += part[(size_t)r * width * NQ + i];
    const int q = NQ == 2 && i >= width ? 1 : 0;
    const int ch = (int)blockIdx.x * width + i - q * width;
    if (ch < C) atomicAdd(out + (size_t)q * C + ch, v * scale);
  }
}

// The pixels p0, p0 + step, ... below P in batches whose loads are in flight together: U at a time, and what is left over in
// batches of halves of it (a wait each, where single pixels would wait U - 1 times).  batch(count, first pixel)
template <int N> struct Count { static constexpr int value = N; };
template <int U, typename Fn>
__device__ __forceinline__ void pixel_batches(long long p, long long step, long long P, Fn batch) {
  for (; p + (U - 1) * step < P; p += U * step) batch(Count<U>(), p);
  if constexpr (U > 4) if (p + 3 * step < P) { batch(Count<4>(), p); p += 4 * step; }
  if constexpr (U > 2) if (p + step < P) { batch(Count<2>(), p); p += 2 * step; }
  if (U > 1 && p < P) batch(Count<1>(), p);
}

// Per-channel constants of a block's slots meet in shared memory ([n][8 * slots]): computed or loaded once per block with
// coalesced reads, then eight consecutive ones per thread.  Read from global memory by every thread (32 bytes apart per
// lane) they were 39 of the 52 us of a 32 x 56 x 56 x 192 normalisation.
template <int N, typename Fn>
__device__ __forceinline__ void slot_consts(const SlotMap& s, int C, float* sh, float (&v)[N][8], Fn fn) {
  const int width = s.cvb * 8, c0 = (int)blockIdx.x * width;
  for (int i = threadIdx.x; i < width && c0 + i < C; i += blockDim.x) {
    float o[N];
    fn(c0 + i, o);
#pragma unroll
    for (int n = 0; n < N; ++n) sh[n * width + i] = o[n];
  }
  __syncthreads();
  if (s.on) {
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const float4 a = *reinterpret_cast<const float4*>(sh + n * width + s.slot * 8);
      const float4 b = *reinterpret_cast<const float4*>(sh + n * width + s.slot * 8 + 4);
      v[n][0] = a.x; v[n][1] = a.y; v[n][2] = a.z; v[n][3] = a.w; v[n][4] = b.x; v[n][5] = b.y; v[n][6] = b.z; v[n][7] = b.w;
    }
  }
}

// MODE 0: out[c] += sum x, out[C+c] += sum x^2                  (BN forward statistics)
// MODE 1: out[c] += sum dy', out[C+c] += sum dy' * xhat          (BN backward; dy' = dy masked by y>0 if relu)
// MODE 2: out[c] += scale * sum x                                (bias gradient)
// MODE 3: as 1, dy' = dy where the forward pass left a bit (y then points to the bit bytes, one per 8-channel vector)
template <int MODE>
__device__ __forceinline__ void channel_reduce_body(const bf16* __restrict__ x, const bf16* __restrict__ dy,
                                                    const bf16* __restrict__ y, const float* __restrict__ mean_rstd,
                                                    float* __restrict__ out, long long P, int C, long long ldx,
                                                    long long lddy, int relu, float scale) {
  extern __shared__ __align__(16) float sacc[];  // [rows][(1 or 2) * 8 * slots]
  constexpr bool BWD = MODE == 1 || MODE == 3;
  const uint8_t* bits = reinterpret_cast<const uint8_t*>(y);
  const long long cv = C >> 3;
  const SlotMap m(C);
  float a0[8], a1[8], mr[2][8];
#pragma unroll
  for (int e = 0; e < 8; ++e) { a0[e] = 0.f; a1[e] = 0.f; }
  if (BWD) {
    slot_consts(m, C, sacc, mr, [&](int c, float (&o)[2]) { o[0] = mean_rstd[c]; o[1] = mean_rstd[C + c]; });
    __syncthreads();              // the partial sums go to the same shared memory
  }
  if (m.on) {
    auto add = [&](const Bf8& xv, const Bf8& dv, const Bf8& yv, uint32_t on) {
      if (BWD) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float d = bf(dv.v[e]);
          if (MODE == 3 ? !(on >> e & 1u) : relu && !(bf(yv.v[e]) > 0.f)) d = 0.f;
          a0[e] += d;
          a1[e] += d * (bf(xv.v[e]) - mr[0][e]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) { const float f = bf(xv.v[e]); a0[e] += f; if (MODE == 0) a1[e] += f * f; }
      }
    };
    // two pixels where there are three tensors to load: four took 153 registers, one block per SM (BatchNorm backward of
    // 100352 x 192 by its output 73 us, 56 with two)
    pixel_batches<MODE == 1 ? 2 : MODE == 3 ? 4 : 8>(m.p0, m.step, P, [&](auto count, long long p) {
      constexpr int U = decltype(count)::value;
      Bf8 xv[U], dv[U], yv[U];
      uint32_t on[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        xv[u] = ld8(x + (p + u * m.step) * ldx + m.c);
        on[u] = 0u;
        if (BWD) dv[u] = ld8(dy + (p + u * m.step) * lddy + m.c);
        if (MODE == 3) on[u] = bits[(p + u * m.step) * cv + (m.c >> 3)];
        if (MODE == 1) {
          if (relu) yv[u] = ld8(y + (p + u * m.step) * lddy + m.c);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) add(xv[u], dv[u], yv[u], on[u]);
    });
    if (BWD) {
#pragma unroll
      for (int e = 0; e < 8; ++e) a1[e] *= mr[1][e];
    }
  }
  slot_sums<MODE == 2 ? 1 : 2>(m, a0, a1, out, C, MODE == 2 ? scale : 1.f, sacc);
}
// Blocks per SM of the channel kernels (launch bounds and grids).  Two with eight pixels of a thread in flight (four where
// there are two tensors to load, two where there are three) instead of four with four: the same bytes in flight, half the
// atomics and constants.  BatchNorm with ReLU bits, forward and backward, us: 100352 x 192 61.3 -> 57.4, 25088 x 192 24.5 ->
// 22.0, 25088 x 320 32.2 -> 28.7, 25600 x 144 22.8 -> 20.0, 50000 x 48 18.1 -> 15.7, 6272 x 160 12.8 -> 11.8; one block per SM
// with eight pixels of the sums 62.1, 20.9, 28.3, 18.4, 16.4, 12.8.
constexpr int kChannelBlocks = 2;
// The kernels of a BatchNorm fill the SMs' registers.  Blocks of the next one that come up while the last of this are running
// lie two to the SMs that were done first, and its own end is as ragged, so over a large tensor they wait for the end.
// Forward and backward, us, next blocks at once / at the end: 100352 x 192 57.5 / 55.4, x 128 37.4 / 33.8, x 64 22.1 / 21.2,
// 300000 x 32 28.1 / 26.5, 25088 x 320 29.2 / 27.7, x 192 22.1 / 21.7, 6272 x 160 12.2 / 12.3.  In a module of branches the
// small ones lose by it, since other branches have the SMs meanwhile (32 x 14 x 14 178.4 / 181.3, 7 x 7 99.4 / 104.9).
__device__ __forceinline__ void batchnorm_enter(long long P, int C) {
  geeps_pdl_wait();
  if (P * C <= 5LL << 20) geeps_pdl_trigger();
}
enum { MASK_NONE = 0, MASK_Y = 1, MASK_BITS = 2 };      // what the backward pass reads a ReLU mask from
template <int MODE>
__global__ void __launch_bounds__(256, kChannelBlocks)
channel_reduce_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dy, const bf16* __restrict__ y,
                      const float* __restrict__ mean_rstd, float* __restrict__ out, long long P, int C,
                      long long ldx, long long lddy, int relu, float scale) {
  if (MODE == 2) geeps_pdl_enter(); else batchnorm_enter(P, C);
  channel_reduce_body<MODE>(x, dy, y, mean_rstd, out, P, C, ldx, lddy, relu, scale);
}

// any C, any pitch: one thread per column (small P: FC bias gradients with odd widths)
__global__ void colsum_simple_kernel(const bf16* __restrict__ x, float* __restrict__ out, long long P, int C,
                                     long long ldx, float scale, int accumulate) {
  geeps_pdl_enter();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float a = 0.f;
  for (long long p = 0; p < P; ++p) a += bf(x[p * ldx + c]);
  out[c] = a * scale + (accumulate ? out[c] : 0.f);
}

// sums -> mean / rstd (+ running statistics with Caffe-style moving average); in place where sums == mean_rstd: a thread
// reads its two sums before it writes its two results
__global__ void bn_finalize_kernel(const float* sums, float* mean_rstd,
                                   float* running_mean, float* running_var, int C, float inv_count, float eps,
                                   float momentum) {
  geeps_pdl_enter();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const float m = sums[c] * inv_count;
  float var = sums[C + c] * inv_count - m * m;
  var = fmaxf(var, 0.f);
  mean_rstd[c] = m;
  mean_rstd[C + c] = rsqrtf(var + eps);
  if (running_mean) {
    running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * m;
    running_var[c] = (1.f - momentum) * running_var[c] + momentum * var;
  }
}

// y = (x - m) * k + b, k = gamma / std, through ReLU where asked: the pixel loop of both normalisation kernels.
// bits (optional): one byte per 8-channel vector with bit e set where y[e] > 0, all that the ReLU backward needs of y.
__device__ __forceinline__ void bn_apply_pixels(const SlotMap& s, const bf16* __restrict__ x, bf16* __restrict__ y,
                                                const float (&mkb)[3][8], long long P,
                                                long long ldx, long long ldy, int relu, uint8_t* bits, int cv) {
  auto mark = [&](long long p, const Bf8& o) {
    uint32_t on = 0u;
#pragma unroll
    for (int e = 0; e < 8; ++e) on |= bf(o.v[e]) > 0.f ? 1u << e : 0u;
    bits[p * cv + (s.c >> 3)] = (uint8_t)on;
  };
  auto one = [&](const Bf8& v) {
    Bf8 o;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float f = fmaf(bf(v.v[e]) - mkb[0][e], mkb[1][e], mkb[2][e]);
      if (relu) f = fmaxf(f, 0.f);
      o.v[e] = __float2bfloat16(f);
    }
    return o;
  };
  pixel_batches<8>(s.p0, s.step, P, [&](auto count, long long p) {
    constexpr int U = decltype(count)::value;
    Bf8 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = ld8(x + (p + u * s.step) * ldx + s.c);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const Bf8 o = one(v[u]);
      st8(y + (p + u * s.step) * ldy + s.c, o);
      if (bits) mark(p + u * s.step, o);
    }
  });
}

__global__ void __launch_bounds__(256)
bn_apply_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, const float* __restrict__ mean_rstd,
                const float* __restrict__ gamma, const float* __restrict__ beta, long long P, int C,
                long long ldx, long long ldy, int relu) {
  geeps_pdl_enter();
  extern __shared__ __align__(16) float sacc[];
  const SlotMap s(C);
  float mkb[3][8];
  slot_consts(s, C, sacc, mkb, [&](int c, float (&o)[3]) { o[0] = mean_rstd[c]; o[1] = mean_rstd[C + c] * gamma[c]; o[2] = beta[c]; });
  if (!s.on) return;
  bn_apply_pixels(s, x, y, mkb, P, ldx, ldy, relu, nullptr, 0);
}

// Normalisation with the statistics finalised inside: every block derives mean and 1/std of its channels from
// the channel sums (no separate finalisation launch); the blocks of the first pixels also store mean / rstd for the
// backward pass, update the running statistics and zero `zero_after` (2 C floats: the scratch of the NEXT reduction
// of this layer, e.g. the backward one, so that no memset node sits in front of it).
__device__ __forceinline__ void bn_apply_fused_body(const bf16* __restrict__ x, bf16* __restrict__ y,
                                                    const float* sums, float* mean_rstd,
                                                    float* running_mean, float* running_var,
                                                    const float* __restrict__ gamma, const float* __restrict__ beta,
                                                    float* zero_after, long long P, int C, long long ldx, long long ldy,
                                                    int relu, float inv_count, float eps, float momentum, uint8_t* bits) {
  extern __shared__ __align__(16) float sacc[];
  const SlotMap s(C);
  float mkb[3][8];
  slot_consts(s, C, sacc, mkb, [&](int c, float (&o)[3]) {
    const float m = sums[c] * inv_count;
    const float var = fmaxf(sums[C + c] * inv_count - m * m, 0.f);
    const float r = rsqrtf(var + eps);
    o[0] = m; o[1] = r * gamma[c]; o[2] = beta[c];
    if (blockIdx.y == 0 && P > 0) {
      mean_rstd[c] = m;
      mean_rstd[C + c] = r;
      if (running_mean) {
        running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * m;
        running_var[c] = (1.f - momentum) * running_var[c] + momentum * var;
      }
      if (zero_after) { zero_after[c] = 0.f; zero_after[C + c] = 0.f; }
    }
  });
  if (!s.on) return;
  bn_apply_pixels(s, x, y, mkb, P, ldx, ldy, relu, bits, C >> 3);
}
__global__ void __launch_bounds__(256, kChannelBlocks)
bn_apply_fused_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, const float* __restrict__ sums,
                      float* __restrict__ mean_rstd, float* running_mean, float* running_var,
                      const float* __restrict__ gamma, const float* __restrict__ beta, float* zero_after, long long P,
                      int C, long long ldx, long long ldy, int relu, float inv_count, float eps, float momentum, uint8_t* bits) {
  batchnorm_enter(P, C);
  bn_apply_fused_body(x, y, sums, mean_rstd, running_mean, running_var, gamma, beta, zero_after, P, C, ldx, ldy, relu,
                      inv_count, eps, momentum, bits);
}

// dx = gamma * rstd * (dy' - sum_dy/P - xhat * sum_dy_xhat/P); also emits dgamma, dbeta (scaled).
template <int MASK>
__device__ __forceinline__ void bn_backward_body(const bf16* __restrict__ x, const bf16* __restrict__ dy,
                                                 const bf16* __restrict__ y, bf16* __restrict__ dx,
                                                 const float* mean_rstd, const float* __restrict__ gamma,
                                                 const float* sums, float* dgamma, float* dbeta, long long P, int C,
                                                 long long ldx, long long lddy, long long lddx, int relu,
                                                 float grad_scale, float* zero_after) {
  extern __shared__ __align__(16) float sacc[];
  const uint8_t* bits = reinterpret_cast<const uint8_t*>(y);
  const long long cv = C >> 3;
  const SlotMap s(C);
  const float invP = 1.f / (float)P;
  float q[4][8];                    // mean, gamma / std, sum_dy / P, sum_dy_xhat / (P std)
  slot_consts(s, C, sacc, q, [&](int c, float (&o)[4]) {
    const float rs = mean_rstd[C + c], s0 = sums[c], s1 = sums[C + c];
    o[0] = mean_rstd[c]; o[1] = gamma[c] * rs; o[2] = s0 * invP; o[3] = rs * (s1 * invP);
    if (blockIdx.y == 0) {
      if (dbeta) dbeta[c] = s0 * grad_scale;
      if (dgamma) dgamma[c] = s1 * grad_scale;
      // the scratch of this layer's next forward reduction (nobody reads it during the backward pass)
      if (zero_after) { zero_after[c] = 0.f; zero_after[C + c] = 0.f; }
    }
  });
  if (!s.on) return;
  auto one = [&](const Bf8& xv, const Bf8& dv, const Bf8& yv, uint32_t on) {
    Bf8 o;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float d = bf(dv.v[e]);
      if (MASK == MASK_BITS ? !(on >> e & 1u) : MASK == MASK_Y && relu && !(bf(yv.v[e]) > 0.f)) d = 0.f;
      o.v[e] = __float2bfloat16(q[1][e] * (d - q[2][e] - (bf(xv.v[e]) - q[0][e]) * q[3][e]));
    }
    return o;
  };
  pixel_batches<MASK == MASK_Y ? 2 : 4>(s.p0, s.step, P, [&](auto count, long long p) {
    constexpr int U = decltype(count)::value;
    Bf8 xv[U], dv[U], yv[U];
    uint32_t on[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      xv[u] = ld8(x + (p + u * s.step) * ldx + s.c);
      dv[u] = ld8(dy + (p + u * s.step) * lddy + s.c);
      on[u] = MASK == MASK_BITS ? bits[(p + u * s.step) * cv + (s.c >> 3)] : 0u;
      if (MASK == MASK_Y && relu) yv[u] = ld8(y + (p + u * s.step) * lddy + s.c);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) st8(dx + (p + u * s.step) * lddx + s.c, one(xv[u], dv[u], yv[u], on[u]));
  });
}
template <int MASK>
__global__ void __launch_bounds__(256, kChannelBlocks)
bn_backward_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dy, const bf16* __restrict__ y,
                   bf16* __restrict__ dx, const float* __restrict__ mean_rstd, const float* __restrict__ gamma,
                   const float* __restrict__ sums, float* dgamma, float* dbeta, long long P, int C,
                   long long ldx, long long lddy, long long lddx, int relu, float grad_scale, float* zero_after) {
  batchnorm_enter(P, C);
  bn_backward_body<MASK>(x, dy, y, dx, mean_rstd, gamma, sums, dgamma, dbeta, P, C, ldx, lddy, lddx, relu, grad_scale,
                         zero_after);
}

// ---- one launch per direction: reduction, grid barrier, normalisation (cooperative launch: all blocks resident) ----
// bar[0] counts arrivals, bar[1] counts blocks that are done (the last one resets both for the next launch), bar[2]
// is set when a block gave up waiting (it then skips the second phase: the output stays stale and mean_rstd[0] is
// made NaN so that the failure shows in the loss).
__device__ __forceinline__ bool bn_grid_barrier(int* bar, int nblocks) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1);
    s_ok = geeps_wait_ge(bar, nblocks, 1000000000ull, nullptr) ? 1 : 0;
    __threadfence();
  }
  __syncthreads();
  return s_ok != 0;
}
__device__ __forceinline__ void bn_grid_done(int* bar, int nblocks) {
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(bar + 1, 1) == nblocks - 1) {
    bar[0] = 0; bar[1] = 0;
    __threadfence();
  }
}
__global__ void __launch_bounds__(256)
bn_forward_coop_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, float* sums, float* mean_rstd,
                       float* running_mean, float* running_var, const float* __restrict__ gamma,
                       const float* __restrict__ beta, float* zero_after, int* bar, long long P, int C, long long ldx,
                       long long ldy, int relu, float inv_count, float eps, float momentum, uint8_t* bits) {
  geeps_pdl_enter();
  channel_reduce_body<0>(x, nullptr, nullptr, nullptr, sums, P, C, ldx, 0, 0, 1.f);
  if (bn_grid_barrier(bar, (int)(gridDim.x * gridDim.y)))
    bn_apply_fused_body(x, y, sums, mean_rstd, running_mean, running_var, gamma, beta, zero_after, P, C, ldx, ldy, relu,
                        inv_count, eps, momentum, bits);
  else if (threadIdx.x == 0) { bar[2] = 1; mean_rstd[0] = __int_as_float(0x7fc00000); }
  bn_grid_done(bar, (int)(gridDim.x * gridDim.y));
}
template <bool BITS>      // y points to the mask bits
__global__ void __launch_bounds__(256)
bn_backward_coop_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dy, const bf16* __restrict__ y,
                        bf16* __restrict__ dx, float* mean_rstd, const float* __restrict__ gamma, float* sums,
                        float* dgamma, float* dbeta, float* zero_after, int* bar, long long P, int C, long long ldx,
                        long long lddy, long long lddx, int relu, float grad_scale) {
  geeps_pdl_enter();
  channel_reduce_body<BITS ? 3 : 1>(x, dy, y, mean_rstd, sums, P, C, ldx, lddy, relu, 1.f);
  if (bn_grid_barrier(bar, (int)(gridDim.x * gridDim.y)))
    bn_backward_body<BITS ? MASK_BITS : MASK_Y>(x, dy, y, dx, mean_rstd, gamma, sums, dgamma, dbeta, P, C, ldx, lddy, lddx,
                                                relu, grad_scale, zero_after);
  else if (threadIdx.x == 0) { bar[2] = 1; mean_rstd[0] = __int_as_float(0x7fc00000); }
  bn_grid_done(bar, (int)(gridDim.x * gridDim.y));
}

// ---------------- ReLU backward / dropout ----------------
__global__ void __launch_bounds__(256)
relu_backward_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ y, bf16* __restrict__ dx, long long n8) {
  geeps_pdl_enter();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += stride) {
    Bf8 d = ld8(dy + i * 8), v = ld8(y + i * 8), o;
#pragma unroll
    for (int e = 0; e < 8; ++e) o.v[e] = bf(v.v[e]) > 0.f ? d.v[e] : __float2bfloat16(0.f);
    st8(dx + i * 8, o);
  }
}

// 2-D variant with row pitches (channel slices of concat tensors)
__global__ void __launch_bounds__(256)
relu_backward_2d_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ y, bf16* __restrict__ dx, long long P,
                        int C, long long lddy, long long ldy, long long lddx) {
  geeps_pdl_enter();
  const int cv = C >> 3;
  const long long total = P * cv;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % cv) * 8;
    const long long p = i / cv;
    Bf8 d = ld8(dy + p * lddy + c), v = ld8(y + p * ldy + c), o;
#pragma unroll
    for (int e = 0; e < 8; ++e) o.v[e] = bf(v.v[e]) > 0.f ? d.v[e] : __float2bfloat16(0.f);
    st8(dx + p * lddx + c, o);
  }
}
// dst = bf16(relu ? max(src, 0) : src) over a [P][C] fp32 matrix with row pitches: the finishing pass of a split-K
// GEMM whose partial sums were reduce-added in fp32
__global__ void __launch_bounds__(256)
f32_to_bf16_2d_kernel(const float* __restrict__ src, bf16* __restrict__ dst, long long P, int C, long long lds,
                      long long ldd, int relu) {
  geeps_pdl_enter();
  const int cv = C >> 3;
  const long long total = P * cv;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const float lo = relu ? 0.f : -INFINITY;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % cv) * 8;
    const long long p = i / cv;
    const float4 a = *reinterpret_cast<const float4*>(src + p * lds + c);
    const float4 b = *reinterpret_cast<const float4*>(src + p * lds + c + 4);
    *reinterpret_cast<uint4*>(dst + p * ldd + c) =
        make_uint4(pack_bf16x2(fmaxf(a.x, lo), fmaxf(a.y, lo)), pack_bf16x2(fmaxf(a.z, lo), fmaxf(a.w, lo)),
                   pack_bf16x2(fmaxf(b.x, lo), fmaxf(b.y, lo)), pack_bf16x2(fmaxf(b.z, lo), fmaxf(b.w, lo)));
  }
}
// ReLU backward fused with the per-channel sums of its result (the bias gradient of the layer whose output y is):
// dx = y > 0 ? dy : 0, out[c] += sum over pixels of dx.  Four blocks per SM with eight pixels of a thread in flight; eight with
// four: 43264 x 384 22.3 us, 18.0 now, 43264 x 256 16.4, 12.4, 186624 x 256 53.4, 50.9 (of which 44 are the bytes).
// `clear`: the weight gradient that the next kernels add to, zeroed on the way.
__global__ void __launch_bounds__(256)
relu_backward_colsum_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ y, bf16* __restrict__ dx,
                            float* __restrict__ out, long long P, int C, long long lddy, long long ldy, long long lddx,
                            float* __restrict__ clear, long long clear_n, int clear_head) {
  geeps_pdl_enter();
  extern __shared__ __align__(16) float sacc[];  // [rows][8 * slots]
  clear_range(clear, clear_n, clear_head, ((long long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x,
              (long long)gridDim.y * gridDim.x * blockDim.x);
  const SlotMap m(C);
  float a[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) a[e] = 0.f;
  if (m.on) {
    auto one = [&](const Bf8& d, const Bf8& v) {
      Bf8 o;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const bool on = bf(v.v[e]) > 0.f;
        o.v[e] = on ? d.v[e] : __float2bfloat16(0.f);
        a[e] += on ? bf(d.v[e]) : 0.f;
      }
      return o;
    };
    pixel_batches<8>(m.p0, m.step, P, [&](auto count, long long p) {
      constexpr int U = decltype(count)::value;
      Bf8 d[U], v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        d[u] = ld8(dy + (p + u * m.step) * lddy + m.c);
        v[u] = ld8(y + (p + u * m.step) * ldy + m.c);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) st8(dx + (p + u * m.step) * lddx + m.c, one(d[u], v[u]));
    });
  }
  slot_sums<1>(m, a, a, out, C, 1.f, sacc);
}
// dst += the sum of N sources over 2-D views (branch gradients): one pass and one rounding for up to three of them
struct AddSrc { const bf16* p[3]; long long ld[3]; };
// One vector per thread and step over the whole matrix; a dense one (every pitch equal to C) needs no coordinates.  Bound
// by memory.  One source of 6272 x 576: a 64-bit division per vector 4.2 us, a thread that keeps its channels (and its
// pixels one after the other) 5.1, this 3.7, pitched 4.1; three sources 5.1 -> 3.7 us.
template <int N, bool DENSE>
__global__ void __launch_bounds__(256)
add_2d_kernel(bf16* __restrict__ dst, const AddSrc src, long long total, int cv, long long ldd) {
  geeps_pdl_enter();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    // a pixel number of 32 bits is found by a 32-bit division
    const long long p = DENSE ? 0 : (total <= 0xffffffffLL ? (long long)((unsigned)i / (unsigned)cv) : i / cv);
    const long long c = (i - p * cv) * 8;
    Bf8 a = ld8(dst + p * ldd + c), v[N], o;
#pragma unroll
    for (int n = 0; n < N; ++n) v[n] = ld8(src.p[n] + p * src.ld[n] + c);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float f = bf(a.v[e]);
#pragma unroll
      for (int n = 0; n < N; ++n) f += bf(v[n].v[e]);
      o.v[e] = __float2bfloat16(f);
    }
    st8(dst + p * ldd + c, o);
  }
}

__device__ __forceinline__ uint32_t mix32(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return (uint32_t)((z ^ (z >> 31)) >> 32);
}
// y = x * keep(seed, idx) / (1 - p); the same call with dy as input gives dx.  VEC: eight values a thread and step (n a
// multiple of 8, both pointers on 16 bytes): fewer, wider accesses and an eighth of the blocks, which also have to find room
// beside a parameter push that holds half of every SM.  256 x 4096 5.4 -> 2.9 us, 6.5 M values 12.8 -> 9.5.
template <bool VEC>
__global__ void __launch_bounds__(256)
dropout_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, long long n, float p, unsigned long long seed,
               const int* __restrict__ step_ref) {
  geeps_pdl_enter();
  if (step_ref != nullptr) seed += (unsigned long long)(long long)*step_ref;
  const float inv = 1.f / (1.f - p);
  const uint32_t thresh = (uint32_t)(p * 4294967296.0);
  auto one = [&](bf16 v, long long i) {
    return mix32(seed * 0x100000001B3ull + (uint64_t)i) >= thresh ? __float2bfloat16(bf(v) * inv) : __float2bfloat16(0.f);
  };
  const long long stride = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (VEC) {
    for (long long i = first * 8; i < n; i += stride * 8) {
      Bf8 v = ld8(x + i);
#pragma unroll
      for (int e = 0; e < 8; ++e) v.v[e] = one(v.v[e], i + e);
      st8(y + i, v);
    }
  } else {
    for (long long i = first; i < n; i += stride) y[i] = one(x[i], i);
  }
}

// ---------------- LRN across channels ----------------
// Forward keeps r = 1 / scale per element in bf16 for the backward pass (scale = k + alpha/n * window sum of x^2):
// half the bytes of an fp32 scale buffer in both directions, and the backward needs 1/scale (for dy*y/scale) and
// scale^-beta = r^beta only.
__global__ void __launch_bounds__(256)
lrn_forward_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, bf16* __restrict__ scale, long long P, int C,
                   int size, float alpha, float beta, float k) {
  geeps_pdl_enter();
  const long long total = P * C;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int half = size / 2;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % C);
    const bf16* row = x + (i - c);
    float s = 0.f;
    const int lo = max(0, c - half), hi = min(C - 1, c + half);
    for (int j = lo; j <= hi; ++j) { float f = bf(row[j]); s += f * f; }
    const float sc = k + alpha / (float)size * s;
    scale[i] = __float2bfloat16(__frcp_rn(sc));
    y[i] = __float2bfloat16(bf(row[c]) * __powf(sc, -beta));
  }
}
__global__ void __launch_bounds__(256)
lrn_backward_kernel(const bf16* __restrict__ x, const bf16* __restrict__ y, const bf16* __restrict__ scale,
                    const bf16* __restrict__ dy, bf16* __restrict__ dx, long long P, int C, int size, float alpha,
                    float beta, int relu_mask) {
  geeps_pdl_enter();
  const long long total = P * C;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int half = size / 2;
  const float coef = 2.f * alpha * beta / (float)size;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % C);
    const long long base = i - c;
    float acc = 0.f;
    const int lo = max(0, c - half), hi = min(C - 1, c + half);
    for (int j = lo; j <= hi; ++j) acc += bf(dy[base + j]) * bf(y[base + j]) * bf(scale[base + j]);
    const float xi = bf(x[i]);
    const float d = bf(dy[i]) * __powf(bf(scale[i]), beta) - coef * xi * acc;
    dx[i] = __float2bfloat16((relu_mask && xi <= 0.f) ? 0.f : d);
  }
}

// Vector forms: one thread owns 8 consecutive channels of a pixel and slides the window over the
// 24 channels around them (window half-width <= 8); each squared value / ratio is computed once.
template <int HALF>
__global__ void __launch_bounds__(256)
lrn_forward_v8_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, bf16* __restrict__ scale, long long P, int C,
                      int size, float alpha, float beta, float k) {
  geeps_pdl_enter();
  const int cv = C >> 3;
  const long long total = P * cv;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const float a_n = alpha / (float)size;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % cv) * 8;
    const long long base = (i / cv) * C;
    float sq[24];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      const int cc = c + (v - 1) * 8;
      if (cc >= 0 && cc < C) {
        Bf8 t = ld8(x + base + cc);
#pragma unroll
        for (int e = 0; e < 8; ++e) { float f = bf(t.v[e]); sq[v * 8 + e] = v == 1 ? f : f * f; }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) sq[v * 8 + e] = 0.f;
      }
    }
    float xv[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) { xv[e] = sq[8 + e]; sq[8 + e] = xv[e] * xv[e]; }
    Bf8 o, r;
    float s = 0.f;       // sliding window over the 2*HALF+1 channels around output e
#pragma unroll
    for (int j = 8 - HALF; j <= 8 + HALF; ++j) s += sq[j];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sc = k + a_n * s;
      o.v[e] = __float2bfloat16(xv[e] * __powf(sc, -beta));
      r.v[e] = __float2bfloat16(__frcp_rn(sc));
      if (e < 7) s += sq[8 + e + HALF + 1] - sq[8 + e - HALF];
    }
    st8(y + base + c, o);
    st8(scale + base + c, r);
  }
}
template <int HALF>
__global__ void __launch_bounds__(256)
lrn_backward_v8_kernel(const bf16* __restrict__ x, const bf16* __restrict__ y, const bf16* __restrict__ scale,
                       const bf16* __restrict__ dy, bf16* __restrict__ dx, long long P, int C, int size, float alpha,
                       float beta, int relu_mask, float* __restrict__ colsum) {
  geeps_pdl_enter();
  // colsum (optional): per-channel sums of dx over all pixels - the bias gradient of the convolution whose
  // ReLU is folded in here.  The host sizes the grid so that gridDim * blockDim is a multiple of C/8: every
  // thread then keeps one channel group for all its pixels and sums in registers.
  extern __shared__ float lrn_cs[];
  const int cv = C >> 3;
  const long long total = P * cv;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const float coef = 2.f * alpha * beta / (float)size;
  float cs[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) cs[e] = 0.f;
  if (colsum != nullptr) {
    for (int j = threadIdx.x; j < C; j += blockDim.x) lrn_cs[j] = 0.f;
    __syncthreads();
  }
  const int c_fixed = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) % cv) * 8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % cv) * 8;
    const long long base = (i / cv) * C;
    float ratio[24], dyc[8], scc[8];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      const int cc = c + (v - 1) * 8;
      if (cc >= 0 && cc < C) {
        Bf8 d = ld8(dy + base + cc), yy = ld8(y + base + cc), rr = ld8(scale + base + cc);   // rr = 1 / scale
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          ratio[v * 8 + e] = bf(d.v[e]) * bf(yy.v[e]) * bf(rr.v[e]);
          if (v == 1) { dyc[e] = bf(d.v[e]); scc[e] = bf(rr.v[e]); }
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) ratio[v * 8 + e] = 0.f;
      }
    }
    Bf8 xv = ld8(x + base + c), o;
    float acc = 0.f;
#pragma unroll
    for (int j = 8 - HALF; j <= 8 + HALF; ++j) acc += ratio[j];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float xe = bf(xv.v[e]);
      // relu_mask: x is the output of a ReLU whose backward is folded in here (no gradient where it clipped)
      o.v[e] = __float2bfloat16((relu_mask && xe <= 0.f) ? 0.f : dyc[e] * __powf(scc[e], beta) - coef * xe * acc);
      cs[e] += bf(o.v[e]);
      if (e < 7) acc += ratio[8 + e + HALF + 1] - ratio[8 + e - HALF];
    }
    st8(dx + base + c, o);
  }
  if (colsum != nullptr) {
#pragma unroll
    for (int e = 0; e < 8; ++e) atomicAdd(&lrn_cs[c_fixed + e], cs[e]);
    __syncthreads();
    for (int j = threadIdx.x; j < C; j += blockDim.x) atomicAdd(colsum + j, lrn_cs[j]);
  }
}

// NCHW fp32 -> NHWC bf16, one thread per pixel: reads are coalesced along W in every channel plane
template <typename T>
__global__ void __launch_bounds__(256)
nchw_to_nhwc_pix_kernel(const T* __restrict__ x, bf16* __restrict__ y, int B, int C, int HW, int Cpad) {
  geeps_pdl_enter();
  const long long total = (long long)B * HW;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const long long b = i / HW, p = i % HW;
    const T* src = x + b * C * HW + p;
    bf16* dst = y + i * Cpad;
    for (int c0 = 0; c0 < Cpad; c0 += 4) {
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = (c0 + e < C) ? in_val(src + (long long)(c0 + e) * HW) : 0.f;
      *reinterpret_cast<uint2*>(dst + c0) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    }
  }
}

// NCHW fp32 -> space-to-depth NHWC bf16: y[b][hs][ws][(dy*S + dx)*C + c] = x[b][c][hs*S + dy][ws*S + dx]
// (zero past the image edge and in the channel padding).  A stride-S convolution over x is then a
// stride-1 convolution with ceil(k/S) taps per dimension over y.  One thread per output pixel; the
// 4 x 3-channel case keeps the pixel's 48 values in registers and reads 16 contiguous bytes per (c, dy).
template <int S, int C, typename T>
__global__ void __launch_bounds__(256)
nchw_to_s2d_kernel(const T* __restrict__ x, bf16* __restrict__ y, int B, int H, int W, int Hs, int Ws, int Cpad) {
  geeps_pdl_enter();
  constexpr int N = S * S * C;
  const long long total = (long long)B * Hs * Ws;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int ws = (int)(i % Ws);
    const long long t = i / Ws;
    const int hs = (int)(t % Hs);
    const long long b = t / Hs;
    float v[N];
#pragma unroll
    for (int c = 0; c < C; ++c) {
#pragma unroll
      for (int dy = 0; dy < S; ++dy) {
        const int h = hs * S + dy;
        const T* row = x + ((b * C + c) * H + h) * (long long)W;
#pragma unroll
        for (int dx = 0; dx < S; ++dx) {
          const int w = ws * S + dx;
          v[(dy * S + dx) * C + c] = (h < H && w < W) ? in_val(row + w) : 0.f;
        }
      }
    }
    bf16* dst = y + i * Cpad;
#pragma unroll
    for (int j = 0; j + 8 <= N; j += 8)
      *reinterpret_cast<uint4*>(dst + j) = make_uint4(pack_bf16x2(v[j], v[j + 1]), pack_bf16x2(v[j + 2], v[j + 3]),
                                                      pack_bf16x2(v[j + 4], v[j + 5]), pack_bf16x2(v[j + 6], v[j + 7]));
    int j = N & ~7;
    if ((N & 7) == 0)
      for (; j + 8 <= Cpad; j += 8) *reinterpret_cast<uint4*>(dst + j) = make_uint4(0, 0, 0, 0);
    for (; j < Cpad; ++j) dst[j] = __float2bfloat16(j < N ? v[j] : 0.f);
  }
}

// The same layout for S = 4, C = 3 with coalesced traffic on both sides: a block of four warps converts 32
// consecutive output pixels of one output row.  Warp dy reads, for each colour, the 128 consecutive input elements of
// image row 4 hs + dy that those pixels cover (32 consecutive elements per load), the values meet in a [32 pixels][Cpad]
// tile in shared memory, and the tile leaves as one contiguous run of 32 * Cpad * 2 bytes in 16-byte stores.
template <typename T>
__global__ void __launch_bounds__(128)
nchw_to_s2d43_tile_kernel(const T* __restrict__ x, bf16* __restrict__ y, int B, int H, int W, int Hs, int Ws, int Cpad,
                          int segs) {
  geeps_pdl_enter();
  constexpr int S = 4, C = 3, PIX = 32, PITCH = 72;      // tile row pitch in elements: 144 bytes staggers the banks
  __shared__ __align__(16) bf16 tile[PIX * PITCH];
  const int lane = threadIdx.x & 31, dy = threadIdx.x >> 5;
  long long blk = blockIdx.x;
  const int seg = (int)(blk % segs); blk /= segs;
  const int hs = (int)(blk % Hs);
  const long long b = blk / Hs;
  const int ws0 = seg * PIX;
  // channels past S * S * C are zero (this warp's share of them: pixel `lane`, slots 48 + 4 dy .. + 4, when they exist)
  for (int j = S * S * C + dy * 4; j < Cpad && j < S * S * C + dy * 4 + 4; ++j) tile[lane * PITCH + j] = __float2bfloat16(0.f);
  const int h = hs * S + dy;
  // the 128 consecutive input elements of this image row that the 32 pixels cover, 32 at a time: every load
  // instruction of the warp is one contiguous run (also when x is pinned host memory read over PCIe)
  const int wbase = ws0 * S;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const T* row = x + ((b * C + c) * H + h) * (long long)W;
#pragma unroll
    for (int i = 0; i < S; ++i) {
      const int e = i * 32 + lane;                      // element of the run: pixel e / 4, column offset e % 4
      const int w = wbase + e;
      const float v = (h < H && w < W) ? in_val(row + w) : 0.f;
      tile[(e >> 2) * PITCH + (dy * S + (e & 3)) * C + c] = __float2bfloat16(v);
    }
  }
  __syncthreads();
  const int per_pix = Cpad >> 3;                          // 16-byte pieces per pixel
  const int npix = min(PIX, Ws - ws0);
  bf16* dst = y + ((b * Hs + hs) * (long long)Ws + ws0) * Cpad;
  for (int i = threadIdx.x; i < npix * per_pix; i += blockDim.x) {
    const int px = i / per_pix, piece = i - px * per_pix;
    *reinterpret_cast<uint4*>(dst + (long long)i * 8) = *reinterpret_cast<const uint4*>(tile + px * PITCH + piece * 8);
  }
}

// any S, C: one thread per output element
template <typename T>
__global__ void __launch_bounds__(256)
nchw_to_s2d_generic_kernel(const T* __restrict__ x, bf16* __restrict__ y, int B, int C, int H, int W, int S,
                           int Hs, int Ws, int Cpad) {
  geeps_pdl_enter();
  const long long total = (long long)B * Hs * Ws * Cpad;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int j = (int)(i % Cpad);
    long long t = i / Cpad;
    const int ws = (int)(t % Ws); t /= Ws;
    const int hs = (int)(t % Hs);
    const long long b = t / Hs;
    float v = 0.f;
    if (j < S * S * C) {
      const int c = j % C, q = j / C, dx = q % S, dy = q / S;
      const int h = hs * S + dy, w = ws * S + dx;
      if (h < H && w < W) v = in_val(x + ((b * C + c) * H + h) * (long long)W + w);
    }
    y[i] = __float2bfloat16(v);
  }
}

// ---- data transformer: uint8 NCHW source images -> cropped / mirrored / mean-subtracted / scaled bf16 activations ----
// The work of Caffe's DataTransformer (crop_size, mirror, mean_value, scale), done on the device so that the host ships
// one byte per value.  aug (NULL: centre crop, no mirror) holds {h_off, w_off, mirror} per image.
struct XformDev {
  const uint8_t* x;
  const int* aug;
  int Hin, Win;          // source image
  int H, W;              // cropped image (what the network sees)
  int h_off, w_off;      // centre crop, used when aug == NULL
  float mean[4], scale;
};

__device__ __forceinline__ void xform_image(const XformDev& t, long long b, int& h_off, int& w_off, int& mirror) {
  if (t.aug != nullptr) {
    // out-of-range offsets are clamped: a bad entry reads a valid window instead of another image
    h_off = min(max(t.aug[b * 3 + 0], 0), t.Hin - t.H);
    w_off = min(max(t.aug[b * 3 + 1], 0), t.Win - t.W);
    mirror = t.aug[b * 3 + 2] != 0;
  } else {
    h_off = t.h_off; w_off = t.w_off; mirror = 0;
  }
}

// ---- S = 4, C = 3 space-to-depth, 8- and 16-bit sources ----
// Two lanes make one output pixel (two image rows of four columns each): a lane fetches the four columns of a colour as
// the one to three aligned 32-bit words that cover them, converts them in registers and builds three 16-byte pieces of
// the pixel; a warp's 16 pixels meet in shared memory and leave as one contiguous run.  256 images of 8 bits, cropped to
// 227 x 227: one element per load and 2-byte shared-memory stores, 32 pixels of one output row per block, 59 us; this
// 30 us, of which the 106 MB written are 16.
// An 8-bit source may start and end inside a word (a batch slice, odd image sizes): the lanes whose words could reach past
// it fetch by elements, every other lane by words (by elements throughout: 423 us).
struct U8Quads {
  static constexpr bool kBytes = true;
  XformDev t;
  const uint8_t* end;       // one past the source
  int h_off, w_off, mirror;
  __device__ __forceinline__ void image(long long b) { xform_image(t, b, h_off, w_off, mirror); }
  __device__ __forceinline__ int height() const { return t.H; }
  __device__ __forceinline__ int pitch() const { return t.Win; }
  __device__ __forceinline__ long long plane() const { return (long long)t.Hin * t.Win; }
  __device__ __forceinline__ int width() const { return t.W; }
  __device__ __forceinline__ const uint8_t* row(long long b, int c, int h) const {
    return t.x + ((b * 3 + c) * t.Hin + (h + h_off)) * (long long)t.Win + w_off;
  }
  __device__ __forceinline__ uint32_t byte(long long b, int c, int h, int w) const {
    return __ldg(row(b, c, h) + (mirror ? t.W - 1 - w : w));
  }
  __device__ __forceinline__ const uint8_t* quad_at(long long b, int c, int h, int w) const {
    return row(b, c, h) + (mirror ? t.W - 4 - w : w);
  }
  // are all words around columns w .. w + 3 of rows h .. h1, every colour, inside the source?
  __device__ __forceinline__ bool inside(long long b, int h, int h1, int w) const {
    const uint8_t* first = quad_at(b, 0, h, w);
    return first - ((uintptr_t)first & 3) >= t.x && end - quad_at(b, 2, h1, w) >= 8;
  }
  // columns w .. w + 3, a byte each (the second word is read only when it holds one of the columns)
  __device__ __forceinline__ uint32_t quad(const uint8_t* p) const {
    const uint32_t sh = (uint32_t)((uintptr_t)p & 3) * 8;
    const uint32_t* q = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
    const uint32_t lo = __ldg(q), hi = sh ? __ldg(q + 1) : 0u;
    const uint32_t v = __funnelshift_r(lo, hi, sh);
    return mirror ? __byte_perm(v, 0, 0x0123) : v;
  }
  // (byte - mean) * scale of byte i of u and byte j of v, packed; 2^23 + byte is exact; m: minus the two colours' means
  __device__ __forceinline__ uint32_t two(uint32_t u, int i, uint32_t v, int j, float2 m) const {
    const float2 f = make_float2(__uint_as_float(__byte_perm(u, 0x4b000000u, 0x7650u | (uint32_t)i)),
                                 __uint_as_float(__byte_perm(v, 0x4b000000u, 0x7650u | (uint32_t)j)));
    const float2 base = make_float2(-8388608.f, -8388608.f), k = make_float2(t.scale, t.scale);
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;\n\tadd.rn.f32x2 %0, %0, %3;\n\tmul.rn.f32x2 %0, %0, %4;"
        : "=&l"(r)
        : "l"(reinterpret_cast<const unsigned long long&>(f)), "l"(reinterpret_cast<const unsigned long long&>(base)),
          "l"(reinterpret_cast<const unsigned long long&>(m)), "l"(reinterpret_cast<const unsigned long long&>(k)));
    const float2 o = reinterpret_cast<float2&>(r);
    return pack_bf16x2(o.x, o.y);
  }
  // the twelve values of a row, column-major, colour fastest; columns from n on are zero (n >= 4: none)
  __device__ __forceinline__ void row12(const uint32_t (&v)[3], int n, uint32_t* o) const {
    const float2 m01 = make_float2(-t.mean[0], -t.mean[1]), m20 = make_float2(-t.mean[2], -t.mean[0]),
                 m12 = make_float2(-t.mean[1], -t.mean[2]);
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
      o[3 * (k / 2)] = two(v[0], k, v[1], k, m01);
      o[3 * (k / 2) + 1] = two(v[2], k, v[0], k + 1, m20);
      o[3 * (k / 2) + 2] = two(v[1], k + 1, v[2], k + 1, m12);
    }
    if (n < 4) {
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const int first = 2 * i / 3, second = (2 * i + 1) / 3;       // columns of the word's halves
        if (second >= n) o[i] &= first >= n ? 0u : 0xffffu;
      }
    }
  }
};
struct Bf16Quads {
  static constexpr bool kBytes = false;
  const bf16* x;
  int H, W;
  __device__ __forceinline__ void image(long long) {}
  __device__ __forceinline__ int height() const { return H; }
  __device__ __forceinline__ int width() const { return W; }
  __device__ __forceinline__ uint32_t one(long long b, int c, int h, int w) const {
    return (uint32_t)__bfloat16_as_ushort(x[((b * 3 + c) * H + h) * (long long)W + w]);
  }
  __device__ __forceinline__ bool inside(long long, int, int, int) const { return true; }   // whole words: see the launch
  __device__ __forceinline__ uint2 quad(long long b, int c, int h, int w) const {
    const bf16* p = x + ((b * 3 + c) * H + h) * (long long)W + w;
    const bool odd = ((uintptr_t)p & 2) != 0;
    const uint32_t* q = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
    const uint32_t w0 = __ldg(q), w1 = __ldg(q + 1), w2 = odd ? __ldg(q + 2) : 0u;
    return odd ? make_uint2(__funnelshift_r(w0, w1, 16), __funnelshift_r(w1, w2, 16)) : make_uint2(w0, w1);
  }
};
template <typename Src>
__global__ void __launch_bounds__(256)
s2d43_quad_kernel(Src src, bf16* __restrict__ y, unsigned npix, int Hs, int Ws, int Cpad) {
  __shared__ uint4 tile[8][16 * 8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane & 1, px = lane >> 1;
  const unsigned base = (blockIdx.x * (blockDim.x >> 5) + warp) * 16u;
  if (base >= npix) return;                       // whole warps: nothing below meets another warp
  const unsigned pix = base + px;
  const int per_pix = Cpad >> 3;
  uint32_t o[12];
#pragma unroll
  for (int i = 0; i < 12; ++i) o[i] = 0u;
  if (pix < npix) {
    const unsigned row = pix / (unsigned)Ws, b = row / (unsigned)Hs;
    const int w = (int)(pix - row * Ws) * 4, h0 = (int)(row - b * Hs) * 4 + half * 2;
    src.image(b);
    const int last = src.height() - 1, wq = min(w, src.width() - 4);
    // All fetches of a lane are in flight together, then masked.  (A branch per colour that fetched the one to three
    // columns of a ragged right edge waited for each: 256 images 45 us, 35 us without; one image 4.9 and 2.5 us.)
    const bool words = wq >= 0 && src.inside(b, min(h0, last), min(h0 + 1, last), wq);
    if constexpr (Src::kBytes) {
      // bytes stay bytes until they are packed in the output's order (converted a colour at a time and interleaved as
      // 16-bit values: 256 images 33.8 us, 29.8 now, of which the 157 MB in and out are 24)
      const int shift = (w - wq) * 8;    // past the right edge: the last four columns, shifted
      uint32_t v[2][3];
      if (words) {
        const uint8_t* at = src.quad_at(b, 0, min(h0, last), wq);
        const long long plane = src.plane(), down = h0 < last ? src.pitch() : 0;
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            v[d][c] = src.quad(at + (c * plane + d * down));
            v[d][c] = shift < 32 ? v[d][c] >> shift : 0u;
          }
      } else {
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            v[d][c] = 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) v[d][c] |= src.byte(b, c, min(h0 + d, last), min(w + k, src.width() - 1)) << (8 * k);
          }
      }
#pragma unroll
      for (int d = 0; d < 2; ++d) src.row12(v[d], h0 + d <= last ? src.width() - w : 0, o + 6 * d);
    } else {
      unsigned long long q[2][3];          // four columns of 16 bits
      if (words) {
        const int shift = (w - wq) * 16;
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const uint2 v = src.quad(b, c, min(h0 + d, last), wq);
            q[d][c] = shift < 64 ? ((unsigned long long)v.y << 32 | v.x) >> shift : 0ull;
          }
      } else {
        const int n = src.width() - w;
        const unsigned long long keep = n >= 4 ? ~0ull : (n > 0 ? (1ull << (16 * n)) - 1 : 0ull);
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            unsigned long long v = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              v |= (unsigned long long)src.one(b, c, min(h0 + d, last), min(w + k, src.width() - 1)) << (16 * k);
            q[d][c] = v & keep;
          }
      }
      // interleave: column-major, colour fastest
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        uint32_t lo[3], hi[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          lo[c] = h0 + d <= last ? (uint32_t)q[d][c] : 0u;
          hi[c] = h0 + d <= last ? (uint32_t)(q[d][c] >> 32) : 0u;
        }
        o[6 * d + 0] = __byte_perm(lo[0], lo[1], 0x5410);
        o[6 * d + 1] = __byte_perm(lo[2], lo[0], 0x7610);
        o[6 * d + 2] = __byte_perm(lo[1], lo[2], 0x7632);
        o[6 * d + 3] = __byte_perm(hi[0], hi[1], 0x5410);
        o[6 * d + 4] = __byte_perm(hi[2], hi[0], 0x7610);
        o[6 * d + 5] = __byte_perm(hi[1], hi[2], 0x7632);
      }
    }
  }
  // pieces of a pixel XOR-ed with the pixel number: the 16-byte stores spread over the banks
  uint4* mine = tile[warp] + px * 8;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    mine[(half * 3 + i) ^ (px & 7)] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
  mine[(6 + half) ^ (px & 7)] = make_uint4(0u, 0u, 0u, 0u);     // channels past 48
  __syncwarp();
  const int n = (int)min(16u, npix - base) * per_pix;
  uint4* dst = reinterpret_cast<uint4*>(y) + (long long)base * per_pix;
  for (int i = lane; i < n; i += 32) {
    const int p = per_pix == 8 ? i >> 3 : i / per_pix, k = i - p * per_pix;
    dst[i] = tile[warp][p * 8 + (k ^ (p & 7))];
  }
}
// what the kernel asks of the output and of the pixel count (its indexes are 32 bits wide)
inline bool s2d43_quads_ok(const void* y, long long npix, int Cpad) {
  return ((uintptr_t)y & 15) == 0 && Cpad % 8 == 0 && Cpad >= 48 && Cpad <= 64 && npix > 0 && npix < 0x7fffff00LL;
}
// Eight warps a block, fewer where that would leave SMs without a block (one image of 227 x 227: 26 blocks of eight).
// An ordinary launch: thousands of short blocks, each of which would wait for the step before (19.4 -> 19.8 us at batch 121).
template <typename Src>
void launch_s2d43_quads(const Src& src, void* y, long long npix, int Hs, int Ws, int Cpad, cudaStream_t st) {
  const long long warps = (npix + 15) / 16;
  long long per_block = warps / (2 * geeps_sm_count());
  per_block = per_block < 1 ? 1 : (per_block > 8 ? 8 : per_block);
  s2d43_quad_kernel<<<(unsigned)((warps + per_block - 1) / per_block), (unsigned)(32 * per_block), 0, st>>>(
      src, (bf16*)y, (unsigned)npix, Hs, Ws, Cpad);
}

// any S >= 1 (S = 1: plain NHWC) and C <= 4: one thread per output element
__global__ void __launch_bounds__(256)
u8_xform_generic_kernel(XformDev t, bf16* __restrict__ y, int B, int C, int S, int Hs, int Ws, int Cpad) {
  geeps_pdl_enter();
  const long long total = (long long)B * Hs * Ws * Cpad;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int j = (int)(i % Cpad);
    long long r = i / Cpad;
    const int ws = (int)(r % Ws); r /= Ws;
    const int hs = (int)(r % Hs);
    const long long b = r / Hs;
    float v = 0.f;
    if (j < S * S * C) {
      const int c = j % C, q = j / C, dx = q % S, dy = q / S;
      const int h = hs * S + dy, w = ws * S + dx;
      if (h < t.H && w < t.W) {
        int h_off, w_off, mirror;
        xform_image(t, b, h_off, w_off, mirror);
        const uint8_t* row = t.x + ((b * C + c) * t.Hin + (h + h_off)) * (long long)t.Win + w_off;
        v = ((float)__ldg(row + (mirror ? t.W - 1 - w : w)) - t.mean[c]) * t.scale;
      }
    }
    y[i] = __float2bfloat16(v);
  }
}

// g[r][c] = 0 where mask[c] == 0
__global__ void __launch_bounds__(256)
col_mask_kernel(float* __restrict__ g, const uint8_t* __restrict__ mask, long long rows, int cols, long long ld) {
  geeps_pdl_enter();
  const long long total = rows * cols;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % cols);
    if (!mask[c]) g[(i / cols) * ld + c] = 0.f;
  }
}

// ---------------- pooling (NHWC, 8 channels per thread) ----------------
// Output may be a channel slice of a wider tensor (pitch ldy, offset applied by the caller).
// ---- packed helpers for max pooling: 8 channels at a time, two per 32-bit register ----
// Window code per 16-bit lane.
__device__ __forceinline__ uint32_t dup16(uint32_t code) { return code | (code << 16); }
// acc (4 x bf16x2) += d where argmax byte == code.  `pk` holds the 8 argmax bytes, `d` the 8 gradients.
__device__ __forceinline__ void pool_bwd_accum(__nv_bfloat162 (&acc)[4], const uint2 pk, const uint4 d, uint32_t code) {
  const uint32_t c4 = code * 0x01010101u;
  const uint32_t m0 = __vcmpeq4(pk.x, c4), m1 = __vcmpeq4(pk.y, c4);     // 0xff per matching channel
  if ((m0 | m1) == 0) return;
  const uint32_t dv[4] = {d.x, d.y, d.z, d.w};
  const uint32_t mk[4] = {__byte_perm(m0, 0, 0x1100), __byte_perm(m0, 0, 0x3322), __byte_perm(m1, 0, 0x1100),
                          __byte_perm(m1, 0, 0x3322)};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t sel = dv[j] & mk[j];
    acc[j] = __hadd2(acc[j], *reinterpret_cast<const __nv_bfloat162*>(&sel));
  }
}
__device__ __forceinline__ uint4 pool_bwd_pack(const __nv_bfloat162 (&acc)[4]) {
  return make_uint4(*reinterpret_cast<const uint32_t*>(&acc[0]), *reinterpret_cast<const uint32_t*>(&acc[1]),
                    *reinterpret_cast<const uint32_t*>(&acc[2]), *reinterpret_cast<const uint32_t*>(&acc[3]));
}

// One block per output row (b, oh): threadIdx.x walks the 8-channel vectors of a pixel, threadIdx.y the
// pixels of the row, so no thread ever divides to find its coordinates and a warp reads contiguous pixels.
__global__ void __launch_bounds__(256)
maxpool_forward_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, uint8_t* __restrict__ argmax,
                       const GeepsPoolGeom g, int relu_mask) {
  geeps_pdl_enter();
  const int cv = g.C >> 3;
  const int oh = blockIdx.x % g.OH, b = blockIdx.x / g.OH;
  const int ih0 = oh * g.stride - g.pad;
  const int kh_lo = max(0, -ih0), kh_hi = min(g.K, g.H - ih0);
  const bf16* xb = x + (long long)b * g.H * g.W * g.ldx;
  const long long orow = ((long long)b * g.OH + oh) * g.OW;
  for (int ow = threadIdx.y; ow < g.OW; ow += blockDim.y) {
    const int iw0 = ow * g.stride - g.pad;
    const int kw_lo = max(0, -iw0), kw_hi = min(g.K, g.W - iw0);
    for (int cvi = threadIdx.x; cvi < cv; cvi += blockDim.x) {
      const int c = cvi * 8;
      // packed: best value and window code per 16-bit lane; strict > keeps the first maximum
      const uint32_t neg = 0xff7fff7fu;                 // two bf16 lowest finite values
      __nv_bfloat162 best[4];
      uint32_t arg[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) { best[j] = *reinterpret_cast<const __nv_bfloat162*>(&neg); arg[j] = 0x00ff00ffu; }
      for (int kh = kh_lo; kh < kh_hi; ++kh) {
        const bf16* xr = xb + ((long long)(ih0 + kh) * g.W + iw0) * g.ldx + c;
        for (int kw = kw_lo; kw < kw_hi; ++kw) {
          const uint4 v = *reinterpret_cast<const uint4*>(xr + (long long)kw * g.ldx);
          const uint32_t vv[4] = {v.x, v.y, v.z, v.w};
          const uint32_t code = dup16((uint32_t)(kh * g.K + kw));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 x2 = *reinterpret_cast<const __nv_bfloat162*>(&vv[j]);
            const uint32_t gt = __hgt2_mask(x2, best[j]);
            best[j] = __hmax2(best[j], x2);
            arg[j] = (arg[j] & ~gt) | (code & gt);
          }
        }
      }
      // A window without a positive value names none, so the backward pass leaves out what the ReLU in front masks and that layer
      // reads dx for its column sums only (43264 x 256: 22 MB instead of 44 and 22 written; AlexNet's step 2128 / 2115 us).
      if (relu_mask) {
        const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) arg[j] |= ~__hgt2_mask(best[j], zero) & 0x00ff00ffu;
      }
      const long long opix = orow + ow;
      *reinterpret_cast<uint4*>(y + opix * g.ldy + c) = pool_bwd_pack(best);
      uint2 pk;      // 16-bit lanes -> bytes
      pk.x = __byte_perm(arg[0], arg[1], 0x6420);
      pk.y = __byte_perm(arg[2], arg[3], 0x6420);
      *reinterpret_cast<uint2*>(argmax + opix * g.C + c) = pk;
    }
  }
}
// One block per input row (b, ih).  The output rows whose window covers ih are the same for the whole
// block, the output columns covering iw are a short range: only those windows are visited.
__global__ void __launch_bounds__(256)
maxpool_backward_kernel(const bf16* __restrict__ dy, const uint8_t* __restrict__ argmax, bf16* __restrict__ dx,
                        const GeepsPoolGeom g, int accumulate) {
  geeps_pdl_enter();
  const int cv = g.C >> 3;
  const int ih = blockIdx.x % g.H, b = blockIdx.x / g.H;
  const int th = ih + g.pad;
  // oh * stride <= th <= oh * stride + K - 1
  const int oh_lo = max(0, (th - g.K + g.stride) / g.stride), oh_hi = min(g.OH - 1, th / g.stride);
  const long long obase = (long long)b * g.OH * g.OW;
  bf16* drow = dx + ((long long)b * g.H + ih) * g.W * g.ldx;
  for (int iw = threadIdx.y; iw < g.W; iw += blockDim.y) {
    const int tw = iw + g.pad;
    const int ow_lo = max(0, (tw - g.K + g.stride) / g.stride), ow_hi = min(g.OW - 1, tw / g.stride);
    for (int cvi = threadIdx.x; cvi < cv; cvi += blockDim.x) {
      const int c = cvi * 8;
      __nv_bfloat162 acc[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = __floats2bfloat162_rn(0.f, 0.f);
      for (int oh = oh_lo; oh <= oh_hi; ++oh) {
        const int kh = th - oh * g.stride;
        for (int ow = ow_lo; ow <= ow_hi; ++ow) {
          const int code = kh * g.K + (tw - ow * g.stride);
          const long long opix = obase + (long long)oh * g.OW + ow;
          const uint2 pk = *reinterpret_cast<const uint2*>(argmax + opix * g.C + c);
          const uint4 d = *reinterpret_cast<const uint4*>(dy + opix * g.ldy + c);
          pool_bwd_accum(acc, pk, d, (uint32_t)code);
        }
      }
      bf16* dst = drow + (long long)iw * g.ldx + c;
      if (accumulate) {
        const uint4 old = *reinterpret_cast<const uint4*>(dst);
        const uint32_t ov[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] = __hadd2(acc[j], *reinterpret_cast<const __nv_bfloat162*>(&ov[j]));
      }
      *reinterpret_cast<uint4*>(dst) = pool_bwd_pack(acc);
    }
  }
}

// Same product, staged through shared memory: a block owns `stride` consecutive input rows of one image; the few
// output rows whose windows cover them (dy and argmax) are copied into shared memory once and every input
// pixel then gathers from there.  The direct kernel re-reads each dy / argmax element from L2 for every input
// pixel of its window (K*K times); here it crosses L2 -> SM once per block.
__global__ void __launch_bounds__(256)
maxpool_backward_smem_kernel(const bf16* __restrict__ dy, const uint8_t* __restrict__ argmax, bf16* __restrict__ dx,
                             const GeepsPoolGeom g, int accumulate, int rows_per_block, int max_oh) {
  geeps_pdl_enter();
  extern __shared__ __align__(16) uint8_t pool_smem[];
  const int cv = g.C >> 3;
  const int row_blocks = (g.H + rows_per_block - 1) / rows_per_block;
  const int rb = blockIdx.x % row_blocks, b = blockIdx.x / row_blocks;
  const int ih_lo = rb * rows_per_block, ih_hi = min(g.H, ih_lo + rows_per_block);      // [lo, hi)
  const int oh_lo = max(0, (ih_lo + g.pad - g.K + g.stride) / g.stride);
  const int oh_hi = min(g.OH - 1, (ih_hi - 1 + g.pad) / g.stride);
  const int n_oh = oh_hi - oh_lo + 1;
  bf16* s_dy = reinterpret_cast<bf16*>(pool_smem);                                        // [max_oh][OW][C]
  uint8_t* s_arg = pool_smem + (size_t)max_oh * g.OW * g.C * sizeof(bf16);                // [max_oh][OW][C]
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nthreads = blockDim.x * blockDim.y;
  if (n_oh > 0) {
    const long long obase = ((long long)b * g.OH + oh_lo) * g.OW;
    const int vecs = n_oh * g.OW * cv;
    for (int v = tid; v < vecs; v += nthreads) {
      const int pix = v / cv, c = (v - pix * cv) * 8;
      *reinterpret_cast<uint4*>(s_dy + (size_t)pix * g.C + c) =
          *reinterpret_cast<const uint4*>(dy + (obase + pix) * g.ldy + c);
      *reinterpret_cast<uint2*>(s_arg + (size_t)pix * g.C + c) =
          *reinterpret_cast<const uint2*>(argmax + (obase + pix) * g.C + c);
    }
  }
  __syncthreads();
  for (int ih = ih_lo; ih < ih_hi; ++ih) {
    const int th = ih + g.pad;
    const int r_lo = max(oh_lo, (th - g.K + g.stride) / g.stride), r_hi = min(oh_hi, th / g.stride);
    bf16* drow = dx + ((long long)b * g.H + ih) * g.W * g.ldx;
    for (int iw = threadIdx.y; iw < g.W; iw += blockDim.y) {
      const int tw = iw + g.pad;
      const int ow_lo = max(0, (tw - g.K + g.stride) / g.stride), ow_hi = min(g.OW - 1, tw / g.stride);
      for (int cvi = threadIdx.x; cvi < cv; cvi += blockDim.x) {
        const int c = cvi * 8;
        __nv_bfloat162 acc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] = __floats2bfloat162_rn(0.f, 0.f);
        for (int oh = r_lo; oh <= r_hi; ++oh) {
          const int kh = th - oh * g.stride;
          for (int ow = ow_lo; ow <= ow_hi; ++ow) {
            const int code = kh * g.K + (tw - ow * g.stride);
            const size_t sp = ((size_t)(oh - oh_lo) * g.OW + ow) * g.C + c;
            pool_bwd_accum(acc, *reinterpret_cast<const uint2*>(s_arg + sp), *reinterpret_cast<const uint4*>(s_dy + sp),
                           (uint32_t)code);
          }
        }
        bf16* dst = drow + (long long)iw * g.ldx + c;
        if (accumulate) {
          const uint4 old = *reinterpret_cast<const uint4*>(dst);
          const uint32_t ov[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[j] = __hadd2(acc[j], *reinterpret_cast<const __nv_bfloat162*>(&ov[j]));
        }
        *reinterpret_cast<uint4*>(dst) = pool_bwd_pack(acc);
      }
    }
  }
}
// 3 x 3 windows at stride 2: the four pixels of a quad (even padded row and column first) lie in four windows, which a thread
// loads once, all at a time, for 8 channels.  No shared memory to fill first, so nothing waits for a block's slowest load;
// each pixel adds its windows in the order of the other kernels.  us, windows staged in shared memory / so: 256 x 13 x 13 x 256
// 21.1 / 9.6 (the bytes 4.5), 100 x 13 x 13 x 256 11.4 / 5.4, 8 x 13 x 13 x 256 7.9 / 3.0, 32 x 14 x 14 x 576 15.9 / 4.2, 32 x
// 56 x 56 x 64 15.2 / 6.4.
__global__ void __launch_bounds__(256)
maxpool3s2_backward_kernel(const bf16* __restrict__ dy, const uint8_t* __restrict__ argmax, bf16* __restrict__ dx,
                           const GeepsPoolGeom g, int accumulate, unsigned quads_h, unsigned quads_w, unsigned total) {
  geeps_pdl_enter();
  const unsigned item = blockIdx.x * blockDim.x + threadIdx.x;
  if (item >= total) return;
  const unsigned cv = (unsigned)g.C >> 3;
  const unsigned q = item / cv, row = q / quads_w, b = row / quads_h;
  const int c = (int)(item - q * cv) * 8;
  const int wr = (g.pad >> 1) + (int)(row - b * quads_h), wc = (g.pad >> 1) + (int)(q - row * quads_w);   // last windows of the quad
  uint4 d[2][2];
  uint2 k[2][2];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int oh = wr - 1 + r, ow = wc - 1 + s;
      d[r][s] = make_uint4(0, 0, 0, 0);
      k[r][s] = make_uint2(0xffffffffu, 0xffffffffu);      // no element of a window
      if (oh >= 0 && oh < g.OH && ow >= 0 && ow < g.OW) {
        const long long opix = ((long long)b * g.OH + oh) * g.OW + ow;
        d[r][s] = *reinterpret_cast<const uint4*>(dy + opix * g.ldy + c);
        k[r][s] = *reinterpret_cast<const uint2*>(argmax + opix * g.C + c);
      }
    }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int ih = 2 * wr + u - g.pad, iw = 2 * wc + v - g.pad;
      if (ih < 0 || ih >= g.H || iw < 0 || iw >= g.W) continue;
      __nv_bfloat162 acc[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
      for (int r = u; r < 2; ++r)           // an odd row is the middle of one window, an even one the last and first of two
#pragma unroll
        for (int s = v; s < 2; ++s) {
          const int kh = u ? 1 : 2 - 2 * r, kw = v ? 1 : 2 - 2 * s;
          pool_bwd_accum(acc, k[r][s], d[r][s], (uint32_t)(kh * 3 + kw));
        }
      bf16* dst = dx + (((long long)b * g.H + ih) * g.W + iw) * g.ldx + c;
      if (accumulate) {
        const uint4 old = *reinterpret_cast<const uint4*>(dst);
        const uint32_t ov[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] = __hadd2(acc[j], *reinterpret_cast<const __nv_bfloat162*>(&ov[j]));
      }
      *reinterpret_cast<uint4*>(dst) = pool_bwd_pack(acc);
    }
}

// Caffe average pooling: divisor is the window area clipped to the padded extent.
__device__ __forceinline__ int avg_area(int o, int stride, int pad, int K, int size) {
  const int s = o * stride - pad;
  const int e = min(s + K, size + pad);
  return e - s;
}
// threadIdx.x is the 8-channel vector of a pixel and threadIdx.y (with blockIdx.y) the pixel, so nothing is divided to
// find columns and only the windows that cover a pixel are visited (a 64-bit division chain per vector: 14 and 17.5 us on
// 32 x 14 x 14 x 576, this 10 and 15).  A block stays in one row, whose coordinates and window rows are then the same for
// all its threads (forward 17.5 us on 32 x 56 x 56 x 64, 21 with a row per thread).  ROWS: several rows per block, on
// threadIdx.z, where a row has work for 128 threads or fewer and at most three windows (taps) per direction cover a pixel;
// the loads of a window row are in flight together.  512 x 5 x 5 x 24, forward and backward: one row per 256 threads 8.1
// and 10.8 us, one row per block of its size 4.5 and 5.7, this 2.8 and 3.4.  (Larger windows, such as the global pooling
// at the end of a network, are bound by the taps of a thread: 100 x 8 x 8 x 336, one row 9.2 us, grouped 9.9.)
template <bool ROWS>
__device__ __forceinline__ unsigned pool_row() { return ROWS ? blockIdx.x * blockDim.z + threadIdx.z : blockIdx.x; }

template <bool ROWS>
__global__ void __launch_bounds__(256)
avgpool_forward_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, const GeepsPoolGeom g) {
  geeps_pdl_enter();
  const int cv = g.C >> 3;
  const unsigned row = pool_row<ROWS>();
  if (ROWS && row >= (unsigned)g.B * (unsigned)g.OH) return;
  const int oh = row % g.OH, b = row / g.OH;
  const int ih0 = oh * g.stride - g.pad;
  const int kh_lo = max(0, -ih0), kh_hi = min(g.K, g.H - ih0);
  const int area_h = avg_area(oh, g.stride, g.pad, g.K, g.H);
  const long long orow = ((long long)b * g.OH + oh) * g.OW;
  for (int ow = blockIdx.y * blockDim.y + threadIdx.y; ow < g.OW; ow += blockDim.y * gridDim.y) {
    const int iw0 = ow * g.stride - g.pad;
    const int kw_lo = max(0, -iw0), kw_hi = min(g.K, g.W - iw0);
    const float inv = __frcp_rn((float)(area_h * avg_area(ow, g.stride, g.pad, g.K, g.W)));
    for (int cvi = threadIdx.x; cvi < cv; cvi += blockDim.x) {
      const int c = cvi * 8;
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
      for (int kh = kh_lo; kh < kh_hi; ++kh) {
        const bf16* xr = x + (((long long)b * g.H + ih0 + kh) * g.W + iw0) * g.ldx + c;
        if (ROWS) {
          Bf8 v[3];
#pragma unroll
          for (int kw = 0; kw < 3; ++kw) v[kw] = kw >= kw_lo && kw < kw_hi ? ld8(xr + (long long)kw * g.ldx) : zero8();
#pragma unroll
          for (int kw = 0; kw < 3; ++kw)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += bf(v[kw].v[e]);
        } else {
#pragma unroll 3
          for (int kw = kw_lo; kw < kw_hi; ++kw) {
            const Bf8 v = ld8(xr + (long long)kw * g.ldx);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += bf(v.v[e]);
          }
        }
      }
      Bf8 o;
#pragma unroll
      for (int e = 0; e < 8; ++e) o.v[e] = __float2bfloat16(acc[e] * inv);
      st8(y + (orow + ow) * g.ldy + c, o);
    }
  }
}
template <bool ROWS>
__global__ void __launch_bounds__(256)
avgpool_backward_kernel(const bf16* __restrict__ dy, bf16* __restrict__ dx, const GeepsPoolGeom g, int accumulate) {
  geeps_pdl_enter();
  const int cv = g.C >> 3;
  const unsigned row = pool_row<ROWS>();
  if (ROWS && row >= (unsigned)g.B * (unsigned)g.H) return;
  const int ih = row % g.H, b = row / g.H;
  const int th = ih + g.pad;
  // oh * stride <= th <= oh * stride + K - 1
  const int oh_lo = max(0, (th - g.K + g.stride) / g.stride), oh_hi = min(g.OH - 1, th / g.stride);
  bf16* drow = dx + ((long long)b * g.H + ih) * g.W * g.ldx;
  const float inv_full = __frcp_rn((float)(g.K * g.K));
  for (int iw = blockIdx.y * blockDim.y + threadIdx.y; iw < g.W; iw += blockDim.y * gridDim.y) {
    const int tw = iw + g.pad;
    const int ow_lo = max(0, (tw - g.K + g.stride) / g.stride), ow_hi = min(g.OW - 1, tw / g.stride);
    for (int cvi = threadIdx.x; cvi < cv; cvi += blockDim.x) {
      const int c = cvi * 8;
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
      for (int oh = oh_hi; oh >= oh_lo; --oh) {             // the order of the window rows and columns
        const int area_h = avg_area(oh, g.stride, g.pad, g.K, g.H);
        const bf16* src = dy + (((long long)b * g.OH + oh) * g.OW) * g.ldy + c;
        if (ROWS) {
          Bf8 d[3];
#pragma unroll
          for (int i = 0; i < 3; ++i) d[i] = ow_hi - i >= ow_lo ? ld8(src + (long long)(ow_hi - i) * g.ldy) : zero8();
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const int area = area_h * avg_area(ow_hi - i, g.stride, g.pad, g.K, g.W);
            const float inv = area == g.K * g.K ? inv_full : ow_hi - i >= ow_lo ? __frcp_rn((float)area) : 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += bf(d[i].v[e]) * inv;
          }
        } else {
#pragma unroll 3
          for (int ow = ow_hi; ow >= ow_lo; --ow) {
            const float inv = __frcp_rn((float)(area_h * avg_area(ow, g.stride, g.pad, g.K, g.W)));
            const Bf8 d = ld8(src + (long long)ow * g.ldy);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += bf(d.v[e]) * inv;
          }
        }
      }
      bf16* dst = drow + (long long)iw * g.ldx + c;
      Bf8 o;
      if (accumulate) {
        const Bf8 old = ld8(dst);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += bf(old.v[e]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) o.v[e] = __float2bfloat16(acc[e]);
      st8(dst, o);
    }
  }
}

// Average pooling of 3 x 3 windows at stride 1 (the pooling branch of an Inception module), where every window has the
// same area: both directions are the same stencil over in[o + off .. o + off + 2], forward the sum in row order and then
// the division, backward each term divided, in the opposite order; sums, orders and bits are those of the kernels above.
// A thread takes R output rows of a column: with four an input row is read by 1.5 outputs instead of three, its 18 loads
// are in flight at once, and the coordinates are found once.  Forward adds the bf16 values as they are (mixed-precision
// sums), backward multiplies pairs; captured chain, us,
// forward and backward: 32 x 14 x 14 x 576 on the kernels above 10.0, 14.8, this 6.6, 6.6 (two rows a thread 6.2, 8.1, one 7.9,
// 8.9; unpacked single products 7.5, 10.6);
// 100 x 32 x 32 x 96 23.8, 34.9, now 13.4, 13.6.  Backward by one row a thread spills at five blocks per SM (2 x 28 x 28 x 320 2.86,
// at four 2.75, 512 x 5 x 5 x 24 2.62, 2.50), forward it does not.
template <bool BWD, int R>
__global__ void __launch_bounds__(256, R > 1 ? 2 : BWD ? 4 : 5)
avgpool3_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, int H, int W, int OH, int OW, int cv, long long ldi,
                long long ldo, int off, int blocks_h, int total, int accumulate) {
  geeps_pdl_enter();
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= total) return;
  const int c = i % cv * 8;
  int t = i / cv;
  const int ow = t % OW;
  t /= OW;
  const int b = t / blocks_h, oh0 = (t - b * blocks_h) * R;
  const float inv = __frcp_rn(9.f);
  uint4 v[R + 2][3];
#pragma unroll
  for (int r = 0; r < R + 2; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int h = oh0 + off + r, w = ow + off + k;
      v[r][k] = (unsigned)h < (unsigned)H && (unsigned)w < (unsigned)W
                    ? *reinterpret_cast<const uint4*>(in + (((long long)b * H + h) * W + w) * ldi + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
  for (int o = 0; o < R; ++o) {
    if (oh0 + o >= OH) break;
    float2 acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = 0; n < 9; ++n) {
      const uint4& d = BWD ? v[o + 2 - n / 3][2 - n % 3] : v[o + n / 3][n % 3];
      const uint32_t w[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (BWD) {
          const float2 f = make_float2(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xffff0000u)), m = make_float2(inv, inv);
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<unsigned long long&>(acc[k]))
              : "l"(reinterpret_cast<const unsigned long long&>(f)), "l"(reinterpret_cast<const unsigned long long&>(m)));
        } else {
          asm("{.reg .b16 l, h; mov.b32 {l, h}, %2; add.f32.bf16 %0, l, %0; add.f32.bf16 %1, h, %1;}"
              : "+f"(acc[k].x), "+f"(acc[k].y) : "r"(w[k]));
        }
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + (((long long)b * OH + oh0 + o) * OW + ow) * ldo + c);
    if (BWD && accumulate) {
      const uint4 old = *dst;
      const uint32_t w[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) { acc[k].x += __uint_as_float(w[k] << 16); acc[k].y += __uint_as_float(w[k] & 0xffff0000u); }
    }
    const float m = BWD ? 1.f : inv;
    *dst = make_uint4(pack_bf16x2(acc[0].x * m, acc[0].y * m), pack_bf16x2(acc[1].x * m, acc[1].y * m),
                      pack_bf16x2(acc[2].x * m, acc[2].y * m), pack_bf16x2(acc[3].x * m, acc[3].y * m));
  }
}

// ---------------- softmax cross-entropy (one CTA per sample) ----------------
__device__ __forceinline__ float block_reduce(float v, bool is_max, float* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float t = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmaxf(v, t) : v + t;
  }
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sh[lane] : (is_max ? -3.0e38f : 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float t = __shfl_xor_sync(0xffffffffu, v, o);
      v = is_max ? fmaxf(v, t) : v + t;
    }
    if (lane == 0) sh[0] = v;
  }
  __syncthreads();
  return sh[0];
}
// loss_sum += -log softmax(logits[b])[label[b]] * loss_scale;  dlogits = (softmax - onehot) * grad_scale
// Rows below 4096 classes: 256 threads, one value at a time; three passes over at most 16 KB that stay in L1.
__global__ void __launch_bounds__(256)
softmax_ce_small_kernel(const float* __restrict__ logits, const long long* __restrict__ labels, float* loss_sum,
                  float* __restrict__ per_sample, bf16* __restrict__ dlogits, int C, long long ldl, long long ldd,
                  float loss_scale, float grad_scale, int* status) {
  geeps_pdl_enter();
  __shared__ float sh[32];
  const int b = blockIdx.x;
  const float* row = logits + (long long)b * ldl;
  float mx = -3.0e38f;
  for (int c = threadIdx.x; c < C; c += blockDim.x) mx = fmaxf(mx, row[c]);
  mx = block_reduce(mx, true, sh);
  float s = 0.f;
  for (int c = threadIdx.x; c < C; c += blockDim.x) s += __expf(row[c] - mx);
  s = block_reduce(s, false, sh);
  long long lab = labels[b];
  if (lab < 0 || lab >= C) {
    if (threadIdx.x == 0) geeps_report(status, GEEPS_ERR_BOUNDS, 30, b, (int)lab);
    lab = 0;
  }
  const float inv = 1.f / s;
  if (dlogits != nullptr) {
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      float pr = __expf(row[c] - mx) * inv;
      dlogits[(long long)b * ldd + c] = __float2bfloat16((pr - (c == lab ? 1.f : 0.f)) * grad_scale);
    }
  }
  if (threadIdx.x == 0) {
    const float l = -(row[lab] - mx - __logf(s));
    if (per_sample) per_sample[b] = l;
    if (loss_sum) atomicAdd(loss_sum, l * loss_scale);
  }
}

// One block per sample.  The row is read once: up to R * 8 values per thread stay in registers between the maximum, the
// sum and the gradient (a row past that is read again).  With a batch of 32 the 32 blocks are all there is, so each has
// up to 1024 threads; VEC (pitches and bases of 16 bytes) moves 32 bytes in and 16 out per thread and step.
// 32 x 21841 classes: 54 us (256 threads, three scalar passes) -> 8 us; bound by one SM's load latency.
template <bool VEC>
__global__ void __launch_bounds__(1024)
softmax_ce_kernel(const float* __restrict__ logits, const long long* __restrict__ labels, float* loss_sum,
                  float* __restrict__ per_sample, bf16* __restrict__ dlogits, int C, long long ldl, long long ldd,
                  float loss_scale, float grad_scale, int* status) {
  geeps_pdl_enter();
  __shared__ float sh[32];
  constexpr int R = 3;
  const int b = blockIdx.x, T = blockDim.x, tid = threadIdx.x;
  const float* row = logits + (long long)b * ldl;
  // value e of this thread in step r: eight consecutive classes, or (unaligned rows) eight strided ones
  auto col = [&](int r, int e) { return VEC ? (r * T + tid) * 8 + e : (r * 8 + e) * T + tid; };
  auto load = [&](int r, float (&o)[8]) {
    if (VEC && col(r, 7) < C) {
      const float4 lo = *reinterpret_cast<const float4*>(row + col(r, 0)), hi = *reinterpret_cast<const float4*>(row + col(r, 4));
      o[0] = lo.x; o[1] = lo.y; o[2] = lo.z; o[3] = lo.w; o[4] = hi.x; o[5] = hi.y; o[6] = hi.z; o[7] = hi.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = col(r, e) < C ? row[col(r, e)] : -INFINITY;
    }
  };
  const int steps = (C + 8 * T - 1) / (8 * T);
  float v[R][8], w[8];
  float mx = -3.0e38f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    load(r, v[r]);
#pragma unroll
    for (int e = 0; e < 8; ++e) mx = fmaxf(mx, v[r][e]);
  }
  for (int r = R; r < steps; ++r) {
    load(r, w);
#pragma unroll
    for (int e = 0; e < 8; ++e) mx = fmaxf(mx, w[e]);
  }
  mx = block_reduce(mx, true, sh);
  float s = 0.f;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (col(r, e) < C) s += __expf(v[r][e] - mx);
  for (int r = R; r < steps; ++r) {
    load(r, w);
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (col(r, e) < C) s += __expf(w[e] - mx);
  }
  s = block_reduce(s, false, sh);
  long long lab = labels[b];
  if (lab < 0 || lab >= C) {
    if (tid == 0) geeps_report(status, GEEPS_ERR_BOUNDS, 30, b, (int)lab);
    lab = 0;
  }
  const float inv = 1.f / s;
  if (dlogits != nullptr) {
    bf16* drow = dlogits + (long long)b * ldd;
    auto store = [&](int r, const float (&l)[8]) {
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = (__expf(l[e] - mx) * inv - (col(r, e) == (int)lab ? 1.f : 0.f)) * grad_scale;
      if (VEC && col(r, 7) < C) {
        *reinterpret_cast<uint4*>(drow + col(r, 0)) = make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]),
                                                                 pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (col(r, e) < C) drow[col(r, e)] = __float2bfloat16(o[e]);
      }
    };
#pragma unroll
    for (int r = 0; r < R; ++r) store(r, v[r]);
    for (int r = R; r < steps; ++r) { load(r, w); store(r, w); }
  }
  if (tid == 0) {
    const float l = -(row[lab] - mx - __logf(s));
    if (per_sample) per_sample[b] = l;
    if (loss_sum) atomicAdd(loss_sum, l * loss_scale);
  }
}

}  // namespace

#define CK() ((int)cudaGetLastError())

template <typename T>
static int nchw_to_nhwc_launch(const T* x, void* y, int B, int C, int H, int W, int Cpad, cudaStream_t st) {
  const long long n = (long long)B * H * W * Cpad;
  if (Cpad % 4 == 0)
    geeps_launch_plain(nchw_to_nhwc_pix_kernel<T>, grid_1d((long long)B * H * W), 256, 0, st, x, (bf16*)y, B, C, H * W, Cpad);
  else
    geeps_launch_plain(nchw_f32_to_nhwc_bf16_kernel<T>, grid_1d(n), 256, 0, st, x, (bf16*)y, B, C, H, W, Cpad);
  return CK();
}

template <typename T>
static int nchw_to_s2d_launch(const T* x, void* y, int B, int C, int H, int W, int S, int Hs, int Ws, int Cpad,
                              cudaStream_t st) {
  if constexpr (sizeof(T) == 2) {
    const long long npix = (long long)B * Hs * Ws;
    if (S == 4 && C == 3 && s2d43_quads_ok(y, npix, Cpad) && ((uintptr_t)x & 3) == 0 && (long long)B * 3 * H * W % 2 == 0) {
      launch_s2d43_quads(Bf16Quads{(const bf16*)x, H, W}, y, npix, Hs, Ws, Cpad, st);
      return CK();
    }
  }
  if (S == 4 && C == 3 && Cpad % 8 == 0 && Cpad >= 48 && Cpad <= 64 && (((uintptr_t)y) & 15) == 0) {
    const int segs = (Ws + 31) / 32;
    geeps_launch_plain(nchw_to_s2d43_tile_kernel<T>, (unsigned)((long long)B * Hs * segs), 128, 0, st, x, (bf16*)y, B, H, W, Hs, Ws, Cpad,
                                                                                      segs);
  } else if (S == 4 && C == 3)
    geeps_launch_plain(nchw_to_s2d_kernel<4, 3, T>, grid_1d((long long)B * Hs * Ws), 256, 0, st, x, (bf16*)y, B, H, W, Hs, Ws, Cpad);
  else
    geeps_launch_plain(nchw_to_s2d_generic_kernel<T>, grid_1d((long long)B * Hs * Ws * Cpad), 256, 0, st, x, (bf16*)y, B, C, H, W, S,
                                                                                         Hs, Ws, Cpad);
  return CK();
}

extern "C" {

int geeps_nchw_to_nhwc_bf16(const void* x, int x_is_bf16, void* y, int B, int C, int H, int W, int Cpad, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  return x_is_bf16 ? nchw_to_nhwc_launch((const bf16*)x, y, B, C, H, W, Cpad, st)
                   : nchw_to_nhwc_launch((const float*)x, y, B, C, H, W, Cpad, st);
}
int geeps_nchw_f32_to_nhwc_bf16(const float* x, void* y, int B, int C, int H, int W, int Cpad, void* stream) {
  return geeps_nchw_to_nhwc_bf16(x, 0, y, B, C, H, W, Cpad, stream);
}

int geeps_nchw_to_s2d_bf16(const void* x, int x_is_bf16, void* y, int B, int C, int H, int W, int S, int Hs, int Ws,
                           int Cpad, void* stream) {
  if (S <= 0 || Cpad < S * S * C || (Cpad & 7)) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  return x_is_bf16 ? nchw_to_s2d_launch((const bf16*)x, y, B, C, H, W, S, Hs, Ws, Cpad, st)
                   : nchw_to_s2d_launch((const float*)x, y, B, C, H, W, S, Hs, Ws, Cpad, st);
}

int geeps_u8_transform_bf16(const GeepsU8Transform* p, void* stream) {
  if (p == nullptr || p->x == nullptr || p->y == nullptr) return (int)cudaErrorInvalidValue;
  const int S = p->S < 1 ? 1 : p->S;
  if (p->C < 1 || p->C > 4 || p->B < 1 || p->H < 1 || p->W < 1 || p->Hin < p->H || p->Win < p->W ||
      p->Cpad < S * S * p->C || p->Hs < 1 || p->Ws < 1)
    return (int)cudaErrorInvalidValue;
  // every source element an output position can name lies inside the cropped image
  if ((long long)(p->Hs - 1) * S >= p->H || (long long)(p->Ws - 1) * S >= p->W) return (int)cudaErrorInvalidValue;
  XformDev t;
  t.x = p->x; t.aug = p->aug;
  t.Hin = p->Hin; t.Win = p->Win; t.H = p->H; t.W = p->W;
  t.h_off = (p->Hin - p->H) / 2; t.w_off = (p->Win - p->W) / 2;
  for (int c = 0; c < 4; ++c) t.mean[c] = p->mean[c];
  t.scale = p->scale;
  cudaStream_t st = (cudaStream_t)stream;
  const long long npix = (long long)p->B * p->Hs * p->Ws;
  if (S == 4 && p->C == 3 && s2d43_quads_ok(p->y, npix, p->Cpad)) {
    U8Quads q;
    q.t = t;
    q.end = p->x + (long long)p->B * 3 * p->Hin * p->Win;
    launch_s2d43_quads(q, p->y, npix, p->Hs, p->Ws, p->Cpad, st);
  } else {
    geeps_launch_plain(u8_xform_generic_kernel, grid_1d((long long)p->B * p->Hs * p->Ws * p->Cpad), 256, 0, st, t, (bf16*)p->y, p->B, p->C,
                                                                                              S, p->Hs, p->Ws, p->Cpad);
  }
  return CK();
}

int geeps_col_mask_f32(float* g, const unsigned char* mask, long long rows, int cols, long long ld, void* stream) {
  geeps_launch_plain(col_mask_kernel, grid_1d(rows * cols), 256, 0, (cudaStream_t)stream, g, mask, rows, cols, ld);
  return CK();
}

int geeps_im2col(const void* x, void* col, const GeepsConvGeom* g, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const long long rows = (long long)g->B * g->OH * g->OW;
  const int kd = g->KH * g->KW * g->Cg;
  if (g->ldcol > kd)
    geeps_launch_plain(zero_col_pad_kernel, grid_1d(rows * (g->ldcol - kd)), 256, 0, st, (bf16*)col, rows, kd, g->ldcol);
  const bool a8 = (g->Cg % 8 == 0) && (g->C % 8 == 0) && (g->c0 % 8 == 0) && (g->ldcol % 8 == 0);
  const bool a4 = (g->Cg % 4 == 0) && (g->C % 4 == 0) && (g->c0 % 4 == 0) && (g->ldcol % 4 == 0);
  const int wgrid = grid_1d(rows * 32);   // one warp per patch-matrix row
  if (a8) geeps_launch_plain(im2col_kernel<8>, wgrid, 256, 0, st, (const bf16*)x, (bf16*)col, *g);
  else if (a4) geeps_launch_plain(im2col_kernel<4>, wgrid, 256, 0, st, (const bf16*)x, (bf16*)col, *g);
  else geeps_launch_plain(im2col_kernel<1>, wgrid, 256, 0, st, (const bf16*)x, (bf16*)col, *g);
  return CK();
}

int geeps_col2im(const void* dcol, void* dx, const GeepsConvGeom* g, int accumulate, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const long long pix = (long long)g->B * g->H * g->W;
  const bool a8 = (g->Cg % 8 == 0) && (g->C % 8 == 0) && (g->c0 % 8 == 0) && (g->ldcol % 8 == 0);
  if (a8) geeps_launch_plain(col2im_kernel<8>, grid_1d(pix * (g->Cg / 8)), 256, 0, st, (const bf16*)dcol, (bf16*)dx, *g, accumulate);
  else geeps_launch_plain(col2im_kernel<1>, grid_1d(pix * g->Cg), 256, 0, st, (const bf16*)dcol, (bf16*)dx, *g, accumulate);
  return CK();
}

// More than one block a SM and less than two: one.  Blocks that come up before their predecessor has left (geeps_launch)
// pair up on the SMs with room, and the step waits for those.  BatchNorm forward and backward, us, ordinary launches /
// dependent / dependent with this: 8 x 56 x 56 x 64, 196 blocks 13.0 / 14.6 / 12.7; 64 x 14 x 14 x 160, 261 blocks 16.6 /
// 18.1 / 15.2; 32 x 28 x 28 x 48, 149 blocks 14.3 / 13.7 / 11.9.  In an Inception module of 31 x 28 x 28 x 352 ordinary
// launches of these layers cost 10 us (313), dependent ones 302, with this 298.
static SlotGrid balanced(SlotGrid g) {
  const unsigned one = (unsigned)geeps_sm_count() / g.grid.x;
  if (g.grid.y > one && g.grid.y < 2 * one) g.grid.y = one;
  return g;
}
// reductions: one batch of four pixels per thread where that leaves SMs idle
static SlotGrid reduce_grid(int mode, long long P, int C) {
  return balanced(slot_grid(P, C, 4, kChannelBlocks, mode == 2 ? 1 : 2));
}
// element-wise passes with per-channel constants
static SlotGrid apply_grid(long long P, int C) {
  SlotGrid g = balanced(slot_grid(P, C, 4, kChannelBlocks, 0));
  g.smem = ((size_t)(C / 8) + g.grid.x - 1) / g.grid.x * 8 * 4 * sizeof(float);      // four constants per channel
  return g;
}
// ReLU mask with column sums
static SlotGrid relu_colsum_grid(long long P, int C) { return slot_grid(P, C, 4, 4, 1); }

int geeps_bn_forward(const void* x, void* y, const float* gamma, const float* beta, float* sums,
                     float* mean_rstd, float* running_mean, float* running_var, long long P, int C,
                     long long ldx, long long ldy, float eps, float momentum, int relu, void* stream) {
  if (C % 8) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  geeps_clear_f32(sums, 2LL * C, st);
  const SlotGrid rg = reduce_grid(0, P, C), ag = apply_grid(P, C);
  geeps_launch(channel_reduce_kernel<0>, rg.grid, rg.threads, rg.smem, st,
      (const bf16*)x, nullptr, nullptr, nullptr, sums, P, C, ldx, 0, 0, 1.f);
  geeps_launch(bn_finalize_kernel, (C + 127) / 128, 128, 0, st, sums, mean_rstd, running_mean, running_var, C,
                                                      1.f / (float)P, eps, momentum);
  geeps_launch(bn_apply_kernel, ag.grid, ag.threads, ag.smem, st, (const bf16*)x, (bf16*)y, mean_rstd, gamma, beta, P, C, ldx,
                                                        ldy, relu);
  return CK();
}

// the ReLU mask, where there is one, read from the output
static int bn_backward_by_output(const void* x, const void* dy, const void* y, void* dx, const float* mean_rstd,
                                 const float* gamma, float* sums, float* dgamma, float* dbeta, float* zero_after, long long P,
                                 int C, long long ldx, long long lddy, long long lddx, int relu, float grad_scale,
                                 cudaStream_t st) {
  const SlotGrid rg = reduce_grid(1, P, C), ag = apply_grid(P, C);
  geeps_launch(channel_reduce_kernel<1>, rg.grid, rg.threads, rg.smem, st,
      (const bf16*)x, (const bf16*)dy, (const bf16*)y, mean_rstd, sums, P, C, ldx, lddy, relu, 1.f);
  geeps_launch(relu ? bn_backward_kernel<MASK_Y> : bn_backward_kernel<MASK_NONE>, ag.grid, ag.threads, ag.smem, st,
               (const bf16*)x, (const bf16*)dy, (const bf16*)y, (bf16*)dx, mean_rstd, gamma, sums, dgamma, dbeta, P, C, ldx,
               lddy, lddx, relu, grad_scale, zero_after);
  return CK();
}
int geeps_bn_backward(const void* x, const void* dy, const void* y, void* dx, const float* mean_rstd,
                      const float* gamma, float* sums, float* dgamma, float* dbeta, long long P, int C,
                      long long ldx, long long lddy, long long lddx, int relu, float grad_scale, void* stream) {
  if (C % 8) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  geeps_clear_f32(sums, 2LL * C, st);
  return bn_backward_by_output(x, dy, y, dx, mean_rstd, gamma, sums, dgamma, dbeta, nullptr, P, C, ldx, lddy, lddx, relu,
                               grad_scale, st);
}

// The training-loop forms: `sums` must be zero on entry (2 C floats) and `zero_after` (or NULL) is zeroed for the
// layer's next reduction, so a BatchNorm layer that alternates forward and backward needs no memset and no separate
// finalisation launch: 2 launches per direction instead of 4 and 3.
// grid of a single-launch BatchNorm kernel: enough blocks for the reduction, never more than can be resident at
// once beside other kernels (the blocks wait for one another at the grid barrier)
static SlotGrid bn_coop_grid(long long P, int C) {
  SlotGrid g = slot_grid(P, C, 4, 1, 2);
  const size_t consts = apply_grid(P, C).smem;
  if (g.smem < consts) g.smem = consts;
  return g;
}
static bool bn_coop_enabled() {
  static int v = -1;
  // off by default: with at most one block per SM and a grid barrier the single launch is slower than two full-width
  // launches (Inception-BN-22K 5.84 against 5.65 ms per step, small net 1.96 against 1.95 ms).  The batches of the two launches serve
  // it too, though the backward form by the mask bits spills 16 bytes with them: 25088 x 192 forward 14.0 -> 11.3, backward 16.6 ->
  // 15.2 us, 6272 x 160 8.4 -> 7.6, 9.7 -> 9.4, 49 x 1024 11.2 -> 10.8, 11.3 -> 11.4
  if (v < 0) { const char* e = getenv("GEEPS_BN_COOP"); v = e ? atoi(e) : 0; }
  return v != 0;
}

int geeps_bn_forward_fused_bits(const void* x, void* y, const float* gamma, const float* beta, float* sums,
                                float* mean_rstd, float* running_mean, float* running_var, float* zero_after,
                                int* barrier, unsigned char* bits, long long P, int C, long long ldx, long long ldy,
                                float eps, float momentum, int relu, void* stream) {
  if (C % 8) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  if (barrier != nullptr && bn_coop_enabled()) {
    const bf16* xx = (const bf16*)x; bf16* yy = (bf16*)y;
    float inv_count = 1.f / (float)P;
    void* args[] = {&xx, &yy, &sums, &mean_rstd, &running_mean, &running_var, &gamma, &beta, &zero_after, &barrier,
                    &P, &C, &ldx, &ldy, &relu, &inv_count, &eps, &momentum, &bits};
    const SlotGrid cg = bn_coop_grid(P, C);
    cudaError_t e = cudaLaunchCooperativeKernel((void*)bn_forward_coop_kernel, cg.grid, dim3(cg.threads), args, cg.smem, st);
    return e == cudaSuccess ? CK() : (int)e;
  }
  const SlotGrid rg = reduce_grid(0, P, C), ag = apply_grid(P, C);
  geeps_launch(channel_reduce_kernel<0>, rg.grid, rg.threads, rg.smem, st,
      (const bf16*)x, nullptr, nullptr, nullptr, sums, P, C, ldx, 0, 0, 1.f);
  geeps_launch(bn_apply_fused_kernel, ag.grid, ag.threads, ag.smem, st, (const bf16*)x, (bf16*)y, sums, mean_rstd, running_mean,
                                                              running_var, gamma, beta, zero_after, P, C, ldx, ldy, relu,
                                                              1.f / (float)P, eps, momentum, bits);
  return CK();
}
int geeps_bn_backward_fused_bits(const void* x, const void* dy, const void* y, const unsigned char* bits, void* dx,
                                 float* mean_rstd, const float* gamma, float* sums, float* dgamma, float* dbeta,
                                 float* zero_after, int* barrier, long long P, int C, long long ldx, long long lddy,
                                 long long lddx, int relu, float grad_scale, void* stream) {
  if (C % 8) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  if (barrier != nullptr && bn_coop_enabled()) {
    const bool by_bits = bits != nullptr && relu;
    const bf16* xx = (const bf16*)x; const bf16* dd = (const bf16*)dy; const bf16* yy = (const bf16*)(by_bits ? bits : y);
    bf16* dxx = (bf16*)dx;
    void* args[] = {&xx, &dd, &yy, &dxx, &mean_rstd, &gamma, &sums, &dgamma, &dbeta, &zero_after, &barrier,
                    &P, &C, &ldx, &lddy, &lddx, &relu, &grad_scale};
    const SlotGrid cg = bn_coop_grid(P, C);
    void* kernel = by_bits ? (void*)bn_backward_coop_kernel<true> : (void*)bn_backward_coop_kernel<false>;
    cudaError_t e = cudaLaunchCooperativeKernel(kernel, cg.grid, dim3(cg.threads), args, cg.smem, st);
    return e == cudaSuccess ? CK() : (int)e;
  }
  if (bits != nullptr && relu) {
    const SlotGrid rg = reduce_grid(3, P, C), ag = apply_grid(P, C);
    geeps_launch(channel_reduce_kernel<3>, rg.grid, rg.threads, rg.smem, st, (const bf16*)x, (const bf16*)dy, (const bf16*)bits,
                                                                   mean_rstd, sums, P, C, ldx, lddy, relu, 1.f);
    geeps_launch(bn_backward_kernel<MASK_BITS>, ag.grid, ag.threads, ag.smem, st, (const bf16*)x, (const bf16*)dy, (const bf16*)bits, (bf16*)dx,
                                                             mean_rstd, gamma, sums, dgamma, dbeta, P, C, ldx, lddy, lddx,
                                                             relu, grad_scale, zero_after);
    return CK();
  }
  return bn_backward_by_output(x, dy, y, dx, mean_rstd, gamma, sums, dgamma, dbeta, zero_after, P, C, ldx, lddy, lddx, relu,
                               grad_scale, st);
}

int geeps_colsum(const void* x, float* out, long long P, int C, long long ldx, float scale, int zero_first,
                 void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if ((C % 8) || (ldx % 8) || C > 4096) {
    geeps_launch(colsum_simple_kernel, (C + 127) / 128, 128, 0, st, (const bf16*)x, out, P, C, ldx, scale, !zero_first);
    return CK();
  }
  if (zero_first) geeps_clear_f32(out, C, st);
  const SlotGrid rg = reduce_grid(2, P, C);
  geeps_launch(channel_reduce_kernel<2>, rg.grid, rg.threads, rg.smem, st,
      (const bf16*)x, nullptr, nullptr, nullptr, out, P, C, ldx, 0, 0, scale);
  return CK();
}

int geeps_copy_f32(float* dst, const float* src, long long n, void* stream) {
  return (int)cudaMemcpyAsync(dst, src, sizeof(float) * (size_t)n, cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
}

int geeps_relu_backward(const void* dy, const void* y, void* dx, long long n, void* stream) {
  if (n % 8) return (int)cudaErrorInvalidValue;
  geeps_launch_plain(relu_backward_kernel, grid_1d(n / 8), 256, 0, (cudaStream_t)stream, (const bf16*)dy, (const bf16*)y, (bf16*)dx, n / 8);
  return CK();
}

int geeps_relu_backward_2d(const void* dy, const void* y, void* dx, long long P, int C, long long lddy, long long ldy,
                           long long lddx, void* stream) {
  if (C % 8 || lddy % 8 || ldy % 8 || lddx % 8) return (int)cudaErrorInvalidValue;
  geeps_launch_plain(relu_backward_2d_kernel, grid_1d(P * (C / 8)), 256, 0, (cudaStream_t)stream, (const bf16*)dy, (const bf16*)y,
                                                                                 (bf16*)dx, P, C, lddy, ldy, lddx);
  return CK();
}
int geeps_relu_backward_colsum(const void* dy, const void* y, void* dx, float* colsum, long long P, int C,
                               long long lddy, long long ldy, long long lddx, void* stream) {
  return geeps_relu_backward_colsum_clear(dy, y, dx, colsum, P, C, lddy, ldy, lddx, nullptr, 0, stream);
}
// Zeros to the clear_n values at `clear` as well: on the way in a short pass, where a launch for them in front of each group's
// weight gradient costs more than its bytes (backward passes of layers, us, a launch each / so: 1000 x 48 from 80 channels
// 15.5 / 13.7, two groups 1922 x 96 from 128 31.2 / 27.2, 6100 x 232 from 88 32.0 / 29.8, 22275 x 176 from 40 49.9 / 46.8).
// After a long pass they keep a launch, one for all groups: the blocks of a weight gradient that follows it directly come up
// in the order in which its blocks leave, on other SMs than the tiles they share lie well on (44800 x 264 from 144, 5 x 5
// 295.5 us, 306.3 without the launch; 93600 x 352 from 88 632, 650; though 43264 x 384 from 256 145.8, 143.2).
int geeps_relu_backward_colsum_clear(const void* dy, const void* y, void* dx, float* colsum, long long P, int C,
                                     long long lddy, long long ldy, long long lddx, float* clear, long long clear_n, void* stream) {
  if (C % 8 || lddy % 8 || ldy % 8 || lddx % 8 || C > 8192 || clear_n < 0 || (clear_n > 0 && !clear)) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  geeps_clear_f32(colsum, C, st);
  const bool apart = P * C > (1LL << 22);
  float* const along = apart ? nullptr : clear;
  const long long along_n = apart ? 0 : clear_n;
  const SlotGrid rg = relu_colsum_grid(P, C);
  geeps_launch_plain(relu_backward_colsum_kernel, rg.grid, rg.threads, rg.smem, st,
      (const bf16*)dy, (const bf16*)y, (bf16*)dx, colsum, P, C, lddy, ldy, lddx, along, along_n, (int)clear_head(along, along_n));
  if (apart && clear_n > 0) geeps_clear_f32(clear, clear_n, st);
  return CK();
}
int geeps_f32_to_bf16_2d(const float* src, void* dst, long long P, int C, long long lds, long long ldd, int relu,
                         void* stream) {
  if (C % 8 || lds % 4 || ldd % 8 || ((uintptr_t)src & 15) || ((uintptr_t)dst & 15)) return (int)cudaErrorInvalidValue;
  geeps_launch_plain(f32_to_bf16_2d_kernel, grid_1d(P * (C / 8)), 256, 0, (cudaStream_t)stream, src, (bf16*)dst, P, C, lds, ldd, relu);
  return CK();
}
int geeps_add_bf16_2d_n(void* dst, const void* s0, const void* s1, const void* s2, long long P, int C, long long ldd,
                        long long ld0, long long ld1, long long ld2, void* stream) {
  const int n = s2 ? 3 : (s1 ? 2 : 1);
  if (C % 8 || ldd % 8 || ld0 % 8 || (n > 1 && ld1 % 8) || (n > 2 && ld2 % 8) || !s0 || (s2 && !s1))
    return (int)cudaErrorInvalidValue;
  const AddSrc src = {{(const bf16*)s0, (const bf16*)s1, (const bf16*)s2}, {ld0, ld1, ld2}};
  const long long total = P * (C / 8);
  const bool dense = ldd == C && ld0 == C && (n < 2 || ld1 == C) && (n < 3 || ld2 == C);
  const int grid = grid_1d(total);
  cudaStream_t st = (cudaStream_t)stream;
#define ADD_2D(N, DENSE) geeps_launch_plain(add_2d_kernel<N, DENSE>, grid, 256, 0, st, (bf16*)dst, src, total, C / 8, ldd)
  if (dense) { if (n == 3) ADD_2D(3, true); else if (n == 2) ADD_2D(2, true); else ADD_2D(1, true); }
  else { if (n == 3) ADD_2D(3, false); else if (n == 2) ADD_2D(2, false); else ADD_2D(1, false); }
#undef ADD_2D
  return CK();
}

int geeps_dropout(const void* x, void* y, long long n, float p, unsigned long long seed, void* stream) {
  return geeps_dropout_ref(x, y, n, p, seed, nullptr, stream);
}
int geeps_dropout_ref(const void* x, void* y, long long n, float p, unsigned long long seed, const int* step_ref,
                      void* stream) {
  const bool vec = n % 8 == 0 && (((uintptr_t)x | (uintptr_t)y) & 15) == 0;
  geeps_launch_plain(vec ? dropout_kernel<true> : dropout_kernel<false>, grid_1d(vec ? n / 8 : n), 256, 0, (cudaStream_t)stream,
                     (const bf16*)x, (bf16*)y, n, p, seed, step_ref);
  return CK();
}

int geeps_lrn_forward(const void* x, void* y, void* rscale, long long P, int C, int size, float alpha, float beta,
                      float k, void* stream) {
  const int g8 = grid_1d(P * (C / 8));
  cudaStream_t st8 = (cudaStream_t)stream;
  if (C % 8 == 0 && size == 5)
    geeps_launch_plain(lrn_forward_v8_kernel<2>, g8, 256, 0, st8, (const bf16*)x, (bf16*)y, (bf16*)rscale, P, C, size, alpha, beta, k);
  else if (C % 8 == 0 && size == 3)
    geeps_launch_plain(lrn_forward_v8_kernel<1>, g8, 256, 0, st8, (const bf16*)x, (bf16*)y, (bf16*)rscale, P, C, size, alpha, beta, k);
  else if (C % 8 == 0 && size == 7)
    geeps_launch_plain(lrn_forward_v8_kernel<3>, g8, 256, 0, st8, (const bf16*)x, (bf16*)y, (bf16*)rscale, P, C, size, alpha, beta, k);
  else
    geeps_launch_plain(lrn_forward_kernel, grid_1d(P * C), 256, 0, (cudaStream_t)stream, (const bf16*)x, (bf16*)y, (bf16*)rscale, P, C, size,
                                                                        alpha, beta, k);
  return CK();
}
int geeps_lrn_backward(const void* x, const void* y, const void* rscale, const void* dy, void* dx, long long P,
                       int C, int size, float alpha, float beta, int relu_mask, float* colsum, void* stream) {
  int g8 = grid_1d(P * (C / 8));
  cudaStream_t st8 = (cudaStream_t)stream;
  size_t cs_smem = 0;
  if (colsum != nullptr) {
    if (C % 8 || (size != 3 && size != 5 && size != 7) || C > 8192) return (int)cudaErrorInvalidValue;
    // gridDim * 256 must be a multiple of C/8 (one channel group per thread): round the grid down to a multiple of m
    int cv = C / 8, a = cv, b = 256;
    while (b) { int t = a % b; a = b; b = t; }
    const int m = cv / a;
    g8 = g8 >= m ? g8 / m * m : m;
    cs_smem = sizeof(float) * C;
    geeps_clear_f32(colsum, C, st8);
  }
  if (C % 8 == 0 && size == 5)
    geeps_launch_plain(lrn_backward_v8_kernel<2>, g8, 256, cs_smem, st8, (const bf16*)x, (const bf16*)y, (const bf16*)rscale, (const bf16*)dy, (bf16*)dx, P, C, size, alpha, beta, relu_mask, colsum);
  else if (C % 8 == 0 && size == 3)
    geeps_launch_plain(lrn_backward_v8_kernel<1>, g8, 256, cs_smem, st8, (const bf16*)x, (const bf16*)y, (const bf16*)rscale, (const bf16*)dy, (bf16*)dx, P, C, size, alpha, beta, relu_mask, colsum);
  else if (C % 8 == 0 && size == 7)
    geeps_launch_plain(lrn_backward_v8_kernel<3>, g8, 256, cs_smem, st8, (const bf16*)x, (const bf16*)y, (const bf16*)rscale, (const bf16*)dy, (bf16*)dx, P, C, size, alpha, beta, relu_mask, colsum);
  else
    geeps_launch_plain(lrn_backward_kernel, grid_1d(P * C), 256, 0, (cudaStream_t)stream, (const bf16*)x, (const bf16*)y, (const bf16*)rscale,
                                                                         (const bf16*)dy, (bf16*)dx, P, C, size, alpha,
                                                                         beta, relu_mask);
  return CK();
}

static int maxpool_forward(const void* x, void* y, void* argmax, const GeepsPoolGeom* g, int relu_mask, void* stream) {
  if (g->C % 8 || g->ldx % 8 || g->ldy % 8 || g->K * g->K > 255) return (int)cudaErrorInvalidValue;
  geeps_launch_plain(maxpool_forward_kernel, g->B * g->OH, pool_block(g->C / 8), 0, (cudaStream_t)stream, (const bf16*)x, (bf16*)y,
                                                                                        (uint8_t*)argmax, *g, relu_mask);
  return CK();
}
int geeps_maxpool_forward(const void* x, void* y, void* argmax, const GeepsPoolGeom* g, void* stream) {
  return maxpool_forward(x, y, argmax, g, 0, stream);
}
int geeps_maxpool_forward_relu(const void* x, void* y, void* argmax, const GeepsPoolGeom* g, void* stream) {
  return maxpool_forward(x, y, argmax, g, 1, stream);
}
int geeps_maxpool_backward(const void* dy, const void* argmax, void* dx, const GeepsPoolGeom* g, int accumulate,
                           void* stream) {
  if (g->C % 8 || g->ldx % 8 || g->ldy % 8) return (int)cudaErrorInvalidValue;
  if (g->K == 3 && g->stride == 2 && g->pad >= 0 && g->H > 0 && g->W > 0) {
    const long long qh = ((g->H + g->pad - 1) >> 1) - (g->pad >> 1) + 1, qw = ((g->W + g->pad - 1) >> 1) - (g->pad >> 1) + 1;
    const long long total = g->B * qh * qw * (g->C / 8);
    if (total > 0 && total < (1LL << 31)) {
      geeps_launch_plain(maxpool3s2_backward_kernel, (int)((total + 255) / 256), 256, 0, (cudaStream_t)stream, (const bf16*)dy,
          (const uint8_t*)argmax, (bf16*)dx, *g, accumulate, (unsigned)qh, (unsigned)qw, (unsigned)total);
      return CK();
    }
  }
  // other overlapping windows: stage the covering output rows in shared memory when they fit
  const int rows_per_block = g->stride > 1 ? 2 * g->stride : 2;
  const int max_oh = (rows_per_block + g->K - 2) / g->stride + 1;
  const size_t smem = (size_t)max_oh * g->OW * g->C * 3;
  if (g->K > g->stride && smem <= 96 * 1024) {
    static bool attr_set = false;
    if (!attr_set) {
      cudaFuncSetAttribute(maxpool_backward_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      attr_set = true;
    }
    const int row_blocks = (g->H + rows_per_block - 1) / rows_per_block;
    geeps_launch_plain(maxpool_backward_smem_kernel, g->B * row_blocks, pool_block(g->C / 8), smem, (cudaStream_t)stream,
        (const bf16*)dy, (const uint8_t*)argmax, (bf16*)dx, *g, accumulate, rows_per_block, max_oh);
    return CK();
  }
  geeps_launch_plain(maxpool_backward_kernel, g->B * g->H, pool_block(g->C / 8), 0, (cudaStream_t)stream,
      (const bf16*)dy, (const uint8_t*)argmax, (bf16*)dx, *g, accumulate);
  return CK();
}
int geeps_channel_blocks(long long P, int C, int* out) { return geeps_channel_pass_blocks(0, P, C, out); }
int geeps_channel_pass_blocks(int pass, long long P, int C, int* out) {
  if (pass < 0 || pass > 3) return (int)cudaErrorInvalidValue;
  const SlotGrid g = pass == 3 ? relu_colsum_grid(P, C) : pass == 2 ? apply_grid(P, C) : reduce_grid(pass == 1 ? 2 : 0, P, C);
  out[0] = (int)g.grid.x; out[1] = (int)g.grid.y; out[2] = g.threads; out[3] = (int)g.smem;
  return 0;
}
int geeps_avgpool_blocks(int C, int width, long long rows, int group, int* out) {
  const PoolGrid g = avgpool_grid(C / 8, width, rows, group != 0);
  const unsigned v[5] = {g.grid.x, g.grid.y, g.block.x, g.block.y, g.block.z};
  for (int i = 0; i < 5; ++i) out[i] = (int)v[i];
  return 0;
}
// 3 x 3 windows at stride 1 that lie in the padded image (each then has nine pixels of it), 32-bit thread numbers
static bool avgpool3_ok(const GeepsPoolGeom* g) {
  return g->K == 3 && g->stride == 1 && g->pad >= 0 && g->OH == g->H + 2 * g->pad - 2 && g->OW == g->W + 2 * g->pad - 2 &&
         g->OH > 0 && g->OW > 0 && g->B > 0 && g->C >= 8 && (long long)g->B * (g->H + 2 * g->pad) * (g->W + 2 * g->pad) * (g->C / 8) < (1LL << 30);
}
// Four rows a thread where that leaves a full set of resident threads, else one: 4 x 14 x 14 x 576 2.9 and 2.9 us with four
// rows, 2.7 and 2.7 with one; 100 x 8 x 8 x 336 4.1 and 4.0, 5.6 and 6.3; 512 x 5 x 5 x 24 2.9 and 2.9, 2.3 and 2.4.
static int avgpool3(bool bwd, const void* in, void* out, const GeepsPoolGeom* g, int accumulate, cudaStream_t st) {
  const int H = bwd ? g->OH : g->H, W = bwd ? g->OW : g->W, OH = bwd ? g->H : g->OH, OW = bwd ? g->W : g->OW, cv = g->C / 8;
  const bool four = (long long)g->B * OH * OW * cv >= 512LL * geeps_sm_count();
  const int blocks_h = four ? (OH + 3) / 4 : OH, total = g->B * blocks_h * OW * cv;
  geeps_launch_plain(bwd ? (four ? avgpool3_kernel<true, 4> : avgpool3_kernel<true, 1>)
                         : (four ? avgpool3_kernel<false, 4> : avgpool3_kernel<false, 1>), (total + 255) / 256, 256, 0, st,
                     (const bf16*)in, (bf16*)out, H, W, OH, OW, cv, bwd ? g->ldy : g->ldx, bwd ? g->ldx : g->ldy,
                     bwd ? g->pad - 2 : -g->pad, blocks_h, total, accumulate);
  return CK();
}
int geeps_avgpool_forward(const void* x, void* y, const GeepsPoolGeom* g, void* stream) {
  if (g->C % 8 || g->ldx % 8 || g->ldy % 8) return (int)cudaErrorInvalidValue;
  if (avgpool3_ok(g)) return avgpool3(false, x, y, g, 0, (cudaStream_t)stream);
  const PoolGrid pg = avgpool_grid(g->C / 8, g->OW, (long long)g->B * g->OH, g->K <= 3);
  cudaStream_t st = (cudaStream_t)stream;
  if (pg.grid.x == 0) return 0;
  if (pg.block.z == 1) geeps_launch_plain(avgpool_forward_kernel<false>, pg.grid, pg.block, 0, st, (const bf16*)x, (bf16*)y, *g);
  else geeps_launch_plain(avgpool_forward_kernel<true>, pg.grid, pg.block, 0, st, (const bf16*)x, (bf16*)y, *g);
  return CK();
}
int geeps_avgpool_backward(const void* dy, void* dx, const GeepsPoolGeom* g, int accumulate, void* stream) {
  if (g->C % 8 || g->ldx % 8 || g->ldy % 8) return (int)cudaErrorInvalidValue;
  if (avgpool3_ok(g)) return avgpool3(true, dy, dx, g, accumulate, (cudaStream_t)stream);
  const PoolGrid pg = avgpool_grid(g->C / 8, g->W, (long long)g->B * g->H, g->K <= 3 * g->stride);
  cudaStream_t st = (cudaStream_t)stream;
  if (pg.grid.x == 0) return 0;
  if (pg.block.z == 1)
    geeps_launch_plain(avgpool_backward_kernel<false>, pg.grid, pg.block, 0, st, (const bf16*)dy, (bf16*)dx, *g, accumulate);
  else
    geeps_launch_plain(avgpool_backward_kernel<true>, pg.grid, pg.block, 0, st, (const bf16*)dy, (bf16*)dx, *g, accumulate);
  return CK();
}

int geeps_softmax_ce(const float* logits, const long long* labels, float* loss_sum, float* per_sample,
                     void* dlogits, int B, int C, long long ldl, long long ldd, float loss_scale, float grad_scale,
                     int zero_loss, int* status, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (zero_loss && loss_sum) geeps_clear_f32(loss_sum, 1, st);
  // Narrow rows keep the order in which 256 threads have always summed them.  The register kernel takes the same time up to
  // 1000 classes and less from there (32 x 2000 8.5 -> 6.5 us, 32 x 4000 10.5 -> 7.0, 256 x 4000 10.6 -> 8.7; rows off a
  // 16-byte boundary 8.5, 8.5 and 10.6), 32 x 6000 12.6 -> 8.5, 32 x 21841 54 -> 8.
  if (C < 4096) {
    geeps_launch(softmax_ce_small_kernel, B, 256, 0, st, logits, labels, loss_sum, per_sample, (bf16*)dlogits, C, ldl, ldd, loss_scale,
                                               grad_scale, status);
    return CK();
  }
  int threads = (C / 8 + 31) / 32 * 32;
  threads = threads > 1024 ? 1024 : threads;
  const bool vec = ldl % 4 == 0 && ((uintptr_t)logits & 15) == 0 &&
                   (dlogits == nullptr || (ldd % 8 == 0 && ((uintptr_t)dlogits & 15) == 0));
  if (vec)
    geeps_launch(softmax_ce_kernel<true>, B, threads, 0, st, logits, labels, loss_sum, per_sample, (bf16*)dlogits, C, ldl, ldd,
                                                   loss_scale, grad_scale, status);
  else
    geeps_launch(softmax_ce_kernel<false>, B, threads, 0, st, logits, labels, loss_sum, per_sample, (bf16*)dlogits, C, ldl, ldd,
                                                    loss_scale, grad_scale, status);
  return CK();
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// BatchNorm forward for callers that must not allocate device memory.
//
// geeps_bn_forward needs 2*C floats of scratch for the per-channel sums and leaves it to the caller to provide them.  Two
// kinds of callers of this library cannot do that: code running under the parameter server's memory plan, where every
// byte of the GPU budget has been handed out before the first clock, and plain C/C++ hosts that link the library without
// any device allocator of their own and must not pay cudaMalloc's device-wide synchronisation inside their step loop.
// For them the sums are formed in the 2*C floats that receive mean and 1/std, and finalised in place: nothing is shared
// between calls, so calls on several streams, threads or ranks may overlap and the call may be captured.
// ---------------------------------------------------------------------------------------------
#include <stdio.h>

extern "C" {

int geeps_bn_noalloc_max_channels() { return GEEPS_BN_NOALLOC_MAX_CHANNELS; }

int geeps_bn_forward_noalloc(const void* x, void* y, const float* gamma, const float* beta, float* mean_rstd,
                             float* running_mean, float* running_var, long long P, int C, long long ldx,
                             long long ldy, float eps, float momentum, int relu, void* stream) {
  if (C <= 0 || C % 8) return (int)cudaErrorInvalidValue;
  if (C > GEEPS_BN_NOALLOC_MAX_CHANNELS) {
    fprintf(stderr, "geeps_bn_forward_noalloc: %d channels exceed the limit of %d channels; "
                    "use geeps_bn_forward with caller-provided scratch\n", C, GEEPS_BN_NOALLOC_MAX_CHANNELS);
    return GEEPS_ERR_NOALLOC_TOO_LARGE;
  }
  return geeps_bn_forward(x, y, gamma, beta, mean_rstd, mean_rstd, running_mean, running_var, P, C, ldx, ldy, eps, momentum,
                          relu, stream);
}

}  // extern "C"
