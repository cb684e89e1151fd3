// Shared device helpers for every sm_100a kernel in this library.
//
// Conventions used by all kernels:
//  * A parameter-server row is 128 fp32 values = 512 bytes (same row shape as
//    include/geeps-user-defined-types.hpp:55-57 of the reference).
//  * No kernel traps, asserts or spins forever.  A wait that runs out of its
//    time budget, or an index that fails a bounds check, records a code in a
//    caller-provided 4-word status block and the kernel returns normally.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#define GEEPS_ROW_FLOATS 128
#define GEEPS_ROW_BYTES 512

// status[0] = first error code (0 = ok), status[1] = kernel id,
// status[2] = detail (flag index / row index), status[3] = observed value.
enum GeepsStatusCode : int {
  GEEPS_OK = 0,
  GEEPS_ERR_TIMEOUT = 1,       // a bounded wait expired
  GEEPS_ERR_BOUNDS = 2,        // an index failed a software bounds check
  GEEPS_ERR_ALIGN = 3,         // a pointer failed an alignment check
};

enum GeepsKernelId : int {
  KID_ROW_GATHER = 1, KID_ROW_SCATTER = 2, KID_ROW_SCATTER_ADD = 3, KID_ROW_AXPY = 4,
  KID_PUSH_APPLY = 10, KID_PULL = 11, KID_PUSHPULL = 12, KID_FLAG_WAIT = 13,
  KID_GEMM_TC = 20, KID_GEMM_SIMT = 21, KID_PULL_GEMM = 22, KID_CONV_TC = 23,
};

// Number of SMs of the current device (cudaDevAttrMultiProcessorCount), read once per device and cached:
// grids are sized from it, never from a literal.
inline int geeps_sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); dev = 0; }
  int n = cached[dev];
  if (n <= 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) { cudaGetLastError(); n = 148; }
    cached[dev] = n;
  }
  return n;
}

// Programmatic dependent launch: a kernel launched with geeps_launch() may start while its predecessor in the stream
// drains - its blocks become resident as the predecessor's leave - and must call geeps_pdl_wait(), in every thread and
// before it touches global memory, which returns when the predecessor is complete and its writes are visible.  Since every
// kernel waits for its own predecessor that way, a kernel that is complete has all work enqueued before it behind it, and
// later launches of any kind (library kernels, copies, events) order themselves as after an ordinary launch.
__device__ __forceinline__ void geeps_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The blocks of the next kernel may start, as far as there is room for them, once every block has called this (or left).
// Called before the wait of its own kernel has returned it would let a third kernel in; all kernels call it after.
// Where it stands: in the tensor-core kernels behind the last load of a block, whose shared memory leaves no room for
// another block before (the pair GEMM has none: its successor comes up when it ends); in the others at the start, except the
// passes of a BatchNorm over a large tensor (batchnorm_enter).
__device__ __forceinline__ void geeps_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void geeps_pdl_enter() { geeps_pdl_wait(); geeps_pdl_trigger(); }

template <typename... P, typename... A>
inline void geeps_launch_as(int dependent, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);      // an error is also what cudaGetLastError() returns
}
// Which launch a kernel gets (us in a captured chain of 16, ordinary / dependent, unless said otherwise).
// geeps_launch, dependent: tensor-core kernels, channel sums, BatchNorm, softmax.  They have at most as many blocks as fit at
// once (softmax: one a row), and in a network's chains the way from one kernel to the next is what is gained: 32 x 14 x 14, 128 ->
// 160, 3 x 3 7.9 / 7.0; GEMM 6272 x 160, K = 576 5.6 / 4.8; BatchNorm of 100 x 16 x 16 x 144 forward and backward 22.6 / 21.2;
// softmax of 256 x 1000 7.6 / 6.6; an Inception module with BatchNorm's launches ordinary 199, dependent 193, its classifier
// 82.3, 80.9.  Forward and backward of 60 convolution layers take 4 % less.  Not every kernel gains: CTAs of a part of a wave
// come up where the predecessor leaves room, and the other way round 35 x 8 x 8, 72 -> 312 takes 9.7 / 11.5 after itself.
// geeps_launch_plain: kernels of many short blocks.  Early blocks wait on the SMs that have room first, as many as fit, and the
// other SMs run dry: max pooling of 32 x 14 x 14 x 576 12.1 / 15.1, its backward at 608 channels 19.2 / 23.5; average pooling
// of 8 x 14 x 14 x 576 4.1 / 4.4, backward 5.5 / 6.1; LRN + pooling backward of 2 x 43 x 43 x 88 8.8 / 10.2; layouts: fp32 to
// space-to-depth at 16 x 227 x 227 3.9 / 4.2 (72 channels, 32 x 224 x 224 8.3 / 9.3), to NHWC at 100 x 32 x 32 2.3 / 2.5, from
// 8 bits 9.1 / 9.6; the sum of three gradients of 16 Mi values 13.6 / 14.6, the ReLU mask 11.3 / 11.9.  Where a size does not
// suffer it gains 0.1 to 0.3.  In a network: Inception module 192.0 / 192.8, AlexNet's training step 2212 / 2218.
template <typename... P, typename... A>
inline void geeps_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  geeps_launch_as(1, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}
template <typename... P, typename... A>
inline void geeps_launch_plain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  geeps_launch_as(0, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}

__device__ __forceinline__ void geeps_report(int* status, int code, int kid, int detail, int seen) {
  if (status == nullptr) return;
  if (atomicCAS(status, 0, code) == 0) {
    status[1] = kid;
    status[2] = detail;
    status[3] = seen;
    __threadfence_system();
  }
}

__device__ __forceinline__ uint64_t geeps_globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---- system-scope flag words (monotone clock stamps; wait for >= expected) ----
__device__ __forceinline__ int ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(int* p, int v) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed_sys(const int* p) {
  int v;
  asm volatile("ld.relaxed.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Spin until *flag >= expected or budget_ns elapses.  Returns true on success.
// The polls are relaxed loads spaced by a sleep that backs off to 4 us, and one acquire load orders the
// data behind the flag once it has been seen: a waiting warp shares its SM with compute kernels (the
// persistent tensor-core kernels assign tiles statically, so one slowed SM slows the whole kernel), and
// system-scope acquires issued every microsecond were measurably slowing them.
__device__ __forceinline__ bool geeps_wait_ge(const int* flag, int expected, uint64_t budget_ns,
                                              int* seen_out) {
  int v = ld_acquire_sys(flag);
  if (v >= expected) { if (seen_out) *seen_out = v; return true; }
  const uint64_t t0 = geeps_globaltimer();
  unsigned backoff = 64;
  for (;;) {
    v = ld_relaxed_sys(flag);
    if (v >= expected) {
      v = ld_acquire_sys(flag);
      if (seen_out) *seen_out = v;
      return true;
    }
    if (geeps_globaltimer() - t0 > budget_ns) { if (seen_out) *seen_out = v; return false; }
    __nanosleep(backoff);
    if (backoff < 4096) backoff <<= 1;
  }
}

// 16-byte vector helpers
__device__ __forceinline__ float4 ld_f4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st_f4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
// Zeros to c[0, n) by the threads at, at + stride, ...: `head` single values up to a 16-byte boundary, vectors, the rest
__device__ __forceinline__ void clear_range(float* c, long long n, int head, long long at, long long stride) {
  if (at < head) c[at] = 0.f;
  const long long n4 = (n - head) >> 2;
  for (long long i = at; i < n4; i += stride) st_f4(c + head + 4 * i, make_float4(0.f, 0.f, 0.f, 0.f));
  const long long tail = head + 4 * n4;
  if (at < n - tail) c[tail + at] = 0.f;
}
inline long long clear_head(const float* c, long long n) {
  const long long head = ((16 - ((uintptr_t)c & 15)) & 15) / 4;
  return head < n ? head : n;
}
__device__ __forceinline__ float4 ld_f4_nc_stream(const float* p) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
// Weak 16-byte load that bypasses the (non-coherent) L1 and is served from L2 / the peer.  Correct for data
// that was completely written before this kernel started or before a flag this kernel's stream waited on
// (stream order and the release / acquire on the flag order those writes before this load).
__device__ __forceinline__ float4 ld_f4_cg(const float* p) {
  float4 v;
  asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
// Volatile-strength peer load: data written by another GPU during this kernel must
// not be served from a stale L1 line.
__device__ __forceinline__ float4 ld_f4_peer(const float* p) {
  float4 v;
  asm volatile("ld.relaxed.sys.global.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}

// ---- NVSwitch multicast (multimem) accesses through a multicast mapping: 16-byte aligned addresses ----
// sum over every bound device of the float4 at this offset, added in the switch
__device__ __forceinline__ float4 multimem_ld_reduce_f4(const float* p) {
  float4 v;
  asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
// store to every bound device
__device__ __forceinline__ void multimem_st_f4(float* p, float4 v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};"
               ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void multimem_st_bf16x4(void* p, uint2 v) {
  asm volatile("multimem.st.relaxed.sys.global.v2.bf16x2 [%0], {%1,%2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
