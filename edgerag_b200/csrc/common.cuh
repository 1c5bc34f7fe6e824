// Shared helpers of the sm_100a kernels: element conversion, reductions, error reporting.
//
// Every exported function is `extern "C"`, takes raw device pointers and a stream, launches on
// that stream, allocates nothing, and returns 0 or a negative code whose text `erb_last_error()`
// gives.  Each source is compiled twice, into one library per element type (float for the 32-bit
// path, bfloat16 for serving), so a run builds and loads only the type it uses.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

// Each source is compiled once per element type: -DERB_ELEM=0 (float) or 1 (bfloat16).
#ifndef ERB_ELEM
#error "compile with -DERB_ELEM=0 (float) or -DERB_ELEM=1 (bfloat16)"
#endif
#if ERB_ELEM == 0
typedef float elem_t;
#else
typedef __nv_bfloat16 elem_t;
#endif

#define ERB_OK 0
#define ERB_ERR_ARG -1
#define ERB_ERR_CUDA -2
#define ERB_ERR_UNSUPPORTED -3

namespace erb {

// One message buffer per library; written by the host wrappers only.
inline char* error_buffer() {
  static thread_local char buf[512];
  return buf;
}

inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(error_buffer(), 512, fmt, ap);
  va_end(ap);
  return code;
}

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return ERB_OK;
}

// Streaming multiprocessors of the current device (asked once per device).
inline int sm_count() {
  static int counts[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
  if (!counts[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
    counts[dev] = n;
  }
  return counts[dev];
}

template <typename T> struct Elem;
template <> struct Elem<float> {
  static __device__ __forceinline__ float load(const float* p) { return *p; }
  static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
  static __device__ __forceinline__ float round(float v) { return v; }
};
template <> struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float load(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
  static __device__ __forceinline__ float round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
};

// Loads `N` consecutive elements (N * sizeof(T) must be 16 bytes, pointer 16-byte aligned) as floats.
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* out) {
  uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __bfloat1622float2(h[i]);
    out[2 * i] = f.x;
    out[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void load4(const float* p, float* out) {
  float4 raw = *reinterpret_cast<const float4*>(p);
  out[0] = raw.x; out[1] = raw.y; out[2] = raw.z; out[3] = raw.w;
}

// Four neighbouring elements as floats (pointers aligned to four elements).
template <typename T> struct Pack4;
template <> struct Pack4<float> {
  static __device__ __forceinline__ void load(const float* p, float* v) { load4(p, v); }
  static __device__ __forceinline__ void store(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <> struct Pack4<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* v) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(raw.x << 16); v[1] = __uint_as_float(raw.x & 0xffff0000u);
    v[2] = __uint_as_float(raw.y << 16); v[3] = __uint_as_float(raw.y & 0xffff0000u);
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float* v) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
  }
};

// silu(g) * u in float.  Where the result is rounded to 16 bits (ERB_ELEM == 1) the exponential and the
// division are the fast forms (relative error about 2^-21, far below that rounding); the 32-bit path keeps
// the exact ones.  Every kernel that gates (the gate kernel, the gated epilogues of the products for few
// rows) calls this, so that they agree to the bit.
__device__ __forceinline__ float silu_mul(float g, float u) {
#if ERB_ELEM == 1
  return __fdividef(g, 1.f + __expf(-g)) * u;
#else
  return g / (1.f + expf(-g)) * u;
#endif
}

// x * sigmoid(z) in float (an entry of an output gate), in the forms of silu_mul.
__device__ __forceinline__ float sigmoid_mul(float x, float z) {
#if ERB_ELEM == 1
  return __fdividef(x, 1.f + __expf(-z));
#else
  return x / (1.f + expf(-z));
#endif
}

// gelu(g) * u with the tanh form of gelu, 0.5 g (1 + tanh(sqrt(2/pi) (g + 0.044715 g^3))), in float.  Every
// kernel that gates this way calls this, so that they agree to the bit.
__device__ __forceinline__ float gelu_tanh_mul(float g, float u) {
  const float inner = 0.7978845608028654f * fmaf(0.044715f * g * g, g, g);
  return 0.5f * g * (1.f + tanhf(inner)) * u;
}

// The gate of a gated unit with bounded branches: g = min(g, limit), u = clamp(u, -limit, limit) for limit > 0;
// act 0: g * sigmoid(alpha g) * (u + shift); act 1: gelu_tanh(g) * (u + shift).
#define ERB_GLU_SIGMOID 0
#define ERB_GLU_GELU_TANH 1
__device__ __forceinline__ float glu_gate(float g, float u, int act, float limit, float alpha, float shift) {
  if (limit > 0.f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
  }
  if (act == ERB_GLU_GELU_TANH) return gelu_tanh_mul(g, u + shift);
#if ERB_ELEM == 1
  return __fdividef(g, 1.f + __expf(-alpha * g)) * (u + shift);
#else
  return g / (1.f + expf(-alpha * g)) * (u + shift);
#endif
}

// A barrier among `count` threads of a block (a multiple of 32).
__device__ __forceinline__ void named_barrier(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Two floats that one instruction multiplies and adds (both rounded as fmaf rounds one).
struct Two {
  unsigned long long v;
  __device__ __forceinline__ Two() {}
  __device__ __forceinline__ Two(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
  __device__ __forceinline__ explicit Two(float a) : Two(a, a) {}
  __device__ __forceinline__ void get(float& a, float& b) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
};
__device__ __forceinline__ Two operator*(Two a, Two b) {
  Two d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ Two operator+(Two a, Two b) {
  Two d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) {
  Two d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}

// v * sigmoid(v) of two values in float, without a division's and expf's side branches: 2^(-v log2 e) with the rounding of the product carried along,
// and a reciprocal refined once.  As near to v * sigmoid(v) as v / (1 + expf(-v)) is (tests/test_silu_rows.py), in 11 instructions a value
// instead of 25; infinities and NaN as there.
__device__ __forceinline__ Two silu_two(Two v) {
  const Two z = v * Two(-1.f), hi = z * Two(1.44269502f), lo = fma2(z, Two(1.92596299e-8f), fma2(z, Two(1.44269502f), hi * Two(-1.f)));
  float h0, h1, l0, l1, e0, e1;
  hi.get(h0, h1);
  lo.get(l0, l1);
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(h0));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(h1));
  // (the carried rounding is no number where v is infinite, and nothing where 2^hi is none)
  l0 = fabsf(h0) < 128.f ? l0 : 0.f;
  l1 = fabsf(h1) < 128.f ? l1 : 0.f;
  // a quarter of 1 + e: its reciprocal is then a normal number wherever e is finite; where e is infinite the reciprocal is zero
  const Two e(e0, e1), d = fma2(fma2(e * Two(0.693147181f), Two(l0, l1), e), Two(0.25f), Two(0.25f));
  float d0, d1, y0, y1;
  d.get(d0, d1);
  d0 = fminf(d0, 3.402823466e38f);
  d1 = fminf(d1, 3.402823466e38f);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(d0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(d1));
  const Two y(y0, y1), r = fma2(Two(-d0, -d1), y, Two(1.f));
  return v * Two(0.25f) * fma2(y, r, y);
}

// The same of one value: the same operations, the same bits.
__device__ __forceinline__ float silu_one(float v) {
  const float z = -v, hi = __fmul_rn(z, 1.44269502f), low = __fmaf_rn(z, 1.92596299e-8f, __fmaf_rn(z, 1.44269502f, -hi));
  float e, y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(hi));
  const float l = fabsf(hi) < 128.f ? low : 0.f;
  const float d = fminf(__fmaf_rn(__fmaf_rn(__fmul_rn(e, 0.693147181f), l, e), 0.25f, 0.25f), 3.402823466e38f);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return __fmul_rn(__fmul_rn(v, 0.25f), __fmaf_rn(y, __fmaf_rn(-d, y, 1.f), y));
}

// The nth request (from 0) with more than one token, or -1; the whole warp asks.
__device__ __forceinline__ int nth_portion(const int* __restrict__ seq_starts, int n_seqs, int nth) {
  const int lane = threadIdx.x & 31;
  for (int s0 = 0; s0 < n_seqs; s0 += 32) {
    const int s = s0 + lane;
    unsigned more = __ballot_sync(0xffffffffu, s < n_seqs && seq_starts[min(s, n_seqs - 1) + 1] - seq_starts[min(s, n_seqs - 1)] > 1);
    const int here = __popc(more);
    if (nth < here) {
      for (; nth > 0; --nth) more &= more - 1;
      return s0 + __ffs(more) - 1;
    }
    nth -= here;
  }
  return -1;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over the block in a fixed order (warp trees, then the first warp over the warp sums);
// every thread gets the result.  `scratch` holds 32 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? scratch[lane] : 0.f;
  t = warp_sum(t);
  return t;
}
__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? scratch[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

// One rotary pair (x[j], x[j + half]) turned by the angle whose cosine and sine are given.  Written
// with explicit roundings so that every kernel that rotates gives the same bits.
__device__ __forceinline__ void rotate_pair(float a, float b, float cs, float sn, float& lo, float& hi) {
  lo = __fmaf_rn(a, cs, -__fmul_rn(b, sn));
  hi = __fmaf_rn(b, cs, __fmul_rn(a, sn));
}

// The first key a query at position `pos` sees.  `window` > 0: the last `window` keys; `window` < 0: the keys of the
// query's own chunk, chunks being runs of -window positions counted from position 0 of the sequence; 0: every key.
__host__ __device__ __forceinline__ int first_visible_key(int pos, int window) {
  if (window > 0) return pos - window + 1 > 0 ? pos - window + 1 : 0;
  if (window < 0) return pos - pos % (-window);
  return 0;
}

// Chained launches.  Kernels that run back to back in the decode step are launched with
// programmatic stream serialization: the next kernel's blocks may be scheduled while the previous
// kernel drains, which hides the launch latency between the many short kernels of a step.  Every
// such kernel calls chain_wait() before it touches memory, which blocks until the previous kernel
// has completed and its writes are visible; so the data flow is that of ordinary stream order.
// EDGERAG_B200_NO_CHAIN=1 in the environment turns the attribute off.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

inline bool chain_enabled() {
  static const bool on = [] {
    const char* v = getenv("EDGERAG_B200_NO_CHAIN");
    return !(v && v[0] == '1');
  }();
  return on;
}

template <typename... KArgs, typename... Args>
inline void launch_chained(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                           Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chain_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);   // errors surface in check_launch()
}

}  // namespace erb

#define ERB_EXPORT extern "C" __attribute__((visibility("default")))

// Each library exports its own copy under a library-specific name via this macro.
#define ERB_DEFINE_LAST_ERROR(name) \
  ERB_EXPORT const char* name() { return erb::error_buffer(); }
