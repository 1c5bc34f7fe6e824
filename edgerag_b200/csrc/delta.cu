// The gated delta rule over ragged batches, with every request's state kept in a slot between steps.
//
// Per token and head h (queries and keys of head h / (H / G); d entries each, values dv entries):
//   q, k: unit vectors, x / sqrt(sum(x^2) + 1e-6), q also times d^-1/2         (from the convolved, activated rows)
//   beta = sigmoid(b_h),   g = exp(-exp(A_log_h) * softplus(a_h + dt_bias_h))    (b, a: columns of the input product)
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q               S: d x dv, float, one per request and head
// so the read-out sees the token's own write.  Column p of S depends on the other columns through nothing but k, q, g
// and beta, which gives the kernel its shape: a thread owns up to 16 entries of one column, the threads of a column are
// neighbouring lanes, and per token the two dot products S^T k and S^T q are finished with lane shuffles:
//   a = (S_old^T k)_p,  c = (S_old^T q)_p,   u = beta (v_p - g a),   S_new = g S_old + k u,   o_p = g c + u (k . q).
// Everything here is float whatever the element type T of the rows.  The state is stored transposed, [dv][d], so
// that the lanes of a column read neighbouring addresses.  (The walk issues about 100 instructions a token and warp; a
// first form that indexed its rows with a run-time stride issued 430 and took four times as long.)
//
// Two kernels.  `prepare` is parallel over the tokens and leaves, as floats in a scratch, what the walk needs of a token:
// per key head the unit query (scaled) and the unit key, per head (beta, g, k . q), and the value.  `scan` walks a
// request's tokens; a block stages 16 tokens at a time in shared memory with asynchronous copies, the next 16 on their
// way while these are walked.
//
// A request's tokens of one step are neighbours in the batch (rows seq_starts[s] .. seq_starts[s+1]), its slot is
// state_slots[s].  Walked, every (request, head, column) is one thread group's, token after token, and the arithmetic of a
// token does not depend on how the sequence was cut into steps or on what else the step holds.
//
// Portions of prompts (bfloat16 rows, keys of 64 or 128, values of a multiple of 16) are taken 64 tokens at a time, as products
// of matrices, where chunks_pay says so: see delta_chunk_kernel.  The two forms differ by rounding, and which of them a portion
// gets depends on the step; a caller for whom that matters gives `longest` as 1.
#include <limits.h>
#include <math.h>

#include "common.cuh"
#if ERB_ELEM == 1
#include "mma_split.cuh"
#include "tc_common.cuh"
#endif

using namespace erb;

ERB_DEFINE_LAST_ERROR(erb_last_error)

namespace {

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

__device__ __forceinline__ void copy16_async(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int kDeltaChunk = 16;    // tokens staged in shared memory at a time
constexpr int kDeltaRows = 16;     // entries of a column that a thread holds at most
constexpr int kPrepWarps = 4;

__host__ __device__ __forceinline__ int pad4(int v) { return (v + 3) & ~3; }

// The scratch of one step: qk [tokens][G][2][pad4(d)], then sc [tokens][H][4] = (beta, g, k . q, 0), then
// vf [tokens][H][pad4(dv)], all float.
struct DeltaScratch {
  float* qk;
  float* sc;
  float* vf;
};
__host__ __device__ inline size_t delta_scratch_floats(int n_tokens, int H, int G, int d, int dv) {
  return (size_t)n_tokens * ((size_t)G * 2 * pad4(d) + (size_t)H * 4 + (size_t)H * pad4(dv));
}
__host__ __device__ inline DeltaScratch delta_scratch(float* base, int n_tokens, int H, int G, int d, int dv) {
  DeltaScratch s;
  s.qk = base;
  s.sc = s.qk + (size_t)n_tokens * G * 2 * pad4(d);
  s.vf = s.sc + (size_t)n_tokens * H * 4;
  return s;
}

// One warp: a token's unit query (scaled) and unit key, dp entries each (zeros behind the first d).  Returns k . q.
template <typename T>
__device__ __forceinline__ float unit_rows(const T* __restrict__ qs, const T* __restrict__ ks, int d, int dp, float q_scale, int lane, float* qd,
                                           float* kd) {
  float sk = 0.f, sq = 0.f;
  for (int n = lane; n < d; n += 32) {
    const float kv = Elem<T>::load(ks + n), qv = Elem<T>::load(qs + n);
    sk = fmaf(kv, kv, sk);
    sq = fmaf(qv, qv, sq);
  }
  // (the roots, the decay and the write strength once per token in double, rounded once: their errors would otherwise
  //  compound along the recurrence)
  const float rk = (float)(1.0 / sqrt((double)warp_sum(sk) + 1e-6));
  const float rq = (float)((double)q_scale / sqrt((double)warp_sum(sq) + 1e-6));
  float kq = 0.f;
  for (int n = lane; n < dp; n += 32) {
    const float kv = n < d ? Elem<T>::load(ks + n) * rk : 0.f, qv = n < d ? Elem<T>::load(qs + n) * rq : 0.f;
    kd[n] = kv;
    qd[n] = qv;
    kq = fmaf(kv, qv, kq);
  }
  return warp_sum(kq);
}

// (beta, g, k . q) of a token's head; `raw`: the token's row of the input product.
template <typename T>
__device__ __forceinline__ float4 head_scalars(const T* __restrict__ raw, int off_b, int off_a, int h, const float* __restrict__ dt_bias,
                                               const float* __restrict__ a_log, float kq) {
  const float beta = (float)(1.0 / (1.0 + exp(-(double)Elem<T>::load(raw + off_b + h))));
  const double z = (double)(Elem<T>::load(raw + off_a + h) + dt_bias[h]);
  const float g = (float)exp(-exp((double)a_log[h]) * (z > 30.0 ? z : log1p(exp(z))));
  return make_float4(beta, g, kq, 0.f);
}

// One warp per (token, key head): the unit vectors, then the scalars and values of the heads that use this key head.
template <typename T>
__global__ void __launch_bounds__(kPrepWarps * 32)
delta_prepare_kernel(const T* __restrict__ qkv, int channels, const T* __restrict__ proj, int ld, int off_b, int off_a,
                     const float* __restrict__ dt_bias, const float* __restrict__ a_log, DeltaScratch out, int n_items, int H,
                     int G, int d, int dv, float q_scale, const int* __restrict__ singles) {
  chain_wait();
  const int item = blockIdx.x * kPrepWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= n_items) return;
  // `at`: the token's place in the scratch.  With `singles` (the step's seq_starts) an item is a request, and only requests of
  // one token are prepared, each at its own number.
  const int at = item / G, kh = item % G;
  if (singles && singles[at + 1] - singles[at] != 1) return;
  const int t = singles ? singles[at] : at;
  const int dp = pad4(d), dvp = pad4(dv), rep = H / G;
  const T* row = qkv + (size_t)t * channels;
  float* qd = out.qk + ((size_t)at * G + kh) * 2 * dp;
  const float kq = unit_rows(row + kh * d, row + G * d + kh * d, d, dp, q_scale, lane, qd, qd + dp);
  const T* raw = proj + (size_t)t * ld;
  for (int r = 0; r < rep; ++r) {
    const int h = kh * rep + r;
    if (lane == 0) *reinterpret_cast<float4*>(out.sc + ((size_t)at * H + h) * 4) = head_scalars(raw, off_b, off_a, h, dt_bias, a_log, kq);
    const T* vs = row + 2 * G * d + h * dv;
    float* vd = out.vf + ((size_t)at * H + h) * dvp;
    for (int n = lane; n < dvp; n += 32) vd[n] = n < dv ? Elem<T>::load(vs + n) : 0.f;
  }
}

// The walk along one request's tokens, for PB columns of a head from p0 on.  Thread (l, p) holds 16 rows of column p, four runs of
// four neighbours: rows 4 (l + L j) .. + 3 for j = 0 .. 3, so that the lanes of a column read neighbouring 16-byte pieces of a
// key.  PB is a multiple of 4.  Shared memory: two stages of [chunk][2][16 L] + [chunk][PB] + [chunk][4] floats; a staged
// query or key has room for 16 L entries, the ones past pad4(d) zeroed once, so that the walk reads without a test.
// `stage(c0, nc, qk_s, v_s, sc_s)` brings nc tokens from c0 on; it may copy asynchronously, one group of copies at a time.  All threads
// of the block come here; with SPARE there may be more than the L * PB that walk.
template <int L, bool SPARE, typename Stage>
__device__ __forceinline__ void walk_tokens(float* smem, const Stage& stage, float* __restrict__ state, const int* __restrict__ seq_starts,
                                            const int* __restrict__ state_slots, float* __restrict__ out, int H, int d, int dv, int PB, int h, int seq,
                                            int p0) {
  const int dp = pad4(d);
  constexpr int RS = 16 * L;                                   // floats of a staged query or key
  const int stage_floats = kDeltaChunk * (2 * RS + PB + 4);
  const bool walks = !SPARE || (int)threadIdx.x < L * PB;
  const int l = threadIdx.x % L, p = threadIdx.x / L;
  const int col = p0 + p;
  const bool live = walks && col < dv;
  const int start = seq_starts[seq], n_tok = seq_starts[seq + 1] - start;
  float* s_glob = state + (((size_t)state_slots[seq] * H + h) * dv + (live ? col : 0)) * d;
  int row_of[4];                                               // first row of each run
#pragma unroll
  for (int j = 0; j < 4; ++j) row_of[j] = 4 * (l + L * j);
  if (dp < RS) {                                               // the tails that no copy writes
    for (int idx = threadIdx.x; idx < 2 * kDeltaChunk * 2 * (RS - dp); idx += blockDim.x) {
      const int row = idx / (RS - dp), e = idx % (RS - dp);   // row: (stage, token, q or k)
      smem[(row / (2 * kDeltaChunk)) * stage_floats + (row % (2 * kDeltaChunk)) * RS + dp + e] = 0.f;
    }
  }
  float S[kDeltaRows];
#pragma unroll
  for (int i = 0; i < kDeltaRows; ++i) {
    const int n = row_of[i / 4] + (i & 3);
    S[i] = (live && n < d) ? s_glob[n] : 0.f;
  }
  auto bring = [&](int c0, int buf) {
    float* qk_s = smem + buf * stage_floats;
    float* v_s = qk_s + kDeltaChunk * 2 * RS;
    stage(c0, min(kDeltaChunk, n_tok - c0), qk_s, v_s, v_s + kDeltaChunk * PB);
    copies_commit();
  };
  if (n_tok > 0) bring(0, 0);
  float* out_p = out + (size_t)start * H * dv + h * dv + col;
  for (int c0 = 0, buf = 0; c0 < n_tok; c0 += kDeltaChunk, buf ^= 1) {
    const int nc = min(kDeltaChunk, n_tok - c0);
    if (c0 + kDeltaChunk < n_tok) {
      bring(c0 + kDeltaChunk, buf ^ 1);                        // (that stage was read two rounds ago: the barrier below has passed)
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
    const float* qk_s = smem + buf * stage_floats;
    const float* v_s = qk_s + kDeltaChunk * 2 * RS;
    const float* sc_s = v_s + kDeltaChunk * PB;
    if (walks) {
#pragma unroll 2
      for (int c = 0; c < nc; ++c) {
        const float* qc = qk_s + c * 2 * RS;
        const float* kc = qc + RS;
        float4 kv[4], qv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          kv[j] = *reinterpret_cast<const float4*>(kc + row_of[j]);
          qv[j] = *reinterpret_cast<const float4*>(qc + row_of[j]);
        }
        float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          a0 = fmaf(S[4 * j], kv[j].x, a0); a0 = fmaf(S[4 * j + 1], kv[j].y, a0);
          a0 = fmaf(S[4 * j + 2], kv[j].z, a0); a0 = fmaf(S[4 * j + 3], kv[j].w, a0);
          b0 = fmaf(S[4 * j], qv[j].x, b0); b0 = fmaf(S[4 * j + 1], qv[j].y, b0);
          b0 = fmaf(S[4 * j + 2], qv[j].z, b0); b0 = fmaf(S[4 * j + 3], qv[j].w, b0);
          a1 = fmaf(S[4 * j + 4], kv[j + 1].x, a1); a1 = fmaf(S[4 * j + 5], kv[j + 1].y, a1);
          a1 = fmaf(S[4 * j + 6], kv[j + 1].z, a1); a1 = fmaf(S[4 * j + 7], kv[j + 1].w, a1);
          b1 = fmaf(S[4 * j + 4], qv[j + 1].x, b1); b1 = fmaf(S[4 * j + 5], qv[j + 1].y, b1);
          b1 = fmaf(S[4 * j + 6], qv[j + 1].z, b1); b1 = fmaf(S[4 * j + 7], qv[j + 1].w, b1);
        }
        float a = a0 + a1, b = b0 + b1;
#pragma unroll
        for (int o = 1; o < L; o <<= 1) {                // the lanes of a column: a butterfly, the same sum on each
          a += __shfl_xor_sync(0xffffffffu, a, o);
          b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        const float4 sc = *reinterpret_cast<const float4*>(sc_s + 4 * c);     // beta, g, k . q
        const float g = sc.y;
        const float u = sc.x * (v_s[c * PB + p] - g * a);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          S[4 * j] = fmaf(g, S[4 * j], kv[j].x * u);
          S[4 * j + 1] = fmaf(g, S[4 * j + 1], kv[j].y * u);
          S[4 * j + 2] = fmaf(g, S[4 * j + 2], kv[j].z * u);
          S[4 * j + 3] = fmaf(g, S[4 * j + 3], kv[j].w * u);
        }
        if (l == 0 && live) out_p[(size_t)(c0 + c) * H * dv] = fmaf(g, b, u * sc.z);
      }
    }
    __syncthreads();                                   // (the stage is free for the copies of the round after next)
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < kDeltaRows; ++i) {
      const int n = row_of[i / 4] + (i & 3);
      if (n < d) s_glob[n] = S[i];
    }
  }
}

// grid (H, requests, column blocks), block L * PB threads: what `prepare` left of the tokens, walked.
template <int L>
__global__ void __launch_bounds__(512)
delta_scan_kernel(DeltaScratch in, float* __restrict__ state, const int* __restrict__ seq_starts,
                  const int* __restrict__ state_slots, float* __restrict__ out, int H, int G, int d, int dv, int PB, bool singles) {
  chain_wait();
  if (singles && seq_starts[blockIdx.y + 1] - seq_starts[blockIdx.y] != 1) return;       // (the chunk kernel's)
  extern __shared__ __align__(16) float smem[];
  const int dp = pad4(d), dvp = pad4(dv), h = blockIdx.x, kh = h / (H / G), seq = blockIdx.y, p0 = blockIdx.z * PB;
  constexpr int RS = 16 * L;
  const int first = singles ? seq : seq_starts[seq];           // place in the scratch
  const int qk4 = 2 * dp / 4, v4 = PB / 4;                     // 16-byte pieces of a token's rows
  const int pb_live = min(PB, dvp - p0);                       // columns of this block that the scratch holds
  auto stage = [&](int c0, int nc, float* qk_s, float* v_s, float* sc_s) {
    for (int idx = threadIdx.x; idx < nc * qk4; idx += blockDim.x) {
      const int c = idx / qk4, j = idx % qk4;                  // piece j of the token's [q | k]: to row 2 c or 2 c + 1
      const int which = 4 * j >= dp, e = 4 * j - which * dp;
      copy16_async(qk_s + (2 * c + which) * RS + e, in.qk + ((size_t)(first + c0 + c) * G + kh) * 2 * dp + 4 * j);
    }
    for (int idx = threadIdx.x; idx < nc * v4; idx += blockDim.x) {
      const int c = idx / v4, j = idx % v4;
      if (4 * j < pb_live) copy16_async(v_s + c * PB + 4 * j, in.vf + ((size_t)(first + c0 + c) * H + h) * dvp + p0 + 4 * j);
    }
    for (int c = threadIdx.x; c < nc; c += blockDim.x)
      copy16_async(sc_s + 4 * c, in.sc + ((size_t)(first + c0 + c) * H + h) * 4);
  };
  walk_tokens<L, false>(smem, stage, state, seq_starts, state_slots, out, H, d, dv, PB, h, seq, p0);
}

// One warp per (token, head): out = o / sqrt(mean(o^2) + eps) * weight[entry of the head] * silu(gate), o float.
constexpr int kNormWarps = 4;
template <typename T>
__global__ void __launch_bounds__(kNormWarps * 32)
head_norm_gate_kernel(const float* __restrict__ o, const T* __restrict__ gate, int gate_ld, const float* __restrict__ weight,
                      T* __restrict__ out, int n_items, int H, int dv, float eps) {
  chain_wait();
  const int item = blockIdx.x * kNormWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= n_items) return;
  const int t = item / H, h = item % H;
  const float* src = o + ((size_t)t * H + h) * dv;
  float ss = 0.f;
  for (int i = lane; i < dv; i += 32) ss = fmaf(src[i], src[i], ss);
  const float rs = rsqrtf(warp_sum(ss) / (float)dv + eps);
  const T* gt = gate + (size_t)t * gate_ld + h * dv;
  T* dst = out + ((size_t)t * H + h) * dv;
  for (int i = lane; i < dv; i += 32)
    Elem<T>::store(dst + i, src[i] * rs * weight[i] * silu_f(Elem<T>::load(gt + i)));
}

// The same for heads of at most 512 values in aligned runs of four: a lane reads four neighbours at a time and keeps them for the
// store.  2,048 tokens of 16 heads of 128: 11.9 us by the kernel above, 9.7 us; 8 tokens 2.95 us and 2.1 us.
template <typename T, int V>
__global__ void __launch_bounds__(kNormWarps * 32)
head_norm_gate_vec_kernel(const float* __restrict__ o, const T* __restrict__ gate, int gate_ld, const float* __restrict__ weight,
                          T* __restrict__ out, int n_items, int H, int dv, float eps) {
  chain_wait();
  const int item = blockIdx.x * kNormWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= n_items) return;
  const int t = item / H, h = item % H;
  const float* src = o + (size_t)item * dv;
  const T* gt = gate + (size_t)t * gate_ld + h * dv;
  float v[V][4], z[V][4], ss = 0.f;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int e = 4 * lane + 128 * j;
    if (e < dv) {
      load4(src + e, v[j]);
      Pack4<T>::load(gt + e, z[j]);
#pragma unroll
      for (int i = 0; i < 4; ++i) ss = fmaf(v[j][i], v[j][i], ss);
    }
  }
  const float rs = rsqrtf(warp_sum(ss) / (float)dv + eps);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int e = 4 * lane + 128 * j;
    if (e < dv) {
      float w[4];
      load4(weight + e, w);
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = v[j][i] * rs * w[i] * silu_f(z[j][i]);
      Pack4<T>::store(out + (size_t)item * dv + e, w);
    }
  }
}

#if ERB_ELEM == 1
// ---------------------------------------------------------------------------------------------
// 64 tokens at a time.  With c_t the sum of the logarithms of the chunk's decays up to and with token t, S the state before the
// chunk and u_t the token's write (u = beta (v - S^T k) with the state of its time),
//     u_t + beta_t sum_{s < t} exp(c_t - c_s) (k_t . k_s) u_s  =  beta_t (v_t - exp(c_t) S^T k_t)
//     o_t = exp(c_t) S^T q_t + sum_{s <= t} exp(c_t - c_s) (q_t . k_s) u_s
//     S  <- exp(c_64) S + sum_s exp(c_64 - c_s) k_s u_s^T
// The first line is a triangular system (I + A) U = R whose matrix does not depend on the state: a first kernel, parallel over
// (chunk, head), makes T = (I + A)^-1 in float and P T, with P the weights of the second line, so that U = T R and P U = (P T) R come from R side by
// side; the second kernel, parallel over (request, head, 16 columns of values), walks the chunks with products of matrices alone.  The raw
// queries and keys are bfloat16 as they are (their lengths are factors of rows and columns); every other operand goes in as three bfloat16
// pieces (mma_split.cuh), so that nothing is rounded to 16 bits.  c is summed in double and kept as two floats.
//
// The product of a chunk's 128 rows of keys and queries with the state is tcgen05's, its sums in TMEM (two, over half of a row's entries each: the unit
// cuts its sums); the triangular ones and the state's are mma.sync.  What bounds it: the three dependent phases of a chunk, 4,500 clocks
// (700 the first product, 1,100 R, 900 U, 1,700 the state), and the 64 KB of operands a block reads of it, which four warps bring that do
// nothing else.  The walk takes 0.46 us a token (2,048 tokens of 16 heads of 128 x 128: 971 us with its preparing); both kernels of the chunks
// 105.7 us (27 of it the first); 115.6 us with all products by mma.sync and o from U, 143.6 us while the warps that make the products also asked
// for the copies, 2,300 of a chunk's 6,200 clocks, and the first kernel made its roots one after the other.  (All products by tcgen05: 104.7 us, and the
// state a twentieth further from float64.)  Error against float64: o 1.6e-7, the state 1.0e-7, not above the walk's.
//
// Every wait for a product is bounded; a thread that gives up raises a block-wide flag, all warps still come to the barriers of the remaining
// chunks, and the block frees its TMEM.  It then records 8000000 in *status and returns, or, where the caller named no status word, walks its
// portion like the block that finds a number that is not finite.
constexpr int kChunk = 64, kChunkCols = 16, kChunkWarps = 16, kCopyWarps = 4, kIssueWarp = 15, kChunkPrepWarps = 8;
constexpr int kPieceElems = kChunk * kChunk;

// What the first kernel leaves of one (chunk, head): P T and T, each as three pieces [64][64] (laid
// out as shared memory has them; tiles of 16 x 16 above the diagonal are not written), per token (beta, exp(c) / |k|, exp(c) / |q|, exp(c_64 - c) / |k|), exp(c_64).
struct ChunkRecord {
  __nv_bfloat16 pt[3][kPieceElems];
  __nv_bfloat16 t[3][kPieceElems];
  float4 sc[kChunk];
  float4 total;
};
static_assert(sizeof(ChunkRecord) == 4 * 12548, "copied 16 bytes at a time; the size that callers give the scratch by");

// where entry (r, c) of such a piece lies: rows of 128 bytes, 16-byte pieces exchanged by the row's number
__device__ __forceinline__ int entry(int r, int c) { return r * kChunk + ((c & ~7) ^ ((r & 7) << 3)) + (c & 7); }

// Chunks before request `seq` (requests of one token have none).
__device__ __forceinline__ int chunks_before(const int* seq_starts, int seq) {
  int n = 0;
  for (int s = threadIdx.x & 31; s < seq; s += 32) {
    const int len = seq_starts[s + 1] - seq_starts[s];
    n += len > 1 ? (len + kChunk - 1) / kChunk : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}

// The products of two operands in three pieces each that matter, sums by their size.
__device__ __forceinline__ void six_products(float (&acc)[3][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
  mma16816(acc[0], a[0], b[0][0], b[0][1]);
  mma16816(acc[1], a[0], b[1][0], b[1][1]);
  mma16816(acc[2], a[0], b[2][0], b[2][1]);
  mma16816(acc[1], a[1], b[0][0], b[0][1]);
  mma16816(acc[2], a[1], b[1][0], b[1][1]);
  mma16816(acc[2], a[2], b[0][0], b[0][1]);
}

template <int D>
struct DeltaPrepSmem {
  __nv_bfloat16 k[kChunk][D + 8], q[kChunk][D + 8];
  float a[kChunk][kChunk + 4];                                 // A, then T in its place
  float x[3][16][17];
  float beta[kChunk], ik[kChunk], iq[kChunk], hi[kChunk], lo[kChunk], grown[kChunk], left[kChunk];
  double sums[2];
  alignas(16) __nv_bfloat16 p[3][kChunk][kChunk + 8];          // P in pieces
  alignas(16) __nv_bfloat16 t[D < 128 ? 3 : 1][kChunk][kChunk + 8];      // T in pieces (keys of 128: in the place of k and q)
};

template <int D>
__global__ void __launch_bounds__(kChunkPrepWarps * 32)
delta_chunk_prepare_kernel(const __nv_bfloat16* __restrict__ qkv, int channels, const __nv_bfloat16* __restrict__ proj, int ld, int off_b,
                           int off_a, const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                           const int* __restrict__ seq_starts, int n_seqs, ChunkRecord* __restrict__ records, int H, int G, float q_scale) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DeltaPrepSmem<D>& sm = *reinterpret_cast<DeltaPrepSmem<D>*>(smem_raw);
  auto &ks = sm.k, &qs = sm.q;
  auto &a_s = sm.a;
  auto &x_s = sm.x;
  auto &beta_s = sm.beta, &ik_s = sm.ik, &iq_s = sm.iq, &hi_s = sm.hi, &lo_s = sm.lo, &grown_s = sm.grown, &left_s = sm.left;
  const int h = blockIdx.x, kh = h / (H / G), warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qr = lane >> 2, qc = lane & 3;
  int seq = -1, c = (int)blockIdx.y, start = 0, n_tok = 0;     // chunk c of request seq
  for (int s = 0; s < n_seqs; ++s) {
    start = seq_starts[s];
    n_tok = seq_starts[s + 1] - start;
    const int chunks = n_tok > 1 ? (n_tok + kChunk - 1) / kChunk : 0;
    if (c < chunks) { seq = s; break; }
    c -= chunks;
  }
  if (seq < 0) return;                                         // (the grid is an upper bound)
  const int c0 = c * kChunk;
  ChunkRecord& rec = records[(size_t)blockIdx.y * H + h];
  for (int idx = threadIdx.x; idx < kChunk * (D / 8); idx += blockDim.x) {
    const int r = idx / (D / 8), e = 8 * (idx % (D / 8));
    const bool real = c0 + r < n_tok;
    const __nv_bfloat16* src = qkv + (size_t)(start + (real ? c0 + r : 0)) * channels + kh * D + e;
    copy16_or_zero(&qs[r][e], src, real);
    copy16_or_zero(&ks[r][e], src + G * D, real);
  }
  copy_commit();
  // Per token, in double and rounded once: warps 0 and 1 the decays, 2 and 3 the write strengths, the others the roots of the lengths, whose
  // sums they make a row at a time and keep in a lane each.  (One warp for decays and strengths and a root after every row: 13,000 clocks of a
  // block's 32,000.)
  float raw = 0.f;
  const int tok = 32 * (warp & 1) + lane;
  if (warp < 4 && c0 + tok < n_tok) raw = __bfloat162float(proj[(size_t)(start + c0 + tok) * ld + (warp < 2 ? off_a : off_b) + h]);
  copy_wait<0>();
  __syncthreads();
  if (warp < 2) {
    double cum = 0.0;
    if (c0 + tok < n_tok) {
      const double z = (double)(raw + dt_bias[h]);
      cum = -exp((double)a_log[h]) * (z > 30.0 ? z : log1p(exp(z)));
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, cum, o);
      if (lane >= o) cum += v;
    }
    if (lane == 31) sm.sums[warp] = cum;
    named_barrier(1, 64);
    const double all = sm.sums[0] + sm.sums[1];
    if (warp == 1) cum += sm.sums[0];
    const double l2 = cum * 1.4426950408889634;
    hi_s[tok] = (float)l2;
    lo_s[tok] = (float)(l2 - (double)(float)l2);
    grown_s[tok] = (float)exp(cum);
    left_s[tok] = (float)exp(all - cum);
    if (tok == kChunk - 1) rec.total = make_float4(grown_s[tok], 0.f, 0.f, 0.f);
  } else if (warp < 4) {
    beta_s[tok] = c0 + tok < n_tok ? (float)(1.0 / (1.0 + exp(-(double)raw))) : 0.f;
  } else {
    constexpr int kRows = kChunk / (kChunkPrepWarps - 4);
    float sum_k = 0.f, sum_q = 0.f;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int r = kRows * (warp - 4) + i;
      float sk = 0.f, sq = 0.f;
#pragma unroll
      for (int e = 0; e < D / 64; ++e) {
        const float2 kv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ks[r][2 * lane + 64 * e]));
        const float2 qv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qs[r][2 * lane + 64 * e]));
        sk = fmaf(kv.x, kv.x, sk); sk = fmaf(kv.y, kv.y, sk);
        sq = fmaf(qv.x, qv.x, sq); sq = fmaf(qv.y, qv.y, sq);
      }
      sk = warp_sum(sk);
      sq = warp_sum(sq);
      if (lane == i) { sum_k = sk; sum_q = sq; }
    }
    if (lane < kRows) {
      ik_s[kRows * (warp - 4) + lane] = (float)(1.0 / sqrt((double)sum_k + 1e-6));
      iq_s[kRows * (warp - 4) + lane] = (float)((double)q_scale / sqrt((double)sum_q + 1e-6));
    }
  }
  __syncthreads();
  if (threadIdx.x < kChunk) {
    const int r = threadIdx.x;
    rec.sc[r] = make_float4(beta_s[r], grown_s[r] * ik_s[r], grown_s[r] * iq_s[r], left_s[r] * ik_s[r]);
  }
  // the tiles on and below the diagonal: 10 of k . k, 10 of q . k
  for (int item = warp; item < 20; item += kChunkPrepWarps) {
    const bool is_q = item >= 10;
    const int tile = is_q ? item - 10 : item, tr = tile < 1 ? 0 : tile < 3 ? 1 : tile < 6 ? 2 : 3;
    const int row = 16 * tr, col = 16 * (tile - tr * (tr + 1) / 2);
    float acc[2][2][4] = {};
#pragma unroll
    for (int k = 0; k < D / 16; ++k) {
      uint32_t a[4], b[4];
      ldmatrix4(a, is_q ? &qs[row + (lane & 15)][16 * k + 8 * (lane >> 4)] : &ks[row + (lane & 15)][16 * k + 8 * (lane >> 4)]);
      ldmatrix4(b, &ks[col + (lane & 7) + 8 * (lane >> 4)][16 * k + 8 * ((lane >> 3) & 1)]);
      mma16816(acc[k & 1][0], a, b[0], b[1]);
      mma16816(acc[k & 1][1], a, b[2], b[3]);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = row + qr + 8 * j, s = col + 8 * nt + 2 * qc;
        float v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float decay = exp2f((hi_s[r] - hi_s[s + i]) + (lo_s[r] - lo_s[s + i]));
          const float dot = (acc[0][nt][2 * j + i] + acc[1][nt][2 * j + i]) * ik_s[s + i];
          v[i] = is_q ? (s + i <= r ? dot * iq_s[r] * decay : 0.f) : (s + i < r ? dot * ik_s[r] * decay * beta_s[r] : 0.f);
        }
        if (is_q) {
          uint32_t piece[3];
          split_pair(v[0], v[1], piece);
#pragma unroll
          for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(&sm.p[k][r][s]) = piece[k];
        } else {
          a_s[r][s] = v[0];
          a_s[r][s + 1] = v[1];
        }
      }
  }
  __syncthreads();
  // T = (I + A)^-1 in place of A, by blocks of 16: the diagonal ones column by column, then the others by rising distance from
  // the diagonal, T_ij = -T_ii sum_k A_ik T_kj (k from j to i - 1).  The tiles of A at distances 1 and 2 are used again after T has
  // taken their places, so each thread keeps its rows of them in registers; only (3, 0) is read where it was.  X holds a distance's sums.
  float tcol[16];
  if (warp < 4 && lane < 16) {
    const int b = 16 * warp;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float v = i == lane ? 1.f : 0.f;
#pragma unroll
      for (int k = 0; k < i; ++k) v = fmaf(-a_s[b + i][b + k], tcol[k], v);
      tcol[i] = v;
    }
  }
  __syncthreads();
  if (warp < 4 && lane < 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) a_s[16 * warp + i][16 * warp + lane] = tcol[i];
  }
  __syncthreads();
  {
    const int er = threadIdx.x >> 4, ec = threadIdx.x & 15;    // a thread's entry of a tile
    float a_keep[3][16];                                       // this thread's rows of A at distance 1 (tiles (1,0), (2,1), (3,2)): row er
    float a_keep2[2][16];                                      // and at distance 2 (tiles (2,0), (3,1))
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int k = 0; k < 16; ++k) a_keep[b][k] = a_s[16 * (b + 1) + er][16 * b + k];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int k = 0; k < 16; ++k) a_keep2[b][k] = a_s[16 * (b + 2) + er][16 * b + k];
#pragma unroll
    for (int dist = 1; dist < 4; ++dist) {
      __syncthreads();
#pragma unroll
      for (int b = 0; b < 4 - dist; ++b) {                     // tile (b + dist, b)
        const int i = b + dist;
        float x = 0.f;
#pragma unroll
        for (int kb = b; kb < i; ++kb) {                       // A tile (i, kb), at distance i - kb
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const float av = i - kb == 1 ? a_keep[kb][k] : i - kb == 2 ? a_keep2[kb < 2 ? kb : 0][k] : a_s[16 * i + er][16 * kb + k];
            x = fmaf(av, a_s[16 * kb + k][16 * b + ec], x);
          }
        }
        x_s[b][er][ec] = x;
      }
      __syncthreads();
#pragma unroll
      for (int b = 0; b < 4 - dist; ++b) {
        const int i = b + dist;
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) v = fmaf(a_s[16 * i + er][16 * i + k], x_s[b][k][ec], v);
        a_s[16 * i + er][16 * b + ec] = -v;
      }
    }
  }
  __syncthreads();
  static_assert(sizeof(sm.p) <= sizeof(sm.k) + sizeof(sm.q) || D < 128, "T's pieces take the keys' and queries' place");
  __nv_bfloat16 (*t_s)[kChunk][kChunk + 8] = D < 128 ? sm.t : reinterpret_cast<__nv_bfloat16 (*)[kChunk][kChunk + 8]>(&ks[0][0]);
  for (int idx = threadIdx.x; idx < kPieceElems / 4; idx += blockDim.x) {
    const int r = idx / (kChunk / 4), e = 4 * (idx % (kChunk / 4));
    if (e >= 16 * (r / 16 + 1)) continue;
    const float4 v = *reinterpret_cast<const float4*>(&a_s[r][e]);
    uint32_t p01[3], p23[3];
    split_pair(v.x, v.y, p01);
    split_pair(v.z, v.w, p23);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      *reinterpret_cast<uint2*>(&rec.t[k][entry(r, e)]) = make_uint2(p01[k], p23[k]);
      *reinterpret_cast<uint2*>(&t_s[k][r][e]) = make_uint2(p01[k], p23[k]);
    }
  }
  __syncthreads();
  // P T, 16 x 8 at a time on and below the diagonal's tiles, the six products of pieces that matter
  for (int item = warp; item < 20; item += kChunkPrepWarps) {
    const int tile = item >> 1, tr = tile < 1 ? 0 : tile < 3 ? 1 : tile < 6 ? 2 : 3;
    const int row = 16 * tr, first = 16 * (tile - tr * (tr + 1) / 2), col = first + 8 * (item & 1);
    float acc[3][4] = {};
    for (int k = first; k <= row; k += 16) {
      uint32_t a[3][4], b[3][2];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        ldmatrix4(a[i], &sm.p[i][row + (lane & 15)][k + 8 * (lane >> 4)]);
        ldmatrix2t(b[i], &t_s[i][k + (lane & 15)][col]);
      }
      six_products(acc, a, b);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint32_t piece[3];
      split_pair((acc[2][2 * j] + acc[1][2 * j]) + acc[0][2 * j], (acc[2][2 * j + 1] + acc[1][2 * j + 1]) + acc[0][2 * j + 1], piece);
#pragma unroll
      for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(&rec.pt[k][entry(row + qr + 8 * j, col + 2 * qc)]) = piece[k];
    }
  }
}

// grid (H, requests, columns / 16).  Phases of a chunk, a barrier after each:
//   1  S^T k and S^T q, one product of 128 rows; R = beta (v - exp(c) S^T k), exp(c) S^T q
//   2  warps 0-7: U = T R, as the state will take it;  warps 8-15: o = (P T) R + exp(c) S^T q
//   3  the state, in accumulators (a tile of 16 keys x 8 values a warp)
// Four more warps copy the next chunk's operands meanwhile.
//
// The products are causal for finite numbers only: above the diagonal T and the weights are zeros, and 0 * inf is no number; nor are
// the pieces of an infinity, or the differences of c where a decay is exactly zero.  Whatever is not finite makes an o of its own
// token or the last state not finite, so both are looked at (one multiplication an output), and a block that finds one walks its
// portion once more from the state as it was, with the bits of delta_scan_kernel.  (2,048 tokens of 16 heads of 128 x 128, both
// kernels: 142.5 us without the look, 143.7 us with it, before the steps above.)
template <int D>
struct DeltaChunkSmem {
  static constexpr int LdC = kChunkCols + 8;                   // rows 16 bytes longer than a power of two: no bank conflicts
  struct alignas(1024) Stage {
    __nv_bfloat16 kq[D / 64][2 * kChunk][64];                  // the keys' rows, then the queries', 64 entries at a time; 128-byte swizzle
    __nv_bfloat16 v[kChunk][LdC];
    ChunkRecord rec;
  } stage[2];
  // the state before the chunk, a row per key: of 4 columns the three pieces and 4 entries of nothing, then the next 4; 128-byte swizzle
  __nv_bfloat16 s[D][64];
  __nv_bfloat16 r[3][kChunk][LdC];
  __nv_bfloat16 w[3][kChunk][LdC];                             // exp(c_64 - c) / |k| u
  alignas(16) float qs[kChunk][kChunkCols + 4];                // exp(c) / |q| S^T q
  uint64_t bar;                                                // the products with the state are there
  int abort;
  uint32_t tmem;
};
static_assert(sizeof(DeltaChunkSmem<128>::Stage) % 1024 == 0 && offsetof(DeltaChunkSmem<128>, s) % 1024 == 0 && offsetof(DeltaChunkSmem<64>, s) % 1024 == 0 &&
                  offsetof(DeltaChunkSmem<128>, r) % 16 == 0 && offsetof(DeltaChunkSmem<128>, qs) % 16 == 0 && offsetof(DeltaChunkSmem<64>, qs) % 16 == 0 &&
                  offsetof(DeltaChunkSmem<128>, bar) % 8 == 0 && offsetof(DeltaChunkSmem<64>, bar) % 8 == 0 &&
                  offsetof(DeltaChunkSmem<128>::Stage, v) % 16 == 0 && offsetof(DeltaChunkSmem<128>::Stage, rec) % 16 == 0 &&
                  offsetof(DeltaChunkSmem<64>::Stage, rec) % 16 == 0 && sizeof(DeltaChunkSmem<128>) + 1024 <= 232448, "tiles start where their swizzle does");
// entry `col` (under 64) of row `row` in a tile of 128-byte rows with the 128-byte swizzle
__device__ __forceinline__ int swizzled(int row, int col) { return (((col >> 3) ^ (row & 7)) << 3) + (col & 7); }

template <int D>
__global__ void __launch_bounds__((kChunkWarps + kCopyWarps) * 32)
delta_chunk_kernel(const __nv_bfloat16* __restrict__ qkv, int channels, const ChunkRecord* __restrict__ records, float* __restrict__ state,
                   const int* __restrict__ seq_starts, const int* __restrict__ state_slots, float* __restrict__ out, int H, int G, int dv,
                   const __nv_bfloat16* __restrict__ proj, int ld, int off_b, int off_a, const float* __restrict__ dt_bias,
                   const float* __restrict__ a_log, float q_scale, int n_seqs, int* __restrict__ status) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char smem_all[];
  unsigned char* smem_raw = smem_all + ((1024u - (smem_u32(smem_all) & 1023u)) & 1023u);
  typedef DeltaChunkSmem<D> Smem;
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int h = blockIdx.x, p0 = blockIdx.z * kChunkCols, kh = h / (H / G);
  const int seq = (int)gridDim.y == n_seqs ? (int)blockIdx.y : nth_portion(seq_starts, n_seqs, blockIdx.y);
  if (seq < 0) return;
  const int start = seq_starts[seq], n_tok = seq_starts[seq + 1] - start;
  if (n_tok <= 1) return;                                      // (a single token is walked)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qr = lane >> 2, qc = lane & 3;
  const int n_chunks = (n_tok + kChunk - 1) / kChunk;
  const ChunkRecord* rec0 = records + (size_t)chunks_before(seq_starts, seq) * H + h;
  const __nv_bfloat16* rows = qkv + (size_t)start * channels;
  volatile int* abort_flag = &sm.abort;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&sm.bar), 1);
    sm.abort = 0;
    mbar_init_fence();
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(128) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem, 0);
  constexpr int kColHalf = 64;                                 // columns of TMEM: three pieces' sums over the first half of the keys; over the others

  if (warp >= kChunkWarps) {                                   // the copies: a chunk's operands while the one before is worked on
    const int t = threadIdx.x - kChunkWarps * 32;
    constexpr int kThreads = kCopyWarps * 32, kRow = D / 8, kRows = kThreads / kRow;      // 16-byte pieces of a row; rows a round of the threads
    const int r0 = t / kRow, e0 = 8 * (t % kRow);
    int at[3];                                                 // where this thread's pieces of P and T lie: those not above the diagonal's tiles
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      int n = t + kThreads * i, tile = 0;
      while (n >= 32 * (tile + 1)) n -= 32 * ++tile;           // (16 rows of 2 (tile + 1) pieces)
      at[i] = t + kThreads * i < 320 ? entry(16 * tile + n / (2 * (tile + 1)), 8 * (n % (2 * (tile + 1)))) : -1;
    }
    for (int c = 0; c < n_chunks; ++c) {
      typename Smem::Stage& st = sm.stage[c & 1];
      const int left = n_tok - c * kChunk;                     // tokens from this chunk on (rows behind the request's are zeros)
      const ChunkRecord* rec = rec0 + (size_t)c * H;
      const __nv_bfloat16* src = rows + (size_t)(c * kChunk) * channels;
#pragma unroll
      for (int i = 0; i < kChunk / kRows; ++i) {
        const int r = r0 + kRows * i;
        const __nv_bfloat16* row = src + (size_t)(r < left ? r : 0) * channels + kh * D + e0;
        copy16_or_zero(&st.kq[e0 >> 6][kChunk + r][swizzled(r, e0 & 63)], row, r < left);
        copy16_or_zero(&st.kq[e0 >> 6][r][swizzled(r, e0 & 63)], row + G * D, r < left);
      }
      {
        const int r = t >> 1, e = 8 * (t & 1);
        copy16_or_zero(&st.v[r][e], src + (size_t)(r < left ? r : 0) * channels + 2 * G * D + h * dv + p0 + e, r < left);
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (at[i] >= 0)
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            copy16_or_zero(&st.rec.pt[k][at[i]], &rec->pt[k][at[i]], true);
            copy16_or_zero(&st.rec.t[k][at[i]], &rec->t[k][at[i]], true);
          }
      if (t < kChunk) copy16_or_zero(&st.rec.sc[t], &rec->sc[t], true);
      else if (t == kChunk) copy16_or_zero(&st.rec.total, &rec->total, true);
      copy_commit();
      copy_wait<0>();
      fence_async_proxy();
      __syncthreads();                                         // (a chunk's first barrier)
    }
  }
  // the state (stored [values][keys]): warp w holds keys 16 (w mod D/16) .. + 15, values 8 (w div D/16) .. + 7
  constexpr int kStateWarps = D / 8;
  const int s_row = 16 * (warp % (D / 16)), s_col = 8 * (warp / (D / 16));
  float S[4];
  float* s_glob = state + (((size_t)state_slots[seq] * H + h) * dv + p0) * D;
  auto publish = [&]() {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint32_t piece[3];
      split_pair(S[2 * j], S[2 * j + 1], piece);
#pragma unroll
      for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(&sm.s[s_row + qr + 8 * j][swizzled(qr, 4 * ((s_col + 2 * qc) & ~3) + 4 * k + (2 * qc & 3))]) = piece[k];
    }
    fence_async_proxy();
  };
  if (warp < kStateWarps) {
#pragma unroll
    for (int i = 0; i < 4; ++i) S[i] = s_glob[(size_t)(s_col + 2 * qc + (i & 1)) * D + s_row + qr + 8 * (i >> 1)];
    publish();
  }
  const int row = 16 * ((warp & 7) >> 1), col = 8 * (warp & 1);       // a warp's tile of R, U and o
  // 16 x 8 of M X for a lower-triangular M in pieces (swizzled rows) and X in pieces, the six products that matter
  auto triangular = [&](const __nv_bfloat16 (*m)[kPieceElems], const __nv_bfloat16 (*x)[kChunk][Smem::LdC], float* result) {
    float acc[3][4] = {};
    for (int k = 0; k <= row; k += 16) {
      uint32_t a[3][4], b[3][2];
      const int r = row + (lane & 15), e = (k >> 3) + (lane >> 4);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        ldmatrix4(a[i], &m[i][entry(r, 8 * e)]);
        ldmatrix2t(b[i], &x[i][k + (lane & 15)][col]);
      }
      six_products(acc, a, b);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) result[i] = (acc[2][i] + acc[1][i]) + acc[0][i];
  };
  float probe = 0.f;                                           // no number once a result was not finite
  for (int c = 0; c < n_chunks && warp < kChunkWarps; ++c) {
    typename Smem::Stage& st = sm.stage[c & 1];
    __syncthreads();                                           // chunk c's operands and the state's pieces are there
    if (warp == kIssueWarp) {                                  // S^T of keys and queries, rows as they came: the whole warp, one elected lane issues
      constexpr uint32_t kIdesc = mma_idesc(2 * kChunk, 64, true);
      const uint64_t da = make_desc(smem_u32(&st.kq[0][0][0])), db = make_desc(smem_u32(&sm.s[0][0]));
      fence_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          mma_bf16(tmem + (k / (D / 32)) * kColHalf, da + (k >> 2) * (2 * kChunk * 128 >> 4) + 2 * (k & 3), db + k * (16 * 128 >> 4), kIdesc, k % (D / 32) > 0);
        mma_commit(smem_u32(&sm.bar));
      }
      __syncwarp();
    }
    mbar_wait_or_abort(smem_u32(&sm.bar), c & 1, abort_flag);
    __syncwarp();
    fence_after_sync();
    {
      // a thread: row 32 (warp mod 4) + lane, keys' rows first; columns 4 (warp div 4) .. + 3
      const int quad = warp & 3, t = 32 * (quad & 1) + lane, first = 4 * (warp >> 2);
      float sum[4], low[16], high[16];
      tmem_ld16(tmem + ((uint32_t)(32 * quad) << 16) + 4 * first, low);
      tmem_ld16(tmem + ((uint32_t)(32 * quad) << 16) + kColHalf + 4 * first, high);
      tmem_ld_wait();
      fence_before_sync();
#pragma unroll
      for (int i = 0; i < 4; ++i) sum[i] = ((low[8 + i] + high[8 + i]) + (low[4 + i] + high[4 + i])) + (low[i] + high[i]);
      const float4 sc = st.rec.sc[t];
      if (quad < 2) {
        const uint2 in = *reinterpret_cast<const uint2*>(&st.v[t][first]);
        uint32_t p01[3], p23[3];
        split_pair(sc.x * fmaf(-sc.y, sum[0], __uint_as_float(in.x << 16)), sc.x * fmaf(-sc.y, sum[1], __uint_as_float(in.x & 0xffff0000u)), p01);
        split_pair(sc.x * fmaf(-sc.y, sum[2], __uint_as_float(in.y << 16)), sc.x * fmaf(-sc.y, sum[3], __uint_as_float(in.y & 0xffff0000u)), p23);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(&sm.r[k][t][first]) = make_uint2(p01[k], p23[k]);
      } else {
        *reinterpret_cast<float4*>(&sm.qs[t][first]) = make_float4(sc.z * sum[0], sc.z * sum[1], sc.z * sum[2], sc.z * sum[3]);
      }
    }
    named_barrier(1, kChunkWarps * 32);                        // R is there
    if (warp < 8) {
      float u[4];
      triangular(st.rec.t, sm.r, u);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = row + qr + 8 * j;
        const float left = st.rec.sc[r].w;
        uint32_t weighted[3];
        split_pair(left * u[2 * j], left * u[2 * j + 1], weighted);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(&sm.w[k][r][col + 2 * qc]) = weighted[k];
      }
    } else {
      float own[4];
      triangular(st.rec.pt, sm.r, own);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = row + qr + 8 * j;
        if (c * kChunk + r < n_tok) {
          const float2 q = *reinterpret_cast<const float2*>(&sm.qs[r][col + 2 * qc]);
          const float2 o = make_float2(q.x + own[2 * j], q.y + own[2 * j + 1]);
          probe = fmaf(o.x, 0.f, fmaf(o.y, 0.f, probe));
          *reinterpret_cast<float2*>(out + ((size_t)(start + c * kChunk + r) * H + h) * dv + p0 + col + 2 * qc) = o;
        }
      }
    }
    named_barrier(1, kChunkWarps * 32);                        // U is there
    if (warp < kStateWarps) {
      float add[3][4] = {};
#pragma unroll
      for (int k = 0; k < kChunk / 16; ++k) {
        uint32_t kt[4], b[3][2];                               // K^T: 16 keys x 16 tokens
        const int e = s_row + 8 * ((lane >> 3) & 1);
        ldmatrix4t(kt, &st.kq[e >> 6][16 * k + (lane & 7) + 8 * (lane >> 4)][swizzled(lane, e & 63)]);
#pragma unroll
        for (int piece = 0; piece < 3; ++piece) {
          ldmatrix2t(b[piece], &sm.w[piece][16 * k + (lane & 15)][s_col]);
          mma16816(add[piece], kt, b[piece][0], b[piece][1]);
        }
      }
      const float total = st.rec.total.x;
#pragma unroll
      for (int i = 0; i < 4; ++i) S[i] = fmaf(total, S[i], (add[2][i] + add[1][i]) + add[0][i]);
      publish();
    }
  }
  if (warp < kStateWarps) {
#pragma unroll
    for (int i = 0; i < 4; ++i) probe = fmaf(S[i], 0.f, probe);
  }
  const bool odd = __syncthreads_or(!(probe == 0.f)), gave_up = *abort_flag != 0;
  if (gave_up && threadIdx.x == 0 && status) atomicCAS(status, 0, 8000000);
  __syncthreads();
  if (warp == kIssueWarp) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128) : "memory");
  }
  if (gave_up && status) return;
  if (odd || gave_up) {
    static_assert(2 * kDeltaChunk * (2 * D + kChunkCols + 4) * sizeof(float) <= offsetof(Smem, bar) && D / 16 * kChunkCols <= kChunkWarps * 32, "the walk has room");
    auto prepared = [&](int c0, int nc, float* qk_s, float* v_s, float* sc_s) {      // what `prepare` makes of a token, a warp each
      for (int t = warp; t < nc; t += kChunkWarps) {
        const __nv_bfloat16* at = rows + (size_t)(c0 + t) * channels;
        const float kq = unit_rows(at + kh * D, at + G * D + kh * D, D, D, q_scale, lane, qk_s + 2 * t * D, qk_s + (2 * t + 1) * D);
        if (lane == 0)
          *reinterpret_cast<float4*>(sc_s + 4 * t) = head_scalars(proj + (size_t)(start + c0 + t) * ld, off_b, off_a, h, dt_bias, a_log, kq);
        if (lane < kChunkCols) v_s[t * kChunkCols + lane] = __bfloat162float(at[2 * G * D + h * dv + p0 + lane]);
      }
    };
    walk_tokens<D / 16, true>(reinterpret_cast<float*>(smem_raw), prepared, state, seq_starts, state_slots, out, H, D, dv, kChunkCols, h, seq, p0);
    return;
  }
  if (warp < kStateWarps) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s_glob[(size_t)(s_col + 2 * qc + (i & 1)) * D + s_row + qr + 8 * (i >> 1)] = S[i];
  }
}

inline bool chunk_sizes(int d, int dv) { return (d == 64 || d == 128) && dv % kChunkCols == 0; }
inline long long chunk_records(int n_tokens, int n_seqs, int H) { return (long long)(n_tokens / kChunk + n_seqs) * H; }

// Floats that portions in chunks need: the chunks' records, and the walk's scratch for requests of one token.
inline long long chunk_scratch_floats(int n_tokens, int n_seqs, int H, int G, int d, int dv) {
  return chunk_records(n_tokens, n_seqs, H) * (long long)(sizeof(ChunkRecord) / 4) + (long long)delta_scratch_floats(n_seqs, H, G, d, dv);
}

// Whether the chunks are the faster form: both costs in microseconds, fitted to the times of 1 to 64 requests of 16 to 2,048 tokens
// (4 to 16 heads of 64 x 48 and 128 x 128).  The walk is taken for 0.49 us a token of the longest portion (0.46 now) or, when the GPU is full,
// its blocks' tokens and states; the chunks cost two more launches, 2.8 us a chunk of the longest portion or as many rounds of blocks as
// the SMs need, a block an SM, and requests of one token are then walked by themselves.  Of 297 layouts three of 36 and 44 tokens get chunks
// where the walk is faster, by 3.2 us at most.  One request: from 34 tokens on (16 heads of 128 x 128: 28 tokens 18.7 us walked, 17.4 in a chunk;
// 36 21.5 | 17.2; 4 of 64 x 48: 36 14.5 | 15.5); 32 requests of equal length: from about 65.
inline bool chunks_pay(int blocks, int n_tokens, int n_seqs, int longest) {
  if (longest < 34) return false;
  const double extra = (double)n_tokens - n_seqs - (longest - 1);      // tokens beyond one of the other requests
  const double others = fmax(0.0, fmin(extra, n_seqs - 1.0)), singles = n_seqs - 1.0 - others;
  const double own = (longest + 63) / 64, chunks = own + (others > 0.0 ? others + extra / 64.0 : 0.0);
  const double walk = fmax(6.0 + 0.49 * longest, blocks * (0.00086 * n_tokens + 0.0024 * n_seqs));
  const double rounds = ceil(blocks * (1.0 + others) / sm_count());
  return fmax(14.5 + 2.8 * own, 4.0 + rounds * (4.0 + 2.2 * chunks / (1.0 + others))) + 0.003 * blocks * singles < walk;
}
#endif  // ERB_ELEM == 1

}  // namespace

ERB_EXPORT int erb_delta_scan(const void* qkv, int channels, const void* proj, int ld, int off_b, int off_a,
                              const float* dt_bias, const float* a_log, float* state, const int* seq_starts,
                              const int* state_slots, float* out, float* scratch, long long scratch_floats, int n_seqs, int n_tokens,
                              int longest, int portions, int H, int G, int d, int dv, int* status, void* stream) {
  if (n_seqs <= 0 || n_tokens <= 0) return ERB_OK;
  if (H <= 0 || G <= 0 || H % G || d <= 0 || dv <= 0 || d > 32 * kDeltaRows)
    return fail(ERB_ERR_ARG, "delta_scan: bad sizes (%d heads over %d, keys of %d up to %d)", H, G, d, 32 * kDeltaRows);
  if (channels < 2 * G * d + H * dv) return fail(ERB_ERR_ARG, "delta_scan: rows too narrow");
  if (!scratch || ((uintptr_t)scratch & 15)) return fail(ERB_ERR_ARG, "delta_scan: the scratch must be 16-byte aligned");
  if (portions <= 0 || portions > n_seqs) portions = n_seqs;
  bool singles = false;                  // whether the walk is left with the requests of one token
  int walk_tokens = n_tokens;
#if ERB_ELEM == 1
  if (chunk_sizes(d, dv) && n_tokens > n_seqs && chunks_pay(H * (dv / kChunkCols), n_tokens, n_seqs, longest) && channels % 8 == 0 &&
      !(((uintptr_t)qkv | (uintptr_t)scratch) & 15) && !((uintptr_t)out & 7) && n_tokens / kChunk + n_seqs <= 65535 &&
      scratch_floats >= chunk_scratch_floats(n_tokens, n_seqs, H, G, d, dv)) {
    ChunkRecord* records = reinterpret_cast<ChunkRecord*>(scratch);
    auto prep = d == 64 ? delta_chunk_prepare_kernel<64> : delta_chunk_prepare_kernel<128>;
    const size_t prep_bytes = d == 64 ? sizeof(DeltaPrepSmem<64>) : sizeof(DeltaPrepSmem<128>);
    cudaError_t e = cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep_bytes);
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "delta_scan: %s", cudaGetErrorString(e));
    launch_chained(prep, dim3(H, n_tokens / kChunk + portions), dim3(kChunkPrepWarps * 32), prep_bytes, (cudaStream_t)stream, (const elem_t*)qkv,
                   channels, (const elem_t*)proj, ld, off_b, off_a, dt_bias, a_log, seq_starts, n_seqs, records, H, G, 1.f / sqrtf((float)d));
    int rc = check_launch("delta_chunk_prepare");
    if (rc) return rc;
    const size_t bytes = 1024 + (d == 64 ? sizeof(DeltaChunkSmem<64>) : sizeof(DeltaChunkSmem<128>));
    auto kern = d == 64 ? delta_chunk_kernel<64> : delta_chunk_kernel<128>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "delta_scan: %s", cudaGetErrorString(e));
    launch_chained(kern, dim3(H, portions, dv / kChunkCols), dim3((kChunkWarps + kCopyWarps) * 32), bytes, (cudaStream_t)stream, (const elem_t*)qkv,
                   channels, records, state, seq_starts, state_slots, out, H, G, dv, (const elem_t*)proj, ld, off_b, off_a, dt_bias, a_log,
                   1.f / sqrtf((float)d), n_seqs, status);
    if ((rc = check_launch("delta_chunk")) || n_seqs == 1) return rc;
    singles = true;
    walk_tokens = n_seqs;
    scratch += chunk_records(n_tokens, n_seqs, H) * (long long)(sizeof(ChunkRecord) / 4);
  }
#endif
  const DeltaScratch sc = delta_scratch(scratch, walk_tokens, H, G, d, dv);
  const long long items = (long long)walk_tokens * G;
  if (items > 0x7fffffffLL) return fail(ERB_ERR_UNSUPPORTED, "delta_scan: %d tokens of %d key heads", n_tokens, G);
  launch_chained(delta_prepare_kernel<elem_t>, dim3((unsigned)((items + kPrepWarps - 1) / kPrepWarps)), dim3(kPrepWarps * 32), 0,
                 (cudaStream_t)stream, (const elem_t*)qkv, channels, (const elem_t*)proj, ld, off_b, off_a, dt_bias, a_log, sc,
                 (int)items, H, G, d, dv, 1.f / sqrtf((float)d), singles ? seq_starts : nullptr);
  int rc = check_launch("delta_prepare");
  if (rc) return rc;
  int L = 1;
  while (L * kDeltaRows < d) L <<= 1;
  // columns per block: whole warps, up to 256 threads, fewer where that gives the GPU too few blocks; at least 4
  int PB = 256 / L;
  while (PB * L > 32 && PB / 2 >= dv && PB > 4) PB >>= 1;
  while (PB * L > 64 && PB > 4 && (long long)H * n_seqs * ((dv + PB - 1) / PB) < 2LL * sm_count()) PB >>= 1;
  const int cblocks = (dv + PB - 1) / PB;
  const size_t smem = sizeof(float) * 2 * ((size_t)kDeltaChunk * (2 * 16 * L + PB + 4));
#define ERB_DELTA_CASE(LL)                                                                                              \
  case LL: {                                                                                                            \
    auto kern = delta_scan_kernel<LL>;                                                                                  \
    if (smem > 48 * 1024) {                                                                                             \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);               \
      if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "delta_scan: %s", cudaGetErrorString(e));                        \
    }                                                                                                                   \
    launch_chained(kern, dim3(H, n_seqs, cblocks), dim3(LL * PB), smem, (cudaStream_t)stream, sc, state, seq_starts,    \
                   state_slots, out, H, G, d, dv, PB, singles);                                                         \
  } break;
  switch (L) {
    ERB_DELTA_CASE(1)
    ERB_DELTA_CASE(2)
    ERB_DELTA_CASE(4)
    ERB_DELTA_CASE(8)
    ERB_DELTA_CASE(16)
    default:
      ERB_DELTA_CASE(32)
  }
#undef ERB_DELTA_CASE
  return check_launch("delta_scan");
}

ERB_EXPORT int erb_head_norm_gate(const float* o, const void* gate, int gate_ld, const float* weight, void* out, int n_tokens,
                                  int H, int dv, float eps, void* stream) {
  if (n_tokens <= 0) return ERB_OK;
  if (H <= 0 || dv <= 0) return fail(ERB_ERR_ARG, "head_norm_gate: bad sizes");
  const long long items = (long long)n_tokens * H;
  if (items > 0x7fffffffLL) return fail(ERB_ERR_UNSUPPORTED, "head_norm_gate: %d tokens of %d heads", n_tokens, H);
  const uintptr_t elem_bits = 4 * sizeof(elem_t) - 1;
  if (dv % 4 == 0 && dv <= 512 && gate_ld % 4 == 0 && !(((uintptr_t)o | (uintptr_t)weight) & 15) && !(((uintptr_t)gate | (uintptr_t)out) & elem_bits)) {
    auto kern = dv <= 128 ? head_norm_gate_vec_kernel<elem_t, 1> : dv <= 256 ? head_norm_gate_vec_kernel<elem_t, 2> : head_norm_gate_vec_kernel<elem_t, 4>;
    launch_chained(kern, dim3((unsigned)((items + kNormWarps - 1) / kNormWarps)), dim3(kNormWarps * 32), 0, (cudaStream_t)stream, o,
                   (const elem_t*)gate, gate_ld, weight, (elem_t*)out, (int)items, H, dv, eps);
    return check_launch("head_norm_gate");
  }
  launch_chained(head_norm_gate_kernel<elem_t>, dim3((unsigned)((items + kNormWarps - 1) / kNormWarps)), dim3(kNormWarps * 32), 0,
                 (cudaStream_t)stream, o, (const elem_t*)gate, gate_ld, weight, (elem_t*)out, (int)items, H, dv, eps);
  return check_launch("head_norm_gate");
}
