// A selective state-space mixer (the "state-space duality" form with a scalar decay per head) over
// ragged batches, with the state of every request kept in slots between steps.
//
// Per token the input projection gives  z (inner) | x (inner) | B (G*N) | C (G*N) | dt (H);  inner = H * P.
//   1. short causal convolution per channel over x|B|C with bias, then silu; the inputs of the last
//      taps-1 tokens of a request are part of its state, so a portion may start anywhere;
//   2. dt = softplus(dt + dt_bias);   per head h (group g = h / (H / G)):
//        S <- exp(-exp(A_log_h) dt) S + dt B_g x_h^T     (S: N x P, float, one per request and head)
//        y_h = S^T C_g + D_h x_h;
//   3. y * silu(z), unit RMS in equal parts of the row (each by its own mean square), times a weight.
// The decay, dt, the state, y and the norm are float; x, B, C arrive in the element type T.
//
// A request's tokens of one step are neighbours in the batch (rows seq_starts[s] .. seq_starts[s+1]),
// its slot is state_slots[s].  Every (request, head, block of columns) is scanned by exactly one block: token after token, or
// (bfloat16, the sizes of ssm_chunk_kernel) 128 or 64 tokens at a time as products of matrices.
#include <limits.h>
#include <math.h>
#include <stddef.h>

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

// One block per token; threads over channels.  conv_state: [slots][taps-1][channels] float, oldest first.
template <typename T>
__global__ void __launch_bounds__(256)
conv_silu_kernel(const T* __restrict__ proj, int ld, int off, int channels, int taps, const T* __restrict__ weight,
                 const T* __restrict__ bias, const float* __restrict__ conv_state, const int* __restrict__ seq_of_token,
                 const int* __restrict__ seq_starts, const int* __restrict__ state_slots, T* __restrict__ out) {
  chain_wait();
  const int t = blockIdx.x;
  const int seq = seq_of_token[t];
  const int start = seq_starts[seq];
  const int i = t - start;                                    // index of the token inside its portion
  const float* old = conv_state + (size_t)state_slots[seq] * (taps - 1) * channels;
  for (int ch = blockIdx.y * blockDim.x + threadIdx.x; ch < channels; ch += gridDim.y * blockDim.x) {
    float acc = bias ? Elem<T>::load(bias + ch) : 0.f;
    for (int j = 0; j < taps; ++j) {
      const int r = i - (taps - 1 - j);                        // portion index of the input under tap j
      const float v = r >= 0 ? Elem<T>::load(proj + (size_t)(start + r) * ld + off + ch)
                             : old[(size_t)(taps - 1 + r) * channels + ch];
      acc = fmaf(Elem<T>::load(weight + (size_t)ch * taps + j), v, acc);
    }
#if ERB_ELEM == 1
    Elem<T>::store(out + (size_t)t * channels + ch, silu_one(acc));      // (as conv_silu_vec_kernel: the same bits)
#else
    Elem<T>::store(out + (size_t)t * channels + ch, silu_f(acc));
#endif
  }
}

#if ERB_ELEM == 1
// The same for four taps and rows whose channels come in aligned runs of eight (bfloat16 build): a thread owns eight channels
// of TT neighbouring tokens, keeps its weights in registers and reads every input once with 16-byte loads instead of four
// times with 2-byte ones.  The sums are made in the same order: their bits are those of the kernel above, and silu is as near (silu_two).
// 2,048 tokens of 6,144 channels: 70 us by the kernel above, 25.6 us with its arithmetic, 17.5 us with two channels an
// instruction, tokens of one request without looking each one's request up, and this silu, four tokens a thread (two 21.8, eight 19.6 us);
// 64 single tokens 16 us and 3.6 us.
template <int TT>
__global__ void __launch_bounds__(128, TT == 1 ? 7 : 5)         // (one token a thread: 72 registers, so that 1,000 blocks are one wave)
conv_silu_vec_kernel(const __nv_bfloat16* __restrict__ proj, int ld, int off, int channels, const __nv_bfloat16* __restrict__ weight,
                     const __nv_bfloat16* __restrict__ bias, const float* __restrict__ conv_state, const int* __restrict__ seq_of_token,
                     const int* __restrict__ seq_starts, const int* __restrict__ state_slots, __nv_bfloat16* __restrict__ out, int n_tokens) {
  constexpr int TAPS = 4;
  chain_wait();
  const int ch = 8 * (blockIdx.y * blockDim.x + threadIdx.x), t0 = blockIdx.x * TT;
  if (ch >= channels) return;
  const int first = seq_of_token[t0], place = t0 - seq_starts[first];      // the first token's request, and its index there
  uint4 raw[TT + TAPS - 1];                                   // inputs t0 - (TAPS - 1) .. t0 + TT - 1
#pragma unroll
  for (int k = 0; k < TT + TAPS - 1; ++k) {
    const int t = t0 + k - (TAPS - 1);
    raw[k] = make_uint4(0, 0, 0, 0);
    if (t >= 0 && t < n_tokens) raw[k] = *reinterpret_cast<const uint4*>(proj + (size_t)t * ld + off + ch);
  }
  Two w[TAPS][4], b[4];                                       // pairs of channels
  {
    float v[8 * TAPS], u[8] = {};
#pragma unroll
    for (int i = 0; i < TAPS; ++i) load8(weight + (size_t)ch * TAPS + 8 * i, v + 8 * i);     // [channel][tap]
    if (bias) load8(bias + ch, u);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      b[e] = Two(u[2 * e], u[2 * e + 1]);
#pragma unroll
      for (int j = 0; j < TAPS; ++j) w[j][e] = Two(v[2 * e * TAPS + j], v[(2 * e + 1) * TAPS + j]);
    }
  }
  // tokens of one request that have their earlier inputs in this portion need no look at the request
  const bool plain = TT > 1 && place >= TAPS - 1 && seq_of_token[min(t0 + TT, n_tokens) - 1] == first;
#pragma unroll
  for (int k = 0; k < TT; ++k) {
    const int t = t0 + k;
    if (t >= n_tokens) break;
    Two acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = b[e];
    int i = TT > 1 ? TAPS : place, seq = first;
    if (TT > 1 && !plain) {
      seq = seq_of_token[t];
      i = t - seq_starts[seq];
    }
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {
      const int r = i - (TAPS - 1 - j);                        // portion index of the input under tap j
      Two v[4];
      if (r >= 0) {
        const uint32_t u[4] = {raw[k + j].x, raw[k + j].y, raw[k + j].z, raw[k + j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = Two(__uint_as_float(u[e] << 16), __uint_as_float(u[e] & 0xffff0000u));
      } else {
        const float* old = conv_state + ((size_t)state_slots[seq] * (TAPS - 1) + TAPS - 1 + r) * channels + ch;
        float x[8];
        load4(old, x);
        load4(old + 4, x + 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = Two(x[2 * e], x[2 * e + 1]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = fma2(w[j][e], v[e], acc[e]);
    }
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float s0, s1;
      silu_two(acc[e]).get(s0, s1);
      const __nv_bfloat162 p = __floats2bfloat162_rn(s0, s1);
      o[e] = *reinterpret_cast<const uint32_t*>(&p);
    }
    *reinterpret_cast<uint4*>(out + (size_t)t * channels + ch) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

#endif

// One block per request: the last taps-1 inputs of (old state, then the portion) become the state.
template <typename T>
__global__ void __launch_bounds__(256)
conv_state_update_kernel(const T* __restrict__ proj, int ld, int off, int channels, int taps, float* __restrict__ conv_state,
                         const int* __restrict__ seq_starts, const int* __restrict__ state_slots) {
  chain_wait();
  const int seq = blockIdx.x;
  const int start = seq_starts[seq], n = seq_starts[seq + 1] - start;
  const int K = taps - 1;
  float* st = conv_state + (size_t)state_slots[seq] * K * channels;
  for (int ch = blockIdx.y * blockDim.x + threadIdx.x; ch < channels; ch += gridDim.y * blockDim.x) {
    for (int k = 0; k < K; ++k) {                             // rising k: entry k + n is read before it is written
      const int src = k + n;
      st[(size_t)k * channels + ch] = src < K ? st[(size_t)src * channels + ch]
                                              : Elem<T>::load(proj + (size_t)(start + src - K) * ld + off + ch);
    }
  }
}

// Rows [q heads | k heads | v heads] of a fused product made ready for attention by a short causal convolution per channel:
//   u = row + bias,   y_t = sum_j w[j] u_(t - (taps - 1 - j))   (u before the sequence's start: zero; no taps: y = u)
// in float, from the portion's own rows and, before its first token, from the request's record of biased inputs (float
// [slots][taps - 1][channels], oldest first).  q goes to rows of its own, k and v to the token's cache slot (page *
// page_size + offset; negative: not written).  A thread owns four neighbouring channels of one token.  A sequence with one
// token in the step gets its record moved on by the same thread (nobody else reads those channels of that record); the
// records of longer portions are moved on by qkv_conv_state_kernel, after this kernel.
// weight: float [taps][channels].
template <typename T>
__global__ void __launch_bounds__(128)
qkv_conv_kernel(const T* __restrict__ proj, int ld, const float* __restrict__ bias, const float* __restrict__ weight, int taps,
                float* __restrict__ conv_state, const int* __restrict__ seq_of_token, const int* __restrict__ seq_starts,
                const int* __restrict__ state_slots, const int* __restrict__ slots, T* __restrict__ q_out,
                T* __restrict__ k_pages, T* __restrict__ v_pages, int nq, int nkv, int D, int page_size) {
  chain_wait();
  const int t = blockIdx.x, ch = 4 * (blockIdx.y * blockDim.x + threadIdx.x);
  const int qw = nq * D, kw = nkv * D, channels = qw + 2 * kw;
  if (ch >= channels) return;
  float b[4] = {0.f, 0.f, 0.f, 0.f};
  if (bias) load4(bias + ch, b);
  auto input = [&](int row, float* u) {
    Pack4<T>::load(proj + (size_t)row * ld + ch, u);
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] += b[i];
  };
  float y[4], u[4];
  input(t, u);
  if (taps <= 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = u[i];
  } else {
    const int seq = seq_of_token[t], start = seq_starts[seq], n = seq_starts[seq + 1] - start, i0 = t - start;
    float* rec = conv_state ? conv_state + (size_t)state_slots[seq] * (taps - 1) * channels + ch : nullptr;
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = 0.f;
    for (int j = 0; j < taps; ++j) {
      const int r = i0 - (taps - 1 - j);               // index inside the portion of the input under tap j
      float x[4], w[4];
      if (j == taps - 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = u[i];
      } else if (r >= 0) {
        input(start + r, x);
      } else {
        load4(rec + (size_t)(taps - 1 + r) * channels, x);
      }
      load4(weight + (size_t)j * channels + ch, w);
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = fmaf(w[i], x[i], y[i]);
    }
    if (n == 1 && taps > 1) {
      for (int k = 0; k + 1 < taps - 1; ++k)
        *reinterpret_cast<float4*>(rec + (size_t)k * channels) = *reinterpret_cast<const float4*>(rec + (size_t)(k + 1) * channels);
      *reinterpret_cast<float4*>(rec + (size_t)(taps - 2) * channels) = make_float4(u[0], u[1], u[2], u[3]);
    }
  }
  if (ch < qw) {
    Pack4<T>::store(q_out + (size_t)t * qw + ch, y);
    return;
  }
  const int slot = slots ? slots[t] : -1;
  if (slot < 0) return;
  const bool is_k = ch < qw + kw;
  const int c = ch - qw - (is_k ? 0 : kw), head = c / D, e = c % D;
  T* pages = is_k ? k_pages : v_pages;
  Pack4<T>::store(pages + (((size_t)(slot / page_size) * nkv + head) * page_size + slot % page_size) * D + e, y);
}

// The records of the sequences with more than one token in the step: the last taps - 1 of (record, then the biased rows).
template <typename T>
__global__ void __launch_bounds__(128)
qkv_conv_state_kernel(const T* __restrict__ proj, int ld, const float* __restrict__ bias, int taps, float* __restrict__ conv_state,
                      const int* __restrict__ seq_starts, const int* __restrict__ state_slots, int first_seq, int channels) {
  chain_wait();
  const int seq = first_seq + blockIdx.x, ch = 4 * (blockIdx.y * blockDim.x + threadIdx.x);
  const int start = seq_starts[seq], n = seq_starts[seq + 1] - start, K = taps - 1;
  if (n <= 1 || ch >= channels) return;
  float* rec = conv_state + (size_t)state_slots[seq] * K * channels + ch;
  float b[4] = {0.f, 0.f, 0.f, 0.f};
  if (bias) load4(bias + ch, b);
  for (int k = 0; k < K; ++k) {                        // rising k: entry k + n is read before it is written
    const int src = k + n;
    float x[4];
    if (src < K) {
      load4(rec + (size_t)src * channels, x);
    } else {
      Pack4<T>::load(proj + (size_t)(start + src - K) * ld + ch, x);
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] += b[i];
    }
    *reinterpret_cast<float4*>(rec + (size_t)k * channels) = make_float4(x[0], x[1], x[2], x[3]);
  }
}

constexpr int kScanChunk = 16;     // tokens staged in shared memory at a time

// One block per (head, request); thread (l, p): column p of the state, rows l * NL .. l * NL + NL - 1, in
// registers.  A chunk of tokens is staged (B, C, x, dt, decay as floats), scanned without a barrier (every
// thread leaves its partial y per token in shared memory), then the L partial sums of a column are added in order.
template <typename T, int NLMAX>
__global__ void __launch_bounds__(512)
ssm_scan_kernel(const T* __restrict__ xbc, int channels, const T* __restrict__ proj, int ld, int off_dt,
                const float* __restrict__ dt_bias, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                float* __restrict__ state, const int* __restrict__ seq_starts, const int* __restrict__ state_slots,
                float* __restrict__ y, int H, int P, int N, int G, int L, int NL) {
  chain_wait();
  extern __shared__ float smem[];
  float* b_s = smem;                                   // [chunk][N]
  float* c_s = b_s + kScanChunk * N;                   // [chunk][N]
  float* x_s = c_s + kScanChunk * N;                   // [chunk][P]
  float* dt_s = x_s + kScanChunk * P;                  // [chunk]
  float* decay_s = dt_s + kScanChunk;                  // [chunk]
  float* part_s = decay_s + kScanChunk;                // [chunk][L][P]
  const int h = blockIdx.x, seq = blockIdx.y;
  const int g = h / (H / G);
  const int inner = H * P;
  const int p = threadIdx.x % P, l = threadIdx.x / P;
  const int n0 = l * NL;
  const int start = seq_starts[seq], n_tok = seq_starts[seq + 1] - start;
  float* s_glob = state + (((size_t)state_slots[seq] * H + h) * N) * P;
  float S[NLMAX];
#pragma unroll
  for (int i = 0; i < NLMAX; ++i) S[i] = (i < NL && n0 + i < N) ? s_glob[(size_t)(n0 + i) * P + p] : 0.f;
  const float a = -expf(a_log[h]), bias = dt_bias[h], dskip = d_skip[h];
  for (int c0 = 0; c0 < n_tok; c0 += kScanChunk) {
    const int nc = min(kScanChunk, n_tok - c0);
    __syncthreads();                                   // (the chunk before has been read)
    for (int idx = threadIdx.x; idx < nc * N; idx += blockDim.x) {
      const int k = idx / N, n = idx % N;
      const T* row = xbc + (size_t)(start + c0 + k) * channels;
      b_s[idx] = Elem<T>::load(row + inner + g * N + n);
      c_s[idx] = Elem<T>::load(row + inner + G * N + g * N + n);
    }
    for (int idx = threadIdx.x; idx < nc * P; idx += blockDim.x) {
      const int k = idx / P, pp = idx % P;
      x_s[idx] = Elem<T>::load(xbc + (size_t)(start + c0 + k) * channels + h * P + pp);
    }
    for (int k = threadIdx.x; k < nc; k += blockDim.x) {
      const float dt = softplus_f(Elem<T>::load(proj + (size_t)(start + c0 + k) * ld + off_dt + h) + bias);
      dt_s[k] = dt;
      decay_s[k] = expf(a * dt);
    }
    __syncthreads();
    for (int k = 0; k < nc; ++k) {
      const float decay = decay_s[k], dx = dt_s[k] * x_s[k * P + p];
      const float* bk = b_s + k * N + n0;
      const float* ck = c_s + k * N + n0;
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < NLMAX; ++i) {
        if (i < NL && n0 + i < N) {
          S[i] = fmaf(decay, S[i], bk[i] * dx);
          sum = fmaf(S[i], ck[i], sum);
        }
      }
      part_s[(k * L + l) * P + p] = sum;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nc * P; idx += blockDim.x) {
      const int k = idx / P, pp = idx % P;
      float sum = 0.f;
      for (int ll = 0; ll < L; ++ll) sum += part_s[(k * L + ll) * P + pp];
      y[(size_t)(start + c0 + k) * inner + h * P + pp] = sum + dskip * x_s[idx];
    }
  }
#pragma unroll
  for (int i = 0; i < NLMAX; ++i)
    if (i < NL && n0 + i < N) s_glob[(size_t)(n0 + i) * P + p] = S[i];
}

// The same scan for states whose row count is a multiple of NL (8 or 16): a block owns PB (16 or 32) columns of
// one head's state, thread (l, p) rows NL l .. NL l + NL - 1 of column p, so a head gives P / PB blocks of
// N / NL * PB light threads (more warps in flight to hide the dependent steps of a token, and a warp reads B and C
// as 16-byte broadcasts).  Same arithmetic per state entry; the partial sums of a column are added in the order of l.
// All threads of the block come here; with SPARE there may be more than the N / NL * PB that walk.
template <typename T, int NL, bool SPARE>
__device__ __forceinline__ void scan_tokens(float* smem, const T* __restrict__ xbc, int channels, const T* __restrict__ proj, int ld, int off_dt,
                                            const float* __restrict__ dt_bias, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                                            float* __restrict__ state, const int* __restrict__ seq_starts, const int* __restrict__ state_slots,
                                            float* __restrict__ y, int H, int P, int N, int G, int PB, int h, int seq, int p0) {
  const int L = N / NL;
  float* b_s = smem;                                   // [chunk][N]
  float* c_s = b_s + kScanChunk * N;                   // [chunk][N]
  float* x_s = c_s + kScanChunk * N;                   // [chunk][PB]
  float* dt_s = x_s + kScanChunk * PB;                 // [chunk]
  float* decay_s = dt_s + kScanChunk;                  // [chunk]
  float* part_s = decay_s + kScanChunk;                // [chunk][L][PB]
  const int g = h / (H / G);
  const int inner = H * P;
  const bool walks = !SPARE || (int)threadIdx.x < L * PB;
  const int p = threadIdx.x % PB, l = walks ? threadIdx.x / PB : 0;
  const int n0 = l * NL;
  const int start = seq_starts[seq], n_tok = seq_starts[seq + 1] - start;
  float* s_glob = state + (((size_t)state_slots[seq] * H + h) * N + n0) * P + p0 + p;
  float S[NL];
#pragma unroll
  for (int i = 0; i < NL; ++i) S[i] = s_glob[(size_t)i * P];
  const float a = -expf(a_log[h]), bias = dt_bias[h], dskip = d_skip[h];
  for (int c0 = 0; c0 < n_tok; c0 += kScanChunk) {
    const int nc = min(kScanChunk, n_tok - c0);
    __syncthreads();
    for (int idx = threadIdx.x; idx < nc * N; idx += blockDim.x) {
      const int k = idx / N, n = idx % N;
      const T* row = xbc + (size_t)(start + c0 + k) * channels;
      b_s[idx] = Elem<T>::load(row + inner + g * N + n);
      c_s[idx] = Elem<T>::load(row + inner + G * N + g * N + n);
    }
    for (int idx = threadIdx.x; idx < nc * PB; idx += blockDim.x) {
      const int k = idx / PB, pp = idx % PB;
      x_s[idx] = Elem<T>::load(xbc + (size_t)(start + c0 + k) * channels + h * P + p0 + pp);
    }
    for (int k = threadIdx.x; k < nc; k += blockDim.x) {
      const float dt = softplus_f(Elem<T>::load(proj + (size_t)(start + c0 + k) * ld + off_dt + h) + bias);
      dt_s[k] = dt;
      decay_s[k] = expf(a * dt);
    }
    __syncthreads();
    if (walks) {
      for (int k = 0; k < nc; ++k) {
        const float decay = decay_s[k], dx = dt_s[k] * x_s[k * PB + p];
        const float4* bk = reinterpret_cast<const float4*>(b_s + k * N + n0);
        const float4* ck = reinterpret_cast<const float4*>(c_s + k * N + n0);
        float sum = 0.f;
#pragma unroll
        for (int i4 = 0; i4 < NL / 4; ++i4) {
          const float4 b = bk[i4], c = ck[i4];
          S[4 * i4] = fmaf(decay, S[4 * i4], b.x * dx);         sum = fmaf(S[4 * i4], c.x, sum);
          S[4 * i4 + 1] = fmaf(decay, S[4 * i4 + 1], b.y * dx); sum = fmaf(S[4 * i4 + 1], c.y, sum);
          S[4 * i4 + 2] = fmaf(decay, S[4 * i4 + 2], b.z * dx); sum = fmaf(S[4 * i4 + 2], c.z, sum);
          S[4 * i4 + 3] = fmaf(decay, S[4 * i4 + 3], b.w * dx); sum = fmaf(S[4 * i4 + 3], c.w, sum);
        }
        part_s[(k * L + l) * PB + p] = sum;
      }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nc * PB; idx += blockDim.x) {
      const int k = idx / PB, pp = idx % PB;
      float sum = 0.f;
      for (int ll = 0; ll < L; ++ll) sum += part_s[(k * L + ll) * PB + pp];
      y[(size_t)(start + c0 + k) * inner + h * P + p0 + pp] = sum + dskip * x_s[idx];
    }
  }
  if (walks) {
#pragma unroll
    for (int i = 0; i < NL; ++i) s_glob[(size_t)i * P] = S[i];
  }
}
__host__ __device__ constexpr size_t scan_smem(int N, int PB, int L) { return sizeof(float) * ((size_t)kScanChunk * (2 * N + PB + 2 + (size_t)L * PB)); }

template <typename T, int NL>
__global__ void __launch_bounds__(512)
ssm_scan16_kernel(const T* __restrict__ xbc, int channels, const T* __restrict__ proj, int ld, int off_dt,
                  const float* __restrict__ dt_bias, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                  float* __restrict__ state, const int* __restrict__ seq_starts, const int* __restrict__ state_slots,
                  float* __restrict__ y, int H, int P, int N, int G, int PB, int most_tokens) {
  chain_wait();
  extern __shared__ __align__(16) float smem[];
  if (seq_starts[blockIdx.y + 1] - seq_starts[blockIdx.y] > most_tokens) return;      // (longer portions: the chunk kernel's)
  scan_tokens<T, NL, false>(smem, xbc, channels, proj, ld, off_dt, dt_bias, a_log, d_skip, state, seq_starts, state_slots, y, H, P, N, G, PB,
                            blockIdx.x, blockIdx.y, blockIdx.z * PB);
}

#if ERB_ELEM == 1
// The scan of portions of prompts, 128 tokens at a time.  With c_t the sum of the logarithms of the chunk's decays up to and
// with token t, and S the state before the chunk,
//     y_t = exp(c_t) S^T C_t + sum_{s <= t} (C_t . B_s) dt_s exp(c_t - c_s) x_s + D x_t
//     S  <- exp(c_128) S + sum_s B_s (dt_s exp(c_128 - c_s) x_s)^T
// which are products of matrices, here on tcgen05 with their sums in TMEM.  C, B and x are bfloat16 as they are; every operand that is
// not (the weights of the second sum, the state, the weighted x of the third) goes in as three bfloat16 pieces (mma_split.cuh), so
// nothing is rounded to 16 bits.  c is summed in double and kept as two floats, since its differences, not its values, matter.
//
// Block: one (head, request, 32 columns).  Sixteen warps do what is between the products, an issuing warp asks for the products, four warps
// make the steps and decays a chunk ahead and store the outputs of the chunk before, one of their lanes brings the next chunk's rows by TMA
// tensor copies.  Per chunk c:
//   G = C B^T                       as two sums over half of the state's rows each (the unit cuts its sums; one sum of 128 was a third
//                                   further from float64), issued while the chunk before is finished
//   Y0 = C S while the weights' pieces are made from G, as the left operand in TMEM; then dS = B^T (weighted x), and Y1 = (weights) x,
//   its first half of the tokens as soon as those weights are there
//   the state in registers, S <- exp(c_128) S + dS, and its pieces; the next chunk's weighted x; y = exp(c_t) Y0 + Y1 + D x
// The pieces of the state and of the weighted x are neighbouring columns of one product: a product of 32 columns costs as much as one
// of 96 (54 clocks, the left operand's reads).  Only the state's own line waits for the chunk before.  A weight's decay is one
// exponential where t and s lie in the same 32 tokens; elsewhere it is the product of two factors, from s to the end of its 32 and on to the
// last token before t's 32, and from there to t, which are made once a token, in double, and rounded once.
//
// What bounds it: a chunk's line, about 5,300 clocks: G read 700, the weights 2,500 (shared memory serves the products' operands meanwhile),
// dS awaited and the state published 1,000, weighted x 700, outputs 400.  2,048 tokens of 64 heads of 64 x 128: 53.3 us; 64.5 us with an
// exponential a weight, a lone lane issuing (110 clocks a product; an elected lane of a whole warp has what they take in uniform
// registers) and steps, stores and weighted x in the line; 132 us in chunks of 64 by mma.sync, 566 us walked.  (The weighted x made by the step warps:
// 55 us; there they are the longer line.)  Error against float64 1.2e-7 for y, 7.4e-8 for the state, as those.
//
// The products are causal for finite numbers only: above the diagonal the weights are zeros, and 0 * inf is no number; nor are the
// pieces of an infinity, or the differences of c where a decay is exactly zero; and a chunk's last rows may be another request's.
// Whatever is not finite makes a y of its own token or the last state not finite, so both are looked at (one multiplication an output),
// and a block that finds one walks its portion once more from the state as it was, token after token like ssm_scan16_kernel and with
// its bits.
//
// Every wait for a product, a copy or warps is bounded; a thread that gives up raises a block-wide flag, all warps still come to the
// barriers of the remaining chunks, the block lets its copies land and frees its TMEM.  It then records 7000000 in *status and returns, or, where
// the caller named no status word, walks its portion like the block that finds a number that is not finite.
constexpr int kChunk = 128, kChunkCols = 32, kChunkWarps = 16, kIssueWarp = 16, kStepWarp = 17, kStepWarps = 4,
              kChunkThreads = 32 * (kStepWarp + kStepWarps);

struct ChunkSmem {
  uint8_t c[2][2][kChunk * 128];             // two stages; blocks of 64 state rows, 128-byte rows of a token, 128-byte swizzle
  uint8_t b[2][2][kChunk * 128];
  uint8_t x[2][kChunk * 64];                 // 64-byte rows of a token, 64-byte swizzle; so are the pieces
  uint8_t w[3][kChunk * 64];                 // the weighted x
  uint8_t s[3][kChunk * 64];                 // the state before the chunk: a row per state row
  float dt[2][kChunk], hi[2][kChunk], lo[2][kChunk];           // step, c_t / ln 2 in two floats
  float grown[2][kChunk], weight[2][kChunk];                   // exp(c_t), dt_t exp(c_128 - c_t)
  float fall[2][kChunk], rise[2][3][kChunk];                   // exp(c_t - c_r), r the last token before t's 32; dt_s exp(c_r - c_s) for the later 32s' r
  alignas(16) float out[kChunk][kChunkCols + 4];               // a chunk's y on its way to whole lines
  double decay[kStepWarps];                                    // of 32 tokens each
  uint64_t bars[12];
  int abort;
  uint32_t tmem;
};
static_assert(offsetof(ChunkSmem, dt) % 16 == 0 && offsetof(ChunkSmem, hi) % 16 == 0 && offsetof(ChunkSmem, lo) % 16 == 0 &&
                  offsetof(ChunkSmem, out) % 16 == 0 && offsetof(ChunkSmem, rise) % 16 == 0 && (kChunkCols + 4) % 4 == 0 && offsetof(ChunkSmem, bars) % 8 == 0 &&
                  offsetof(ChunkSmem, decay) % 8 == 0 && offsetof(ChunkSmem, b) % 1024 == 0 && offsetof(ChunkSmem, x) % 1024 == 0 &&
                  offsetof(ChunkSmem, w) % 1024 == 0 && offsetof(ChunkSmem, s) % 1024 == 0, "read 16 bytes at a time; tiles start where their swizzle does");
// byte offset of 16-byte piece c of row r in a tile of 64-byte rows with the 64-byte swizzle
__device__ __forceinline__ uint32_t swz64(int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); }
// Tiles of 64-byte rows as an operand whose columns are its outer side: 512 bytes between groups of 8 rows, a tile from 32 columns to the next.
__device__ __forceinline__ uint64_t desc_rows64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | (uint64_t)((kChunk * 64) >> 4) << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
// split_pair for a pair that is held as one operand.
__device__ __forceinline__ void split_two(Two x, uint32_t* piece) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float a, b;
    x.get(a, b);
    const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    piece[k] = *reinterpret_cast<const uint32_t*>(&p);
    if (k < 2) x = fma2(Two(-1.f), Two(__uint_as_float(piece[k] << 16), __uint_as_float(piece[k] & 0xffff0000u)), x);
  }
}

template <int N>
__global__ void __launch_bounds__(kChunkThreads, 1)
ssm_chunk_kernel(const __grid_constant__ CUtensorMap map_bc, const __grid_constant__ CUtensorMap map_x, const __nv_bfloat16* __restrict__ xbc,
                 int channels, const __nv_bfloat16* __restrict__ proj, int ld, int off_dt, const float* __restrict__ dt_bias,
                 const float* __restrict__ a_log, const float* __restrict__ d_skip, float* __restrict__ state,
                 const int* __restrict__ seq_starts, const int* __restrict__ state_slots, float* __restrict__ y, int H, int P, int G,
                 int n_seqs, int* __restrict__ status) {
  chain_wait();
  // (a block of single tokens would hold an SM's shared memory for half a microsecond only to leave: 31 of them beside a portion 14 us)
  const int h = blockIdx.x, p0 = blockIdx.z * kChunkCols;
  const int seq = (int)gridDim.y == n_seqs ? (int)blockIdx.y : nth_portion(seq_starts, n_seqs, blockIdx.y);
  if (seq < 0) return;
  const int start = seq_starts[seq], n_tok = seq_starts[seq + 1] - start;
  if (n_tok <= 1) return;                                      // (a single token: the scan kernel's)
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  ChunkSmem& sm = *reinterpret_cast<ChunkSmem*>(smem);
  const int g = h / (H / G), inner = H * P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_chunks = (n_tok + kChunk - 1) / kChunk;
  // G there; the weights' pieces of the chunk's first and last 64 tokens; the weighted x's; dS there; Y there; the state's pieces; a stage's rows
  // (two); the outputs of the chunk before read; those stored and the next chunk's steps there; the first half of Y1 from the
  // two smaller pieces there
  constexpr int kBarG = 0, kBarP1 = 1, kBarP2 = 2, kBarW = 3, kBarD = 4, kBarY = 5, kBarS = 6, kBarL = 7, kBarR = 9, kBarT = 10, kBarH = 11;
  auto bar = [&](int which) { return smem_u32(&sm.bars[which]); };
  volatile int* abort_flag = &sm.abort;
  if (threadIdx.x == 0) {
    for (int i : {kBarG, kBarD, kBarY, kBarL, kBarL + 1, kBarR, kBarH}) mbar_init(bar(i), 1);
    mbar_init(bar(kBarT), kStepWarps);
    for (int i : {kBarP1, kBarP2, kBarW, kBarS}) mbar_init(bar(i), kChunkWarps);
    sm.abort = 0;
    mbar_init_fence();
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sm.tmem;
  // columns of TMEM.  G's first sum, then dS by three pieces: 0; Y0 by the state's three pieces; Y1; the weights' pieces for the chunk's last 64
  // tokens, 3 x 32, then for its first 64; G's second sum lies over two of those and the 64 columns behind them
  constexpr uint32_t kColD = 0, kColY0 = 128, kColY1 = 224, kColM = 352, kColG = 384;
  auto col_m = [](int unit, int piece) { return kColM - (unit >> 2) * 96 + 32 * piece + 8 * (unit & 3); };
  constexpr int kTopThreads = 32 * (kChunkWarps + kStepWarps);
  float probe = 0.f;                                           // no number once a result was not finite

  // the state: thread (row n, quarter qt) holds columns 8 qt .. 8 qt + 7 of row n
  const int quad = warp & 3, qt = (warp >> 2) & 3, row = 32 * quad + lane;
  float S[8];
  float* s_glob = state + (((size_t)state_slots[seq] * H + h) * N + row) * P + p0 + 8 * qt;
  const bool holds = warp < kChunkWarps && row < N;

  if (warp < kChunkWarps) {
    const uint32_t t_lane = tmem + ((uint32_t)(32 * quad) << 16);
    auto publish = [&]() {                                     // the state's pieces
      uint32_t piece[4][3];
#pragma unroll
      for (int i = 0; i < 4; ++i) split_two(Two(S[2 * i], S[2 * i + 1]), piece[i]);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        *reinterpret_cast<uint4*>(sm.s[k] + swz64(row, qt)) = make_uint4(piece[0][k], piece[1][k], piece[2][k], piece[3][k]);
    };
    auto arrive = [&](int which) {                             // this warp's part is in place for the products
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(which));
    };
    auto wait = [&](int which, uint32_t parity) {
      mbar_wait_or_abort(bar(which), parity, abort_flag);
      __syncwarp();
    };
    auto no_weights = [&](int u, int piece) {                  // zeros in the unit of 16 columns from a piece on: it lies above the diagonal
      const uint32_t zero[8] = {};
      for (; piece < 3; ++piece) tmem_st8(t_lane + col_m(u, piece), zero);
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) S[i] = 0.f;
    if (holds) {
#pragma unroll
      for (int i = 0; i < 8; i += 2) {                         // (states are 8-byte aligned)
        const float2 v = *reinterpret_cast<const float2*>(s_glob + i);
        S[i] = v.x; S[i + 1] = v.y;
      }
    }
    publish();
    for (int u = qt; u < 8; u += 4)
      if (u >= 2 * (quad + 1)) no_weights(u, 0);
    tmem_st_wait();
    fence_before_sync();
    fence_async_proxy();
    arrive(kBarS);
    auto weigh = [&](int c) {                                  // weighted x: tokens 32 (warp / 4) .. + 31, columns 8 (warp % 4) .. + 7
      const int st = c & 1, t = 32 * qt + lane;
      wait(kBarL + st, (c >> 1) & 1);
      const float f = sm.weight[st][t];
      const uint4 in = *reinterpret_cast<const uint4*>(sm.x[st] + swz64(t, quad));
      const uint32_t q[4] = {in.x, in.y, in.z, in.w};
      uint32_t piece[4][3];
#pragma unroll
      for (int i = 0; i < 4; ++i) split_two(Two(f) * Two(__uint_as_float(q[i] << 16), __uint_as_float(q[i] & 0xffff0000u)), piece[i]);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        *reinterpret_cast<uint4*>(sm.w[k] + swz64(t, quad)) = make_uint4(piece[0][k], piece[1][k], piece[2][k], piece[3][k]);
      fence_async_proxy();
      arrive(kBarW);
    };
    wait(kBarT, 0);
    weigh(0);
    const float dskip = d_skip[h];
    for (int c = 0; c < n_chunks; ++c) {
      const int st = c & 1;
      const uint32_t par = c & 1;
      named_barrier(1, kTopThreads);                           // this chunk's steps are there, everybody is done with the chunk before
      if (threadIdx.x == 0) mbar_arrive(bar(kBarR));
      __syncwarp();
      wait(kBarG, par);
      fence_after_sync();
      float gram[2][16];                                       // units qt and qt + 4 of these 32 tokens: 16 columns each
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int u = qt + 4 * i;
        if (u < 2 * (quad + 1)) {                              // (the same for the warp)
          float more[16];
          tmem_ld16(t_lane + 16 * u, gram[i]);
          tmem_ld16(t_lane + kColG + 16 * u, more);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) gram[i][j] += more[j];
        }
      }
      fence_before_sync();
      named_barrier(4 + quad, 128);                            // the weights take the place of the second sum: all four warps have read it
      const Two hi_t(sm.hi[st][row]), lo_t(sm.lo[st][row]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int u = qt + 4 * i;
        if (u < 2 * (quad + 1)) {
          uint32_t piece[8][3];
          if (u < 2 * quad) {                                  // (the same for the warp) before these tokens' group: two factors
            const Two fall(sm.fall[st][row]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float4 f = *reinterpret_cast<const float4*>(&sm.rise[st][quad - 1][16 * u + 4 * j]);
              split_two(Two(gram[i][4 * j], gram[i][4 * j + 1]) * Two(f.x, f.y) * fall, piece[2 * j]);
              split_two(Two(gram[i][4 * j + 2], gram[i][4 * j + 3]) * Two(f.z, f.w) * fall, piece[2 * j + 1]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int s0 = 16 * u + 4 * j;
              const float4 hs = *reinterpret_cast<const float4*>(&sm.hi[st][s0]), ls = *reinterpret_cast<const float4*>(&sm.lo[st][s0]);
              const float4 ds = *reinterpret_cast<const float4*>(&sm.dt[st][s0]);
              const Two h2[2] = {Two(hs.x, hs.y), Two(hs.z, hs.w)}, l2[2] = {Two(ls.x, ls.y), Two(ls.z, ls.w)}, d2[2] = {Two(ds.x, ds.y), Two(ds.z, ds.w)};
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                const Two gap = fma2(Two(-1.f), h2[k], hi_t) + fma2(Two(-1.f), l2[k], lo_t);
                float e0, e1, w0, w1;
                gap.get(e0, e1);
                (Two(gram[i][4 * j + 2 * k], gram[i][4 * j + 2 * k + 1]) * d2[k] * Two(fast_exp2(e0), fast_exp2(e1))).get(w0, w1);
                split_two(Two(s0 + 2 * k <= row ? w0 : 0.f, s0 + 2 * k + 1 <= row ? w1 : 0.f), piece[2 * j + k]);
              }
            }
          }
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            uint32_t out[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) out[j] = piece[j][k];
            tmem_st8(t_lane + col_m(u, k), out);
          }
        } else if (u < 4) {
          no_weights(u, 1);                                    // (the second sum lay over two of the pieces)
        }
        tmem_st_wait();
        fence_before_sync();
        arrive(i == 0 ? kBarP1 : kBarP2);
      }
      // the state
      wait(kBarD, par);
      fence_after_sync();
      float v[8], v1[8], v2[8];
      tmem_ld8(t_lane + kColD + 8 * qt, v);
      tmem_ld8(t_lane + kColD + 32 + 8 * qt, v1);
      tmem_ld8(t_lane + kColD + 64 + 8 * qt, v2);
      tmem_ld_wait();
      if (holds) {
        const float total = sm.grown[st][kChunk - 1];
#pragma unroll
        for (int i = 0; i < 8; ++i) S[i] = fmaf(total, S[i], (v2[i] + v1[i]) + v[i]);
      }
      publish();
      fence_before_sync();
      fence_async_proxy();
      arrive(kBarS);
      wait(kBarT, par ^ 1);
      if (c + 1 < n_chunks) weigh(c + 1);
      // the outputs of token `row`
      wait(kBarY, par);
      fence_after_sync();
      float own[8];
      tmem_ld8(t_lane + kColY0 + 8 * qt, v);
      tmem_ld8(t_lane + kColY0 + 32 + 8 * qt, v1);
      tmem_ld8(t_lane + kColY0 + 64 + 8 * qt, v2);
      tmem_ld8(t_lane + kColY1 + 8 * qt, own);
      tmem_ld_wait();
      fence_before_sync();
      {
        const float grown = sm.grown[st][row];
        const uint4 in = *reinterpret_cast<const uint4*>(sm.x[st] + swz64(row, qt));
        const uint32_t q[4] = {in.x, in.y, in.z, in.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[2 * i] = fmaf(grown, (v2[2 * i] + v1[2 * i]) + v[2 * i], own[2 * i]) + dskip * __uint_as_float(q[i] << 16);
          v[2 * i + 1] = fmaf(grown, (v2[2 * i + 1] + v1[2 * i + 1]) + v[2 * i + 1], own[2 * i + 1]) + dskip * __uint_as_float(q[i] & 0xffff0000u);
        }
        if (c * kChunk + row < n_tok)
#pragma unroll
          for (int i = 0; i < 8; ++i) probe = fmaf(v[i], 0.f, probe);
        *reinterpret_cast<float4*>(&sm.out[row][8 * qt]) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(&sm.out[row][8 * qt + 4]) = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) probe = fmaf(S[i], 0.f, probe);
    named_barrier(1, kTopThreads);
  } else if (warp == kIssueWarp) {
    // The whole warp walks the chunks and one elected lane issues: what a product takes then lies in uniform registers (a lone lane
    // took 110 clocks a product, 56 products a chunk).
    constexpr uint32_t kIdescG = mma_idesc(128, kChunk, false), kIdesc1 = mma_idesc(128, kChunkCols, true),
                       kIdesc3 = mma_idesc(128, 3 * kChunkCols, true), kIdescT = kIdesc3 | (1u << 15);
    constexpr uint64_t kBlock = (kChunk * 128) >> 4;           // from a tile's first 64 state rows to its others, in 16-byte pieces
    constexpr uint64_t kPiece = (kChunk * 64) >> 4;
    const bool elected = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const int chunks = __shfl_sync(0xffffffffu, n_chunks, 0);
    const uint64_t ds = desc_rows64(smem_u32(sm.s[0])), dw = desc_rows64(smem_u32(sm.w[0])), dx0 = desc_rows64(smem_u32(sm.x[0]));
    const uint64_t dc0 = make_desc(smem_u32(sm.c[0][0])), db0 = make_desc(smem_u32(sm.b[0][0]));
    bool ok = true;
    auto wait = [&](int which, uint32_t parity) {
      if (ok) ok = mbar_wait_or_abort(bar(which), parity, abort_flag);
      return ok = __all_sync(0xffffffffu, ok) != 0;
    };
    auto issue_g = [&](int c, int half) {                      // a sum of G over half of the state's rows
      const uint64_t dc = dc0 + (c & 1) * 2 * kBlock, db = db0 + (c & 1) * 2 * kBlock;
#pragma unroll
      for (int i = 0; i < N / 32; ++i) {
        const int k = half * (N / 32) + i;
        mma_bf16(tm + half * kColG, dc + (k >> 2) * kBlock + 2 * (k & 3), db + (k >> 2) * kBlock + 2 * (k & 3), kIdescG, i > 0);
      }
    };
    auto issue_y1 = [&](uint64_t dx, int half, int p) {        // the part of Y1 from a piece of the weights for half of the chunk's tokens
#pragma unroll
      for (int i = 0; i < kChunk / 32; ++i) {
        const int k = half * (kChunk / 32) + i;
        mma_bf16_a_tmem(tm + kColY1, tm + col_m(k, p), dx + 64 * k, kIdesc1, half || p < 2 || i > 0);
      }
    };
    if (wait(kBarS, 0) && wait(kBarL, 0)) {
      fence_after_sync();
      if (elected) {
        issue_g(0, 0);
        issue_g(0, 1);
        mma_commit(bar(kBarG));
      }
      __syncwarp();
    }
    for (int c = 0; c < chunks && ok; ++c) {
      const int st = c & 1;
      const bool more = c + 1 < chunks;
      // dS = B^T (weighted x): B's rows are its tokens, 64 state rows to a block
      const uint64_t dc = dc0 + st * 2 * kBlock, dx = dx0 + st * kPiece, db = ((db0 + st * 2 * kBlock) & ~((uint64_t)0x3fff << 16)) | (kBlock << 16);
      if (!wait(kBarR, c & 1)) break;
      fence_after_sync();
      if (elected) {
#pragma unroll
        for (int k = 0; k < N / 16; ++k)                       // Y0 = C S
          mma_bf16(tm + kColY0, dc + (k >> 2) * kBlock + 2 * (k & 3), ds + 64 * k, kIdesc3, k > 0);
      }
      __syncwarp();
      if (!wait(kBarW, c & 1) || !wait(kBarP1, c & 1)) break;  // (all of G has been read)
      fence_after_sync();
      if (elected) {
#pragma unroll
        for (int k = 0; k < kChunk / 16; ++k) mma_bf16(tm + kColD, db + 128 * k, dw + 64 * k, kIdescT, k > 0);
        mma_commit(bar(kBarD));                                // (the state's pieces have been read, too)
        issue_y1(dx, 0, 2);                                    // (the smallest pieces first)
        issue_y1(dx, 0, 1);
        mma_commit(bar(kBarH));
        issue_y1(dx, 0, 0);
      }
      __syncwarp();
      // G's second sum lies over the two smaller pieces of these weights, and nothing says that products of other shapes and sums are finished
      // in the order of issue: it waits for their commit.  The weights for the second half are still being made meanwhile.
      if (!wait(kBarH, c & 1)) break;
      if (more) {
        if (!wait(kBarL + (st ^ 1), ((c + 1) >> 1) & 1)) break;
        fence_after_sync();
        if (elected) issue_g(c + 1, 1);
        __syncwarp();
      }
      if (!wait(kBarP2, c & 1)) break;
      fence_after_sync();
      if (elected) {
#pragma unroll
        for (int p = 2; p >= 0; --p) issue_y1(dx, 1, p);
        mma_commit(bar(kBarY));
      }
      __syncwarp();
      if (more) {
        if (!wait(kBarS, (c + 1) & 1)) break;                  // (dS has been read)
        fence_after_sync();
        if (elected) {
          issue_g(c + 1, 0);
          mma_commit(bar(kBarG));
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else {                                                     // steps and decays: token 32 w + lane of a chunk
    const int w = warp - kStepWarp, r = 32 * w + lane;
    const float a = -expf(a_log[h]), bias = dt_bias[h];
    auto load_stage = [&](int c) {                             // (rows behind the request's are looked at by nothing that is kept)
      const int st = c & 1, at = start + c * kChunk;
      const uint32_t full = bar(kBarL + st);
      mbar_expect(full, (N > 64 ? 4 : 2) * kChunk * 128 + kChunk * 64);
      for (int j = 0; j < (N > 64 ? 2 : 1); ++j) {
        tma_load_box(smem_u32(sm.c[st][j]), &map_bc, inner + (G + g) * N + 64 * j, at, full);
        tma_load_box(smem_u32(sm.b[st][j]), &map_bc, inner + g * N + 64 * j, at, full);
      }
      tma_load_box(smem_u32(sm.x[st]), &map_x, h * P + p0, at, full);
    };
    float dt, hi, lo, fall, rise[kStepWarps - 1], grown, weight;   // of a chunk's token, on their way
    auto raw_step = [&](int c) { return c * kChunk + r < n_tok ? __bfloat162float(proj[(size_t)(start + c * kChunk + r) * ld + off_dt + h]) : 0.f; };
    auto make_steps = [&](int c, float raw_dt) {
      dt = c * kChunk + r < n_tok ? softplus_f(raw_dt + bias) : 0.f;
      double cum = (double)a * (double)dt;                     // inclusive sums over the group's lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, cum, o);
        if (lane >= o) cum += v;
      }
      const double sum = __shfl_sync(0xffffffffu, cum, 31), l2 = cum * 1.4426950408889634;
      hi = (float)l2;
      lo = (float)(l2 - (double)hi);
      double from = exp(cum), to = (double)dt * exp(sum - cum);     // from the group's start, to its end
      fall = (float)from;
      named_barrier(2, 32 * kStepWarps);                       // (all have read the decays of the chunk before)
      if (lane == 31) sm.decay[w] = from;
      named_barrier(2, 32 * kStepWarps);
#pragma unroll
      for (int i = 0; i < kStepWarps; ++i) {
        if (i < w) from *= sm.decay[i];
        if (i > w) {
          rise[i > 0 ? i - 1 : 0] = (float)to;
          to *= sm.decay[i];
        }
      }
      grown = (float)from;
      weight = (float)to;
    };
    auto place_steps = [&](int c) {
      const int st = c & 1;
      sm.dt[st][r] = dt;
      sm.hi[st][r] = hi;
      sm.lo[st][r] = lo;
      sm.fall[st][r] = fall;
      sm.grown[st][r] = grown;
#pragma unroll
      for (int i = 1; i < kStepWarps; ++i)
        if (i > w) sm.rise[st][i - 1][r] = rise[i - 1];
      sm.weight[st][r] = weight;
    };
    auto store = [&](int c) {                                  // the outputs of chunk c: eight lanes a token, whole lines
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = 32 * w + 4 * i + (lane >> 3), e = 4 * (lane & 7);
        if (c * kChunk + t < n_tok)
          *reinterpret_cast<float4*>(y + (size_t)(start + c * kChunk + t) * inner + h * P + p0 + e) = *reinterpret_cast<const float4*>(&sm.out[t][e]);
      }
    };
    const bool copies = w == 0 && lane == 0;
    if (copies) load_stage(0);
    __syncwarp();
    float raw_dt = raw_step(1);                                // asked for before it is used
    make_steps(0, raw_step(0));
    place_steps(0);
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(kBarT));
    if (n_chunks > 1) make_steps(1, raw_dt);
    raw_dt = raw_step(2);
    for (int c = 0; c < n_chunks; ++c) {
      const bool more = c + 1 < n_chunks;
      named_barrier(1, kTopThreads);
      if (copies && more) load_stage(c + 1);
      __syncwarp();
      if (more) place_steps(c + 1);
      if (c > 0) store(c - 1);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kBarT));
      if (c + 2 < n_chunks) make_steps(c + 2, raw_dt);
      raw_dt = raw_step(c + 3);
    }
    named_barrier(1, kTopThreads);
    store(n_chunks - 1);
  }
  const bool odd = __syncthreads_or(!(probe == 0.f));
  const bool gave_up = *abort_flag != 0;
  if (gave_up && threadIdx.x == 0) {
    for (int c = max(0, n_chunks - 2); c < n_chunks; ++c) mbar_wait(bar(kBarL + (c & 1)), (c >> 1) & 1);
    if (status) atomicCAS(status, 0, 7000000);
  }
  __syncthreads();
  if (warp == kIssueWarp) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (gave_up && status) return;
  if (odd || gave_up) {                                        // (in room that no copy and no barrier uses)
    static_assert(offsetof(ChunkSmem, w) + scan_smem(N, kChunkCols, N / 8) <= offsetof(ChunkSmem, bars) && N / 8 * kChunkCols <= kChunkWarps * 32,
                  "the walk has room");
    scan_tokens<__nv_bfloat16, 8, true>(reinterpret_cast<float*>(sm.w), xbc, channels, proj, ld, off_dt, dt_bias, a_log, d_skip, state,
                                        seq_starts, state_slots, y, H, P, N, G, kChunkCols, h, seq, p0);
    return;
  }
  if (holds) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) *reinterpret_cast<float2*>(s_glob + i) = make_float2(S[i], S[i + 1]);
  }
}

// The same sums 64 tokens at a time with mma.sync, for portions of at most 64 tokens (longer ones it takes, too, a chunk after the other): without
// TMEM to fetch and give back, copies through descriptors and a chunk of 128 rows, of which half or more would be zeros, a portion of up to 64
// tokens takes 7.5 us instead of 10.0 (64 heads of 64 x 128; 8 of 32 x 32 5.1 | 6.9), eight of 40 46.1 | 64.1, one of 64 beside 31 single tokens 41.6 |
// 56.2; at 65 tokens and more the kernel above is as fast or faster (300 tokens 23 | 14).
// Block: one (head, request, 32 columns), 16 warps of products and one that makes the next chunk's steps and decays; the state stays in the
// accumulators' registers.  Between the two barriers of a chunk the work is cut into pieces of about the same length: first 10 of the warps make a
// tile of the weights (C B^T below the diagonal) each, the others the weighted x, and every warp 16 rows x 8 columns of the part of y that comes from
// the state; then the same 16 x 8 of the part within the chunk, and 16 rows of the state.  What is not finite is walked, as above.
constexpr int kShortChunk = 64, kShortWarps = 16;

template <int N>
struct ShortSmem {
  static constexpr int LdN = N + 8, LdP = kChunkCols + 8, LdM = kShortChunk + 8;   // rows 16 bytes longer than a power of two: no bank conflicts
  __nv_bfloat16 c[2][kShortChunk][LdN];
  __nv_bfloat16 b[2][kShortChunk][LdN];
  __nv_bfloat16 x[2][kShortChunk][LdP];
  __nv_bfloat16 s[3][N][LdP];                                  // the state before the chunk, in pieces
  __nv_bfloat16 w[3][kShortChunk][LdP];                             // the weighted x, in pieces
  __nv_bfloat16 m[3][kShortChunk][LdM];                             // the weights of the sum within the chunk, in pieces (tiles above the diagonal unused)
  float dt[2][kShortChunk], hi[2][kShortChunk], lo[2][kShortChunk];           // step, c_t / ln 2 in two floats
  float grown[2][kShortChunk], weight[2][kShortChunk];                   // exp(c_t), dt_t exp(c_64 - c_t)
  float total[2];                                              // exp(c_64)
};

template <int N>
__global__ void __launch_bounds__((kShortWarps + 1) * 32)
ssm_short_kernel(const __nv_bfloat16* __restrict__ xbc, int channels, const __nv_bfloat16* __restrict__ proj, int ld, int off_dt,
                 const float* __restrict__ dt_bias, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                 float* __restrict__ state, const int* __restrict__ seq_starts, const int* __restrict__ state_slots,
                 float* __restrict__ y, int H, int P, int G, int n_seqs) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ShortSmem<N>& sm = *reinterpret_cast<ShortSmem<N>*>(smem_raw);
  const int h = blockIdx.x, p0 = blockIdx.z * kChunkCols;
  const int seq = (int)gridDim.y == n_seqs ? (int)blockIdx.y : nth_portion(seq_starts, n_seqs, blockIdx.y);
  if (seq < 0) return;
  const int start = seq_starts[seq], n_tok = seq_starts[seq + 1] - start;
  if (n_tok <= 1) return;                                      // (a single token: the scan kernel's)
  const int g = h / (H / G), inner = H * P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qr = lane >> 2, qc = lane & 3;
  const int n_chunks = (n_tok + kShortChunk - 1) / kShortChunk;
  const __nv_bfloat16* rows = xbc + (size_t)start * channels;

  auto load_stage = [&](int c) {                               // the threads of the products
    const int buf = c & 1, c0 = c * kShortChunk;
    for (int idx = threadIdx.x; idx < kShortChunk * (N / 8); idx += kShortWarps * 32) {
      const int r = idx / (N / 8), e = 8 * (idx % (N / 8));
      const bool real = c0 + r < n_tok;
      const __nv_bfloat16* src = rows + (size_t)(real ? c0 + r : 0) * channels + inner + g * N + e;
      copy16_or_zero(&sm.b[buf][r][e], src, real);
      copy16_or_zero(&sm.c[buf][r][e], src + G * N, real);
    }
    if (threadIdx.x < kShortChunk * (kChunkCols / 8)) {
      const int r = threadIdx.x / (kChunkCols / 8), e = 8 * (threadIdx.x % (kChunkCols / 8));
      const bool real = c0 + r < n_tok;
      copy16_or_zero(&sm.x[buf][r][e], rows + (size_t)(real ? c0 + r : 0) * channels + h * P + p0 + e, real);
    }
    copy_commit();
  };
  const float a = -expf(a_log[h]), bias = dt_bias[h];
  auto make_steps = [&](int c) {                               // the last warp: tokens 2 lane and 2 lane + 1 of chunk c
    const int buf = c & 1, t0 = c * kShortChunk + 2 * lane;
    float dt[2];
    double la[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      dt[i] = t0 + i < n_tok ? softplus_f(__bfloat162float(proj[(size_t)(start + t0 + i) * ld + off_dt + h]) + bias) : 0.f;
      la[i] = (double)a * (double)dt[i];
    }
    double sum = la[0] + la[1];                                // inclusive scan over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    const double all = __shfl_sync(0xffffffffu, sum, 31);
    const double cum[2] = {sum - la[1], sum};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 2 * lane + i;
      const double l2 = cum[i] * 1.4426950408889634;
      const float hi = (float)l2;
      sm.dt[buf][r] = dt[i];
      sm.hi[buf][r] = hi;
      sm.lo[buf][r] = (float)(l2 - (double)hi);
      sm.grown[buf][r] = (float)exp(cum[i]);
      sm.weight[buf][r] = (float)((double)dt[i] * exp(all - cum[i]));
    }
    if (lane == 0) sm.total[buf] = (float)exp(all);
  };

  // the state: warp w holds rows 16 (w mod N/16) .. + 15, columns 8 NTW (w div N/16) .. + 8 NTW - 1
  constexpr int kRowTiles = N / 16, kColGroups = kShortWarps / kRowTiles < 4 ? kShortWarps / kRowTiles : 4, NTW = 4 / kColGroups;
  const bool holds_state = warp < kRowTiles * kColGroups;
  const int s_row = 16 * (warp % kRowTiles), s_col = 8 * NTW * (warp / kRowTiles);
  float S[NTW][4];
  float* s_glob = state + ((size_t)state_slots[seq] * H + h) * N * P + p0;
  auto publish = [&]() {                                       // the state's pieces to shared memory
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t piece[3];
        split_pair(S[nt][2 * j], S[nt][2 * j + 1], piece);
#pragma unroll
        for (int k = 0; k < 3; ++k)
          *reinterpret_cast<uint32_t*>(&sm.s[k][s_row + qr + 8 * j][s_col + 8 * nt + 2 * qc]) = piece[k];
      }
  };
  if (warp < kShortWarps) load_stage(0);
  else make_steps(0);
  if (holds_state) {
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float2 v = *reinterpret_cast<const float2*>(s_glob + (size_t)(s_row + qr + 8 * j) * P + s_col + 8 * nt + 2 * qc);
        S[nt][2 * j] = v.x;
        S[nt][2 * j + 1] = v.y;
      }
    publish();
  }
  const int y_row = 16 * (warp >> 2), y_col = 8 * (warp & 3);
  // the tile of the weights that a warp makes: warps 0 .. 9 take the tiles (row, column) on and below the diagonal
  const int m_tr = warp < 1 ? 0 : warp < 3 ? 1 : warp < 6 ? 2 : 3;
  const int m_row = 16 * m_tr, m_col = 16 * (warp - m_tr * (m_tr + 1) / 2);
  const float dskip = d_skip[h];
  float probe = 0.f;                                           // no number once a result was not finite
  for (int c = 0; c < n_chunks; ++c) {
    const int buf = c & 1;
    if (warp < kShortWarps) copy_wait<0>();
    __syncthreads();                                           // chunk c's rows, steps and state pieces are there; stage c - 1 is free
    if (warp == kShortWarps) {
      if (c + 1 < n_chunks) make_steps(c + 1);
      __syncthreads();
      continue;
    }
    if (c + 1 < n_chunks) load_stage(c + 1);
    // the part of y that comes from the state
    float inter[3][4] = {};
#pragma unroll
    for (int k = 0; k < N / 16; k += 2) {
      uint32_t cf[2][4], b[3][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) ldmatrix4(cf[i], &sm.c[buf][y_row + (lane & 15)][16 * (k + i) + 8 * (lane >> 4)]);
#pragma unroll
      for (int piece = 0; piece < 3; ++piece) ldmatrix4t(b[piece], &sm.s[piece][16 * k + lane][y_col]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int piece = 0; piece < 3; ++piece) mma16816(inter[piece], cf[i], b[piece][2 * i], b[piece][2 * i + 1]);
    }
    if (warp < 10) {                                           // a tile of the weights
      float gram[2][2][4] = {};                                // (two chains: a product does not wait for the one before it)
#pragma unroll
      for (int k = 0; k < N / 16; ++k) {
        uint32_t cf[4], b[4];
        ldmatrix4(cf, &sm.c[buf][m_row + (lane & 15)][16 * k + 8 * (lane >> 4)]);
        ldmatrix4(b, &sm.b[buf][m_col + (lane & 7) + 8 * (lane >> 4)][16 * k + 8 * ((lane >> 3) & 1)]);
        mma16816(gram[k & 1][0], cf, b[0], b[1]);
        mma16816(gram[k & 1][1], cf, b[2], b[3]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int s = m_col + 8 * nt + 2 * qc;
        const float2 hs = *reinterpret_cast<const float2*>(&sm.hi[buf][s]), ls = *reinterpret_cast<const float2*>(&sm.lo[buf][s]);
        const float2 ds = *reinterpret_cast<const float2*>(&sm.dt[buf][s]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int r = m_row + qr + 8 * j;
          const float hi = sm.hi[buf][r], lo = sm.lo[buf][r];
          const float v0 = s <= r ? (gram[0][nt][2 * j] + gram[1][nt][2 * j]) * ds.x * exp2f((hi - hs.x) + (lo - ls.x)) : 0.f;
          const float v1 = s + 1 <= r ? (gram[0][nt][2 * j + 1] + gram[1][nt][2 * j + 1]) * ds.y * exp2f((hi - hs.y) + (lo - ls.y)) : 0.f;
          uint32_t piece[3];
          split_pair(v0, v1, piece);
#pragma unroll
          for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(&sm.m[k][r][s]) = piece[k];
        }
      }
    } else {                                                   // weighted x in pieces: 4 columns of one token at a time
      for (int idx = threadIdx.x - 320; idx < kShortChunk * (kChunkCols / 4); idx += 192) {
        const int r = idx >> 3, e = 4 * (idx & 7);
        float v[4];
        Pack4<__nv_bfloat16>::load(&sm.x[buf][r][e], v);
        const float f = sm.weight[buf][r];
        uint32_t p01[3], p23[3];
        split_pair(f * v[0], f * v[1], p01);
        split_pair(f * v[2], f * v[3], p23);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(&sm.w[k][r][e]) = make_uint2(p01[k], p23[k]);
      }
    }
    __syncthreads();                                           // weights and weighted x are complete; nobody reads the state's pieces any more
    float add[3][NTW][4] = {};
    if (holds_state) {
#pragma unroll
      for (int k = 0; k < kShortChunk / 16; ++k) {
        uint32_t bt[4], b[3][4];                               // B^T: 16 state rows x 16 tokens
        ldmatrix4t(bt, &sm.b[buf][16 * k + (lane & 7) + 8 * (lane >> 4)][s_row + 8 * ((lane >> 3) & 1)]);
#pragma unroll
        for (int piece = 0; piece < 3; ++piece) {
          if (NTW == 2) ldmatrix4t(b[piece], &sm.w[piece][16 * k + (lane & 15)][s_col + 8 * (lane >> 4)]);
          else ldmatrix2t(b[piece], &sm.w[piece][16 * k + (lane & 15)][s_col]);
        }
#pragma unroll
        for (int piece = 0; piece < 3; ++piece)
#pragma unroll
          for (int nt = 0; nt < NTW; ++nt) mma16816(add[piece][nt], bt, b[piece][2 * nt], b[piece][2 * nt + 1]);
      }
    }
    float intra[3][4] = {};                                    // the part of y from the chunk's own tokens
    for (int k = 0; k <= (warp >> 2); k += 2) {
      uint32_t xb[4], mf[3][4];
      ldmatrix4t(xb, &sm.x[buf][16 * k + lane][y_col]);        // (rows 16 k .. + 31: the second half may lie behind the diagonal)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (k + i > (warp >> 2)) break;
#pragma unroll
        for (int piece = 0; piece < 3; ++piece) ldmatrix4(mf[piece], &sm.m[piece][y_row + (lane & 15)][16 * (k + i) + 8 * (lane >> 4)]);
#pragma unroll
        for (int piece = 0; piece < 3; ++piece) mma16816(intra[piece], mf[piece], xb[2 * i], xb[2 * i + 1]);
      }
    }
    if (holds_state) {
      const float total = sm.total[buf];
#pragma unroll
      for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[nt][i] = fmaf(total, S[nt][i], (add[2][nt][i] + add[1][nt][i]) + add[0][nt][i]);
      publish();
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = y_row + qr + 8 * j, col = y_col + 2 * qc;
      if (c * kShortChunk + r < n_tok) {
        const float grown = sm.grown[buf][r];
        const float2 xv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&sm.x[buf][r][col]));
        float v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int q = 2 * j + i;
          const float before = (inter[2][q] + inter[1][q]) + inter[0][q], own = (intra[2][q] + intra[1][q]) + intra[0][q];
          v[i] = fmaf(grown, before, own) + dskip * (i ? xv.y : xv.x);
          probe = fmaf(v[i], 0.f, probe);
        }
        *reinterpret_cast<float2*>(y + (size_t)(start + c * kShortChunk + r) * inner + h * P + p0 + col) = make_float2(v[0], v[1]);
      }
    }
  }
  if (holds_state) {
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) probe = fmaf(S[nt][i], 0.f, probe);
  }
  if (__syncthreads_or(!(probe == 0.f))) {
    static_assert(scan_smem(N, kChunkCols, N / 8) <= sizeof(ShortSmem<N>) && N / 8 * kChunkCols <= kShortWarps * 32, "the walk has room");
    scan_tokens<__nv_bfloat16, 8, true>(reinterpret_cast<float*>(smem_raw), xbc, channels, proj, ld, off_dt, dt_bias, a_log, d_skip, state,
                                        seq_starts, state_slots, y, H, P, N, G, kChunkCols, h, seq, p0);
    return;
  }
  if (holds_state) {
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        *reinterpret_cast<float2*>(s_glob + (size_t)(s_row + qr + 8 * j) * P + s_col + 8 * nt + 2 * qc) =
            make_float2(S[nt][2 * j], S[nt][2 * j + 1]);
  }
}
#endif  // ERB_ELEM == 1

// One block per (token, part): out = unit_rms(y * silu(z)) * weight over the part's entries.  `gate` may
// be null (no gate), `x` is float (X32) or T.
template <typename T, bool X32>
__global__ void __launch_bounds__(256)
gated_group_norm_kernel(const void* __restrict__ x_, int x_ld, const T* __restrict__ gate, int gate_ld,
                        const float* __restrict__ weight, T* __restrict__ out, int out_ld, int width, int parts, float eps) {
  chain_wait();
  __shared__ float scratch[32];
  const int t = blockIdx.x, part = blockIdx.y;
  const int per = width / parts, lo = part * per;
  float ss = 0.f;
  auto value = [&](int i) {
    float v = X32 ? static_cast<const float*>(x_)[(size_t)t * x_ld + i] : Elem<T>::load(static_cast<const T*>(x_) + (size_t)t * x_ld + i);
    if (gate) v *= silu_f(Elem<T>::load(gate + (size_t)t * gate_ld + i));
    return v;
  };
  for (int i = lo + threadIdx.x; i < lo + per; i += blockDim.x) {
    const float v = value(i);
    ss += v * v;
  }
  const float rs = rsqrtf(block_sum(ss, scratch) / (float)per + eps);
  for (int i = lo + threadIdx.x; i < lo + per; i += blockDim.x)
    Elem<T>::store(out + (size_t)t * out_ld + i, value(i) * rs * weight[i]);
}

// The same for parts of 128 V entries (V up to 8) and rows whose parts start aligned: a warp per (token, part), 4 V entries a
// lane held in registers between the sum and the store, so that nothing is read or gated twice.
// 2,048 tokens of 8 parts of 512: 42 us by the kernel above, 11.4 us; one token 2.9 us by both.
template <typename T, bool X32, int V>
__global__ void __launch_bounds__(128)
gated_group_norm_vec_kernel(const void* __restrict__ x_, int x_ld, const T* __restrict__ gate, int gate_ld,
                            const float* __restrict__ weight, T* __restrict__ out, int out_ld, int n_items, int parts, float eps) {
  chain_wait();
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= n_items) return;
  constexpr int per = 128 * V;
  const int t = item / parts, lo = (item % parts) * per + 4 * lane;
  float v[V][4], ss = 0.f;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    if (X32) load4(static_cast<const float*>(x_) + (size_t)t * x_ld + lo + 128 * j, v[j]);
    else Pack4<T>::load(static_cast<const T*>(x_) + (size_t)t * x_ld + lo + 128 * j, v[j]);
  }
  if (gate) {
    float z[V][4];
#pragma unroll
    for (int j = 0; j < V; ++j) Pack4<T>::load(gate + (size_t)t * gate_ld + lo + 128 * j, z[j]);
#pragma unroll
    for (int j = 0; j < V; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) v[j][i] *= silu_f(z[j][i]);
  }
#pragma unroll
  for (int j = 0; j < V; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = fmaf(v[j][i], v[j][i], ss);
  const float rs = rsqrtf(warp_sum(ss) / (float)per + eps);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    float w[4];
    load4(weight + lo + 128 * j, w);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = v[j][i] * rs * w[i];
    Pack4<T>::store(out + (size_t)t * out_ld + lo + 128 * j, w);
  }
}

#if ERB_ELEM == 1
// Which form is the fastest: a chunk's tokens of the kernel that takes portions in chunks, 0 for the walk.  The costs in microseconds, fitted to the
// kernels' times over 1 to 64 requests of 2 to 2,048 tokens (64 heads of 64 x 128 and 32 of 64 x 64; of 196 pairs measured one is decided
// wrongly, 33.4 us against 30.3).  The walk costs 0.27 us a token of the longest portion or, when the GPU is full, its blocks' tokens and states;
// a chunk of 128 tokens costs 2.8 us for the longest portion, or as many rounds of blocks as the SMs need, a block an SM.  Portions of at most 64
// tokens take the kernel for those (its header), at its latency or its blocks.  One request: from 17 tokens on (64 x 128: 16 tokens 6.7 us walked,
// 7.1 in a chunk; 20 8.5 | 7.3; 8 of 32 x 32: 16 5.9 | 5.0); eight of 24 tokens are walked (41.8 | 45.5), of 32 not (52.0 | 45.8).
inline int chunk_of(int blocks, int N, int n_tokens, int n_seqs, int longest) {
  if (longest <= 1) return 0;
  const double size = N / 128.0, extra = (double)n_tokens - n_seqs - (longest - 1);      // tokens beyond one of the other requests
  const double others = fmax(0.0, extra < n_seqs - 1 ? extra : n_seqs - 1);
  const double walk = fmax(3.0 + 0.27 * longest, blocks * size * (0.00165 * n_tokens + 0.008 * n_seqs));
  if (longest <= kShortChunk) {
    const double busy = 0.036 * blocks * (1.0 + (others > 0.0 ? others + extra / kShortChunk : 0.0));
    return fmax(4.6 + 2.75 * size, busy) < fmax(3.0 + 0.27 * longest, blocks * size * (0.0015 * n_tokens + 0.008 * n_seqs)) ? kShortChunk : 0;
  }
  const double longest_chunks = (longest + kChunk - 1) / kChunk, chunks = longest_chunks + (others > 0.0 ? others + extra / kChunk : 0.0);
  const double rounds = ceil(blocks * (1.0 + others) / sm_count());
  return fmax(7.0 + 2.7 * longest_chunks, rounds * (2.6 + 2.8 * size + 2.9 * chunks / (1.0 + others))) < walk ? kChunk : 0;
}
#endif

}  // namespace

ERB_EXPORT int erb_conv_silu(const void* proj, int n_tokens, int ld, int off, int channels, int taps, const void* weight,
                             const void* bias, const float* conv_state, const int* seq_of_token, const int* seq_starts,
                             const int* state_slots, void* out, void* stream) {
  if (n_tokens <= 0) return ERB_OK;
  if (channels <= 0 || taps < 1 || (taps > 1 && !conv_state)) return fail(ERB_ERR_ARG, "conv_silu: bad sizes");
#if ERB_ELEM == 1
  // Few channels of few tokens: the kernel above, whose threads have less to do one after the other (8 tokens of 6,144 channels 1.9 us
  // there, 2.5 here; 256 of 72 1.8 | 2.5); from 64 tokens on it gives a token's channels to one block (64 of 1,024 3.1 | 2.5, of
  // 6,144 12.6 | 2.9).  Four tokens a thread read the weights and the inputs seldom: from about 700 tokens of 6,144 channels on (8.7 us, and
  // 10.2 with one token a thread and the earlier arithmetic; 256 tokens 5.6 us with four, 5.2 with one).
  const long long sums = (long long)n_tokens * channels;
  if ((sums >= 100000 || (n_tokens >= 64 && channels >= 1024)) && taps == 4 && channels % 8 == 0 && ld % 8 == 0 && off % 8 == 0 &&
      !(((uintptr_t)proj | (uintptr_t)weight | (uintptr_t)bias | (uintptr_t)conv_state | (uintptr_t)out) & 15)) {
    const int per = sums >= 4000000 ? 4 : 1;
    launch_chained(per == 4 ? conv_silu_vec_kernel<4> : conv_silu_vec_kernel<1>,
                   dim3((n_tokens + per - 1) / per, (channels / 8 + 127) / 128), dim3(128), 0, (cudaStream_t)stream, (const elem_t*)proj,
                   ld, off, channels, (const elem_t*)weight, (const elem_t*)bias, conv_state, seq_of_token, seq_starts, state_slots,
                   (elem_t*)out, n_tokens);
    return check_launch("conv_silu");
  }
#endif
  launch_chained(conv_silu_kernel<elem_t>, dim3(n_tokens, n_tokens < 64 ? (channels + 255) / 256 : 1), dim3(256), 0, (cudaStream_t)stream, (const elem_t*)proj, ld, off,
                 channels, taps, (const elem_t*)weight, (const elem_t*)bias, conv_state, seq_of_token, seq_starts, state_slots,
                 (elem_t*)out);
  return check_launch("conv_silu");
}

ERB_EXPORT int erb_conv_state_update(const void* proj, int n_seqs, int ld, int off, int channels, int taps, float* conv_state,
                                     const int* seq_starts, const int* state_slots, void* stream) {
  if (n_seqs <= 0 || taps <= 1) return ERB_OK;
  launch_chained(conv_state_update_kernel<elem_t>, dim3(n_seqs, (channels + 255) / 256), dim3(256), 0, (cudaStream_t)stream, (const elem_t*)proj, ld,
                 off, channels, taps, conv_state, seq_starts, state_slots);
  return check_launch("conv_state_update");
}

ERB_EXPORT int erb_ssm_scan(const void* xbc, int channels, const void* proj, int ld, int off_dt, const float* dt_bias,
                            const float* a_log, const float* d_skip, float* state, const int* seq_starts,
                            const int* state_slots, float* y, int n_seqs, int n_tokens, int longest, int portions, int H, int P, int N, int G,
                            int* status, void* stream) {
  if (n_seqs <= 0) return ERB_OK;
  if (H <= 0 || P <= 0 || N <= 0 || G <= 0 || H % G || P > 512) return fail(ERB_ERR_ARG, "ssm_scan: bad sizes (columns of at most 512)");
  if (portions <= 0 || portions > n_seqs) portions = n_seqs;
  int most_tokens = INT_MAX;            // what the scan takes: every portion, or single tokens beside the chunk kernel's portions
#if ERB_ELEM == 1
  const bool fits = (N == 32 || N == 64 || N == 128) && P % kChunkCols == 0 && channels % 8 == 0 && !((uintptr_t)xbc & 15) &&
                    !((uintptr_t)state & 7) && !((uintptr_t)y & 7);
  int chunk = fits ? chunk_of(H * (P / kChunkCols), N, n_tokens, n_seqs, longest) : 0;
  if (chunk == kChunk && ((uintptr_t)y & 15)) chunk = kShortChunk;      // (its stores are of 8 bytes; the other's of 16 cost it a twentieth in two forms)
  if (chunk == kShortChunk) {
    const size_t bytes = N == 32 ? sizeof(ShortSmem<32>) : N == 64 ? sizeof(ShortSmem<64>) : sizeof(ShortSmem<128>);
    auto kern = N == 32 ? ssm_short_kernel<32> : N == 64 ? ssm_short_kernel<64> : ssm_short_kernel<128>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "ssm_scan: %s", cudaGetErrorString(e));
    launch_chained(kern, dim3(H, portions, P / kChunkCols), dim3((kShortWarps + 1) * 32), bytes, (cudaStream_t)stream, (const elem_t*)xbc, channels,
                   (const elem_t*)proj, ld, off_dt, dt_bias, a_log, d_skip, state, seq_starts, state_slots, y, H, P, G, n_seqs);
    const int rc = check_launch("ssm_short");
    if (rc || n_seqs == 1) return rc;
    most_tokens = 1;
    n_tokens = n_seqs;                  // (below: the shape for single tokens)
  } else if (chunk == kChunk) {
    constexpr size_t bytes = sizeof(ChunkSmem) + 1024;
    auto kern = N == 32 ? ssm_chunk_kernel<32> : N == 64 ? ssm_chunk_kernel<64> : ssm_chunk_kernel<128>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "ssm_scan: %s", cudaGetErrorString(e));
    CUtensorMap bc, x;
    int rc;
    if ((rc = rows_map(&bc, xbc, n_tokens, channels, channels, kChunk, "ssm_scan")) ||
        (rc = rows_map(&x, xbc, n_tokens, channels, channels, kChunk, "ssm_scan", kChunkCols)))
      return rc;
    launch_chained(kern, dim3(H, portions, P / kChunkCols), dim3(kChunkThreads), bytes, (cudaStream_t)stream, bc, x,
                   (const elem_t*)xbc, channels, (const elem_t*)proj, ld, off_dt, dt_bias, a_log, d_skip, state, seq_starts,
                   state_slots, y, H, P, G, n_seqs, status);
    rc = check_launch("ssm_chunk");
    if (rc || n_seqs == 1) return rc;
    most_tokens = 1;
    n_tokens = n_seqs;                  // (below: the shape for single tokens)
  }
#endif
  const int PB = P % 32 == 0 ? 32 : (P % 16 == 0 ? 16 : 0);
  // rows per thread: 16 for a step of single tokens (fewer, busier threads: the step is the state's read and write),
  // 8 where portions are walked and that still gives a block of at most 512 threads (twice the warps to hide a token's
  // dependent steps).  The two differ in the order in which a column's partial sums are added, that is by rounding.
  const int NLc = (n_tokens > n_seqs && N % 8 == 0 && (N / 8) * PB <= 512) ? 8 : 16;
  if (PB && N % NLc == 0 && (N / NLc) * PB <= 512) {
    const int L = N / NLc;
    const size_t smem16 = scan_smem(N, PB, L);
    auto kern = NLc == 8 ? ssm_scan16_kernel<elem_t, 8> : ssm_scan16_kernel<elem_t, 16>;
    if (smem16 > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem16);
      if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "ssm_scan: %s", cudaGetErrorString(e));
    }
    launch_chained(kern, dim3(H, n_seqs, P / PB), dim3(L * PB), smem16, (cudaStream_t)stream,
                   (const elem_t*)xbc, channels, (const elem_t*)proj, ld, off_dt, dt_bias, a_log, d_skip, state, seq_starts,
                   state_slots, y, H, P, N, G, PB, most_tokens);
    return check_launch("ssm_scan");
  }
  int L = 512 / P;                       // threads that share a column of the state
  if (L > 4) L = 4;
  if (L > N) L = N;
  int NL = (N + L - 1) / L;
  if (NL > 64) return fail(ERB_ERR_UNSUPPORTED, "ssm_scan: a state of %d rows with columns of %d (at most %d rows)", N, P, 64 * L);
  const size_t smem = sizeof(float) * ((size_t)kScanChunk * (2 * N + P + 2 + (size_t)L * P));
  if (smem > 200 * 1024) return fail(ERB_ERR_UNSUPPORTED, "ssm_scan: sizes need %zu bytes of shared memory", smem);
  auto kernel = NL <= 16 ? ssm_scan_kernel<elem_t, 16> : ssm_scan_kernel<elem_t, 64>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "ssm_scan: %s", cudaGetErrorString(e));
  }
  launch_chained(kernel, dim3(H, n_seqs), dim3(L * P), smem, (cudaStream_t)stream, (const elem_t*)xbc, channels,
                 (const elem_t*)proj, ld, off_dt, dt_bias, a_log, d_skip, state, seq_starts, state_slots, y, H, P, N, G, L, NL);
  return check_launch("ssm_scan");
}

ERB_EXPORT int erb_gated_group_norm(const void* x, int x_is_float, int x_ld, const void* gate, int gate_ld, const float* weight,
                                    void* out, int out_ld, int n_tokens, int width, int parts, float eps, void* stream) {
  if (n_tokens <= 0) return ERB_OK;
  if (width <= 0 || parts <= 0 || width % parts) return fail(ERB_ERR_ARG, "gated_group_norm: the parts must divide the width");
  const int per = width / parts, V = per / 128;
  const uintptr_t elem_bits = 4 * sizeof(elem_t) - 1, x_bits = x_is_float ? 15 : elem_bits;
  if (per % 128 == 0 && (V == 1 || V == 2 || V == 4 || V == 8) && x_ld % 4 == 0 && out_ld % 4 == 0 && (!gate || gate_ld % 4 == 0) &&
      !(((uintptr_t)gate | (uintptr_t)out) & elem_bits) && !((uintptr_t)x & x_bits) && !((uintptr_t)weight & 15) &&
      (long long)n_tokens * parts <= 0x7fffffffLL) {
    const int n_items = n_tokens * parts;
#define ERB_GROUP_NORM(X32, VV)                                                                                            \
  launch_chained(gated_group_norm_vec_kernel<elem_t, X32, VV>, dim3((n_items + 3) / 4), dim3(128), 0, (cudaStream_t)stream, x, x_ld, \
                 (const elem_t*)gate, gate_ld, weight, (elem_t*)out, out_ld, n_items, parts, eps)
    if (x_is_float) { if (V == 1) ERB_GROUP_NORM(true, 1); else if (V == 2) ERB_GROUP_NORM(true, 2); else if (V == 4) ERB_GROUP_NORM(true, 4); else ERB_GROUP_NORM(true, 8); }
    else { if (V == 1) ERB_GROUP_NORM(false, 1); else if (V == 2) ERB_GROUP_NORM(false, 2); else if (V == 4) ERB_GROUP_NORM(false, 4); else ERB_GROUP_NORM(false, 8); }
#undef ERB_GROUP_NORM
    return check_launch("gated_group_norm");
  }
  if (x_is_float)
    launch_chained(gated_group_norm_kernel<elem_t, true>, dim3(n_tokens, parts), dim3(256), 0, (cudaStream_t)stream, x, x_ld,
                   (const elem_t*)gate, gate_ld, weight, (elem_t*)out, out_ld, width, parts, eps);
  else
    launch_chained(gated_group_norm_kernel<elem_t, false>, dim3(n_tokens, parts), dim3(256), 0, (cudaStream_t)stream, x, x_ld,
                   (const elem_t*)gate, gate_ld, weight, (elem_t*)out, out_ld, width, parts, eps);
  return check_launch("gated_group_norm");
}

// taps 0: no convolution; otherwise `weight` float [taps][channels] and, for taps > 1, the records `conv_state`.
// Sequences before `first_portion` bring one token each.
ERB_EXPORT int erb_qkv_conv(const void* proj, int ld, const float* bias, const float* weight, int taps, float* conv_state,
                            const int* seq_of_token, const int* seq_starts, const int* state_slots, const int* slots, void* q_out,
                            void* k_pages, void* v_pages, int n_tokens, int n_seqs, int first_portion, int nq, int nkv, int D,
                            int page_size, void* stream) {
  if (n_tokens <= 0) return ERB_OK;
  const int channels = (nq + 2 * nkv) * D;
  if (nq <= 0 || nkv <= 0 || D <= 0 || D % 4 || ld % 4 || ld < channels || taps < 0 || page_size <= 0 || (taps > 0 && !weight) ||
      (taps > 1 && !conv_state) || (slots && (!k_pages || !v_pages)))
    return fail(ERB_ERR_ARG, "qkv_conv: bad sizes (heads of %d, rows of %d) or missing tensors", D, ld);
  const int y = (channels / 4 + 127) / 128;
  launch_chained(qkv_conv_kernel<elem_t>, dim3(n_tokens, y), dim3(128), 0, (cudaStream_t)stream, (const elem_t*)proj, ld, bias, weight,
                 taps, conv_state, seq_of_token, seq_starts, state_slots, slots, (elem_t*)q_out, (elem_t*)k_pages, (elem_t*)v_pages,
                 nq, nkv, D, page_size);
  int rc = check_launch("qkv_conv");
  if (rc || taps <= 1 || n_seqs <= first_portion) return rc;
  launch_chained(qkv_conv_state_kernel<elem_t>, dim3(n_seqs - first_portion, y), dim3(128), 0, (cudaStream_t)stream,
                 (const elem_t*)proj, ld, bias, taps, conv_state, seq_starts, state_slots, first_portion, channels);
  return check_launch("qkv_conv_state");
}
