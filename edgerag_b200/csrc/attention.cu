// Causal grouped-query attention over cache pages, for any element type and head size.
//
// These are the general kernels: CUDA-core arithmetic in float, any head size that is a multiple
// of 8 up to 128 or of 16 up to 256, any page size, any number of heads and groups, an optional window.  They serve
// the 32-bit path and every shape the tensor-core kernels do not take.
//
// Cache layout (one layer): pages[page][kv head][offset][D]; a token at logical position p of a
// sequence lives in page block_table[seq][p / page_size] at offset p % page_size.  Keys are
// stored already rotated.  A query at position p sees keys max(0, p - window + 1) .. p
// (window <= 0: all keys 0 .. p) and, with a window, also the keys 0 .. keep_first - 1 whatever their
// distance.  A negative `window` stands for a mask of chunks: the query sees the keys from the start of its own run of
// -window positions (runs counted from position 0 of the sequence) up to itself.  Query head h reads kv head h / (nq / nkv).
// With `penalty` (float [2][nq]: r1 of every query head, then r2) the scaled score of a key d positions back is lowered by
// r1 * ln(1 + r2 * d).  With `softcap` c > 0 the scaled score s becomes c * tanh(s / c); a launch takes one of the two.
// With `gate` (rows of nq * D entries, `gate_stride` apart, row t for output row t) every output entry is multiplied by the
// sigmoid of its entry of the gate before it is rounded.
//
// Both kernels give every thread its own keys and its own online-softmax state (running max,
// denominator, float accumulator of D values), so the inner loop has no cross-thread traffic;
// states are merged once at the end, in a fixed order.
#include <mutex>

#include "common.cuh"

using namespace erb;

ERB_DEFINE_LAST_ERROR(erb_last_error)

namespace {

template <typename T> struct Vec;  // 16-byte vectors
template <> struct Vec<float> { static constexpr int N = 4; };
template <> struct Vec<__nv_bfloat16> { static constexpr int N = 8; };

template <typename T, int N>
__device__ __forceinline__ void load_vec(const T* p, float* out);
template <>
__device__ __forceinline__ void load_vec<float, 4>(const float* p, float* out) { load4(p, out); }
template <>
__device__ __forceinline__ void load_vec<__nv_bfloat16, 8>(const __nv_bfloat16* p, float* out) { load8(p, out); }

// One thread's online-softmax state over the keys it visits.
template <int D>
struct LaneState {
  float m = -INFINITY, l = 0.f;
  float acc[D];
  __device__ __forceinline__ void init() {
#pragma unroll
    for (int d = 0; d < D; ++d) acc[d] = 0.f;
  }
  // Visit one key: k and v point at the D elements of the key and the value row.
  template <typename T>
  __device__ __forceinline__ void visit(const float* q_smem, const T* k, const T* v, float scale, float lower, float softcap) {
    constexpr int N = Vec<T>::N;
    float s = 0.f;
#pragma unroll
    for (int d0 = 0; d0 < D; d0 += N) {
      float kk[N];
      load_vec<T, N>(k + d0, kk);
#pragma unroll
      for (int i = 0; i < N; ++i) s = fmaf(q_smem[d0 + i], kk[i], s);
    }
    s = fmaf(s, scale, -lower);
    if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    float p;
    if (s > m) {
      const float alpha = expf(m - s);  // exp(-inf) = 0 on the first key
      l *= alpha;
#pragma unroll
      for (int d = 0; d < D; ++d) acc[d] *= alpha;
      m = s;
      p = 1.f;
    } else {
      p = expf(s - m);
    }
    l += p;
#pragma unroll
    for (int d0 = 0; d0 < D; d0 += N) {
      float vv[N];
      load_vec<T, N>(v + d0, vv);
#pragma unroll
      for (int i = 0; i < N; ++i) acc[d0 + i] = fmaf(p, vv[i], acc[d0 + i]);
    }
  }
};

// Merge the 32 states of a warp.  `stage` is the warp's shared area of 32 * (D + 1) floats.
// Afterwards lane x holds, for each i with d = x + 32 i < D, the warp's sum for column d in
// out[i]; the warp's max and denominator are returned in m_w / l_w (same on every lane).
template <int D>
__device__ __forceinline__ void warp_merge(LaneState<D>& st, float* stage, float& m_w, float& l_w,
                                           float* out /* (D + 31) / 32 */) {
  const int lane = threadIdx.x & 31;
  m_w = warp_max(st.m);
  const float f = (st.m == -INFINITY) ? 0.f : expf(st.m - m_w);
  l_w = warp_sum(st.l * f);
  float* mine = stage + lane * (D + 1);
#pragma unroll
  for (int d = 0; d < D; ++d) mine[d] = st.acc[d] * f;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < (D + 31) / 32; ++i) {
    const int d = lane + 32 * i;
    float sum = 0.f;
    if (d < D) {
#pragma unroll 8
      for (int j = 0; j < 32; ++j) sum += stage[j * (D + 1) + d];
    }
    out[i] = sum;
  }
  __syncwarp();
}

// What a head's distance penalty takes off the score of a key `dist` positions back (no penalty: 0).
struct Penalty {
  float r1 = 0.f, r2 = 0.f;
  __device__ __forceinline__ Penalty(const float* table, int head, int n_heads) {
    if (table) { r1 = table[head]; r2 = table[n_heads + head]; }
  }
  __device__ __forceinline__ float at(int dist) const { return r1 != 0.f ? r1 * log1pf(r2 * (float)dist) : 0.f; }
};

constexpr int kRowWarps = 4;  // warps (query rows) per block in the row kernel

// ---------------------------------------------------------------------------------------------
// Row kernel: one warp per (query token, query head).  Handles portions of prompts and decoded
// tokens alike; the only per-token inputs are its sequence and its position.
// ---------------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(kRowWarps * 32)
attention_rows_kernel(const T* __restrict__ q, int q_row_stride, const T* __restrict__ k_pages,
                      const T* __restrict__ v_pages, const int* __restrict__ block_tables, int max_pages,
                      const int* __restrict__ seq_of_token, const int* __restrict__ positions,
                      T* __restrict__ out, int out_row_stride, int n_tokens, int nq, int nkv,
                      int page_size, int window, int keep_first, float scale, const float* __restrict__ penalty, float softcap,
                      const T* __restrict__ gate, int gate_stride) {
  chain_wait();
  extern __shared__ float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* q_s = smem + warp * D;
  float* stage = smem + kRowWarps * D + warp * 32 * (D + 1);
  const int t = blockIdx.x * kRowWarps + warp;
  const int h = blockIdx.y;
  if (t >= n_tokens) return;  // warps are independent: no block-wide barrier below
  const T* q_row = q + (size_t)t * q_row_stride + (size_t)h * D;
  for (int d = lane; d < D; d += 32) q_s[d] = Elem<T>::load(q_row + d);
  __syncwarp();

  const int seq = seq_of_token[t], pos = positions[t];
  const int kvh = h / (nq / nkv);
  const int* bt = block_tables + (size_t)seq * max_pages;
  const int k_lo = first_visible_key(pos, window);

  LaneState<D> st;
  st.init();
  const Penalty pen(penalty, h, nq);
  const int kept = min(keep_first, k_lo);     // the first keys that the window would hide
  for (int k = lane; k < kept; k += 32) {
    const int page = bt[k / page_size];
    const size_t row = (((size_t)page * nkv + kvh) * page_size + (k % page_size)) * D;
    st.template visit<T>(q_s, k_pages + row, v_pages + row, scale, pen.at(pos - k), softcap);
  }
  for (int k = k_lo + lane; k <= pos; k += 32) {
    const int page = bt[k / page_size];
    const size_t row = (((size_t)page * nkv + kvh) * page_size + (k % page_size)) * D;
    st.template visit<T>(q_s, k_pages + row, v_pages + row, scale, pen.at(pos - k), softcap);
  }
  float m_w, l_w, o[(D + 31) / 32];
  warp_merge<D>(st, stage, m_w, l_w, o);
  const float inv = 1.f / l_w;
  T* o_row = out + (size_t)t * out_row_stride + (size_t)h * D;
#pragma unroll
  for (int i = 0; i < (D + 31) / 32; ++i) {
    const int d = lane + 32 * i;
    if (d < D) Elem<T>::store(o_row + d, gate ? sigmoid_mul(o[i] * inv, Elem<T>::load(gate + (size_t)t * gate_stride + h * D + d)) : o[i] * inv);
  }
}

#if ERB_ELEM == 0
// ---------------------------------------------------------------------------------------------
// Portions of prompts in 32 bits: a block takes 32 neighbouring tokens of one head and walks the keys in tiles of 64 that it copies
// to shared memory once for all of them (the row kernel above lets every lane fetch keys of its own, row after row).  A
// thread owns two rows: with 15 others it makes their 128 scores of a tile (keys tx, tx + 16, ...), takes the rows' maximum, and
// adds P V for four columns (eight of heads of 128); P passes through shared memory within the half-warp.  P V is summed 32 keys at a
// time and then onto the accumulator, so that its rounding is no worse than that of the row kernel's 32 partial sums.
// Tiles start at absolute multiples of 64 positions, and a tile that a row does not see changes nothing of it: a row's
// result does not depend on the other tokens.  Tokens of several sequences in a block are taken one sequence after the other.
// The even tiles and the odd ones (counted from position 0) are walked apart, and the two maxima, sums and accumulators are put together at
// the end in that order, so that a row's result depends on nothing but its own keys.  A block has two groups of 256 threads, each with
// buffers of its own, for the two halves, or one group, which walks one after the other: the same bits.  One group, two blocks an SM, where
// there are many blocks, or more than SMs with walks so short that one of two groups would often stand idle (the caller counts; 32 heads, one
// group | two: 16 portions of 32 tokens 21.4 | 31.1 us, 2 of 333 89 | 98, 2,048 tokens 926 | 1,008).
// Bound by the reads of shared memory and the multiplications, about alike, and for few blocks by a tile's chain (5 us), which is why
// there are two groups.  9 heads of 64 over 3 kv heads, row kernel | one group | two: 333 tokens 94 | 31 | 26 us, 96 tokens 15 | 13.5 | 11.1,
// 333 behind 7,000 2,896 | 613 | 459, 2,048 tokens 2,354 | 345 | 329; 8 heads of 128, 333 behind 100 246 | 69 | 56.  (Four groups of 128 threads
// with four rows each: 2,048 tokens 276, but 16 portions of 32 tokens 12.8 instead of 8.5.)
// ---------------------------------------------------------------------------------------------
constexpr int kTileRows = 32, kTileKeys = 64, kTileThreads = 256, kTileParts = 2;       // (threads of a group; even and odd tiles)
template <int D> __host__ __device__ constexpr int tile_group_floats() { return 2 * kTileKeys * (D + 4) + kTileRows * (kTileKeys + 4); }
template <int D> __host__ __device__ constexpr int tile_part_floats() { return 2 * (2 + 4 * (D / 64)) + 1; }      // of a thread, odd: no bank conflicts
template <int D, int GROUPS> constexpr size_t tile_smem() {
  return sizeof(float) * (kTileRows * (D + 4) + GROUPS * tile_group_floats<D>() + (GROUPS == 1 ? kTileThreads * tile_part_floats<D>() : 0));
}

template <int D, int GROUPS>
__global__ void __launch_bounds__(GROUPS * kTileThreads, kTileParts / GROUPS)
attention_tile_kernel(const float* __restrict__ q, int q_row_stride, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                      const int* __restrict__ block_tables, int max_pages, const int* __restrict__ seq_of_token,
                      const int* __restrict__ positions, float* __restrict__ out, int out_row_stride, int n_tokens, int nq, int nkv,
                      int page_size, int window, int keep_first, float scale, const float* __restrict__ penalty, float softcap,
                      const float* __restrict__ gate, int gate_stride) {
  chain_wait();
  constexpr int LD = D + 4, LP = kTileKeys + 4, kGroups = D / 64;
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;                             // [kTileRows][LD]
  const int group = threadIdx.x / kTileThreads;
  float* k_s = q_s + kTileRows * LD + group * tile_group_floats<D>();       // [kTileKeys][LD]
  float* v_s = k_s + kTileKeys * LD;
  float* p_s = v_s + kTileKeys * LD;             // [kTileRows][LP]
  const int t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * kTileRows, n_here = min(kTileRows, n_tokens - t0);   // (the longest walks first)
  const int h = blockIdx.y, kvh = h / (nq / nkv);
  const int tid = threadIdx.x % kTileThreads, lane = tid & 31, tx = tid & 15, r0 = 2 * (tid >> 4);
  for (int i = threadIdx.x; i < kTileRows * D; i += GROUPS * kTileThreads) {
    const int r = i / D, d = i % D;
    q_s[r * LD + d] = r < n_here ? q[(size_t)(t0 + r) * q_row_stride + (size_t)h * D + d] : 0.f;
  }
  // lane r of every warp knows row r
  const int t_lane = t0 + min(lane, n_here - 1);
  const int seq_l = seq_of_token[t_lane], pos_l = positions[t_lane], lo_l = first_visible_key(pos_l, window);
  const int pos0 = __shfl_sync(0xffffffffu, pos_l, r0), pos1 = __shfl_sync(0xffffffffu, pos_l, r0 + 1);
  const int lo0 = __shfl_sync(0xffffffffu, lo_l, r0), lo1 = __shfl_sync(0xffffffffu, lo_l, r0 + 1);
  const Penalty pen(penalty, h, nq);
  const int page_shift = (page_size & (page_size - 1)) == 0 ? __ffs(page_size) - 1 : -1;
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kTileThreads) : "memory"); };
  __syncthreads();                               // (q is there)

  for (int begin = 0, end; begin < n_here; begin = end) {          // runs of one sequence
    const int seq = __shfl_sync(0xffffffffu, seq_l, begin);
    const unsigned other = __ballot_sync(0xffffffffu, lane >= begin && (lane >= n_here || seq_l != seq));
    end = other ? __ffs(other) - 1 : kTileRows;
    const bool in = lane >= begin && lane < end;
    const int hi = __reduce_max_sync(0xffffffffu, in ? pos_l : INT_MIN), pos_min = __reduce_min_sync(0xffffffffu, in ? pos_l : INT_MAX);
    const int lo = __reduce_min_sync(0xffffffffu, in ? lo_l : INT_MAX), lo_max = __reduce_max_sync(0xffffffffu, in ? lo_l : INT_MIN);
    const int* bt = block_tables + (size_t)seq * max_pages;
    float m[2], l[2], acc[2][4 * kGroups];
    // where a thread leaves what the odd tiles gave: of two groups the second one's buffers, whose tiles are done with by then
    float* odd = q_s + kTileRows * LD + tile_group_floats<D>() + tid * tile_part_floats<D>();
    auto leave = [&]() {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        odd[i] = m[i];
        odd[2 + i] = l[i];
#pragma unroll
        for (int c = 0; c < 4 * kGroups; ++c) odd[4 + 4 * kGroups * i + c] = acc[i][c];
      }
    };
#pragma unroll 1
    for (int walk = GROUPS == 1 ? kTileParts - 1 : group; walk >= (GROUPS == 1 ? 0 : group); --walk) {
#pragma unroll
      for (int i = 0; i < 2; ++i) { m[i] = -INFINITY; l[i] = 0.f; }
#pragma unroll
      for (int i = 0; i < 4 * kGroups; ++i) acc[0][i] = acc[1][i] = 0.f;
      for (int j = 0; j * kTileKeys <= hi; ++j) {
        if (j * kTileKeys >= keep_first) j = max(j, lo / kTileKeys);         // past the kept first keys: on to the first that a row sees
        if (j % kTileParts != walk) continue;
        const int k0 = j * kTileKeys;
        group_sync();                                                         // (the tile before is done with)
        constexpr int kRowsAtOnce = 4 * kTileThreads / D, kBatch = 4;       // rows that the group's threads copy at a time
        const int r_own = tid / (D / 4), c = 4 * (tid % (D / 4));
#pragma unroll
        for (int first = 0; first < kTileKeys; first += kRowsAtOnce * kBatch) {
          int page[kBatch];                        // (the loads of several rows under way at once: their pages, then keys and values)
          float4 kv[kBatch], vv[kBatch];
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            const int k = k0 + first + i * kRowsAtOnce + r_own;
            page[i] = k <= hi ? bt[page_shift >= 0 ? k >> page_shift : k / page_size] : -1;
          }
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            const int k = k0 + first + i * kRowsAtOnce + r_own;
            kv[i] = vv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (page[i] >= 0) {
              const size_t row = (((size_t)page[i] * nkv + kvh) * page_size + (page_shift >= 0 ? k & (page_size - 1) : k % page_size)) * D + c;
              kv[i] = *reinterpret_cast<const float4*>(k_pages + row);
              vv[i] = *reinterpret_cast<const float4*>(v_pages + row);
            }
          }
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            const int r = first + i * kRowsAtOnce + r_own;
            *reinterpret_cast<float4*>(k_s + r * LD + c) = kv[i];
            *reinterpret_cast<float4*>(v_s + r * LD + c) = vv[i];
          }
        }
        group_sync();
        const bool whole = k0 + kTileKeys - 1 <= pos_min && (k0 >= lo_max || k0 + kTileKeys <= keep_first);    // every row sees every key
        float s[2][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) s[0][u] = s[1][u] = 0.f;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
          const float4 a = *reinterpret_cast<const float4*>(q_s + r0 * LD + d), b = *reinterpret_cast<const float4*>(q_s + (r0 + 1) * LD + d);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 k4 = *reinterpret_cast<const float4*>(k_s + (tx + 16 * u) * LD + d);
            s[0][u] = fmaf(a.x, k4.x, s[0][u]); s[0][u] = fmaf(a.y, k4.y, s[0][u]); s[0][u] = fmaf(a.z, k4.z, s[0][u]); s[0][u] = fmaf(a.w, k4.w, s[0][u]);
            s[1][u] = fmaf(b.x, k4.x, s[1][u]); s[1][u] = fmaf(b.y, k4.y, s[1][u]); s[1][u] = fmaf(b.z, k4.z, s[1][u]); s[1][u] = fmaf(b.w, k4.w, s[1][u]);
          }
        }
        float alpha[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int pos = i ? pos1 : pos0, first = i ? lo1 : lo0;
          bool seen[4];
          float top = m[i];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = k0 + tx + 16 * u;
            seen[u] = whole || (k <= pos && (k >= first || k < keep_first));
            float v = fmaf(s[i][u], scale, -pen.at(seen[u] ? pos - k : 0));
            if (softcap > 0.f) v = softcap * tanhf(v / softcap);
            s[i][u] = v;
            if (seen[u]) top = fmaxf(top, v);
          }
#pragma unroll
          for (int o = 8; o; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
          alpha[i] = m[i] == top ? 1.f : expf(m[i] - top);
          m[i] = top;
          const float ref = top == -INFINITY ? 0.f : top;
          float sum = 0.f;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float p = s[i][u] == ref ? 1.f : expf(s[i][u] - ref);
            if (seen[u]) sum += p;
            p_s[(r0 + i) * LP + tx + 16 * u] = seen[u] ? p : -1.f;           // (below 0: not seen, whatever its value holds)
          }
          l[i] = l[i] * alpha[i] + sum;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4 * kGroups; ++i) { acc[0][i] *= alpha[0]; acc[1][i] *= alpha[1]; }
        auto products = [&](auto masked) {
#pragma unroll 1
          for (int k1 = 0; k1 < kTileKeys; k1 += 32) {
            float part[2][4 * kGroups];
#pragma unroll
            for (int i = 0; i < 4 * kGroups; ++i) part[0][i] = part[1][i] = 0.f;
#pragma unroll 2
            for (int k = k1; k < k1 + 32; k += 4) {
              float p[2][4];
              *reinterpret_cast<float4*>(p[0]) = *reinterpret_cast<const float4*>(p_s + r0 * LP + k);
              *reinterpret_cast<float4*>(p[1]) = *reinterpret_cast<const float4*>(p_s + (r0 + 1) * LP + k);
#pragma unroll
              for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int g = 0; g < kGroups; ++g) {
                  float v[4];
                  *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(v_s + (k + u) * LD + 64 * g + 4 * tx);
#pragma unroll
                  for (int i = 0; i < 2; ++i) {
                    if (decltype(masked)::value && p[i][u] < 0.f) continue;
#pragma unroll
                    for (int c = 0; c < 4; ++c) part[i][4 * g + c] = fmaf(p[i][u], v[c], part[i][4 * g + c]);
                  }
                }
            }
#pragma unroll
            for (int i = 0; i < 4 * kGroups; ++i) { acc[0][i] += part[0][i]; acc[1][i] += part[1][i]; }
          }
        };
        if (whole) products(std::false_type{}); else products(std::true_type{});
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int o = 8; o; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
      if (GROUPS == 1 && walk > 0) leave();
    }
    if (GROUPS > 1) {
      __syncthreads();                           // (the tiles are done with)
      if (group > 0) leave();
      __syncthreads();
    }
    if (group == 0) {                            // both parts of these rows
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float top = fmaxf(m[i], odd[i]), ref = top == -INFINITY ? 0.f : top;
        // (a maximum of +inf is its own: its part's sum holds such keys with weight 1)
        const float f0 = m[i] == top ? 1.f : expf(m[i] - ref);
        l[i] *= f0;
#pragma unroll
        for (int c = 0; c < 4 * kGroups; ++c) acc[i][c] *= f0;
        if (odd[i] == -INFINITY && odd[2 + i] == 0.f) continue;            // (saw no key of this row)
        const float f = odd[i] == top ? 1.f : expf(odd[i] - ref);
        l[i] = fmaf(odd[2 + i], f, l[i]);
#pragma unroll
        for (int c = 0; c < 4 * kGroups; ++c) acc[i][c] = fmaf(odd[4 + 4 * kGroups * i + c], f, acc[i][c]);
      }
    }
    if (GROUPS > 1) __syncthreads();             // (the next run's tiles come into that room)
    if (group > 0) continue;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = r0 + i, t = t0 + r;
      if (r < begin || r >= end) continue;
      const float inv = 1.f / l[i];
#pragma unroll
      for (int g = 0; g < kGroups; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int d = 64 * g + 4 * tx + c;
          const float v = acc[i][4 * g + c] * inv;
          out[(size_t)t * out_row_stride + (size_t)h * D + d] = gate ? sigmoid_mul(v, gate[(size_t)t * gate_stride + h * D + d]) : v;
        }
    }
  }
}

template <int D, int GROUPS>
int launch_tiles(const void* q, int q_row_stride, const void* k_pages, const void* v_pages, const int* block_tables, int max_pages,
                 const int* seq_of_token, const int* positions, void* out, int out_row_stride, int n_tokens, int nq, int nkv, int page_size,
                 int window, int keep_first, float scale, const float* penalty, float softcap, const void* gate, int gate_stride,
                 cudaStream_t s) {
  const dim3 grid((n_tokens + kTileRows - 1) / kTileRows, nq);
  auto kern = attention_tile_kernel<D, GROUPS>;
  constexpr size_t smem = tile_smem<D, GROUPS>();
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "attention_rows: %s", cudaGetErrorString(e));
  launch_chained(kern, grid, dim3(GROUPS * kTileThreads), smem, s, (const float*)q, q_row_stride,
                 (const float*)k_pages, (const float*)v_pages, block_tables, max_pages, seq_of_token, positions, (float*)out, out_row_stride,
                 n_tokens, nq, nkv, page_size, window, keep_first, scale, penalty, softcap, (const float*)gate, gate_stride);
  return check_launch("attention_tile");
}
#endif

// ---------------------------------------------------------------------------------------------
// Decode kernel: one query token per sequence; the keys of a sequence are cut into splits of
// `split_keys` keys, one block per (split, query head, sequence).  Partial results (max,
// denominator, unnormalised accumulator) go to scratch; the combine kernel merges the splits in
// order.  The split size is a constant of the launch, so a sequence's result does not depend on
// what else is in the batch.
// ---------------------------------------------------------------------------------------------
constexpr int kDecodeWarps = 4;

template <typename T, int D>
__global__ void __launch_bounds__(kDecodeWarps * 32)
attention_decode_split_kernel(const T* __restrict__ q, int q_row_stride, const T* __restrict__ k_pages,
                              const T* __restrict__ v_pages, const int* __restrict__ block_tables,
                              int max_pages, const int* __restrict__ token_of_seq,
                              const int* __restrict__ positions, float* __restrict__ part_acc,
                              float* __restrict__ part_ml, int max_splits, int nq, int nkv, int page_size,
                              int window, int keep_first, int split_keys, float scale, const float* __restrict__ penalty,
                              float softcap) {
  chain_wait();
  extern __shared__ float smem[];
  float* q_s = smem;                                   // D
  float* stage = smem + D;                             // kDecodeWarps * 32 * (D + 1)
  float* warp_out = stage + kDecodeWarps * 32 * (D + 1);  // kDecodeWarps * (D + 2)
  const int split = blockIdx.x, h = blockIdx.y, seq = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = token_of_seq[seq];
  const int pos = positions[t];
  const int k_lo = first_visible_key(pos, window);
  // Splits are aligned to multiples of split_keys in absolute key positions.
  const int first_split = k_lo / split_keys;
  const int begin = max(k_lo, (first_split + split) * split_keys);
  const int end = min(pos + 1, (first_split + split + 1) * split_keys);
  if (begin >= end) return;  // this split does not exist for this sequence
  const int kept = split == 0 ? min(keep_first, k_lo) : 0;   // the first split also takes the keys kept before the window

  const T* q_row = q + (size_t)t * q_row_stride + (size_t)h * D;
  for (int d = threadIdx.x; d < D; d += blockDim.x) q_s[d] = Elem<T>::load(q_row + d);
  __syncthreads();

  const int kvh = h / (nq / nkv);
  const int* bt = block_tables + (size_t)seq * max_pages;
  LaneState<D> st;
  st.init();
  const Penalty pen(penalty, h, nq);
  for (int k = (int)threadIdx.x; k < kept; k += kDecodeWarps * 32) {
    const int page = bt[k / page_size];
    const size_t row = (((size_t)page * nkv + kvh) * page_size + (k % page_size)) * D;
    st.template visit<T>(q_s, k_pages + row, v_pages + row, scale, pen.at(pos - k), softcap);
  }
  for (int k = begin + (int)threadIdx.x; k < end; k += kDecodeWarps * 32) {
    const int page = bt[k / page_size];
    const size_t row = (((size_t)page * nkv + kvh) * page_size + (k % page_size)) * D;
    st.template visit<T>(q_s, k_pages + row, v_pages + row, scale, pen.at(pos - k), softcap);
  }
  float m_w, l_w, o[(D + 31) / 32];
  warp_merge<D>(st, stage + warp * 32 * (D + 1), m_w, l_w, o);
  float* wo = warp_out + warp * (D + 2);
#pragma unroll
  for (int i = 0; i < (D + 31) / 32; ++i) {
    const int d = lane + 32 * i;
    if (d < D) wo[d] = o[i];
  }
  if (lane == 0) { wo[D] = m_w; wo[D + 1] = l_w; }
  __syncthreads();
  // Merge the warps in order.
  float m_b = -INFINITY;
#pragma unroll
  for (int w = 0; w < kDecodeWarps; ++w) m_b = fmaxf(m_b, warp_out[w * (D + 2) + D]);
  const size_t slot = ((size_t)seq * nq + h) * max_splits + split;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kDecodeWarps; ++w) {
      const float mw = warp_out[w * (D + 2) + D];
      const float f = (mw == -INFINITY) ? 0.f : expf(mw - m_b);
      sum += warp_out[w * (D + 2) + d] * f;
    }
    part_acc[slot * D + d] = sum;
  }
  if (threadIdx.x == 0) {
    float l_b = 0.f;
#pragma unroll
    for (int w = 0; w < kDecodeWarps; ++w) {
      const float mw = warp_out[w * (D + 2) + D];
      const float f = (mw == -INFINITY) ? 0.f : expf(mw - m_b);
      l_b += warp_out[w * (D + 2) + D + 1] * f;
    }
    part_ml[slot * 2] = m_b;
    part_ml[slot * 2 + 1] = l_b;
  }
}

template <typename T>
__global__ void attention_decode_combine_kernel(const float* __restrict__ part_acc,
                                                const float* __restrict__ part_ml,
                                                const int* __restrict__ token_of_seq,
                                                const int* __restrict__ positions, T* __restrict__ out,
                                                int out_row_stride, int max_splits, int nq, int head_dim,
                                                int window, int split_keys, const T* __restrict__ gate, int gate_stride) {
  chain_wait();
  const int h = blockIdx.x, seq = blockIdx.y;
  const int t = token_of_seq[seq];
  const int pos = positions[t];
  const int k_lo = first_visible_key(pos, window);
  // never beyond what the split kernel's grid wrote (a caller that understates max_splits gets the
  // first max_splits splits merged, not its neighbours' scratch)
  const int n_splits = min(pos / split_keys - k_lo / split_keys + 1, max_splits);
  const size_t base = ((size_t)seq * nq + h) * max_splits;
  float m = -INFINITY;
  for (int s = 0; s < n_splits; ++s) m = fmaxf(m, part_ml[(base + s) * 2]);
  float l = 0.f;
  for (int s = 0; s < n_splits; ++s) l += part_ml[(base + s) * 2 + 1] * expf(part_ml[(base + s) * 2] - m);
  const float inv = 1.f / l;
  T* o_row = out + (size_t)t * out_row_stride + (size_t)h * head_dim;
  for (int d = threadIdx.x; d < head_dim; d += blockDim.x) {
    float sum = 0.f;
    for (int s = 0; s < n_splits; ++s)
      sum += part_acc[(base + s) * head_dim + d] * expf(part_ml[(base + s) * 2] - m);
    Elem<T>::store(o_row + d, gate ? sigmoid_mul(sum * inv, Elem<T>::load(gate + (size_t)t * gate_stride + h * head_dim + d)) : sum * inv);
  }
}

template <typename T, int D>
int launch_rows(const void* q, int q_row_stride, const void* k_pages, const void* v_pages,
                const int* block_tables, int max_pages, const int* seq_of_token, const int* positions,
                void* out, int out_row_stride, int n_tokens, int nq, int nkv, int page_size, int window,
                int keep_first, float scale, const float* penalty, float softcap, const void* gate, int gate_stride, cudaStream_t s) {
  const size_t smem = (size_t)(kRowWarps * D + kRowWarps * 32 * (D + 1)) * sizeof(float);
  auto kern = attention_rows_kernel<T, D>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "attention_rows: %s", cudaGetErrorString(e));
  }
  dim3 grid((n_tokens + kRowWarps - 1) / kRowWarps, nq);
  launch_chained(kern, dim3(grid), dim3(kRowWarps * 32), smem, s, (const T*)q, q_row_stride, (const T*)k_pages, (const T*)v_pages,
      block_tables, max_pages, seq_of_token, positions, (T*)out, out_row_stride, n_tokens, nq, nkv,
      page_size, window, keep_first, scale, penalty, softcap, (const T*)gate, gate_stride);
  return check_launch("attention_rows");
}

template <typename T, int D>
int launch_decode(const void* q, int q_row_stride, const void* k_pages, const void* v_pages,
                  const int* block_tables, int max_pages, const int* token_of_seq, const int* positions,
                  void* out, int out_row_stride, float* part_acc, float* part_ml, int max_splits, int n_seqs,
                  int nq, int nkv, int page_size, int window, int keep_first, int split_keys, float scale, const float* penalty,
                  float softcap, const void* gate, int gate_stride, cudaStream_t s) {
  const size_t smem =
      (size_t)(D + kDecodeWarps * 32 * (D + 1) + kDecodeWarps * (D + 2)) * sizeof(float);
  auto kern = attention_decode_split_kernel<T, D>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "attention_decode: %s", cudaGetErrorString(e));
  }
  dim3 grid(max_splits, nq, n_seqs);
  launch_chained(kern, dim3(grid), dim3(kDecodeWarps * 32), smem, s, (const T*)q, q_row_stride, (const T*)k_pages,
      (const T*)v_pages, block_tables, max_pages, token_of_seq, positions, part_acc, part_ml, max_splits,
      nq, nkv, page_size, window, keep_first, split_keys, scale, penalty, softcap);
  int rc = check_launch("attention_decode_split");
  if (rc) return rc;
  launch_chained(attention_decode_combine_kernel<T>, dim3(dim3(nq, n_seqs)), dim3(64), 0, s, part_acc, part_ml, token_of_seq,
      positions, (T*)out, out_row_stride, max_splits, nq, D, window, split_keys, (const T*)gate, gate_stride);
  return check_launch("attention_decode_combine");
}

int check_common(const char* who, int nq, int nkv, int head_dim, int page_size, int max_pages) {
  if (nq <= 0 || nkv <= 0 || nq % nkv) return fail(ERB_ERR_ARG, "%s: %d query heads / %d kv heads", who, nq, nkv);
  if (head_dim < 8 || head_dim > 256 || (head_dim <= 128 ? head_dim % 8 : head_dim % 16))
    return fail(ERB_ERR_UNSUPPORTED, "%s: head_dim %d is not a multiple of 8 up to 128 or of 16 up to 256", who, head_dim);
  if (page_size <= 0 || max_pages <= 0) return fail(ERB_ERR_ARG, "%s: bad page_size/max_pages", who);
  return ERB_OK;
}

}  // namespace

#define ERB_DISPATCH_D(FN, ...)                                                                \
  switch (head_dim) {                                                                          \
    case 8: return FN<elem_t, 8>(__VA_ARGS__);     case 24: return FN<elem_t, 24>(__VA_ARGS__);   \
    case 40: return FN<elem_t, 40>(__VA_ARGS__);   case 56: return FN<elem_t, 56>(__VA_ARGS__);   \
    case 72: return FN<elem_t, 72>(__VA_ARGS__);   case 88: return FN<elem_t, 88>(__VA_ARGS__);   \
    case 104: return FN<elem_t, 104>(__VA_ARGS__); case 120: return FN<elem_t, 120>(__VA_ARGS__); \
    case 16: return FN<elem_t, 16>(__VA_ARGS__);   case 32: return FN<elem_t, 32>(__VA_ARGS__);   \
    case 48: return FN<elem_t, 48>(__VA_ARGS__);   case 64: return FN<elem_t, 64>(__VA_ARGS__);   \
    case 80: return FN<elem_t, 80>(__VA_ARGS__);   case 96: return FN<elem_t, 96>(__VA_ARGS__);   \
    case 112: return FN<elem_t, 112>(__VA_ARGS__); case 128: return FN<elem_t, 128>(__VA_ARGS__); \
    case 144: return FN<elem_t, 144>(__VA_ARGS__); case 160: return FN<elem_t, 160>(__VA_ARGS__); \
    case 176: return FN<elem_t, 176>(__VA_ARGS__); case 192: return FN<elem_t, 192>(__VA_ARGS__); \
    case 208: return FN<elem_t, 208>(__VA_ARGS__); case 224: return FN<elem_t, 224>(__VA_ARGS__); \
    case 240: return FN<elem_t, 240>(__VA_ARGS__); case 256: return FN<elem_t, 256>(__VA_ARGS__); \
  }

// q: [n_tokens, ...] with `q_row_stride` elements between rows, head h at column h * head_dim.
// out: the same shape convention.  block_tables: int32 [n_seqs, max_pages].  tiled: the tokens are portions of prompts, for the kernel
// that takes 32 neighbouring ones together (32 bits, heads of 64 and 128; else without meaning); 2: heads of 64 by one group of threads a block.
ERB_EXPORT int erb_attention_rows(const void* q, int q_row_stride, const void* k_pages, const void* v_pages,
                                  const int* block_tables, int max_pages, const int* seq_of_token,
                                  const int* positions, void* out, int out_row_stride, int n_tokens, int nq,
                                  int nkv, int head_dim, int page_size, int window, int keep_first, float scale,
                                  const float* penalty, float softcap, const void* gate, int gate_stride, int tiled, void* stream) {
  if (n_tokens <= 0) return ERB_OK;
  if (penalty && softcap > 0.f) return fail(ERB_ERR_UNSUPPORTED, "attention_rows: a penalty and a cap of the scores exclude each other");
  int rc = check_common("attention_rows", nq, nkv, head_dim, page_size, max_pages);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
#if ERB_ELEM == 0
  if (tiled && (head_dim == 64 || head_dim == 128) && !(((uintptr_t)k_pages | (uintptr_t)v_pages) & 15))
    return (head_dim == 128 ? launch_tiles<128, 2> : tiled == 2 ? launch_tiles<64, 1> : launch_tiles<64, 2>)(
        q, q_row_stride, k_pages, v_pages, block_tables, max_pages, seq_of_token, positions, out, out_row_stride, n_tokens, nq, nkv, page_size,
        window, window > 0 ? keep_first : 0, scale, penalty, softcap, gate, gate_stride, s);
#endif
  ERB_DISPATCH_D(launch_rows, q, q_row_stride, k_pages, v_pages, block_tables, max_pages, seq_of_token,
                 positions, out, out_row_stride, n_tokens, nq, nkv, page_size, window, window > 0 ? keep_first : 0, scale, penalty,
                 softcap, gate, gate_stride, s)
  return fail(ERB_ERR_UNSUPPORTED, "attention_rows: head_dim %d", head_dim);
}

// Scratch the caller provides: part_acc float [n_seqs * nq * max_splits * head_dim],
// part_ml float [n_seqs * nq * max_splits * 2], with max_splits >= the largest number of splits
// any sequence of the batch has (its visible key range cut at multiples of split_keys).
ERB_EXPORT int erb_attention_decode(const void* q, int q_row_stride, const void* k_pages,
                                    const void* v_pages, const int* block_tables, int max_pages,
                                    const int* token_of_seq, const int* positions, void* out,
                                    int out_row_stride, float* part_acc, float* part_ml, int max_splits,
                                    int n_seqs, int nq, int nkv, int head_dim, int page_size, int window,
                                    int keep_first, int split_keys, float scale, const float* penalty, float softcap,
                                    const void* gate, int gate_stride, void* stream) {
  if (n_seqs <= 0) return ERB_OK;
  if (penalty && softcap > 0.f) return fail(ERB_ERR_UNSUPPORTED, "attention_decode: a penalty and a cap of the scores exclude each other");
  int rc = check_common("attention_decode", nq, nkv, head_dim, page_size, max_pages);
  if (rc) return rc;
  if (max_splits <= 0 || split_keys <= 0 || !part_acc || !part_ml)
    return fail(ERB_ERR_ARG, "attention_decode: scratch or split arguments missing");
  if (n_seqs > 65535 || nq > 65535) return fail(ERB_ERR_UNSUPPORTED, "attention_decode: grid too large");
  cudaStream_t s = (cudaStream_t)stream;
  ERB_DISPATCH_D(launch_decode, q, q_row_stride, k_pages, v_pages, block_tables, max_pages, token_of_seq,
                 positions, out, out_row_stride, part_acc, part_ml, max_splits, n_seqs, nq, nkv, page_size,
                 window, window > 0 ? keep_first : 0, split_keys, scale, penalty, softcap, gate, gate_stride, s)
  return fail(ERB_ERR_UNSUPPORTED, "attention_decode: head_dim %d", head_dim);
}

// ---------------------------------------------------------------------------------------------
// The variant for callers that cannot allocate: scratch in a file-scope device array.
// See attention_noalloc.h for the contract.
// ---------------------------------------------------------------------------------------------
#include "attention_noalloc.h"

static __device__ __align__(256) float g_static_decode_scratch[ERB_STATIC_SCRATCH_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
// Device address of the array on each device; looked up once per device by the first call there.
// In host code the array's name is only a handle for the runtime, not a device pointer.
float* g_static_scratch_addr[kMaxDevices] = {nullptr};
std::mutex g_static_scratch_mutex;

int static_scratch_for_current_device(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "attention_decode_static: cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return fail(ERB_ERR_UNSUPPORTED, "attention_decode_static: device %d", dev);
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  if (!g_static_scratch_addr[dev]) {
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_static_decode_scratch);
    if (e != cudaSuccess || !p)
      return fail(ERB_ERR_CUDA, "attention_decode_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    g_static_scratch_addr[dev] = p;
  }
  *out = g_static_scratch_addr[dev];
  return ERB_OK;
}
}  // namespace

ERB_EXPORT long long erb_attention_decode_static_floats(int n_seqs, int nq, int head_dim, int max_splits) {
  return (long long)n_seqs * nq * max_splits * (head_dim + 2);
}

ERB_EXPORT int erb_attention_decode_static(const void* q, int q_row_stride, const void* k_pages,
                                           const void* v_pages, const int* block_tables, int max_pages,
                                           const int* token_of_seq, const int* positions, void* out,
                                           int out_row_stride, int max_splits, int n_seqs, int nq, int nkv,
                                           int head_dim, int page_size, int window, int split_keys,
                                           float scale, void* stream) {
  if (n_seqs <= 0) return ERB_OK;
  if (max_splits <= 0 || nq <= 0 || head_dim <= 0)
    return fail(ERB_ERR_ARG, "attention_decode_static: bad sizes");
  const long long need = erb_attention_decode_static_floats(n_seqs, nq, head_dim, max_splits);
  if (need > (long long)ERB_STATIC_SCRATCH_FLOATS)
    return fail(ERB_ERR_UNSUPPORTED,
                "attention_decode_static: %lld floats of scratch needed (sequences %d x heads %d x splits %d x "
                "(head_dim %d + 2)), the built-in array holds %d; use erb_attention_decode with caller scratch",
                need, n_seqs, nq, max_splits, head_dim, (int)ERB_STATIC_SCRATCH_FLOATS);
  float* base = nullptr;
  int rc = static_scratch_for_current_device(&base);
  if (rc) return rc;
  float* part_acc = base;
  float* part_ml = base + (size_t)n_seqs * nq * max_splits * head_dim;
  return erb_attention_decode(q, q_row_stride, k_pages, v_pages, block_tables, max_pages, token_of_seq,
                              positions, out, out_row_stride, part_acc, part_ml, max_splits, n_seqs, nq, nkv,
                              head_dim, page_size, window, 0, split_keys, scale, nullptr, 0.f, nullptr, 0, stream);
}
