// Causal attention for portions of prompts whose value rows are wider than 64 entries, on the 5th-generation tensor cores
// (tcgen05 + TMEM), warps specialised by role as in attention_prefill.cu.  Two forms of one kernel (bfloat16):
//
//   differential   two softmax maps of 64 entries per head over the same values: a block owns 128 tokens of one head; its two
//                  query tiles are the two maps, each with keys of its own, both with the same value tile.  Keys and values
//                  come from the cache's pages.  The difference of the maps, the head norm and the constant are in the epilogue.
//   rows           keys of up to 192 entries made of a part per head and a part that all heads share, values of 64 or 128, one
//                  softmax: a block owns 256 tokens of one head as two query tiles that use the same keys and values.  Keys and
//                  values lie in rows of plain buffers (the up-projected latents of a portion's context).  Sinks and a gate per
//                  head are in the epilogue.
//
//   warp 18 (copy)    brings the key and the value blocks of a tile of 64 keys by TMA tensor copies, three or four tiles of each in
//                     flight
//   warps 16, 17      issue S_t(j) = Q_t K(j)^T (M 128, N 64) and O_t += P_t(j) V(j) (M 128, N 64 or 128) for query tile 0 and 1;
//                     S, O and P in TMEM
//   warps 0-7, 8-15   softmax of query tile 0 and 1: two threads per row, each with 32 of a tile's 64 keys
//
// A tile's scores have two places in TMEM, and P takes the place of the scores that it was made of: S_t(j + 1) is there when the
// softmax of S_t(j) ends, and the softmax warps need not wait for a product in a step.  The place of S_t(j) is taken by
// S_t(j + 2) only once P_t(j) V(j) has been seen to end.  Every hand-over is an mbarrier, every wait for one is bounded: a thread that
// gives up raises a block-wide flag, the block records a code in *status, lets its copies land, frees its TMEM and returns.  The
// barriers between softmax warps have no limit; all their warps come to each of them, whatever their waits give (pair_rounds.h).
//
// P goes into the second product as two bfloat16 pieces, its rounding and what that leaves: the reference maximum moves seldom, so
// the largest weight of a row is no longer exactly 1, and rounding it once would lose 4 % of accuracy against a kernel that
// moves it with every tile.  The tensor cores have the room for the second piece.
//
// What bounds it: the exponentials and what is done to a score besides (17 instructions of all warps a score with a cap, 11.5 without); the tensor
// cores wait for them.  Tiles of 64 keys leave room in TMEM for two accumulators of 128 columns beside the scores, and in shared
// memory for three to four tiles beside the queries; that, and boxes of 64 columns, is why heads and values are of 64 or 128 (the
// differential form of 64 and 128: other sizes are diff_attention.cu's).  Differential, 2,048 tokens of 16 heads, capped: 240 us by the mma.sync
// kernel of diff_attention.cu, 71 us by this; without a cap 185 us and 56 us.
// Rows, 2,048 tokens of 16 heads of 128 + 64 and 128: about 50 us beside 20 us of gathering and up-projecting, where the kernel over
// latents of 512 took 705 us.
#include <limits.h>
#include <stdarg.h>
#include <stdio.h>

#undef ERB_ELEM
#define ERB_ELEM 1
#include "pair_rounds.h"
#include "tc_common.cuh"

using namespace erb;

ERB_DEFINE_LAST_ERROR(erb_last_error)

namespace {

constexpr int BM = 128, BN = 64;
constexpr int kSoftmaxWarps = 16, kIssueWarp = 16, kCopyWarp = 18, kThreads = 608;      // (warps 16 and 17 issue)
constexpr uint32_t kQBlock = BM * 128, kKvBlock = BN * 128;       // bytes of 64 columns of a query tile, of a key or value tile
constexpr uint32_t kTmemCols = 512, kColO = 256;     // scores, and P in their place: 2 tiles x 2 x 64; O: 2 x 128
__device__ __forceinline__ constexpr uint32_t col_s(int t, int j) { return (uint32_t)((2 * t + (j & 1)) * BN); }
constexpr float kSumLimit = 1048576.f;    // a tile's sum of P from which on the reference maximum is moved (2^20)
constexpr uint32_t kExchangeBytes = 2 * BM * 2 * 4;      // a float per (query tile, row, half of its keys)
constexpr int kExchangeLd = 132;          // floats of a row of the second map's result on its way to the first map's threads

struct WideArgs {
  const __nv_bfloat16* q;          // differential: [token][head][2][64]; rows: [token][head][dim + rot] (only the first dim read)
  int q_ld, q_head;                // elements between tokens, between heads
  const __nv_bfloat16* q_rot;      // rows: the turned parts, [token][head][64], zeros behind the rotated entries
  const int* block_tables;
  int max_pages, page_size, kv_heads;
  const int* seq_starts;
  const int* positions;
  int n_seqs, heads;
  int kv_rows, k_col, v_col, kv_head, rot_col;   // rows: buffer rows per sequence; columns of a head's keys and values, of the shared part
  float scale_log2, cap_in, cap_out;
  int window;
  const float* sink;
  const __nv_bfloat16* gate;
  int gate_ld;
  float lambda, eps, out_scale;
  __nv_bfloat16* out;              // [token][head][VB * 64]
  int* status;
};

template <bool DIFF, int KB, int VB>
__host__ __device__ constexpr uint32_t q_bytes() { return 2 * (DIFF ? 1 : KB) * kQBlock; }
template <bool DIFF, int KB, int VB>
__host__ __device__ constexpr int stages() { return KB == 3 ? 3 : 4; }
template <bool DIFF, int KB, int VB>
__host__ __device__ constexpr uint32_t smem_bytes() {
  return q_bytes<DIFF, KB, VB>() + stages<DIFF, KB, VB>() * (KB + VB) * kKvBlock + kExchangeBytes + 8 * (4 * stages<DIFF, KB, VB>() + 12) + 16 + 1024;
}

template <bool DIFF, int KB, int VB, bool CAP>
__global__ void __launch_bounds__(kThreads, 1)
attention_wide_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const WideArgs a) {
  constexpr int ST = stages<DIFF, KB, VB>();
  constexpr uint32_t kQ = q_bytes<DIFF, KB, VB>(), kKeys = KB * kKvBlock, kValues = VB * kKvBlock;      // bytes of a tile
  constexpr int kRows = DIFF ? BM : 2 * BM;                     // tokens of a block
  // barriers: key and value tiles there and free again; per query tile and place (even and odd steps): S there, P written,
  // P V done.  Two of each, since a waiting thread may lag one step, and a barrier's parity tells two steps apart but not three
  constexpr int kBarKFull = 0, kBarKEmpty = ST, kBarVFull = 2 * ST, kBarVEmpty = 3 * ST, kBarS = 4 * ST, kBarP = kBarS + 4,
                kBarPv = kBarP + 4, kNumBars = kBarPv + 4;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;                 // the swizzle repeats every 1024 bytes
  uint8_t* smem = smem_raw + (base - raw);
  const uint32_t sQ = base, sK = sQ + kQ, sV = sK + ST * kKeys, bars = sV + ST * kValues + kExchangeBytes;
  float* shared_rows = reinterpret_cast<float*>(smem + kQ + ST * (kKeys + kValues));      // [query tile][row][half]
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + (bars - base) + 8 * kNumBars);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + (bars - base) + 8 * kNumBars + 8);
  auto bar = [&](int which) { return bars + 8u * (uint32_t)which; };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.x;

  // later rows of a prompt see more keys: the last rows of every head start first
  int tile = (int)(gridDim.y - 1 - blockIdx.y), seq = -1, q0 = 0, rows = 0, seq_q0 = 0;
  for (int s = 0; s < a.n_seqs; ++s) {
    const int begin = a.seq_starts[s], len = a.seq_starts[s + 1] - begin, n_tiles = (len + kRows - 1) / kRows;
    if (tile < n_tiles) { seq = s; seq_q0 = begin; q0 = begin + tile * kRows; rows = min(kRows, len - tile * kRows); break; }
    tile -= n_tiles;
  }
  if (seq < 0) return;                                          // (the grid is an upper bound)
  if (*reinterpret_cast<volatile int*>(a.status) != 0) return;  // an earlier block gave up: do not pile on

  if (tid == 0) {
    for (int s = 0; s < ST; ++s) {                     // (free again: told by both issuing warps)
      mbar_init(bar(kBarKFull + s), 1); mbar_init(bar(kBarVFull + s), 1);
      mbar_init(bar(kBarKEmpty + s), 2); mbar_init(bar(kBarVEmpty + s), 2);
    }
    for (int i = 0; i < 4; ++i) { mbar_init(bar(kBarS + i), 1); mbar_init(bar(kBarP + i), 8); mbar_init(bar(kBarPv + i), 1); }    // (P: an arrival per warp of the group)
    *s_abort = 0;
    mbar_init_fence();
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  chain_wait();     // queries, positions, keys and values are written by the kernels before this one

  const int pos0 = a.positions[q0], last_key = pos0 + rows - 1;
  const int lo_block = first_visible_key(pos0, a.window), key_first = lo_block & ~(BN - 1);
  const int rows_t[2] = {min(rows, BM), DIFF ? rows : max(rows - BM, 0)};
  const int n_end[2] = {(pos0 + rows_t[0] - 1 - key_first) / BN + 1, rows_t[1] > 0 ? (last_key - key_first) / BN + 1 : 0};
  const int n_kv = max(n_end[0], n_end[1]);
  const int valid_last = last_key - (key_first + (n_kv - 1) * BN) + 1;        // keys of the last tile

  if (warp < kSoftmaxWarps) {
    // query tiles: a warp copies four whole 128-byte rows at a time; rows past the portion's end are zeros
    constexpr int QB = DIFF ? 1 : KB;
    for (int idx = tid; idx < 2 * QB * BM * 8; idx += kSoftmaxWarps * 32) {
      const int c = idx & 7, r = (idx >> 3) & (BM - 1), block = (idx >> 10) % QB, t = (idx >> 10) / QB;
      const int row = DIFF ? r : t * BM + r;
      const bool valid = row < rows;
      const size_t tok = (size_t)(q0 + (valid ? row : 0));
      const __nv_bfloat16* src = DIFF ? a.q + tok * a.q_ld + h * a.q_head + 64 * t + 8 * c
                               : block < KB - 1 ? a.q + tok * a.q_ld + h * a.q_head + 64 * block + 8 * c
                                                : a.q_rot + (tok * a.heads + h) * 64 + 8 * c;
      cp_async16(sQ + (t * QB + block) * kQBlock + swz(r, c), src, valid);
    }
    cp_async_commit();
    cp_async_wait<0>();
    fence_async_proxy();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  int copies_k = 0, copies_v = 0;       // tiles the copy warp has asked for

  if (warp == kCopyWarp) {
    bool ok = true;
    auto wait = [&](int which, uint32_t parity) {      // the first lane polls, the others sleep in the vote
      bool mine = true;
      if (lane == 0) mine = mbar_wait_or_abort(bar(which), parity, s_abort);
      return __all_sync(0xffffffffu, mine) != 0;
    };
    if (DIFF) {
      // lane i brings piece i of a tile: a page, or the part of one that a tile of 64 keys covers
      const int* bt = a.block_tables + (size_t)seq * a.max_pages;
      const int piece = min(a.page_size, BN), pieces = BN / piece, kvh = h / (a.heads / a.kv_heads);
      const uint32_t piece_bytes = (uint32_t)piece * 128u;
      auto row_of = [&](int j) {                        // first pool row of this lane's piece, or -1 (behind the last key, or before every window)
        const int key = key_first + j * BN + lane * piece;
        if (j >= n_kv || lane >= pieces || key > last_key || (a.window != 0 && key + piece <= lo_block)) return -1;
        return (bt[key / a.page_size] * a.kv_heads + kvh) * a.page_size + key % a.page_size;
      };
      // (`row`: this lane's piece, or -1; zero_rest: rows that are not brought become zeros)
      auto bring = [&](int j, int row, const CUtensorMap* map, uint32_t dst, int blocks, uint32_t full, bool zero_rest) {
        const int n = __popc(__ballot_sync(0xffffffffu, row >= 0));
        if (zero_rest && row < 0 && lane < pieces && key_first + j * BN + lane * piece <= last_key) {
          // nobody sees these rows (their P is zero), but whatever an earlier tile left there would spoil 0 * x if it were no number
          for (int b = 0; b < blocks; ++b) {
            uint4* z = reinterpret_cast<uint4*>(smem + (dst - base) + lane * piece_bytes + b * kKvBlock);
            for (uint32_t i = 0; i < piece_bytes / 16; ++i) z[i] = make_uint4(0, 0, 0, 0);
          }
          fence_async_proxy();
        }
        __syncwarp();
        if (lane == 0) mbar_expect(full, (uint32_t)(n * blocks) * piece_bytes);
        __syncwarp();
        if (row >= 0)
          for (int b = 0; b < blocks; ++b) tma_load_box(dst + lane * piece_bytes + b * kKvBlock, map, 64 * b, row, full);
      };
      int row_next = row_of(0);
      for (int j = 0; j < n_kv && ok; ++j) {
        const int st = j % ST, row = row_next;
        row_next = row_of(j + 1);
        if (j >= ST) ok = wait(kBarKEmpty + st, ((j / ST) - 1) & 1);
        if (!ok) break;
        bring(j, row, &map_k, sK + st * kKeys, KB, bar(kBarKFull + st), false);
        copies_k = j + 1;
        if (j >= ST) ok = wait(kBarVEmpty + st, ((j / ST) - 1) & 1);
        if (!ok) break;
        bring(j, row, &map_v, sV + st * kValues, VB, bar(kBarVFull + st), true);
        copies_v = j + 1;
      }
    } else if (lane == 0) {
      // buffer row 0 of a sequence is the first key of the tile that holds the first key its portion sees
      const int row0 = seq * a.kv_rows + key_first - (first_visible_key(a.positions[seq_q0], a.window) & ~(BN - 1));
      for (int j = 0; j < n_kv && ok; ++j) {
        const int st = j % ST, row = row0 + j * BN;
        if (j >= ST) ok = mbar_wait_or_abort(bar(kBarKEmpty + st), ((j / ST) - 1) & 1, s_abort);
        if (!ok) break;
        mbar_expect(bar(kBarKFull + st), kKeys);
#pragma unroll
        for (int b = 0; b < KB - 1; ++b)
          tma_load_box(sK + st * kKeys + b * kKvBlock, &map_k, h * a.kv_head + a.k_col + 64 * b, row, bar(kBarKFull + st));
        tma_load_box(sK + st * kKeys + (KB - 1) * kKvBlock, &map_v, a.rot_col, row, bar(kBarKFull + st));      // (the second map: the latents' rows)
        copies_k = j + 1;
        if (j >= ST) ok = mbar_wait_or_abort(bar(kBarVEmpty + st), ((j / ST) - 1) & 1, s_abort);
        if (!ok) break;
        mbar_expect(bar(kBarVFull + st), kValues);
#pragma unroll
        for (int b = 0; b < VB; ++b)
          tma_load_box(sV + st * kValues + b * kKvBlock, &map_k, h * a.kv_head + a.v_col + 64 * b, row, bar(kBarVFull + st));
        copies_v = j + 1;
      }
    }
  } else if (warp >= kIssueWarp) {
    // The whole warp walks the steps and one elected lane issues: what a product takes then lies in uniform registers.  (A lone lane
    // that made descriptors in its own registers took 4,000 clocks a step to issue both tiles' 24 products, one such warp for both
    // tiles 2,000 beside six waits of 250.)
    constexpr uint32_t kIdescS = mma_idesc(BM, BN, false), kIdescO = mma_idesc(BM, 64 * VB, true);
    const bool elected = elect_one();
    const int t = __shfl_sync(0xffffffffu, warp - kIssueWarp, 0), n = __shfl_sync(0xffffffffu, n_end[t], 0), n_all = __shfl_sync(0xffffffffu, n_kv, 0);
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t dq = make_desc(sQ), dk = make_desc(sK);
    const uint64_t dv = (make_desc(sV) & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(kKvBlock >> 4) << 16);      // 64 columns of V apart: a block
    bool ok = true;
    auto wait = [&](int which, uint32_t parity) {
      if (ok) ok = mbar_wait_or_abort(bar(which), parity, s_abort);
      ok = __all_sync(0xffffffffu, ok) != 0;
    };
    auto issue_s = [&](int j) {                         // S_t(j) = Q_t K(j)^T; K(j) is free again behind it
      const int st = j % ST;
      wait(kBarKFull + st, (j / ST) & 1);
      if (!ok) return;
      const uint64_t keys = dk + (uint64_t)(st * (kKeys >> 4));
      const uint32_t d = tm + col_s(t, j);
      if (elected) {
#pragma unroll
        for (int b = 0; b < (DIFF ? 1 : KB); ++b)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_bf16(d, dq + (uint64_t)((t * (DIFF ? 1 : KB) + b) * (kQBlock >> 4) + 2 * k), keys + (uint64_t)((DIFF ? t : b) * (kKvBlock >> 4) + 2 * k),
                     kIdescS, b + k > 0);
        mma_commit(bar(kBarS + 2 * t + (j & 1)));
        mma_commit(bar(kBarKEmpty + st));
      }
      __syncwarp();
    };
    if (n > 0) issue_s(0);
    if (n > 1) issue_s(1);
    for (int j = 0; j < n && ok; ++j) {                 // O_t += P_t(j) V(j): 16 keys a step, 8 columns of each piece of P, 2048 bytes of V
      const int st = j % ST;
      wait(kBarVFull + st, (j / ST) & 1);
      if (DIFF && j == n_all - 1 && ok) {
        // rows behind the last key may hold anything (unwritten slots of the page, an earlier tile): their P is zero, but
        // 0 * NaN would spoil the product (both warps make them zeros, whichever comes first)
        for (int idx = lane; idx < VB * (BN - valid_last) * 8; idx += 32) {
          const int r = idx >> 3, b = r / (BN - valid_last);
          *reinterpret_cast<uint4*>(smem + (sV - base) + st * kValues + b * kKvBlock + swz(valid_last + r % (BN - valid_last), idx & 7)) =
              make_uint4(0, 0, 0, 0);
        }
        fence_async_proxy();
        __syncwarp();
      }
      wait(kBarP + 2 * t + (j & 1), (j >> 1) & 1);
      if (!ok) break;
      fence_after_sync();
      const uint64_t values = dv + (uint64_t)(st * (kValues >> 4));
      const uint32_t d = tm + kColO + t * 128, p = tm + col_s(t, j), more = j > 0 ? 1u : 0u;
      if (elected) {
#pragma unroll
        for (int k = 0; k < BN / 16; ++k) {
          mma_bf16_a_tmem(d, p + k * 8, values + (uint64_t)(k * (2048 >> 4)), kIdescO, k > 0 ? 1u : more);
          mma_bf16_a_tmem(d, p + BN / 2 + k * 8, values + (uint64_t)(k * (2048 >> 4)), kIdescO, 1u);
        }
        mma_commit(bar(kBarPv + 2 * t + (j & 1)));
        mma_commit(bar(kBarVEmpty + st));
      }
      __syncwarp();
      if (j + 2 < n) {
        wait(kBarPv + 2 * t + (j & 1), (j >> 1) & 1);   // P_t(j) V(j) has left the place (the softmax is busy with S_t(j + 1))
        if (ok) issue_s(j + 2);
      }
    }
    // tiles that only the other query tile uses are free for this one (each once it is there: the copies' phases stay in step)
    for (int j = n; j < n_all && ok; ++j) {
      wait(kBarKFull + j % ST, (j / ST) & 1);
      if (ok && lane == 0) mbar_arrive(bar(kBarKEmpty + j % ST));
      wait(kBarVFull + j % ST, (j / ST) & 1);
      if (ok && lane == 0) mbar_arrive(bar(kBarVEmpty + j % ST));
    }
  } else {
    // warp w of a group reaches the TMEM lanes of rows 32 (w & 3) .. + 31 and takes the keys 32 (w >> 2) .. + 31 of every tile
    const int t = warp >> 3, quarter = warp & 3, half = (warp >> 2) & 1, row = quarter * 32 + lane;
    const int tile_pos0 = pos0 + (DIFF ? 0 : t * BM), my_pos = min(tile_pos0 + row, last_key);     // (rows past the end see no garbage)
    const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t t_o = t_lane + kColO + t * 128 + half * 32 * VB;        // this thread's half of the accumulator's columns
    const int pair_barrier = 1 + t * 4 + quarter;                          // the two warps that share these rows
    float* mine = shared_rows + (t * BM + row) * 2 + half;
    const float* partners = shared_rows + (t * BM + row) * 2 + (half ^ 1);
    bool ok = true;
    auto wait = [&](int which, uint32_t parity) {        // the same answer for every lane: TMEM loads are collective
      return __all_sync(0xffffffffu, mbar_wait_or_abort(bar(which), parity, s_abort)) != 0;
    };
    float m_ref = -INFINITY, l_run = 0.f;                // l_run: this thread's half of the row's sum
    const int win_lo = first_visible_key(my_pos, a.window);
    auto hidden = [&](int key) { return key > my_pos || key < win_lo; };
    const int n_mine = n_end[t];
    for (int j = 0; j < n_mine; ++j) {
      PairRounds pair(j == 0);
      if (!wait(kBarS + 2 * t + (j & 1), (j >> 1) & 1)) {
        // the partner may have found the scores there: to its barriers, then out with it
        do {
          if (pair.search()) named_barrier(pair_barrier, 64);
          named_barrier_any(pair_barrier, 64, true);
        } while (pair.again());
        ok = false;
        break;
      }
      fence_after_sync();
      const uint32_t t_s = t_lane + col_s(t, j);
      const int tile_key0 = key_first + j * BN, key0 = tile_key0 + 32 * half;
      const bool edge = tile_key0 + BN - 1 > tile_pos0 || (a.window != 0 && tile_key0 < first_visible_key(tile_pos0 + BM - 1, a.window));
      // The exponentials are taken against the reference maximum of the tiles before; only on the first tile, or where a row's sum
      // shows that the reference is far too low, is the tile's maximum searched, the reference moved, O and the sum rescaled, and
      // the tile's P made again (P is a floating-point number: a reference that is low by twenty powers of two costs no precision).
      float l_tile = 0.f;
      uint32_t high[16], low[16];                        // P in two pieces, pairs of neighbouring keys
      bool capped = false;                               // the scores have been replaced by capped ones in the log2 domain
      for (;;) {
        if (pair.search()) {
          float m_raw = -INFINITY;
          {
            float s[32];
            tmem_ld32(t_s + 32 * half, s);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) m_raw = fmaxf(m_raw, (edge && hidden(key0 + i)) ? -INFINITY : s[i]);
          }
          // (the cap is monotonic.  A row may see nothing of its first tiles: its reference then stays at a finite floor)
          *mine = CAP ? (m_raw == -INFINITY ? -1e30f : capped ? m_raw : capped_score(m_raw * (a.cap_in * 2.8853900817779268f), a.cap_out))
                      : fmaxf(m_raw * a.scale_log2, -1e30f);
          named_barrier(pair_barrier, 64);
          const float m_tile = fmaxf(*mine, *partners);
          float alpha = 1.f;
          if (m_tile > m_ref) {
            alpha = fast_exp2(m_ref - m_tile);           // 0 on the first tile
            m_ref = m_tile;
          }
          l_run *= alpha;
          if (j > 0) {
            if (wait(kBarPv + 2 * t + ((j - 1) & 1), ((j - 1) >> 1) & 1)) {      // P V of the tile before must have landed
              fence_after_sync();
#pragma unroll 1
              for (int c = 0; c < VB; ++c) {
                float acc[32];
                tmem_ld32(t_o + 32 * c, acc);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] *= alpha;
                tmem_st32(t_o + 32 * c, acc);
              }
            }
          }
        }
        float even, odd;
        for (;;) {
          Two l2[2] = {Two(0.f), Two(0.f)};
          float s[2][16], big = 0.f;
          tmem_ld16(t_s + 32 * half, s[0]);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            tmem_ld_wait();
            if (c == 0) tmem_ld16(t_s + 32 * half + 16, s[1]);
            float* sc = s[c];
            const Two ref2(-m_ref);
            if (CAP && !capped) {
              const Two in2(a.cap_in), out2(a.cap_in * a.cap_out);
#pragma unroll
              for (int i = 0; i < 16; i += 2) {
                big = fmaxf(big, fmaxf(fabsf(sc[i]), fabsf(sc[i + 1])));
                const Two s2(sc[i], sc[i + 1]), x = s2 * in2, y = x * x;
                Two p = fma2(Two(kTanh5), y, Two(kTanh4));
                p = fma2(p, y, Two(kTanh3));
                p = fma2(p, y, Two(kTanh2));
                p = fma2(p, y, Two(kTanh1));
                p = fma2(p, y, Two(kTanh0));
                fma2(s2 * out2, p, ref2).get(sc[i], sc[i + 1]);
              }
            } else {
              const Two scale2(CAP ? 1.f : a.scale_log2);
#pragma unroll
              for (int i = 0; i < 16; i += 2) fma2(Two(sc[i], sc[i + 1]), scale2, ref2).get(sc[i], sc[i + 1]);
            }
            if (edge) {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (hidden(key0 + 16 * c + i)) sc[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float p0 = fast_exp2(sc[2 * i]), p1 = fast_exp2(sc[2 * i + 1]);
              const Two p(p0, p1);
              l2[i & 1] = l2[i & 1] + p;
              const __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
              const uint32_t hi = *reinterpret_cast<const uint32_t*>(&b);
              float r0, r1;
              (p + Two(__uint_as_float((hi << 16) ^ 0x80000000u), __uint_as_float((hi & 0xffff0000u) ^ 0x80000000u))).get(r0, r1);
              const __nv_bfloat162 e = __floats2bfloat162_rn(r0, r1);
              high[8 * c + i] = hi;
              low[8 * c + i] = *reinterpret_cast<const uint32_t*>(&e);
            }
          }
          (l2[0] + l2[1]).get(even, odd);
          if (!CAP || capped || !__any_sync(0xffffffffu, !(big * a.cap_in <= 1.f))) break;
          // some score lies beyond the polynomial: the scores are capped in their place by the exact form, and the tile is taken again
          const float x_in = a.cap_in * 2.8853900817779268f;
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            float x[16];
            tmem_ld16(t_s + 32 * half + 16 * c, x);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = capped_score(x[i] * x_in, a.cap_out);
            tmem_st16(t_s + 32 * half + 16 * c, reinterpret_cast<const uint32_t*>(x));
          }
          tmem_st_wait();
          capped = true;
        }
        l_tile = even + odd;
        // both threads of a row have to agree on the reference (and behind this barrier both have read their scores)
        if (!named_barrier_any(pair_barrier, 64, pair.vote(!(l_tile < kSumLimit), s_abort))) break;
        if (!pair.again()) { ok = false; break; }
      }
      if (!ok) break;
      tmem_st16(t_s + 16 * half, high);                  // (in the scores' place: 32 columns of pairs of each piece)
      tmem_st16(t_s + BN / 2 + 16 * half, low);
      tmem_st_wait();
      l_run += l_tile;
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kBarP + 2 * t + (j & 1)));
    }
    if (n_mine > 0 && ok) {
      ok = wait(kBarPv + 2 * t + ((n_mine - 1) & 1), ((n_mine - 1) >> 1) & 1);
      fence_after_sync();
    }
    *mine = l_run;                                       // (behind the last vote: the partner has read the maximum)
    named_barrier(9, kSoftmaxWarps * 32);
    const float l_row = l_run + *partners;
    const size_t tok = (size_t)(q0 + (DIFF ? row : t * BM + row));
    __nv_bfloat16* dst = a.out + (tok * a.heads + h) * (VB * 64) + half * 32 * VB;
    auto store32 = [&](__nv_bfloat16* to, const float* v, float f) {
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(v[i + 2 * e] * f, v[i + 2 * e + 1] * f);
          w[e] = *reinterpret_cast<const uint32_t*>(&b);
        }
        *reinterpret_cast<uint4*>(to + i) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    };
    if (DIFF) {
      // the second map's rows go to the first map's threads through the key and value stages, which nobody uses any more
      float* exchange = reinterpret_cast<float*>(smem + kQ) + row * kExchangeLd + half * 32 * VB;
      if (t == 1 && ok) {
        const float f = a.lambda / l_row;
#pragma unroll
        for (int c = 0; c < VB; ++c) {
          float acc[32];
          tmem_ld32(t_o + 32 * c, acc);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(exchange + 32 * c + i) = make_float4(f * acc[i], f * acc[i + 1], f * acc[i + 2], f * acc[i + 3]);
        }
      }
      named_barrier(9, kSoftmaxWarps * 32);
      if (t == 0) {
        const float inv = 1.f / l_row;
        float acc[VB][32], ss = 0.f;
        if (ok) {
#pragma unroll
          for (int c = 0; c < VB; ++c) tmem_ld32(t_o + 32 * c, acc[c]);
          tmem_ld_wait();
        }
#pragma unroll
        for (int c = 0; c < VB; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 o2 = *reinterpret_cast<const float4*>(exchange + 32 * c + i);
            acc[c][i] = fmaf(acc[c][i], inv, -o2.x);
            acc[c][i + 1] = fmaf(acc[c][i + 1], inv, -o2.y);
            acc[c][i + 2] = fmaf(acc[c][i + 2], inv, -o2.z);
            acc[c][i + 3] = fmaf(acc[c][i + 3], inv, -o2.w);
#pragma unroll
            for (int e = 0; e < 4; ++e) ss = fmaf(acc[c][i + e], acc[c][i + e], ss);
          }
        float* squares = shared_rows + 2 * BM;           // (the second tile's places, whose sums have been read)
        squares[row * 2 + half] = ss;
        named_barrier(pair_barrier, 64);
        const float f = rsqrtf((ss + squares[row * 2 + (half ^ 1)]) / (float)(64 * VB) + a.eps) * a.out_scale;
        if (ok && row < rows) {
#pragma unroll
          for (int c = 0; c < VB; ++c) store32(dst + 32 * c, acc[c], f);
        }
      }
    } else if (ok && n_mine > 0) {
      const bool valid = row < rows_t[t];
      float f = 1.f / (a.sink ? l_row + exp2f(fmaf(a.sink[h], 1.4426950408889634f, -m_ref)) : l_row);
      if (a.gate && valid) f *= 1.f / (1.f + expf(-__bfloat162float(a.gate[tok * a.gate_ld + h])));
#pragma unroll
      for (int c = 0; c < VB; ++c) {
        float acc[32];
        tmem_ld32(t_o + 32 * c, acc);
        tmem_ld_wait();
        if (valid) store32(dst + 32 * c, acc, f);
      }
    }
  }

  fence_before_sync();
  __syncthreads();
  if (*s_abort) {
    // copies that were asked for may still be on their way: let them land before the shared memory is given back
    if (warp == kCopyWarp && lane == 0) {
      for (int i = max(0, copies_k - ST); i < copies_k; ++i) mbar_wait(bar(kBarKFull + i % ST), (i / ST) & 1);
      for (int i = max(0, copies_v - ST); i < copies_v; ++i) mbar_wait(bar(kBarVFull + i % ST), (i / ST) & 1);
    }
    if (tid == 0) atomicCAS(a.status, 0, 1000000 + (int)(blockIdx.y * gridDim.x + blockIdx.x));
    __syncthreads();
  }
  if (warp == kIssueWarp) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// The cache rows that a portion's tokens see, gathered into plain rows: row r of sequence s is key g + r, g the first key of the
// tile of 64 that holds the first key its first token sees; zeros before that key and behind the last one.  A warp per row.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const __nv_bfloat16* __restrict__ pages, const int* __restrict__ block_tables, int max_pages,
                     const int* __restrict__ seq_starts, const int* __restrict__ positions, int rows, int kv_rows, int width, int page_size,
                     int window, __nv_bfloat16* __restrict__ out) {
  chain_wait();
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  const int s = r / kv_rows;
  const int lo = first_visible_key(positions[seq_starts[s]], window), key = (lo & ~(BN - 1)) + r - s * kv_rows;
  const bool real = key >= lo && key <= positions[seq_starts[s + 1] - 1];
  const uint4* src = reinterpret_cast<const uint4*>(
      pages + (real ? ((size_t)block_tables[(size_t)s * max_pages + key / page_size] * page_size + key % page_size) * width : 0));
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)r * width);
  for (int c = lane; c < width / 8; c += 32) dst[c] = real ? src[c] : make_uint4(0, 0, 0, 0);
}

// The rotated parts of the queries: row t holds, per head, `dim` unrotated then `rot` rotated entries; the latter go, turned, to
// out[token][head][64], zeros behind them.  Pairs (2i, 2i + 1), angle = position * inv_freq[i] in float, cosines and sines times
// rot_mult.  A block per token: the angles once for all heads.
__global__ void __launch_bounds__(128)
latent_q_rows_kernel(const __nv_bfloat16* __restrict__ q, int ld, int heads, int dim, int rot, const int* __restrict__ positions,
                     const float* __restrict__ inv_freq, int rot_dims, float rot_mult, __nv_bfloat16* __restrict__ out) {
  chain_wait();
  __shared__ float2 turn[32];
  const int t = blockIdx.x;
  if (threadIdx.x < 32) {
    float sn = 0.f, cs = 1.f;
    if (2 * (int)threadIdx.x < rot_dims) {
      sincosf((float)positions[t] * inv_freq[threadIdx.x], &sn, &cs);
      sn *= rot_mult; cs *= rot_mult;
    }
    turn[threadIdx.x] = make_float2(cs, sn);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < heads * 32; idx += blockDim.x) {
    const int h = idx >> 5, i = idx & 31;
    __nv_bfloat162 v = __floats2bfloat162_rn(0.f, 0.f);
    if (2 * i < rot) {
      const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(q + (size_t)t * ld + (size_t)h * (dim + rot) + dim + 2 * i));
      const float2 c = turn[i];
      v = __floats2bfloat162_rn(u.x * c.x - u.y * c.y, u.y * c.x + u.x * c.y);
    }
    *reinterpret_cast<__nv_bfloat162*>(out + ((size_t)t * heads + h) * 64 + 2 * i) = v;
  }
}

template <bool DIFF, int KB, int VB, bool CAP>
int launch(const CUtensorMap& mk, const CUtensorMap& mv, const WideArgs& a, int n_blocks, void* stream, const char* who) {
  auto kern = attention_wide_kernel<DIFF, KB, VB, CAP>;
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<DIFF, KB, VB>());
    if (e != cudaSuccess) return fail(ERB_ERR_CUDA, "%s: %s", who, cudaGetErrorString(e));
    configured = true;
  }
  launch_chained(kern, dim3(a.heads, n_blocks), dim3(kThreads), smem_bytes<DIFF, KB, VB>(), (cudaStream_t)stream, mk, mv, a);
  return check_launch(who);
}

}  // namespace

// Differential attention over portions (maps of 64, values of 128, pages of 8 to 128 tokens, a power of two).  q: [token][head][2][64],
// rotated, not scaled; seq_starts: int32 [n_seqs + 1] offsets of the sequences to process (consecutive rows of block_tables);
// n_blocks: sum over them of ceil(length / 128) (an upper bound is fine).  window > 0: a row sees its last `window` keys.
// softcap > 0: a scaled score s becomes softcap * tanh(s / softcap).
ERB_EXPORT int erb_attention_wide_diff(const void* q, const void* k_pages, const void* v_pages, int n_pool_pages, const int* block_tables,
                                       int max_pages, const int* seq_starts, const int* positions, void* out, int n_seqs, int n_blocks,
                                       int heads, int kv_heads, int page_size, int window, float scale, float softcap, float lambda,
                                       float eps, float out_scale, int* status, void* stream) {
  if (n_seqs <= 0 || n_blocks <= 0) return ERB_OK;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || n_blocks > 65535 || max_pages <= 0 || n_pool_pages <= 0 || !status || window < 0 ||
      !(scale > 0.f))
    return fail(ERB_ERR_ARG, "attention_wide_diff: bad sizes or a missing status word");
  if (page_size < 8 || page_size > 128 || (page_size & (page_size - 1)) || (((uintptr_t)q | (uintptr_t)out) & 15) ||
      (((uintptr_t)k_pages | (uintptr_t)v_pages) & 127))
    return fail(ERB_ERR_UNSUPPORTED, "attention_wide_diff: pages of %d, or rows that are not aligned", page_size);
  const unsigned long long pool_rows = (unsigned long long)n_pool_pages * kv_heads * page_size;
  if (pool_rows > 0x7fffffffull) return fail(ERB_ERR_UNSUPPORTED, "attention_wide_diff: pool too large for 32-bit row coordinates");
  const unsigned box = page_size < BN ? (unsigned)page_size : (unsigned)BN;
  CUtensorMap mk, mv;
  int rc;
  if ((rc = rows_map(&mk, k_pages, pool_rows, 128, 128, box, "attention_wide_diff")) ||
      (rc = rows_map(&mv, v_pages, pool_rows, 128, 128, box, "attention_wide_diff")))
    return rc;
  WideArgs a = {};
  a.q = (const __nv_bfloat16*)q; a.q_ld = heads * 128; a.q_head = 128;
  a.block_tables = block_tables; a.max_pages = max_pages; a.page_size = page_size; a.kv_heads = kv_heads;
  a.seq_starts = seq_starts; a.positions = positions; a.n_seqs = n_seqs; a.heads = heads;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.cap_in = softcap > 0.f ? scale / softcap : 0.f; a.cap_out = softcap * 1.4426950408889634f;
  a.window = window; a.lambda = lambda; a.eps = eps; a.out_scale = out_scale;
  a.out = (__nv_bfloat16*)out; a.status = status;
  return softcap > 0.f ? launch<true, 2, 2, true>(mk, mv, a, n_blocks, stream, "attention_wide_diff")
                       : launch<true, 2, 2, false>(mk, mv, a, n_blocks, stream, "attention_wide_diff");
}

// The cache rows of `n_seqs` portions as plain rows: out [n_seqs * kv_rows][width]; kv_rows a multiple of 64 that covers, from the
// tile of 64 keys with the first key a portion's first token sees, all of its keys.
ERB_EXPORT int erb_latent_gather(const void* pages, const int* block_tables, int max_pages, const int* seq_starts, const int* positions,
                                 int n_seqs, int kv_rows, int width, int page_size, int window, void* out, void* stream) {
  if (n_seqs <= 0 || kv_rows <= 0) return ERB_OK;
  if (kv_rows % BN || width <= 0 || width % 8 || page_size <= 0 || max_pages <= 0 || window < 0 || (long long)n_seqs * kv_rows > 0x7fffffffLL ||
      (((uintptr_t)pages | (uintptr_t)out) & 15))
    return fail(ERB_ERR_ARG, "latent_gather: bad sizes (rows of %d, %d a sequence) or alignment", width, kv_rows);
  const int rows = n_seqs * kv_rows;
  launch_chained(latent_gather_kernel, dim3((rows + 7) / 8), dim3(256), 0, (cudaStream_t)stream, (const __nv_bfloat16*)pages, block_tables,
                 max_pages, seq_starts, positions, rows, kv_rows, width, page_size, window, (__nv_bfloat16*)out);
  return check_launch("latent_gather");
}

ERB_EXPORT int erb_latent_q_rows(const void* q, int n_tokens, int ld, int heads, int dim, int rot, const int* positions, const float* inv_freq,
                                 int rot_dims, float rot_mult, void* out, void* stream) {
  if (n_tokens <= 0) return ERB_OK;
  if (heads <= 0 || dim % 2 || rot % 2 || rot < 0 || rot > 64 || ld % 2 || rot_dims > rot || rot_dims % 2 || (rot_dims > 0 && !inv_freq) ||
      (((uintptr_t)q | (uintptr_t)out) & 3))
    return fail(ERB_ERR_ARG, "latent_q_rows: bad sizes (rotated parts of %d, at most 64)", rot);
  launch_chained(latent_q_rows_kernel, dim3(n_tokens), dim3(128), 0, (cudaStream_t)stream, (const __nv_bfloat16*)q, ld, heads, dim, rot,
                 positions, inv_freq, rot_dims, rot_mult, (__nv_bfloat16*)out);
  return check_launch("latent_q_rows");
}

// Attention over rows: keys of a head are [dim | shared rot], values v_dim.  q: [token][head][dim + rot] (rows q_ld apart, the first
// `dim` entries of a head are read), q_rot: [token][head][64] from erb_latent_q_rows; kv: [n_seqs * kv_rows][heads][dim + v_dim];
// latents: [n_seqs * kv_rows][rank + rot] from erb_latent_gather, whose last `rot` columns are the keys' shared part.  All token rows
// start at the batch's first token; seq_starts as for erb_attention_wide_diff; n_blocks: sum of ceil(length / 256).  sink: float
// [heads] or null; gate: [token][head] logits (rows gate_ld apart) or null; out: [token][head][v_dim].
ERB_EXPORT int erb_attention_wide_rows(const void* q, int q_ld, const void* q_rot, const void* kv, const void* latents, const int* seq_starts,
                                       const int* positions, void* out, int n_seqs, int kv_rows, int n_blocks, int heads, int dim, int rot,
                                       int v_dim, int rank, int window, float scale, const float* sink, const void* gate, int gate_ld,
                                       int* status, void* stream) {
  if (n_seqs <= 0 || n_blocks <= 0) return ERB_OK;
  if ((dim != 64 && dim != 128) || (v_dim != 64 && v_dim != 128) || rot <= 0 || rot > 64 || rot % 8 || rank <= 0 || rank % 8)
    return fail(ERB_ERR_UNSUPPORTED, "attention_wide_rows: heads of %d + %d and %d over latents of %d", dim, rot, v_dim, rank);
  if (heads <= 0 || n_blocks > 65535 || kv_rows <= 0 || kv_rows % BN || !status || window < 0 || !(scale > 0.f) ||
      (long long)n_seqs * kv_rows > 0x7fffffffLL)
    return fail(ERB_ERR_ARG, "attention_wide_rows: bad sizes or a missing status word");
  if (q_ld % 8 || (((uintptr_t)q | (uintptr_t)q_rot | (uintptr_t)out | (uintptr_t)kv | (uintptr_t)latents) & 15))
    return fail(ERB_ERR_UNSUPPORTED, "attention_wide_rows: rows must be 16-byte aligned");
  const unsigned long long rows = (unsigned long long)n_seqs * kv_rows;
  const unsigned kv_ld = (unsigned)heads * (dim + v_dim), lat_ld = (unsigned)(rank + rot);
  CUtensorMap mk, ml;
  int rc;
  if ((rc = rows_map(&mk, kv, rows, kv_ld, kv_ld, BN, "attention_wide_rows")) ||
      (rc = rows_map(&ml, latents, rows, lat_ld, lat_ld, BN, "attention_wide_rows")))
    return rc;
  WideArgs a = {};
  a.q = (const __nv_bfloat16*)q; a.q_ld = q_ld; a.q_head = dim + rot; a.q_rot = (const __nv_bfloat16*)q_rot;
  a.seq_starts = seq_starts; a.positions = positions; a.n_seqs = n_seqs; a.heads = heads;
  a.kv_rows = kv_rows; a.k_col = 0; a.v_col = dim; a.kv_head = dim + v_dim; a.rot_col = rank;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.window = window; a.sink = sink; a.gate = (const __nv_bfloat16*)gate; a.gate_ld = gate_ld;
  a.out = (__nv_bfloat16*)out; a.status = status;
  if (dim == 64) return v_dim == 64 ? launch<false, 2, 1, false>(mk, ml, a, n_blocks, stream, "attention_wide_rows")
                                    : launch<false, 2, 2, false>(mk, ml, a, n_blocks, stream, "attention_wide_rows");
  return v_dim == 64 ? launch<false, 3, 1, false>(mk, ml, a, n_blocks, stream, "attention_wide_rows")
                     : launch<false, 3, 2, false>(mk, ml, a, n_blocks, stream, "attention_wide_rows");
}
