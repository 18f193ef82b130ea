// Causal grouped-query attention for steps that bring many tokens per sequence, on the
// 5th-generation tensor cores. A block owns two query tiles of 128 rows that share every K and V
// page it reads; S = Q K^T, P and O all live in tensor memory:
//
//   tensor memory (512 columns): S0 | S1 | O0 | O1. P_t, rounded to bfloat16, overwrites the first
//   64 columns of S_t (two keys per 32-bit column) and is the A operand of O_t += P_t V.
//   shared memory: Q0, Q1, and K and V double-buffered (128-byte swizzle, filled by TMA).
//
// Warps 0..3 run the softmax of tile 0 and warps 4..7 that of tile 1 (thread = query row = tensor-memory lane, all 128 keys
// of a block); lane 0 of warp 8 issues every MMA, lane 0 of warp 9 the TMA loads, in the order
//   ... PV0(j-1) QK0(j) PV1(j-1) QK1(j) PV0(j) QK0(j+1) ...
// so that while one tile's rows are in the softmax the tensor core works for the other tile.
//
// What bounds it is a tile's chain: softmax of a block, its P V, the next block's Q K^T (tensor memory has no room for a
// second S per tile). Per block of 128 keys a tile spends 1,800 clocks in the softmax (reading S 50, maximum 370,
// exponentials and packing 1,260 where the special-function unit alone takes 1,024, storing P 120), 1,030 in its 16 MMAs and
// about 600 on the barriers between them. A thread keeps its 128 scores in registers: the softmax warps take 216 each and the
// other four warps 72 (setmaxnreg; of the 168 that 384 threads start with). With 168 the compiler spilled some 100 bytes a
// thread, and the exponentials took 2,000 clocks, twice the rate of the unit, in every arrangement of the warps that was
// tried; a path of its own for blocks that some row sees in part cost as much (the compiler moved the exponentials of both
// paths in front of the branch), so scores that a row does not see become minus infinity first and there is one path.
// 2,048 tokens, 32 heads in groups of four: 45 us (49 before); four prompts of 957 to 1,531, 40 heads in groups of five:
// 105 (166 with query tiles of 128 rows fetched by the threads; 120 while the three rows that whole tokens leave empty counted as
// rows that see nothing, so that their warp masked every block).
// Per key block of 128 keys (two cache pages) and tile:
//   S = Q K^T                                   [issuer]   -> s_full
//   row max; p = exp2(S*c - m) rounded to bfloat16 -> tensor memory  [softmax]  -> p_ready
//   O += P V   (V as an MN-major B operand)     [issuer]
// O stays in tensor memory across key blocks. The reference maximum m of a row moves only when the
// row's maximum has grown by more than 2^8 since it was set (then the warp rescales its O rows in
// tensor memory); until then p <= 2^8, which float32 sums and bfloat16 probabilities hold without
// loss. The final division by the row's sum undoes the choice of m exactly as with a running maximum.
//
// Numerics as in the other attention kernels of this library (and the reference's,
// engine/kernels/attention.py:9-11,104-122 of willzeng274/kernel-rush-kawk): scores, maxima and sums
// in float32, probabilities rounded to bfloat16 before P.V, the output accumulated in float32. A
// query at position p sees keys max(0, p - window + 1)..p. The rows of a tile are (token, group
// member) pairs of one kv head, row R -> token R / G, head kh * G + R % G, so all G query heads of a
// kv head share one read of K and V (attention.py:70-73). Every barrier wait is bounded.
//
// WIDE: attention whose softmax weights are 32-bit quantities (krk_sink_prefill_tcgen05). A weight reaches P V as two bfloat16
// halves, p = hi + lo (16 bits of mantissa), which take the two halves of S's columns in tensor memory, and each instruction of
// P V comes twice, for the pages that some row of the tile sees. A row may start from a softmax sink (maximum = its head's
// sink, sum 1, no value); rows of the output may lie apart, are multiplied by a number and by the sigmoid of a gate per head or
// per element. SHAPED: scores are capped
// (c tanh(s / c) = c (1 - 2 / (1 + e^(2 s / c)))) and lose a slope times the distance of query and key before the softmax.
// 2,048 tokens, a window of 1,024, 16 heads of 128 in groups of four: 37 us (45 with the softmax of both tiles in all eight
// warps; the mma.sync kernel 116, of 37 at that instruction's measured rate, 550 TFLOP/s, for 19 GFLOP); 12 heads in groups of
// three, no slopes, 37 (43; 75).
//
// Compiled once per head size, for head sizes 64 and 128: -DKRK_HEAD_DIM=<D>.
#include "tcgen05.cuh"

#ifndef KRK_HEAD_DIM
#error "compile with -DKRK_HEAD_DIM=<head size>"
#endif

#if KRK_HEAD_DIM == 64 || KRK_HEAD_DIM == 128

namespace {

using namespace tc;

constexpr int D = KRK_HEAD_DIM;
constexpr int ROWS = 128;              // query rows per tile
constexpr int KEYS = 128;              // keys per block iteration: two pages
constexpr int DB = D / 64;             // 64-wide blocks of the head dimension
constexpr int THREADS = 384;           // 8 softmax warps, the warps that issue the MMAs, load and allocate, one idle
constexpr uint32_t SUB = 128 * 128;    // bytes of a [128 rows x 64 bf16] swizzled sub-tile
constexpr uint32_t TILE_BYTES = DB * SUB;  // a Q, K or V tile
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t TMEM_O = 256;       // O_t starts at column 256 + t * D; S_t at t * 128
constexpr float LOG2E = 1.4426950408889634f;
constexpr int PAGE_IDS = 1024;         // page-table entries a block keeps in shared memory (64 K keys)
constexpr float RESCALE_STEP = 8.f;    // in log2 units: the reference maximum moves when outgrown by 2^8

enum Bar { K_FULL = 0, V_FULL = 2, K_FREE = 4, V_FREE = 6, S_FULL = 8, P_READY = 10, O_DONE = 12, Q_FULL = 14, N_BARS = 15 };

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// byte offset of the 16-byte piece `chunk` (8 elements) of row `r` inside a swizzled [128 x 64] sub-tile
__device__ __forceinline__ uint32_t swz(int r, int chunk) { return (uint32_t)r * 128u + (uint32_t)((chunk ^ (r & 7)) << 4); }

struct TileRange {
  int lo, hi;  // key blocks the tile can see; lo > hi: the tile has no rows
  __device__ __forceinline__ bool has(int j) const { return j >= lo && j <= hi; }
};

__device__ __forceinline__ TileRange tile_range(int row_begin, int rows, int n_rows, int G, int q_len, int start, int window) {
  TileRange t;
  if (row_begin >= n_rows) { t.lo = 1; t.hi = 0; return t; }
  const int first_tok = row_begin / G;
  const int last_tok = min(q_len - 1, (row_begin + rows - 1) / G);
  t.lo = window > 0 ? max(0, start + first_tok - window + 1) / KEYS : 0;
  t.hi = (start + last_tok) / KEYS;
  return t;
}

// The first and the last page that some row of a tile sees, of the sequence's.
__device__ __forceinline__ int first_page(int row_begin, int G, int start, int window) {
  return window > 0 ? max(0, start + row_begin / G - window + 1) / KRK_PAGE : 0;
}
__device__ __forceinline__ int last_page(int row_begin, int rows, int G, int q_len, int start) {
  return (start + min(q_len - 1, (row_begin + rows - 1) / G)) / KRK_PAGE;
}

// What the wide form adds; see the opening text.
struct Extras {
  const float *sink, *slopes;  // per query head, either may be null
  float cap_log2, in_cap;      // softcap in log2 units, and what an exponent of 2 (x, in log2 units) is multiplied by; 0: none
  float in_tanh, small;        // scale / softcap, and the score up to which the tangent's argument is at most 0.65
  float out_scale;
  const bf16* gate;
  int gate_stride, gate_mode;  // 0: none, 1: a column per head, 2: a column per element
  int out_stride;
};

template <bool WIDE, int SHAPE>
__global__ void __launch_bounds__(THREADS, 1)
attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                         const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_o, int q_by_tma, int rows, bf16* __restrict__ out, const bf16* __restrict__ qkv, int q_stride, int HQ, int HKV,
                         const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                         const int* __restrict__ seq_qlen, const int* __restrict__ cu_q, const int* __restrict__ table,
                         int width, float scale_log2, int window, int* __restrict__ error, const Extras ex) {
  constexpr bool SHAPED = SHAPE != 0;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = base;                    // two tiles
  unsigned char* k_s = q_s + 2 * TILE_BYTES;    // two stages
  unsigned char* v_s = k_s + 2 * TILE_BYTES;    // two stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + 2 * TILE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + N_BARS);
  int* pages_s = reinterpret_cast<int*>(tmem_slot + 2);  // [PAGE_IDS] the block's page-table entries, from page 2 * j_lo on
  volatile int* gave_up = pages_s + PAGE_IDS;  // [2] per tile

  // blockIdx.x counts (row pair, kv head) with the pair as the slow index, descending: blocks start in
  // launch order, so the pairs with the most key blocks, of every kv head, run first and the short ones
  // fill the tail
  const int seq = blockIdx.y, kh = blockIdx.x % HKV;
  const int pair = gridDim.x / HKV - 1 - blockIdx.x / HKV;
  const int G = HQ / HKV;
  // all four before the first is used: one trip to memory
  const int q_len = seq_qlen[seq], start = seq_start[seq], slot = seq_slot[seq], row0 = cu_q[seq];
  const int n_rows = q_len * G;
  const int pair_row = pair * 2 * rows;
  if (pair_row >= n_rows) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const TileRange r0 = tile_range(pair_row, rows, n_rows, G, q_len, start, window);
  const TileRange r1 = tile_range(pair_row + rows, rows, n_rows, G, q_len, start, window);
  const int j_lo = r0.lo;                                   // tile 0 exists and starts no later than tile 1
  const int j_hi = r1.lo <= r1.hi ? max(r0.hi, r1.hi) : r0.hi;
  const int n = j_hi - j_lo + 1;

  // TMA loads: the first ones by the issuer (warp 8, lane 0) before the block's first barrier, the rest by the loader
  auto load_tile = [&](unsigned char* dst, const CUtensorMap* map, uint64_t* bar, int i) {
    mbar_expect_tx(bar, TILE_BYTES);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      // from shared memory: a load from the page table here would stand between the issuing thread's MMAs
      const int at = 2 * i + half;
      const int page = at < PAGE_IDS ? pages_s[at] : table[(size_t)slot * width + (2 * (j_lo + i) + half) % width];
      const int row = (page * HKV + kh) * KRK_PAGE;
#pragma unroll
      for (int h = 0; h < DB; ++h) tma_load_2d(dst + h * SUB + half * (64 * 128), map, bar, h * 64, row);
    }
  };
  auto load_k = [&](int i) { load_tile(k_s + (i & 1) * TILE_BYTES, &map_k, bars + K_FULL + (i & 1), i); };
  auto load_v = [&](int i) { load_tile(v_s + (i & 1) * TILE_BYTES, &map_v, bars + V_FULL + (i & 1), i); };

  if (warp == 9 && lane < 4) {
    const CUtensorMap* map = lane == 0 ? &map_k : lane == 1 ? &map_v : lane == 2 ? &map_q : &map_o;
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
  }
  if (warp == 8) {
    // The block's first loads in the order of what they wait for: the error word and the page-table entries are
    // requested together, the query tiles (which need neither) go out before either has arrived.
    // A block of this step that gave up on a wait (codes from 3 on): the others do no work. The host reads and
    // clears the word at the end of every step, so a flag never outlives the step that raised it.
    const int error_now = *reinterpret_cast<volatile int*>(error);
    int page_here[PAGE_IDS / 32 > 4 ? 4 : PAGE_IDS / 32];  // the first 128 entries, one load per lane and round
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = lane + 32 * q;
      page_here[q] = i < min(2 * n, PAGE_IDS) ? table[(size_t)slot * width + (2 * j_lo + i) % width] : 0;
    }
    if (lane == 0) {
      for (int i = 0; i < N_BARS; ++i) mbar_init(bars + i, (i == P_READY || i == P_READY + 1) ? ROWS / 32 : 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      gave_up[0] = gave_up[1] = 0;
      if (q_by_tma) {
        // a query tile is a box of whole tokens x G heads x 64 dims per 64-wide block of the head: its rows land in
        // (token, group member) order, which is the tile's row order
        const int tiles_here = r1.lo <= r1.hi ? 2 : 1;
        mbar_expect_tx(bars + Q_FULL, tiles_here * DB * rows * 128);
        for (int t = 0; t < tiles_here; ++t)
#pragma unroll
          for (int h = 0; h < DB; ++h)
            tma_load_3d(q_s + t * TILE_BYTES + h * SUB, &map_q, bars + Q_FULL, h * 64, kh * G, row0 + (pair_row + t * rows) / G);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (lane + 32 * q < min(2 * n, PAGE_IDS)) pages_s[lane + 32 * q] = page_here[q];
    for (int i = lane + 128; i < min(2 * n, PAGE_IDS); i += 32) pages_s[i] = table[(size_t)slot * width + (2 * j_lo + i) % width];
    __syncwarp();
    if (lane == 0) {
      tmem_slot[1] = (uint32_t)(error_now >= 3);
      if (error_now < 3) {
        load_k(0);
        load_v(0);
        if (n > 1) load_k(1);
      } else if (q_by_tma) {
        mbar_wait(bars + Q_FULL, 0);  // nothing else is asked for, and the block, which has nothing to do, stays until the query tiles are here
      }
    }
  } else if (warp == 10) {  // beside the loads of warp 8
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (!q_by_tma) {
    // the query tiles by hand: row r, 16-byte piece c -> swizzled K-major sub-tiles; rows past the end are zero
    for (int i = threadIdx.x; i < 2 * ROWS * (D / 8); i += THREADS) {
      const int r = i / (D / 8), c = i % (D / 8);
      const int R = pair_row + r;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (R < n_rows) v = *reinterpret_cast<const uint4*>(qkv + (size_t)(row0 + R / G) * q_stride + (size_t)(kh * G + R % G) * D + c * 8);
      *reinterpret_cast<uint4*>(q_s + (r / ROWS) * TILE_BYTES + (c / 8) * SUB + swz(r % ROWS, c % 8)) = v;
    }
    fence_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const bool dead = tmem_slot[1] != 0;

  if (dead) {
    // nothing to do
  } else if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 8) {
    if (lane == 0) {
      // ---- issuer: TMA loads and MMAs ----
      // a negative scale: the products leave negated (the descriptor's bit for A), and the softmax takes the scale's size, so that maxima
      // before it are maxima after it and a score that is not seen is minus infinity
      const uint32_t idesc_s = (!WIDE && scale_log2 < 0.f ? 1u << 13 : 0u) | (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(KEYS >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
      constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
      bool ok = true;
      auto give_up = [&](int code) { atomicExch(error, code); ok = false; };
      auto qk = [&](int t, int i) {  // S_t = Q_t K_i^T
        const unsigned char* q = q_s + t * TILE_BYTES;
        const unsigned char* k = k_s + (i & 1) * TILE_BYTES;
#pragma unroll
        for (int h = 0; h < DB; ++h)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_bf16(tmem + t * 128, umma_desc_sw128(q + h * SUB + kk * 32, 16, 1024),
                      umma_desc_sw128(k + h * SUB + kk * 32, 16, 1024), idesc_s, (h > 0 || kk > 0) ? 1u : 0u);
        umma_commit(bars + S_FULL + t);
      };
      // WIDE: whether a tile's first block has a first page, and its last block a second one, that no row of it sees. Such a page
      // stays out of P V: its weights are zero, but its values may be anything (the second page of a sequence's last block
      // may belong to another sequence), and zero times infinity is not zero.
      bool skip_first[2], skip_last[2];
      auto pv = [&](int t, int i, bool first, bool last) {  // O_t (+)= P_t V_i, 16 keys (8 columns of P) per instruction
        const unsigned char* v = v_s + (i & 1) * TILE_BYTES;
        if constexpr (WIDE) {
          const bool skip = first && skip_first[t];
          auto page = [&](int k0) {
#pragma unroll
            for (int ks = k0; ks < k0 + KEYS / 32; ++ks) {
              umma_bf16_tmem_a(tmem + TMEM_O + t * D, tmem + t * 128 + ks * 8, umma_desc_sw128(v + ks * 16 * 128, SUB, 1024),
                               idesc_o, (first && ks == 0) || (skip && ks == KEYS / 32) ? 0u : 1u);
              // the weights' low halves
              umma_bf16_tmem_a(tmem + TMEM_O + t * D, tmem + t * 128 + 64 + ks * 8, umma_desc_sw128(v + ks * 16 * 128, SUB, 1024),
                               idesc_o, 1u);
            }
          };
          if (!skip) page(0);
          if (!(last && skip_last[t])) page(KEYS / 32);
        } else {
#pragma unroll
          for (int ks = 0; ks < KEYS / 16; ++ks)
            umma_bf16_tmem_a(tmem + TMEM_O + t * D, tmem + t * 128 + ks * 8, umma_desc_sw128(v + ks * 16 * 128, SUB, 1024),
                             idesc_o, (first && ks == 0) ? 0u : 1u);
        }
      };
      const TileRange rng[2] = {r0, r1};
      if (q_by_tma && !mbar_wait(bars + Q_FULL, 0)) give_up(14);
      if (ok && !mbar_wait(bars + K_FULL, 0)) give_up(6);
      if (ok) {
        tc_fence_after();
        if (r0.has(j_lo)) qk(0, 0);
        if (r1.has(j_lo)) qk(1, 0);
        umma_commit(bars + K_FREE);
      }
      if constexpr (WIDE) {  // here, while the first scores are on their way
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          skip_first[t] = first_page(pair_row + t * rows, G, start, window) & 1;
          skip_last[t] = !(last_page(pair_row + t * rows, rows, G, q_len, start) & 1);
        }
      }
      for (int i = 0; i < n && ok; ++i) {
        const int j = j_lo + i, b = i & 1;
        bool v_ready = false, k_ready = false;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (rng[t].has(j)) {
            if (!mbar_wait(bars + P_READY + t, (j - rng[t].lo) & 1)) { give_up(8); break; }
            if (!v_ready) {
              if (!mbar_wait(bars + V_FULL + b, (i >> 1) & 1)) { give_up(9); break; }
              v_ready = true;
            }
            tc_fence_after();
            pv(t, i, j == rng[t].lo, j == rng[t].hi);
            if (j == rng[t].hi) umma_commit(bars + O_DONE + t);
          }
          if (t == 1) umma_commit(bars + V_FREE + b);
          if (i + 1 < n) {
            if (rng[t].has(j + 1)) {
              if (!k_ready) {
                if (!mbar_wait(bars + K_FULL + ((i + 1) & 1), ((i + 1) >> 1) & 1)) { give_up(10); break; }
                k_ready = true;
              }
              tc_fence_after();
              qk(t, i + 1);
            }
            if (t == 1) umma_commit(bars + K_FREE + ((i + 1) & 1));
          }
        }
      }
    }
    } else if (warp == 9) {
    if (lane == 0) {
      // ---- loader: the TMA loads after the first ones. A thread of its own: issuing a load takes the time of
      // several MMAs, and the issuer's instruction stream is what bounds the kernel.
      for (int i = 0; i < n; ++i) {
        if (i + 1 < n) {  // V of the next block goes where block i - 1's was
          if (i >= 1 && !mbar_wait(bars + V_FREE + ((i + 1) & 1), ((i - 1) >> 1) & 1)) { atomicExch(error, 7); break; }
          load_v(i + 1);
        }
        if (i + 2 < n) {  // K of block i + 2 goes where block i's was
          if (!mbar_wait(bars + K_FREE + (i & 1), (i >> 1) & 1)) { atomicExch(error, 11); break; }
          load_k(i + 2);
        }
      }
    }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ---- softmax: warps 0..3 have tile 0, warps 4..7 tile 1; thread = query row (its tensor-memory lane), whole key blocks.
    const int t = warp >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const TileRange rng = t ? r1 : r0;
    const uint32_t tmem_s = tmem + t * 128 + lane_addr, tmem_o = tmem + TMEM_O + t * D + lane_addr;
    // a thread without a row (a tile of fewer than 128, or the sequence's last) is where the last row is, so that its warp's blocks are seen
    // whole when its rows see them whole: its scores are anything, decide nothing and go nowhere
    const int rows_here = min(rows, n_rows - pair_row - t * rows);
    const int R = pair_row + t * rows + min(r, rows_here - 1);
    const bool valid = r < rows_here;
    const int pos = start + R / G;
    const int low = window > 0 ? max(0, pos - window + 1) : 0;
    float m = -INFINITY, slope = 0.f;
    float2 l2 = make_float2(0.f, 0.f);
    if constexpr (WIDE) {
      const int head = kh * G + R % G;
      if (ex.sink) {
        // a sink at minus infinity, or so low that it is in log2 units, is none: nothing is summed before the first key
        m = ex.sink[head] * LOG2E;
        l2.x = m != -INFINITY ? 1.f : 0.f;
      }
      if (SHAPED && ex.slopes) slope = ex.slopes[head] * LOG2E;
    }
    const float scale_size = WIDE ? scale_log2 : fabsf(scale_log2);  // a negative scale's sign is in the scores already
    const float2 scale2 = make_float2(scale_size, scale_size);
    constexpr uint32_t unseen = 0xff800000u;  // minus infinity: a score whose weight is zero
    bool ok = true, loud = false;  // a block of the warp had a capped score beyond the series' range: it is not looked for again
    for (int j = rng.lo; j <= rng.hi; ++j) {
      const int key0 = j * KEYS;
      // the row sees keys first..first + span of the block: (unsigned)(i - first) <= span; none of them: no i passes
      const bool none = pos < max(low, key0);
      const unsigned first = none ? (unsigned)KEYS : (unsigned)max(low - key0, 0);
      const unsigned span = none ? 0u : (unsigned)(pos - key0) - first;
      const bool whole = __all_sync(0xffffffffu, key0 + KEYS - 1 <= pos && key0 >= low);
      // tensor-memory loads and stores are warp-wide: a warp gives up as a whole
      if (!__all_sync(0xffffffffu, mbar_wait(bars + S_FULL + t, (j - rng.lo) & 1))) {
        if (lane == 0) atomicExch(error, 12);
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t s[KEYS];
#pragma unroll
      for (int q = 0; q < KEYS / 32; ++q) tmem_ld_32x32(tmem_s + 32 * q, *reinterpret_cast<uint32_t(*)[32]>(s + 32 * q));
      tmem_wait_ld();
      if constexpr (SHAPED) {  // in log2 units from here on; the slope's distance counted from the block's first key
        const float away = slope * (float)(pos - key0);
        const float2 slope2 = make_float2(slope, slope), away2 = make_float2(-away, -away);
        auto two = [&](int i) { return make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])); };
        auto keep = [&](int i, float2 x) {  // less the slope's share
          x = __ffma2_rn(slope2, make_float2((float)i, (float)(i + 1)), x);
          s[i] = __float_as_uint(x.x);
          s[i + 1] = __float_as_uint(x.y);
        };
        if constexpr (SHAPE == 2) {
          if (!loud) {
            float most = 0.f;
            if (!whole) {  // by the scores that count alone: a row's bits do not depend on what lies in pages and rows that it does not see
#pragma unroll
              for (int i = 0; i < KEYS; ++i)
                if ((unsigned)i - first > span) s[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < KEYS; i += 2) most = fmaxf(fmaxf(most, fabsf(__uint_as_float(s[i]))), fabsf(__uint_as_float(s[i + 1])));
            loud = __any_sync(0xffffffffu, valid && most > ex.small);
          }
          if (loud) {
#pragma unroll
            for (int i = 0; i < KEYS; i += 2) {
              float2 x = __fmul2_rn(two(i), scale2);
              x.x = ex.cap_log2 * (1.f - __fdividef(2.f, 1.f + fast_exp2(x.x * ex.in_cap)));
              x.y = ex.cap_log2 * (1.f - __fdividef(2.f, 1.f + fast_exp2(x.y * ex.in_cap)));
              keep(i, __fadd2_rn(x, away2));
            }
          } else {
            // tanh(u) = u + u z P(z), z = u^2, for |u| up to 0.65: the series' terms from u^3 on divided by u^3, fitted in Chebyshev
            // points over z; off by at most 9.4e-8 of tanh(u) in float32 (the form above by 1.7e-7 of 1). Scores that are small beside the
            // cap are the rule where queries and keys are normalised, and the exponentials' unit, which would do three things a score, does
            // one: 2,048 tokens of 16 heads behind a cap of 30, 94 us and 84 here.
            const float2 into = make_float2(ex.in_tanh, ex.in_tanh), cap2 = make_float2(ex.cap_log2, ex.cap_log2);
            constexpr float P[5] = {-0.333333284f, 0.133326009f, -0.0538258478f, 0.0208813194f, -0.00593298022f};
#pragma unroll
            for (int i = 0; i < KEYS; i += 2) {
              const float2 u = __fmul2_rn(two(i), into), z = __fmul2_rn(u, u);
              float2 q = make_float2(P[4], P[4]);
#pragma unroll
              for (int k = 3; k >= 0; --k) q = __ffma2_rn(q, z, make_float2(P[k], P[k]));
              keep(i, __ffma2_rn(__ffma2_rn(__fmul2_rn(u, z), q, u), cap2, away2));
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < KEYS; i += 2) keep(i, __ffma2_rn(two(i), scale2, away2));
        }
      }
      if (!whole) {
#pragma unroll
        for (int i = 0; i < KEYS; ++i)
          if ((unsigned)i - first > span) s[i] = unseen;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < KEYS; i += 8)
#pragma unroll
          for (int q = 0; q < 4; ++q) mx4[q] = fmaxf(fmaxf(mx4[q], __uint_as_float(s[i + q])), __uint_as_float(s[i + 4 + q]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const float m_new = fmaxf(m, SHAPED ? mx : mx * scale_size);
      const bool outgrown = valid && m != -INFINITY && m_new - m > RESCALE_STEP;
      if (__any_sync(0xffffffffu, outgrown)) {
        // the warp moves its rows' reference maxima and scales its rows of O; the block's P.V has not been issued and the
        // one before it is complete (S of this block came after it), so nothing else touches these rows of O
        const float alpha = m == -INFINITY ? 1.f : fast_exp2(m - m_new);
        // a row that starts from a sink may outgrow it in the tile's first block, when there is no O yet
#pragma unroll 1
        for (int c0 = 0; c0 < ((WIDE && j == rng.lo) ? 0 : D); c0 += 32) {
          uint32_t o[32];
          tmem_ld_32x32(tmem_o + c0, o);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(tmem_o + c0, o);
        }
        l2.x *= alpha;
        l2.y *= alpha;
        m = m_new;
      } else if (m == -INFINITY) {
        m = m_new;  // no key seen before this block: O and the sums are still zero
      }
      const float m_safe = m == -INFINITY ? 0.f : m;
      const float2 minus_m = make_float2(-m_safe, -m_safe);
      // A block's weights are added up by themselves: thousands of them one by one onto the row's sum, which all round the same way
      // where the weights are alike, drift by up to 1e-4 at 16,384 keys
      float2 sum = make_float2(0.f, 0.f);
#pragma unroll
      for (int i0 = 0; i0 < KEYS; i0 += 32) {
        uint32_t pk[16], pl[WIDE ? 16 : 1];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float2 x = make_float2(__uint_as_float(s[i0 + i]), __uint_as_float(s[i0 + i + 1]));
          x = SHAPED ? __fadd2_rn(x, minus_m) : __ffma2_rn(x, scale2, minus_m);
          const float2 p = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          sum = __fadd2_rn(sum, p);
          const __nv_bfloat162 h = __floats2bfloat162_rn(p.x, p.y);
          const uint32_t hi = *reinterpret_cast<const uint32_t*>(&h);
          pk[i / 2] = hi;
          if constexpr (WIDE) {
            const float2 rest = __fadd2_rn(p, make_float2(-__uint_as_float(hi << 16), -__uint_as_float(hi & 0xffff0000u)));
            const __nv_bfloat162 d = __floats2bfloat162_rn(rest.x, rest.y);
            pl[i / 2] = *reinterpret_cast<const uint32_t*>(&d);
          }
        }
        tmem_st_32x16(tmem_s + i0 / 2, pk);
        if constexpr (WIDE) tmem_st_32x16(tmem_s + KEYS / 2 + i0 / 2, pl);
      }
      l2 = __fadd2_rn(l2, sum);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + P_READY + t);
    }
    if (rng.lo <= rng.hi) {  // the same for every thread of the tile's four warps
      // O_t, divided by the row sums and rounded, goes through shared memory: a thread holds a row, and rows are 2 * D bytes
      // apart at best in the output. It is staged in the tile's query buffer, which its MMAs are done with, in the query
      // tile's own layout (128-byte swizzle), and leaves as the query tile came: one tiled store per 64-wide block of the
      // head when the tile is whole, else 16-byte pieces by all threads of the tile, consecutive threads storing consecutive
      // pieces (the rows of a token lie side by side in the output).
      const bool fine = ok && __all_sync(0xffffffffu, mbar_wait(bars + O_DONE + t, 0));
      unsigned char* stage = q_s + t * TILE_BYTES;
      if (fine) {
        tc_fence_after();
        int row = R;
        asm volatile("" : "+r"(row));  // its token and head are worked out again: they are not kept in registers through the walk
        const int tok = row / G, head = kh * G + row % G;
        float inv = valid ? (WIDE ? ex.out_scale : 1.0f) / (l2.x + l2.y) : 0.f;
        if (WIDE && ex.gate_mode == 1 && valid)
          inv /= 1.0f + expf(-__bfloat162float(ex.gate[(size_t)(row0 + tok) * ex.gate_stride + head]));
        if (WIDE && ex.gate_mode == 2) {
          // a gate per element: eight columns at a time, a loop of its own (unrolled into the other one it was code of 50 KB
          // that every block jumped over, 3 to 9 us)
          const bf16* g = ex.gate + (size_t)(row0 + tok) * ex.gate_stride + (size_t)head * D;
          const bool pieces = valid && ex.gate_stride % 8 == 0 && ((uintptr_t)ex.gate & 15) == 0;
#pragma unroll 2
          for (int c0 = 0; c0 < D; c0 += 8) {
            uint32_t o[8];
            tmem_ld_32x8(tmem_o + c0, o);
            uint4 gv = make_uint4(0, 0, 0, 0);
            if (pieces) gv = *reinterpret_cast<const uint4*>(g + c0);
            else if (valid) {
              bf16* e = reinterpret_cast<bf16*>(&gv);
              for (int i = 0; i < 8; ++i) e[i] = g[c0 + i];
            }
            tmem_wait_ld();
            const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&gv);
            uint4 pk;
            __nv_bfloat162* pp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              pp[e] = __floats2bfloat162_rn(__uint_as_float(o[2 * e]) / (1.0f + expf(-__low2float(g2[e]))) * inv,
                                            __uint_as_float(o[2 * e + 1]) / (1.0f + expf(-__high2float(g2[e]))) * inv);
            *reinterpret_cast<uint4*>(stage + (c0 / 64) * SUB + swz(r, (c0 / 8) % 8)) = pk;
          }
        } else {
#pragma unroll
          for (int c0 = 0; c0 < D; c0 += 32) {
            uint32_t o[32];
            tmem_ld_32x32(tmem_o + c0, o);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
              uint4 pk;
              __nv_bfloat162* pp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
              for (int e = 0; e < 4; ++e)
                pp[e] = __floats2bfloat162_rn(__uint_as_float(o[c + 2 * e]) * inv, __uint_as_float(o[c + 2 * e + 1]) * inv);
              const int piece = (c0 + c) / 8;
              *reinterpret_cast<uint4*>(stage + (piece / 8) * SUB + swz(r, piece % 8)) = pk;
            }
          }
        }
        fence_async_smem();
      } else if (lane == 0) {
        if (ok) atomicExch(error, 13);
        gave_up[t] = 1;
      }
      asm volatile("bar.sync %0, 128;" ::"r"(1 + t) : "memory");  // the tile's four warps
      if (!gave_up[t]) {
        const int row_begin = pair_row + t * rows;
        if (q_by_tma && row_begin + rows <= n_rows) {
          if (quad == 0 && lane == 0) {
#pragma unroll
            for (int h = 0; h < DB; ++h) tma_store_3d(&map_o, stage + h * SUB, h * 64, kh * G, row0 + row_begin / G);
            tma_store_commit();
            tma_store_wait_read();  // shared memory is given up when the block ends
          }
        } else {
#pragma unroll 4
          for (int k = 0; k < ROWS * (D / 8) / 128; ++k) {
            const int p = quad * 32 + lane + 128 * k;
            const int row = p / (D / 8), piece = p % (D / 8);
            const int R = row_begin + row;
            if (row < rows && R < n_rows)
              *reinterpret_cast<uint4*>(out + (size_t)(row0 + R / G) * (WIDE ? ex.out_stride : HQ * D) + (size_t)(kh * G + R % G) * D + piece * 8) =
                  *reinterpret_cast<const uint4*>(stage + (piece / 8) * SUB + swz(row, piece % 8));
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

constexpr size_t SMEM_BYTES = 6 * TILE_BYTES + 1024 + N_BARS * 8 + 64 + PAGE_IDS * sizeof(int) + 16;

template <bool WIDE, int SHAPE>
int launch_tcgen05(bf16* out, const bf16* q, int q_stride, int HQ, int HKV, const int* seq_slot, const int* seq_start,
                   const int* seq_qlen, const int* cu_q, const int* table, int width, const void* k_cache, const void* v_cache,
                   int n_pages, int n_seqs, int max_q_len, int total_rows, float scale, int window, int* error, const Extras& ex,
                   cudaStream_t stream) {
  const int G = HQ / HKV;
  // The query tiles come and go by TMA where whole tokens (G rows each) fill most of a tile; a tile then has that many rows.
  // Fetched by the threads, the two tiles take 8 us at G of 5 where TMA takes 2 (of 30 for a block with twelve blocks of keys), so the
  // rows left empty cost less down to 112 of 128, and down to 96 where the shorter tiles make no more rounds of one block an SM. One
  // prompt of 2,048, one kv head of 128, threads / TMA: G of 5 (125 rows, 8 kv heads) 80 / 61 us, 25 (125) 45 / 41, 28 (112) 50 / 45, 22 (110) 45 /
  // 41, 26 (104) 47 / 45; three rounds for two: 37 (111) 61 / 63, 33 (99) 57 / 63 (heads of 64: 47 / 57), but 700 tokens, one round, 26 / 21.
  const int whole = G <= ROWS ? ROWS / G * G : 0;
  auto rounds = [&](int rows_a_tile) { return (((long long)max_q_len * G + 2 * rows_a_tile - 1) / (2 * rows_a_tile) * HKV * n_seqs + 147) / 148; };
  const int q_by_tma = whole >= 112 || (whole >= 96 && rounds(whole) <= rounds(ROWS)) ? 1 : 0;
  const int tile_rows = q_by_tma ? whole : ROWS;
  const long long tiles = ((long long)max_q_len * G + 2 * tile_rows - 1) / (2 * tile_rows);
  if (tiles * HKV > 0x7fffffffLL || n_seqs > 65535) return -3;
  CUtensorMap map_k, map_v;
  const long long rows = (long long)n_pages * HKV * KRK_PAGE;
  int rc = make_map_bf16(&map_k, k_cache, rows, D, D, 64);
  if (rc) return rc;
  rc = make_map_bf16(&map_v, v_cache, rows, D, D, 64);
  if (rc) return rc;
  CUtensorMap map_q = map_k, map_o = map_k;
  if (q_by_tma) {
    rc = make_map_bf16_3d(&map_q, q, D, HQ, total_rows, D, q_stride, G, tile_rows / G);
    if (rc) return rc;
    rc = make_map_bf16_3d(&map_o, out, D, HQ, total_rows, D, ex.out_stride, G, tile_rows / G);
    if (rc) return rc;
  }
  if (scale == 0.f) scale = 1e-30f;  // weights of zero are made by scores of minus infinity: the scale must not be zero
  auto kern = attention_tcgen05_kernel<WIDE, SHAPE>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  kern<<<dim3((unsigned)(tiles * HKV), n_seqs, 1), THREADS, SMEM_BYTES, stream>>>(
      map_k, map_v, map_q, map_o, q_by_tma, tile_rows, out, q, q_stride, HQ, HKV, seq_slot, seq_start, seq_qlen, cu_q, table, width,
      scale * LOG2E, window, error, ex);
  KRK_CHECK_LAUNCH();
  return 0;
}

}  // namespace

// Same arguments as krk_attention_prefill plus the cache's number of pages and the number of rows of qkv
// (for the TMA maps) and the device error word. The keys and values of the step's own rows must be in the cache already.
KRK_API int krk_attention_prefill_tcgen05(void* out, const void* qkv, int q_stride, int HQ, int HKV,
                                          const int* seq_slot, const int* seq_start, const int* seq_qlen,
                                          const int* cu_q, const int* table, int width, const void* k_cache,
                                          const void* v_cache, int n_pages, int n_seqs, int max_q_len, int total_rows,
                                          float scale, int window, int* error, cudaStream_t stream) {
  if (n_seqs == 0 || max_q_len == 0) return 0;
  if ((q_stride % 8) || ((uintptr_t)qkv & 15) || ((uintptr_t)out & 15)) return -2;
  Extras ex = {};
  ex.out_stride = HQ * D;
  return launch_tcgen05<false, 0>((bf16*)out, (const bf16*)qkv, q_stride, HQ, HKV, seq_slot, seq_start, seq_qlen, cu_q, table, width,
                                      k_cache, v_cache, n_pages, n_seqs, max_q_len, total_rows, scale, window, error, ex, stream);
}

// krk_sink_window_prefill (attention_mma.cu) on the 5th-generation tensor cores: the same arguments plus the cache's number of
// pages, the number of rows of the queries and the error word, less the kept first keys, which it does not take. -2: rows or
// columns off 16-byte boundaries, or a scale that is not positive (maxima are taken before it).
KRK_API int krk_sink_prefill_tcgen05(void* out, int out_stride, float out_scale, const void* q, int q_stride, int HQ, int HKV,
                                     const float* sink, const int* seq_slot, const int* seq_start, const int* seq_qlen,
                                     const int* cu_q, const int* table, int width, const void* k_cache, const void* v_cache,
                                     int n_pages, int n_seqs, int max_q_len, int total_rows, float scale, int window, const void* gate,
                                     int gate_stride, int gate_mode, const float* slopes, float softcap, int* error,
                                     cudaStream_t stream) {
  if (n_seqs == 0 || max_q_len == 0) return 0;
  if (q_stride % 8 || out_stride % 8 || ((uintptr_t)q & 15) || ((uintptr_t)out & 15) || !(scale > 0.f)) return -2;
  Extras ex = {};
  ex.sink = sink; ex.slopes = slopes; ex.out_scale = out_scale; ex.out_stride = out_stride;
  ex.cap_log2 = softcap * LOG2E; ex.in_cap = softcap > 0.f ? 2.f / softcap : 0.f;
  ex.in_tanh = softcap > 0.f ? scale / softcap : 0.f; ex.small = softcap > 0.f ? 0.65f * (softcap / scale) : 0.f;
  ex.gate = (const bf16*)gate; ex.gate_stride = gate_stride; ex.gate_mode = gate ? gate_mode : 0;
  auto go = softcap > 0.f ? launch_tcgen05<true, 2> : slopes ? launch_tcgen05<true, 1> : launch_tcgen05<true, 0>;
  return go((bf16*)out, (const bf16*)q, q_stride, HQ, HKV, seq_slot, seq_start, seq_qlen, cu_q, table, width, k_cache, v_cache, n_pages,
            n_seqs, max_q_len, total_rows, scale, window, error, ex, stream);
}

#endif  // head sizes served by this kernel
