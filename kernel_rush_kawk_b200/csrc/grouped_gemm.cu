// The routed experts' products of many rows in one launch on the 5th-generation tensor cores, the rows of an expert
// wherever the routing put their number: C[r, :] = act(A[r, :] W_e^T) for the rows r of expert e, offsets[e] <= r <
// offsets[e + 1], W [E, N, K]. Gated: W [E, 2N, K] holds every expert's gate rows and then its up rows, and C = act(g, u) with g
// and u multiplied by the row's weight first where there is one (a router that weighs an expert's input). The offsets stay on the device.
//
// Bound by the weights' bytes (64 experts of 2,048 x 1,408, 2,048 rows of six: 738 and 369 MB, 113 and 56 us, against 88 and 44 us of
// products). Blocks work in pairs (cta_group::2): 256 rows of W_e are the product's M, each block's shared memory holding 128 of them,
// and an expert's rows are its N, 32 to 256 of them, each block holding half. So what a product costs follows the rows that there are,
// in steps of 32 instead of 128, every weight is fetched once for up to 256 rows, an SM takes in 16 KB of weights and its half of the rows
// for as much work as a block alone does with 16 and 32 KB, and a tile's accumulator fills half of tensor memory: while its eight
// reading warps turn one tile into C, the next one is multiplied. Pairs stay and walk the tiles (74 pairs, the tiles of a row tile
// side by side), so that loads go on over the seams; products of few tiles take single blocks (by_blocks, below). With a single-block tile of
// 256 rows by 256 columns, launched per tile, the two products took 195 and 105 us, now 163 and 85; 4,000 rows 352 and 187 -> 280 and 150; 200 rows, where nothing but the weights
// counts, 163 and 81 -> 120 and 65. Asking weights into L2 ahead of the ring was measured and is slower (eight blocks of k: 219
// against 189 us, single blocks); rows in copies of 16 instead of 128, 64, 32 and 16: 200 against 167 us.
//
// Warp 0 of either block drives TMA (64 elements of K a stage, 128-byte swizzle) and counts on the first block's barriers; warp 1 of
// the first block issues tcgen05.mma for both; warps 2..9 read the accumulator back. There a lane is a column of C and what a thread
// holds are rows, so a warp turns 32 x 32 of them through a patch of shared memory. Gated, gate and up rows alternate in the tile, so
// that neighbouring lanes hold a column's two products. Rows beyond the expert's, the next one's or zeros, are not stored.
// Every wait is bounded: one that runs out sets the error word, and the blocks leave after freeing their tensor memory.
#include "mma.cuh"  // times_logistic
#include "tcgen05.cuh"

namespace {

using namespace tc;

constexpr int BK = 64, UMMA_K = 16;
constexpr int SMS = 148;
constexpr int READERS = 8;  // warps that read accumulators: two to a quarter of tensor memory's lanes
constexpr int THREADS = 64 + 32 * READERS;

// SILU: silu(g) u of the two products as they would have been stored; CLAMPED:
// g' = min(g, limit), u' = clamp(u, -limit, limit), g' sigmoid(slope g') (u' + 1), nothing rounded before the end
enum Form { SILU, CLAMPED, PLAIN, SQUARED };

// SHORT: single-token steps, which may come here or, with fewer pairs, to few_experts.cu, are as exact here as there. There eight warps share
// a sum's k, and the activation is expf and a division. The tensor cores cut off every sum: one accumulator for all of 2,048 k left 2.0e-3
// of the activations next to the correctly rounded ones. So tiles are of up to 32 rows and have eight accumulators, a block of k each in
// turn, which are added when they are read back.
constexpr int SHORT_ROWS = 32, SHORT_SUMS = 8;

template <Form FORM, bool SHORT>
__device__ __forceinline__ float gated_act_of(float g, float u, float limit, float slope) {
  if (FORM == CLAMPED) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    if (SHORT) return times_logistic(g, slope * g) * (u + 1.0f);
    return __fdividef(g, 1.0f + __expf(-slope * g)) * (u + 1.0f);
  }
  g = round_to<bf16>(g);
  if (SHORT) return silu_near(g) * round_to<bf16>(u);
  return __fdividef(g, 1.0f + __expf(-g)) * round_to<bf16>(u);
}

constexpr uint32_t W_BYTES = 128 * BK * 2;      // a block's half of the pair's weights
constexpr int BOXES = 4, BIGGEST = 128;         // rows come in copies of 128, 64, 32 and 16: many small ones would bound the kernel
struct RowMaps { CUtensorMap of[BOXES]; };
constexpr int BUF_COLS = 256;                   // tensor memory of an accumulator; there are two
constexpr int PATCH_PITCH = 80;                 // bytes of a row of a warp's patch for the transpose: 16-byte reads of 32 rows meet no bank twice
constexpr int PATCH_BYTES = 32 * PATCH_PITCH;
constexpr int RING_BYTES = 200 * 1024, MOST_STAGES = 10;
constexpr size_t SMEM_BYTES = 1024 + (size_t)RING_BYTES + READERS * PATCH_BYTES + (2 * MOST_STAGES + 5) * 8 + 16;

// Which expert and rows the row tile `y` is, over all experts' row tiles in order: an expert's rows in as few equal tiles of up to
// `most` rows as hold them, in multiples of 32. A warp's own: 32 experts' tile counts at a time, kept between calls, since a
// block asks for its tiles in ascending order.
struct RowTiles {
  const int* offsets;
  int E, most, e0, before, lo, hi, count, incl;  // experts e0 + lane; `before`: row tiles of the experts before e0
  __device__ RowTiles(const int* offsets_, int E_, int most_) : offsets(offsets_), E(E_), most(most_), e0(0), before(0) { load(); }
  __device__ void load() {
    const int lane = threadIdx.x & 31, mine = e0 + lane;
    lo = mine < E ? offsets[mine] : 0;
    hi = mine < E ? offsets[mine + 1] : 0;
    incl = count = tiles_of(hi - lo);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int p = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += p;
    }
  }
  __device__ int tiles_of(int rows) const { return (rows + most - 1) / most; }
  __device__ int each(int rows) const { return rows ? ((rows + tiles_of(rows) - 1) / tiles_of(rows) + 31) / 32 * 32 : 0; }
  // rows of the biggest tile
  __device__ int biggest() const {
    int n = 32;
    for (int i = threadIdx.x & 31; i < E; i += 32) n = max(n, each(offsets[i + 1] - offsets[i]));
    return __reduce_max_sync(0xffffffffu, n);
  }
  // false: there are not so many
  __device__ bool find(int y, int& e, int& m0, int& rows) {
    for (int all = __shfl_sync(0xffffffffu, incl, 31); y - before >= all; all = __shfl_sync(0xffffffffu, incl, 31)) {
      if (e0 + 32 >= E) return false;
      before += all;
      e0 += 32;
      load();
    }
    const int t = y - before, first = incl - count;
    const int src = __ffs(__ballot_sync(0xffffffffu, t < incl && t >= first)) - 1;
    const int rows_each = each(hi - lo), from = lo + (t - first) * rows_each;
    e = e0 + src;
    m0 = __shfl_sync(0xffffffffu, from, src);
    rows = __shfl_sync(0xffffffffu, min(rows_each, hi - from), src);
    return true;
  }
};

template <Form FORM, bool SHORT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS)
grouped_gemm_kernel(const __grid_constant__ RowMaps maps_a, const __grid_constant__ CUtensorMap map_w, bf16* __restrict__ C,
                    const int* __restrict__ offsets, int E, int N, int K, int most, const float* __restrict__ row_weights,
                    float limit, float slope, int* __restrict__ error) {
  constexpr bool GATED = FORM == SILU || FORM == CLAMPED;
  constexpr int BC = GATED ? 64 : 128;  // columns of C a block makes of a tile; the pair twice as many
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* patches = tiles + RING_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(patches + READERS * PATCH_BYTES);  // the first block's: copies of both have landed
  uint64_t* empty_bar = full_bar + MOST_STAGES;   // either block's: the products have read a stage
  uint64_t* acc_full = empty_bar + MOST_STAGES;   // either block's
  uint64_t* acc_empty = acc_full + 2;        // the first block's: the reading warps of both are through
  uint64_t* drain_bar = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  int* issued = reinterpret_cast<int*>(tmem_slot + 1);  // blocks of k that were asked for, where a wait ran out; else -1
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < MOST_STAGES; ++s) {
      mbar_init(full_bar + s, 1);
      mbar_init(empty_bar + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + b, 1);
      mbar_init(acc_empty + b, 2 * READERS);
    }
    mbar_init(drain_bar, 1);
    *issued = -1;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BUF_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the other block's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();
  grid_dependency_wait();
  RowTiles tiles_of(offsets, E, most);
  const uint32_t stage_bytes = W_BYTES + (uint32_t)tiles_of.biggest() / 2 * BK * 2;
  const int stages = min(MOST_STAGES, (int)(RING_BYTES / stage_bytes));
  const int k_blocks = (K + BK - 1) / BK, cols = (N + 2 * BC - 1) / (2 * BC);
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  int e, m0, rows;

  if (warp == 0) {
    int s = 0, asked = 0;
    uint32_t parity = 1;  // of the round before: a first round finds its stages empty
    bool ok = true;
    for (int t = pair; ok && tiles_of.find(t / cols, e, m0, rows); t += pairs) {
      if (lane == 0) {
        const int half = (rows + 31) / 32 * 16;  // rows that each block of the pair brings
        const int f0 = (t % cols * 2 + (int)rank) * BC, first = m0 + (int)rank * half;
        const uint32_t bytes = 2 * (W_BYTES + (uint32_t)half * BK * 2);
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(empty_bar + s, parity)) {
            atomicExch(error, 3);
            *issued = asked;
            ok = false;
            break;
          }
          unsigned char* stage = tiles + s * stage_bytes;
          const uint32_t bar = cluster_address(full_bar + s, 0);
          if (rank == 0) mbar_expect_tx(full_bar + s, bytes);
          if (GATED) tma_load_3d_pair(stage, &map_w, bar, kb * BK, 0, 2 * e * N + f0);
          else tma_load_2d_pair(stage, &map_w, bar, kb * BK, e * N + f0);
          int r = 0;
#pragma unroll
          for (int b = 0; b < BOXES; ++b)
            if (half & (BIGGEST >> b)) {
              tma_load_2d_pair(stage + W_BYTES + r * (BK * 2), &maps_a.of[b], bar, kb * BK, first + r);
              r += BIGGEST >> b;
            }
          ++asked;
          if (++s == stages) { s = 0; parity ^= 1; }
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
    }
    if (lane == 0 && ok)  // the last stages' releases, too, have arrived before the block leaves
      for (int i = 0; i < stages; ++i) {
        if (!mbar_wait(empty_bar + s, parity)) {
          atomicExch(error, 3);
          *issued = asked;
          break;
        }
        if (++s == stages) { s = 0; parity ^= 1; }
      }
  } else if (warp == 1) {
    int s = 0, buf = 0;
    uint32_t parity = 0, acc_parity = 1;
    bool ok = rank == 0;
    for (int t = pair; ok && tiles_of.find(t / cols, e, m0, rows); t += pairs) {
      if (lane == 0) {
        const uint32_t idesc = umma_idesc(256, (rows + 31) / 32 * 32);
        const uint32_t acc = tmem_base + (uint32_t)buf * BUF_COLS;
        ok = mbar_wait(acc_empty + buf, acc_parity);  // both blocks have read what was there
        tc_fence_after();
        for (int kb = 0; ok && kb < k_blocks; ++kb) {
          if (!mbar_wait(full_bar + s, parity)) {
            ok = false;
            break;
          }
          tc_fence_after();
          unsigned char* stage = tiles + s * stage_bytes;
          const uint64_t w_desc = umma_desc(stage), r_desc = umma_desc(stage + W_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t adv = (uint64_t)((k * UMMA_K * 2) >> 4);
            if (SHORT) umma_bf16_pair(acc + kb % SHORT_SUMS * SHORT_ROWS, w_desc + adv, r_desc + adv, idesc, (kb >= SHORT_SUMS || k > 0) ? 1u : 0u);
            else umma_bf16_pair(acc, w_desc + adv, r_desc + adv, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_pair(empty_bar + s);
          if (++s == stages) { s = 0; parity ^= 1; }
        }
        if (ok) {
          umma_commit_pair(acc_full + buf);
        } else {  // products on their way end before tensor memory is freed
          atomicExch(error, 4);
          umma_commit_pair(drain_bar);
          mbar_wait(drain_bar, 0, WAIT_LIMIT_NS / 20);
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      buf ^= 1;
      acc_parity ^= buf == 0;
    }
  } else {
    const int quarter = warp & 3;
    unsigned char* patch = patches + (warp - 2) * PATCH_BYTES;
    int buf = 0;
    uint32_t parity = 0;
    for (int t = pair; tiles_of.find(t / cols, e, m0, rows); t += pairs) {
      if (!mbar_wait(acc_full + buf, parity)) {
        if (lane == 0) atomicExch(error, 5);
        break;
      }
      __syncwarp();
      tc_fence_after();
      const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * BUF_COLS;
      constexpr int MINE = BC / 4;  // features of this warp
      const int f0 = (t % cols * 2 + (int)rank) * BC + quarter * MINE;
      if (f0 < N) {
        for (int c0 = (warp - 2) / 4 * 32; c0 < rows; c0 += 32 * (READERS / 4)) {
          uint32_t v[32];
          tmem_ld_32x32(acc + (uint32_t)c0, v);
          const int row = m0 + c0 + lane;
          const bool live = c0 + lane < rows;
          float by = 1.f;
          if (GATED && row_weights && live) by = row_weights[row];
          tmem_wait_ld();
          if constexpr (SHORT) {
#pragma unroll 1
            for (int i = 1; i < min(SHORT_SUMS, k_blocks); ++i) {
              uint32_t more[32];
              tmem_ld_32x32(acc + (uint32_t)(i * SHORT_ROWS), more);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(more[j]));
            }
          }
          if constexpr (GATED) {
            // an even lane has a feature's gate and the odd one after it the same feature's up: they share the rows, the even ones to
            // the even lane
            const bool odd = lane & 1;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float a = __uint_as_float(v[2 * j]), b = __uint_as_float(v[2 * j + 1]);
              const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
              float g = odd ? got : a, u = odd ? b : got;
              if (row_weights) {
                const float w = __shfl_sync(0xffffffffu, by, 2 * j + (odd ? 1 : 0));
                g *= w;
                u *= w;
              }
              *reinterpret_cast<bf16*>(patch + (2 * j + (odd ? 1 : 0)) * PATCH_PITCH + (lane >> 1) * 2) =
                  from_float<bf16>(gated_act_of<FORM, SHORT>(g, u, limit, slope));
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              float z = __uint_as_float(v[j]);
              if (FORM == SQUARED) {  // squared relu of the product as it would have been stored
                z = round_to<bf16>(z);
                z = z > 0.f ? z * z : 0.f;
              }
              *reinterpret_cast<bf16*>(patch + j * PATCH_PITCH + lane * 2) = from_float<bf16>(z);
            }
          }
          __syncwarp();
          if (live) {
            bf16* dst = C + (size_t)row * N + f0;
#pragma unroll
            for (int j = 0; j < MINE; j += 8)  // N is a multiple of 8
              if (f0 + j < N) *reinterpret_cast<uint4*>(dst + j) = *reinterpret_cast<const uint4*>(patch + lane * PATCH_PITCH + j * 2);
          }
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_address(acc_empty + buf, 0));
      buf ^= 1;
      parity ^= buf == 0;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (rank == 0 && threadIdx.x == 0 && *issued >= 0)  // copies on their way end before shared memory is given up
    for (int i = max(0, *issued - stages); i < *issued; ++i) mbar_wait(full_bar + i % stages, (uint32_t)(i / stages) & 1u, WAIT_LIMIT_NS / 20);
  __syncthreads();
  cluster_sync();  // neither block's barriers are signalled any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * BUF_COLS) : "memory");
  }
}

// The same by single blocks, 128 of an expert's rows against BN rows of its weights (gated: 128 gate rows and their up rows), a tile each: for
// products of few tiles, which pairs would do in fewer and larger pieces than the SMs are (by_blocks). The rows are the product's M here, so a
// lane is a row of C. Tile for tile the sums are the same bits.
constexpr int BLOCK_THREADS = 192, BLOCK_STAGES = 4;
constexpr uint32_t A_BYTES = 128 * BK * 2;

template <int BN> constexpr size_t block_smem() { return (size_t)BLOCK_STAGES * (A_BYTES + BN * BK * 2) + 1024 + (2 * BLOCK_STAGES + 1) * 8 + 16; }

template <Form FORM, int BN>
__global__ void __launch_bounds__(BLOCK_THREADS)
grouped_block_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, bf16* __restrict__ C,
                     const int* __restrict__ offsets, int E, int N, int K, const float* __restrict__ row_weights, float limit,
                     float slope, int* __restrict__ error) {
  constexpr bool GATED = FORM == SILU || FORM == CLAMPED;
  static_assert(!GATED || BN == 256, "a gate tile and an up tile of 128 rows each");
  constexpr int BC = GATED ? BN / 2 : BN;  // columns of C a block makes
  constexpr uint32_t STAGE_BYTES = A_BYTES + BN * BK * 2;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + (size_t)BLOCK_STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + BLOCK_STAGES;
  uint64_t* acc_bar = empty_bar + BLOCK_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  int* issued = reinterpret_cast<int*>(tmem_slot + 1);  // blocks of k that were asked for, where a wait ran out; else -1
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  grid_dependency_wait();
  RowTiles tiles_of(offsets, E, 128);
  int e, m0, rows;
  if (!tiles_of.find(blockIdx.y, e, m0, rows)) return;  // the same for the whole block
  const int n0 = blockIdx.x * BC, k_blocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < BLOCK_STAGES; ++s) {
      mbar_init(full_bar + s, 1);
      mbar_init(empty_bar + s, 1);
    }
    mbar_init(acc_bar, 1);
    *issued = -1;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();

  if (warp == 0 && lane == 0) {
    for (int kb = 0; kb < k_blocks; ++kb) {
      const int s = kb % BLOCK_STAGES;
      if (kb >= BLOCK_STAGES && !mbar_wait(empty_bar + s, ((kb / BLOCK_STAGES) - 1) & 1)) {
        atomicExch(error, 3);
        *issued = kb;
        break;
      }
      unsigned char* stage = tiles + (size_t)s * STAGE_BYTES;
      mbar_expect_tx(full_bar + s, STAGE_BYTES);
      tma_load_2d(stage, &map_a, full_bar + s, kb * BK, m0);
#pragma unroll
      for (int h = 0; h < BN / 128; ++h)
        tma_load_2d(stage + A_BYTES + h * (128 * BK * 2), &map_w, full_bar + s, kb * BK, GATED ? (2 * e + h) * N + n0 : e * N + n0 + 128 * h);
    }
  } else if (warp == 1 && lane == 0) {
    constexpr uint32_t idesc = umma_idesc(128, BN);
    for (int kb = 0; kb < k_blocks; ++kb) {
      const int s = kb % BLOCK_STAGES;
      if (!mbar_wait(full_bar + s, (kb / BLOCK_STAGES) & 1)) {
        atomicExch(error, 4);
        break;
      }
      tc_fence_after();
      unsigned char* stage = tiles + (size_t)s * STAGE_BYTES;
      const uint64_t a_desc = umma_desc(stage), b_desc = umma_desc(stage + A_BYTES);
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) {
        const uint64_t adv = (uint64_t)((k * UMMA_K * 2) >> 4);
        umma_bf16(tmem_base, a_desc + adv, b_desc + adv, idesc, (kb > 0 || k > 0) ? 1u : 0u);
      }
      umma_commit(empty_bar + s);
    }
    umma_commit(acc_bar);  // arrives even after a failed wait, so the epilogue moves on
  } else if (warp >= 2) {
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const bool ok = mbar_wait(acc_bar, 0);
    if (!ok && lane == 0) atomicExch(error, 5);
    __syncwarp();
    tc_fence_after();
    if (ok) {
      const float by = GATED && row_weights && row < rows ? row_weights[m0 + row] : 1.f;
#pragma unroll 1
      for (int c0 = 0; c0 < BC && n0 + c0 < N; c0 += 32) {
        uint32_t g[32], u[GATED ? 32 : 1];
        tmem_ld_32x32(acc + (uint32_t)c0, g);
        if constexpr (GATED) tmem_ld_32x32(acc + (uint32_t)(BC + c0), u);
        tmem_wait_ld();
        if (row < rows) {
          bf16* dst = C + (size_t)(m0 + row) * N + n0 + c0;
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              v[i] = __uint_as_float(g[j + i]);
              if constexpr (GATED) {
                v[i] = gated_act_of<FORM, false>(by * v[i], by * __uint_as_float(u[j + i]), limit, slope);
              } else if (FORM == SQUARED) {  // squared relu of the product as it would have been stored
                const float z = round_to<bf16>(v[i]);
                v[i] = z > 0.f ? z * z : 0.f;
              }
            }
            uint4 pk;
            __nv_bfloat162* two = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
            for (int q = 0; q < 4; ++q) two[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
            if (n0 + c0 + j < N) *reinterpret_cast<uint4*>(dst + j) = pk;  // N is a multiple of 8
          }
        }
        __syncwarp();
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (threadIdx.x == 0 && *issued >= 0)  // copies on their way end before shared memory is given up
    for (int i = max(0, *issued - BLOCK_STAGES); i < *issued; ++i)
      mbar_wait(full_bar + i % BLOCK_STAGES, (uint32_t)(i / BLOCK_STAGES) & 1u, WAIT_LIMIT_NS / 20);
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(BN) : "memory");
  }
}

// Whether single blocks are the faster ones: where their tiles, an expert's last one half filled, are one round over the SMs (two of a
// short k, or of up to 1,024 where the second is nearly full), and the pairs' larger ones would be a second round that is nearly empty
// (gated, whose epilogue takes a single block's lanes longer), or leave SMs idle: an expert's rows are a tile's or nearly, or its
// columns half of one. Pairs and blocks, us: gated, 8 experts of 512 x 1,024, 2,048 rows 13.9 and 17.1, 4,096 rows 20.8 and 13.4, of 16
// 22.2 and 35.7; plain, 16 of 512 x 1,024, 1,024 rows 10.4 and 11.2, 2,048 11.9 and 10.3, 4,096 14.5 and 11.7, 8,192 21.4 and 14.2; 16
// of 1,024 x 512, 8,192 rows 23.7 and 18.7; of 1,024 x 1,024, 4,096 rows 23.2 and 24.4, 8,192 27.8 and 25.4; 8 of 1,024 x 512,
// 4,096 rows 16.6 and 8.4; 64 of 128 x 512, 64 rows 7.7 and 5.6, 8,192 10.4 and 6.5.
bool by_blocks(int rows, int E, int N, int K, bool gated) {
  const int experts = rows < E ? rows : E;
  const long long cols = (N + (gated || N <= 128 ? 127 : 255)) / (gated || N <= 128 ? 128 : 256);
  const long long blocks = (rows / 128 + (experts + 1) / 2) * cols;
  const bool second = !gated && (K <= 512 || (K <= 1024 && blocks > 9 * SMS / 5));
  if (blocks > (second ? 2 * SMS : SMS)) return false;
  if (gated) return (rows / 256 + experts / 2) * cols > SMS / 2;
  return N <= 128 || rows >= 96LL * E;
}

template <Form FORM, int BN>
int launch_blocks(bf16* C, const bf16* A, const bf16* W, const int* offsets, int rows, int E, int N, int K, const float* row_weights,
                  float limit, float slope, int* error, cudaStream_t stream) {
  constexpr bool GATED = FORM == SILU || FORM == CLAMPED;
  CUtensorMap map_a, map_w;
  int rc = make_map_bf16(&map_a, A, rows, K, K, 128);
  if (rc) return rc;
  rc = make_map_bf16(&map_w, W, (long long)E * N * (GATED ? 2 : 1), K, K, 128);
  if (rc) return rc;
  auto kern = grouped_block_kernel<FORM, BN>;
  const cudaError_t set = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)block_smem<BN>());
  if (set != cudaSuccess) return (int)set;
  constexpr int BC = GATED ? BN / 2 : BN;
  const long long row_tiles = rows / 128 + (rows < E ? rows : E);  // an expert leaves at most one tile partly filled
  if (row_tiles > 65535) return -3;
  return (int)launch_pdl(kern, dim3((unsigned)((N + BC - 1) / BC), (unsigned)row_tiles), dim3(BLOCK_THREADS), block_smem<BN>(), stream, map_a,
                         map_w, C, offsets, E, N, K, row_weights, limit, slope, error);
}

template <Form FORM, bool SHORT>
int launch_pairs(bf16* C, const bf16* A, const bf16* W, const int* offsets, int rows, int E, int N, int K, const float* row_weights,
                 float limit, float slope, int* error, cudaStream_t stream) {
  constexpr int most = SHORT ? SHORT_ROWS : 256;
  constexpr bool GATED = FORM == SILU || FORM == CLAMPED;
  RowMaps maps_a;
  CUtensorMap map_w;
  int rc;
  for (int b = 0; b < BOXES; ++b)
    if ((rc = make_map_bf16(&maps_a.of[b], A, rows, K, K, BIGGEST >> b))) return rc;
  // gated: rows [e 2 N + n] and, N rows further on, [e 2 N + N + n]: a box of 64 features brings each gate row and its up row in turn
  rc = GATED ? make_map_bf16_3d(&map_w, W, K, 2, 2LL * E * N - N, (long long)N * K, K, 2, 64)
             : make_map_bf16(&map_w, W, (long long)E * N, K, K, 128);
  if (rc) return rc;
  auto kern = grouped_gemm_kernel<FORM, SHORT>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int cols = (N + (GATED ? 127 : 255)) / (GATED ? 128 : 256);
  const long long work = (rows / most + (long long)(rows < E ? rows : E)) * cols;  // tiles at most: an expert leaves one partly filled
  if (work + SMS > 0x7fffffffLL) return -3;
  return (int)launch_pdl(kern, dim3((unsigned)(2 * work < SMS ? 2 * work : SMS)), dim3(THREADS), SMEM_BYTES, stream, maps_a, map_w, C,
                         offsets, E, N, K, most, row_weights, limit, slope, error);
}

}  // namespace

// C [rows, N] = act(A [rows, K] W_e^T) over the experts' rows (offsets int32 [E + 1] on the device; rows is the most there
// can be). act: -1 none, 5 squared relu. N and K multiples of 8, K at least 64, 16-byte aligned bases. `gated`: W [E, 2N, K],
// act 0 (silu) or 3 (clamped swish with its limit and slope), row_weights [rows] or null. `route` 0: pairs of blocks; 1: pairs or
// single blocks, by sizes; 2: a single-token step's tiles.
KRK_API int krk_grouped_gemm(void* C, const void* A, const void* W, const int* offsets, int rows, int E, int N, int K, int act,
                             int gated, int route, const float* row_weights, float limit, float slope, int* error,
                             cudaStream_t stream) {
  if (rows == 0 || N == 0 || E == 0) return 0;
  if (N % 8 || K % 8 || K < 64 || (((uintptr_t)A | (uintptr_t)W | (uintptr_t)C) & 15) || 2LL * E * N > 0x7fffffffLL) return -2;
  if (gated ? (act != 0 && act != 3) : ((act != -1 && act != 5) || row_weights)) return -2;
  auto with = [&](auto go) { return go((bf16*)C, (const bf16*)A, (const bf16*)W, offsets, rows, E, N, K, row_weights, limit, slope, error, stream); };
  const bool blocks = route == 1 && by_blocks(rows, E, N, K, gated), narrow = N <= 128, single = route == 2;
  if (gated && act == 3) return with(blocks ? launch_blocks<CLAMPED, 256> : single ? launch_pairs<CLAMPED, true> : launch_pairs<CLAMPED, false>);
  if (gated) return with(blocks ? launch_blocks<SILU, 256> : single ? launch_pairs<SILU, true> : launch_pairs<SILU, false>);
  if (act == 5)
    return with(blocks ? (narrow ? launch_blocks<SQUARED, 128> : launch_blocks<SQUARED, 256>) : single ? launch_pairs<SQUARED, true> : launch_pairs<SQUARED, false>);
  return with(blocks ? (narrow ? launch_blocks<PLAIN, 128> : launch_blocks<PLAIN, 256>) : single ? launch_pairs<PLAIN, true> : launch_pairs<PLAIN, false>);
}
