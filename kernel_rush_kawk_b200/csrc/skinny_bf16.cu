// Decode-time matrix product for few rows: out[M, N] = act(x)[M, K] * W[N, K]^T,
// bfloat16, M <= 16, with SwiGLU (or another gate, see the entry) folded into the epilogue.
//
// At decode the projections are pure weight streaming (the reference says so of
// its own skinny kernel, engine/kernels/gemm.py:1-10 of willzeng274/kernel-rush-kawk).
// Here the weights are the 16-row operand of the tensor-core instruction ("swap
// A and B"): a warp owns 16 output features (rows of W) and a slice of K; each
// lane reads 16 contiguous bytes of a weight row straight from global memory into
// the A fragment, the batch rows are the 8-wide B operand. The K index inside a
// 32-wide chunk is permuted identically for both operands (a dot product does not
// care), which is what lets one 16-byte load fill a fragment. No weight byte goes
// through shared memory. The warps of a block split K and reduce through shared
// memory in a fixed order, so results are reproducible.
//
// Epilogue (swiglu): rows n and N + n of W are gate and up; out = round(round(silu(round(g))) * round(u))
// (gemm.py:108-113).
//
// The residual add and the RMSNorm before a product stay a kernel of their own (elementwise.cu), although the reference
// folds them into its product (gemm.py:22-51): done in every block's prologue they stand between the block's first
// weights and its first use of them, while the separate kernel runs under the ring-fulls that these blocks have asked
// for already. Measured, a captured layer after 500 tokens, prologue against kernel: 4B shape 47.3 / 45.3 us at one
// row, 57.4 / 46.6 at two; 8B 79.0 / 74.0 and 84.8 / 75.6; 14B 128.4 / 121.1 and 139.8 / 123.1.
//
// A product with few output features (N of some thousands) has too few 16-row tiles to keep
// every SM's memory pipe full: what bounds a block is the bytes it has in flight, and one block
// of eight warps per SM holds 64 KB. Such products split K as well: the KSPLIT blocks of a
// thread-block cluster stream a quarter of K each for the same tile, five small blocks share an
// SM, and the partial sums meet in the first block's shared memory (distributed shared memory,
// added in block order, so the result does not depend on timing).
#include <cooperative_groups.h>

#define KRK_TRACE_OWNER  // with -DKRK_TRACE this file keeps the timeline buffer
#include "mma.cuh"

namespace {

constexpr int CHUNK = 32;        // k values per fragment load
constexpr int RING_LOADS = 8;    // 16-row tile chunks in flight per thread (32 bytes each)
// With two batch tiles whose rows ride in the ring (9 to 16 rows) a stage is a third larger, and
// at 8 loads an 8-warp block takes 131 KB of shared memory: one block per SM. Six keep two blocks per SM;
// a decode step at 16 sequences of the 4B shape: 2.79 ms against 3.08 ms with 8 (and 2.96 / 3.06 / 3.30 ms
// with 5 / 7 / 4; the library product: 2.83 ms).
constexpr int RING_LOADS_TWO_TILES = 6;
// five 4-warp blocks of a K-split product share an SM: 40 KB each with the ring, the reduction buffer and the inbox
constexpr int RING_LOADS_KSPLIT = 6, RING_LOADS_KSPLIT_TWO_TILES = 4;
template <int NT, int KSPLIT = 1, int RING = 0>
__host__ __device__ constexpr int ring_loads() {
  return RING > 0 ? RING : (KSPLIT > 1) ? (NT == 2 ? RING_LOADS_KSPLIT_TWO_TILES : RING_LOADS_KSPLIT)
                      : NT == 2 ? RING_LOADS_TWO_TILES : RING_LOADS;
}

// NT: 8-row batch tiles (1 or 2). RT: 16-row weight tiles per block; with SWIGLU the
// block streams RT gate tiles and RT up tiles.
//
// Weight bytes travel global -> shared memory with cp.async into a ring that is
// private to each thread: a thread later reads back exactly the 16-byte pieces it
// copied itself, so the ring needs no barrier, only cp.async.wait_group. The first
// ring-full of copies is issued before anything else (before the wait on the
// previous kernel), so the memory system is busy from the
// block's first instruction.
template <int WARPS, int NT, int RT, int SWIGLU, typename TOut, int KSPLIT = 1, int RING = 0>
__global__ void __launch_bounds__(WARPS * 32)
skinny_kernel(TOut* __restrict__ out, const bf16* __restrict__ x, const bf16* __restrict__ W,
              int M, int N, int K, float limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KRK_TRACE_DECL
  constexpr int THREADS = WARPS * 32;
  constexpr int TILES = SWIGLU ? 2 * RT : RT;  // 16-row weight tiles this block streams
  constexpr int STAGES = ring_loads<NT, KSPLIT, RING>() / TILES;
  constexpr int SLOTS = TILES * 2 + NT;          // 16-byte pieces per thread and stage: weights, and the batch rows
  constexpr size_t RING_BYTES = (size_t)STAGES * SLOTS * THREADS * 16;
  uint4* ring = reinterpret_cast<uint4*>(smem_raw);                                 // [STAGES][SLOTS][THREADS]
  float* red = reinterpret_cast<float*>(smem_raw + RING_BYTES);                       // [WARPS][TILES*NT*4*32]
  constexpr size_t RED_BYTES = (size_t)WARPS * TILES * NT * 4 * 32 * sizeof(float);
  float* inbox = reinterpret_cast<float*>(smem_raw + RING_BYTES + RED_BYTES);         // [KSPLIT - 1][outputs]
  static_assert(KSPLIT == 1 || !SWIGLU, "K is split only for the plain product");
  if (KSPLIT > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // "I have started"

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int ks = KSPLIT > 1 ? blockIdx.x % KSPLIT : 0;  // this block's part of K: its rank in the cluster

  // weight rows of this block's tiles, clamped so that edge tiles read valid memory
  const int n0 = (blockIdx.x / KSPLIT) * 16 * RT;
  const bf16* wrow[TILES][2];
#pragma unroll
  for (int s = 0; s < TILES; ++s) {
    const int tile_row = n0 + (s % RT) * 16 + (SWIGLU && s >= RT ? N : 0);
    const int limit = (SWIGLU && s >= RT ? 2 * N : N) - 1;
    wrow[s][0] = W + (size_t)min(tile_row + g, limit) * K + 8 * t;
    wrow[s][1] = W + (size_t)min(tile_row + g + 8, limit) * K + 8 * t;
  }
  const int n_chunks = K / CHUNK;
  const int per_block = (n_chunks + KSPLIT - 1) / KSPLIT;
  const int b_begin = ks * per_block, b_end = min(n_chunks, b_begin + per_block);
  const int per_warp = (max(0, b_end - b_begin) + WARPS - 1) / WARPS;
  const int c_begin = b_begin + warp * per_warp, c_end = min(b_end, c_begin + per_warp);
  const int nc = max(0, c_end - c_begin);

  // batch rows of the B fragments
  const bf16* xsrc[NT];
  bool xok[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int m = 8 * j + g;
    xok[j] = m < M;
    xsrc[j] = x + (size_t)min(m, M - 1) * K + 8 * t;
  }

  const uint64_t stream_policy = l2_evict_first_policy();
  auto issue_w = [&](int i) {  // weights of chunk i of this warp's slice into stage i % STAGES
    if (i < nc) {
      uint4* dst = ring + ((size_t)(i % STAGES) * SLOTS) * THREADS + threadIdx.x;
      const size_t off = (size_t)(c_begin + i) * CHUNK;
#pragma unroll
      for (int s = 0; s < TILES; ++s) {
        cp_async_16_stream(dst + (s * 2 + 0) * THREADS, wrow[s][0] + off, stream_policy);
        cp_async_16_stream(dst + (s * 2 + 1) * THREADS, wrow[s][1] + off, stream_policy);
      }
    }
  };
  auto issue_x = [&](int i) {  // the batch rows' piece of chunk i
    if (i < nc) {
      uint4* dst = ring + ((size_t)(i % STAGES) * SLOTS + TILES * 2) * THREADS + threadIdx.x;
      const size_t off = (size_t)(c_begin + i) * CHUNK;
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (xok[j]) cp_async_16(dst + j * THREADS, xsrc[j] + off);
    }
  };
  // Weights are written by no kernel: their copies start before the wait on the previous
  // kernel. Activations come from it: their copies start after the wait. One commit group
  // per stage, empty or not, so that group counting stays simple.
#pragma unroll
  for (int i = 0; i < STAGES; ++i) issue_w(i);
  // The next kernel's blocks may start at once: they prefetch their weights beside this kernel.
  // (Letting them in only after this kernel's streaming was measured: slower.)
  grid_launch_dependents();
  grid_dependency_wait();  // x comes from an earlier kernel
  KRK_TRACE_READY
#pragma unroll
  for (int i = 0; i < STAGES; ++i) {
    issue_x(i);
    cp_async_commit();
  }

  float acc[TILES][NT][4];
#pragma unroll
  for (int s = 0; s < TILES; ++s)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[s][j][c] = 0.f;

  for (int i = 0; i < nc; ++i) {
    cp_async_wait<STAGES - 1>();  // all but the newest STAGES-1 groups are complete: chunk i has landed
    const uint4* src = ring + ((size_t)(i % STAGES) * SLOTS) * THREADS + threadIdx.x;
    uint4 wa[TILES][2];
#pragma unroll
    for (int s = 0; s < TILES; ++s) {
      wa[s][0] = src[(s * 2 + 0) * THREADS];
      wa[s][1] = src[(s * 2 + 1) * THREADS];
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      uint4 xb = make_uint4(0, 0, 0, 0);
      if (xok[j]) xb = src[(TILES * 2 + j) * THREADS];
#pragma unroll
      for (int s = 0; s < TILES; ++s) {
        mma_bf16_16816(acc[s][j], wa[s][0].x, wa[s][1].x, wa[s][0].y, wa[s][1].y, xb.x, xb.y);
        mma_bf16_16816(acc[s][j], wa[s][0].z, wa[s][1].z, wa[s][0].w, wa[s][1].w, xb.z, xb.w);
      }
    }
    issue_w(i + STAGES);  // refill the stage just consumed (its values are in registers and used)
    issue_x(i + STAGES);
    cp_async_commit();
  }
  cp_async_wait<0>();

  // reduce over the warps in a fixed order
  constexpr int PER_WARP = TILES * NT * 4 * 32;
#pragma unroll
  for (int s = 0; s < TILES; ++s)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[warp * PER_WARP + ((s * NT + j) * 4 + c) * 32 + lane] = acc[s][j][c];
  __syncthreads();

  // outputs of this block: RT*16 features x NT*8 batch rows
  constexpr int OUTS = RT * 16 * NT * 8;
  if (KSPLIT > 1) {
    // every block of the cluster but the first adds its warps' parts and puts the sums into the first block's
    // inbox; one cluster barrier later the first block holds them all
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every block of the cluster has started
    if (ks != 0) {
      float* dst = cluster.map_shared_rank(inbox, 0) + (size_t)(ks - 1) * OUTS;
      for (int o = threadIdx.x; o < OUTS; o += THREADS) {
        const int m = o % (NT * 8), f = o / (NT * 8);
        const int tile = f / 16, r = f % 16;
        const int j = m / 8, col = m % 8;
        const int src_lane = (r % 8) * 4 + col / 2, reg = (r / 8) * 2 + (col & 1);
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) v += red[w * PER_WARP + ((tile * NT + j) * 4 + reg) * 32 + src_lane];
        dst[o] = v;
      }
    }
    cluster.sync();
  }
  for (int o = threadIdx.x; o < OUTS; o += THREADS) {
    const int m = o % (NT * 8), f = o / (NT * 8);  // batch row, feature within the block
    const int tile = f / 16, r = f % 16;
    const int j = m / 8, col = m % 8;
    // accumulator (row r, column col) of tile: lane = (r % 8) * 4 + col / 2, register (r / 8) * 2 + col % 2
    const int src_lane = (r % 8) * 4 + col / 2, reg = (r / 8) * 2 + (col & 1);
    float v = 0.f, v2 = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      v += red[w * PER_WARP + ((tile * NT + j) * 4 + reg) * 32 + src_lane];
      if (SWIGLU) v2 += red[w * PER_WARP + (((RT + tile) * NT + j) * 4 + reg) * 32 + src_lane];
    }
    if (KSPLIT > 1) {
      if (ks == 0) {
#pragma unroll
        for (int r = 0; r < KSPLIT - 1; ++r) v += inbox[r * OUTS + o];  // the other blocks' parts, in block order
      } else {
        continue;
      }
    }
    const int n = n0 + f;
    if (m < M && n < N) {
      if (SWIGLU == 2) {  // tanh form of GELU on the gate, gate and up as accumulated (float32), rounded once
        v = 0.5f * v * (1.0f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v))) * v2;
      } else if (SWIGLU == 3) {  // clamped inputs, g' sigmoid(1.702 g') (u' + 1)
        const float gate = fminf(v, limit), up = fminf(fmaxf(v2, -limit), limit);
        v = gate / (1.0f + expf(-1.702f * gate)) * (up + 1.0f);
      } else if (SWIGLU) {
        const float gate = round_to<bf16>(v), up = round_to<bf16>(v2);
        v = round_to<bf16>(gate / (1.0f + expf(-gate))) * up;
      } else if (limit < 0.f) {  // squared relu of the product as it would have been stored
        v = round_to<bf16>(v);
        v = v > 0.f ? v * v : 0.f;
      }
      out[(size_t)m * N + n] = from_float<TOut>(v);
    }
  }
  KRK_TRACE_END(K)
}

template <int WARPS, int NT, int RT, int SWIGLU, typename TOut, int KSPLIT = 1, int RING = 0>
int launch_warps(void* out, const void* x, const void* W, int M, int N, int K, float limit,
           cudaStream_t stream) {
  constexpr int THREADS = WARPS * 32;
  constexpr int TILES = SWIGLU ? 2 * RT : RT;
  constexpr int STAGES = ring_loads<NT, KSPLIT, RING>() / TILES;
  constexpr int SLOTS = TILES * 2 + NT;
  size_t smem = (size_t)STAGES * SLOTS * THREADS * 16 + (size_t)WARPS * TILES * NT * 4 * 32 * sizeof(float) +
                (size_t)(KSPLIT - 1) * RT * 16 * NT * 8 * sizeof(float);
  if (smem > 220 * 1024) return -2;
  auto kern = skinny_kernel<WARPS, NT, RT, SWIGLU, TOut, KSPLIT, RING>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  const int blocks = (N + 16 * RT - 1) / (16 * RT);
  if (KSPLIT > 1) {  // the blocks of a cluster share a tile and split K
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks * KSPLIT);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = KSPLIT;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    static const bool plain = getenv("KRK_NO_PDL") != nullptr;
    cfg.attrs = attr;
    cfg.numAttrs = plain ? 1 : 2;
    return (int)cudaLaunchKernelEx(&cfg, kern, (TOut*)out, (const bf16*)x, (const bf16*)W, M, N, K, limit);
  }
  cudaError_t e = launch_pdl(kern, dim3(blocks), dim3(THREADS), smem, stream, (TOut*)out, (const bf16*)x, (const bf16*)W, M,
                             N, K, limit);
  if (e != cudaSuccess) return (int)e;
  return 0;
}

// Blocks of 8 warps hold more bytes in flight each; blocks of 4 warps are small enough for
// five of them to share an SM. With between two and five blocks per SM the small ones all
// fit at once (one wave, no straggling second wave of a few blocks); otherwise the large.
template <int NT, int RT, int SWIGLU, typename TOut>
int launch(void* out, const void* x, const void* W, int M, int N, int K, float limit,
           cudaStream_t stream) {
  const int blocks = (N + 16 * RT - 1) / (16 * RT);
  // Between two and three blocks per SM: small blocks, but with rings as deep as three of them fit beside one
  // another, since what bounds a block is the bytes it has in flight (the depth makes no difference inside a step:
  // eight loads against eleven at eight rows, six against eight at sixteen, each within 0.3 %).
  if constexpr (!SWIGLU && RT == 1) {
    if (blocks > 2 * 148 && blocks <= 3 * 148)
      return launch_warps<4, NT, RT, SWIGLU, TOut, 1, (NT == 1 ? 11 : 8)>(out, x, W, M, N, K, limit, stream);
  }
  if (blocks > 2 * 148 && blocks <= 5 * 148)
    return launch_warps<4, NT, RT, SWIGLU, TOut>(out, x, W, M, N, K, limit, stream);
  // few tiles (about one per SM): split K four ways over a cluster, so that four to five small blocks an SM
  // have their bytes in flight instead of one large one
  if constexpr (!SWIGLU && RT == 1) {
    if (blocks * 4 <= 5 * 148 && K >= 4 * 4 * CHUNK * 4)
      return launch_warps<4, NT, RT, SWIGLU, TOut, 4>(out, x, W, M, N, K, limit, stream);
  }
  // (a ring twice as deep for kernels of about one block per SM was measured: slower, because the
  // next kernel's blocks then no longer fit beside it to prefetch their weights)
  return launch_warps<8, NT, RT, SWIGLU, TOut>(out, x, W, M, N, K, limit, stream);
}

template <int NT, int SWIGLU, typename TOut>
int pick_rt(void* out, const void* x, const void* W, int M, int N, int K, float limit, cudaStream_t stream) {
  if constexpr (!SWIGLU) {
    // Two row tiles a block where the blocks of one tile would be more than three an SM: a block asks for the batch rows' pieces beside
    // every weight tile's, and two tiles share them. us at 16 rows, one tile / two: 7,168 outputs of 5,120 19.5 / 15.7, 8,192 of
    // 2,560 11.3 / 8.7, 9,216 of 12,288 47.6 / 42.3; at 8 rows 16.4 / 13.9, 9.3 / 7.9, 42.6 / 40.1; at one 13.5 / 12.9, 7.8 / 7.3, 39.4 / 39.2.
    const int tiles = (N + 15) / 16, pairs = (N + 31) / 32;
    if (tiles > 3 * 148) return launch<NT, 2, SWIGLU, TOut>(out, x, W, M, N, K, limit, stream);
    // Between two and three blocks of one tile an SM, and long rows: two tiles a block as well, and K split three ways over a cluster, while
    // that leaves room for the clusters' placing (500 of 592 blocks, 5,312 outputs; 528 ran over). us, one tile / two split: 5,120 outputs
    // of 5,120 at 16 rows 14.7 / 11.5, at 8 11.5 / 10.0, at one 9.9 / 9.6; of 17,408 42.7 / 36.9, 36.0 / 33.8, 32.9 / 32.8. The clusters' start
    // and meeting is a fixed cost, so short rows lose: from K of 4,608 on every width at 1, 8, 9 and 16 rows gains (5,312 outputs 9.2 / 9.1,
    // 10.8 / 9.5, 12.2 / 10.2, 13.4 / 12.5; 4,752 8.8 / 8.5, 10.5 / 8.9, 10.2 / 9.7, 13.9 / 10.2), at 4,352 5,312 outputs of 16 rows lose (11.0 /
    // 12.5), at 4,096 of 9 as well (9.7 / 11.4), at 2,048 all but 16 rows of the narrowest, at 1,024 all (5,120 outputs 2.7 / 3.5, 2.9 /
    // 3.7, 3.2 / 4.5, 3.9 / 5.0). (Two ways, for 6,144 outputs, gained alone, 7.2 -> 6.7 at 8 rows of 2,560, and lost in a step, 51.6 ->
    // 52.4 a layer.)
    if (tiles > 2 * 148 && pairs * 3 <= 500 && K >= 4608)
      return launch_warps<4, NT, 2, SWIGLU, TOut, 3, (NT == 1 ? 8 : 6)>(out, x, W, M, N, K, limit, stream);
  }
  return launch<NT, 1, SWIGLU, TOut>(out, x, W, M, N, K, limit, stream);
}

template <int SWIGLU, typename TOut>
int pick_nt(void* out, const void* x, const void* W, int M, int N, int K, float limit, cudaStream_t stream) {
  if (M <= 8) return pick_rt<1, SWIGLU, TOut>(out, x, W, M, N, K, limit, stream);
  return pick_rt<2, SWIGLU, TOut>(out, x, W, M, N, K, limit, stream);
}

}  // namespace

#ifdef KRK_TRACE
KRK_API int krk_trace_dump(unsigned long long* host, unsigned int cap, unsigned int* count) {
  cudaDeviceSynchronize();
  cudaMemcpyFromSymbol(count, krk_trace_count, sizeof(unsigned int));
  unsigned int n = *count < cap ? *count : cap;
  if (n > KRK_TRACE_CAP) n = KRK_TRACE_CAP;
  cudaMemcpyFromSymbol(host, krk_trace_buf, (size_t)n * 4 * sizeof(unsigned long long));
  unsigned int zero = 0;
  cudaMemcpyToSymbol(krk_trace_count, &zero, sizeof(unsigned int));
  return 0;
}
#endif

// out [M, N] (bfloat16 or float32), x [M, K] bfloat16 contiguous, W [N, K] ([2N, K] with a gate) bfloat16
// contiguous. Needs M <= 16 and K % 32 == 0. gate: 0 none, 1 SwiGLU, 2 the tanh form of GELU, 3 gate and up clamped
// at `limit`, swish with slope 1.702 times (up + 1), 4 no gate but the squared relu of the plain product.
KRK_API int krk_skinny_linear(void* out, const void* x, const void* W, int M, int N, int K, float limit, int gate,
                              int out_dtype, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  if (M > 16 || K % CHUNK || K <= 0) return -2;
  if (gate != 0 && out_dtype != KRK_DTYPE_BF16) return -4;
  if (gate == 4) return pick_nt<0, bf16>(out, x, W, M, N, K, -1.f, stream);
  if (gate == 3) return pick_nt<3, bf16>(out, x, W, M, N, K, limit, stream);
  if (gate == 2) return pick_nt<2, bf16>(out, x, W, M, N, K, 0.f, stream);
  if (gate) return pick_nt<1, bf16>(out, x, W, M, N, K, 0.f, stream);
  if (out_dtype == KRK_DTYPE_F32) return pick_nt<0, float>(out, x, W, M, N, K, 0.f, stream);
  return pick_nt<0, bf16>(out, x, W, M, N, K, 0.f, stream);
}
