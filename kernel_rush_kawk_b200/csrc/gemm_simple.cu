// C[M, N] = A[M, K] * W[N, K]^T with float32 multiply-adds on the CUDA cores.
//
// This is the matrix product of the true 32-bit path: no tensor cores, no
// reduced-precision mode, and every output element is one chain of fused
// multiply-adds over k in ascending order, whichever kernel below computes it, so
// a row's result does not depend on how many other rows the call has. Weights are
// [out, in] as in the reference (y = x W^T, no bias:
// engine/model.py:295,299,301 of willzeng274/kernel-rush-kawk).
//
// Three kernels share that sum:
//
// * gemm_f32_tile: more than 16 float32 rows. Bound by the multiply-add pipe and, close behind it, by shared-memory reads,
//   so a thread holds up to 8 x 8 outputs, operands come k-major through two shared-memory buffers, and the next slice
//   is in registers while this one is multiplied. 1,024 rows of 19,456 x 2,560: 1.99 ms, 51 of the pipe's 72 TFLOP/s
//   (measured with independent chains); 360 rows of 6,144 x 2,560: 259 us, 44 TFLOP/s (the general kernel: 2.0 ms).
//   Packed multiply-adds (fma.rn.f32x2) were measured and are slower here (274 to 294 us): the copies that pair an
//   operand with itself cost more than the pipe's register reads gain.
// * gemm_f32_few: up to 16 float32 rows. Bound by the weights' bytes: each is read once, by bulk copies a slice or two ahead; a
//   thread owns one or two output columns of one or two rows. One row of 151,936 x 2,560: 235 us, 6.6 TB/s; three rows 226,
//   of 2,560 x 9,728 35 us, where the chain of K multiply-adds is the bound (20 us at four clocks each; copies of 16 bytes by
//   all threads: 265 and 46; the general kernel: 1.9 ms and 570 us of 2,560 x 4,096).
// * gemm_nt: everything else (bfloat16 inputs with float32 output at odd sizes, for output-head logits at many
//   positions; float32 rows whose size or alignment does not allow 16-byte accesses). 64x64 output tile, k in slices of
//   16, 256 threads with a 4x4 micro-tile each.
#include "mma.cuh"      // the cache policy of streamed weights
#include "tcgen05.cuh"  // mbarriers

namespace {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
gemm_nt_kernel(TOut* __restrict__ C, const TIn* __restrict__ A, const TIn* __restrict__ W, int M, int N, int K,
               int lda, int ldw, int ldc) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  const int lr = tid / 4, lk = (tid % 4) * 4;  // this thread loads row lr, k = lk..lk+3 of both tiles
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + lk + j;
      const int am = m0 + lr, wn = n0 + lr;
      As[lk + j][lr] = (am < M && k < K) ? to_float<TIn>(A[(size_t)am * lda + k]) : 0.f;
      Ws[lk + j][lr] = (wn < N && k < K) ? to_float<TIn>(W[(size_t)wn * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = As[k][tm + i]; w[i] = Ws[k][tn + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = m0 + tm + i, n = n0 + tn + j;
      if (m < M && n < N) C[(size_t)m * ldc + n] = from_float<TOut>(acc[i][j]);
    }
}

template <typename TIn, typename TOut>
int launch(void* C, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return -3;
  gemm_nt_kernel<TIn, TOut><<<grid, 256, 0, stream>>>((TOut*)C, (const TIn*)A, (const TIn*)W, M, N, K, lda, ldw, ldc);
  KRK_CHECK_LAUNCH();
  return 0;
}

// ---- float32, more than 16 rows --------------------------------------------------------------------------------
// 128 threads; thread (ty, tx) of 8 x 16 holds MG groups of 4 rows and NG groups of 4 columns, the groups 32 rows (64
// columns) apart. A warp covers 4 x 8 of the threads' places, neighbouring lanes sharing a column or differing in their
// row alone: a warp's 16-byte read then takes 2 cycles of the SM's shared memory (measured; 4 where every fourth lane
// shares). The fragments of the next k are read before this one's are multiplied.
constexpr int TK = 16;  // k per slice

template <int MG, int NG>
__global__ void __launch_bounds__(128, MG * NG == 4 ? 3 : 4)
gemm_f32_tile_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                     int lda, int ldw, int ldc) {
  constexpr int TM = 32 * MG, TN = 64 * NG;
  // Row k of a slice starts 8 floats further for every four k, so that the 32 stores of a warp (8 rows or columns of four
  // k that are four apart) fall into different banks; rows stay on 16-byte boundaries.
  constexpr int AP = TM + 28, WP = TN + 28;
#define KRK_SKEW(k) (8 * (((k) >> 2) & 3))
  __shared__ __align__(16) float As[2][TK][AP];
  __shared__ __align__(16) float Ws[2][TK][WP];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (warp >> 1) * 8 + ((lane & 15) >> 1), ty = (warp & 1) * 4 + (lane & 1) + 2 * (lane >> 4);
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  const int lk = (tid & 3) * 4, lr = tid >> 2;  // this thread loads k = lk..lk+3 of rows lr, lr + 32, ...
  float acc[4 * MG][4 * NG];
#pragma unroll
  for (int i = 0; i < 4 * MG; ++i)
#pragma unroll
    for (int j = 0; j < 4 * NG; ++j) acc[i][j] = 0.f;
  float4 ar[MG], wr[2 * NG];
  auto fetch = [&](int k0) {  // zeros beyond the matrices' ends (K is a multiple of 4)
    const bool in = k0 + lk < K;
#pragma unroll
    for (int i = 0; i < MG; ++i) {
      const int m = m0 + lr + 32 * i;
      ar[i] = in && m < M ? *reinterpret_cast<const float4*>(A + (size_t)m * lda + k0 + lk) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 2 * NG; ++i) {
      const int n = n0 + lr + 32 * i;
      wr[i] = in && n < N ? *reinterpret_cast<const float4*>(W + (size_t)n * ldw + k0 + lk) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto stage = [&](int b) {
    const int at = lr + KRK_SKEW(lk);
#pragma unroll
    for (int i = 0; i < MG; ++i) {
      As[b][lk][at + 32 * i] = ar[i].x; As[b][lk + 1][at + 32 * i] = ar[i].y;
      As[b][lk + 2][at + 32 * i] = ar[i].z; As[b][lk + 3][at + 32 * i] = ar[i].w;
    }
#pragma unroll
    for (int i = 0; i < 2 * NG; ++i) {
      Ws[b][lk][at + 32 * i] = wr[i].x; Ws[b][lk + 1][at + 32 * i] = wr[i].y;
      Ws[b][lk + 2][at + 32 * i] = wr[i].z; Ws[b][lk + 3][at + 32 * i] = wr[i].w;
    }
  };
  fetch(0);
  stage(0);
  __syncthreads();
  const int slices = (K + TK - 1) / TK;
  for (int s = 0; s < slices; ++s) {
    const int b = s & 1;
    if (s + 1 < slices) fetch((s + 1) * TK);
    float4 w[2][NG];
    float4 a[2][MG];
    auto read = [&](int f, int k) {
#pragma unroll
      for (int g = 0; g < NG; ++g) w[f][g] = *reinterpret_cast<const float4*>(&Ws[b][k][64 * g + 4 * tx + KRK_SKEW(k)]);
#pragma unroll
      for (int g = 0; g < MG; ++g) a[f][g] = *reinterpret_cast<const float4*>(&As[b][k][32 * g + 4 * ty + KRK_SKEW(k)]);
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      if (k + 1 < TK) read((k + 1) & 1, k + 1);
#pragma unroll
      for (int g = 0; g < MG; ++g) {
        const float4 v = a[k & 1][g];
        const float av[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < NG; ++j) {
            const float4 u = w[k & 1][j];
            acc[4 * g + i][4 * j] = fmaf(av[i], u.x, acc[4 * g + i][4 * j]);
            acc[4 * g + i][4 * j + 1] = fmaf(av[i], u.y, acc[4 * g + i][4 * j + 1]);
            acc[4 * g + i][4 * j + 2] = fmaf(av[i], u.z, acc[4 * g + i][4 * j + 2]);
            acc[4 * g + i][4 * j + 3] = fmaf(av[i], u.w, acc[4 * g + i][4 * j + 3]);
          }
      }
    }
    if (s + 1 < slices) {
      stage(b ^ 1);  // the slice before, which was there, was multiplied before the last barrier
      __syncthreads();
    }
  }
#undef KRK_SKEW
  const bool wide = (ldc & 3) == 0;  // C's rows start on 16-byte boundaries (its base does: the caller checks)
#pragma unroll
  for (int g = 0; g < MG; ++g)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + 32 * g + 4 * ty + i;
      if (m >= M) continue;
#pragma unroll
      for (int h = 0; h < NG; ++h) {
        const int n = n0 + 64 * h + 4 * tx;
        float* c = C + (size_t)m * ldc + n;
        const float4 v = make_float4(acc[4 * g + i][4 * h], acc[4 * g + i][4 * h + 1], acc[4 * g + i][4 * h + 2], acc[4 * g + i][4 * h + 3]);
        if (wide && n + 4 <= N) {
          *reinterpret_cast<float4*>(c) = v;
        } else {
          const float* f = reinterpret_cast<const float*>(&v);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < N) c[j] = f[j];
        }
      }
    }
}

// ---- float32, up to 16 rows ------------------------------------------------------------------------------------
// A block owns 16 * CPT columns (a thread c, c + 16); a group of 16 threads takes RPT rows, a warp has two groups, and there are as many
// warps as the rows ask for. A slice is SLICE k of the columns' weights and of the rows. One more warp asks for slices, a bulk copy a
// column (1 KB), as far ahead as the ring is deep, so that the others only wait and multiply: with 16-byte copies by all threads, asking
// for a slice took 600 to 1,200 clocks of the 1,200 that its 256 multiply-adds take in their chain (256 x 4, and the reads).
// Beyond 8 rows, where shared-memory reads are the bound, a thread's two rows of two columns read half as much for a
// multiply-add as one of one.
constexpr int FEW_MAX_DEPTH = 3;
constexpr int FEW_BARS = 2 * FEW_MAX_DEPTH * 8;  // bytes before the ring: slice is here, slice is free

template <int RPT, int CPT, int SLICE>
__global__ void __launch_bounds__(160)
gemm_f32_few_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                    int lda, int ldw, int ldc, int depth, int* __restrict__ error) {
  constexpr int COLS = 16 * CPT, PITCH = SLICE + 4;
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* free_ = full + FEW_MAX_DEPTH;
  float* ring = reinterpret_cast<float*>(smem + FEW_BARS);
  const int stage_floats = (COLS + M) * PITCH;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, readers = (blockDim.x >> 5) - 1;
  const int n0 = blockIdx.x * COLS;
  const int slices = (K + SLICE - 1) / SLICE;
  if (tid == 0) {
    for (int i = 0; i < depth; ++i) {
      tc::mbar_init(full + i, 1);
      tc::mbar_init(free_ + i, readers);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (warp == readers) {  // the copies: a lane has columns (or rows) lane, lane + 32 of a slice
    const int cols = min(COLS, N - n0);
    const uint64_t policy = l2_evict_first_policy();
    for (int s = 0, b = 0, round = 0; s < slices; ++s) {
      if (round > 0 && !__all_sync(0xffffffffu, tc::mbar_wait(free_ + b, (round - 1) & 1))) {  // a reader has given up, and says so
        tc::wait_for_copies(full, depth, s);
        return;
      }
      const int bytes = min(SLICE, K - s * SLICE) * 4;
      if (lane == 0) tc::mbar_expect_tx(full + b, (cols + M) * bytes);
      __syncwarp();
      float* dst = ring + b * stage_floats;
      for (int r = lane; r < cols; r += 32)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                     ::"r"(tc::smem_u32(dst + r * PITCH)), "l"(W + (size_t)(n0 + r) * ldw + s * SLICE), "r"(bytes), "r"(tc::smem_u32(full + b)), "l"(policy)
                     : "memory");
      if (lane < M)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(tc::smem_u32(dst + (COLS + lane) * PITCH)), "l"(A + (size_t)lane * lda + s * SLICE), "r"(bytes), "r"(tc::smem_u32(full + b))
                     : "memory");
      if (++b == depth) { b = 0; ++round; }
    }
    return;  // what has been asked for is read, or waited for by the reader that gives up
  }
  // neighbouring lanes share a column and differ in their rows
  const int col = lane >> 1, group = 2 * warp + (lane & 1);
  float acc[RPT][CPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int c = 0; c < CPT; ++c) acc[r][c] = 0.f;
  const int row0 = group * RPT;
  int xat[RPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r) xat[r] = (COLS + min(row0 + r, M - 1)) * PITCH;
  bool here = true;
  for (int s = 0, b = 0, round = 0; s < slices; ++s) {
    // a wait that runs out: the warp's outputs are NaN
    here = __all_sync(0xffffffffu, tc::mbar_wait(full + b, round & 1));
    if (!here) {  // a place that it hands back no more is not filled again: what may be on its way is a ring from here
      tc::wait_for_copies(full, depth, min(slices, s + depth));
      break;
    }
    const float* base = ring + b * stage_floats;
    const float* w = base + col * PITCH;
    constexpr int AHEAD = 4;  // pieces of four k in registers while as many are multiplied
    const int kn = min(SLICE, K - s * SLICE);
    float4 w4[2][AHEAD][CPT], x4[2][AHEAD][RPT];
    auto read = [&](int f, int k0) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
#pragma unroll
        for (int c = 0; c < CPT; ++c) w4[f][i][c] = *reinterpret_cast<const float4*>(w + 16 * c * PITCH + k0 + 4 * i);
#pragma unroll
        for (int r = 0; r < RPT; ++r) x4[f][i][r] = *reinterpret_cast<const float4*>(base + xat[r] + k0 + 4 * i);
      }
    };
    auto multiply = [&](int f, int i) {
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < CPT; ++c) acc[r][c] = fmaf(x4[f][i][r].x, w4[f][i][c].x, acc[r][c]);
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < CPT; ++c) acc[r][c] = fmaf(x4[f][i][r].y, w4[f][i][c].y, acc[r][c]);
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < CPT; ++c) acc[r][c] = fmaf(x4[f][i][r].z, w4[f][i][c].z, acc[r][c]);
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < CPT; ++c) acc[r][c] = fmaf(x4[f][i][r].w, w4[f][i][c].w, acc[r][c]);
    };
    if (kn == SLICE) {
      read(0, 0);
#pragma unroll
      for (int p = 0; p < SLICE / (4 * AHEAD); ++p) {
        if (p + 1 < SLICE / (4 * AHEAD)) read((p + 1) & 1, (p + 1) * 4 * AHEAD);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) multiply(p & 1, i);
      }
    } else {
      for (int k = 0; k < kn; k += 4) {
#pragma unroll
        for (int c = 0; c < CPT; ++c) w4[0][0][c] = *reinterpret_cast<const float4*>(w + 16 * c * PITCH + k);
#pragma unroll
        for (int r = 0; r < RPT; ++r) x4[0][0][r] = *reinterpret_cast<const float4*>(base + xat[r] + k);
        multiply(0, 0);
      }
    }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(free_ + b);
    if (++b == depth) { b = 0; ++round; }
  }
  if (!here && lane == 0 && error) atomicExch(error, 20);
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int c = 0; c < CPT; ++c)
      if (row0 + r < M && n0 + col + 16 * c < N) C[(size_t)(row0 + r) * ldc + n0 + col + 16 * c] = here ? acc[r][c] : NAN;
}

template <int MG, int NG>
int launch_tile(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  dim3 grid((N + 64 * NG - 1) / (64 * NG), (M + 32 * MG - 1) / (32 * MG));
  if (grid.y > 65535) return -3;
  gemm_f32_tile_kernel<MG, NG><<<grid, 128, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
  KRK_CHECK_LAUNCH();
  return 0;
}

template <int RPT, int CPT, int SLICE>
int launch_few(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int* error, cudaStream_t stream) {
  constexpr size_t per_row = (SLICE + 4) * sizeof(float);
  const size_t stage = (16 * CPT + M) * per_row;  // 17 to 50 KB
  const int blocks = (N + 16 * CPT - 1) / (16 * CPT);
  // Two slices of the ring leave an SM more blocks than three, three cover more of a slice's way. Where a thread has one output, what
  // decides is how many blocks the SMs take in full rounds (three rows of K 2,560, two slices and three: N of 2,560 17.8 and 16.4 us, 6,144
  // 20.3 and 19.0, 8,192 22.6 and 29.3, 12,288 (K 4,096) 51.6 and 44.3, 19,456 43.0 and 44.0, 151,936 239 and 256). Two rows by two columns are
  // bound by the multiplying warps' own reads, which only other blocks cover: two slices at every size measured, where three were within 2 %
  // or worse (K 2,560, two and three: five rows in slices of 128, N of 151,936 277 and 365 us; sixteen rows in slices of 256, one
  // block an SM with three, 19,456 79 and 108, 151,936 438 and 698; twelve of 9,728 48 and 61).
  auto rounds = [&](int depth) {
    const long long held = max(1LL, (long long)(227 * 1024 / (FEW_BARS + depth * stage + 1024)));
    return (blocks + 148 * held - 1) / (148 * held) * held;
  };
  const int depth = RPT == 1 && rounds(3) < rounds(2) ? 3 : 2;
  // always the most that a call may need: another thread may be about to launch with more rows than this one
  cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<RPT, CPT, SLICE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(FEW_BARS + FEW_MAX_DEPTH * (16 * CPT + 8 * RPT) * per_row));
  if (e != cudaSuccess) return (int)e;
  const int readers = (M + 2 * RPT - 1) / (2 * RPT);
  gemm_f32_few_kernel<RPT, CPT, SLICE><<<blocks, 32 * (readers + 1), FEW_BARS + depth * stage, stream>>>(
      C, A, W, M, N, K, lda, ldw, ldc, depth, error);
  KRK_CHECK_LAUNCH();
  return 0;
}

// float32 in and out with 16-byte rows. -2: not of that kind.
int launch_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int* error, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  if (K < 4 || K % 4 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W | (uintptr_t)C) & 15)) return -2;
  // 16 rows: 79 us of 19,456 x 2,560 and 161 by the tiles below, 438 and 647 of 151,936 x 2,560, 2.5 and 4.0 of 128 x 64.
  // One row of one column a thread reads most of shared memory for a multiply-add and has the most blocks; from five rows
  // on the reads bound it where there are columns enough (eight rows, two by two in slices of 128 and one by one: N of 19,456
  // 45 and 57 us, 151,936 283 and 366; 8,192 27 and 22; five rows 44 and 48, 277 and 284; 12,288 31 and 28). Beyond eight rows two by
  // two always: in slices of 128 to 12 rows of many columns (nine rows: N of 12,288 32 and 41, 151,936 322 and 399; 8,192 28 and 22;
  // sixteen 437 and 438, but 89 and 79 of 19,456).
  if (M <= 8 && (M < 5 || N < 16384)) return launch_few<1, 1, 256>(C, A, W, M, N, K, lda, ldw, ldc, error, stream);
  if (M <= 8 || (M <= 12 && N >= 12288)) return launch_few<2, 2, 128>(C, A, W, M, N, K, lda, ldw, ldc, error, stream);
  if (M <= 16) return launch_few<2, 2, 256>(C, A, W, M, N, K, lda, ldw, ldc, error, stream);
  // Cycles per k on the busiest SM, from the times measured at 17 to 1,024 rows of five matrices: a block alone is bound by
  // its own latency (the first number), several by what a block takes of the SM.
  auto cost = [&](int tm, int tn, int alone, int each) {
    const long long tiles = (long long)((M + tm - 1) / tm) * ((N + tn - 1) / tn);
    const long long all = (tiles + 147) / 148 * each;
    return all > alone ? all : alone;
  };
  const long long c22 = cost(64, 128, 120, 89), c21 = cost(64, 64, 88, 47), c12 = cost(32, 128, 96, 49);
  const long long best = min(c22, min(c21, c12));
  if (best == c22) return launch_tile<2, 2>(C, A, W, M, N, K, lda, ldw, ldc, stream);
  if (best == c21) return launch_tile<2, 1>(C, A, W, M, N, K, lda, ldw, ldc, stream);
  return launch_tile<1, 2>(C, A, W, M, N, K, lda, ldw, ldc, stream);
}

}  // namespace

// in_dtype / out_dtype: KRK_DTYPE_F32 or KRK_DTYPE_BF16. Supported: f32->f32, bf16->f32, bf16->bf16. `error` (device, may be null)
// is set to 20 should a product of few rows give up on a wait, whose outputs are then NaN.
KRK_API int krk_gemm_nt(void* C, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldc,
                        int in_dtype, int out_dtype, int* error, cudaStream_t stream) {
  if (in_dtype == KRK_DTYPE_F32 && out_dtype == KRK_DTYPE_F32) {
    const int rc = launch_f32((float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, error, stream);
    if (rc != -2) return rc;
  }
  if (in_dtype == KRK_DTYPE_F32 && out_dtype == KRK_DTYPE_F32)
    return launch<float, float>(C, A, W, M, N, K, lda, ldw, ldc, stream);
  if (in_dtype == KRK_DTYPE_BF16 && out_dtype == KRK_DTYPE_F32)
    return launch<bf16, float>(C, A, W, M, N, K, lda, ldw, ldc, stream);
  if (in_dtype == KRK_DTYPE_BF16 && out_dtype == KRK_DTYPE_BF16)
    return launch<bf16, bf16>(C, A, W, M, N, K, lda, ldw, ldc, stream);
  return -4;
}

// For the tests of tc::wait_for_copies: a warp asks for `asked` slices of 256 numbers of src into a ring of `depth` places, reads none,
// and leaves the ring in out once the last copies are said to be here. `withheld`: it counts on one more, which it never asks for;
// that wait runs out after limit_us, which the error word says (21). Slice i is in place i % depth.
namespace {
__global__ void copies_kernel(float* out, const float* src, int depth, int asked, int withheld, int* error, unsigned long long limit_ns) {
  __shared__ __align__(16) float ring[8][256];
  __shared__ uint64_t full[8];
  if (threadIdx.x == 0) {
    for (int i = 0; i < depth; ++i) tc::mbar_init(full + i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < depth * 256; i += 32) ring[i / 256][i % 256] = 0.f;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (threadIdx.x == 0) {
    for (int i = 0; i < asked + withheld; ++i) {
      if (i >= depth && !tc::mbar_wait(full + i % depth, (uint32_t)(i / depth - 1) & 1u)) { asked = i; withheld = 0; break; }
      if (i == asked) break;
      tc::mbar_expect_tx(full + i % depth, 1024);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 1024, [%2];"
                   ::"r"(tc::smem_u32(ring[i % depth])), "l"(src + i * 256), "r"(tc::smem_u32(full + i % depth)) : "memory");
    }
  }
  asked = __shfl_sync(0xffffffffu, asked, 0);
  withheld = __shfl_sync(0xffffffffu, withheld, 0);
  if (!__all_sync(0xffffffffu, tc::wait_for_copies(full, depth, asked + withheld, limit_ns)) && threadIdx.x == 0) atomicExch(error, 21);
  for (int i = threadIdx.x; i < depth * 256; i += 32) out[i] = ring[i / 256][i % 256];
}
}  // namespace

KRK_API int krk_selftest_wait_for_copies(float* out, const float* src, int depth, int asked, int withheld, int* error, int limit_us,
                                         cudaStream_t stream) {
  if (depth < 1 || depth > 8 || asked < 0 || asked > 64 || withheld < 0 || withheld > 1 || limit_us < 1 || limit_us > 100000 ||
      (uintptr_t)src % 16)
    return -2;
  copies_kernel<<<1, 32, 0, stream>>>(out, src, depth, asked, withheld, error, (unsigned long long)limit_us * 1000ull);
  KRK_CHECK_LAUNCH();
  return 0;
}
