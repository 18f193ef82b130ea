// Products of routed experts with few rows (single-token steps) in bfloat16: every chosen expert's weights are read once and
// multiplied by all the rows that chose it.
//
// Such a step is bound by the weights' bytes. A warp per (row, expert) pair and output, as routed.cu has it for the 32-bit path and odd
// sizes, reads an expert again for every row that chose it (8 rows of 6 out of 64 experts: 48 pairs of about 35
// experts; 64 rows: 384 pairs of 64) and has one or two rows of weights in flight. Here a block takes 32 rows of one expert's
// matrix (16 of the gate and the same 16 of the up product, or 32 neighbours), its warps take 32-element pieces of them in
// turn, and up to 16 of the expert's rows meet them in one m16n8k16 product, float32 accumulate: the matrix is the product's
// A, 16 bytes a lane straight from memory, 192 bytes of it on the way in each thread. The order of k within a product is free
// as long as both sides agree, so lane t of four takes k = 8 t .. 8 t + 7 of 32 for both: four of them feed one
// instruction, four the next, and neither side passes through shared memory (each is read by one warp alone). The warps' sums meet
// in shared memory, in the order of the warps. An expert chosen by more than 16 rows goes over its weights again, from L2.
//
// 64 experts of 2,048 x 1,408 of which a row takes 6, the whole feed-forward: one row 54 -> 50 us, 8 rows 204 -> 152 (gate/up
// 115 -> 83: 404 MB at 4.9 TB/s; down and sum 92 -> 49), 64 rows 1,354 -> 250.
#include "mma.cuh"

namespace {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int ROWS = 16;   // of an expert in one pass
constexpr int AHEAD = 3;   // pieces of 32 k side by side that a warp has on the way: 192 bytes a row (2 and three blocks an SM, or one
                           // block of 4, are slower: 163 and 216 against 161 us at 8 rows)

enum Form { GATED, PLAIN, DOWN };  // gate and up with an activation; one product with an activation; one product as it is

__device__ __forceinline__ float act_of(float z, int act) {
  if (act == 0) return z / (1.0f + expf(-z));
  if (act == 1) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
  if (act == 5) return z > 0.f ? z * z : 0.f;
  return 1.0f / (1.0f + expf(-z));
}
__device__ __forceinline__ float clamped_swish(float g, float u, float limit, float slope) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.0f + expf(-slope * g)) * (u + 1.0f);
}

struct FewArgs {
  bf16* out;        // [pairs, F]
  const bf16* x;    // rows of K: a pair's own (DOWN), or the row's that chose
  int x_stride;
  const bf16* w;    // [E, (GATED: 2) F, K]
  const int* experts;  // [pairs], -1: none
  int pairs, top, F, K;
  int by_expert;    // blockIdx.y is an expert, or a pair (whose block works if no pair before it has its expert)
  int act;
  const float* in_weights;  // [pairs] or null
  float limit, slope;
};

// The sums over the warp's pieces of k for NT * 8 rows
template <int NT>
__device__ __forceinline__ void products(float (&acc)[2][2][4], const bf16* const (&w)[4], const bf16* const (&x)[2], int K, int warp,
                                         int t4) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][n][c] = 0.f;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int k0 = warp * 32 * AHEAD + 8 * t4; k0 - 8 * t4 < K; k0 += AHEAD * WARPS * 32) {
    uint4 a[AHEAD][4], b[AHEAD][NT];
#pragma unroll
    for (int p = 0; p < AHEAD; ++p) {
      const int k = k0 + p * 32;
      const bool in = k < K;  // K is a multiple of 8
#pragma unroll
      for (int i = 0; i < 4; ++i) a[p][i] = in ? ld_stream_16(w[i] + k) : zero;
#pragma unroll
      for (int n = 0; n < NT; ++n) b[p][n] = in ? *reinterpret_cast<const uint4*>(x[n] + k) : zero;
    }
#pragma unroll
    for (int p = 0; p < AHEAD; ++p)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 lo = a[p][2 * i], hi = a[p][2 * i + 1];
          mma_bf16_16816(acc[i][n], lo.x, hi.x, lo.y, hi.y, b[p][n].x, b[p][n].y);
          mma_bf16_16816(acc[i][n], lo.z, hi.z, lo.w, hi.w, b[p][n].z, b[p][n].w);
        }
  }
}

template <Form FORM>
__global__ void __launch_bounds__(THREADS, 2) few_experts_kernel(FewArgs a) {
  extern __shared__ int list[];  // the expert's pairs, in order
  __shared__ float sums[WARPS][2][ROWS][17];
  __shared__ int counts[WARPS];
  grid_launch_dependents();
  grid_dependency_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  // the list of the expert's pairs, each warp looking through a run of them; the first 32 are asked for together with the
  // expert's number, since a block's time before its first weights is a sixth of its life
  const int run = ((a.pairs + WARPS - 1) / WARPS + 31) / 32 * 32;
  const int lo = warp * run, hi = min(a.pairs, lo + run);
  const int early = lo + lane < hi ? a.experts[lo + lane] : -1;
  const int e = a.by_expert ? (int)blockIdx.y : a.experts[blockIdx.y];
  if (e < 0) return;
  auto found = [&](int i) { return __ballot_sync(0xffffffffu, (i == lo ? early : i + lane < hi ? a.experts[i + lane] : -1) == e); };
  int mine = 0;
  for (int i = lo; i < hi; i += 32) mine += __popc(found(i));
  if (lane == 0) counts[warp] = mine;
  __syncthreads();
  int m = 0, at = 0;
#pragma unroll
  for (int v = 0; v < WARPS; ++v) {
    if (v == warp) at = m;
    m += counts[v];
  }
  if (m == 0) return;
  for (int i = lo; i < hi; i += 32) {
    const unsigned all = found(i);
    if (all >> lane & 1u) list[at + __popc(all & ((1u << lane) - 1u))] = i + lane;
    at += __popc(all);
  }
  __syncthreads();
  if (!a.by_expert && list[0] != (int)blockIdx.y) return;

  const int F = a.F, K = a.K;
  constexpr int COLS = FORM == GATED ? 16 : 32;
  const bf16* we = a.w + (size_t)e * (FORM == GATED ? 2 : 1) * F * K;
  const int f0 = blockIdx.x * COLS;
  const bf16* w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int f = f0 + g + 8 * (i & 1) + (FORM == GATED ? 0 : 16 * (i >> 1));
    w[i] = we + (size_t)(min(f, F - 1) + (FORM == GATED ? F * (i >> 1) : 0)) * K;
  }
  for (int r0 = 0; r0 < m; r0 += ROWS) {
    const int rows = min(ROWS, m - r0);
    const bf16* x[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int pair = list[min(r0 + 8 * n + g, m - 1)];  // a column beyond the last row repeats it and is not stored
      x[n] = FORM == DOWN ? a.x + (size_t)pair * K : a.x + (size_t)(pair / a.top) * a.x_stride;
    }
    float acc[2][2][4];
    if (rows <= 8) products<1>(acc, w, x, K, warp, t4);
    else products<2>(acc, w, x, K, warp, t4);
    if (r0) __syncthreads();  // the sums of the rows before are read
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) sums[warp][i][8 * n + 2 * t4 + (c & 1)][g + 8 * (c >> 1)] = acc[i][n][c];
    __syncthreads();
    const int r = tid >> 4, f = tid & 15;
    if (r < rows) {
      const int pair = list[r0 + r];
      float s[2] = {0.f, 0.f};
#pragma unroll
      for (int v = 0; v < WARPS; ++v) {
        s[0] += sums[v][0][r][f];
        s[1] += sums[v][1][r][f];
      }
      if (FORM != DOWN && a.in_weights) {
        const float by = a.in_weights[pair];
        s[0] *= by;
        s[1] *= by;
      }
      bf16* out = a.out + (size_t)pair * F + f0 + f;
      if (FORM == GATED) {
        // the two products leave in the path's type before the activation, as they do from a product kernel
        if (f0 + f < F)
          *out = from_float<bf16>(a.act == 3 ? clamped_swish(s[0], s[1], a.limit, a.slope)
                                             : act_of(round_to<bf16>(s[0]), a.act) * round_to<bf16>(s[1]));
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (f0 + f + 16 * i < F) out[16 * i] = from_float<bf16>(FORM == PLAIN ? act_of(round_to<bf16>(s[i]), a.act) : s[i]);
      }
    }
  }
}

template <Form FORM>
int launch(FewArgs a, int E, cudaStream_t stream) {
  a.by_expert = a.pairs > E;
  const int cols = (FORM == GATED ? 16 : 32);
  const dim3 grid((unsigned)((a.F + cols - 1) / cols), (unsigned)(a.by_expert ? E : a.pairs));
  return (int)launch_pdl(few_experts_kernel<FORM>, grid, dim3(THREADS), (size_t)a.pairs * sizeof(int), stream, a);
}

}  // namespace

// form 0: out = act(x Wg^T) * (x Wu^T) with w [E, 2 F, K] (act 3: the clamped swish); 1: out = act(x W^T); 2: out = x W^T from a
// row of x per pair. out [rows * top, F]. bfloat16; K a multiple of 8, rows of x and w on 16-byte boundaries, up to 4,096 pairs.
KRK_API int krk_few_experts(void* out, const void* x, int x_stride, const void* w, const int* experts, int rows, int top, int E, int F,
                            int K, int form, int act, const float* in_weights, float limit, float slope, cudaStream_t stream) {
  if (rows == 0) return 0;
  const long long pairs = (long long)rows * top;
  if (pairs > 4096 || E > 65535 || K % 8 || K < 8 || F < 1 || (form != 2 && x_stride % 8) || (((uintptr_t)x | (uintptr_t)w) & 15) ||
      (act == 3 && form == 1) || form < 0 || form > 2)
    return -2;
  FewArgs a;
  a.out = (bf16*)out; a.x = (const bf16*)x; a.x_stride = x_stride; a.w = (const bf16*)w; a.experts = experts;
  a.pairs = (int)pairs; a.top = top; a.F = F; a.K = K; a.by_expert = 0; a.act = act; a.in_weights = in_weights; a.limit = limit;
  a.slope = slope;
  return form == 0 ? launch<GATED>(a, E, stream) : form == 1 ? launch<PLAIN>(a, E, stream) : launch<DOWN>(a, E, stream);
}
