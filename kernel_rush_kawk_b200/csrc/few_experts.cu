// Products of routed experts with few rows (single-token steps) in bfloat16: every chosen expert's weights are read once and
// multiplied by all the rows that chose it.
//
// Such a step is bound by the weights' bytes. A warp per (row, expert) pair and output, as routed.cu has it for the 32-bit path and odd
// sizes, reads an expert again for every row that chose it (8 rows of 6 out of 64 experts: 48 pairs of about 35
// experts; 64 rows: 384 pairs of 64) and has one or two rows of weights in flight. Here a unit is 32 rows of one expert's
// matrix (16 of the gate and the same 16 of the up product, or 32 neighbours) and up to 16 of the expert's rows; a block's warps take
// 32-element pieces of k in turn, and the rows meet them in one m16n8k16 product, float32 accumulate: the matrix is the product's
// A, 16 bytes a lane straight from memory, 192 bytes of it on the way in each thread. The order of k within a product is free
// as long as both sides agree, so lane t of four takes k = 8 t .. 8 t + 7 of 32 for both: four of them feed one
// instruction, four the next, and neither side passes through shared memory (each is read by one warp alone). The warps' sums meet
// in shared memory, in the order of the warps. An expert chosen by more than 16 rows goes over its weights again, from L2.
//
// A unit is short: 2,048 elements of a row are eight pieces a warp, and a block of one unit spends much of its life with nothing on the
// way, before its first weights and behind its last. So two blocks an SM share all units out, each a run of neighbours, and a warp asks
// for a piece of the next unit as soon as it has multiplied one of this. Where all units start at once, or nearly, a block of
// one is left (few_experts_unit_kernel), which needs no tables of the other experts' pairs.
//
// 64 experts of 2,048 x 1,408 of which a row takes 6, the gated and the down product (a block a unit / this, us): one row 25.3 / 23.5, 2
// rows 44.0 / 38.7, 8 rows 114 / 102 (588 MB at 5.75 TB/s), 16 rows 156 / 143, 64 rows 207 / 191; 128 of 1,024 x 512, 8 a row: one row
// 9.1 / 8.8, 8 rows 48.2 / 38.6, 16 rows 77.8 / 55.8.
#include "mma.cuh"

namespace {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int ROWS = 16;   // of an expert in one pass
constexpr int AHEAD = 3;   // pieces of 32 k side by side that a warp has on the way: 192 bytes a row (2 and three blocks an SM, or one
                           // block of 4: 99 and 111 against 102 us at 8 rows, 232 and 225 against 191 at 64)

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
  int E;
  int act;
  const float* in_weights;  // [pairs] or null
  float limit, slope;
};

// Exclusive sums of v over the block's threads, and their total.
__device__ __forceinline__ int scan(int v, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = v;
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    const int o = __shfl_up_sync(0xffffffffu, s, d);
    if (lane >= d) s += o;
  }
  __syncthreads();
  if (lane == 31) warp_sums[warp] = s;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int i = 0; i < WARPS; ++i) {
    if (i < warp) before += warp_sums[i];
    total += warp_sums[i];
  }
  return before + s - v;
}

// What a block knows of the step: the pairs by expert, an expert's in their own order (all blocks have to have the same), and up to
// ROWS of an expert's as a pass.
struct Tables {
  int* list;         // [pairs] the pairs, by expert
  int* pass_expert;  // [passes]
  int* pass_first;   // [passes] its first pair in the list
  int* pass_rows;    // [passes]
  int passes;
  static __host__ __device__ size_t bytes(int pairs, int E) {
    return pairs <= 32 ? (size_t)pairs * 16 : ((size_t)pairs * 5 + 2 * ((E + 31) / 32)) * 4 + (size_t)WARPS * (pairs < E ? pairs : E) * 2;
  }
};

__device__ __forceinline__ Tables tables(const FewArgs& a, int* at0, int* warp_sums) {
  Tables t;
  t.list = at0;
  t.pass_expert = t.list + a.pairs;
  t.pass_first = t.pass_expert + a.pairs;
  t.pass_rows = t.pass_first + a.pairs;
  const int tid = threadIdx.x, lane = tid & 31;
  auto choice = [&](int i) {  // -1: none
    const int e = a.experts[i];
    return (unsigned)e < (unsigned)a.E ? e : -1;
  };
  if (a.pairs <= 32) {  // every warp counts for itself, the first one writes: one barrier
    const int e = lane < a.pairs ? choice(lane) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, e), below = (1u << lane) - 1u;
    const unsigned some = __ballot_sync(0xffffffffu, e >= 0);
    if (__all_sync(0xffffffffu, e < 0 || same == 1u << lane)) {  // no expert twice, as in a step of one row: a pass each
      if (tid < 32 && e >= 0) {
        const int p = __popc(some & below);
        t.pass_expert[p] = e;
        t.pass_first[p] = p;
        t.pass_rows[p] = 1;
        t.list[p] = lane;
      }
      t.passes = __popc(some);
      __syncthreads();
      return t;
    }
    const bool leads = e >= 0 && !(same & below);
    const int m = leads ? __popc(same) : 0;
    int both = m | (m + ROWS - 1) / ROWS << 16;  // its pairs, and its passes: sums of each stay below 2^16
    const int own = both;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int o = __shfl_up_sync(0xffffffffu, both, d);
      if (lane >= d) both += o;
    }
    t.passes = __shfl_sync(0xffffffffu, both, 31) >> 16;
    const int before = both - own, first = before & 0xffff;
    const int leader = __ffs(same) - 1;
    const int place = __shfl_sync(0xffffffffu, first, leader) + __popc(same & below);
    if (tid < 32) {
      for (int q = 0; q * ROWS < m; ++q) {
        const int p = (before >> 16) + q;
        t.pass_expert[p] = e;
        t.pass_first[p] = first + q * ROWS;
        t.pass_rows[p] = min(ROWS, m - q * ROWS);
      }
      if (e >= 0) t.list[place] = lane;
    }
    __syncthreads();
    return t;
  }
  int* number = t.pass_rows + a.pairs;  // [chosen experts]
  const int words = (a.E + 31) / 32, most = min(a.pairs, a.E);
  unsigned* chosen = reinterpret_cast<unsigned*>(number + a.pairs);  // [words] a bit an expert
  int* rank = reinterpret_cast<int*>(chosen + words);                // [words] chosen experts before the word's
  // [WARPS][most] pairs of a chosen expert in a warp's run of pairs; then where the warp's next one goes
  unsigned short* at = reinterpret_cast<unsigned short*>(rank + words);
  for (int i = tid; i < words; i += THREADS) chosen[i] = 0u;
  for (int i = tid; i < WARPS * most; i += THREADS) at[i] = 0;
  const int warp = tid >> 5, run = ((a.pairs + WARPS - 1) / WARPS + 31) / 32 * 32;
  const int lo = warp * run, hi = min(a.pairs, lo + run);
  const int early = lo + lane < hi ? choice(lo + lane) : -1;
  auto expert = [&](int i) { return i == lo ? early : i + lane < hi ? choice(i + lane) : -1; };  // of the run's piece from i on
  __syncthreads();
  for (int i = lo; i < hi; i += 32) {
    const int e = expert(i);
    if (e >= 0) atomicOr(chosen + (e >> 5), 1u << (e & 31));
  }
  __syncthreads();
  auto rank_of = [&](int e) { return rank[e >> 5] + __popc(chosen[e >> 5] & ((1u << (e & 31)) - 1u)); };
  int n_chosen = 0;
  for (int w0 = 0; w0 < words; w0 += THREADS) {
    int total;
    const int before = scan(w0 + tid < words ? __popc(chosen[w0 + tid]) : 0, warp_sums, total);
    if (w0 + tid < words) rank[w0 + tid] = n_chosen + before;
    n_chosen += total;
  }
  __syncthreads();
  for (int i = lo; i < hi; i += 32) {
    const int e = expert(i), r = e < 0 ? -1 : rank_of(e);
    const unsigned same = __match_any_sync(0xffffffffu, r);
    if (r >= 0 && lane == __ffs(same) - 1) {
      number[r] = e;
      at[warp * most + r] += (unsigned short)__popc(same);
    }
    __syncwarp();
  }
  __syncthreads();
  int placed = 0;
  t.passes = 0;
  for (int r0 = 0; r0 < n_chosen; r0 += THREADS) {
    const int r = r0 + tid;
    int m = 0;
    if (r < n_chosen)
      for (int v = 0; v < WARPS; ++v) m += at[v * most + r];
    int pass_total, pair_total;
    const int p = t.passes + scan((m + ROWS - 1) / ROWS, warp_sums, pass_total);
    const int first = placed + scan(m, warp_sums, pair_total);
    for (int q = 0; q * ROWS < m; ++q) {
      t.pass_expert[p + q] = number[r];
      t.pass_first[p + q] = first + q * ROWS;
      t.pass_rows[p + q] = min(ROWS, m - q * ROWS);
    }
    if (r < n_chosen) {
      int next = first;
      for (int v = 0; v < WARPS; ++v) {
        const int n = at[v * most + r];
        at[v * most + r] = (unsigned short)next;
        next += n;
      }
    }
    t.passes += pass_total;
    placed += pair_total;
  }
  __syncthreads();
  for (int i = lo; i < hi; i += 32) {
    const int e = expert(i), r = e < 0 ? -1 : rank_of(e);
    const unsigned same = __match_any_sync(0xffffffffu, r);
    const int next = r >= 0 ? at[warp * most + r] : 0;
    __syncwarp();
    if (r >= 0) {
      t.list[next + __popc(same & ((1u << lane) - 1u))] = i + lane;
      if (lane == __ffs(same) - 1) at[warp * most + r] = (unsigned short)(next + __popc(same));
    }
    __syncwarp();
  }
  __syncthreads();
  return t;
}

// The passes of one expert alone, `e`: each warp looks through a run of the pairs. `first`: the pair without which they are none.
__device__ __forceinline__ Tables tables_of(const FewArgs& a, int e, int early, int first, int* at0, int* counts) {
  Tables t;
  const int most = (a.pairs + ROWS - 1) / ROWS;
  t.list = at0;
  t.pass_expert = t.list + a.pairs;
  t.pass_first = t.pass_expert + most;
  t.pass_rows = t.pass_first + most;
  t.passes = 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int run = ((a.pairs + WARPS - 1) / WARPS + 31) / 32 * 32, lo = warp * run, hi = min(a.pairs, lo + run);
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
  if (m == 0) return t;
  for (int i = lo; i < hi; i += 32) {
    const unsigned all = found(i);
    if (all >> lane & 1u) t.list[at + __popc(all & ((1u << lane) - 1u))] = i + lane;
    at += __popc(all);
  }
  const int passes = (m + ROWS - 1) / ROWS;
  if (tid < passes) {  // up to 256
    t.pass_expert[tid] = e;
    t.pass_first[tid] = tid * ROWS;
    t.pass_rows[tid] = min(ROWS, m - tid * ROWS);
  }
  __syncthreads();
  if (first < 0 || t.list[0] == first) t.passes = passes;
  return t;
}

// `steps` units from (pass, tile) on, a unit being a pass over one of `tiles` tiles of columns from f_base on. A warp's pieces of k follow
// one another over the units' ends: a piece's registers are asked to be filled again as soon as it has been multiplied.
template <Form FORM, int NT>
__device__ __forceinline__ void walk(const FewArgs& a, const Tables& t, float (*sums)[2][ROWS][17], int pass, int tile, int steps, int tiles,
                                     int f_base) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int F = a.F, K = a.K;
  constexpr int COLS = FORM == GATED ? 16 : 32;

  const bf16 *w[4], *x[NT];
  auto aim = [&](int pass, int tile) {
    const bf16* we = a.w + (size_t)t.pass_expert[pass] * (FORM == GATED ? 2 : 1) * F * K;
    const int f0 = f_base + tile * COLS, first = t.pass_first[pass], rows = t.pass_rows[pass];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int f = f0 + g + 8 * (i & 1) + (FORM == GATED ? 0 : 16 * (i >> 1));
      w[i] = we + (size_t)(min(f, F - 1) + (FORM == GATED ? F * (i >> 1) : 0)) * K;
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int pair = t.list[first + min(8 * n + g, rows - 1)];  // a column beyond the last row repeats it and is not stored
      x[n] = FORM == DOWN ? a.x + (size_t)pair * K : a.x + (size_t)(pair / a.top) * a.x_stride;
    }
  };
  uint4 wa[AHEAD][4], xb[AHEAD][NT];
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  auto load = [&](int p, int k) {
    const bool in = k < K;  // K is a multiple of 8
#pragma unroll
    for (int i = 0; i < 4; ++i) wa[p][i] = in ? ld_stream_16(w[i] + k) : zero;
#pragma unroll
    for (int n = 0; n < NT; ++n) xb[p][n] = in ? *reinterpret_cast<const uint4*>(x[n] + k) : zero;
  };
  constexpr int STEP = AHEAD * WARPS * 32;
  const int first = warp * 32 * AHEAD + 8 * t4;
  aim(pass, tile);
#pragma unroll
  for (int p = 0; p < AHEAD; ++p) load(p, first + 32 * p);
  for (int step = 0; step < steps; ++step) {
    const bool last = step + 1 == steps, turn = tile + 1 == tiles;
    float acc[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][n][c] = 0.f;
    for (int k0 = first;; k0 += STEP) {
      const bool more = k0 - 8 * t4 + STEP < K;  // of this unit, for this warp
      const int next = more ? k0 + STEP : first;
      if (!more && !last) aim(pass + turn, turn ? 0 : tile + 1);
#pragma unroll
      for (int p = 0; p < AHEAD; ++p) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint4 lo = wa[p][2 * i], hi = wa[p][2 * i + 1];
            mma_bf16_16816(acc[i][n], lo.x, hi.x, lo.y, hi.y, xb[p][n].x, xb[p][n].y);
            mma_bf16_16816(acc[i][n], lo.z, hi.z, lo.w, hi.w, xb[p][n].z, xb[p][n].w);
          }
        if (more || !last) load(p, next + 32 * p);
      }
      if (!more) break;
    }
    if (step) __syncthreads();  // the sums before are read
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) sums[warp][i][8 * n + 2 * t4 + (c & 1)][g + 8 * (c >> 1)] = acc[i][n][c];
    __syncthreads();
    const int r = tid >> 4, f = tid & 15, f0 = f_base + tile * COLS;
    if (r < t.pass_rows[pass]) {
      const int pair = t.list[t.pass_first[pass] + r];
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
    if (turn) {
      ++pass;
      tile = 0;
    } else {
      ++tile;
    }
  }
}

// A block a tile of one expert's columns: blockIdx.y is the expert, or a pair, whose block works if no pair before it has its expert.
template <Form FORM>
__global__ void __launch_bounds__(THREADS, 2) few_experts_unit_kernel(FewArgs a) {
  extern __shared__ int tables_s[];
  __shared__ float sums[WARPS][2][ROWS][17];
  __shared__ int counts[WARPS];
  grid_launch_dependents();
  grid_dependency_wait();
  // the first choices of a warp's run are asked for together with the expert's number: a block's time before its first weights is a
  // sixth of its life
  const bool by_expert = a.pairs > a.E;
  const int lane = threadIdx.x & 31, run = ((a.pairs + WARPS - 1) / WARPS + 31) / 32 * 32, i = (threadIdx.x >> 5) * run + lane;
  const int early = i < a.pairs ? a.experts[i] : -1;
  const int e = by_expert ? (int)blockIdx.y : a.experts[blockIdx.y];
  if ((unsigned)e >= (unsigned)a.E) return;
  const Tables t = tables_of(a, e, early, by_expert ? -1 : (int)blockIdx.y, tables_s, counts);
  if (t.passes == 0) return;
  const int f_base = blockIdx.x * (FORM == GATED ? 16 : 32);
  if (t.pass_rows[0] > 8) walk<FORM, 2>(a, t, sums, 0, 0, t.passes, 1, f_base);
  else walk<FORM, 1>(a, t, sums, 0, 0, t.passes, 1, f_base);
}

template <Form FORM>
__global__ void __launch_bounds__(THREADS, 2) few_experts_kernel(FewArgs a) {
  extern __shared__ int tables_s[];
  __shared__ float sums[WARPS][2][ROWS][17];
  __shared__ int warp_sums[WARPS];
  grid_launch_dependents();
  grid_dependency_wait();
  const Tables t = tables(a, tables_s, warp_sums);
  constexpr int COLS = FORM == GATED ? 16 : 32;
  const int tiles = (a.F + COLS - 1) / COLS;
  const long long units = (long long)t.passes * tiles;
  long long u0, u1;
  int p0, p1;
  if (units < 1 << 22) {  // 32-bit divisions: those of 64 bits take a quarter of a microsecond here
    const unsigned n = (unsigned)units;
    u0 = n * blockIdx.x / gridDim.x;
    u1 = n * (blockIdx.x + 1) / gridDim.x;
    p0 = (int)((unsigned)u0 / (unsigned)tiles);
    p1 = ((int)u1 - 1) / tiles;
  } else {
    u0 = units * blockIdx.x / gridDim.x;
    u1 = units * (blockIdx.x + 1) / gridDim.x;
    p0 = (int)(u0 / tiles);
    p1 = (int)((u1 - 1) / tiles);
  }
  if (u0 == u1) return;
  const int tile0 = (int)(u0 - (long long)p0 * tiles);
  bool many = false;
  for (int p = p0; p <= p1; ++p) many |= t.pass_rows[p] > 8;
  if (many) walk<FORM, 2>(a, t, sums, p0, tile0, (int)(u1 - u0), tiles, 0);
  else walk<FORM, 1>(a, t, sums, p0, tile0, (int)(u1 - u0), tiles, 0);
}

template <Form FORM>
int launch(const FewArgs& a, cudaStream_t stream) {
  const int tiles = (a.F + (FORM == GATED ? 16 : 32) - 1) / (FORM == GATED ? 16 : 32);
  const int groups = a.pairs > a.E ? a.E : a.pairs;  // experts that may be chosen
  // A block a tile of an expert where that is no more blocks than start at once, and, beyond 32 pairs, where a walking block's tables of
  // all pairs cost 2 us, up to 768: walk / tile, us, the gated and the down product of 8 experts of 128 x 256 3.4 / 2.8 and 3.1 / 2.5 at
  // 32 pairs, 5.5 / 3.4 and 5.2 / 3.2 at 64; 16 of 256 x 1,024 (256 and 512 blocks) 4.8 / 4.2 and 5.0 / 4.8, 7.1 / 4.9 and 7.5 / 5.1; 128
  // of 128 x 512 at 48 pairs (384 and 768) 7.4 / 5.8 and 8.0 / 6.7; 16 of 1,536 x 1,536 at 64, the down product (768) 14.1 / 12.4. Beyond:
  // 12 pairs in 384 blocks of K 1,024 5.1 / 5.4; 64 of 256 x 1,024 at 64 (1,024) 11.8 / 11.8, 16 of 1,024 x 1,024 (1,024) 18.4 / 18.9.
  const long long blocks = (long long)groups * tiles;
  const bool unit = blocks <= 2 * 148 || (a.pairs > 32 && blocks <= 768);
  // the list alone and 16 bytes a pass, 20 KB at most; or 160 KB at 4,096 pairs of 65,535 experts
  const size_t bytes = unit ? ((size_t)a.pairs + 3 * ((a.pairs + ROWS - 1) / ROWS)) * 4 : Tables::bytes(a.pairs, a.E);
  if (bytes > 24 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(few_experts_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)Tables::bytes(4096, 65535));  // one value, whichever thread sets it
    if (e != cudaSuccess) return (int)e;
  }
  const long long most = (long long)(a.pairs < a.E ? a.pairs : a.E + a.pairs / ROWS) * tiles;  // units that there can be
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = unit ? dim3((unsigned)tiles, (unsigned)groups) : dim3((unsigned)(most < 2 * 148 ? most : 2 * 148));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = stream;
  // Loads on their way into registers hold room in the L1 cache, and an SM whose kernel before asked for nearly all of it as shared memory,
  // as the few-row products do, stays divided that way while one of their blocks is left on it: 3.4 TB/s where 5.7 are to be had. So the
  // launch asks for no more shared memory than two blocks need. The whole call behind its router's product, 64 experts of 1,408 x 2,048, 8
  // rows: 200 us as it comes, 130 with 60 % of the SM as shared memory, 126 with 50, 124 with 25 (which is two blocks' need there).
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  const size_t need = 2 * (bytes + sizeof(float) * WARPS * 2 * ROWS * 17 + 1024 + 64) * 100 / (228 * 1024) + 1;
  attr[0].val.sharedMemCarveout = (unsigned)(need < 100 ? need : 100);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  static const bool plain = getenv("KRK_NO_PDL") != nullptr;  // measurement switch: ordinary stream order
  cfg.attrs = attr;
  cfg.numAttrs = plain ? 1 : 2;
  return (int)cudaLaunchKernelEx(&cfg, unit ? few_experts_unit_kernel<FORM> : few_experts_kernel<FORM>, a);
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
  a.pairs = (int)pairs; a.top = top; a.F = F; a.K = K; a.E = E; a.act = act; a.in_weights = in_weights; a.limit = limit;
  a.slope = slope;
  return form == 0 ? launch<GATED>(a, stream) : form == 1 ? launch<PLAIN>(a, stream) : launch<DOWN>(a, stream);
}
