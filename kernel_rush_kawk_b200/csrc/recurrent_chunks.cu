// The recurrences of recurrent.cu over a step's many tokens in chunks of 32, for bfloat16 rows and heads of 64 channels.
//
// The scan of recurrent.cu takes a sequence's tokens one after the other: 0.57 us a token (delta rule) or 0.40 (time
// mixing) whatever the batch, on as many SMs as there are heads and sequences. Here a chunk's tokens become small matrix
// products, and all chunks but for one walk run side by side. The state, the decays and all sums are float32, as they are there.
// Products on the tensor cores take operands as three bfloat16 terms (24 bits), leave out those of two terms that are below
// 2^-24 of the leading one's, and add all of a sum's small products before its leading ones, because the tensor cores cut every sum
// off: outputs that are not the correctly rounded ones, of 1,033 tokens of 8 heads, 2.3e-4 with float32 multiply-adds on the CUDA
// cores, 1.4e-4 here (3.5e-4 with the small products of a slice of k after the leading ones of the slice before). With the state S
// before the chunk, c_t the log decays summed from the chunk's first token to t, and rows of the chunk's tokens:
//
//   time mixing:  o_t = (r_t e^{c_{t-1}}) . S + sum_{s<t} [sum_n r_tn k_sn e^{c_{t-1,n} - c_{s,n}}] v_s + (r_t . bonus k_t) v_t
//                 S' = e^{c_last} S + sum_s (k_s e^{c_last - c_s}) v_s^T
//
//   delta rule, u the unit keys, a the removal rates, y_t = u_t . S_{t-1} (what token t removes along its key):
//     y_t = (u_t e^{c_{t-1}}) . S + sum_{s<t} (B_ts v_s - D_ts y_s),  B_ts = (u_t e^{c_{t-1}}) . (k_s e^{-c_s}), D with a_s u_s for k_s
//     o_t = (r_t e^{c_t}) . S + sum_{s<=t} (P_ts v_s - R_ts y_s),      P, R likewise from r_t e^{c_t}
//     S'  = e^{c_last} (S + sum_s (k_s e^{-c_s}) v_s^T - (a_s u_s e^{-c_s}) y_s^T)
//   y is linear in S: Y = X S + Z with (I + D) X = U and (I + D) Z = B V, U the rows u_t e^{c_{t-1}}. So
//     O = Q S + O_own with Q = Rows - R X, O_own = P V - R Z;   S' = M S + G with M = e^{c_last} (I - A^T X),
//     G = e^{c_last} (K^T V - A^T Z).
//
// Three passes: (1) per (sequence, chunk, head) M, G, Q and O_own (time mixing: G and the summed decays alone); (2) the walk over
// a sequence's chunks, S' = M S + G, split over the value columns, which are independent of one another; it leaves each chunk
// its starting state in G's place and the sequence its final one; (3) per (sequence, chunk, head) the outputs with their norm,
// weight and gate. Chunks of 32: a chunk of 64 needs twice the multiply-adds a token in pass 1 and halves the walk's steps.
//
// Measured: one prompt of 2,048 tokens, delta rule of 8 heads, 1,171 us token by token, 101 here back to back (the passes 58, 33 and 17, each
// alone and from a cold cache); three prompts of 2,553 tokens in all, time mixing of 40 heads, 405 -> 117 us (48, 17 and 66; with float32 on the
// CUDA cores 175). Passes 1 and 3 are bound by instruction issue and latencies (a 0.4 to 0.5 share of the issue slots, 12 to 32 warps an
// SM), the walk by the chain of its steps.
//
// e^{-c_s} must stay in range. The delta rule's decay is at least e^{-decay_scale} a token, so a chunk's is bounded by the
// parameter (the caller asks krk_recurrence_chunk_tokens). Time mixing's has no bound: a chunk in which some channel decays by
// more than e^-40 forms its pair sums by decaying each key token by token, right for any decay and slower.
#include "mma.cuh"
#include "tcgen05.cuh"  // tiled copies and their barriers

namespace {

constexpr int L = 32;         // tokens per chunk
constexpr int N = 64;         // channels of a head
constexpr int PITCH = N + 4;  // rows on 16-byte boundaries; eight neighbouring rows' pieces fall into different banks
constexpr int THREADS = 128, HALF = L / 2;
constexpr int DELTA_THREADS = 256, PART = L * N / DELTA_THREADS;  // pass 1 of the delta rule: a thread has PART tokens of a channel
constexpr float SAFE = 40.f;  // keys up to 1e21 stay finite times e^SAFE
constexpr int WALK_COLS = 4;    // value columns a block of pass 2 walks with
constexpr int WALK_STAGES = 6;  // chunks whose M are on the way, and the one at hand

struct ChunkArgs {
  const bf16 *r, *k, *v, *g, *rate, *lora;
  int r_stride, k_stride, v_stride, g_stride, rate_stride, lora_stride;
  const bf16* w2;
  const float *w0, *rate_bias, *bonus, *norm_w;
  float* state;  // [slots, H, N, N]
  const bf16* last_rows;
  int last_stride, C;
  float* last_state;
  bf16* out;
  int out_stride, out_col;
  float out_scale, eps, decay_scale;
  int H, R;
  const int *cu_q, *seq_qlen, *seq_slot;
  int chunk0, n_chunks;  // the chunks of every sequence that this launch takes
  int* error;
  float* scratch;        // per (sequence, chunk, head): delta M, G, Q, O_own; time mixing G, summed decays and, past e^-SAFE, the decays
};
constexpr int ITEM_DELTA = 2 * N * N + 2 * L * N, ITEM_MIX = N * N + 2 * L * N;

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 widen4(const bf16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
  return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
__device__ __forceinline__ void fma4(float4& d, float a, float4 b) {
  d.x = fmaf(a, b.x, d.x); d.y = fmaf(a, b.y, d.y); d.z = fmaf(a, b.z, d.z); d.w = fmaf(a, b.w, d.w);
}
__device__ __forceinline__ float dot4(float4 a, float4 b, float d) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, d))));
}

// W2 tanh(lora) of tokens t0 .. t0 + T - 1 for one channel
template <int T>
__device__ __forceinline__ void low_rank_rows(const ChunkArgs& a, float (&z)[T], const float* th_s, int channel, int t0) {
  const int RP = (a.R + 7) & ~7;
  const bf16* w2 = a.w2 + (size_t)channel * a.R;
  const bool wide = a.R % 8 == 0 && ((uintptr_t)a.w2 & 7) == 0;  // in pieces of four
#pragma unroll
  for (int t = 0; t < T; ++t) z[t] = 0.f;
  for (int m = 0; m < RP; m += 8) {
    float w[8];
    if (wide) {
      st4(w, widen4(w2 + m));
      st4(w + 4, widen4(w2 + m + 4));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = m + i < a.R ? __bfloat162float(w2[m + i]) : 0.f;
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const float4 x = ld4(th_s + (t0 + t) * RP + m), y = ld4(th_s + (t0 + t) * RP + m + 4);
      z[t] = fmaf(x.w, w[3], fmaf(x.z, w[2], fmaf(x.y, w[1], fmaf(x.x, w[0], z[t]))));
      z[t] = fmaf(y.w, w[7], fmaf(y.z, w[6], fmaf(y.y, w[5], fmaf(y.x, w[4], z[t]))));
    }
  }
}

// tanh of the low-rank input in the path's precision, [L][R rounded up to 8], zeros beyond the tokens and R
__device__ __forceinline__ void load_tanh(const ChunkArgs& a, float* th_s, size_t row0, int nt) {
  const int RP = (a.R + 7) & ~7;
  for (int t = threadIdx.x >> 3; t < L; t += blockDim.x >> 3)
    for (int m = threadIdx.x & 7; m < RP; m += 8)
      th_s[t * RP + m] = t < nt && m < a.R ? round_to<bf16>(tanhf(__bfloat162float(a.lora[(row0 + t) * a.lora_stride + m]))) : 0.f;
}
// A warp's place in a product of 64 columns: 16 columns a warp, lanes 8 x 4, neighbouring lanes sharing a row or a column
// (a warp's 16-byte read of shared memory then takes 2 cycles, not 4).
struct Place {
  int ty, col;
  __device__ Place() {
    const int lane = threadIdx.x & 31;
    ty = (lane & 15) >> 1;
    col = (threadIdx.x >> 5) * 16 + 4 * ((lane & 1) + 2 * (lane >> 4));
  }
};

// ---- products on the tensor cores ----------------------------------------------------------------------------------
// mma.sync m16n8k16, float32 accumulate. Values are bfloat16 already; every other operand is handed over as three bfloat16 terms
// that add up to it, and where both sides are such sums the six products that matter in 32-bit are formed, small ones first.
constexpr int KP = N + 8;   // bfloat16 rows in shared memory: ldmatrix reads eight of them from different banks
constexpr int PP = L + 8;
__device__ __forceinline__ void split3_store(bf16* dst, int apart, float x) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint32_t b = pack_bf16x2(x, 0.f);
    *reinterpret_cast<unsigned short*>(dst + i * apart) = (unsigned short)b;
    x -= __uint_as_float(b << 16);
  }
}
__device__ __forceinline__ void split3_store4(bf16* dst, int apart, float4 x) {
  uint32_t lo[3], hi[3];
  split3_pair(x.x, x.y, lo);
  split3_pair(x.z, x.w, hi);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(dst + i * apart) = make_uint2(lo[i], hi[i]);
}
// Returns whether one of this thread's is not finite: an exponent of ones, to which its lowest bit is added, leaves its field.
__device__ __forceinline__ bool load_raw(bf16* dst, const bf16* src, int stride, size_t row0, int ch0, int nt) {
  uint32_t over = 0u;
#pragma unroll
  for (int i = threadIdx.x; i < L * (N / 4); i += THREADS) {
    const int t = i / (N / 4), c = (i % (N / 4)) * 4;
    const uint2 four = t < nt ? *reinterpret_cast<const uint2*>(src + (row0 + t) * stride + ch0 + c) : make_uint2(0u, 0u);
    *reinterpret_cast<uint2*>(dst + t * KP + c) = four;
    over |= ((four.x & 0x7f807f80u) + 0x00800080u) | ((four.y & 0x7f807f80u) + 0x00800080u);
  }
  return over & 0x80008000u;
}

// The five small products of two operands that are three terms each, into one tile of 16 x 8. The sixth, of the leading terms, is added
// after the small ones of all of a sum's k: the tensor cores cut every sum off, and a small product would cost a large one its last bit.
__device__ __forceinline__ void small33(float (&d)[4], const uint32_t (&x)[3][4], const uint32_t (&y)[3][2]) {
#pragma unroll
  for (int sum = 2; sum >= 1; --sum)
#pragma unroll
    for (int t = 0; t <= sum; ++t) mma_bf16_16816(d, x[t][0], x[t][1], x[t][2], x[t][3], y[sum - t][0], y[sum - t][1]);
}

// ---- pass 1, delta rule ----------------------------------------------------------------------------------------
// Eight warps. A thread makes one channel of eight tokens' rows; six warps multiply [U; Rows] [K; A]^T, a warp four tiles of 16 x 8; four
// solve for a column of [X | Z] a thread, with float32 multiply-adds, while the other four multiply K^T V; then four multiply A^T X
// and four A^T Z, and all of them eight columns of Q and O each. X and Z are kept with their signs turned.
// Two blocks an SM. Bound by its chains and barriers, the substitution's before all. One prompt of 2,048 tokens, 8 heads: 50 us (57 from
// a cold cache; with float32 on the CUDA cores, three blocks of four warps an SM, 63).
__global__ void __launch_bounds__(DELTA_THREADS, 2) delta_chunk_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int TERM = L * KP, ROWS3 = 3 * TERM;       // elements of one term of a chunk's rows, of three
  bf16* ut = reinterpret_cast<bf16*>(sm);              // [3][L][KP] u_t e^{c_{t-1}}; then -X
  bf16* rt = ut + ROWS3;                               // [3][L][KP] r_t e^{c_t}
  bf16* kt = rt + ROWS3;                               // [3][L][KP] k_s e^{-c_s}
  bf16* at = kt + ROWS3;                               // [3][L][KP] a_s u_s e^{-c_s}
  bf16* zt = at + ROWS3;                               // [3][L][KP] -Z
  bf16* pt = zt + ROWS3;                               // [3][L][KP] P beside R
  bf16* vs = pt + ROWS3;                               // [L][KP] the values, what is not finite set aside
  float* us = reinterpret_cast<float*>(vs + TERM);     // [L][PITCH] u_t e^{c_{t-1}}
  float* es = us + L * PITCH;                          // [L][PITCH] B beside D
  float* last = es + L * PITCH;                        // [N] e^{c_last}
  float* sq = last + N;                                // [2][L] |k|^2, of either half of the channels
  float2* total = reinterpret_cast<float2*>(sq + 2 * L);  // [4][N] a part's decays, summed, and what that rounded off
  int* bad = reinterpret_cast<int*>(total + 4 * N);    // [4][N]: the first token that is not finite in a column of X, of Z; with an
                                                       // infinity in a column of the values, with a NaN
  float* th_s = us;                                    // [L][R rounded up], over us and es; gone before they are written
  const int h = blockIdx.x, ci = blockIdx.y, seq = blockIdx.z, ch0 = h * N;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  grid_dependency_wait();
  const int first = (a.chunk0 + ci) * L, nt = min(L, a.seq_qlen[seq] - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const int ch = tid & (N - 1), part = tid / N, t0 = part * PART;
  float r[PART], k[PART], rate[PART];
#pragma unroll
  for (int i = 0; i < PART; ++i) {
    const bool in = t0 + i < nt;
    const size_t row = row0 + t0 + i;
    r[i] = in ? __bfloat162float(a.r[row * a.r_stride + ch0 + ch]) : 0.f;
    k[i] = in ? __bfloat162float(a.k[row * a.k_stride + ch0 + ch]) : 0.f;
    rate[i] = in ? __bfloat162float(a.rate[row * a.rate_stride + ch0 + ch]) : 0.f;
  }
  if (tid < 4 * N) bad[tid] = L;
  load_tanh(a, th_s, row0, nt);
  __syncthreads();
  for (int i = tid; i < L * (N / 4); i += DELTA_THREADS) {  // the values
    const int t = i / (N / 4), c = (i % (N / 4)) * 4;
    const uint2 raw = t < nt ? *reinterpret_cast<const uint2*>(a.v + (row0 + t) * a.v_stride + ch0 + c) : make_uint2(0u, 0u);
    uint32_t two[2] = {raw.x, raw.y};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const bool lo = (two[j] & 0x7f80u) == 0x7f80u, hi = (two[j] & 0x7f800000u) == 0x7f800000u;
      if (lo) atomicMin(bad + (two[j] & 0x7fu ? 3 * N : 2 * N) + c + 2 * j, t);
      if (hi) atomicMin(bad + (two[j] & 0x7f0000u ? 3 * N : 2 * N) + c + 2 * j + 1, t);
      if (lo || hi) two[j] &= (lo ? 0xffff0000u : 0xffffffffu) & (hi ? 0xffffu : 0xffffffffu);
    }
    *reinterpret_cast<uint2*>(vs + t * KP + c) = make_uint2(two[0], two[1]);
  }
  float c[PART], rest[PART];  // the log decays summed over the chunk's tokens (zero decay beyond the last), and what the running sums round off:
                              // a sum of 18 rounds at 1e-6, which e^c would multiply everything by
  {
    low_rank_rows<PART>(a, c, th_s, ch0 + ch, t0);
    const float w0 = a.w0[ch0 + ch];
    float run = 0.f, lost = 0.f;
#pragma unroll
    for (int i = 0; i < PART; ++i) {
      float x = -a.decay_scale * sigmoid_f(c[i] + w0);
      if (t0 + i >= nt) x = 0.f;
      const float sum = run + x, y = sum - run;
      lost += (run - (sum - y)) + (x - y);
      rest[i] = lost;
      c[i] = run = sum;
    }
    total[part * N + ch] = make_float2(run, lost);
#pragma unroll
    for (int i = 0; i < PART; ++i) {
      const float s = warp_sum(k[i] * k[i]);
      if (lane == 0) sq[(warp & 1) * L + t0 + i] = s;
    }
  }
  __syncthreads();  // th_s is no longer read
  {
    float before = 0.f, before1 = 0.f;  // the sums of the parts before
    for (int q = 0; q < part; ++q) {
      const float2 f = total[q * N + ch];
      const float sum = before + f.x, y = sum - before;
      before1 += f.y + ((before - (sum - y)) + (f.x - y));
      before = sum;
    }
    const float bias = a.rate_bias[ch0 + ch];
    float c_prev = before, c1_prev = before1;
#pragma unroll
    for (int i = 0; i < PART; ++i) {
      const int t = t0 + i, at1 = t * KP + ch;
      const float sum = before + c[i], y = sum - before;
      const float c1 = rest[i] + before1 + ((before - (sum - y)) + (c[i] - y));
      const float u = k[i] * rsqrtf(sq[t] + sq[L + t] + 1e-6f), back = expf(-sum) * (1.f - c1), on = expf(sum) * (1.f + c1);
      const float ue = u * (expf(c_prev) * (1.f + c1_prev));
      us[t * PITCH + ch] = ue;
      split3_store(ut + at1, TERM, ue);
      split3_store(rt + at1, TERM, r[i] * on);
      split3_store(kt + at1, TERM, k[i] * back);
      split3_store(at + at1, TERM, sigmoid_f(rate[i] + bias) * u * back);
      c_prev = sum;
      c1_prev = c1;
      if (t == L - 1) last[ch] = on;
    }
  }
  __syncthreads();
  if (warp < 6) {  // [U; Rows] [K; A]^T without the tiles that look ahead
    // warps 0, 3: tokens 0..15 of U, of Rows, against tokens 0..15 of K and A; 1, 4: tokens 16..31 against K; 2, 5: against A
    const int which = warp % 3;
    const bool rows = warp >= 3;
    const int m0 = which ? 16 : 0;
    const bf16* x = rows ? rt : ut;
    float e[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) e[j][q] = 0.f;
#pragma unroll
    for (int leading = 0; leading < 2; ++leading)
#pragma unroll
      for (int kk = 0; kk < N; kk += 16) {
        uint32_t xf[3][4];
#pragma unroll
        for (int t = 0; t < (leading ? 1 : 3); ++t)
          ldmatrix_x4(xf[t][0], xf[t][1], xf[t][2], xf[t][3], x + t * TERM + (m0 + (lane & 15)) * KP + kk + (lane >> 4) * 8);
#pragma unroll
        for (int j = 0; j < 4; j += 2) {  // 16 tokens of K or A
          const bf16* y = (which == 0 ? j == 2 : which == 2) ? at : kt;
          const int s0 = which == 0 ? 0 : j * 8;
          uint32_t y0[3][2], y1[3][2];
#pragma unroll
          for (int t = 0; t < (leading ? 1 : 3); ++t)
            ldmatrix_x4(y0[t][0], y0[t][1], y1[t][0], y1[t][1],
                        y + t * TERM + (s0 + ((lane >> 4) << 3) + (lane & 7)) * KP + kk + ((lane >> 3) & 1) * 8);
          if (leading) {
            mma_bf16_16816(e[j], xf[0][0], xf[0][1], xf[0][2], xf[0][3], y0[0][0], y0[0][1]);
            mma_bf16_16816(e[j + 1], xf[0][0], xf[0][1], xf[0][2], xf[0][3], y1[0][0], y1[0][1]);
          } else {
            small33(e[j], xf, y0);
            small33(e[j + 1], xf, y1);
          }
        }
      }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int s0 = (which == 0 ? (j & 1) * 8 : j * 8) + 2 * t4;              // the token of K or A
      const int col = s0 + ((which == 0 ? j >= 2 : which == 2) ? L : 0);       // B or P in front, D or R behind
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int t = m0 + g + 8 * hh;
        if (!rows) {
          *reinterpret_cast<float2*>(es + t * PITCH + col) = make_float2(s0 < t ? e[j][2 * hh] : 0.f, s0 + 1 < t ? e[j][2 * hh + 1] : 0.f);
        } else {
          uint32_t three[3];
          split3_pair(s0 <= t ? e[j][2 * hh] : 0.f, s0 + 1 <= t ? e[j][2 * hh + 1] : 0.f, three);
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(pt + i * TERM + t * KP + col) = three[i];
        }
      }
    }
  }
  __syncthreads();
  float* item = a.scratch + (((size_t)seq * a.n_chunks + ci) * a.H + h) * ITEM_DELTA;
  const int m0 = (warp & 3) * 16;  // key channels of this warp's tiles of M (warps 0..3) or G (4..7)
  float d[N / 8][4];
#pragma unroll
  for (int n = 0; n < N / 8; ++n)
#pragma unroll
    for (int q = 0; q < 4; ++q) d[n][q] = 0.f;
  // 16 rows of the transpose of a term's rows, of tokens s .. s + 15
  auto transposed = [&](uint32_t (&f)[4], const bf16* rows, int s) {
    ldmatrix_x4_trans(f[0], f[1], f[2], f[3], rows + (s + (lane & 7) + ((lane >> 4) & 1) * 8) * KP + m0 + ((lane >> 3) & 1) * 8);
  };
  auto tokens = [&](uint32_t (&f)[4], const bf16* rows, int s, int n) {  // tokens s .. s + 15 of columns 8 n .. 8 n + 15
    ldmatrix_x4_trans(f[0], f[1], f[2], f[3], rows + (s + (lane & 7) + ((lane >> 3) & 1) * 8) * KP + (n + (lane >> 4)) * 8);
  };
  if (warp < 4) {  // forward substitution, a column of [X | Z] a thread; four partial sums a row
    const bool is_z = warp >= 2;
    const int col = tid & (N - 1);
    float x[L];
    int nonfinite = L;
    if (!is_z) {
#pragma unroll
      for (int t = 0; t < L; ++t) {
        float p[4] = {us[t * PITCH + col], 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < t; s += 4) {
          const float4 e = ld4(es + t * PITCH + L + s);
          p[0] = fmaf(-e.x, x[s], p[0]);
          if (s + 1 < t) p[1] = fmaf(-e.y, x[s + 1], p[1]);
          if (s + 2 < t) p[2] = fmaf(-e.z, x[s + 2], p[2]);
          if (s + 3 < t) p[3] = fmaf(-e.w, x[s + 3], p[3]);
        }
        x[t] = (p[0] + p[1]) + (p[2] + p[3]);
      }
    } else {
      float v[L];
#pragma unroll
      for (int t = 0; t < L; ++t) v[t] = t < nt ? __bfloat162float(a.v[(row0 + t) * a.v_stride + ch0 + col]) : 0.f;
#pragma unroll
      for (int t = 0; t < L; ++t) {
        float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < t; s += 4) {
          const float4 b = ld4(es + t * PITCH + s), e = ld4(es + t * PITCH + L + s);
          p[0] = fmaf(-e.x, x[s], fmaf(b.x, v[s], p[0]));
          if (s + 1 < t) p[1] = fmaf(-e.y, x[s + 1], fmaf(b.y, v[s + 1], p[1]));
          if (s + 2 < t) p[2] = fmaf(-e.z, x[s + 2], fmaf(b.z, v[s + 2], p[2]));
          if (s + 3 < t) p[3] = fmaf(-e.w, x[s + 3], fmaf(b.w, v[s + 3], p[3]));
        }
        x[t] = (p[0] + p[1]) + (p[2] + p[3]);
      }
    }
    bf16* to = (is_z ? zt : ut) + col;
#pragma unroll
    for (int t = L - 1; t >= 0; --t) {
      const bool in = fabsf(x[t]) < INFINITY;
      if (!in) nonfinite = t;
      split3_store(to + t * KP, TERM, in ? -x[t] : 0.f);  // a product would hand what is not finite, times zero, to the tokens before
    }
    bad[(is_z ? N : 0) + col] = nonfinite;
  } else {  // K^T V: the small terms of K
#pragma unroll
    for (int s = 0; s < L; s += 16) {
      uint32_t kf[2][4];
      transposed(kf[0], kt + TERM, s);
      transposed(kf[1], kt + 2 * TERM, s);
#pragma unroll
      for (int n = 0; n < N / 8; n += 2) {
        uint32_t b[4];
        tokens(b, vs, s, n);
#pragma unroll
        for (int t = 1; t >= 0; --t) {
          mma_bf16_16816(d[n], kf[t][0], kf[t][1], kf[t][2], kf[t][3], b[0], b[1]);
          mma_bf16_16816(d[n + 1], kf[t][0], kf[t][1], kf[t][2], kf[t][3], b[2], b[3]);
        }
      }
    }
  }
  __syncthreads();
  // only now: a block of the walk that waited from the start would hold the shared memory that this kernel's blocks need
  grid_launch_dependents();
  {  // M and G: - A^T X, K^T V - A^T Z
    const bool is_g = warp >= 4;
    const bf16* y = is_g ? zt : ut;
#pragma unroll
    for (int s = 0; s < L; s += 16) {
      uint32_t af[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t) transposed(af[t], at + t * TERM, s);
#pragma unroll
      for (int n = 0; n < N / 8; n += 2) {
        uint32_t y0[3][2], y1[3][2];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          uint32_t f[4];
          tokens(f, y + t * TERM, s, n);
          y0[t][0] = f[0]; y0[t][1] = f[1]; y1[t][0] = f[2]; y1[t][1] = f[3];
        }
        small33(d[n], af, y0);
        small33(d[n + 1], af, y1);
      }
    }
#pragma unroll
    for (int s = 0; s < L; s += 16) {
      uint32_t af[4], kf[4];
      transposed(af, at, s);
      transposed(kf, kt, s);
#pragma unroll
      for (int n = 0; n < N / 8; n += 2) {
        uint32_t f[4];
        tokens(f, y, s, n);
        mma_bf16_16816(d[n], af[0], af[1], af[2], af[3], f[0], f[1]);
        mma_bf16_16816(d[n + 1], af[0], af[1], af[2], af[3], f[2], f[3]);
        if (is_g) {
          tokens(f, vs, s, n);
          mma_bf16_16816(d[n], kf[0], kf[1], kf[2], kf[3], f[0], f[1]);
          mma_bf16_16816(d[n + 1], kf[0], kf[1], kf[2], kf[3], f[2], f[3]);
        }
      }
    }
    const int* worst = bad + (is_g ? N : 0);
#pragma unroll
    for (int n = 0; n < N / 8; ++n)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int row = m0 + g + 8 * hh, col = n * 8 + 2 * t4;
        const float w = last[row];
        float v[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          v[j] = d[n][2 * hh + j];
          if (!is_g && row == col + j) v[j] += 1.f;
          if (is_g && min(bad[2 * N + col + j], bad[3 * N + col + j]) < L) {
            // a value that is not finite: the tokens after it have read it (NaN), unless it is the chunk's last
            const bf16* key = kt + (nt - 1) * KP + row;
            const float k0 = __bfloat162float(key[0]), k1 = k0 + (__bfloat162float(key[TERM]) + __bfloat162float(key[2 * TERM]));
            v[j] = fmaf(fabsf(k0) < INFINITY ? k1 : k0, __bfloat162float(a.v[(row0 + nt - 1) * a.v_stride + ch0 + col + j]), v[j]);
          }
          v[j] = worst[col + j] < nt ? NAN : w * v[j];
        }
        *reinterpret_cast<float2*>(item + (is_g ? N * N : 0) + row * N + col) = make_float2(v[0], v[1]);
      }
  }
  {  // Q and O: columns 8 warp .. 8 warp + 7 of Rows - R X and of P V - R Z
    const int c0 = warp * 8, col = c0 + 2 * t4;
    float q[2][4], o[2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j) q[m][j] = o[m][j] = 0.f;
    uint32_t xf[3][4], zf[3][4], vf[4];  // of 32 tokens: two of sixteen
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      ldmatrix_x4_trans(xf[t][0], xf[t][1], xf[t][2], xf[t][3], ut + t * TERM + lane * KP + c0);
      ldmatrix_x4_trans(zf[t][0], zf[t][1], zf[t][2], zf[t][3], zt + t * TERM + lane * KP + c0);
    }
    ldmatrix_x4_trans(vf[0], vf[1], vf[2], vf[3], vs + lane * KP + c0);
#pragma unroll
    for (int leading = 0; leading < 2; ++leading)
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int kk = 0; kk <= m; ++kk) {  // not later tokens
          uint32_t pf[3][4], rf[3][4];
#pragma unroll
          for (int t = 0; t < (leading ? 1 : 3); ++t) {
            const bf16* from = pt + t * TERM + (m * 16 + (lane & 15)) * KP + kk * 16 + (lane >> 4) * 8;
            if (leading || t) ldmatrix_x4(pf[t][0], pf[t][1], pf[t][2], pf[t][3], from);
            ldmatrix_x4(rf[t][0], rf[t][1], rf[t][2], rf[t][3], from + L);
          }
          if (leading) {
            mma_bf16_16816(q[m], rf[0][0], rf[0][1], rf[0][2], rf[0][3], xf[0][2 * kk], xf[0][2 * kk + 1]);
            mma_bf16_16816(o[m], rf[0][0], rf[0][1], rf[0][2], rf[0][3], zf[0][2 * kk], zf[0][2 * kk + 1]);
            mma_bf16_16816(o[m], pf[0][0], pf[0][1], pf[0][2], pf[0][3], vf[2 * kk], vf[2 * kk + 1]);
          } else {
            uint32_t x2[3][2], z2[3][2];
#pragma unroll
            for (int t = 0; t < 3; ++t)
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                x2[t][j] = xf[t][2 * kk + j];
                z2[t][j] = zf[t][2 * kk + j];
              }
            small33(q[m], rf, x2);
            small33(o[m], rf, z2);
#pragma unroll
            for (int t = 2; t >= 1; --t) mma_bf16_16816(o[m], pf[t][0], pf[t][1], pf[t][2], pf[t][3], vf[2 * kk], vf[2 * kk + 1]);
          }
        }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int t = m * 16 + g + 8 * hh;
        float v[2], w[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const bf16* from = rt + t * KP + col + j;
          const float row = __bfloat162float(from[0]) + (__bfloat162float(from[TERM]) + __bfloat162float(from[2 * TERM]));  // r e^c again
          v[j] = t >= bad[col + j] ? NAN : row + q[m][2 * hh + j];
          w[j] = t >= min(bad[N + col + j], bad[3 * N + col + j]) ? NAN : t >= bad[2 * N + col + j] ? INFINITY : o[m][2 * hh + j];
        }
        *reinterpret_cast<float2*>(item + 2 * N * N + t * N + col) = make_float2(v[0], v[1]);
        *reinterpret_cast<float2*>(item + 2 * N * N + L * N + t * N + col) = make_float2(w[0], w[1]);
      }
  }
}

// ---- pass 1, time mixing ---------------------------------------------------------------------------------------
// A thread has its channel's decays in registers, and sums them from either end: the weights e^{c_last - c_s} from the last token
// back and the running sums c_t from the first one on. Neither is a difference of sums, in which a small decay after
// large ones would be lost. Eight blocks an SM: 45 us where seven take 50 and the float32 form took 57 (2,553 tokens, 40 heads).
__global__ void __launch_bounds__(THREADS, 8) mix_chunk_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float sm[];
  bf16* kt = reinterpret_cast<bf16*>(sm);      // [3][L][KP] k_s e^{c_last - c_s}
  bf16* vs = kt + 3 * L * KP;                  // [L][KP]
  bf16* ks = vs + L * KP;                      // [L][KP]
  float* th_s = reinterpret_cast<float*>(ks + L * KP);  // [L][R rounded up]
  float* total = th_s + L * ((a.R + 7) & ~7);  // [2][N]
  const int h = blockIdx.x, ci = blockIdx.y, seq = blockIdx.z, ch0 = h * N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  grid_dependency_wait();
  const int first = (a.chunk0 + ci) * L, nt = min(L, a.seq_qlen[seq] - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const bool odd_key = load_raw(ks, a.k, a.k_stride, row0, ch0, nt), odd_value = load_raw(vs, a.v, a.v_stride, row0, ch0, nt);
  load_tanh(a, th_s, row0, nt);
  const bool odd = __syncthreads_or(odd_key || odd_value);
  float* item = a.scratch + (((size_t)seq * a.n_chunks + ci) * a.H + h) * ITEM_MIX;
  {
    const int ch = threadIdx.x & (N - 1), half = threadIdx.x / N, t0 = half * HALF;
    float x[HALF], run = 0.f;
    low_rank_rows<HALF>(a, x, th_s, ch0 + ch, t0);
    const float w0 = a.w0[ch0 + ch];
#pragma unroll
    for (int t = 0; t < HALF; ++t) {
      x[t] = t0 + t < nt ? -expf(x[t] + w0) : 0.f;  // zero decay beyond the last token
      run += x[t];
    }
    total[half * N + ch] = run;
    __syncthreads();
    grid_launch_dependents();
    const float other = total[(half ^ 1) * N + ch];
    const float before = half ? other : 0.f;
    float after = half ? 0.f : other, c = before;
    run = 0.f;
#pragma unroll
    for (int t = 0; t < HALF; ++t) {
      run += x[t];
      c = before + run;
      item[N * N + (t0 + t) * N + ch] = c;
    }
#pragma unroll
    for (int t = HALF - 1; t >= 0; --t) {
      const int at = (t0 + t) * KP + ch;
      split3_store(kt + at, L * KP, __bfloat162float(ks[at]) * expf(after));
      after += x[t];
    }
    if (__syncthreads_or(half && !(c > -SAFE)))  // pass 3 will form the pair sums from the decays themselves
#pragma unroll
      for (int t = 0; t < HALF; ++t) item[N * N + L * N + (t0 + t) * N + ch] = expf(x[t]);
  }
  const int m0 = warp * 16;  // key channels of this warp
  float g[N / 8][4];
#pragma unroll
  for (int n = 0; n < N / 8; ++n)
#pragma unroll
    for (int c = 0; c < 4; ++c) g[n][c] = 0.f;
  // the small terms of all tokens before the leading ones: the tensor cores cut every sum off
#pragma unroll
  for (int leading = 0; leading < 2; ++leading)
#pragma unroll
    for (int s = 0; s < L; s += 16) {
      uint32_t af[2][4];
#pragma unroll
      for (int t = 0; t < (leading ? 1 : 2); ++t)  // the transpose of the keys' rows
        ldmatrix_x4_trans(af[t][0], af[t][1], af[t][2], af[t][3],
                          kt + ((leading ? 0 : 2 - t) * L + s + (lane & 7) + ((lane >> 4) & 1) * 8) * KP + m0 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int n = 0; n < N / 8; n += 2) {
        uint32_t b[4];
        ldmatrix_x4_trans(b[0], b[1], b[2], b[3], vs + (s + (lane & 7) + ((lane >> 3) & 1) * 8) * KP + (n + (lane >> 4)) * 8);
#pragma unroll
        for (int t = 0; t < (leading ? 1 : 2); ++t) {
          mma_bf16_16816(g[n], af[t][0], af[t][1], af[t][2], af[t][3], b[0], b[1]);
          mma_bf16_16816(g[n + 1], af[t][0], af[t][1], af[t][2], af[t][3], b[2], b[3]);
        }
      }
    }
#pragma unroll
  for (int n = 0; n < N / 8; ++n)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
      *reinterpret_cast<float2*>(item + (m0 + (lane >> 2) + 8 * hh) * N + n * 8 + 2 * (lane & 3)) = make_float2(g[n][2 * hh], g[n][2 * hh + 1]);
  if (odd) {  // the terms of an infinity do not add up to it: what came out not finite, again with multiply-adds
#pragma unroll 1
    for (int i = 0; i < N / 2; ++i) {
      const int n = m0 + (lane >> 2) + (i & 2) * 4, p = (i >> 2) * 8 + 2 * (lane & 3) + (i & 1);  // this thread's own sums
      if (fabsf(item[n * N + p]) < INFINITY) continue;
      float sum = 0.f;
#pragma unroll 1
      for (int t = 0; t < nt; ++t) {
        const bf16* key = kt + t * KP + n;
        const float k0 = __bfloat162float(key[0]), k1 = k0 + (__bfloat162float(key[L * KP]) + __bfloat162float(key[2 * L * KP]));
        sum = fmaf(fabsf(k0) < INFINITY ? k1 : k0, __bfloat162float(vs[t * KP + p]), sum);
      }
      item[n * N + p] = sum;
    }
  }
}

// ---- pass 2 ----------------------------------------------------------------------------------------------------
// Delta rule: a block walks WALK_COLS value columns of one (sequence, head). Four warps have sixteen of the 64 key channels' rows
// each; a lane takes four rows against eight channels, and eight lanes hand their shares round until each has two numbers of
// the new state: one barrier a chunk. A fifth warp asks for the chunks' M and columns of G five chunks ahead, as tiled copies, and waits
// for them. Bound by the chain of a step: the state from shared memory, 32 multiply-adds of four columns, three exchanges, the
// barrier. One prompt of 2,048 tokens, 8 heads, the three passes back to back: 111 us with 16-byte copies by the walkers (32 a step)
// and two barriers, 101 here; the walk by itself 34.0 and 31.6 us, from a cold cache 35.6 and 33.1.
constexpr int WALKERS = 128, WALK_THREADS = WALKERS + 32;
constexpr int WALK_M = N * N, WALK_G = N * WALK_COLS;         // floats of a chunk's M and of its columns of G
constexpr int WALK_SP = 36;                                   // floats from eight channels of the state to the next eight: other banks
__global__ void __launch_bounds__(WALK_THREADS)
delta_walk_kernel(const __grid_constant__ CUtensorMap map_m, const __grid_constant__ CUtensorMap map_g, ChunkArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* ms = reinterpret_cast<float*>(((uintptr_t)sm + 1023) & ~(uintptr_t)1023);  // [WALK_STAGES][2][N][32], 128-byte swizzle
  float* gs = ms + WALK_STAGES * WALK_M;                                            // [WALK_STAGES][N][WALK_COLS]
  float* ss = gs + WALK_STAGES * WALK_G;                                            // [2][N / 8][WALK_SP] the state's columns, in turn
  __shared__ uint64_t full[WALK_STAGES];
  const int p0 = blockIdx.x * WALK_COLS, h = blockIdx.y, seq = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    for (int i = 0; i < WALK_STAGES; ++i) tc::mbar_init(full + i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  grid_dependency_wait();
  const int n_chunks = min(a.n_chunks, (a.seq_qlen[seq] + L - 1) / L - a.chunk0);
  if (n_chunks <= 0) return;
  auto step_sync = [] { asm volatile("bar.sync 1, 160;" ::: "memory"); };
  if (warp == WALKERS / 32) {
    // The fifth warp waits for the copies, so that no walker has to: at a step's barrier the next chunk but one is here. A
    // chunk's place is free when the step before it is over, since the walkers read a chunk a step ahead.
    int asked = 0;
    bool late = false;  // a wait has run out: the step's results are not to be used, which the error word says; no more is asked for or waited for
    auto request = [&](int c) {
      if (c >= n_chunks || late) return;
      asked = c + 1;
      if (lane != 0) return;
      const int b = c % WALK_STAGES, row = ((seq * a.n_chunks + c) * a.H + h) * (ITEM_DELTA / N);
      tc::mbar_expect_tx(full + b, (WALK_M + WALK_G) * sizeof(float));
      tc::tma_load_2d(ms + b * WALK_M, &map_m, full + b, 0, row);
      tc::tma_load_2d(ms + b * WALK_M + N * 32, &map_m, full + b, 32, row);
      tc::tma_load_2d(gs + b * WALK_G, &map_g, full + b, p0, row + N);
    };
    auto wait = [&](int c) {
      if (c >= n_chunks || late || __all_sync(0xffffffffu, tc::mbar_wait(full + c % WALK_STAGES, (c / WALK_STAGES) & 1))) return;
      late = true;
      if (lane == 0) atomicExch(a.error, 24);
    };
    for (int c = 0; c < WALK_STAGES; ++c) request(c);
    wait(0);
    wait(1);
    step_sync();
    for (int c = 0; c < n_chunks; ++c) {
      if (c) request(c + WALK_STAGES - 1);
      wait(c + 2);
      step_sync();
    }
    if (late) tc::wait_for_copies(full, WALK_STAGES, asked);
    return;
  }
  const int kg = lane & 7, half = kg >> 2, r0 = warp * 16 + (lane >> 3) * 4;
  const int row = r0 + 2 * half + ((lane >> 1) & 1), col = 2 * (lane & 1);  // what this lane has of the state: two columns of a channel
  float* items = a.scratch + ((size_t)seq * a.n_chunks * a.H + h) * ITEM_DELTA + N * N + row * N + p0 + col;
  const size_t step = (size_t)a.H * ITEM_DELTA;
  float2* st = reinterpret_cast<float2*>(a.state + ((size_t)a.seq_slot[seq] * a.H + h) * N * N + row * N + p0 + col);
  const int at = (row >> 3) * WALK_SP + (row & 7) * WALK_COLS + col;
  float2 mine = *st;
  *reinterpret_cast<float2*>(ss + at) = mine;
  step_sync();
  int b = 0;
  float4 x[4][2];  // a chunk's M, in registers before the state that it meets is there
  float2 own;
  auto fetch = [&] {
    const float* m = ms + b * WALK_M + half * (N * 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + i;
#pragma unroll
      for (int j = 0; j < 2; ++j)  // the upper channels' lanes take their second four first, for the banks' sake
        x[i][j] = ld4(m + r * 32 + ((((kg & 3) * 2 + (j ^ half)) ^ (r & 7)) << 2));
    }
    own = *reinterpret_cast<const float2*>(gs + b * WALK_G + row * WALK_COLS + col);
  };
  fetch();
  for (int c = 0; c < n_chunks; ++c) {
    const float* s = ss + (c & 1) * (N / 8) * WALK_SP + kg * WALK_SP;
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float* sj = s + (j ^ half) * 16;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 state = ld4(sj + 4 * e);
#pragma unroll
        for (int i = 0; i < 4; ++i) fma4(v[i], e == 0 ? x[i][j].x : e == 1 ? x[i][j].y : e == 2 ? x[i][j].z : x[i][j].w, state);
      }
    }
    const float2 g = own;
    if (++b == WALK_STAGES) b = 0;
    if (c + 1 < n_chunks) fetch();
    *reinterpret_cast<float2*>(items + c * step) = mine;  // the chunk's starting state, in G's place
    auto exchange = [](float keep, float send, int by) { return keep + __shfl_xor_sync(0xffffffffu, send, by); };
    const bool up = half, up1 = lane & 2, up2 = lane & 1;
    float4 w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 k = up ? v[2 + i] : v[i], d = up ? v[i] : v[2 + i];
      w[i] = make_float4(exchange(k.x, d.x, 4), exchange(k.y, d.y, 4), exchange(k.z, d.z, 4), exchange(k.w, d.w, 4));
    }
    const float4 k = up1 ? w[1] : w[0], d = up1 ? w[0] : w[1];
    const float4 y = make_float4(exchange(k.x, d.x, 2), exchange(k.y, d.y, 2), exchange(k.z, d.z, 2), exchange(k.w, d.w, 2));
    mine = make_float2(g.x + exchange(up2 ? y.z : y.x, up2 ? y.x : y.z, 1), g.y + exchange(up2 ? y.w : y.y, up2 ? y.y : y.w, 1));
    *reinterpret_cast<float2*>(ss + ((c + 1) & 1) * (N / 8) * WALK_SP + at) = mine;
    step_sync();  // the new state is here, and the old one is no longer read
  }
  grid_launch_dependents();
  *st = mine;
}

// Time mixing: every element of the state by itself, four neighbours a thread.
__global__ void mix_walk_kernel(ChunkArgs a) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int h = blockIdx.y, seq = blockIdx.z;
  const int n_chunks = min(a.n_chunks, (a.seq_qlen[seq] + L - 1) / L - a.chunk0);
  if (n_chunks <= 0) return;
  const int e = 4 * (blockIdx.x * blockDim.x + threadIdx.x), n = e / N;
  float* st = a.state + ((size_t)a.seq_slot[seq] * a.H + h) * N * N + e;
  float* items = a.scratch + ((size_t)seq * a.n_chunks * a.H + h) * ITEM_MIX;
  const size_t step = (size_t)a.H * ITEM_MIX;
  float4 run = ld4(st);
  for (int c0 = 0; c0 < n_chunks; c0 += 8) {
    float4 own[8];
    float decay[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < n_chunks) {
        own[i] = __ldcg(reinterpret_cast<const float4*>(items + (c0 + i) * step + e));
        decay[i] = __ldcg(items + (c0 + i) * step + N * N + (L - 1) * N + n);
      }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < n_chunks) {
        st4(items + (c0 + i) * step + e, run);
        const float w = expf(decay[i]);
        run = make_float4(fmaf(w, run.x, own[i].x), fmaf(w, run.y, own[i].y), fmaf(w, run.z, own[i].z), fmaf(w, run.w, own[i].w));
      }
  }
  st4(st, run);
}

// ---- pass 3, delta rule ----------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS) delta_finish_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                 // [L][PITCH] rows that meet the state
  float* red = qs + L * PITCH;    // [4][L] sums of squares of a warp's columns
  grid_launch_dependents();
  grid_dependency_wait();
  const int h = blockIdx.x, ci = blockIdx.y, seq = blockIdx.z, ch0 = h * N;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int first = (a.chunk0 + ci) * L, qlen = a.seq_qlen[seq], nt = min(L, qlen - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const float* item = a.scratch + (((size_t)seq * a.n_chunks + ci) * a.H + h) * ITEM_DELTA;
  const Place at;
  // the state before the chunk: a value column is one warp's alone, so it is read from memory where it is used
  const float* start = item + N * N + at.col;
  auto state4 = [&](int n) { return __ldcg(reinterpret_cast<const float4*>(start + n * N)); };
  float4 o[4], s0[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) s0[j] = state4(j);
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = __ldcg(reinterpret_cast<const float4*>(item + 2 * N * N + L * N + (at.ty + 8 * i) * N + at.col));
  for (int i = tid; i < L * (N / 4); i += THREADS)
    cp_async_16(qs + (i / (N / 4)) * PITCH + (i % (N / 4)) * 4, item + 2 * N * N + 4 * i);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll 2
  for (int n = 0; n < N; n += 4) {
    float4 s1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) s1[j] = n + 4 < N ? state4(n + 4 + j) : s0[j];  // the next four rows are on the way
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 q = ld4(qs + (at.ty + 8 * i) * PITCH + n);
      fma4(o[i], q.x, s0[0]);
      fma4(o[i], q.y, s0[1]);
      fma4(o[i], q.z, s0[2]);
      fma4(o[i], q.w, s0[3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) s0[j] = s1[j];
  }
  // per head: divide by the root mean square, weight, gate, scale
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float sq = o[i].x * o[i].x + o[i].y * o[i].y + o[i].z * o[i].z + o[i].w * o[i].w;
    sq += __shfl_xor_sync(0xffffffffu, sq, 1);
    sq += __shfl_xor_sync(0xffffffffu, sq, 16);
    if ((tid & 17) == 0) red[warp * L + at.ty + 8 * i] = sq;
  }
  __syncthreads();
  const float4 w = ld4(a.norm_w + ch0 + at.col);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = at.ty + 8 * i;
    if (t >= nt) continue;
    const float sum = (red[t] + red[L + t]) + (red[2 * L + t] + red[3 * L + t]);
    const float by = rsqrtf(sum / (float)N + a.eps) * a.out_scale;
    const float4 g = widen4(a.g + (row0 + t) * a.g_stride + ch0 + at.col);
    uint2 raw;
    raw.x = pack_bf16x2(o[i].x * by * w.x * sigmoid_f(g.x), o[i].y * by * w.y * sigmoid_f(g.y));
    raw.y = pack_bf16x2(o[i].z * by * w.z * sigmoid_f(g.z), o[i].w * by * w.w * sigmoid_f(g.w));
    *reinterpret_cast<uint2*>(a.out + (row0 + t) * a.out_stride + a.out_col + ch0 + at.col) = raw;
  }
  if (a.last_rows && h == 0 && first + nt == qlen) {  // the sequence's last row, for the next step's token shift
    const bf16* row = a.last_rows + (row0 + nt - 1) * a.last_stride;
    float* dst = a.last_state + (size_t)a.seq_slot[seq] * a.C;
    for (int c = tid; c < a.C; c += THREADS) dst[c] = __bfloat162float(row[c]);
  }
}

// ---- pass 3, time mixing ---------------------------------------------------------------------------------------
// Bound by what surrounds the products: loads, exponentials, splitting and barriers; the tensor cores are busy a quarter of the time. Five
// blocks an SM (six spill: 84 us against 72 in one measurement, 3 sequences of 2,553 tokens, 40 heads; the float32 form 115). A warp makes 16 value columns of all tokens. Of a warp's 16 columns the even ones are one tile of the products and the odd ones
// another: a row's piece of the state is then one 8-byte load for both, and a thread ends with four neighbouring columns.
__global__ void __launch_bounds__(THREADS, 5) mix_finish_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float sm[];
  bf16* qt = reinterpret_cast<bf16*>(sm);  // [3][L][KP] r_t e^{c_{t-1}}
  bf16* kt = qt + 3 * L * KP;              // [3][L][KP] k_s e^{-c_s}; then
  bf16* pt = kt;                           // [3][L][PP] the pair sums
  bf16* vs = kt + 3 * L * KP;              // [L][KP], the columns of 16 ordered as the products want them
  float* red = reinterpret_cast<float*>(vs + L * KP);  // [4][L] sums of squares of a warp's columns
  float* own = red + 4 * L;                // [L] a token's own share, through the bonus
  int* bad = reinterpret_cast<int*>(own + L);  // [2][N]: the first token with an infinity in a value column, with a NaN
  // where a channel forgets too much, as float32, before qt and pt are written
  float* es = sm;                                  // [L][PITCH] decays
  float* rs = reinterpret_cast<float*>(kt);        // [L][PITCH] queries
  float* ps = rs + L * PITCH;                      // [L][L + 4] pair sums
  static_assert(L * PITCH * 4 <= 3 * L * KP * 2 && (L * PITCH + L * (L + 4)) * 4 <= 3 * L * KP * 2 && 3 * L * PP * 2 <= L * PITCH * 4, "room");
  grid_launch_dependents();
  grid_dependency_wait();
  const int h = blockIdx.x, ci = blockIdx.y, seq = blockIdx.z, ch0 = h * N;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int first = (a.chunk0 + ci) * L, qlen = a.seq_qlen[seq], nt = min(L, qlen - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const float* item = a.scratch + (((size_t)seq * a.n_chunks + ci) * a.H + h) * ITEM_MIX;
  const float* cum = item + N * N;
  constexpr int EACH = L * (N / 4) / THREADS;
  const int n = (tid % (N / 4)) * 4, tq = tid / (N / 4);  // this thread's four channels of tokens tq, tq + 8, ...
  bool safe;
  {
    uint2 q[EACH], k[EACH], v[EACH];
    float4 c[EACH], b[EACH];
    const float4 end = __ldcg(reinterpret_cast<const float4*>(cum + (L - 1) * N + n)), by = ld4(a.bonus + ch0 + n);
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
      const int t = tq + i * (THREADS / (N / 4));
      const bool in = t < nt;
      q[i] = in ? *reinterpret_cast<const uint2*>(a.r + (row0 + t) * a.r_stride + ch0 + n) : make_uint2(0u, 0u);
      k[i] = in ? *reinterpret_cast<const uint2*>(a.k + (row0 + t) * a.k_stride + ch0 + n) : make_uint2(0u, 0u);
      v[i] = in ? *reinterpret_cast<const uint2*>(a.v + (row0 + t) * a.v_stride + ch0 + n) : make_uint2(0u, 0u);
      c[i] = __ldcg(reinterpret_cast<const float4*>(cum + t * N + n));
      b[i] = t ? __ldcg(reinterpret_cast<const float4*>(cum + (t - 1) * N + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid < 2 * N) bad[tid] = L;
    safe = !__syncthreads_or(!(end.x > -SAFE) || !(end.y > -SAFE) || !(end.z > -SAFE) || !(end.w > -SAFE));
    auto widen = [](uint2 raw) {
      const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
      return make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
    };
    if (!safe) {  // a token's key, as the tokens after it find it: a thread a token and a quarter of the channels
      const float* decays = cum + L * N;
#pragma unroll
      for (int i = 0; i < EACH; ++i) {
        const int t = tq + i * (THREADS / (N / 4)), at4 = t * PITCH + n;
        st4(rs + at4, widen(q[i]));
        st4(es + at4, __ldcg(reinterpret_cast<const float4*>(decays + t * N + n)));
      }
      const int s = tid >> 2, m0 = (tid & 3) * 4;
      float4 w[N / 16];
#pragma unroll
      for (int j = 0; j < N / 16; ++j)
        w[j] = s < nt ? widen4(a.k + (row0 + s) * a.k_stride + ch0 + m0 + 16 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
      __syncthreads();
      for (int t = 0; t < L; ++t) {
        float d = 0.f;
#pragma unroll
        for (int j = 0; j < N / 16; ++j) d = dot4(ld4(rs + t * PITCH + m0 + 16 * j), w[j], d);
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        if (m0 == 0) ps[t * (L + 4) + s] = s < t ? d : 0.f;
        if (s < t)
#pragma unroll
          for (int j = 0; j < N / 16; ++j) {
            const float4 e = ld4(es + t * PITCH + m0 + 16 * j);
            w[j].x *= e.x; w[j].y *= e.y; w[j].z *= e.z; w[j].w *= e.w;
          }
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
      const int t = tq + i * (THREADS / (N / 4));
      const float4 qf = widen(q[i]), kf = widen(k[i]);
      float bonus = qf.x * by.x * kf.x + qf.y * by.y * kf.y + qf.z * by.z * kf.z + qf.w * by.w * kf.w;
#pragma unroll
      for (int off = 1; off < N / 4; off <<= 1) bonus += __shfl_xor_sync(0xffffffffu, bonus, off);
      if (n == 0) own[t] = bonus;
      split3_store4(qt + t * KP + n, L * KP, make_float4(qf.x * expf(b[i].x), qf.y * expf(b[i].y), qf.z * expf(b[i].z), qf.w * expf(b[i].w)));
      if (safe)
        split3_store4(kt + t * KP + n, L * KP, make_float4(kf.x * expf(-c[i].x), kf.y * expf(-c[i].y), kf.z * expf(-c[i].z), kf.w * expf(-c[i].w)));
      // columns n, n + 2 side by side in the even tile, n + 1, n + 3 in the odd one; what is not finite is set aside, since a product
      // would hand it, times zero, to the tokens before
      uint32_t even = __byte_perm(v[i].x, v[i].y, 0x5410), odd = __byte_perm(v[i].x, v[i].y, 0x7632);
      auto finite = [](uint32_t two) { return (two & 0x7f80u) != 0x7f80u && (two & 0x7f800000u) != 0x7f800000u; };
      if (!finite(even) || !finite(odd)) {
        auto aside = [&](uint32_t& two, int col) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t one = two >> (16 * j) & 0xffffu;
            if ((one & 0x7f80u) != 0x7f80u) continue;
            atomicMin(bad + (one & 0x7fu ? N : 0) + col + 2 * j, t);
            two &= j ? 0x0000ffffu : 0xffff0000u;
          }
        };
        aside(even, n);
        aside(odd, n + 1);
      }
      bf16* to = vs + t * KP + (n & ~15) + ((n & 15) >> 1);
      *reinterpret_cast<uint32_t*>(to) = even;
      *reinterpret_cast<uint32_t*>(to + 8) = odd;
    }
  }
  __syncthreads();
  // the state before the chunk: a value column is one warp's alone, so it comes from memory straight into the products' fragments
  const float* start = item + warp * 16 + 2 * g;
  float2 st[N / 16][4];
#pragma unroll
  for (int kk = 0; kk < N / 16; ++kk)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      st[kk][i] = __ldcg(reinterpret_cast<const float2*>(start + (kk * 16 + 2 * t4 + (i & 1) + 8 * (i >> 1)) * N));
  // pair sums: warp 0 tokens 0..15, warps 1 and 2 tokens 16..31, each against 16 of the tokens before
  const int mt = warp ? 1 : 0, u0 = warp == 2 ? 16 : 0;
  float e[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) e[j][c] = 0.f;
  if (safe && warp < 3) {
#pragma unroll
    for (int leading = 0; leading < 2; ++leading)
#pragma unroll
      for (int kk = 0; kk < N; kk += 16) {
        uint32_t af[3][4], b0[3][2], b1[3][2];
#pragma unroll
        for (int t = 0; t < (leading ? 1 : 3); ++t) {
          ldmatrix_x4(af[t][0], af[t][1], af[t][2], af[t][3], qt + (t * L + mt * 16 + (lane & 15)) * KP + kk + (lane >> 4) * 8);
          ldmatrix_x4(b0[t][0], b0[t][1], b1[t][0], b1[t][1],
                      kt + (t * L + u0 + ((lane >> 4) << 3) + (lane & 7)) * KP + kk + ((lane >> 3) & 1) * 8);
        }
        if (leading) {
          mma_bf16_16816(e[0], af[0][0], af[0][1], af[0][2], af[0][3], b0[0][0], b0[0][1]);
          mma_bf16_16816(e[1], af[0][0], af[0][1], af[0][2], af[0][3], b1[0][0], b1[0][1]);
        } else {
          small33(e[0], af, b0);
          small33(e[1], af, b1);
        }
      }
  }
  if (safe) {
    __syncthreads();  // the keys are no longer read
    if (warp < 3) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int t = mt * 16 + g + 8 * hh, s = u0 + j * 8 + 2 * t4;
          float p[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) p[c] = s + c < t ? e[j][2 * hh + c] : s + c == t ? own[t] : 0.f;
          uint32_t three[3];
          split3_pair(p[0], p[1], three);
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(pt + (i * L + t) * PP + s) = three[i];
        }
    }
  } else {
    for (int i = tid; i < L * (L / 2); i += THREADS) {
      const int t = i / (L / 2), s = (i % (L / 2)) * 2;
      uint32_t three[3];
      split3_pair(s == t ? own[t] : ps[t * (L + 4) + s], s + 1 == t ? own[t] : ps[t * (L + 4) + s + 1], three);
#pragma unroll
      for (int j = 0; j < 3; ++j) *reinterpret_cast<uint32_t*>(pt + (j * L + t) * PP + s) = three[j];
    }
  }
  const int col = warp * 16 + 4 * t4;  // this thread's columns, of tokens g, g + 8, g + 16, g + 24
  uint2 gate[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    gate[i] = g + 8 * i < nt ? *reinterpret_cast<const uint2*>(a.g + (row0 + g + 8 * i) * a.g_stride + ch0 + col) : make_uint2(0u, 0u);
  float o[2][2][4];  // [16 tokens][even, odd columns]
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) o[m][j][c] = 0.f;
  // q . S and the pair sums' products: the small terms of both before the leading ones of both
#pragma unroll
  for (int kk = 0; kk < N / 16; ++kk) {
    uint32_t b[2][2][3];
    split3_pair(st[kk][0].x, st[kk][1].x, b[0][0]);
    split3_pair(st[kk][2].x, st[kk][3].x, b[0][1]);
    split3_pair(st[kk][0].y, st[kk][1].y, b[1][0]);
    split3_pair(st[kk][2].y, st[kk][3].y, b[1][1]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      uint32_t af[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t)
        ldmatrix_x4(af[t][0], af[t][1], af[t][2], af[t][3], qt + (t * L + m * 16 + (lane & 15)) * KP + kk * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int sum = 2; sum >= 1; --sum)
#pragma unroll
        for (int t = 0; t <= sum; ++t)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            mma_bf16_16816(o[m][j], af[t][0], af[t][1], af[t][2], af[t][3], b[j][0][sum - t], b[j][1][sum - t]);
    }
  }
  __syncthreads();  // the pair sums are here
  auto pairs = [&](int t) {  // a term of the pair sums against the values
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      uint32_t b[4];
      ldmatrix_x4_trans(b[0], b[1], b[2], b[3], vs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * KP + warp * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int m = kk; m < 2; ++m) {
        uint32_t af[4];
        ldmatrix_x4(af[0], af[1], af[2], af[3], pt + (t * L + m * 16 + (lane & 15)) * PP + kk * 16 + (lane >> 4) * 8);
        mma_bf16_16816(o[m][0], af[0], af[1], af[2], af[3], b[0], b[1]);
        mma_bf16_16816(o[m][1], af[0], af[1], af[2], af[3], b[2], b[3]);
      }
    }
  };
  pairs(2);
  pairs(1);
#pragma unroll
  for (int kk = 0; kk < N / 16; ++kk)
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      uint32_t af[4];
      ldmatrix_x4(af[0], af[1], af[2], af[3], qt + (m * 16 + (lane & 15)) * KP + kk * 16 + (lane >> 4) * 8);
      mma_bf16_16816(o[m][0], af[0], af[1], af[2], af[3], pack_bf16x2(st[kk][0].x, st[kk][1].x), pack_bf16x2(st[kk][2].x, st[kk][3].x));
      mma_bf16_16816(o[m][1], af[0], af[1], af[2], af[3], pack_bf16x2(st[kk][0].y, st[kk][1].y), pack_bf16x2(st[kk][2].y, st[kk][3].y));
    }
  pairs(0);
  // per head: divide by the root mean square, weight, gate, scale
  const int4 inf = *reinterpret_cast<const int4*>(bad + col), nan = *reinterpret_cast<const int4*>(bad + N + col);
  float4 y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = i >> 1, hh = i & 1, t = g + 8 * i;
    y[i] = make_float4(o[m][0][2 * hh], o[m][1][2 * hh], o[m][0][2 * hh + 1], o[m][1][2 * hh + 1]);
    auto kept = [&](float x, int inf, int nan) { return t >= nan ? NAN : t >= inf ? INFINITY : x; };
    y[i] = make_float4(kept(y[i].x, inf.x, nan.x), kept(y[i].y, inf.y, nan.y), kept(y[i].z, inf.z, nan.z), kept(y[i].w, inf.w, nan.w));
    float sq = y[i].x * y[i].x + y[i].y * y[i].y + y[i].z * y[i].z + y[i].w * y[i].w;
    sq += __shfl_xor_sync(0xffffffffu, sq, 1);
    sq += __shfl_xor_sync(0xffffffffu, sq, 2);
    if (t4 == 0) red[warp * L + t] = sq;
  }
  __syncthreads();
  const float4 w = ld4(a.norm_w + ch0 + col);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = g + 8 * i;
    if (t >= nt) continue;
    const float sum = (red[t] + red[L + t]) + (red[2 * L + t] + red[3 * L + t]);
    const float by = rsqrtf(sum / (float)N + a.eps) * a.out_scale;
    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&gate[i].x), hi = *reinterpret_cast<const __nv_bfloat162*>(&gate[i].y);
    uint2 raw;
    raw.x = pack_bf16x2(y[i].x * by * w.x * silu_near(__low2float(lo)), y[i].y * by * w.y * silu_near(__high2float(lo)));
    raw.y = pack_bf16x2(y[i].z * by * w.z * silu_near(__low2float(hi)), y[i].w * by * w.w * silu_near(__high2float(hi)));
    *reinterpret_cast<uint2*>(a.out + (row0 + t) * a.out_stride + a.out_col + ch0 + col) = raw;
  }
  if (a.last_rows && h == 0 && first + nt == qlen) {  // the sequence's last row, for the next step's token shift
    const bf16* row = a.last_rows + (row0 + nt - 1) * a.last_stride;
    float* dst = a.last_state + (size_t)a.seq_slot[seq] * a.C;
    for (int c = tid; c < a.C; c += THREADS) dst[c] = __bfloat162float(row[c]);
  }
}

template <typename Kernel>
int run(Kernel kernel, dim3 grid, int threads, size_t floats, const ChunkArgs& a, cudaStream_t stream) {
  const size_t smem = floats * sizeof(float);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  return (int)launch_pdl(kernel, grid, dim3(threads), smem, stream, a);
}

}  // namespace

// Tokens per chunk where a step's scan may run in chunks, else 0; *item_floats: scratch of a (sequence, chunk, head).
KRK_API int krk_recurrence_chunk_tokens(int rule, int head, int R, float decay_scale, int* item_floats) {
  *item_floats = rule == 1 ? ITEM_DELTA : ITEM_MIX;
  if (head != N || R < 1 || R > 64) return 0;
  // the delta rule: e^{decay_scale * 32} is what keys and rates are multiplied by at most
  if (rule == 1 && !(decay_scale >= 0.f && decay_scale * L <= 40.f)) return 0;
  return L;
}

// krk_linear_recurrence over chunks chunk0 .. chunk0 + n_chunks - 1 of every sequence, bfloat16 (float32 state), from and to the
// stored state; the caller goes through a step's chunks in order. Rows of four elements on 8-byte boundaries.
KRK_API int krk_recurrence_chunks(int rule, const void* r, int r_stride, const void* k, int k_stride, const void* v, int v_stride,
                                  const void* g, int g_stride, const void* rate, int rate_stride, const void* lora,
                                  int lora_stride, const void* w2, const float* w0, const float* rate_bias, const float* bonus,
                                  const float* norm_w, float* state, const void* last_rows, int last_stride, int C,
                                  float* last_state, void* out, int out_stride, int out_col, float out_scale, float eps,
                                  float decay_scale, int H, int R, int n_seqs, const int* cu_q, const int* seq_qlen,
                                  const int* seq_slot, int chunk0, int n_chunks, float* scratch, int* error, cudaStream_t stream) {
  if (n_seqs == 0 || n_chunks == 0) return 0;
  int item;
  const uintptr_t rows = (uintptr_t)r | (uintptr_t)k | (uintptr_t)v | (uintptr_t)g | (uintptr_t)rate | (uintptr_t)out;
  const uintptr_t floats = (uintptr_t)norm_w | (uintptr_t)state | (uintptr_t)scratch;
  const int strides = r_stride | k_stride | v_stride | g_stride | rate_stride | out_stride | out_col;
  if ((rule != 0 && rule != 1) || (rule == 1 && (!rate || !rate_bias)) || (rule == 0 && !bonus) || !scratch ||
      !krk_recurrence_chunk_tokens(rule, N, R, decay_scale, &item) || (rows & 7) || (strides & 3) || (floats & 15) ||
      n_chunks > 65535 || n_seqs > 65535 || H > 65535)
    return -2;
  ChunkArgs a;
  a.r = (const bf16*)r; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = (const bf16*)g; a.rate = (const bf16*)rate;
  a.lora = (const bf16*)lora; a.r_stride = r_stride; a.k_stride = k_stride; a.v_stride = v_stride; a.g_stride = g_stride;
  a.rate_stride = rate_stride; a.lora_stride = lora_stride; a.w2 = (const bf16*)w2; a.w0 = w0; a.rate_bias = rate_bias;
  a.bonus = bonus; a.norm_w = norm_w; a.state = state; a.last_rows = (const bf16*)last_rows; a.last_stride = last_stride;
  a.C = C; a.last_state = last_state; a.out = (bf16*)out; a.out_stride = out_stride; a.out_col = out_col; a.out_scale = out_scale;
  a.eps = eps; a.decay_scale = decay_scale; a.H = H; a.R = R; a.cu_q = cu_q; a.seq_qlen = seq_qlen; a.seq_slot = seq_slot;
  a.chunk0 = chunk0; a.n_chunks = n_chunks; a.scratch = scratch; a.error = error;
  const dim3 items((unsigned)H, (unsigned)n_chunks, (unsigned)n_seqs);
  int rc;
  const size_t RP = (size_t)((R + 7) & ~7);
  if (rule == 1) {
    // six times three terms of a chunk's rows and the values; two matrices of float32; the small things
    const size_t chunk = 19 * (size_t)L * KP / 2 + 2 * (size_t)L * PITCH + N + 2 * L + 8 * N + 4 * N;
    if ((rc = run(delta_chunk_kernel, items, DELTA_THREADS, chunk, a, stream))) return rc;
    // the scratch as rows of N floats: an item's M, then its G
    CUtensorMap map_m, map_g;
    const long long scratch_rows = (long long)n_seqs * n_chunks * H * (ITEM_DELTA / N);
    if (scratch_rows > 0x7fffffffLL) return -2;
    if ((rc = tc::make_map_f32(&map_m, scratch, scratch_rows, N, N, 32, N, true))) return rc;
    if ((rc = tc::make_map_f32(&map_g, scratch, scratch_rows, N, N, WALK_COLS, N, false))) return rc;
    const size_t walk = (WALK_STAGES * (size_t)(WALK_M + WALK_G) + 2 * (N / 8) * WALK_SP) * sizeof(float) + 1024;
    if ((rc = (int)cudaFuncSetAttribute(delta_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk))) return rc;
    if ((rc = (int)launch_pdl(delta_walk_kernel, dim3(N / WALK_COLS, (unsigned)H, (unsigned)n_seqs), dim3(WALK_THREADS), walk, stream, map_m, map_g, a)))
      return rc;
    return run(delta_finish_kernel, items, THREADS, (size_t)L * PITCH + 4 * L, a, stream);
  }
  const size_t rows_bytes = (size_t)L * KP * sizeof(bf16);  // a term of a chunk's rows
  if ((rc = run(mix_chunk_kernel, items, THREADS, 5 * rows_bytes / sizeof(float) + L * RP + 2 * N, a, stream))) return rc;
  if ((rc = run(mix_walk_kernel, dim3(N * N / 4 / 64, (unsigned)H, (unsigned)n_seqs), 64, 0, a, stream))) return rc;
  return run(mix_finish_kernel, items, THREADS, 7 * rows_bytes / sizeof(float) + 5 * L + 2 * N, a, stream);
}
