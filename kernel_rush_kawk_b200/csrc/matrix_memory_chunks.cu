// The recurrences of matrix_memory.cu over a step's many tokens in chunks of 64, on the tensor cores (mma.sync m16n8k16,
// bfloat16 in, float32 accumulate). Within a chunk, with the state S before it,
//
//   y_t = r_t (q_t . S) + sum_{s <= t} A_ts v_s ,   S' = R S + sum_s (w_s k_s) v_s^T
//
// Per-channel decays (c_t: the log decays summed from the chunk's first token to t): A_ts = (q_t e^{c_t}) . (k_s e^{-c_s}),
// q_t . S is (q_t e^{c_t}) . S, w_s = e^{c_last - c_s}, R = e^{c_last} per key channel. Gated by a running maximum (F_t: the
// log forget gates summed likewise, i_s the log input gates, m the maximum): A_ts = (q_t . k_s) e^{F_t - F_s + i_s - m_t},
// r_t = e^{F_t + m_before - m_t}, w_s = e^{F_last - F_s + i_s - m_last}, R = e^{F_last + m_before - m_last}; the vector n
// beside S is one more value column whose v is 1, and its y is what the gated kind divides by.
//
// q, k and v are bfloat16 already, so a product of two of them is exact. Every operand that is not (decayed queries and
// keys, A, the state) is handed to the tensor cores as three bfloat16 terms that add up to it (24 bits of mantissa); where
// both sides are such sums, the six products that matter in 32-bit are formed. So the arithmetic is that of float32 with the
// sums grouped by chunks.
//
// e^{-c_s} overflows where a chunk forgets everything: where a channel's decay over the chunk passes e^-40 the chunk's A is
// formed pair by pair from e^{c_t - c_s} on the CUDA cores instead (right for any decay, and slow).
//
// A state-space mixer (ssd.cu) is a third kind: q and k are its C and B, one row of each for a group of heads, v its x, the decay
// one number per head and token, and x_s counts dt_s times: A_ts = (C_t . B_s) e^{F_t - F_s} dt_s, r_t = e^{F_t}, w_s = e^{F_last - F_s} dt_s,
// plus skip * x_t in the output. Its log decays are as large as the step sizes make them, so they are summed, kept and subtracted in
// 64-bit: e^{F_t - F_s} is then as exact as the product of the decays that the scan token by token forms. One prompt of 2,048
// tokens, 48 heads of 64 with 128 rows: the scan's three passes on the CUDA cores 403 us, these 97 (25, 30 and 57, each from a
// cold cache; 111 with a block a head).
//
// Three passes: (1) every chunk's own sum_s (w_s k_s) v_s^T; (2) the walk over a sequence's chunks, which leaves every
// chunk its starting state and the sequence its final one; (3) the outputs. A block takes some slices of 64 value
// columns of one (sequence, chunk, head).
#include "mma.cuh"

namespace {

enum Kind { DECAYS, RUNNING_MAX };

constexpr int L = 64;        // tokens per chunk
constexpr int PB = 64;       // value columns per block
constexpr int VPITCH = PB + 8;
constexpr int APITCH = L + 8;
constexpr int THREADS = 256, OUT_THREADS = 512;
constexpr float SAFE = 40.f;

__device__ __forceinline__ float log_sigmoid_f(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

// state-space kind: the log decays summed from the chunk's first token to this one, its step size, e^{F_last - F_s} dt
struct __align__(16) Step {
  double sum;
  float dt, weight;
};

struct ChunkArgs {
  const bf16 *q, *k, *v;
  int q_stride, k_stride, v_stride;
  float q_scale;
  const float* cum;     // [rows, H * N]: log decays summed within the chunk (per-channel kind); or null
  const float4* gates;  // [rows, H]: (f, i, m before, m after) (gated kind); or null
  float *state, *nm;    // [slots, H, N, P], [slots, H, N + 1]
  float* y;             // [rows, H, P]
  float* den;           // [rows, H]: n . q (gated kind)
  float* cs;            // [n_seqs, max_chunks, H, N * P + (gated ? N : 0)]: chunk sums, then chunk starts
  float* cd;            // [n_seqs, max_chunks, H, N]: a chunk's decays
  int H, N, P, max_chunks;
  int slices;  // column slices a block walks
  const Step* steps;    // state-space kind: [H, rows]
  int rows;
  const float* skip;    // state-space kind: [H]
  int per_group;        // heads that share a row of q and k
  int units, parts;     // state-space kind: (head, column slice) pairs a block takes of those of a group; blocks for a group
  int chunk0;           // the chunks of every sequence that this launch takes start here
  const int *cu_q, *seq_qlen, *seq_slot;
};

// eight consecutive floats as three terms of eight bfloat16 each, 16 bytes a term
__device__ __forceinline__ void split3_store8(const float (&f)[8], bf16* dst, size_t apart) {
  uint32_t t[4][3];
#pragma unroll
  for (int j = 0; j < 4; ++j) split3_pair(f[2 * j], f[2 * j + 1], t[j]);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(dst + i * apart) = make_uint4(t[0][i], t[1][i], t[2][i], t[3][i]);
}
__device__ __forceinline__ void widen8(const bf16* p, float (&f)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int j = 0; j < 4; ++j) { f[2 * j] = __low2float(h[j]); f[2 * j + 1] = __high2float(h[j]); }
}

// F[t] = sum of f over the chunk's tokens 0..t (64 of them, zero beyond the last), by one warp
__device__ __forceinline__ void chunk_sums(float* F, const float* f, int lane) {
  const float a = f[2 * lane], b = a + f[2 * lane + 1];
  float run = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float p = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += p;
  }
  const float before = run - b;  // exact enough: log gates of one chunk
  F[2 * lane] = before + a;
  F[2 * lane + 1] = before + b;
}

__device__ __forceinline__ void load_values(bf16* vs, const ChunkArgs& a, size_t row0, int h, int p0, int nt) {
  for (int i = threadIdx.x; i < L * (PB / 8); i += blockDim.x) {
    const int s = i / (PB / 8), c = (i % (PB / 8)) * 8;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (s < nt && p0 + c < a.P) v = *reinterpret_cast<const uint4*>(a.v + (row0 + s) * a.v_stride + (size_t)h * a.P + p0 + c);
    *reinterpret_cast<uint4*>(vs + s * VPITCH + c) = v;
  }
}

// ---- pass 1: the chunk's own sum of (w k) v^T, and its decays ------------------------------------------------
template <Kind KIND>
__global__ void __launch_bounds__(THREADS) chunk_sum_kernel(ChunkArgs a) {
  constexpr bool GATED = KIND == RUNNING_MAX;
  extern __shared__ __align__(16) bf16 sm[];
  __shared__ float fs[L], is_[L], Fs[L], ws[L];
  const int N = a.N, P = a.P, H = a.H, NP = N + 8;
  bf16* kt = sm;                       // [3][L][NP]
  bf16* vs = kt + 3 * (size_t)L * NP;  // [L][VPITCH]
  const int h = blockIdx.y % H, chunk = blockIdx.y / H, seq = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  grid_launch_dependents();
  grid_dependency_wait();
  const int first = (a.chunk0 + chunk) * L, nt = min(L, a.seq_qlen[seq] - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const size_t k_col = (size_t)(h / a.per_group) * N;
  float m_before = 0.f, m_last = 0.f;
  if (GATED) {
    if (threadIdx.x < L) {
      const float4 g = threadIdx.x < nt ? a.gates[(row0 + threadIdx.x) * H + h] : make_float4(0.f, -INFINITY, 0.f, 0.f);
      fs[threadIdx.x] = g.x;
      is_[threadIdx.x] = g.y;
    }
    m_before = a.gates[row0 * H + h].z;
    m_last = a.gates[(row0 + nt - 1) * H + h].w;
    __syncthreads();
    if (warp == 0) {
      chunk_sums(Fs, fs, lane);
      __syncwarp();
      for (int s = lane; s < L; s += 32) ws[s] = s < nt ? expf(Fs[L - 1] - Fs[s] + is_[s] - m_last) : 0.f;
    }
    __syncthreads();
  }
  const float* cum_last = GATED ? nullptr : a.cum + (row0 + nt - 1) * H * N + (size_t)h * N;
  for (int i = threadIdx.x; i < L * (N / 8); i += THREADS) {
    const int s = i / (N / 8), n = (i % (N / 8)) * 8;
    float f[8];
    if (s < nt) {
      widen8(a.k + (row0 + s) * a.k_stride + k_col + n, f);
      if (GATED) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= ws[s];
      } else {
        const float* c = a.cum + (row0 + s) * H * N + (size_t)h * N + n;
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= expf(cum_last[n + j] - c[j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = 0.f;
    }
    split3_store8(f, kt + s * NP + n, (size_t)L * NP);
  }
  __syncthreads();
  const size_t at = ((size_t)seq * a.max_chunks + chunk) * H + h;
  float* cs = a.cs + at * ((size_t)N * P + (GATED ? N : 0));
  if (blockIdx.x == 0) {
    for (int n = threadIdx.x; n < N; n += THREADS) {
      a.cd[at * N + n] = GATED ? expf(Fs[L - 1] + m_before - m_last) : expf(cum_last[n]);
      if (GATED) {
        float d = 0.f;
        for (int s = 0; s < nt; ++s) {
          const bf16* t = kt + s * NP + n;
          d += (__bfloat162float(t[2 * (size_t)L * NP]) + __bfloat162float(t[(size_t)L * NP])) + __bfloat162float(t[0]);
        }
        cs[(size_t)N * P + n] = d;
      }
    }
  }
  for (int slice = blockIdx.x * a.slices; slice < (int)(blockIdx.x + 1) * a.slices && slice * PB < P; ++slice) {
  const int p0 = slice * PB;
  __syncthreads();  // the values of the slice before are no longer read
  load_values(vs, a, row0, h, p0, nt);
  __syncthreads();
  for (int m0 = warp * 16; m0 < N; m0 += 16 * (THREADS / 32)) {
    float acc[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[n][c] = 0.f;
#pragma unroll
    for (int ks = 0; ks < L / 16; ++ks) {
      uint32_t af[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t)  // the transpose of k's rows
        ldmatrix_x4_trans(af[t][0], af[t][1], af[t][2], af[t][3],
                          kt + t * (size_t)L * NP + (ks * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * NP + m0 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        uint32_t b0, b1, b2, b3;
        ldmatrix_x4_trans(b0, b1, b2, b3, vs + (ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * VPITCH + (n + (lane >> 4)) * 8);
#pragma unroll
        for (int t = 2; t >= 0; --t) {  // small terms first
          mma_bf16_16816(acc[n], af[t][0], af[t][1], af[t][2], af[t][3], b0, b1);
          mma_bf16_16816(acc[n + 1], af[t][0], af[t][1], af[t][2], af[t][3], b2, b3);
        }
      }
    }
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int p = p0 + n * 8 + 2 * t4;
      if (p < P) {
        *reinterpret_cast<float2*>(cs + (size_t)(m0 + g) * P + p) = make_float2(acc[n][0], acc[n][1]);
        *reinterpret_cast<float2*>(cs + (size_t)(m0 + g + 8) * P + p) = make_float2(acc[n][2], acc[n][3]);
      }
    }
  }
  }
}

// ---- pass 2: a sequence's chunks in order, four neighbouring elements of the state a thread ------------------
template <bool GATED>
__global__ void chunk_walk_kernel(ChunkArgs a) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int h = blockIdx.y, seq = blockIdx.z;
  const int qlen = a.seq_qlen[seq];
  if (qlen <= 0) return;
  const int n_chunks = min(a.max_chunks, (qlen + L - 1) / L - a.chunk0);
  if (n_chunks <= 0) return;
  const size_t NP = (size_t)a.N * a.P, all = NP + (GATED ? a.N : 0);
  const size_t e = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
  if (e >= all) return;
  const bool matrix = e < NP;
  const int n = (int)(matrix ? e / a.P : e - NP);  // the gated kind's decay is one number for all n
  const size_t head = (size_t)a.seq_slot[seq] * a.H + h;
  float* st = matrix ? a.state + head * NP + e : a.nm + head * (a.N + 1) + n;
  float4 run = matrix ? *reinterpret_cast<const float4*>(st) : make_float4(st[0], st[1], st[2], st[3]);
  float4* cs = reinterpret_cast<float4*>(a.cs + ((size_t)seq * a.max_chunks * a.H + h) * all + e);
  const float* cd = a.cd + ((size_t)seq * a.max_chunks * a.H + h) * a.N + n;
  const size_t step = (size_t)a.H * all / 4, dstep = (size_t)a.H * a.N;
  for (int c0 = 0; c0 < n_chunks; c0 += 8) {
    float4 own[8];
    float decay[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < n_chunks) {
        own[i] = __ldcg(cs + (size_t)(c0 + i) * step);
        decay[i] = __ldcg(cd + (size_t)(c0 + i) * dstep);
      }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < n_chunks) {
        cs[(size_t)(c0 + i) * step] = run;
        run.x = fmaf(decay[i], run.x, own[i].x);
        run.y = fmaf(decay[i], run.y, own[i].y);
        run.z = fmaf(decay[i], run.z, own[i].z);
        run.w = fmaf(decay[i], run.w, own[i].w);
      }
  }
  if (matrix) {
    *reinterpret_cast<float4*>(st) = run;
  } else {
    st[0] = run.x; st[1] = run.y; st[2] = run.z; st[3] = run.w;
  }
}

// ---- pass 3: the outputs -------------------------------------------------------------------------------------
// A is formed once per block, each warp one quarter of the tokens against one quarter of the earlier ones, and left in shared
// memory; then the block walks its column slices. A block's 109 to 144 KB of shared memory leave an SM two or one: sixteen warps
// cover one another's reads and barriers, where eight took 73 us (per-channel
// decays) and 42 (gated) of 1,500 tokens of 8 heads of 128 x 256 and sixteen take 61 and 36.
template <Kind KIND>
__global__ void __launch_bounds__(OUT_THREADS, KIND == RUNNING_MAX ? 2 : 1) chunk_output_kernel(ChunkArgs a) {
  constexpr bool GATED = KIND == RUNNING_MAX;
  extern __shared__ __align__(16) bf16 sm[];
  __shared__ float fs[L], is_[L], Fs[L], ms[L], den[4][L];
  const int N = a.N, P = a.P, H = a.H, NP = N + 8;
  constexpr int TERMS = GATED ? 1 : 3;  // of a query's and a key's row in shared memory
  const size_t q_apart = (size_t)L * NP, s_apart = (size_t)N * VPITCH;
  bf16* qs = sm;                       // [TERMS][L][NP]
  bf16* as = qs + TERMS * q_apart;     // [3][L][APITCH]: A
  bf16* vs = as + 3 * L * APITCH;      // [L][VPITCH]
  bf16* ks = vs + L * VPITCH;          // [TERMS][L][NP]; the state takes its place
  bf16* ss = ks;                       // [3][N][VPITCH]
  const int h = blockIdx.y % H, chunk = blockIdx.y / H, seq = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mt = warp & 3, part = warp >> 2;  // 16 tokens; 16 earlier tokens, later 16 of a slice's columns
  const int g = lane >> 2, t4 = lane & 3;
  grid_launch_dependents();
  grid_dependency_wait();
  const int first = (a.chunk0 + chunk) * L, nt = min(L, a.seq_qlen[seq] - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const float* start = a.cs + (((size_t)seq * a.max_chunks + chunk) * H + h) * ((size_t)N * P + (GATED ? N : 0));
  float m_before = 0.f;
  bool safe = true;

  if (GATED) {
    if (threadIdx.x < L) {
      const float4 gt = threadIdx.x < nt ? a.gates[(row0 + threadIdx.x) * H + h] : make_float4(0.f, -INFINITY, 0.f, 0.f);
      fs[threadIdx.x] = gt.x;
      is_[threadIdx.x] = gt.y;
      ms[threadIdx.x] = gt.w;
    }
    m_before = a.gates[row0 * H + h].z;
    for (int i = threadIdx.x; i < 2 * L * (N / 8); i += OUT_THREADS) {
      const int s = (i / (N / 8)) % L, n = (i % (N / 8)) * 8;
      const bool is_k = i >= L * (N / 8);
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (s < nt) v = *reinterpret_cast<const uint4*>((is_k ? a.k + (row0 + s) * a.k_stride : a.q + (row0 + s) * a.q_stride) + (size_t)h * N + n);
      *reinterpret_cast<uint4*>((is_k ? ks : qs) + s * NP + n) = v;
    }
    __syncthreads();
    if (warp == 0) chunk_sums(Fs, fs, lane);
  } else {
    const float* cl = a.cum + (row0 + nt - 1) * H * N + (size_t)h * N;
    int over = 0;
    for (int n = threadIdx.x; n < N; n += OUT_THREADS) over |= !(cl[n] > -SAFE);
    safe = !__syncthreads_or(over);
    for (int i = threadIdx.x; i < L * (N / 8); i += OUT_THREADS) {
      const int s = i / (N / 8), n = (i % (N / 8)) * 8;
      float f[8], k8[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = k8[j] = 0.f;
      if (s < nt) {
        const float4* c4 = reinterpret_cast<const float4*>(a.cum + (row0 + s) * H * N + (size_t)h * N + n);
        const float4 c0 = c4[0], c1 = c4[1];
        const float e[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        widen8(a.q + (row0 + s) * a.q_stride + (size_t)h * N + n, f);
        if (safe) widen8(a.k + (row0 + s) * a.k_stride + (size_t)h * N + n, k8);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= expf(e[j]);
        if (safe) {
#pragma unroll
          for (int j = 0; j < 8; ++j) k8[j] *= expf(-e[j]);
        }
      }
      split3_store8(f, qs + s * NP + n, q_apart);
      if (safe) split3_store8(k8, ks + s * NP + n, q_apart);
    }
  }
  __syncthreads();

  // A: the warp's 16 tokens against 16 of the chunk's (a tile of later tokens stays zero and is not read)
  float s[2][4];
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int c = 0; c < 4; ++c) s[n][c] = 0.f;
  const int u0 = part * 16;
  if (safe) {
    for (int kk = 0; kk < N / 16; ++kk) {
      if (u0 >= mt * 16 + 16) break;
      uint32_t af[TERMS][4];
#pragma unroll
      for (int t = 0; t < TERMS; ++t)
        ldmatrix_x4(af[t][0], af[t][1], af[t][2], af[t][3], qs + t * q_apart + (mt * 16 + (lane & 15)) * NP + kk * 16 + (lane >> 4) * 8);
      uint32_t b[TERMS][4];
#pragma unroll
      for (int t = 0; t < TERMS; ++t)
        ldmatrix_x4(b[t][0], b[t][1], b[t][2], b[t][3],
                    ks + t * q_apart + (u0 + ((lane >> 4) << 3) + (lane & 7)) * NP + kk * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int sum = TERMS == 1 ? 0 : 2; sum >= 0; --sum)  // small terms first
#pragma unroll
        for (int t = 0; t <= sum; ++t) {
          mma_bf16_16816(s[0], af[t][0], af[t][1], af[t][2], af[t][3], b[sum - t][0], b[sum - t][1]);
          mma_bf16_16816(s[1], af[t][0], af[t][1], af[t][2], af[t][3], b[sum - t][2], b[sum - t][3]);
        }
    }
  } else {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int t = mt * 16 + g + 8 * (c >> 1), u = u0 + n * 8 + 2 * t4 + (c & 1);
        if (u > t || t >= nt) continue;
        const bf16* qr = a.q + (row0 + t) * a.q_stride + (size_t)h * N;
        const bf16* kr = a.k + (row0 + u) * a.k_stride + (size_t)h * N;
        const float* ct = a.cum + (row0 + t) * H * N + (size_t)h * N;
        const float* cu = a.cum + (row0 + u) * H * N + (size_t)h * N;
        float d = 0.f;
        for (int j = 0; j < N; ++j) d += __bfloat162float(qr[j]) * __bfloat162float(kr[j]) * expf(ct[j] - cu[j]);
        s[n][c] = d;
      }
  }
  float rows[2] = {a.q_scale, a.q_scale};  // what q . S is multiplied by
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const int t = mt * 16 + g + 8 * hh;
    float sum = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      float v[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int u = u0 + n * 8 + 2 * t4 + c;
        v[c] = 0.f;
        if (u <= t && t < nt) {
          v[c] = s[n][2 * hh + c] * a.q_scale;
          if (GATED) v[c] *= expf(Fs[t] - Fs[u] + is_[u] - ms[t]);
        }
        sum += v[c];
      }
      uint32_t p[3];
      split3_pair(v[0], v[1], p);
#pragma unroll
      for (int i = 0; i < 3; ++i)
        *reinterpret_cast<uint32_t*>(as + (i * L + t) * APITCH + u0 + n * 8 + 2 * t4) = p[i];
    }
    if (GATED) {
      rows[hh] *= t < nt ? expf(Fs[t] + m_before - ms[t]) : 0.f;
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if (t4 == 0) den[part][t] = sum;
    }
  }
  __syncthreads();  // A is complete, and the keys are no longer read
  if (GATED && blockIdx.x == 0) {
    const float* n0 = start + (size_t)N * P;
    for (int t = warp; t < nt; t += OUT_THREADS / 32) {
      float d = 0.f;
      for (int n = lane; n < N; n += 32) d += __bfloat162float(qs[t * NP + n]) * n0[n];
      d = warp_sum(d);
      if (lane == 0)
        a.den[(row0 + t) * H + h] = ((den[0][t] + den[1][t]) + (den[2][t] + den[3][t])) + a.q_scale * expf(Fs[t] + m_before - ms[t]) * d;
    }
  }

  for (int slice = blockIdx.x * a.slices; slice < (int)(blockIdx.x + 1) * a.slices && slice * PB < P; ++slice) {
    const int p0 = slice * PB;
    load_values(vs, a, row0, h, p0, nt);
    for (int i = threadIdx.x; i < N * (PB / 8); i += OUT_THREADS) {
      const int n = i / (PB / 8), c = (i % (PB / 8)) * 8;
      float f[8];
      if (p0 + c < P) {
        const float4 x = __ldcg(reinterpret_cast<const float4*>(start + (size_t)n * P + p0 + c));
        const float4 y = __ldcg(reinterpret_cast<const float4*>(start + (size_t)n * P + p0 + c + 4));
        f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w; f[4] = y.x; f[5] = y.y; f[6] = y.z; f[7] = y.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = 0.f;
      }
      split3_store8(f, ss + n * VPITCH + c, s_apart);
    }
    __syncthreads();
    float acc[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[n][c] = 0.f;
    for (int kk = 0; kk < N / 16; ++kk) {
      uint32_t af[TERMS][4];
#pragma unroll
      for (int t = 0; t < TERMS; ++t)
        ldmatrix_x4(af[t][0], af[t][1], af[t][2], af[t][3], qs + t * q_apart + (mt * 16 + (lane & 15)) * NP + kk * 16 + (lane >> 4) * 8);
      uint32_t b[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t)
        ldmatrix_x4_trans(b[t][0], b[t][1], b[t][2], b[t][3],
                          ss + t * s_apart + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * VPITCH + (part * 2 + (lane >> 4)) * 8);
#pragma unroll
      for (int sum = 2; sum >= 0; --sum)
#pragma unroll
        for (int t = 0; t < TERMS; ++t) {
          if (sum - t < 0) continue;
          mma_bf16_16816(acc[0], af[t][0], af[t][1], af[t][2], af[t][3], b[sum - t][0], b[sum - t][1]);
          mma_bf16_16816(acc[1], af[t][0], af[t][1], af[t][2], af[t][3], b[sum - t][2], b[sum - t][3]);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[n][c] *= rows[c >> 1];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk > mt) break;  // later tokens
      uint32_t af[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t)
        ldmatrix_x4(af[t][0], af[t][1], af[t][2], af[t][3], as + (t * L + mt * 16 + (lane & 15)) * APITCH + kk * 16 + (lane >> 4) * 8);
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4_trans(b0, b1, b2, b3, vs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * VPITCH + (part * 2 + (lane >> 4)) * 8);
#pragma unroll
      for (int t = 2; t >= 0; --t) {
        mma_bf16_16816(acc[0], af[t][0], af[t][1], af[t][2], af[t][3], b0, b1);
        mma_bf16_16816(acc[1], af[t][0], af[t][1], af[t][2], af[t][3], b2, b3);
      }
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int t = mt * 16 + g + 8 * hh;
      if (t >= nt) continue;
      float* yr = a.y + ((row0 + t) * H + h) * P;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int p = p0 + part * 16 + n * 8 + 2 * t4;
        if (p < P) *reinterpret_cast<float2*>(yr + p) = make_float2(acc[n][2 * hh], acc[n][2 * hh + 1]);
      }
    }
    __syncthreads();  // the state and the values make room for the next slice's
  }
}

// ---- state-space kind ----------------------------------------------------------------------------------------
// A group's heads share the rows of q and k, so a block takes several (head, column slice) units of a group's chunk: what depends on
// q and k alone is done once, and a unit's values, step sizes and state are on their way while the unit before is multiplied (MANY). Two
// blocks an SM: three leave the outputs 80 registers, which spill (69 us against 58, profiled; a block a head 66). Where the units
// are more than two blocks an SM hold and not more than three, a block takes one of them, with no next unit's registers: 450 tokens
// of 48 heads 39.6 us with two units a block, 35.2 here.

// What a unit needs of the chunk's tokens: the raw values of a thread's two pieces of eight, the steps of token threadIdx.x
struct UnitRows {
  uint4 v[2];
  Step step;
  __device__ __forceinline__ void fetch(const ChunkArgs& a, size_t row0, int h, int p0, int nt) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int s = (threadIdx.x >> 3) + 32 * i, c = (threadIdx.x & 7) * 8;
      v[i] = s < nt && p0 + c < a.P ? *reinterpret_cast<const uint4*>(a.v + (row0 + s) * a.v_stride + (size_t)h * a.P + p0 + c)
                                    : make_uint4(0u, 0u, 0u, 0u);
    }
    if (threadIdx.x < nt) step = a.steps[(size_t)h * a.rows + row0 + threadIdx.x];
    else step = {0.0, 0.f, 0.f};
  }
};
static_assert(L * PB / 8 == 2 * THREADS && PB == 64, "two pieces a thread");

// The chunk's own sum_s k_s (w_s v_s)^T: where a token's weight is one number it multiplies the values instead of the keys: they are
// fewer, and the keys stay exact. Warps 4 x 2: 32 key rows and 32 columns each, so that a fragment of the values' terms, which
// bound the kernel (every warp reads them from shared memory), serves two products; the keys' fragments stay in registers.
template <bool MANY>
__global__ void __launch_bounds__(THREADS, MANY ? 2 : 3) ssd_sum_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) bf16 sm[];
  __shared__ float ws[2][L];
  const int N = a.N, P = a.P, H = a.H, NP = N + 8;
  bf16* ks = sm;                       // [L][NP]
  bf16* vs = ks + (size_t)L * NP;      // [3][L][VPITCH]
  const int part = blockIdx.x % a.parts, group = blockIdx.x / a.parts, chunk = blockIdx.y, seq = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  grid_launch_dependents();
  grid_dependency_wait();
  const int first = (a.chunk0 + chunk) * L, nt = min(L, a.seq_qlen[seq] - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const int slices = (P + PB - 1) / PB, u1 = MANY ? min(a.per_group * slices, (part + 1) * a.units) : part + 1;
  int u = MANY ? part * a.units : part;
  UnitRows next;
  next.fetch(a, row0, group * a.per_group + u / slices, u % slices * PB, nt);
  for (int s = warp; s < L; s += THREADS / 32)
    for (int n = lane * 8; n < N; n += 256) {
      bf16* dst = ks + s * NP + n;
      if (s < nt) cp_async_16(dst, a.k + (row0 + s) * a.k_stride + (size_t)group * N + n);
      else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
    }
  cp_async_commit();
  cp_async_wait<0>();
  const int c0 = (warp >> 2) * 32;
  for (; u < u1; ++u) {
    const int h = group * a.per_group + u / slices, p0 = u % slices * PB, b = u & 1;
    const UnitRows now = next;
    if (threadIdx.x < L) ws[b][threadIdx.x] = now.step.weight;
    __syncthreads();  // the weights are here, and the values of the unit before are no longer read
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int s = (threadIdx.x >> 3) + 32 * i, c = (threadIdx.x & 7) * 8;
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&now.v[i]);
      const float w = ws[b][s];
      float f[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) { f[2 * j] = w * __low2float(h2[j]); f[2 * j + 1] = w * __high2float(h2[j]); }
      split3_store8(f, vs + s * VPITCH + c, (size_t)L * VPITCH);
    }
    if (MANY && u + 1 < u1) next.fetch(a, row0, group * a.per_group + (u + 1) / slices, (u + 1) % slices * PB, nt);
    __syncthreads();
    const size_t at = ((size_t)seq * a.max_chunks + chunk) * H + h;
    float* cs = a.cs + at * ((size_t)N * P);
    if (p0 == 0) {
      const float decay = expf((float)a.steps[(size_t)h * a.rows + row0 + nt - 1].sum);
      for (int n = threadIdx.x; n < N; n += THREADS) a.cd[at * N + n] = decay;
    }
    for (int m0 = (warp & 3) * 32; m0 < N; m0 += 128) {
      float acc[2][4][4];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[m][n][c] = 0.f;
#pragma unroll
      for (int kk = 0; kk < L / 16; ++kk) {
        uint32_t af[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)  // the transpose of k's rows (the last 16 columns again where N ends there)
          ldmatrix_x4_trans(af[m][0], af[m][1], af[m][2], af[m][3],
                            ks + (kk * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * NP + min(m0 + 16 * m, N - 16) + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
          uint32_t bf[3][4];
#pragma unroll
          for (int t = 0; t < 3; ++t)
            ldmatrix_x4_trans(bf[t][0], bf[t][1], bf[t][2], bf[t][3],
                              vs + ((size_t)t * L + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * VPITCH + c0 + (n + (lane >> 4)) * 8);
#pragma unroll
          for (int t = 2; t >= 0; --t)  // small terms first
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              mma_bf16_16816(acc[m][n], af[m][0], af[m][1], af[m][2], af[m][3], bf[t][0], bf[t][1]);
              mma_bf16_16816(acc[m][n + 1], af[m][0], af[m][1], af[m][2], af[m][3], bf[t][2], bf[t][3]);
            }
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        if (m0 + 16 * m >= N) break;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const int p = p0 + c0 + n * 8 + 2 * t4;
          if (p < P) {
            float* dst = cs + (size_t)(m0 + 16 * m + g) * P + p;
            *reinterpret_cast<float2*>(dst) = make_float2(acc[m][n][0], acc[m][n][1]);
            *reinterpret_cast<float2*>(dst + 8 * (size_t)P) = make_float2(acc[m][n][2], acc[m][n][3]);
          }
        }
      }
    }
  }
}

// The outputs. A warp takes all 64 tokens of eight value columns, whose part of the state is then its own fragment of the product:
// it never passes through shared memory. C_t . B_s of the chunk, the same for a group's heads, waits in shared memory, each thread's
// own share side by side (or in registers, for one unit).
template <bool MANY>
__global__ void __launch_bounds__(THREADS, MANY ? 2 : 3) ssd_output_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) bf16 sm[];
  __shared__ double fs[L];     // the summed decays
  __shared__ float dts[L];
  __shared__ int bad[2][PB];   // the first token that holds something infinite in a value column
  const int N = a.N, P = a.P, H = a.H, NP = N + 8;
  bf16* qs = sm;                       // [L][NP]
  bf16* vs = qs + (size_t)L * NP;      // [L][VPITCH]
  float* dots = reinterpret_cast<float*>(vs + L * VPITCH);  // [16][THREADS] C_t . B_s
  bf16* ks = reinterpret_cast<bf16*>(dots + 16 * THREADS);  // [L][NP]; then
  bf16* as = ks;                       // [3][L][APITCH]: A
  const int part = blockIdx.x % a.parts, group = blockIdx.x / a.parts, chunk = blockIdx.y, seq = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  grid_launch_dependents();
  grid_dependency_wait();
  const int first = (a.chunk0 + chunk) * L, nt = min(L, a.seq_qlen[seq] - first);
  if (nt <= 0) return;
  const size_t row0 = (size_t)a.cu_q[seq] + first;
  const int slices = (P + PB - 1) / PB, u1 = MANY ? min(a.per_group * slices, (part + 1) * a.units) : part + 1;
  int u = MANY ? part * a.units : part;
  const float* starts = a.cs + ((size_t)seq * a.max_chunks + chunk) * H * N * P;
  constexpr int KB = 8;  // 128 rows of the state at a time
  float own[KB][4];
  auto fetch = [&](int u, int n0) {  // rows n0 .. n0 + 127 of a column of the unit's state, as the product's fragments have them
    const int p = u % slices * PB + warp * 8 + g;
    const float* from = starts + ((size_t)(group * a.per_group + u / slices) * N + n0 + 2 * t4) * P + p;
#pragma unroll
    for (int kk = 0; kk < KB; ++kk) {
      const bool in = p < P && n0 + kk * 16 < N;  // N is a multiple of 16
#pragma unroll
      for (int i = 0; i < 4; ++i) own[kk][i] = in ? __ldcg(from + (size_t)(kk * 16 + (i & 1) + 8 * (i >> 1)) * P) : 0.f;
    }
  };
  UnitRows next;
  next.fetch(a, row0, group * a.per_group + u / slices, u % slices * PB, nt);
  for (int s = warp; s < 2 * L; s += THREADS / 32) {
    const bool is_k = s >= L;
    const int r = s & (L - 1);
    for (int n = lane * 8; n < N; n += 256) {
      bf16* dst = (is_k ? ks : qs) + r * NP + n;
      if (r < nt) cp_async_16(dst, (is_k ? a.k + (row0 + r) * a.k_stride : a.q + (row0 + r) * a.q_stride) + (size_t)group * N + n);
      else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  cp_async_commit();
  fetch(u, 0);
  if (threadIdx.x < 2 * PB) bad[threadIdx.x >> 6][threadIdx.x & 63] = L;
  cp_async_wait<0>();
  __syncthreads();
  // A: the warp's 16 tokens against 32 of the chunk's; two warps have later tokens alone, whose tiles are not read
  const int mt = warp & 3, t0 = (warp >> 2) * 32;
  float own_dots[4][4];
  if (t0 < mt * 16 + 16) {
    auto& s = own_dots;
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) s[n][c] = 0.f;
    for (int kk = 0; kk < N; kk += 16) {
      uint32_t af[4];
      ldmatrix_x4(af[0], af[1], af[2], af[3], qs + (mt * 16 + (lane & 15)) * NP + kk + (lane >> 4) * 8);
#pragma unroll
      for (int n = 0; n < 4; n += 2) {
        uint32_t b[4];
        ldmatrix_x4(b[0], b[1], b[2], b[3], ks + (t0 + n * 8 + ((lane >> 4) << 3) + (lane & 7)) * NP + kk + ((lane >> 3) & 1) * 8);
        mma_bf16_16816(s[n], af[0], af[1], af[2], af[3], b[0], b[1]);
        mma_bf16_16816(s[n + 1], af[0], af[1], af[2], af[3], b[2], b[3]);
      }
    }
    if (MANY)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) dots[(n * 4 + c) * THREADS + threadIdx.x] = s[n][c];
  }
  for (int h_before = -1; u < u1; ++u) {
    const int h = group * a.per_group + u / slices;
    int* worst = bad[u & 1];
    // the values, what is not finite set aside (a zero in its place): a matrix product would hand it, times zero, to the tokens before
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int s = (threadIdx.x >> 3) + 32 * i, c = (threadIdx.x & 7) * 8;
      uint32_t* two = reinterpret_cast<uint32_t*>(&next.v[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool lo = (two[j] & 0x7f80u) == 0x7f80u, hi = (two[j] & 0x7f800000u) == 0x7f800000u;
        if (lo) atomicMin(worst + c + 2 * j, s);
        if (hi) atomicMin(worst + c + 2 * j + 1, s);
        if (lo || hi) two[j] &= (lo ? 0xffff0000u : 0xffffffffu) & (hi ? 0xffffu : 0xffffffffu);
      }
      *reinterpret_cast<uint4*>(vs + s * VPITCH + c) = next.v[i];
    }
    if (threadIdx.x < L) {
      fs[threadIdx.x] = next.step.sum;
      dts[threadIdx.x] = next.step.dt;
    }
    __syncthreads();  // values and steps are here, and the keys (later A) are no longer read
    if (h != h_before && t0 < mt * 16 + 16) {
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int t = mt * 16 + g + 8 * hh;
        const double ft = fs[t];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          float v[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int s = t0 + n * 8 + 2 * t4 + c;
            const float dot = MANY ? dots[(n * 4 + 2 * hh + c) * THREADS + threadIdx.x] : own_dots[n][2 * hh + c];
            v[c] = s <= t && t < nt ? dot * (expf((float)(ft - fs[s])) * dts[s]) : 0.f;
          }
          uint32_t p[3];
          split3_pair(v[0], v[1], p);
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(as + (i * L + t) * APITCH + t0 + n * 8 + 2 * t4) = p[i];
        }
      }
    }
    h_before = h;
    const int p0 = u % slices * PB + warp * 8;
    float acc[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[m][c] = 0.f;
    for (int n0 = 0; n0 < N; n0 += 16 * KB) {
      if (n0) fetch(u, n0);
#pragma unroll
      for (int kk = 0; kk < KB; ++kk) {
        if (n0 + kk * 16 >= N) break;
        uint32_t lo[3], hi[3];
        split3_pair(own[kk][0], own[kk][1], lo);
        split3_pair(own[kk][2], own[kk][3], hi);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          uint32_t af[4];
          ldmatrix_x4(af[0], af[1], af[2], af[3], qs + (m * 16 + (lane & 15)) * NP + n0 + kk * 16 + (lane >> 4) * 8);
#pragma unroll
          for (int t = 2; t >= 0; --t) mma_bf16_16816(acc[m], af[0], af[1], af[2], af[3], lo[t], hi[t]);  // small terms first
        }
      }
    }
    if (MANY && u + 1 < u1) {
      next.fetch(a, row0, group * a.per_group + (u + 1) / slices, (u + 1) % slices * PB, nt);
      fetch(u + 1, 0);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const float e = expf((float)fs[m * 16 + g + 8 * hh]);
        acc[m][2 * hh] *= e;
        acc[m][2 * hh + 1] *= e;
      }
    __syncthreads();  // A is here
#pragma unroll
    for (int kk = 0; kk < 4; kk += 2) {
      uint32_t b[4];  // of 16 tokens, and of the 16 after them
      ldmatrix_x4_trans(b[0], b[1], b[2], b[3], vs + (kk * 16 + lane) * VPITCH + warp * 8);
#pragma unroll
      for (int m = kk; m < 4; ++m)
#pragma unroll
        for (int two = 0; two < 2; ++two) {
          if (kk + two > m) continue;  // later tokens
#pragma unroll
          for (int t = 2; t >= 0; --t) {
            uint32_t af[4];
            ldmatrix_x4(af[0], af[1], af[2], af[3], as + (t * L + m * 16 + (lane & 15)) * APITCH + (kk + two) * 16 + (lane >> 4) * 8);
            mma_bf16_16816(acc[m], af[0], af[1], af[2], af[3], b[2 * two], b[2 * two + 1]);
          }
        }
    }
    const int c0 = warp * 8 + 2 * t4;
    const float skip = a.skip[h];
    if (p0 < P) {  // the whole warp: P is a multiple of 16
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int t = m * 16 + g + 8 * hh;
          if (t >= nt) continue;
          const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(vs + t * VPITCH + c0);
          const float y0 = fmaf(skip, __low2float(x), acc[m][2 * hh]), y1 = fmaf(skip, __high2float(x), acc[m][2 * hh + 1]);
          *reinterpret_cast<float2*>(a.y + ((row0 + t) * H + h) * P + p0 + 2 * t4) =
              make_float2(t >= worst[c0] ? NAN : y0, t >= worst[c0 + 1] ? NAN : y1);
        }
    }
    __syncthreads();  // the values, A and the steps make room for the next unit's
    if (threadIdx.x < PB) worst[threadIdx.x] = L;
  }
}

// ---- log decays summed within chunks -------------------------------------------------------------------------
// cum[row, c]: sum over the chunk's tokens up to the row's of logsigmoid(z) / tau, z = W2 lora + bias. A warp has 32 channels of
// sixteen tokens, a block the chunk: bound by the chain of a token's logarithm, so the tokens are spread (a thread with all 64 of a
// channel: 19 us for 1,500 rows of 1,024 channels, 12 here).
constexpr int DECAY_TOKENS = 16;
__global__ void __launch_bounds__(32 * L / DECAY_TOKENS)
chunk_decays_kernel(float* __restrict__ cum, const bf16* __restrict__ lora, int lora_stride, const bf16* __restrict__ w2,
                    const float* __restrict__ bias, float inv_tau, int channels, int R, const int* __restrict__ cu_q,
                    const int* __restrict__ seq_qlen) {
  extern __shared__ __align__(16) float ls[];  // [R][L]
  __shared__ float total[L / DECAY_TOKENS][32];
  grid_launch_dependents();
  grid_dependency_wait();
  const int chunk = blockIdx.y, seq = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nt = min(L, seq_qlen[seq] - chunk * L);
  if (nt <= 0) return;
  const size_t row0 = (size_t)cu_q[seq] + chunk * L;
  for (int i = threadIdx.x; i < L * R; i += blockDim.x)
    ls[(i % R) * L + i / R] = i / R < nt ? __bfloat162float(lora[(row0 + i / R) * lora_stride + i % R]) : 0.f;
  const int c = blockIdx.x * 32 + lane, t0 = warp * DECAY_TOKENS;
  const bool mine = c < channels;
  __syncthreads();
  float z[DECAY_TOKENS];
  const float b = mine ? bias[c] : 0.f;
#pragma unroll
  for (int t = 0; t < DECAY_TOKENS; ++t) z[t] = b;
  const bool wide = R % 8 == 0 && ((uintptr_t)w2 & 15) == 0;
  for (int m0 = 0; m0 < R; m0 += 8) {
    float w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = 0.f;
    if (mine && wide) {
      widen8(w2 + (size_t)c * R + m0, w);
    } else if (mine) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (m0 + j < R) w[j] = __bfloat162float(w2[(size_t)c * R + m0 + j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (m0 + j >= R) break;
#pragma unroll
      for (int t = 0; t < DECAY_TOKENS; t += 4) {
        const float4 x = *reinterpret_cast<const float4*>(ls + (m0 + j) * L + t0 + t);
        z[t] += w[j] * x.x; z[t + 1] += w[j] * x.y; z[t + 2] += w[j] * x.z; z[t + 3] += w[j] * x.w;
      }
    }
  }
  float run = 0.f;
#pragma unroll
  for (int t = 0; t < DECAY_TOKENS; ++t) {
    if (t0 + t < nt) run += log_sigmoid_f(z[t]) * inv_tau;
    z[t] = run;
  }
  total[warp][lane] = run;
  __syncthreads();
  float before = 0.f;
  for (int w = 0; w < warp; ++w) before += total[w][lane];
#pragma unroll
  for (int t = 0; t < DECAY_TOKENS; ++t)
    if (mine && t0 + t < nt) cum[(row0 + t0 + t) * channels + c] = before + z[t];
}

// state-space kind: dt = softplus(raw + bias), log decay -exp(A_log) dt. Not below FORGOTTEN, whose e^ is zero in 32 bits: sums of
// minus infinity have no difference, and even 64 bits would lose a later token's decay beside a number that is large enough. The
// decays are summed over a chunk's tokens in 64 bits. A warp a chunk and head, a lane two neighbouring tokens.
constexpr float FORGOTTEN = -120.f;
__global__ void __launch_bounds__(256) steps_kernel(Step* __restrict__ steps, const bf16* __restrict__ dt, int dt_stride,
                                                    const float* __restrict__ bias, const float* __restrict__ a_log, int rows, int H,
                                                    const int* __restrict__ cu_q, const int* __restrict__ seq_qlen) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, h = blockIdx.y * 8 + (threadIdx.x >> 5), seq = blockIdx.z;
  const int first = blockIdx.x * L, nt = min(L, seq_qlen[seq] - first);
  if (nt <= 0 || h >= H) return;
  const size_t row0 = (size_t)cu_q[seq] + first;
  const float b = bias[h], rate = expf(a_log[h]);
  float d[2], f[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int t = 2 * lane + j;
    d[j] = f[j] = 0.f;
    if (t < nt) {
      const float z = __bfloat162float(dt[(row0 + t) * dt_stride + h]) + b;
      d[j] = z > 20.f ? z : log1pf(expf(z));
      f[j] = -rate * d[j];
      if (f[j] < FORGOTTEN) f[j] = FORGOTTEN;  // a NaN stays one
    }
  }
  const double two = (double)f[0] + f[1];
  double run = two;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double p = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += p;
  }
  const double sums[2] = {(run - two) + f[0], run}, last = __shfl_sync(0xffffffffu, run, 31);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int t = 2 * lane + j;
    if (t >= nt) continue;
    steps[(size_t)h * rows + row0 + t] = {sums[j], d[j], expf((float)(last - sums[j])) * d[j]};
  }
}

size_t sum_smem(int N) { return (3 * (size_t)L * (N + 8) + (size_t)L * VPITCH) * sizeof(bf16); }
size_t ssd_sum_smem(int N) { return ((size_t)L * (N + 8) + 3 * (size_t)L * VPITCH) * sizeof(bf16); }
size_t output_smem(int N, bool gated) {
  const size_t terms = gated ? 1 : 3, rows = terms * L * (N + 8), state = 3 * (size_t)N * VPITCH;
  return (rows + 3 * (size_t)L * APITCH + (size_t)L * VPITCH + (state > rows ? state : rows)) * sizeof(bf16);
}

size_t ssd_output_smem(int N) {
  const size_t keys = (size_t)L * (N + 8), sums = 3 * (size_t)L * APITCH;
  return ((size_t)L * (N + 8) + (size_t)L * VPITCH + (keys > sums ? keys : sums)) * sizeof(bf16) + 16 * THREADS * sizeof(float);
}

int launch_walk(const ChunkArgs& a, bool gated, int n_seqs, cudaStream_t stream) {
  const size_t all = (size_t)a.N * a.P + (gated ? a.N : 0);
  return (int)launch_pdl(gated ? chunk_walk_kernel<true> : chunk_walk_kernel<false>, dim3((unsigned)((all / 4 + 63) / 64), (unsigned)a.H, (unsigned)n_seqs),
                         dim3(64), 0, stream, a);
}

template <typename Kernel>
int room(Kernel kernel, size_t bytes) {
  return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <Kind KIND>
int launch_chunks(ChunkArgs a, int n_seqs, cudaStream_t stream) {
  constexpr bool GATED = KIND == RUNNING_MAX;
  const size_t s1 = sum_smem(a.N), s3 = output_smem(a.N, GATED);
  const long long heads = (long long)a.H * a.max_chunks;
  if (heads > 65535 || n_seqs > 65535) return -2;
  // what a block does before its first slice is done once per block: as many slices a block as leave every SM three
  const int all_slices = (a.P + PB - 1) / PB;
  const long long most = heads * n_seqs * all_slices;
  a.slices = (int)(most / 444 < 1 ? 1 : most / 444 > all_slices ? all_slices : most / 444);
  const dim3 grid((unsigned)((all_slices + a.slices - 1) / a.slices), (unsigned)heads, (unsigned)n_seqs);
  int rc;
  if ((rc = room(chunk_sum_kernel<KIND>, s1)) || (rc = room(chunk_output_kernel<KIND>, s3))) return rc;
  if ((rc = (int)launch_pdl(chunk_sum_kernel<KIND>, grid, dim3(THREADS), s1, stream, a))) return rc;
  if ((rc = launch_walk(a, GATED, n_seqs, stream))) return rc;
  return (int)launch_pdl(chunk_output_kernel<KIND>, grid, dim3(OUT_THREADS), s3, stream, a);
}

int launch_ssd(ChunkArgs a, int n_seqs, int live, cudaStream_t stream) {
  const size_t s1 = ssd_sum_smem(a.N), s3 = ssd_output_smem(a.N);
  if (a.max_chunks > 65535 || n_seqs > 65535) return -2;
  int rc;
  if ((rc = room(ssd_sum_kernel<true>, s1)) || (rc = room(ssd_sum_kernel<false>, s1)) || (rc = room(ssd_output_kernel<true>, s3)) ||
      (rc = room(ssd_output_kernel<false>, s3)))
    return rc;
  const int groups = a.H / a.per_group, all = a.per_group * ((a.P + PB - 1) / PB);
  // units a block: the fewest rounds of units over the SMs, a block's start counted as a part of one. Blocks of chunks that a shorter
  // sequence does not have leave at once and are not counted (48 heads, sequences of 600, 400 and 300 tokens: 93 us counted, 71).
  // Three blocks an SM of one unit each take 1.4 times as long as two (48 heads, 330 tokens: 33.5 us and 28).
  // The starts, 0.5 for the sums and 0.7 for the outputs, choose the fastest or within 1 % of it of 1, 2, 3, 4 and 6 units for one prompt of
  // 192 to 3,000 tokens of 48 heads in four groups (2,048 tokens, the outputs by 1, 2, 3, 4, 6, 8 and 12: 112, 103, 100, 103, 97, 113 and 142 us).
  // Returns whether it is the form of many.
  auto split = [&](float start) {
    float best = 1e30f;
    bool many = true;
    for (int units = 0; units <= all; ++units) {  // 0: three blocks an SM, one unit each
      const int each = units ? units : 1;
      const long long blocks = (long long)((all + each - 1) / each) * groups * live, at_once = units ? 296 : 444;
      const float cost = (float)((blocks + at_once - 1) / at_once) * (each + start) * (units ? 1.f : 1.4f);
      if (cost < best) {
        best = cost;
        a.units = each;
        many = units > 0;
      }
    }
    a.parts = (all + a.units - 1) / a.units;
    return many;
  };
  auto grid = [&] { return dim3((unsigned)(a.parts * groups), (unsigned)a.max_chunks, (unsigned)n_seqs); };
  const bool many_sums = split(0.5f);
  rc = (int)launch_pdl(many_sums ? ssd_sum_kernel<true> : ssd_sum_kernel<false>, grid(), dim3(THREADS), s1, stream, a);
  if (rc) return rc;
  if ((rc = launch_walk(a, false, n_seqs, stream))) return rc;
  const bool many = split(0.7f);
  return (int)launch_pdl(many ? ssd_output_kernel<true> : ssd_output_kernel<false>, grid(), dim3(THREADS), s3, stream, a);
}

}  // namespace

// Tokens per chunk, and whether head sizes are ones that the chunked passes take.
KRK_API int krk_memory_chunk_tokens(int N, int P, int gated) {
  return N % 16 == 0 && P % 16 == 0 && N >= 16 && sum_smem(N) <= 220 * 1024 && output_smem(N, gated != 0) <= 220 * 1024 ? L : 0;
}

KRK_API int krk_memory_chunk_decays(float* cum, const void* lora, int lora_stride, const void* w2, const float* bias, float tau,
                                    int channels, int R, int n_seqs, int max_q_len, const int* cu_q, const int* seq_qlen,
                                    cudaStream_t stream) {
  if (n_seqs == 0 || max_q_len == 0) return 0;
  const size_t smem = (size_t)L * R * sizeof(float);
  const int chunks = (max_q_len + L - 1) / L;
  if (smem > 48 * 1024 || chunks > 65535 || n_seqs > 65535) return -2;
  if (const int rc = room(chunk_decays_kernel, 48 * 1024)) return rc;  // beside the kernel's own
  const dim3 grid((unsigned)((channels + 31) / 32), (unsigned)chunks, (unsigned)n_seqs);
  return (int)launch_pdl(chunk_decays_kernel, grid, dim3(32 * L / DECAY_TOKENS), smem, stream, cum, (const bf16*)lora, lora_stride, (const bf16*)w2,
                         bias, 1.0f / tau, channels, R, cu_q, seq_qlen);
}

// The scan of krk_memory_scan in chunks, bfloat16. cum (per-channel kind) or gates and nm (gated kind); scratch cs and cd
// for ceil(max_q_len / 64) chunks a sequence. Row starts of q, k and v on 16-byte boundaries.
KRK_API int krk_memory_chunks(float* y, float* den, const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride,
                              float q_scale, const float* cum, const float* gates, float* state, float* nm, float* cs, float* cd,
                              int H, int N, int P, int n_seqs, int max_q_len, const int* cu_q, const int* seq_qlen,
                              const int* seq_slot, cudaStream_t stream) {
  if (n_seqs == 0 || max_q_len == 0) return 0;
  if ((cum == nullptr) == (gates == nullptr) || (gates && (!nm || !den)) || !krk_memory_chunk_tokens(N, P, gates != nullptr) ||
      q_stride % 8 || k_stride % 8 || v_stride % 8 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state | (uintptr_t)cs | (uintptr_t)cum) & 15))
    return -2;
  ChunkArgs a;
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.q_stride = q_stride; a.k_stride = k_stride;
  a.v_stride = v_stride; a.q_scale = q_scale; a.cum = cum; a.gates = (const float4*)gates; a.state = state; a.nm = nm; a.y = y; a.den = den;
  a.cs = cs; a.cd = cd; a.H = H; a.N = N; a.P = P; a.max_chunks = (max_q_len + L - 1) / L; a.slices = 1;
  a.cu_q = cu_q; a.seq_qlen = seq_qlen; a.seq_slot = seq_slot;
  a.steps = nullptr; a.rows = 0; a.skip = nullptr; a.per_group = 1; a.units = a.parts = 1; a.chunk0 = 0;
  return gates ? launch_chunks<RUNNING_MAX>(a, n_seqs, stream) : launch_chunks<DECAYS>(a, n_seqs, stream);
}

// Step sizes and summed log decays [H, rows] of a state-space mixer's rows (bfloat16), a Step of 16 bytes each, for krk_ssd_chunks.
KRK_API int krk_ssd_steps(float* steps, const void* dt, int dt_stride, const float* dt_bias, const float* a_log, int rows, int H,
                          int n_seqs, int max_q_len, const int* cu_q, const int* seq_qlen, cudaStream_t stream) {
  if (rows == 0 || n_seqs == 0 || max_q_len == 0) return 0;
  const int chunks = (max_q_len + L - 1) / L;
  if (H > 8 * 65535 || n_seqs > 65535 || ((uintptr_t)steps & 15)) return -2;
  return (int)launch_pdl(steps_kernel, dim3((unsigned)chunks, (unsigned)((H + 7) / 8), (unsigned)n_seqs), dim3(256), 0, stream, (Step*)steps,
                         (const bf16*)dt, dt_stride, dt_bias, a_log, rows, H, cu_q, seq_qlen);
}

// The scan of a state-space mixer (krk_ssd_scan) over chunks chunk0 .. chunk0 + n_chunks - 1 of every sequence, from and to the
// stored state [slots, H, N, P]; the caller goes through a step's chunks in order. x, B and C bfloat16 with rows on 16-byte
// boundaries; scratch cs and cd for n_chunks chunks a sequence. live: chunks in all that hold tokens.
KRK_API int krk_ssd_chunks(float* y, const void* x, int x_stride, const void* B, int b_stride, const void* C, int c_stride,
                           const float* steps, int rows, const float* skip, float* state, float* cs, float* cd, int H, int P,
                           int N, int G, int n_seqs, int chunk0, int n_chunks, int live, const int* cu_q, const int* seq_qlen,
                           const int* seq_slot, cudaStream_t stream) {
  if (n_seqs == 0 || n_chunks == 0 || live == 0) return 0;
  if (G < 1 || H % G || !krk_memory_chunk_tokens(N, P, 1) || x_stride % 8 || b_stride % 8 || c_stride % 8 ||
      (((uintptr_t)x | (uintptr_t)B | (uintptr_t)C | (uintptr_t)state | (uintptr_t)cs) & 15) || ((uintptr_t)steps & 15))
    return -2;
  ChunkArgs a;
  a.q = (const bf16*)C; a.k = (const bf16*)B; a.v = (const bf16*)x; a.q_stride = c_stride; a.k_stride = b_stride;
  a.v_stride = x_stride; a.q_scale = 1.f; a.cum = nullptr; a.gates = nullptr; a.state = state; a.nm = nullptr; a.y = y; a.den = nullptr;
  a.cs = cs; a.cd = cd; a.H = H; a.N = N; a.P = P; a.max_chunks = n_chunks; a.slices = 1;
  a.cu_q = cu_q; a.seq_qlen = seq_qlen; a.seq_slot = seq_slot;
  a.steps = (const Step*)steps; a.rows = rows; a.skip = skip; a.per_group = H / G; a.chunk0 = chunk0;
  return launch_ssd(a, n_seqs, live, stream);
}
