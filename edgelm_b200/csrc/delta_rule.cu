// The gated delta rule: a recurrent mixer whose state per head is a matrix S [d x e] (float32) that is decayed,
// corrected towards the token's value along the token's key, and read with the token's query:
//
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (the read-out sees the token's own write)
//
// with g in (0, 1) a decay and beta in (0, 1) a step size per token and head.  Two kernels: `delta_prepare` (queries and
// keys to unit vectors, the queries times d^(-1/2); beta = sigmoid(.), g = exp(-exp(A_log) softplus(. + dt_bias))) and
// `delta_scan` (the recurrence over the step's tokens of every sequence, from and to the sequence's state row).
// Everything here is float32 in both precisions.
//
// Tokens of all sequences are packed along the first axis; `seq_tok0[s] .. seq_tok0[s + 1] - 1` are the packed rows of
// the batch's sequence s, `seq_slot[s]` the row of its state.
#include "chunk_mm.cuh"

namespace edgelm {

__device__ __forceinline__ float dr_softplus(float z) { return log1pf(expf(-fabsf(z))) + fmaxf(z, 0.f); }

// qkv [tokens][G d | G d | H e] (after the convolution): every query and key head x <- x / sqrt(sum(x^2) + unit_eps),
// queries also times q_scale.  bg [tokens][2 H]: beta, then the decay, from the raw projections u[t][b_off + h], u[t][a_off + h].
__global__ void __launch_bounds__(128)
delta_prepare_kernel(float* __restrict__ qkv, int C, const float* __restrict__ u, int ldu, int b_off, int a_off,
                     const float* __restrict__ A_log, const float* __restrict__ dt_bias, float* __restrict__ bg, int H, int G, int d,
                     float unit_eps, float q_scale) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
  float* row = qkv + (size_t)t * C;
  for (int v = blockIdx.y * NW + warp; v < 2 * G; v += gridDim.y * NW) {          // the vectors: G query heads, then G key heads
    float* x = row + (size_t)v * d;
    float ss = 0.f;
    for (int i = lane; i < d; i += 32) ss = fmaf(x[i], x[i], ss);
    ss = warp_sum(ss);
    const float inv = (1.0f / sqrtf(ss + unit_eps)) * (v < G ? q_scale : 1.0f);
    for (int i = lane; i < d; i += 32) x[i] *= inv;
  }
  const float* ur = u + (size_t)t * ldu;
  for (int h = blockIdx.y * blockDim.x + threadIdx.x; h < H; h += gridDim.y * blockDim.x) {
    bg[(size_t)t * 2 * H + h] = 1.0f / (1.0f + expf(-ur[b_off + h]));
    bg[(size_t)t * 2 * H + H + h] = expf(-expf(A_log[h]) * dr_softplus(ur[a_off + h] + dt_bias[h]));
  }
}

// A block = 16 CPT columns of one head's state for one sequence.  Eight lanes share CPT neighbouring columns, each lane with
// RPT of their rows in registers (row = sublane * RPT + r; rows beyond d are zeros); S^T k and S^T q are sums over a lane's
// rows and three shuffles.  With CPT > 1 the token's key and query rows are read once for the CPT columns and the columns'
// chains of dependent operations run side by side: fewer instructions a column, for steps with enough (sequence, head) pairs
// to fill the device; for one sequence the chain from one token's state to the next is what takes the time, and one column a
// thread is fastest (measured at the launch).  The step's queries, keys, values, betas and decays come through shared
// memory, DS_TC tokens a stage, the next stage on its way (cp.async) while this one is computed.  State layout:
// [slot][H][e][d] (a column's rows side by side).
constexpr int DS_SUB = 8, DS_GROUPS = 16, DS_THREADS = DS_SUB * DS_GROUPS, DS_TC = 8;

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int RPT, int CPT>
__global__ void __launch_bounds__(DS_THREADS)
delta_scan_kernel(const float* __restrict__ qkv, int C, const float* __restrict__ bg, float* __restrict__ state, float* __restrict__ o,
                  const int32_t* __restrict__ seq_tok0, const int32_t* __restrict__ seq_slot, int H, int G, int d, int e) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int DP = DS_SUB * RPT;                       // padded rows
  constexpr int COLS = DS_GROUPS * CPT;                  // columns a block
  constexpr int NV = RPT / 4;
  constexpr int STAGE = DS_TC * (2 * DP + COLS + 2);     // floats a stage: q, k [DS_TC][DP]; v [DS_TC][COLS]; beta, g [DS_TC]
  __shared__ __align__(16) float sm[2 * STAGE];
  const int s = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * COLS;
  const int g = h / (H / G);
  const int sub = threadIdx.x & (DS_SUB - 1), grp = threadIdx.x >> 3, mycol = col0 + grp * CPT;
  const int t0 = seq_tok0[s], n = seq_tok0[s + 1] - t0;
  float* st = state + ((size_t)seq_slot[s] * H + h) * e * d;
  float S[CPT][RPT];
#pragma unroll
  for (int c = 0; c < CPT; ++c)
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int i = sub * RPT + r;
      S[c][r] = (mycol + c < e && i < d) ? st[(size_t)(mycol + c) * d + i] : 0.f;
    }
  for (int i = threadIdx.x; i < 2 * STAGE; i += DS_THREADS) sm[i] = 0.f;   // (rows beyond d and columns beyond e stay zero)
  __syncthreads();
  const int q_off = g * d, k_off = G * d + g * d, v_off = 2 * G * d + h * e + col0;
  auto load = [&](int chunk) {
    float* b = sm + (chunk & 1) * STAGE;
    const int c0 = chunk * DS_TC, nt = min(DS_TC, n - c0);
    for (int i = threadIdx.x; i < nt * d; i += DS_THREADS) {
      const int tt = i / d, j = i - tt * d;
      const float* src = qkv + (size_t)(t0 + c0 + tt) * C;
      cp_async4(b + tt * DP + j, src + q_off + j);
      cp_async4(b + DS_TC * DP + tt * DP + j, src + k_off + j);
    }
    const int ncol = min(COLS, e - col0);
    for (int i = threadIdx.x; i < nt * ncol; i += DS_THREADS) {
      const int tt = i / ncol, j = i - tt * ncol;
      cp_async4(b + 2 * DS_TC * DP + tt * COLS + j, qkv + (size_t)(t0 + c0 + tt) * C + v_off + j);
    }
    if (threadIdx.x < 2 * nt) {
      const int tt = threadIdx.x >> 1, which = threadIdx.x & 1;
      cp_async4(b + 2 * DS_TC * DP + DS_TC * COLS + which * DS_TC + tt, bg + (size_t)(t0 + c0 + tt) * 2 * H + which * H + h);
    }
    cp_async_commit();
  };
  const int n_chunks = (n + DS_TC - 1) / DS_TC;
  if (n_chunks > 0) load(0);
  for (int c = 0; c < n_chunks; ++c) {
    if (c + 1 < n_chunks) { load(c + 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    __syncthreads();
    const float* b = sm + (c & 1) * STAGE;
    const int nt = min(DS_TC, n - c * DS_TC);
    for (int tt = 0; tt < nt; ++tt) {
      const float* qs = b + tt * DP + sub * RPT;
      const float* kk = b + DS_TC * DP + tt * DP + sub * RPT;
      const float beta = b[2 * DS_TC * DP + DS_TC * COLS + tt], dec = b[2 * DS_TC * DP + DS_TC * COLS + DS_TC + tt];
      float4 k4[NV], q4[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) { k4[i] = *reinterpret_cast<const float4*>(kk + 4 * i); q4[i] = *reinterpret_cast<const float4*>(qs + 4 * i); }
      float v[CPT], ks[CPT], ov[CPT];
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) v[cc] = b[2 * DS_TC * DP + tt * COLS + grp * CPT + cc];
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) {
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int r = 4 * i;
          S[cc][r] *= dec; S[cc][r + 1] *= dec; S[cc][r + 2] *= dec; S[cc][r + 3] *= dec;
          a0 = fmaf(S[cc][r], k4[i].x, a0); a1 = fmaf(S[cc][r + 1], k4[i].y, a1);
          a0 = fmaf(S[cc][r + 2], k4[i].z, a0); a1 = fmaf(S[cc][r + 3], k4[i].w, a1);
        }
        ks[cc] = a0 + a1;
      }
#pragma unroll
      for (int off = 1; off < DS_SUB; off <<= 1)
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) ks[cc] += __shfl_xor_sync(0xffffffffu, ks[cc], off);
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) {
        const float uu = beta * (v[cc] - ks[cc]);
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int r = 4 * i;
          S[cc][r] = fmaf(k4[i].x, uu, S[cc][r]); S[cc][r + 1] = fmaf(k4[i].y, uu, S[cc][r + 1]);
          S[cc][r + 2] = fmaf(k4[i].z, uu, S[cc][r + 2]); S[cc][r + 3] = fmaf(k4[i].w, uu, S[cc][r + 3]);
          a0 = fmaf(S[cc][r], q4[i].x, a0); a1 = fmaf(S[cc][r + 1], q4[i].y, a1);
          a0 = fmaf(S[cc][r + 2], q4[i].z, a0); a1 = fmaf(S[cc][r + 3], q4[i].w, a1);
        }
        ov[cc] = a0 + a1;
      }
#pragma unroll
      for (int off = 1; off < DS_SUB; off <<= 1)
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) ov[cc] += __shfl_xor_sync(0xffffffffu, ov[cc], off);
      if (sub == 0) {
        float* orow = o + (size_t)(t0 + c * DS_TC + tt) * H * e + (size_t)h * e;
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc)
          if (mycol + cc < e) orow[mycol + cc] = ov[cc];
      }
    }
    __syncthreads();     // the stage is free for the load after the next
  }
#pragma unroll
  for (int c = 0; c < CPT; ++c)
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int i = sub * RPT + r;
      if (mycol + c < e && i < d) st[(size_t)(mycol + c) * d + i] = S[c][r];
    }
}

// ------------------------------------------------------------------ the recurrence chunk by chunk
// For prompt steps: with L_t the sum of the logarithms of the decays of a chunk's tokens up to t, S0 the state before the chunk and
// u_t the correction that token t writes,
//
//     u_t = beta_t (v_t - exp(L_t) S0^T k_t - sum_(s < t) exp(L_t - L_s) (k_t . k_s) u_s)
//     o_t = exp(L_t) S0^T q_t + sum_(s <= t) exp(L_t - L_s) (q_t . k_s) u_s
//     S   = exp(L_n) S0 + sum_s exp(L_n - L_s) k_s u_s^T
//
// so the corrections solve (I + A) U = beta V - (beta exp(L) K) S0 with A strictly lower triangular, and what goes from chunk to chunk is
// two small matrix products instead of a chain through every token:
//   1. `delta_chunk_solve`, every (chunk, head) at once: A, then U0 = (I + A)^-1 beta V and W = (I + A)^-1 (beta exp(L) K) by
//      substitution, a thread a column with its 64 values in registers;
//   2. `delta_chunk_states`, the chunks of a (sequence, head) in order, blocks of 16 value channels: U = U0 - W S0, then S;
//   3. `delta_chunk_out`, every (chunk, head) at once: the outputs from U and the kept S0.
// Logarithms, their sums and exponentials and the substitution are double (a decay that is zero in float32 counts as exp(-200)), scores join
// runs of eight float32 products in double, everything else is float32.  (All but the logarithms in float32: outputs 1.7 to 2.2 times as far
// from float64 as the walk's.)
// One (chunk, head) of the scratch: U0, later U, [e][64]; W [64][d]; the keys times exp(L_n - L_s) [d][64]; S0 [e][d].  Then exp(L_n) of each.
// Nine heads of 64, prompts of 333 to 1,700 tokens (4,065 in all): the walk 548 us, this 232 (77 + 106 + 49; all but the logarithms in
// float32 195).  The first waits for its loads, results and unrolled code (double pipe 17 % active), the second is the longest sequence's chain.
constexpr int DC_BLOCK = 16;       // value channels a block of `delta_chunk_states` owns
constexpr int DC_STATE_THREADS = 128;
constexpr int DC_SOLVE_PITCH = CHUNK + 2;

__host__ __device__ inline size_t dc_floats(int d, int e) { return (size_t)(2 * CHUNK) * d + (size_t)CHUNK * e + (size_t)d * e; }

// lg[t] = L_t of the chunk's tokens (from ntok on: the last one's), by the first warp; the block synchronises afterwards
__device__ __forceinline__ void dc_logs(double* lg, const float* __restrict__ bg, int tok0, int ntok, int H, int h) {
  if (threadIdx.x >= 32) return;
  double x[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = 2 * threadIdx.x + i;
    const double z = t < ntok ? log((double)bg[(size_t)(tok0 + t) * 2 * H + H + h]) : 0.0;
    x[i] = z < -200.0 ? -200.0 : z;        // (a NaN stays one)
  }
  chunk_log_sums(lg, x[0], x[1]);
}

// NT 128 threads where the columns fit (two blocks an SM: a thread's 64 doubles are half of its registers), else 256
template <int NT>
__global__ void __launch_bounds__(NT)
delta_chunk_solve_kernel(const float* __restrict__ qkv, int C, const float* __restrict__ bg, float* __restrict__ scratch,
                         float* __restrict__ full, const int32_t* __restrict__ tile_tok0, const int32_t* __restrict__ tile_ntok, int H, int G,
                         int d, int e) {
  extern __shared__ __align__(16) float dc_smem[];
  __shared__ double lg[CHUNK], to_start[CHUNK], to_end[CHUNK];      // L_t, exp(L_t), exp(L_n - L_t)
  __shared__ float beta[CHUNK];
  constexpr int AP = DC_SOLVE_PITCH, NY = NT / 16, RM = CHUNK / NY;
  const int P = chunk_pitch(d);
  double* at = reinterpret_cast<double*>(dc_smem);       // [s][t]: A[t][s]
  float* ks = reinterpret_cast<float*>(at + CHUNK * AP); // [CHUNK][P]
  const int tile = blockIdx.x, h = blockIdx.y, g = h / (H / G), tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  chunk_rows(ks, P, qkv + (size_t)tok0 * C + G * d + g * d, C, CHUNK, ntok, d);
  asm volatile("cp.async.commit_group;" ::: "memory");
  dc_logs(lg, bg, tok0, ntok, H, h);
  if (threadIdx.x >= 64 && threadIdx.x < 64 + CHUNK) {
    const int t = threadIdx.x - 64;
    beta[t] = t < ntok ? bg[(size_t)(tok0 + t) * 2 * H + h] : 0.f;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (threadIdx.x < CHUNK) to_start[threadIdx.x] = exp(lg[threadIdx.x]);
  else if (threadIdx.x < 2 * CHUNK) to_end[threadIdx.x - CHUNK] = exp(lg[CHUNK - 1] - lg[threadIdx.x - CHUNK]);
  {
    double acc[RM][4];
    chunk_mm_runs<NY, RM, 4>(acc, ks, P, CHUNK, ks, P, CHUNK, d);
#pragma unroll
    for (int a = 0; a < RM; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int s = chunk_ty() + NY * a, t = chunk_tx() + 16 * b;
        at[s * AP + t] = s < t ? (double)beta[t] * exp(lg[t] - lg[s]) * acc[a][b] : 0.0;
      }
  }
  __syncthreads();
  const int c = threadIdx.x;
  float* base = scratch + ((size_t)tile * H + h) * dc_floats(d, e);
  if (c == 0) full[(size_t)tile * H + h] = (float)to_start[CHUNK - 1];
  if (c >= d + e) return;
  double x[CHUNK];
  if (c < e) {
    const float* v = qkv + (size_t)tok0 * C + 2 * G * d + (size_t)h * e + c;
#pragma unroll
    for (int t = 0; t < CHUNK; ++t) x[t] = t < ntok ? v[(size_t)t * C] : 0.f;
#pragma unroll
    for (int t = 0; t < CHUNK; ++t) x[t] *= beta[t];
  } else {
    float* kt = base + (size_t)CHUNK * e + (size_t)CHUNK * d + (size_t)(c - e) * CHUNK;
#pragma unroll
    for (int t = 0; t < CHUNK; t += 4) {
      float k[4], out[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        k[i] = ks[(t + i) * P + c - e];
        out[i] = (float)(k[i] * to_end[t + i]);
        x[t + i] = k[i] * (beta[t + i] * to_start[t + i]);
      }
      *reinterpret_cast<float4*>(kt + t) = make_float4(out[0], out[1], out[2], out[3]);
    }
  }
#pragma unroll
  for (int s = 0; s < CHUNK - 1; ++s) {
#pragma unroll
    for (int t = (s + 1) & ~1; t < CHUNK; t += 2) {      // (at [s][t] is zero up to t = s)
      const double2 a = *reinterpret_cast<const double2*>(at + s * AP + t);
      if (t > s) x[t] = fma(-a.x, x[s], x[t]);
      x[t + 1] = fma(-a.y, x[s], x[t + 1]);
    }
  }
  if (c < e) {
#pragma unroll
    for (int t = 0; t < CHUNK; t += 4)
      *reinterpret_cast<float4*>(base + (size_t)c * CHUNK + t) = make_float4((float)x[t], (float)x[t + 1], (float)x[t + 2], (float)x[t + 3]);
  } else {
#pragma unroll
    for (int t = 0; t < CHUNK; ++t) base[(size_t)CHUNK * e + (size_t)t * d + c - e] = (float)x[t];
  }
}

template <int RN>      // ceil(d / 16)
__global__ void __launch_bounds__(DC_STATE_THREADS)
delta_chunk_states_kernel(float* __restrict__ scratch, const float* __restrict__ full, float* __restrict__ state,
                          const int32_t* __restrict__ seq_tok0, const int32_t* __restrict__ seq_slot, int H, int d, int e) {
  extern __shared__ __align__(16) float dc_smem[];
  constexpr int AP = CHUNK + 4;
  const int P = chunk_pitch(d), STAGE = CHUNK * P + d * AP + DC_BLOCK * CHUNK;
  float* ss = dc_smem + 2 * STAGE;           // the state's rows [DC_BLOCK][P]
  float* us = ss + DC_BLOCK * P;             // U [DC_BLOCK][AP]
  const int s = blockIdx.x / H, h = blockIdx.x - s * H, j0 = blockIdx.y * DC_BLOCK, nj = min(DC_BLOCK, e - j0);
  int first = 0;                             // the sequence's first tile: every earlier sequence has ceil(n / CHUNK)
  for (int p = 0; p < s; ++p) first += (seq_tok0[p + 1] - seq_tok0[p] + CHUNK - 1) / CHUNK;
  const int chunks = (seq_tok0[s + 1] - seq_tok0[s] + CHUNK - 1) / CHUNK;
  if (chunks == 0) return;
  const size_t FL = dc_floats(d, e);
  float* st = state + ((size_t)seq_slot[s] * H + h) * e * d + (size_t)j0 * d;
  auto load = [&](int c) {                   // W, the scaled keys, this block's rows of U0
    float* dst = dc_smem + (c & 1) * STAGE;
    const float* base = scratch + ((size_t)(first + c) * H + h) * FL;
    chunk_rows(dst, P, base + (size_t)CHUNK * e, d, CHUNK, CHUNK, d);
    chunk_rows(dst + CHUNK * P, AP, base + (size_t)CHUNK * e + (size_t)CHUNK * d, CHUNK, d, d, CHUNK);
    chunk_rows(dst + CHUNK * P + d * AP, CHUNK, base + (size_t)j0 * CHUNK, CHUNK, DC_BLOCK, nj, CHUNK);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0);
  const int tx = chunk_tx(), ty = chunk_ty();
  float S[2][RN];                            // rows ty + 8 a of the block's channels, key channels tx + 16 b
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < RN; ++b) {
      const int j = ty + 8 * a, i = tx + 16 * b;
      S[a][b] = j < nj && i < d ? st[(size_t)j * d + i] : 0.f;
    }
  float keep_next = full[(size_t)first * H + h];
  for (int c = 0; c < chunks; ++c) {
    float* base = scratch + ((size_t)(first + c) * H + h) * FL;
    float* kept = base + (size_t)CHUNK * e + (size_t)(2 * CHUNK) * d + (size_t)j0 * d;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < RN; ++b) {
        const int j = ty + 8 * a, i = tx + 16 * b;
        if (i < d) {
          ss[j * P + i] = S[a][b];
          if (j < nj) kept[(size_t)j * d + i] = S[a][b];
        }
      }
    const float keep = keep_next;
    if (c + 1 < chunks) {
      load(c + 1);
      keep_next = full[(size_t)(first + c + 1) * H + h];
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* ws = dc_smem + (c & 1) * STAGE;
    const float* u0 = ws + CHUNK * P + d * AP;
    float acc[2][4] = {};
    chunk_mm<8, 2, 4>(acc, ss, P, DC_BLOCK, ws, P, CHUNK, d);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int j = ty + 8 * a, t = tx + 16 * b;
        const float u = u0[j * CHUNK + t] - acc[a][b];
        us[j * AP + t] = u;
        if (j < nj) base[(size_t)(j0 + j) * CHUNK + t] = u;
      }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < RN; ++b) S[a][b] *= keep;
    chunk_mm<8, 2, RN>(S, us, AP, DC_BLOCK, ws + CHUNK * P, AP, d, CHUNK);
    __syncthreads();                         // `ss`, `us` and this stage are free
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < RN; ++b) {
      const int j = ty + 8 * a, i = tx + 16 * b;
      if (j < nj && i < d) st[(size_t)j * d + i] = S[a][b];
    }
}

template <int RN>      // ceil(e / 16)
__global__ void __launch_bounds__(256, RN <= 4 ? 2 : 1)
delta_chunk_out_kernel(const float* __restrict__ qkv, int C, const float* __restrict__ bg, const float* __restrict__ scratch,
                       float* __restrict__ o, const int32_t* __restrict__ tile_tok0, const int32_t* __restrict__ tile_ntok, int H, int G, int d,
                       int e) {
  extern __shared__ __align__(16) float dc_smem[];
  __shared__ double lg[CHUNK];
  constexpr int AP = CHUNK + 4;
  const int P = chunk_pitch(d);
  float* qs = dc_smem;                       // [CHUNK][P]
  float* ks = qs + CHUNK * P;                // [CHUNK][P]
  float* ss = ks + CHUNK * P;                // S0 [e][P]
  float* us = ss + e * P;                    // U [e][AP]
  float* ms = us + e * AP;                   // the chunk's own weights [t][s]
  const int tile = blockIdx.x, h = blockIdx.y, g = h / (H / G), tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  const float* base = scratch + ((size_t)tile * H + h) * dc_floats(d, e);
  const float* row = qkv + (size_t)tok0 * C + g * d;
  chunk_rows(qs, P, row, C, CHUNK, ntok, d);
  chunk_rows(ks, P, row + G * d, C, CHUNK, ntok, d);
  asm volatile("cp.async.commit_group;" ::: "memory");
  chunk_rows(ss, P, base + (size_t)CHUNK * e + (size_t)(2 * CHUNK) * d, d, e, e, d);
  chunk_rows(us, AP, base, CHUNK, e, e, CHUNK);
  asm volatile("cp.async.commit_group;" ::: "memory");
  dc_logs(lg, bg, tok0, ntok, H, h);
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  const int tx = chunk_tx(), ty = chunk_ty();
  {
    double acc[4][4];
    chunk_mm_runs<16, 4, 4>(acc, qs, P, CHUNK, ks, P, CHUNK, d);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int t = ty + 16 * a, s = tx + 16 * b;
        ms[t * AP + s] = s <= t ? (float)(exp(lg[t] - lg[s]) * acc[a][b]) : 0.f;
      }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float acc[4][RN] = {};
  chunk_mm<16, 4, RN>(acc, qs, P, CHUNK, ss, P, e, d);
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const float w = (float)exp(lg[ty + 16 * a]);
#pragma unroll
    for (int b = 0; b < RN; ++b) acc[a][b] *= w;
  }
  chunk_mm<16, 4, RN>(acc, ms, AP, CHUNK, us, AP, e, CHUNK);
  bool all_finite = true;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < RN; ++b) {
      const int t = ty + 16 * a, j = tx + 16 * b;
      if (t >= ntok || j >= e) continue;
      o[(size_t)(tok0 + t) * H * e + (size_t)h * e + j] = acc[a][b];
      all_finite = all_finite && isfinite(acc[a][b]);
    }
  if (all_finite) return;
#pragma unroll 1
  for (int i = 0; i < 4 * RN; ++i) {
    const int t = ty + 16 * (i / RN), j = tx + 16 * (i % RN);
    float* out = o + (size_t)(tok0 + t) * H * e + (size_t)h * e + j;
    if (t < ntok && j < e && !isfinite(*out)) *out = chunk_causal(qs + t * P, ss + j * P, d, (float)exp(lg[t]), ms + t * AP, us + j * AP, t);
  }
}

}  // namespace edgelm

using namespace edgelm;

static int g_delta_columns = 0;
// Columns of the state a thread of `delta_scan` holds (1, 2 or 4; 0: the kernel's own choice).  For measurements.
extern "C" int edgelm_delta_scan_columns(int n) {
  g_delta_columns = (n == 1 || n == 2 || n == 4) ? n : 0;
  return 0;
}

extern "C" int edgelm_delta_prepare(float* qkv, int C, const float* u, int ldu, int b_off, int a_off, const float* A_log,
                                    const float* dt_bias, float* bg, int n_tokens, int H, int G, int d, int e, float unit_eps,
                                    float q_scale, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  EL_REFUSE(n_tokens > 0 && H > 0 && G > 0 && H % G == 0 && d > 0 && e > 0 && C == 2 * G * d + H * e, "delta_prepare: sizes do not fit (heads %d over %d, %d x %d, channels %d)", H, G, d, e, C);
  EL_REFUSE(b_off >= 0 && a_off >= 0 && b_off + H <= ldu && a_off + H <= ldu, "delta_prepare: rows of %d values are too short", ldu);
  const int vec_blocks = n_tokens >= 256 ? 1 : (2 * G + 3) / 4;    // a step of few tokens: a warp a vector
  launch_pdl(pdl_bit_for_tokens(n_tokens), delta_prepare_kernel, dim3(n_tokens, vec_blocks), dim3(128), (size_t)0, stream, qkv, C, u, ldu, b_off, a_off, A_log,
             dt_bias, bg, H, G, d, unit_eps, q_scale);
  EL_LAUNCH_CHECK("delta_prepare");
  return 0;
}

extern "C" int edgelm_delta_scan(const float* qkv, int C, const float* bg, float* state, float* o, const int32_t* seq_tok0,
                                 const int32_t* seq_slot, int n_seqs, int n_tokens, int H, int G, int d, int e, cudaStream_t stream) {
  if (n_seqs == 0) return 0;
  EL_REFUSE(n_seqs > 0 && n_seqs <= 65535 && H > 0 && H <= 65535 && G > 0 && H % G == 0 && C == 2 * G * d + H * e, "delta_scan: sizes do not fit (heads %d over %d, channels %d)", H, G, C);
  EL_REFUSE(d >= 1 && d <= 256 && e >= 1, "delta_scan: a state of %d rows per head is not taken (1 to 256)", d);
  // Columns a thread.  Measured (keys and values of 64, 32 heads): one sequence of 2,048 tokens 0.66 / 0.73 / 0.87 ms with 1 / 2 /
  // 4 columns; eight sequences of 512 tokens 0.39 / 0.30 / 0.29 ms.  (Fewer lanes a column, down to a whole column a thread
  // without any shuffle, were measured too: 0.87 to 0.97 ms for the one sequence.)  So one column while the warps leave the
  // device room, else four (two where a column's rows fill the registers), fewer for value heads so narrow that lanes would
  // idle.  `edgelm_delta_scan_columns` overrides, for measurements.
  const int cpt_max = d <= 128 ? 4 : 2;
  const long long warps1 = (long long)n_seqs * H * ((e + 3) / 4);      // warps with one column a thread
  int cpt = g_delta_columns > 0 ? (g_delta_columns < cpt_max ? g_delta_columns : cpt_max) : (warps1 <= 148 * 16 ? 1 : cpt_max);
  while (cpt > 1 && e <= DS_GROUPS * (cpt / 2)) cpt >>= 1;
  const dim3 grid((e + DS_GROUPS * cpt - 1) / (DS_GROUPS * cpt), H, n_seqs), block(DS_THREADS);
  const int bit = pdl_bit_for_tokens(n_tokens);
#define EL_DS2(RPT, CPT) launch_pdl(bit, delta_scan_kernel<RPT, CPT>, grid, block, (size_t)0, stream, qkv, C, bg, state, o, seq_tok0, seq_slot, H, G, d, e)
#define EL_DS(RPT) do { if (cpt == 4) EL_DS2(RPT, 4); else if (cpt == 2) EL_DS2(RPT, 2); else EL_DS2(RPT, 1); } while (0)
  if (d <= 32) EL_DS(4);
  else if (d <= 64) EL_DS(8);
  else if (d <= 128) EL_DS(16);
  else { if (cpt == 2) EL_DS2(32, 2); else EL_DS2(32, 1); }
#undef EL_DS
#undef EL_DS2
  EL_LAUNCH_CHECK("delta_scan");
  return 0;
}

// 1 if the chunked form takes heads of these sizes (whole pieces of 16 bytes, its tiles in shared memory).
extern "C" int edgelm_delta_chunked_takes(int d, int e) { return d >= 4 && d <= 128 && e >= 4 && e <= 128 && d % 4 == 0 && e % 4 == 0 ? 1 : 0; }

// `edgelm_delta_scan` chunk by chunk (three launches): the step's tokens come as tiles of at most CHUNK consecutive tokens of one
// sequence, in the order of the sequences, every sequence cut from its first row of the step.  scratch: n_tiles H (`dc_floats` + 4) floats.
extern "C" int edgelm_delta_chunked(const float* qkv, int C, const float* bg, float* state, float* o, const int32_t* seq_tok0,
                                    const int32_t* seq_slot, int n_seqs, const int32_t* tile_tok0, const int32_t* tile_ntok, int n_tiles, int H,
                                    int G, int d, int e, float* scratch, cudaStream_t stream) {
  if (n_seqs == 0 || n_tiles == 0) return 0;
  EL_REFUSE(n_seqs > 0 && n_tiles > 0 && H > 0 && H <= 65535 && G > 0 && H % G == 0 && C == 2 * G * d + H * e, "delta_chunked: sizes do not fit (heads %d over %d, channels %d)", H, G, C);
  EL_REFUSE(edgelm_delta_chunked_takes(d, e), "delta_chunked: heads of %d x %d are not taken (use the scan)", d, e);
  EL_REFUSE(scratch != nullptr && (uintptr_t)scratch % 16 == 0 && (uintptr_t)qkv % 16 == 0, "delta_chunked: rows and scratch must be 16-byte aligned");
  const int P = chunk_pitch(d), AP = CHUNK + 4;
  float* full = scratch + (size_t)n_tiles * H * dc_floats(d, e);
  const size_t smem1 = (size_t)CHUNK * DC_SOLVE_PITCH * 8 + (size_t)CHUNK * P * 4;
  auto k1 = d + e <= 128 ? delta_chunk_solve_kernel<128> : delta_chunk_solve_kernel<256>;
  const size_t smem2 = (size_t)(2 * (CHUNK * P + d * AP + DC_BLOCK * CHUNK) + DC_BLOCK * P + DC_BLOCK * AP) * 4;
  const size_t smem3 = (size_t)(2 * CHUNK * P + e * P + e * AP + CHUNK * AP) * 4;
  auto k2 = d <= 64 ? delta_chunk_states_kernel<4> : delta_chunk_states_kernel<8>;
  auto k3 = e <= 64 ? delta_chunk_out_kernel<4> : delta_chunk_out_kernel<8>;
  cudaError_t err = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(k3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem3);
  EL_REFUSE(err == cudaSuccess, "delta_chunked: shared memory refused: %s", cudaGetErrorString(err));
  k1<<<dim3(n_tiles, H), d + e <= 128 ? 128 : 256, smem1, stream>>>(qkv, C, bg, scratch, full, tile_tok0, tile_ntok, H, G, d, e);
  EL_LAUNCH_CHECK("delta_chunk_solve");
  k2<<<dim3(n_seqs * H, (e + DC_BLOCK - 1) / DC_BLOCK), DC_STATE_THREADS, smem2, stream>>>(scratch, full, state, seq_tok0, seq_slot, H, d, e);
  EL_LAUNCH_CHECK("delta_chunk_states");
  k3<<<dim3(n_tiles, H), 256, smem3, stream>>>(qkv, C, bg, scratch, o, tile_tok0, tile_ntok, H, G, d, e);
  EL_LAUNCH_CHECK("delta_chunk_out");
  return 0;
}
