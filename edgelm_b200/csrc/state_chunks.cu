// Prompt steps of the state mixers chunk by chunk: the step's tokens come as tiles of at most CHUNK consecutive tokens of one sequence,
// in the order of the sequences, every sequence cut from its first row of the step.  The walks of recurrent.cu take a token after the
// other (0.27 us each); here everything but a multiply-add per state element and chunk runs for all chunks at once.  States, decays,
// step sizes and sums are float32, logarithms of decays double; scores join runs of eight float32 products in double.
//
// Selective state-space recurrence (S <- a_t S + dt_t B_t x_t^T, y_t = S^T C_t + D x_t, a_t = exp(-exp(A_log) dt_t)), with L_t the sum of
// log a up to token t of the chunk and S0 the state before it:
//     y_t = exp(L_t) S0^T C_t + sum_(s <= t) exp(L_t - L_s) (C_t . B_s) dt_s x_s + D x_t
//     S   = exp(L_n) S0 + sum_s exp(L_n - L_s) dt_s B_s x_s^T
//   1. `ssm_chunk_scores`, per (chunk, group): C_t . B_s, and B transposed, both shared by the group's heads;
//   2. `ssm_chunk_state`, per (chunk, head): the chunk's own sum of the second line;
//   3. `chunk_fold`: the chunks of a sequence in order, element by element: S0 in place of that sum, the state moved on;
//   4. `ssm_chunk_out`, per (chunk, head): the first line.
// Most of the time goes to the products out of shared memory of 2. and 4.  2,048 tokens of one sequence, 64 heads of 128 x 64: the walk
// 597 us, this 230 (state 80, out 126, the other two 24).
//
// Decayed outer-product recurrence with a bonus (o_t = (S + diag(u) k_t v_t^T)^T r_t, S <- diag(w_t) S + k_t v_t^T; a decay per key channel):
//   1. `wkv_chunk_local`, per (chunk, head): the walk over the chunk's tokens from a state of zeros, a thread 8 key channels of 4 value
//      channels in registers; its outputs, its last state, and r_t times the product of the decays before t;
//   2. `chunk_fold`;
//   3. `wkv_chunk_out`, per (chunk, head): what S0 adds to the outputs, one product.
// Most of the time goes to 1. (three multiply-adds a state element and token).  2,048 tokens, 32 heads of 64: the walk 562 us, this
// 148.
#include "chunk_mm.cuh"

namespace edgelm {

// dst [n][pitch] = the transposed rows [CHUNK][n] of `src` (n and ld multiples of 4, 16-byte aligned), row s times w[s]; zeros for the
// rows from `valid` on.  Neighbouring threads take neighbouring rows, so that they store next to each other; four requests a thread
// before the first is used.
__device__ __forceinline__ void chunk_transposed(float* dst, int pitch, const float* __restrict__ src, size_t ld, int valid, int n, const float* w) {
  const int total = CHUNK * (n >> 2);
  for (int base = threadIdx.x; base < total; base += 4 * blockDim.x) {
    float4 v[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int i = base + x * blockDim.x, s = i % CHUNK, c = i / CHUNK * 4;
      v[x] = i < total && s < valid ? *reinterpret_cast<const float4*>(src + (size_t)s * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int i = base + x * blockDim.x, s = i % CHUNK, c = i / CHUNK * 4;
      if (i >= total) break;
      const float f = w ? w[s] : 1.f;
      dst[c * pitch + s] = v[x].x * f;
      dst[(c + 1) * pitch + s] = v[x].y * f;
      dst[(c + 2) * pitch + s] = v[x].z * f;
      dst[(c + 3) * pitch + s] = v[x].w * f;
    }
  }
}

// lg[t]: the sum of -exp(A_log) dt up to token t; dts[t] = dt = softplus(raw + bias) (0 from ntok on).  By the first warp; the block
// synchronises afterwards.
__device__ __forceinline__ void ssm_logs(double* lg, float* dts, const float* __restrict__ raw, int ldu, float bias, float a_log, int tok0, int ntok) {
  if (threadIdx.x >= 32) return;
  const double rate = -(double)expf(a_log);
  double x[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = 2 * threadIdx.x + i;
    const float z = t < ntok ? raw[(size_t)(tok0 + t) * ldu] + bias : 0.f;
    const float dt = t < ntok ? log1pf(expf(-fabsf(z))) + fmaxf(z, 0.f) : 0.f;
    dts[t] = dt;
    const double l = t < ntok ? rate * dt : 0.0;
    x[i] = l < -200.0 ? -200.0 : l;      // (a decay that is zero in float32: sums and differences stay finite; a NaN stays one)
  }
  chunk_log_sums(lg, x[0], x[1]);
}

constexpr int SC_PITCH = CHUNK + 4;

// scores [tile][G][CHUNK][CHUNK], then B transposed [tile][G][N][CHUNK]
__global__ void __launch_bounds__(256, 2)
ssm_chunk_scores_kernel(const float* __restrict__ xbc, int C, int inner, float* __restrict__ shared_part, const int32_t* __restrict__ tile_tok0,
                        const int32_t* __restrict__ tile_ntok, int G, int N) {
  extern __shared__ __align__(16) float sc_smem[];
  const int P = chunk_pitch(N);
  float* bs = sc_smem;
  float* cs = bs + CHUNK * P;
  const int tile = blockIdx.x, g = blockIdx.y, tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  const float* row = xbc + (size_t)tok0 * C + inner + g * N;
  chunk_rows(bs, P, row, C, CHUNK, ntok, N);
  chunk_rows(cs, P, row + G * N, C, CHUNK, ntok, N);
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* out = shared_part + ((size_t)tile * G + g) * (CHUNK * CHUNK + (size_t)CHUNK * N);
  double acc[4][4];
  chunk_mm_runs<16, 4, 4>(acc, cs, P, CHUNK, bs, P, CHUNK, N);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) out[(chunk_ty() + 16 * a) * CHUNK + chunk_tx() + 16 * b] = (float)acc[a][b];
  out += CHUNK * CHUNK;
  for (int i = threadIdx.x; i < CHUNK * N; i += blockDim.x) out[i] = bs[(i % CHUNK) * P + i / CHUNK];
}

// sums [tile][H][P][N], keep [tile][H] = exp(L_n)
template <int RN>      // ceil(N / 16)
__global__ void __launch_bounds__(256, 2)
ssm_chunk_state_kernel(const float* __restrict__ xbc, int C, const float* __restrict__ dt_raw, int ldu, const float* __restrict__ dt_bias,
                       const float* __restrict__ A_log,
                       const float* __restrict__ shared_part, float* __restrict__ sums, float* __restrict__ keep,
                       const int32_t* __restrict__ tile_tok0, const int32_t* __restrict__ tile_ntok, int H, int G, int N, int P) {
  extern __shared__ __align__(16) float sc_smem[];
  __shared__ double lg[CHUNK];
  __shared__ float w[CHUNK];
  float* xt = sc_smem;                       // [P][SC_PITCH]: x_s dt_s exp(L_n - L_s)
  float* bt = xt + P * SC_PITCH;             // [N][SC_PITCH]
  const int tile = blockIdx.x, h = blockIdx.y, g = h / (H / G), tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  chunk_rows(bt, SC_PITCH, shared_part + ((size_t)tile * G + g) * (CHUNK * CHUNK + (size_t)CHUNK * N) + CHUNK * CHUNK, CHUNK, N, N, CHUNK);
  asm volatile("cp.async.commit_group;" ::: "memory");
  ssm_logs(lg, w, dt_raw + h, ldu, dt_bias[h], A_log[h], tok0, ntok);
  __syncthreads();
  if (threadIdx.x < CHUNK) w[threadIdx.x] *= expf((float)(lg[CHUNK - 1] - lg[threadIdx.x]));
  if (threadIdx.x == CHUNK) keep[(size_t)tile * H + h] = expf((float)lg[CHUNK - 1]);
  __syncthreads();
  chunk_transposed(xt, SC_PITCH, xbc + (size_t)tok0 * C + h * P, C, ntok, P, w);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float acc[4][RN] = {};
  chunk_mm<16, 4, RN>(acc, xt, SC_PITCH, P, bt, SC_PITCH, N, CHUNK);
  float* out = sums + ((size_t)tile * H + h) * P * N;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < RN; ++b) {
      const int p = chunk_ty() + 16 * a, n = chunk_tx() + 16 * b;
      if (p < P && n < N) out[(size_t)p * N + n] = acc[a][b];
    }
}

// Per (sequence, head), element by element: the chunks in order; the state before a chunk overwrites the chunk's sum, the slot's
// state moves on.  `keep`: the chunk's decay, [tile][H][cols] (cols 1: one for all elements).  An element's column is its index mod
// `cols`.  A thread requests eight chunks' values before the chain of multiply-adds through them.
__global__ void __launch_bounds__(128)
chunk_fold_kernel(float* __restrict__ sums, const float* __restrict__ keep, float* __restrict__ state, const int32_t* __restrict__ seq_tok0,
                  const int32_t* __restrict__ seq_slot, int H, int elements, int cols) {
  const int s = blockIdx.x / H, h = blockIdx.x - s * H, e = blockIdx.y * blockDim.x + threadIdx.x;
  if (e >= elements) return;
  int first = 0;                             // the sequence's first tile: every earlier sequence has ceil(n / CHUNK)
  for (int p = 0; p < s; ++p) first += (seq_tok0[p + 1] - seq_tok0[p] + CHUNK - 1) / CHUNK;
  const int chunks = (seq_tok0[s + 1] - seq_tok0[s] + CHUNK - 1) / CHUNK;
  if (chunks == 0) return;
  float* sp = state + ((size_t)seq_slot[s] * H + h) * elements + e;
  float* a = sums + ((size_t)first * H + h) * elements + e;
  const float* k = keep + ((size_t)first * H + h) * cols + e % cols;
  const size_t step = (size_t)H * elements, kstep = (size_t)H * cols;
  float S = *sp;
  for (int c0 = 0; c0 < chunks; c0 += 8) {
    float add[8], dec[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      add[x] = c0 + x < chunks ? a[(size_t)(c0 + x) * step] : 0.f;
      dec[x] = c0 + x < chunks ? k[(size_t)(c0 + x) * kstep] : 0.f;
    }
#pragma unroll
    for (int x = 0; x < 8; ++x)
      if (c0 + x < chunks) {
        a[(size_t)(c0 + x) * step] = S;
        S = fmaf(dec[x], S, add[x]);
      }
  }
  *sp = S;
}

__global__ void __launch_bounds__(256, 2)
ssm_chunk_out_kernel(const float* __restrict__ xbc, int C, int inner, const float* __restrict__ dt_raw, int ldu, const float* __restrict__ dt_bias,
                       const float* __restrict__ A_log,
                     const float* __restrict__ Dp, const float* __restrict__ shared_part, const float* __restrict__ before,
                     float* __restrict__ y, const int32_t* __restrict__ tile_tok0, const int32_t* __restrict__ tile_ntok, int H, int G, int N,
                     int P) {
  extern __shared__ __align__(16) float sc_smem[];
  __shared__ double lg[CHUNK];
  __shared__ float dts[CHUNK];
  const int NP = chunk_pitch(N);
  float* cs = sc_smem;                       // C [CHUNK][NP]
  float* ss = cs + CHUNK * NP;               // S0 [P][NP]
  float* ms = ss + P * NP;                   // the chunk's own weights [t][s]
  float* xt = ms + CHUNK * SC_PITCH;         // x transposed [P][SC_PITCH]
  const int tile = blockIdx.x, h = blockIdx.y, g = h / (H / G), tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  chunk_rows(cs, NP, xbc + (size_t)tok0 * C + inner + G * N + g * N, C, CHUNK, ntok, N);
  chunk_rows(ss, NP, before + ((size_t)tile * H + h) * P * N, N, P, P, N);
  chunk_rows(ms, SC_PITCH, shared_part + ((size_t)tile * G + g) * (CHUNK * CHUNK + (size_t)CHUNK * N), CHUNK, CHUNK, CHUNK, CHUNK);
  asm volatile("cp.async.commit_group;" ::: "memory");
  ssm_logs(lg, dts, dt_raw + h, ldu, dt_bias[h], A_log[h], tok0, ntok);
  chunk_transposed(xt, SC_PITCH, xbc + (size_t)tok0 * C + h * P, C, ntok, P, nullptr);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int i = threadIdx.x; i < CHUNK * CHUNK; i += 256) {
    const int t = i / CHUNK, s = i % CHUNK;
    ms[t * SC_PITCH + s] = s <= t ? ms[t * SC_PITCH + s] * (expf((float)(lg[t] - lg[s])) * dts[s]) : 0.f;
  }
  __syncthreads();
  float acc[4][4] = {};
  chunk_mm<16, 4, 4>(acc, cs, NP, CHUNK, ss, NP, P, N);
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const float w = expf((float)lg[chunk_ty() + 16 * a]);
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] *= w;
  }
  chunk_mm<16, 4, 4>(acc, ms, SC_PITCH, CHUNK, xt, SC_PITCH, P, CHUNK);
  const float D = Dp[h];
  bool all_finite = true;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int t = chunk_ty() + 16 * a, p = chunk_tx() + 16 * b;
      if (t >= ntok || p >= P) continue;
      const float v = acc[a][b] + D * xt[p * SC_PITCH + t];
      y[(size_t)(tok0 + t) * H * P + (size_t)h * P + p] = v;
      all_finite = all_finite && isfinite(v);
    }
  if (all_finite) return;
#pragma unroll 1
  for (int i = 0; i < 16; ++i) {
    const int t = chunk_ty() + 16 * (i >> 2), p = chunk_tx() + 16 * (i & 3);
    float* out = y + (size_t)(tok0 + t) * H * P + (size_t)h * P + p;
    if (t < ntok && p < P && !isfinite(*out))
      *out = chunk_causal(cs + t * NP, ss + p * NP, N, expf((float)lg[t]), ms + t * SC_PITCH, xt + p * SC_PITCH, t) + D * xt[p * SC_PITCH + t];
  }
}

// ------------------------------------------------------------------ a decay per key channel
constexpr int WK = 64;             // channels a block holds (heads of up to 64 x 64)
constexpr int WK_THREADS = 128;

// (chunk, head) of the scratch: the last state, later S0, [j][i]; r_t times the decays before t, [CHUNK][K]; the product of all decays [K]
// is kept apart ([tile][H][K]).
__global__ void __launch_bounds__(WK_THREADS)
wkv_chunk_local_kernel(const float* __restrict__ r, const float* __restrict__ kk, const float* __restrict__ v, const float* __restrict__ w,
                       const float* __restrict__ bonus, float* __restrict__ sums, float* __restrict__ faded, float* __restrict__ keep,
                       float* __restrict__ o, const int32_t* __restrict__ tile_tok0, const int32_t* __restrict__ tile_ntok, int H, int K) {
  extern __shared__ __align__(16) float sc_smem[];
  __shared__ float own[CHUNK];               // sum over i of bonus[i] r_t[i] k_t[i]
  float* rs = sc_smem;                       // four times [CHUNK][WK] (channels from K on: zeros)
  float* ks = rs + CHUNK * WK;
  float* vs = ks + CHUNK * WK;
  float* ws = vs + CHUNK * WK;
  const int tile = blockIdx.x, h = blockIdx.y, tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  const size_t ld = (size_t)H * K, at = (size_t)tok0 * ld + (size_t)h * K;
  if (K < WK)
    for (int i = threadIdx.x; i < 4 * CHUNK * WK; i += WK_THREADS) sc_smem[i] = 0.f;
  if (K < WK) __syncthreads();
  chunk_rows(rs, WK, r + at, ld, ntok, ntok, K);
  chunk_rows(ks, WK, kk + at, ld, ntok, ntok, K);
  chunk_rows(vs, WK, v + at, ld, ntok, ntok, K);
  chunk_rows(ws, WK, w + at, ld, ntok, ntok, K);
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  {
    // the outputs' share of S0: r_t times the decays of the tokens before it, two halves of the chunk side by side
    const int i = threadIdx.x & 63, half = threadIdx.x >> 6, begin = half ? min(CHUNK / 2, ntok) : 0, end = half ? ntok : min(CHUNK / 2, ntok);
    if (i < K) {
      double d = 1.0;                        // (in float32 the product's roundings alone were a tenth of the outputs' error)
      for (int t = 0; t < begin; ++t) d *= ws[t * WK + i];
      float* out = faded + (((size_t)tile * H + h) * CHUNK) * K + i;
      for (int t = begin; t < end; ++t) {
        out[(size_t)t * K] = (float)(rs[t * WK + i] * d);
        d *= ws[t * WK + i];
      }
      if (half) keep[((size_t)tile * H + h) * K + i] = (float)d;
    }
  }
  {
    const int t = threadIdx.x >> 1, c0 = (threadIdx.x & 1) * (WK / 2);
    float part[8] = {};                      // (eight short runs: one of 32 was less exact than the walk's sums)
    if (t < ntok)
#pragma unroll
      for (int c = 0; c < WK / 2; ++c)
        if (c0 + c < K) part[c & 7] = fmaf(bonus[h * K + c0 + c], rs[t * WK + c0 + c] * ks[t * WK + c0 + c], part[c & 7]);
    float b = ((part[0] + part[4]) + (part[1] + part[5])) + ((part[2] + part[6]) + (part[3] + part[7]));
    b += __shfl_xor_sync(0xffffffffu, b, 1);
    if ((threadIdx.x & 1) == 0) own[t] = b;
  }
  __syncthreads();
  // eight neighbouring pairs of lanes hold key channels 4 sub .. and 32 + 4 sub .. of the value channels 4 grp ..
  const int lane = threadIdx.x & 31, sub = lane >> 1 & 7, grp = (lane & 1) + (lane >> 4) * 2 + (threadIdx.x >> 5) * 4;
  float S[4][8] = {};
  for (int t = 0; t < ntok; ++t) {
    float rr[8], kv[8], ww[8], vj[4], acc[4];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      *reinterpret_cast<float4*>(rr + 4 * p) = *reinterpret_cast<const float4*>(rs + t * WK + 32 * p + 4 * sub);
      *reinterpret_cast<float4*>(kv + 4 * p) = *reinterpret_cast<const float4*>(ks + t * WK + 32 * p + 4 * sub);
      *reinterpret_cast<float4*>(ww + 4 * p) = *reinterpret_cast<const float4*>(ws + t * WK + 32 * p + 4 * sub);
    }
    *reinterpret_cast<float4*>(vj) = *reinterpret_cast<const float4*>(vs + t * WK + 4 * grp);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a0 = 0.f, a1 = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        a0 = fmaf(S[j][i], rr[i], a0);
        a1 = fmaf(S[j][i + 1], rr[i + 1], a1);
        S[j][i] = fmaf(ww[i], S[j][i], kv[i] * vj[j]);
        S[j][i + 1] = fmaf(ww[i + 1], S[j][i + 1], kv[i + 1] * vj[j]);
      }
      acc[j] = a0 + a1;
    }
    // over the eight sublanes (lane bits 1, 2, 3): two values change hands at each of the first two steps
    const bool b1 = lane & 2, b2 = lane & 4;
    float p0 = (b1 ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, b1 ? acc[0] : acc[2], 2);
    float p1 = (b1 ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, b1 ? acc[1] : acc[3], 2);
    float q = (b2 ? p1 : p0) + __shfl_xor_sync(0xffffffffu, b2 ? p0 : p1, 4);
    q += __shfl_xor_sync(0xffffffffu, q, 8);
    const int j = 4 * grp + (b1 ? 2 : 0) + (b2 ? 1 : 0);
    if ((lane & 8) == 0 && j < K) o[(size_t)(tok0 + t) * ld + (size_t)h * K + j] = fmaf(own[t], vs[t * WK + j], q);
  }
  float* out = sums + ((size_t)tile * H + h) * K * K;
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int p = 0; p < 2; ++p)
      if (4 * grp + j < K && 32 * p + 4 * sub < K)
        *reinterpret_cast<float4*>(out + (size_t)(4 * grp + j) * K + 32 * p + 4 * sub) = make_float4(S[j][4 * p], S[j][4 * p + 1], S[j][4 * p + 2], S[j][4 * p + 3]);
}

__global__ void __launch_bounds__(256, 2)
wkv_chunk_out_kernel(const float* __restrict__ before, const float* __restrict__ faded, float* __restrict__ o,
                     const int32_t* __restrict__ tile_tok0, const int32_t* __restrict__ tile_ntok, int H, int K) {
  extern __shared__ __align__(16) float sc_smem[];
  const int P = chunk_pitch(K), tile = blockIdx.x, h = blockIdx.y, tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  float* fs = sc_smem;                       // [CHUNK][P]
  float* ss = fs + CHUNK * P;                // S0 [j][P]
  chunk_rows(fs, P, faded + ((size_t)tile * H + h) * CHUNK * K, K, CHUNK, ntok, K);
  chunk_rows(ss, P, before + ((size_t)tile * H + h) * K * K, K, K, K, K);
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  double acc[4][4];
  chunk_mm_runs<16, 4, 4>(acc, fs, P, CHUNK, ss, P, K, K);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int t = chunk_ty() + 16 * a, j = chunk_tx() + 16 * b;
      if (t >= ntok || j >= K) continue;
      float* out = o + (size_t)(tok0 + t) * H * K + (size_t)h * K + j;
      *out = (float)(*out + acc[a][b]);
    }
}

}  // namespace edgelm

using namespace edgelm;

// 1 if the chunked forms take heads of these sizes.
extern "C" int edgelm_ssm_chunked_takes(int N, int P) { return N >= 4 && N <= 128 && N % 4 == 0 && P >= 4 && P <= 64 && P % 4 == 0 ? 1 : 0; }
extern "C" int edgelm_wkv_chunked_takes(int K) { return K >= 4 && K <= WK && K % 4 == 0 ? 1 : 0; }

// The recurrence of `edgelm_ssm_scan` over tiles: the raw step sizes at u[t][dt_off + h].  (The tail of the convolution ahead stays as it is.)
// scratch: n_tiles times H P N, G CHUNK (CHUNK + N) and H (in fours) floats.
extern "C" int edgelm_ssm_chunked(const float* xbc, int C, int inner, int G, int N, const float* u, int ldu, int dt_off, const float* dt_bias,
                                  const float* A_log, const float* D, float* state, float* y, const int32_t* seq_tok0, const int32_t* seq_slot, int n_seqs,
                                  const int32_t* tile_tok0, const int32_t* tile_ntok, int n_tiles, int H, int P, float* scratch,
                                  cudaStream_t stream) {
  if (n_seqs == 0 || n_tiles == 0) return 0;
  EL_REFUSE(n_seqs > 0 && n_tiles > 0 && H > 0 && H <= 65535 && G > 0 && H % G == 0 && inner == H * P && C == inner + 2 * G * N, "ssm_chunked: sizes do not fit (heads %d over %d, %d x %d, channels %d)", H, G, N, P, C);
  EL_REFUSE(edgelm_ssm_chunked_takes(N, P), "ssm_chunked: a state of %d x %d a head is not taken (use the scan)", N, P);
  EL_REFUSE(scratch != nullptr && (uintptr_t)scratch % 16 == 0 && (uintptr_t)xbc % 16 == 0, "ssm_chunked: rows and scratch must be 16-byte aligned");
  EL_REFUSE(dt_off >= 0 && dt_off + H <= ldu, "ssm_chunked: rows of %d values are too short", ldu);
  const float* dt_raw = u + dt_off;
  float* sums = scratch;
  float* shared_part = sums + (size_t)n_tiles * H * P * N;
  float* keep = shared_part + (size_t)n_tiles * G * (CHUNK * CHUNK + (size_t)CHUNK * N);
  const int NP = chunk_pitch(N);
  const size_t smem1 = (size_t)2 * CHUNK * NP * 4, smem2 = (size_t)(P + N) * SC_PITCH * 4;
  const size_t smem4 = (size_t)(CHUNK * NP + P * NP + CHUNK * SC_PITCH + P * SC_PITCH) * 4;
  auto k2 = N <= 64 ? ssm_chunk_state_kernel<4> : ssm_chunk_state_kernel<8>;
  cudaError_t err = cudaFuncSetAttribute(ssm_chunk_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(ssm_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem4);
  EL_REFUSE(err == cudaSuccess, "ssm_chunked: shared memory refused: %s", cudaGetErrorString(err));
  ssm_chunk_scores_kernel<<<dim3(n_tiles, G), 256, smem1, stream>>>(xbc, C, inner, shared_part, tile_tok0, tile_ntok, G, N);
  EL_LAUNCH_CHECK("ssm_chunk_scores");
  k2<<<dim3(n_tiles, H), 256, smem2, stream>>>(xbc, C, dt_raw, ldu, dt_bias, A_log, shared_part, sums, keep, tile_tok0, tile_ntok, H, G, N, P);
  EL_LAUNCH_CHECK("ssm_chunk_state");
  chunk_fold_kernel<<<dim3(n_seqs * H, (P * N + 127) / 128), 128, 0, stream>>>(sums, keep, state, seq_tok0, seq_slot, H, P * N, 1);
  EL_LAUNCH_CHECK("ssm_chunk_fold");
  ssm_chunk_out_kernel<<<dim3(n_tiles, H), 256, smem4, stream>>>(xbc, C, inner, dt_raw, ldu, dt_bias, A_log, D, shared_part, sums, y, tile_tok0, tile_ntok, H, G, N, P);
  EL_LAUNCH_CHECK("ssm_chunk_out");
  return 0;
}

// The recurrence of `edgelm_wkv_scan` over tiles; scratch: n_tiles H K (K + CHUNK + 1) floats.
extern "C" int edgelm_wkv_chunked(const float* r, const float* k, const float* v, const float* w, const float* bonus, float* state, float* o,
                                  const int32_t* seq_tok0, const int32_t* seq_slot, int n_seqs, const int32_t* tile_tok0,
                                  const int32_t* tile_ntok, int n_tiles, int H, int K, float* scratch, cudaStream_t stream) {
  if (n_seqs == 0 || n_tiles == 0) return 0;
  EL_REFUSE(n_seqs > 0 && n_tiles > 0 && H > 0 && H <= 65535, "wkv_chunked: bad sizes");
  EL_REFUSE(edgelm_wkv_chunked_takes(K), "wkv_chunked: heads of %d are not taken (use the scan)", K);
  EL_REFUSE(scratch != nullptr && (uintptr_t)scratch % 16 == 0 && ((uintptr_t)r | (uintptr_t)k | (uintptr_t)v | (uintptr_t)w) % 16 == 0, "wkv_chunked: rows and scratch must be 16-byte aligned");
  float* sums = scratch;
  float* faded = sums + (size_t)n_tiles * H * K * K;
  float* keep = faded + (size_t)n_tiles * H * CHUNK * K;
  const size_t smem1 = (size_t)4 * CHUNK * WK * 4, smem3 = (size_t)(CHUNK + K) * chunk_pitch(K) * 4;
  cudaError_t err = cudaFuncSetAttribute(wkv_chunk_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
  EL_REFUSE(err == cudaSuccess, "wkv_chunked: shared memory refused: %s", cudaGetErrorString(err));
  wkv_chunk_local_kernel<<<dim3(n_tiles, H), WK_THREADS, smem1, stream>>>(r, k, v, w, bonus, sums, faded, keep, o, tile_tok0, tile_ntok, H, K);
  EL_LAUNCH_CHECK("wkv_chunk_local");
  chunk_fold_kernel<<<dim3(n_seqs * H, (K * K + 127) / 128), 128, 0, stream>>>(sums, keep, state, seq_tok0, seq_slot, H, K * K, K);
  EL_LAUNCH_CHECK("wkv_chunk_fold");
  wkv_chunk_out_kernel<<<dim3(n_tiles, H), 256, smem3, stream>>>(sums, faded, o, tile_tok0, tile_ntok, H, K);
  EL_LAUNCH_CHECK("wkv_chunk_out");
  return 0;
}
