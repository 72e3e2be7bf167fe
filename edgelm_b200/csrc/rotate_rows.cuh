// Prompt steps: projections of many tokens through bias, filter over time, norm and rotation into queries and cache rows, for heads of
// whole runs of 32 dimensions.  A warp owns one unit (a query head, a key head, or as many value channels) of ROT_TOKENS consecutive
// tokens: lane l holds the run of dk / 32 dimensions from l dk / 32 on (one access of 8 or 16 bytes a token where rows are aligned to a
// run; a rotation's partner is one shuffle away, or in the lane), the filter's taps and inputs stay in registers from token to token, and the
// angles' sines and cosines are computed once a token and block, while the rows, the three in front and the taps are on their way.
// (A token a block, every element computing its own angle and reading its filter's inputs anew, took 271 us for 3,900 tokens of 16 heads
// of two maps of 64 with three taps; dimensions l, l + 32, ... a lane 171, runs 104: a norm's sum is 4 shuffles instead of 20, a
// partner needs no selection.  2,048 tokens of 64 heads of 64: 44 and 37.)  At 1.5 to 2.3 TB/s: angles, filter and norm
// are a fifth, a fifth and an eighth of the time (the longer case without them: 45 us, 3.5 TB/s), and 16 warps an SM what 127 registers leave room
// for; a loop over the tokens with three rows on their way holds more warps and takes 5 to 10 % longer.
#pragma once
#include "common.cuh"

namespace edgelm {

constexpr int ROT_TOKENS = 8, ROT_WARPS = 4;

struct RotateRows {
  const float* qkv;                // [tokens][q | k | v], row pitch ldq
  int ldq;
  const float* bias;               // or null
  const int32_t *tok_pos, *tok_seq, *page_table;
  int table_stride, n_pages, n_tokens, H, G, dv, maps, rot, interleaved;
  const double* freq;
  int* err;
  const float *q_norm, *k_norm;    // weights of the norm ahead of the rotation, or null
  float eps, mult;
  int unit_norm;                   // divide by the root mean square after the rotation
  const float* conv_w;             // [channels][taps], or null
  const float* conv_state;
  const int32_t *seq_tok0, *seq_slot;
  int taps;
};

// The blocks from which on it is ahead of a block a token and four heads: a warp's eight tokens are a chain of some 8 us (with three taps
// 11 to 15), whatever the step.  (A block a token
// and four heads against this: 9 heads of 64, 384 tokens, 336 blocks 7.2 and 8.1 us; 512 tokens, 448 blocks 8.3 and 8.2; 768 tokens, 672
// blocks 11.7 and 9.6; from 500 to 600 blocks 0.59 to 0.88 of the time over ten shapes of heads, 250 to 300 blocks 0.87 to 1.31.)
constexpr int ROT_BLOCKS = 450;

// whether the kernel takes these sizes (dk: what a head's queries and a key row hold, all maps)
inline bool rotate_rows_takes(int n_tokens, int H, int G, int dk, int dv, int maps, int rot, int interleaved, int taps) {
  if (dk < 1 || (long long)((n_tokens + ROT_TOKENS - 1) / ROT_TOKENS) * ((H + G + G * dv / dk + ROT_WARPS - 1) / ROT_WARPS) < ROT_BLOCKS) return false;
  if (n_tokens <= 64 || dk % 32 || dk > 128 || maps < 1 || dk % maps || (dk / maps) % 32 || (dk == 96 && maps > 1) || rot > 128 || (G * dv) % dk || taps > 4) return false;
  return true;
}

// M consecutive values from or to memory, in one access where `whole` says that they lie aligned to their size (M 2 or 4)
template <int M>
__device__ __forceinline__ void load_run(const float* p, bool whole, float* v) {
  if (M == 4 && whole) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[M > 1 ? 1 : 0] = x.y; v[M > 2 ? 2 : 0] = x.z; v[M > 3 ? 3 : 0] = x.w;
  } else if (M == 2 && whole) {
    const float2 x = *reinterpret_cast<const float2*>(p);
    v[0] = x.x; v[M > 1 ? 1 : 0] = x.y;
  } else {
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = p[m];
  }
}
template <int M, typename T>
__device__ __forceinline__ void store_run(T* p, bool whole, const float* v) {
  if (M == 4 && whole) store_piece(p, make_float4(v[0], v[M > 1 ? 1 : 0], v[M > 2 ? 2 : 0], v[M > 3 ? 3 : 0]));
  else if (M == 2 && whole && sizeof(T) == 4) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[M > 1 ? 1 : 0]);
  else if (M == 2 && whole) *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(v[0], v[M > 1 ? 1 : 0]);
  else {
#pragma unroll
    for (int m = 0; m < M; ++m) p[m] = from_f32<T>(v[m]);
  }
}

// Whole runs: bit 0 the projections' rows, bit 1 the queries, bit 2 the cache's rows are aligned to a run of M.
template <typename T, typename TQ, int M>      // M = dk / 32
__global__ void __launch_bounds__(ROT_WARPS * 32)
rotate_rows_kernel(const RotateRows a, TQ* __restrict__ q_out, T* __restrict__ kcache, T* __restrict__ vcache, int whole) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float2 turn[ROT_TOKENS][64];
  __shared__ int place[ROT_TOKENS], seq[ROT_TOKENS], first[ROT_TOKENS];      // page * PAGE + row of a token (-1: none); its sequence and that one's first row
  const int t0 = blockIdx.x * ROT_TOKENS, nt = min(ROT_TOKENS, a.n_tokens - t0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = a.rot >> 1;
  constexpr int DK = 32 * M;
  const int unit = blockIdx.y * ROT_WARPS + warp, n_units = a.H + a.G + a.G * a.dv / DK;
  const int ch0 = unit * DK + lane * M, C = (a.H + a.G) * DK + a.G * a.dv, ds = DK / a.maps;
  const bool value = unit >= a.H + a.G, busy = unit < n_units;
  const float* nw = value ? nullptr : unit < a.H ? a.q_norm : a.k_norm;
  const int j0 = lane * M % ds, lanes = 32 / a.maps;      // this lane's first dimension inside its map; lanes of a map
  // (all that memory gives is on its way while the angles are computed: rows, the three rows in front, taps, weights)
  float in[ROT_TOKENS][M] = {}, ib[M] = {}, past[M][3] = {}, w[M][4] = {}, nwm[M];
  if (busy) {
#pragma unroll
    for (int x = 0; x < ROT_TOKENS; ++x)
      if (x < nt) load_run<M>(a.qkv + (size_t)(t0 + x) * a.ldq + ch0, whole & 1, in[x]);
    if (a.conv_w) {
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j >= 4 - a.taps && t0 - 3 + j >= 0) {
          float v[M];
          load_run<M>(a.qkv + (size_t)(t0 - 3 + j) * a.ldq + ch0, whole & 1, v);
#pragma unroll
          for (int m = 0; m < M; ++m) past[m][j] = v[m];
        }
#pragma unroll
      for (int m = 0; m < M; ++m)              // (aligned to the end: the last tap is [3], the token before [2])
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j >= 4 - a.taps) w[m][j] = a.conv_w[(size_t)(ch0 + m) * a.taps + j - (4 - a.taps)];
    }
    if (a.bias)
#pragma unroll
      for (int m = 0; m < M; ++m) ib[m] = a.bias[ch0 + m];
#pragma unroll
    for (int m = 0; m < M; ++m) nwm[m] = nw ? nw[j0 + m] : 1.f;
  }
  if (threadIdx.x < ROT_TOKENS) {
    const int t = t0 + threadIdx.x, pos = threadIdx.x < nt ? a.tok_pos[t] : -1, s = threadIdx.x < nt ? a.tok_seq[t] : 0;
    int at = -1;
    if (pos >= 0) {
      const int page = a.page_table[(size_t)s * a.table_stride + pos / PAGE];
      if (page >= 0 && page < a.n_pages) at = page * PAGE + pos % PAGE;
      else if (blockIdx.y == 0) atomicOr(a.err, ERR_PAGE_RANGE);
    } else if (threadIdx.x < nt && blockIdx.y == 0) {
      atomicOr(a.err, ERR_POSITION_RANGE);
    }
    place[threadIdx.x] = at;
    seq[threadIdx.x] = s;
    first[threadIdx.x] = a.conv_w && threadIdx.x < nt ? a.seq_tok0[s] : 0;
  }
  for (int i = threadIdx.x; i < nt * half; i += ROT_WARPS * 32) {
    const int x = i / half, j = i - x * half;
    double ang = (double)max(a.tok_pos[t0 + x], 0) * a.freq[j];      // (formed exactly and brought into [-pi, pi] before float32)
    ang -= 6.283185307179586477 * rint(ang * 0.15915494309189533577);
    float sn, cs;
    sincosf((float)ang, &sn, &cs);
    turn[x][j] = make_float2(cs * a.mult, sn * a.mult);
  }
  __syncthreads();
  if (!busy) return;
  // half a rotation away: in the lane `half / M` further, or (half no whole run: M 3, or fewer than a run) a dimension of some lane's
  const bool whole_lanes = half % M == 0, front = j0 < half;
  const int away = front ? lane + half / M : lane - half / M;
  const int vi = ch0 - (a.H + a.G) * DK, vg = vi / a.dv, vj = vi - vg * a.dv;      // (value channels: their head and place in it)
#pragma unroll
  for (int x = 0; x < ROT_TOKENS; ++x)
#pragma unroll
    for (int m = 0; m < M; ++m) in[x][m] += ib[m];
  if (a.conv_w) {
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int j = 0; j < 3; ++j) past[m][j] = j >= 4 - a.taps ? past[m][j] + ib[m] : 0.f;
#pragma unroll
    for (int x = 0; x < ROT_TOKENS; ++x) {
      if (x >= nt) break;
      const int s = seq[x], k = t0 + x - first[x];
      if (x == 0 ? k < 3 : k == 0) {           // the inputs before this token that are no rows of the step: the sequence's tail
        const float* tail = a.conv_state + (size_t)a.seq_slot[s] * (a.taps - 1) * C;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int r = k - 3 + j, row = a.taps - 1 + r;
          if (r < 0 && j >= 4 - a.taps)
#pragma unroll
            for (int m = 0; m < M; ++m) past[m][j] = row >= 0 ? tail[(size_t)row * C + ch0 + m] : 0.f;
        }
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const float now = in[x][m];
        in[x][m] = fmaf(w[m][3], now, fmaf(w[m][2], past[m][2], fmaf(w[m][1], past[m][1], w[m][0] * past[m][0])));
        past[m][0] = a.taps > 3 ? past[m][1] : 0.f;      // (inputs in front of the filter count as zeros: 0 times an infinity is none)
        past[m][1] = a.taps > 2 ? past[m][2] : 0.f;
        past[m][2] = a.taps > 1 ? now : 0.f;
      }
    }
  }
  if (value) {
#pragma unroll
    for (int x = 0; x < ROT_TOKENS; ++x) {
      if (x >= nt || place[x] < 0) continue;
      T* rows = vcache + ((size_t)(place[x] / PAGE) * a.G * PAGE + place[x] % PAGE) * a.dv;
      if (a.dv % M == 0) {                     // a lane's run lies in one head's values
        store_run<M>(rows + (size_t)vg * PAGE * a.dv + vj, whole & 4, in[x]);
      } else {
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const int g = (vi + m) / a.dv;
          rows[(size_t)g * PAGE * a.dv + vi + m - g * a.dv] = from_f32<T>(in[x][m]);
        }
      }
    }
    return;
  }
#pragma unroll
  for (int x = 0; x < ROT_TOKENS; ++x) {
    float v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = in[x][m];
    if (nw) {
      float ss = 0.f;
#pragma unroll
      for (int m = 0; m < M; ++m) ss = fmaf(v[m], v[m], ss);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
        if (o < lanes) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float inv = 1.0f / sqrtf(ss / (float)ds + a.eps);
#pragma unroll
      for (int m = 0; m < M; ++m) v[m] = v[m] * inv * nwm[m];
    }
    if (a.rot) {
      float other[M];
      if (a.interleaved && M % 2 == 0) {       // the other of a neighbouring pair lies in this lane
#pragma unroll
        for (int m = 0; m < M; ++m) other[m] = v[m ^ (M > 1)];
      } else if (!a.interleaved && whole_lanes) {
#pragma unroll
        for (int m = 0; m < M; ++m) other[m] = __shfl_sync(0xffffffffu, v[m], away & 31);
      } else {
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const int j = j0 + m, p = a.interleaved ? j ^ 1 : j < half ? j + half : j - half, d = lane * M - j0 + p;
          other[m] = 0.f;
#pragma unroll
          for (int e = 0; e < M; ++e) {
            const float got = __shfl_sync(0xffffffffu, v[e], d / M);
            if (d % M == e) other[m] = got;
          }
        }
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int j = j0 + m;
        if (j < a.rot) {
          const bool first_of = a.interleaved ? (j & 1) == 0 : j < half;
          const float2 tr = turn[x][a.interleaved ? j >> 1 : j < half ? j : j - half];
          v[m] = first_of ? v[m] * tr.x - other[m] * tr.y : v[m] * tr.x + other[m] * tr.y;
        }
      }
    }
    if (a.unit_norm) {
      float ss = 0.f;
#pragma unroll
      for (int m = 0; m < M; ++m) ss = fmaf(v[m], v[m], ss);
      const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)DK + a.eps);
#pragma unroll
      for (int m = 0; m < M; ++m) v[m] *= inv;
    }
    // (rows without a place are computed like the others, so that the tokens' chains interleave, and not stored)
    if (x >= nt || place[x] < 0) continue;
    if (unit < a.H) store_run<M>(q_out + ((size_t)(t0 + x) * a.H + unit) * DK + lane * M, whole & 2, v);
    else store_run<M>(kcache + (((size_t)(place[x] / PAGE) * a.G + unit - a.H) * PAGE + place[x] % PAGE) * DK + lane * M, whole & 4, v);
  }
}

template <typename T, typename TQ>
inline void launch_rotate_rows(const RotateRows& a, int dk, TQ* q_out, T* kcache, T* vcache, cudaStream_t stream) {
  const dim3 grid((a.n_tokens + ROT_TOKENS - 1) / ROT_TOKENS, (a.H + a.G + a.G * a.dv / dk + ROT_WARPS - 1) / ROT_WARPS), block(ROT_WARPS * 32);
  const auto aligned = [&](const void* p, size_t row, size_t item) { return (uintptr_t)p % (item * (dk / 32)) == 0 && row % (dk / 32) == 0; };
  const int whole = (aligned(a.qkv, a.ldq, 4) ? 1 : 0) | (aligned(q_out, dk, sizeof(TQ)) ? 2 : 0) |
                    (aligned(kcache, dk, sizeof(T)) && aligned(vcache, a.dv, sizeof(T)) ? 4 : 0);
  if (dk == 32) rotate_rows_kernel<T, TQ, 1><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache, whole);
  else if (dk == 64) rotate_rows_kernel<T, TQ, 2><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache, whole);
  else if (dk == 96) rotate_rows_kernel<T, TQ, 3><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache, whole);
  else rotate_rows_kernel<T, TQ, 4><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache, whole);
}

}  // namespace edgelm
