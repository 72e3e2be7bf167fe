// Prompt steps: projections of many tokens through bias, filter over time, norm and rotation into queries and cache rows, for heads of
// whole runs of 32 dimensions.  A warp owns one unit (a query head, a key head, or as many value channels) of ROT_TOKENS consecutive
// tokens: lane l holds the dimensions l, l + 32, ... in registers, a rotation's partner lies in the same lane or a shuffle away, the
// filter's taps and inputs stay in registers from token to token, and the angles' sines and cosines are computed once a token and block.
// (A token a block, every element computing its own angle and reading its filter's inputs anew, took 271 us for 3,900 tokens of 16 heads
// of two maps of 64 with three taps; this 156; 2,048 tokens of 64 heads of 64 94 and 45.)  The projection is read once, queries and cache rows are written once: at 45 us
// about 1.1 TB/s, so what takes the time is a warp's chain of eight tokens and its instructions, not memory.
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
  if (n_tokens <= 64 || dk % 32 || dk > 128 || maps < 1 || dk % maps || (dk / maps) % 32 || rot > 128 || (G * dv) % dk || taps > 4) return false;
  const int half = rot / 2;
  return rot == 0 || interleaved || half % 32 == 0 || (half < 32 && (half & (half - 1)) == 0);
}

template <typename T, typename TQ, int M>      // M = dk / 32
__global__ void __launch_bounds__(ROT_WARPS * 32)
rotate_rows_kernel(const RotateRows a, TQ* __restrict__ q_out, T* __restrict__ kcache, T* __restrict__ vcache) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float2 turn[ROT_TOKENS][64];
  __shared__ int place[ROT_TOKENS], seq[ROT_TOKENS];      // page * PAGE + row of a token (-1: none)
  const int t0 = blockIdx.x * ROT_TOKENS, nt = min(ROT_TOKENS, a.n_tokens - t0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = a.rot >> 1;
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
  constexpr int DK = 32 * M;
  const int unit = blockIdx.y * ROT_WARPS + warp, n_units = a.H + a.G + a.G * a.dv / DK;
  if (unit >= n_units) return;
  const bool value = unit >= a.H + a.G;
  const int ch0 = unit * DK + lane, C = (a.H + a.G) * DK + a.G * a.dv, ds = DK / a.maps;
  float in[ROT_TOKENS][M], ib[M];
#pragma unroll
  for (int m = 0; m < M; ++m) ib[m] = a.bias ? a.bias[ch0 + 32 * m] : 0.f;
#pragma unroll
  for (int x = 0; x < ROT_TOKENS; ++x)
#pragma unroll
    for (int m = 0; m < M; ++m) in[x][m] = (x < nt ? a.qkv[(size_t)(t0 + x) * a.ldq + ch0 + 32 * m] : 0.f) + ib[m];
  if (a.conv_w) {
    float w[M][4], past[M][3];                 // (aligned to the end: the last tap is [3], the token before [2])
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j) w[m][j] = j >= 4 - a.taps ? a.conv_w[(size_t)(ch0 + 32 * m) * a.taps + j - (4 - a.taps)] : 0.f;
#pragma unroll
    for (int x = 0; x < ROT_TOKENS; ++x) {
      if (x >= nt) break;
      const int s = seq[x], k = t0 + x - a.seq_tok0[s];
      if (x == 0 || k == 0) {                  // the inputs before this token: rows of the step, or the sequence's tail
        const float* tail = a.conv_state + (size_t)a.seq_slot[s] * (a.taps - 1) * C;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int r = k - 3 + j, row = a.taps - 1 + r;
#pragma unroll
          for (int m = 0; m < M; ++m)
            past[m][j] = j < 4 - a.taps ? 0.f : r >= 0 ? a.qkv[(size_t)(t0 + x - k + r) * a.ldq + ch0 + 32 * m] + ib[m]
                                : (row >= 0 ? tail[(size_t)row * C + ch0 + 32 * m] : 0.f);
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
    for (int m = 0; m < M; ++m) {
      const int i = ch0 + 32 * m - (a.H + a.G) * DK, g = i / a.dv, j = i - g * a.dv;
#pragma unroll
      for (int x = 0; x < ROT_TOKENS; ++x)
        if (x < nt && place[x] >= 0) vcache[(((size_t)(place[x] / PAGE) * a.G + g) * PAGE + place[x] % PAGE) * a.dv + j] = from_f32<T>(in[x][m]);
    }
    return;
  }
  const float* nw = unit < a.H ? a.q_norm : a.k_norm;
  float nwm[M];
#pragma unroll
  for (int m = 0; m < M; ++m) nwm[m] = nw ? nw[lane + 32 * m % ds] : 1.f;
#pragma unroll
  for (int x = 0; x < ROT_TOKENS; ++x) {
    if (x >= nt || place[x] < 0) continue;
    float v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = in[x][m];
    if (nw) {
      float ss[M];                             // a map's sum of squares, then its factor, at each of its runs
#pragma unroll
      for (int m = 0; m < M; ++m) ss[m] = v[m] * v[m];
#pragma unroll
      for (int m = 1; m < M; ++m)
        if (32 * m % ds != 0) ss[m] += ss[m - 1];
#pragma unroll
      for (int m = M - 2; m >= 0; --m)
        if (32 * (m + 1) % ds != 0) ss[m] = ss[m + 1];
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (32 * m % ds == 0) ss[m] = 1.0f / sqrtf(warp_sum(ss[m]) / (float)ds + a.eps);
        else ss[m] = ss[m - 1];
#pragma unroll
      for (int m = 0; m < M; ++m) v[m] = v[m] * ss[m] * nwm[m];
    }
    if (a.rot) {
      float out[M];
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int j = lane + 32 * m % ds;      // dimension inside its map
        // the partner: the other of a neighbouring pair, half a rotation away in this lane, or in another
        float other;
        int at;
        bool first;
        if (a.interleaved) {
          other = __shfl_xor_sync(0xffffffffu, v[m], 1);
          at = j >> 1;
          first = (j & 1) == 0;
        } else {
          first = j < half;
          at = first ? j : j - half;
          if (half >= 32) {
            other = 0.f;
#pragma unroll
            for (int p = 0; p < M; ++p)
              if (p == (first ? m + half / 32 : m - half / 32)) other = v[p];
          } else {
            other = __shfl_xor_sync(0xffffffffu, v[m], half);
          }
        }
        out[m] = v[m];
        if (j < a.rot) {
          const float2 tr = turn[x][at];
          out[m] = first ? v[m] * tr.x - other * tr.y : v[m] * tr.x + other * tr.y;
        }
      }
#pragma unroll
      for (int m = 0; m < M; ++m) v[m] = out[m];
    }
    if (a.unit_norm) {
      float ss = 0.f;
#pragma unroll
      for (int m = 0; m < M; ++m) ss = fmaf(v[m], v[m], ss);
      const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)DK + a.eps);
#pragma unroll
      for (int m = 0; m < M; ++m) v[m] *= inv;
    }
    if (unit < a.H) {
      TQ* dst = q_out + ((size_t)(t0 + x) * a.H + unit) * DK + lane;
#pragma unroll
      for (int m = 0; m < M; ++m) dst[32 * m] = from_f32<TQ>(v[m]);
    } else {
      T* dst = kcache + (((size_t)(place[x] / PAGE) * a.G + unit - a.H) * PAGE + place[x] % PAGE) * DK + lane;
#pragma unroll
      for (int m = 0; m < M; ++m) dst[32 * m] = from_f32<T>(v[m]);
    }
  }
}

template <typename T, typename TQ>
inline void launch_rotate_rows(const RotateRows& a, int dk, TQ* q_out, T* kcache, T* vcache, cudaStream_t stream) {
  const dim3 grid((a.n_tokens + ROT_TOKENS - 1) / ROT_TOKENS, (a.H + a.G + a.G * a.dv / dk + ROT_WARPS - 1) / ROT_WARPS), block(ROT_WARPS * 32);
  if (dk == 32) rotate_rows_kernel<T, TQ, 1><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache);
  else if (dk == 64) rotate_rows_kernel<T, TQ, 2><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache);
  else if (dk == 96) rotate_rows_kernel<T, TQ, 3><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache);
  else rotate_rows_kernel<T, TQ, 4><<<grid, block, 0, stream>>>(a, q_out, kcache, vcache);
}

}  // namespace edgelm
