// Sliding-window attention with pooled blocks behind the window, over the paged cache.
//
// A token at position i sees the keys j with 0 <= i - j < window, and one pooled key and value per block of P
// consecutive positions that lies wholly before the window (block b = positions bP .. bP + P - 1 is seen iff
// bP + P - 1 <= i - window).  A pooled key (value) is the mean of the block's P keys (values) as the cache holds
// them.  Tokens and blocks share one softmax.
//
// Cache layout: keys [page][kv_head][PAGE][dk], values [page][kv_head][PAGE][dv] in the compute type, as the other
// attention kernels keep them; pooled keys and values in float32, [page][kv_head][R][dk or dv], where a block's
// row lives in the page that holds the block's LAST position e = bP + P - 1: page e / PAGE, row b - (PAGE * (e / PAGE)) / P
// (R = ceil(PAGE / P) rows a page are enough: that many block ends fall into one page at most).
//
// Three kernels: (1) bias, partial rotation, per-head unit RMS norm of q and k, append of k and v; (2) the pooled
// rows of the blocks that the step's tokens complete; (3) attention.  Scores, softmax, norms, angles: float32.
#include "mma_split.cuh"
#include "rotate_rows.cuh"

namespace edgelm {

constexpr int PW_WARPS = 4;

// qkv: [tokens][H dk + G dk + G dv] float32 (the stacked projection), biases float32 (may be null).
// The first `rot` dimensions of each query and key head are rotated: (u, v) = (x[i], x[i + rot/2]) becomes
// (u cos a - v sin a, v cos a + u sin a), a = position * freq[i]; then the head is divided by its root mean square.
template <typename T>
__global__ void __launch_bounds__(PW_WARPS * 32)
qk_rope_norm_append_kernel(const float* __restrict__ qkv, const float* __restrict__ bias, T* __restrict__ q_out,
                           const int32_t* __restrict__ tok_pos, const int32_t* __restrict__ tok_seq,
                           const int32_t* __restrict__ page_table, int table_stride, int n_pages, T* __restrict__ kcache,
                           T* __restrict__ vcache, int H, int G, int dk, int dv, int rot, const double* __restrict__ freq,
                           float eps, int unit_norm, int* __restrict__ err) {
  pdl_launch_dependents();
  pdl_wait();   // (launched as a programmatic dependent: nothing is read or written before the kernel ahead is done)
  extern __shared__ float stage[];   // PW_WARPS rows of dk floats
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pos = tok_pos[t];
  if (pos < 0) {
    if (threadIdx.x == 0 && blockIdx.y == 0) atomicOr(err, ERR_POSITION_RANGE);
    return;
  }
  const int page = page_table[(size_t)tok_seq[t] * table_stride + pos / PAGE];
  if (page < 0 || page >= n_pages) {
    if (threadIdx.x == 0 && blockIdx.y == 0) atomicOr(err, ERR_PAGE_RANGE);
    return;
  }
  const int in_page = pos % PAGE, half = rot >> 1;
  const int ld = H * dk + G * dk + G * dv;
  const float* row = qkv + (size_t)t * ld;
  float* sh = stage + warp * dk;
  const double dpos = (double)pos;
  // a warp a head (query heads, then key heads); the blocks of a token stand side by side over the heads
  for (int head = blockIdx.y * PW_WARPS + warp; head < H + G; head += gridDim.y * PW_WARPS) {
    const float* src = row + (size_t)head * dk;
    const float* b = bias ? bias + (size_t)head * dk : nullptr;
    for (int i = lane; i < dk; i += 32) sh[i] = src[i] + (b ? b[i] : 0.f);
    __syncwarp();
    float ss = 0.f;
    float val[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int i = lane + 32 * m;
      float x = 0.f;
      if (i < dk) {
        x = sh[i];
        if (i < rot) {
          const int f = i < half ? i : i - half;
          // the angle position * f is formed exactly and brought into [-pi, pi] before it is rounded to float32: at
          // position 1,000 a float32 product alone is off by up to 3e-5 rad, which is most of a float32 model's error
          double a = dpos * freq[f];
          a -= 6.283185307179586477 * rint(a * 0.15915494309189533577);
          float sn, cs;
          sincosf((float)a, &sn, &cs);
          x = i < half ? sh[i] * cs - sh[i + half] * sn : sh[i] * cs + sh[i - half] * sn;
        }
      }
      val[m] = x;
      ss = fmaf(x, x, ss);
    }
    ss = warp_sum(ss);
    const float inv = unit_norm ? 1.0f / sqrtf(ss / (float)dk + eps) : 1.0f;
    T* dst = head < H ? q_out + ((size_t)t * H + head) * dk : kcache + (((size_t)page * G + (head - H)) * PAGE + in_page) * dk;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int i = lane + 32 * m;
      if (i < dk) dst[i] = from_f32<T>(val[m] * inv);
    }
    __syncwarp();
  }
  const float* vrow = row + (size_t)(H + G) * dk;
  const float* vb = bias ? bias + (size_t)(H + G) * dk : nullptr;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < G * dv; i += gridDim.y * blockDim.x) {
    const int g = i / dv, j = i - g * dv;
    vcache[(((size_t)page * G + g) * PAGE + in_page) * dv + j] = from_f32<T>(vrow[i] + (vb ? vb[i] : 0.f));
  }
}

// The pooled rows of the blocks that end at a token of this step.  A block of threads looks at `run` consecutive tokens, a lane a token; in
// prompt steps as many as a block has, up to POOL_RUN, so that there is about one pooled row to a block of threads and few find nothing to
// do.  (A token a block, 16 a block and so many: 2,048 tokens, 32 heads, blocks of 64 82, 37 and 29 us, blocks of 4 69, 32 and 25; two heads,
// blocks of 4 5.6, 9.8 and 3.9; 65 tokens, blocks of 4 3.2, 9.4 and 3.3.)
constexpr int POOL_RUN = 16;

template <typename T>
__global__ void pool_blocks_kernel(const int32_t* __restrict__ tok_pos, const int32_t* __restrict__ tok_seq,
                                   const int32_t* __restrict__ page_table, int table_stride, int n_pages,
                                   const T* __restrict__ kcache, const T* __restrict__ vcache, float* __restrict__ pk,
                                   float* __restrict__ pv, int G, int dk, int dv, int P, int R, int* __restrict__ err, int n_tokens, int run) {
  pdl_launch_dependents();
  pdl_wait();   // (launched as a programmatic dependent: nothing is read or written before the kernel ahead is done)
  const int t0 = blockIdx.x * run, lane = threadIdx.x & 31;
  const int mine = lane < run && t0 + lane < n_tokens ? tok_pos[t0 + lane] : -1;
  for (unsigned ends = __ballot_sync(0xffffffffu, mine >= 0 && (mine + 1) % P == 0); ends != 0; ends &= ends - 1) {
    const int x = __ffs(ends) - 1, t = t0 + x, pos = __shfl_sync(0xffffffffu, mine, x);
    const int b = (pos + 1) / P - 1;
    const int32_t* table = page_table + (size_t)tok_seq[t] * table_stride;
    const int dst_page = table[pos / PAGE];
    if (dst_page < 0 || dst_page >= n_pages) {
      if (threadIdx.x == 0 && blockIdx.y == 0) atomicOr(err, ERR_PAGE_RANGE);
      continue;
    }
    const int rowi = b - (PAGE * (pos / PAGE)) / P;
    const float invP = 1.0f / (float)P;
    // a block per (token that ends a block, key/value head); a thread a channel of the key, then of the value: the rows
    // of a block lie side by side in a page, so neighbouring threads read neighbouring addresses, eight rows in flight
    const int g = blockIdx.y;
    for (int i = threadIdx.x; i < dk + dv; i += blockDim.x) {
      const bool is_k = i < dk;
      const int d = is_k ? dk : dv, c = is_k ? i : i - dk;
      const T* base = is_k ? kcache : vcache;
      float acc = 0.f;
#pragma unroll 8
      for (int j = 0; j < P; ++j) {
        const int p = b * P + j;
        const int page = table[p / PAGE];
        if (page < 0 || page >= n_pages) continue;   // (flagged by the append of that token's step)
        acc += to_f32(base[(((size_t)page * G + g) * PAGE + p % PAGE) * d + c]);
      }
      float* dst = is_k ? pk : pv;
      dst[(((size_t)dst_page * G + g) * R + rowi) * d + c] = acc * invP;
    }
  }
}

// ---- the attention kernel
// A block per (token, query head); its NW warps take the keys in turns of 32 (a lane a key: pooled blocks first, then
// the window's tokens), each with its own running maximum, denominator and weighted values (float32), merged at the end
// through shared memory.  A lane reads its key 16 bytes at a time where the layout allows; for the weighted values the
// lanes stand side by side over the value's dimensions, two each.

// q . k over n dimensions, q float32 in shared memory; four running sums.
template <typename TK>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const TK* __restrict__ k, int n, bool vec);

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ q, const float* __restrict__ k, int n, bool vec) {
  float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  int i = 0;
  if (vec) {
    for (; i + 4 <= n; i += 4) {
      const float4 kv = *reinterpret_cast<const float4*>(k + i);
      const float4 qv = *reinterpret_cast<const float4*>(q + i);
      a0 = fmaf(qv.x, kv.x, a0); a1 = fmaf(qv.y, kv.y, a1); a2 = fmaf(qv.z, kv.z, a2); a3 = fmaf(qv.w, kv.w, a3);
    }
  }
  for (; i < n; ++i) a0 = fmaf(q[i], k[i], a0);
  return (a0 + a1) + (a2 + a3);
}

template <>
__device__ __forceinline__ float dot_row<__nv_bfloat16>(const float* __restrict__ q, const __nv_bfloat16* __restrict__ k, int n, bool vec) {
  float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  int i = 0;
  if (vec) {
    for (; i + 8 <= n; i += 8) {
      const uint4 kv = *reinterpret_cast<const uint4*>(k + i);
      const float4 q0 = *reinterpret_cast<const float4*>(q + i), q1 = *reinterpret_cast<const float4*>(q + i + 4);
      a0 = fmaf(q0.x, __uint_as_float(kv.x << 16), a0); a1 = fmaf(q0.y, __uint_as_float(kv.x & 0xffff0000u), a1);
      a2 = fmaf(q0.z, __uint_as_float(kv.y << 16), a2); a3 = fmaf(q0.w, __uint_as_float(kv.y & 0xffff0000u), a3);
      a0 = fmaf(q1.x, __uint_as_float(kv.z << 16), a0); a1 = fmaf(q1.y, __uint_as_float(kv.z & 0xffff0000u), a1);
      a2 = fmaf(q1.z, __uint_as_float(kv.w << 16), a2); a3 = fmaf(q1.w, __uint_as_float(kv.w & 0xffff0000u), a3);
    }
  }
  for (; i < n; ++i) a0 = fmaf(q[i], __bfloat162float(k[i]), a0);
  return (a0 + a1) + (a2 + a3);
}

// two neighbouring values of a row
__device__ __forceinline__ float2 load_pair(const float* p, bool pair) {
  return pair ? *reinterpret_cast<const float2*>(p) : make_float2(p[0], 0.f);
}
__device__ __forceinline__ float2 load_pair(const __nv_bfloat16* p, bool pair) {
  if (!pair) return make_float2(__bfloat162float(p[0]), 0.f);
  const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

constexpr int PW_MAX_WARPS = 8;

// Dynamic shared memory: the query (dk floats, 16-byte aligned), then per warp its maximum, its denominator and dv values.
// This one takes key and value heads of any sizes; those of 32, 64 or 128 dimensions alike go to the kernel of whole rows below, where a load
// instruction of a warp covers whole rows.  (For 2,048 tokens at once, 32 heads, window 1,024, that costs more in shuffles than it saves in loads, 5.2
// ms against 3.8; single tokens wait for memory, and prompt steps have kernels of their own.)
// DVR: how many pairs of value dimensions a lane holds (value heads of up to 64 DVR dimensions).
template <typename T, int DVR>
__global__ void __launch_bounds__(PW_MAX_WARPS * 32)
pooled_window_attn_kernel(const T* __restrict__ q, T* __restrict__ out, const T* __restrict__ kcache, const T* __restrict__ vcache,
                          const float* __restrict__ pk, const float* __restrict__ pv, const int32_t* __restrict__ tok_pos,
                          const int32_t* __restrict__ tok_seq, const int32_t* __restrict__ page_table, int table_stride,
                          int n_pages, int H, int G, int dk, int dv, float scale, int window, int P, int R, int vec_k, int pair_v) {
  pdl_launch_dependents();
  pdl_wait();   // (launched as a programmatic dependent: nothing is read or written before the kernel ahead is done)
  extern __shared__ __align__(16) float smem[];
  const int t = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
  const int dkp = (dk + 3) & ~3;
  float* qh = smem;
  float* wm = smem + dkp;          // [NW] maxima
  float* wl = wm + NW;             // [NW] denominators
  float* wo = wl + NW;             // [NW][dv]
  const int pos = tok_pos[t];
  if (pos < 0) return;
  const int g = h / (H / G);
  const int32_t* table = page_table + (size_t)tok_seq[t] * table_stride;
  const T* qrow = q + ((size_t)t * H + h) * dk;
  for (int i = threadIdx.x; i < dk; i += blockDim.x) qh[i] = to_f32(qrow[i]) * scale;
  __syncthreads();
  const int lo = max(0, pos - window + 1), n_win = pos - lo + 1;
  const int n_blocks = (P > 0 && pos - window >= 0) ? (pos - window + 1) / P : 0;
  const int blk_chunks = (n_blocks + 31) >> 5, n_chunks = blk_chunks + ((n_win + 31) >> 5);
  float m = -INFINITY, l = 0.f;
  bool nan = false;                // some key of this warp's scored not a number
  float o[2 * DVR];                // dimensions 2 lane + 64 r and the one after it
#pragma unroll
  for (int r = 0; r < 2 * DVR; ++r) o[r] = 0.f;
  for (int c = warp; c < n_chunks; c += NW) {
    const bool pooled = c < blk_chunks;
    const int e0 = pooled ? c * 32 : (c - blk_chunks) * 32;
    const int n_here = min(32, (pooled ? n_blocks : n_win) - e0);
    float sc = -INFINITY;
    int vrow = -1;                 // this lane's key: the row of its value
    if (lane < n_here) {
      if (pooled) {
        const int e = e0 + lane, end = e * P + P - 1;
        const int page = table[end / PAGE];
        if (page >= 0 && page < n_pages) {
          vrow = (page * G + g) * R + (e - (PAGE * (end / PAGE)) / P);
          sc = dot_row<float>(qh, pk + (size_t)vrow * dk, dk, (dk & 3) == 0);
        }
      } else {
        const int p = lo + e0 + lane;
        const int page = table[p / PAGE];
        if (page >= 0 && page < n_pages) {
          vrow = (page * G + g) * PAGE + p % PAGE;
          sc = dot_row<T>(qh, kcache + (size_t)vrow * dk, dk, vec_k != 0);
        }
      }
    }
    const float m_new = fmaxf(m, warp_max(sc));
    nan = nan || __any_sync(0xffffffffu, sc != sc);     // (a maximum drops it)
    if (m_new == -INFINITY) continue;
    const float w = sc == -INFINITY ? 0.f : expf(sc - m_new);
    const float corr = m == -INFINITY ? 0.f : expf(m - m_new);
    l = l * corr + warp_sum(w);
    m = m_new;
#pragma unroll
    for (int r = 0; r < 2 * DVR; ++r) o[r] *= corr;
    if (pooled) {
      const bool pair = (dv & 1) == 0;
      for (int j = 0; j < n_here; ++j) {
        const float wj = __shfl_sync(0xffffffffu, w, j);
        const int vr_i = __shfl_sync(0xffffffffu, vrow, j);
        if (vr_i < 0) continue;
        const float* vr = pv + (size_t)vr_i * dv;
#pragma unroll
        for (int r = 0; r < DVR; ++r) {
          const int d = 2 * lane + 64 * r;
          if (d < dv) {
            const float2 x = load_pair(vr + d, pair);
            o[2 * r] = fmaf(wj, x.x, o[2 * r]);
            if (d + 1 < dv) o[2 * r + 1] = fmaf(wj, pair ? x.y : vr[d + 1], o[2 * r + 1]);
          }
        }
      }
    } else {
#pragma unroll 4
      for (int j = 0; j < n_here; ++j) {
        const float wj = __shfl_sync(0xffffffffu, w, j);
        const int vr_i = __shfl_sync(0xffffffffu, vrow, j);
        if (vr_i < 0) continue;
        const T* vr = vcache + (size_t)vr_i * dv;
#pragma unroll
        for (int r = 0; r < DVR; ++r) {
          const int d = 2 * lane + 64 * r;
          if (d < dv) {
            const float2 x = load_pair(vr + d, pair_v != 0);
            o[2 * r] = fmaf(wj, x.x, o[2 * r]);
            if (d + 1 < dv) o[2 * r + 1] = fmaf(wj, pair_v ? x.y : to_f32(vr[d + 1]), o[2 * r + 1]);
          }
        }
      }
    }
  }
  // merge the warps' partial results in a fixed order
  if (lane == 0) { wm[warp] = nan ? NAN : m; wl[warp] = l; }
#pragma unroll
  for (int r = 0; r < DVR; ++r) {
    const int d = 2 * lane + 64 * r;
    if (d < dv) wo[warp * dv + d] = o[2 * r];
    if (d + 1 < dv) wo[warp * dv + d + 1] = o[2 * r + 1];
  }
  __syncthreads();
  float M = -INFINITY;
  for (int w2 = 0; w2 < NW; ++w2) M = fmaxf(M, wm[w2]);
  float L = 0.f;
  for (int w2 = 0; w2 < NW; ++w2) L += wm[w2] == -INFINITY ? 0.f : wl[w2] * expf(wm[w2] - M);
  const float inv = L == 0.f ? 0.f : 1.0f / L;      // (0: no key was seen; a denominator that is not a number goes on)
  for (int d = threadIdx.x; d < dv; d += blockDim.x) {
    float acc = 0.f;
    for (int w2 = 0; w2 < NW; ++w2)
      if (wm[w2] != -INFINITY) acc = fmaf(wo[w2 * dv + d], expf(wm[w2] - M), acc);
    out[((size_t)t * H + h) * dv + d] = from_f32<T>(acc * inv);
  }
}

// The same for key and value heads of D dimensions alike, rows of whole 16-byte pieces: a load instruction of a warp covers 32 / LPR whole
// rows, and a warp's 32 keys and values (fewer of rows over 128 bytes) are requested together, before the first score is known.  (In the kernel above a
// lane reads a key by itself and the warp walks its values one after the other, a trip to memory or four keys at a time: 16 tokens of 9
// heads, window 512: 54 us.)  A warp takes a run of the window's keys and a run of the pooled rows (float32 rows: lanes of 4 dimensions),
// each with a maximum, a denominator and an output of its own; all are merged in order through shared memory.  Bound by four trips to
// memory in a chain (position, page, rows, merge), which is why a block has as many warps as keep a run at 32 keys where blocks are few.
template <typename T, int D>
struct PwRow {
  static constexpr int EPL = 16 / sizeof(T), LPR = D / EPL, RPI = 32 / LPR;      // elements a lane, lanes a row, rows an instruction
  static constexpr int ITS = RPI >= 4 ? 32 / RPI : 8, KEYS = ITS * RPI;                           // instructions in flight (8 at most), their rows
};
__device__ __forceinline__ void pw_unpack(const uint4& u, float* v, const float*) {
  v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
}
__device__ __forceinline__ void pw_unpack(const uint4& u, float* v, const __nv_bfloat16*) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
// A run of rows [begin, end) through one query: `row_of(r)` is the row's number in `keys` and `values` (-1: none).  A run with a score that
// is not a number has such a maximum: the merge hands it on (of the scores' maximum alone it would vanish where the run has no other score).
template <typename T, int D, typename RowOf>
__device__ __forceinline__ void pw_run(const T* __restrict__ keys, const T* __restrict__ values, const float* qh, int begin, int end, int lane, RowOf row_of,
                                       float& m, float& l, float* slot) {
  using R = PwRow<T, D>;
  const int part = lane % R::LPR, grp = lane / R::LPR;
  float qv[R::EPL], o[R::EPL] = {};
  bool nan = false;
#pragma unroll
  for (int e = 0; e < R::EPL; ++e) qv[e] = qh[part * R::EPL + e];
  for (int r0 = begin; r0 < end; r0 += R::KEYS) {
    uint4 kv[R::ITS], vv[R::ITS];
    bool there[R::ITS];
#pragma unroll
    for (int i = 0; i < R::ITS; ++i) {
      const int r = r0 + i * R::RPI + grp, row = r < end ? row_of(r) : -1;
      there[i] = row >= 0;
      kv[i] = there[i] ? *reinterpret_cast<const uint4*>(keys + (size_t)row * D + part * R::EPL) : make_uint4(0, 0, 0, 0);
      vv[i] = there[i] ? *reinterpret_cast<const uint4*>(values + (size_t)row * D + part * R::EPL) : make_uint4(0, 0, 0, 0);
    }
    float sc[R::ITS], m_new = m;
#pragma unroll
    for (int i = 0; i < R::ITS; ++i) {
      float k[R::EPL], d = 0.f;
      pw_unpack(kv[i], k, keys);
#pragma unroll
      for (int e = 0; e < R::EPL; ++e) d = fmaf(qv[e], k[e], d);
#pragma unroll
      for (int x = 1; x < R::LPR; x <<= 1) d += __shfl_xor_sync(0xffffffffu, d, x);
      sc[i] = there[i] ? d : -INFINITY;
      nan = nan || sc[i] != sc[i];
      m_new = fmaxf(m_new, sc[i]);
    }
    m_new = warp_max(m_new);
    if (m_new == -INFINITY) continue;
    const float corr = m == -INFINITY ? 0.f : expf(m - m_new);
    float sum = 0.f;
#pragma unroll
    for (int e = 0; e < R::EPL; ++e) o[e] *= corr;
#pragma unroll
    for (int i = 0; i < R::ITS; ++i) {
      if (!there[i]) continue;
      float v[R::EPL];
      const float w = expf(sc[i] - m_new);
      sum += w;
      pw_unpack(vv[i], v, values);
#pragma unroll
      for (int e = 0; e < R::EPL; ++e) o[e] = fmaf(w, v[e], o[e]);
    }
    l = l * corr + sum;                        // (this lane's rows)
    m = m_new;
  }
  if (__any_sync(0xffffffffu, nan)) m = NAN;
#pragma unroll
  for (int x = R::LPR; x < 32; x <<= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
    for (int e = 0; e < R::EPL; ++e) o[e] += __shfl_xor_sync(0xffffffffu, o[e], x);
  }
  if (grp == 0)
#pragma unroll
    for (int e = 0; e < R::EPL; ++e) slot[part * R::EPL + e] = o[e];
}

constexpr int PWR_MAX_WARPS = 16;
template <typename T, int D>
__global__ void __launch_bounds__(PWR_MAX_WARPS * 32)
pooled_window_attn_rows_kernel(const T* __restrict__ q, T* __restrict__ out, const T* __restrict__ kcache, const T* __restrict__ vcache,
                               const float* __restrict__ pk, const float* __restrict__ pv, const int32_t* __restrict__ tok_pos,
                               const int32_t* __restrict__ tok_seq, const int32_t* __restrict__ page_table, int table_stride,
                               int n_pages, int H, int G, float scale, int window, int P, int R) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float qh[D], wm[2 * PWR_MAX_WARPS], wl[2 * PWR_MAX_WARPS], wo[2 * PWR_MAX_WARPS][D];      // (a warp's window run, its pooled run)
  const int t = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
  const int pos = tok_pos[t];
  if (pos < 0) return;
  const int g = h / (H / G);
  const int32_t* table = page_table + (size_t)tok_seq[t] * table_stride;
  for (int i = threadIdx.x; i < D; i += blockDim.x) qh[i] = to_f32(q[((size_t)t * H + h) * D + i]) * scale;
  __syncthreads();
  const int lo = max(0, pos - window + 1), n_win = pos - lo + 1;
  const int n_blocks = (P > 0 && pos - window >= 0) ? (pos - window + 1) / P : 0;
  float m = -INFINITY, l = 0.f;
  pw_run<T, D>(kcache, vcache, qh, (int)((long long)n_win * warp / NW), (int)((long long)n_win * (warp + 1) / NW), lane, [&](int r) {
    const int p = lo + r, page = table[p / PAGE];
    return page >= 0 && page < n_pages ? (page * G + g) * PAGE + p % PAGE : -1;
  }, m, l, wo[2 * warp]);
  if (lane == 0) { wm[2 * warp] = m; wl[2 * warp] = l; }
  m = -INFINITY, l = 0.f;
  if (n_blocks)
    pw_run<float, D>(pk, pv, qh, n_blocks * warp / NW, n_blocks * (warp + 1) / NW, lane, [&](int e) {
      const int end = e * P + P - 1, page = table[end / PAGE];
      return page >= 0 && page < n_pages ? (page * G + g) * R + (e - (PAGE * (end / PAGE)) / P) : -1;
    }, m, l, wo[2 * warp + 1]);
  if (lane == 0) { wm[2 * warp + 1] = m; wl[2 * warp + 1] = l; }
  __syncthreads();
  if (threadIdx.x < D) {
    // (four sums side by side: one of up to 32 runs after the other rounds more often than the runs themselves)
    float M = -INFINITY, Ls[4] = {}, accs[4] = {};
    for (int w = 0; w < 2 * NW; ++w) M = fmaxf(M, wm[w]);
#pragma unroll 2
    for (int w0 = 0; w0 < 2 * NW; w0 += 4) {
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int w = min(w0 + x, 2 * NW - 1);
        const bool on = w0 + x < 2 * NW && wm[w] != -INFINITY;
        const float f = expf(wm[w] - M), l = fmaf(wl[w], f, Ls[x]), o = fmaf(wo[w][threadIdx.x], f, accs[x]);
        Ls[x] = on ? l : Ls[x];
        accs[x] = on ? o : accs[x];
      }
    }
    const float L = (Ls[0] + Ls[1]) + (Ls[2] + Ls[3]), acc = (accs[0] + accs[1]) + (accs[2] + accs[3]);
    out[((size_t)t * H + h) * D + threadIdx.x] = from_f32<T>(L == 0.f ? 0.f : acc * (1.0f / L));   // (0: no key was seen)
  }
}

// ---- the attention kernel of prompt steps
// A block = up to 32 (token, query head) rows of one key/value head and of one run of consecutive tokens (a tile of the
// step's metadata); 64 keys with their values are staged in shared memory as float32 once for all the rows: first the
// pooled rows that the tile's last token sees (gathered through the page table), then the window's pages.  A warp owns
// four rows, so a key element read from shared memory serves four multiply-adds; lanes own keys for the scores and
// value dimensions for the weighted sum.  Scores, maxima, exponentials, sums and weighted values are float32.  A row sees
// pooled block e iff e < its own count of seen blocks, and key p iff first <= p <= its position.
constexpr int TW_RW = 4, TW_WARPS = 8, TW_ROWS = TW_RW * TW_WARPS, TW_KEYS = PAGE;

template <typename T, int NC>    // NC = ceil(dv / 32): value dimensions a lane owns
__global__ void __launch_bounds__(TW_WARPS * 32)
pooled_window_attn_tiled_kernel(const T* __restrict__ q, T* __restrict__ out, const T* __restrict__ kcache, const T* __restrict__ vcache,
                                const float* __restrict__ pk, const float* __restrict__ pv, const int32_t* __restrict__ page_table,
                                int table_stride, int n_pages, const int32_t* __restrict__ tile_seq, const int32_t* __restrict__ tile_tok0,
                                const int32_t* __restrict__ tile_ntok, const int32_t* __restrict__ tile_pos0, int H, int G, int dk,
                                int dv, float scale, int window, int P, int R) {
  extern __shared__ float tw_smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int ks = dk + 1;                        // padded key row: lanes read different rows
  float* Ks = tw_smem;                          // [TW_KEYS][dk + 1]
  float* Vs = Ks + TW_KEYS * ks;                // [TW_KEYS][dv]
  float* Qs = Vs + TW_KEYS * dv;                // [TW_ROWS][dk]
  float* Ps = Qs + TW_ROWS * dk;                // [TW_ROWS][TW_KEYS]
  const int tile = blockIdx.x, g = blockIdx.y, grp = H / G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int seq = tile_seq[tile], tok0 = tile_tok0[tile], ntok = tile_ntok[tile], pos0 = tile_pos0[tile];
  const int32_t* pages = page_table + (size_t)seq * table_stride;
  const int rows_total = ntok * grp, row_base = blockIdx.z * TW_ROWS;
  if (row_base >= rows_total) return;
  const int rows_here = min(TW_ROWS, rows_total - row_base);
  const int last_pos = pos0 + (row_base + rows_here - 1) / grp, first_pos = pos0 + row_base / grp;
  for (int i = threadIdx.x; i < rows_here * dk; i += blockDim.x) {
    const int r = i / dk, d = i - r * dk;
    const int rr = row_base + r, tok = rr / grp, head = g * grp + rr % grp;
    Qs[r * dk + d] = to_f32(q[((size_t)(tok0 + tok) * H + head) * dk + d]);
  }
  float m[TW_RW], l[TW_RW], acc[TW_RW][NC];
  int limit[TW_RW], first[TW_RW], seen[TW_RW];
#pragma unroll
  for (int r = 0; r < TW_RW; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
    const int rr = row_base + warp * TW_RW + r;
    limit[r] = rr < rows_total ? pos0 + rr / grp : -1;                       // the row's own position; -1: no row
    first[r] = max(0, limit[r] - window + 1);
    seen[r] = (P > 0 && limit[r] - window >= 0) ? (limit[r] - window + 1) / P : 0;   // pooled blocks wholly before its window
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[r][c] = 0.f;
  }
  // what a warp does with the 64 staged keys whose indices (block numbers, or positions) start at `base`: row r sees
  // index i iff lo[r] <= i <= hi[r]
  auto process = [&](int base, const int (&lo)[TW_RW], const int (&hi)[TW_RW], int valid) {
    int any_hi = -1, any_lo = 0x7fffffff;
#pragma unroll
    for (int r = 0; r < TW_RW; ++r)
      if (hi[r] >= lo[r]) { any_hi = max(any_hi, hi[r]); any_lo = min(any_lo, lo[r]); }
    if (base > any_hi || base + TW_KEYS - 1 < any_lo) return;     // none of this warp's rows sees any of these keys
    const int i0 = base + lane, i1 = i0 + 32;
    float s0[TW_RW] = {}, s1[TW_RW] = {};
    const float* k0 = Ks + lane * ks;
    const float* k1 = Ks + (lane + 32) * ks;
    const float* qw = Qs + warp * TW_RW * dk;
    for (int d = 0; d < dk; ++d) {
      const float a = k0[d], b = k1[d];
#pragma unroll
      for (int r = 0; r < TW_RW; ++r) {
        const float qv = qw[r * dk + d];
        s0[r] = fmaf(qv, a, s0[r]);
        s1[r] = fmaf(qv, b, s1[r]);
      }
    }
    float corr[TW_RW];
#pragma unroll
    for (int r = 0; r < TW_RW; ++r) {
      const float a = i0 >= lo[r] && i0 <= hi[r] ? s0[r] * scale : -INFINITY;
      const float b = i1 >= lo[r] && i1 <= hi[r] ? s1[r] * scale : -INFINITY;
      const float mx = fmaxf(m[r], warp_max(fmaxf(a, b)));
      float p0 = 0.f, p1 = 0.f;
      corr[r] = 1.f;
      if (mx != -INFINITY) {      // uniform over the warp
        corr[r] = expf(m[r] - mx);
        p0 = expf(a - mx);
        p1 = expf(b - mx);
        l[r] = l[r] * corr[r] + warp_sum(p0 + p1);
        m[r] = mx;
      }
      Ps[(warp * TW_RW + r) * TW_KEYS + lane] = p0;
      Ps[(warp * TW_RW + r) * TW_KEYS + lane + 32] = p1;
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < TW_RW; ++r)
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[r][c] *= corr[r];
    const float* pw = Ps + warp * TW_RW * TW_KEYS;
    for (int j = 0; j < valid; ++j) {
      float v[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int d = lane + 32 * c;
        v[c] = d < dv ? Vs[j * dv + d] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < TW_RW; ++r) {
        const float pj = pw[r * TW_KEYS + j];
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[r][c] = fmaf(pj, v[c], acc[r][c]);
      }
    }
    __syncwarp();
  };
  // 1. the pooled rows that the block's last token sees
  const int blocks_seen = (P > 0 && last_pos - window >= 0) ? (last_pos - window + 1) / P : 0;
  int zero[TW_RW], top[TW_RW];
#pragma unroll
  for (int r = 0; r < TW_RW; ++r) { zero[r] = 0; top[r] = limit[r] < 0 ? -1 : seen[r] - 1; }
  for (int e0 = 0; e0 < blocks_seen; e0 += TW_KEYS) {
    const int valid = min(TW_KEYS, blocks_seen - e0);
    __syncthreads();              // the keys staged before are no longer read (and the queries are staged)
    for (int i = threadIdx.x; i < TW_KEYS * (dk + dv); i += blockDim.x) {
      const int j = i / (dk + dv), c = i - j * (dk + dv);
      float val = 0.f;
      if (j < valid) {
        const int e = e0 + j, end = e * P + P - 1;
        const int page = pages[end / PAGE];
        if (page >= 0 && page < n_pages) {
          const size_t rowi = ((size_t)page * G + g) * R + (e - (PAGE * (end / PAGE)) / P);
          val = c < dk ? pk[rowi * dk + c] : pv[rowi * dv + (c - dk)];
        }
      }
      if (c < dk) Ks[j * ks + c] = val; else Vs[j * dv + (c - dk)] = val;
    }
    __syncthreads();
    process(e0, zero, top, valid);
  }
  // 2. the window's pages: from the page of the first row's first key to the page of the last row's position
  const int kt_begin = max(0, first_pos - window + 1) / PAGE, kt_end = last_pos / PAGE;
  for (int kt = kt_begin; kt <= kt_end; ++kt) {
    const int page = pages[kt];
    const bool held = page >= 0 && page < n_pages;
    const T* kp = kcache + ((size_t)(held ? page : 0) * G + g) * PAGE * dk;
    const T* vp = vcache + ((size_t)(held ? page : 0) * G + g) * PAGE * dv;
    const int valid = held ? min(PAGE, last_pos + 1 - kt * PAGE) : 0;   // rows of the page that hold this block's keys
    __syncthreads();
    for (int i = threadIdx.x; i < PAGE * dk; i += blockDim.x) {
      const int j = i / dk, d = i - j * dk;
      Ks[j * ks + d] = j < valid ? to_f32(kp[i]) : 0.f;   // what lies behind is not this sequence's: never let it in
    }
    for (int i = threadIdx.x; i < PAGE * dv; i += blockDim.x) Vs[i] = i / dv < valid ? to_f32(vp[i]) : 0.f;
    __syncthreads();
    process(kt * PAGE, first, limit, valid);
  }
#pragma unroll
  for (int r = 0; r < TW_RW; ++r) {
    const int rr = row_base + warp * TW_RW + r;
    if (rr >= rows_total) continue;
    const int tok = rr / grp, head = g * grp + rr % grp;
    const float inv = l[r] > 0.f ? 1.0f / l[r] : 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int d = lane + 32 * c;
      if (d < dv) out[((size_t)(tok0 + tok) * H + head) * dv + d] = from_f32<T>(acc[r][c] * inv);
    }
  }
}

// ---- prompt steps on the tensor cores (bfloat16 cache, key and value heads of one size of 32, 64, 96 or 128)
// A block of four warps: 64 consecutive new tokens of one sequence, one query head, 16 rows a warp; the keys 64 at a time for the
// window's pages (copied by cp.async, two stages), 32 at a time for the pooled rows, which come first.  Scores of page keys are
// products of bfloat16 numbers summed in float32; the float32 weights, and the pooled rows' float32 keys and values, go as three
// bfloat16 terms (8 + 8 + 8 bits of their mantissas), weights times pooled values as the six products of terms that float32 can
// tell from zero.  Scores, maxima, exponentials, denominators and outputs are float32, as on the CUDA cores.
// 2,048 tokens, 32 heads of 64, a window of 1,024, blocks of 64: 1,131 us there, 145 us here (three small matrix
// instructions for every page value, in chains with the exponentials: the tensor pipe is active 44 % of the time, half of the issue slots used).
constexpr int PM_WARPS = 4, PM_ROWS = 16 * PM_WARPS, PM_POOLED = 32;

// S[NT tiles of 8 keys] = Q K^T, the keys in TERMS tiles of `tile` elements one after the other (the smallest term first)
template <int HDT, int NT, int TERMS>
__device__ __forceinline__ void pm_scores(float (&s)[NT][4], const uint32_t (&qa)[HDT][4], const __nv_bfloat16* ks, int tile, int lane) {
  constexpr int PITCH = HDT * 16 + 8;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
#pragma unroll
    for (int t = TERMS - 1; t >= 0; --t)
#pragma unroll
      for (int d = 0; d < HDT; d += 2) {
        const int mi = lane >> 3;
        uint32_t b0, b1, b2, b3;
        sp_ldmatrix_x4(sp_smem(ks + t * tile + (nt * 8 + (lane & 7)) * PITCH + (d + (mi >> 1)) * 16 + (mi & 1) * 8), b0, b1, b2, b3);
        sp_mma(s[nt], qa[d][0], qa[d][1], qa[d][2], qa[d][3], b0, b1);
        sp_mma(s[nt], qa[d + 1][0], qa[d + 1][1], qa[d + 1][2], qa[d + 1][3], b2, b3);
      }
  }
}

// running maximum, denominator and outputs of the lane's two rows over NT tiles of keys whose scores (in units of log 2, -inf: not
// seen) are in `s`, with the values in TERMS tiles
template <int VDT, int NT, int TERMS>
__device__ __forceinline__ void pm_gather(float (&s)[NT][4], float (&o)[VDT * 2][4], float& mA, float& mB, float& lA, float& lB,
                                          const __nv_bfloat16* vs, int tile, int lane) {
  constexpr int PITCH = VDT * 16 + 8;
  float mxA = -INFINITY, mxB = -INFINITY;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    mxA = fmaxf(mxA, fmaxf(s[nt][0], s[nt][1]));
    mxB = fmaxf(mxB, fmaxf(s[nt][2], s[nt][3]));
  }
#pragma unroll
  for (int off = 1; off < 4; off <<= 1) {
    mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, off));
    mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, off));
  }
  const float nmA = fmaxf(mA, mxA), nmB = fmaxf(mB, mxB);
  const float refA = nmA == -INFINITY ? 0.f : nmA, refB = nmB == -INFINITY ? 0.f : nmB;      // (a row that sees no key yet)
  const float corrA = exp2f(mA - refA), corrB = exp2f(mB - refB);
  float sumA = 0.f, sumB = 0.f;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    s[nt][0] = exp2f(s[nt][0] - refA);
    s[nt][1] = exp2f(s[nt][1] - refA);
    s[nt][2] = exp2f(s[nt][2] - refB);
    s[nt][3] = exp2f(s[nt][3] - refB);
    sumA += s[nt][0] + s[nt][1];
    sumB += s[nt][2] + s[nt][3];
  }
#pragma unroll
  for (int off = 1; off < 4; off <<= 1) {
    sumA += __shfl_xor_sync(0xffffffffu, sumA, off);
    sumB += __shfl_xor_sync(0xffffffffu, sumB, off);
  }
  lA = lA * corrA + sumA;
  lB = lB * corrB + sumB;
  mA = nmA;
  mB = nmB;
  if (__any_sync(0xffffffffu, corrA != 1.f || corrB != 1.f)) {
#pragma unroll
    for (int i = 0; i < VDT * 2; ++i) {
      o[i][0] *= corrA;
      o[i][1] *= corrA;
      o[i][2] *= corrB;
      o[i][3] *= corrB;
    }
  }
#pragma unroll
  for (int kt = 0; kt < NT / 2; ++kt) {
    uint32_t a[3][4];
    sp_split(s[2 * kt][0], s[2 * kt][1], a[0][0], a[1][0], a[2][0]);
    sp_split(s[2 * kt][2], s[2 * kt][3], a[0][1], a[1][1], a[2][1]);
    sp_split(s[2 * kt + 1][0], s[2 * kt + 1][1], a[0][2], a[1][2], a[2][2]);
    sp_split(s[2 * kt + 1][2], s[2 * kt + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
    for (int v = TERMS - 1; v >= 0; --v)
#pragma unroll
      for (int dt = 0; dt < VDT * 2; dt += 2) {
        const int mi = lane >> 3;
        uint32_t b0, b1, b2, b3;
        sp_ldmatrix_x4_trans(sp_smem(vs + v * tile + (kt * 16 + (mi & 1) * 8 + (lane & 7)) * PITCH + (dt + (mi >> 1)) * 8), b0, b1, b2, b3);
#pragma unroll
        for (int t = 2 - v; t >= 0; --t) {      // (terms whose places add up to more than 2 are under float32's last bit)
          sp_mma(o[dt], a[t][0], a[t][1], a[t][2], a[t][3], b0, b1);
          sp_mma(o[dt + 1], a[t][0], a[t][1], a[t][2], a[t][3], b2, b3);
        }
      }
  }
}

template <int HDT>
__global__ void __launch_bounds__(PM_WARPS * 32)
pooled_window_attn_mma_kernel(const __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ kcache,
                              const __nv_bfloat16* __restrict__ vcache, const float* __restrict__ pk, const float* __restrict__ pv,
                              const int32_t* __restrict__ page_table, int table_stride, int n_pages, const int32_t* __restrict__ tile_seq,
                              const int32_t* __restrict__ tile_tok0, const int32_t* __restrict__ tile_ntok,
                              const int32_t* __restrict__ tile_pos0, int H, int G, float scale, int window, int P, int R) {
  constexpr int HD = HDT * 16, PITCH = HD + 8, PIECES = HD / 8, STAGE = 2 * PAGE * PITCH, TERM = PM_POOLED * PITCH;
  extern __shared__ __align__(16) uint8_t pm_raw[];
  __nv_bfloat16* sm = reinterpret_cast<__nv_bfloat16*>(pm_raw);      // two stages (keys | values), or three terms of pooled keys | values
  const int tile = blockIdx.x, head = blockIdx.y, g = head / (H / G);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
  const int tok0 = tile_tok0[tile], ntok = tile_ntok[tile], pos0 = tile_pos0[tile];
  const int32_t* table = page_table + (size_t)tile_seq[tile] * table_stride;
  const int rowA = warp * 16 + gid, rowB = rowA + 8;
  const int posA = rowA < ntok ? pos0 + rowA : -1, posB = rowB < ntok ? pos0 + rowB : -1;      // (-1: no such row, nothing is seen)
  const int n_keys = pos0 + ntok, first_page = max(0, pos0 - window + 1) / PAGE, end_page = (n_keys + PAGE - 1) / PAGE;
  const float scale2 = scale * 1.4426950408889634f;                  // scores in units of log 2
  auto page_of = [&](int i) {
    const int page = table[i];
    return page < n_pages ? page : -1;
  };
  auto load_page = [&](int i, int stage) {
    const int page = page_of(i), valid = page >= 0 ? min(PAGE, n_keys - i * PAGE) : 0;      // (rows past the last key: zeros)
    const size_t row0 = ((size_t)max(page, 0) * G + g) * PAGE;
    __nv_bfloat16* ks = sm + stage * STAGE;
    for (int e = threadIdx.x; e < PAGE * PIECES; e += PM_WARPS * 32) {
      const int r = e / PIECES, c = (e - r * PIECES) * 8, bytes = r < valid ? 16 : 0;
      sp_cp16(sp_smem(ks + r * PITCH + c), bytes ? kcache + (row0 + r) * HD + c : kcache, bytes);
      sp_cp16(sp_smem(ks + PAGE * PITCH + r * PITCH + c), bytes ? vcache + (row0 + r) * HD + c : vcache, bytes);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint32_t qa[HDT][4];
  {
    const uint32_t* qA = reinterpret_cast<const uint32_t*>(q + ((size_t)(tok0 + min(rowA, ntok - 1)) * H + head) * HD) + tig;
    const uint32_t* qB = reinterpret_cast<const uint32_t*>(q + ((size_t)(tok0 + min(rowB, ntok - 1)) * H + head) * HD) + tig;
#pragma unroll
    for (int d = 0; d < HDT; ++d) {
      qa[d][0] = qA[d * 8];
      qa[d][1] = qB[d * 8];
      qa[d][2] = qA[d * 8 + 4];
      qa[d][3] = qB[d * 8 + 4];
    }
  }
  float o[HDT * 2][4];
#pragma unroll
  for (int i = 0; i < HDT * 2; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float mA = -INFINITY, mB = -INFINITY, lA = 0.f, lB = 0.f;

  // the pooled rows of the blocks that the tile's last token sees, 32 at a time: each value as three terms
  auto blocks_seen = [&](int pos) { return P > 0 && pos >= window ? (pos - window + 1) / P : 0; };
  const int nbA = blocks_seen(posA), nbB = blocks_seen(posB), nb = blocks_seen(n_keys - 1);
  for (int b0 = 0; b0 < nb; b0 += PM_POOLED) {
    __syncthreads();
    for (int e = threadIdx.x; e < PM_POOLED * (HD / 2) * 2; e += PM_WARPS * 32) {
      const int which = e / (PM_POOLED * (HD / 2)), r = e / (HD / 2) % PM_POOLED, c = e % (HD / 2) * 2, b = b0 + r;
      float2 x = make_float2(0.f, 0.f);
      if (b < nb) {
        const int end = b * P + P - 1, page = page_of(end / PAGE);
        if (page >= 0) x = *reinterpret_cast<const float2*>((which ? pv : pk) + (((size_t)page * G + g) * R + b - PAGE * (end / PAGE) / P) * HD + c);
      }
      uint32_t t1, t2, t3;
      sp_split(x.x, x.y, t1, t2, t3);
      __nv_bfloat16* dst = sm + which * 3 * TERM + r * PITCH + c;
      *reinterpret_cast<uint32_t*>(dst) = t1;
      *reinterpret_cast<uint32_t*>(dst + TERM) = t2;
      *reinterpret_cast<uint32_t*>(dst + 2 * TERM) = t3;
    }
    __syncthreads();
    float s[PM_POOLED / 8][4];
    pm_scores<HDT, PM_POOLED / 8, 3>(s, qa, sm, TERM, lane);
#pragma unroll
    for (int nt = 0; nt < PM_POOLED / 8; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[nt][j] = b0 + nt * 8 + tig * 2 + (j & 1) < (j < 2 ? nbA : nbB) ? s[nt][j] * scale2 : -INFINITY;
    pm_gather<HDT, PM_POOLED / 8, 3>(s, o, mA, mB, lA, lB, sm + 3 * TERM, TERM, lane);
  }
  if (nb > 0) __syncthreads();
  // the window's pages
  const int warp_last = warp * 16 < ntok ? pos0 + min(ntok - 1, warp * 16 + 15) : -1, warp_first = pos0 + warp * 16 - window + 1;
  load_page(first_page, 0);
  for (int i = first_page; i < end_page; ++i) {
    const int stage = (i - first_page) & 1;
    if (i + 1 < end_page) {
      load_page(i + 1, stage ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (i * PAGE <= warp_last && i * PAGE + PAGE > warp_first) {      // else: no row of this warp sees a key of the page
      const __nv_bfloat16* ks = sm + stage * STAGE;
      float s[PAGE / 8][4];
      pm_scores<HDT, PAGE / 8, 1>(s, qa, ks, 0, lane);
      // every row sees the whole page: no mask
      const bool whole = warp * 16 + 15 < ntok && i * PAGE + PAGE - 1 <= pos0 + warp * 16 && i * PAGE >= warp_first + 15;
#pragma unroll
      for (int nt = 0; nt < PAGE / 8; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = i * PAGE + nt * 8 + tig * 2 + (j & 1), pos = j < 2 ? posA : posB;
          s[nt][j] = whole || (key <= pos && key > pos - window) ? s[nt][j] * scale2 : -INFINITY;
        }
      pm_gather<HDT, PAGE / 8, 1>(s, o, mA, mB, lA, lB, ks + PAGE * PITCH, 0, lane);
    }
    __syncthreads();
  }
  const float invA = lA > 0.f ? 1.0f / lA : 0.f, invB = lB > 0.f ? 1.0f / lB : 0.f;
#pragma unroll
  for (int dt = 0; dt < HDT * 2; ++dt) {
    const int d = dt * 8 + tig * 2;
    if (rowA < ntok) *reinterpret_cast<__nv_bfloat162*>(out + ((size_t)(tok0 + rowA) * H + head) * HD + d) = __floats2bfloat162_rn(o[dt][0] * invA, o[dt][1] * invA);
    if (rowB < ntok) *reinterpret_cast<__nv_bfloat162*>(out + ((size_t)(tok0 + rowB) * H + head) * HD + d) = __floats2bfloat162_rn(o[dt][2] * invB, o[dt][3] * invB);
  }
}

}  // namespace edgelm

using namespace edgelm;

extern "C" int edgelm_qk_rope_norm_append(const float* qkv, const float* bias, void* q_out, int dtype, const int32_t* tok_pos,
                                          const int32_t* tok_seq, const int32_t* page_table, int table_stride, int n_pages,
                                          void* kcache, void* vcache, int n_tokens, int H, int G, int dk, int dv, int rot,
                                          const double* freq, float eps, int unit_norm, int* err, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  EL_REFUSE(n_tokens > 0 && H > 0 && G > 0 && H % G == 0, "qk_rope_norm_append: %d query heads over %d key/value heads", H, G);
  EL_REFUSE(dk >= 1 && dk <= 256 && dv >= 1 && dv <= 256, "qk_rope_norm_append: head sizes %d / %d are not taken (1 to 256)", dk, dv);
  EL_REFUSE(rot >= 0 && rot <= dk && rot % 2 == 0, "qk_rope_norm_append: %d rotated dimensions of %d", rot, dk);
  EL_REFUSE(dtype == DT_F32 || dtype == DT_BF16, "qk_rope_norm_append: unknown dtype code %d", dtype);
  if (rotate_rows_takes(n_tokens, H, G, dk, dv, 1, rot, 0, 0)) {      // (prompt steps, heads of whole runs of 32)
    const RotateRows rows{qkv, (H + G) * dk + G * dv, bias, tok_pos, tok_seq, page_table, table_stride, n_pages, n_tokens, H, G, dv, 1, rot, 0, freq, err,
                          nullptr, nullptr, eps, 1.f, unit_norm, nullptr, nullptr, nullptr, nullptr, 0};
    if (dtype == DT_F32) launch_rotate_rows(rows, dk, (float*)q_out, (float*)kcache, (float*)vcache, stream);
    else launch_rotate_rows(rows, dk, (__nv_bfloat16*)q_out, (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, stream);
    EL_LAUNCH_CHECK("rotate_rows");
    return 0;
  }
  const size_t smem = (size_t)PW_WARPS * dk * sizeof(float);
  if (dtype == DT_F32)
    launch_pdl(pdl_bit_for_tokens(n_tokens), qk_rope_norm_append_kernel<float>, dim3(n_tokens, (H + G + PW_WARPS - 1) / PW_WARPS), dim3(PW_WARPS * 32), (size_t)(smem), stream, qkv, bias, (float*)q_out, tok_pos, tok_seq, page_table, table_stride, n_pages,
                                                                              (float*)kcache, (float*)vcache, H, G, dk, dv, rot, freq, eps, unit_norm, err);
  else
    launch_pdl(pdl_bit_for_tokens(n_tokens), qk_rope_norm_append_kernel<__nv_bfloat16>, dim3(n_tokens, (H + G + PW_WARPS - 1) / PW_WARPS), dim3(PW_WARPS * 32), (size_t)(smem), stream, qkv, bias, (__nv_bfloat16*)q_out, tok_pos, tok_seq, page_table, table_stride, n_pages,
                                                                                      (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, H, G, dk, dv, rot, freq, eps, unit_norm, err);
  EL_LAUNCH_CHECK("qk_rope_norm_append");
  return 0;
}

extern "C" int edgelm_pool_blocks(const int32_t* tok_pos, const int32_t* tok_seq, const int32_t* page_table, int table_stride,
                                  int n_pages, const void* kcache, const void* vcache, int dtype, float* pk, float* pv,
                                  int n_tokens, int G, int dk, int dv, int P, int R, int* err, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  EL_REFUSE(n_tokens > 0 && G > 0 && dk > 0 && dv > 0 && P >= 1 && R == (PAGE + P - 1) / P, "pool_blocks: bad sizes (block %d, rows a page %d)", P, R);
  // (blocks of few tokens: as long a run as leaves eight blocks of threads an SM)
  const long long shared = (long long)n_tokens * G / (8 * 148);
  const int want = P > shared ? P : (int)shared, run = n_tokens <= 64 ? 1 : want < POOL_RUN ? want : POOL_RUN, runs = (n_tokens + run - 1) / run;
  if (dtype == DT_F32)
    launch_pdl(pdl_bit_for_tokens(n_tokens), pool_blocks_kernel<float>, dim3(runs, G), dim3(128), (size_t)(0), stream, tok_pos, tok_seq, page_table, table_stride, n_pages, (const float*)kcache, (const float*)vcache, pk, pv, G, dk, dv, P, R, err, n_tokens, run);
  else if (dtype == DT_BF16)
    launch_pdl(pdl_bit_for_tokens(n_tokens), pool_blocks_kernel<__nv_bfloat16>, dim3(runs, G), dim3(128), (size_t)(0), stream, tok_pos, tok_seq, page_table, table_stride, n_pages, (const __nv_bfloat16*)kcache, (const __nv_bfloat16*)vcache, pk, pv, G, dk, dv, P, R, err, n_tokens, run);
  else
    EL_REFUSE(false, "pool_blocks: unknown dtype code %d", dtype);
  EL_LAUNCH_CHECK("pool_blocks");
  return 0;
}

extern "C" int edgelm_pooled_window_attn(const void* q, void* out, const void* kcache, const void* vcache, int dtype, const float* pk,
                                         const float* pv, const int32_t* tok_pos, const int32_t* tok_seq, const int32_t* page_table,
                                         int table_stride, int n_pages, int n_tokens, int H, int G, int dk, int dv, float scale,
                                         int window, int P, int R, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  EL_REFUSE(n_tokens > 0 && H > 0 && G > 0 && H % G == 0, "pooled_window_attn: %d query heads over %d key/value heads", H, G);
  EL_REFUSE(dk >= 1 && dk <= 256 && dv >= 1 && dv <= 256, "pooled_window_attn: head sizes %d / %d are not taken (1 to 256)", dk, dv);
  EL_REFUSE(window >= 1 && P >= 0 && (P == 0 || R == (PAGE + P - 1) / P), "pooled_window_attn: window %d, block %d, rows a page %d", window, P, R);
  // few (token, head) pairs (a decode step): more warps a block share one query's keys
  const int nw = (long long)n_tokens * H >= 2 * 148 * 4 ? 4 : PW_MAX_WARPS;
  const dim3 grid(n_tokens, H), block(nw * 32);
  const size_t smem = (size_t)(((dk + 3) & ~3) + 2 * nw + nw * dv) * sizeof(float);
  const int esz = dtype == DT_F32 ? 4 : 2;
  const int vec_k = ((size_t)dk * esz) % 16 == 0 && (uintptr_t)kcache % 16 == 0;
  const int pair_v = dv % 2 == 0 && (uintptr_t)vcache % 8 == 0;
  EL_REFUSE(P == 0 || ((uintptr_t)pk % 16 == 0 && (uintptr_t)pv % 8 == 0), "pooled_window_attn: the pooled rows are not 16-byte aligned");
  EL_REFUSE((long long)n_pages * G * (PAGE > R ? PAGE : R) < (1ll << 31), "pooled_window_attn: more cache rows than a 32-bit index counts");
  if (dk == dv && (dk == 32 || dk == 64 || dk == 128) && vec_k && (uintptr_t)vcache % 16 == 0 && (P == 0 || (uintptr_t)pv % 16 == 0)) {
    // warps a block: a run of 32 keys a warp where blocks are few (the chain of trips counts), fewer and longer runs where there are many
    const long long blocks = (long long)n_tokens * H;
    const int most = blocks >= 148 * 12 ? 4 : blocks >= 148 * 4 ? 8 : PWR_MAX_WARPS, warps = max(1, min(most, (window + 31) / 32));
    const dim3 threads(max(warps * 32, dk));
#define EL_PWR(TT, DD) launch_pdl(pdl_bit_for_tokens(n_tokens), pooled_window_attn_rows_kernel<TT, DD>, grid, threads, (size_t)0, stream, (const TT*)q, (TT*)out, \
      (const TT*)kcache, (const TT*)vcache, pk, pv, tok_pos, tok_seq, page_table, table_stride, n_pages, H, G, scale, window, P, R)
    if (dtype == DT_F32) {
      if (dk == 32) EL_PWR(float, 32); else if (dk == 64) EL_PWR(float, 64); else EL_PWR(float, 128);
    } else if (dtype == DT_BF16) {
      if (dk == 32) EL_PWR(__nv_bfloat16, 32); else if (dk == 64) EL_PWR(__nv_bfloat16, 64); else EL_PWR(__nv_bfloat16, 128);
    } else
      EL_REFUSE(false, "pooled_window_attn: unknown dtype code %d", dtype);
#undef EL_PWR
    EL_LAUNCH_CHECK("pooled_window_attn");
    return 0;
  }
  const int dvr = dv <= 64 ? 1 : (dv <= 128 ? 2 : 4);
#define EL_PWA(TT, DVR) launch_pdl(pdl_bit_for_tokens(n_tokens), pooled_window_attn_kernel<TT, DVR>, dim3(grid), dim3(block), (size_t)(smem), stream, (const TT*)q, (TT*)out, (const TT*)kcache, (const TT*)vcache, pk, pv, \
      tok_pos, tok_seq, page_table, table_stride, n_pages, H, G, dk, dv, scale, window, P, R, vec_k, pair_v)
  if (dtype == DT_F32) {
    if (dvr == 1) EL_PWA(float, 1); else if (dvr == 2) EL_PWA(float, 2); else EL_PWA(float, 4);
  } else if (dtype == DT_BF16) {
    if (dvr == 1) EL_PWA(__nv_bfloat16, 1); else if (dvr == 2) EL_PWA(__nv_bfloat16, 2); else EL_PWA(__nv_bfloat16, 4);
  } else
    EL_REFUSE(false, "pooled_window_attn: unknown dtype code %d", dtype);
#undef EL_PWA
  EL_LAUNCH_CHECK("pooled_window_attn");
  return 0;
}

// The same attention for prompt steps: tiles (runs of at most `max_tile_tokens` consecutive tokens of one sequence, as
// the step's metadata lists them) instead of single tokens; `max_tile_tokens` x (H / G) rows are dealt to blocks of 32.
template <typename T, int NC>
static int launch_tiled(const void* q, void* out, const void* kc, const void* vc, const float* pk, const float* pv,
                        const int32_t* page_table, int table_stride, int n_pages, const int32_t* tile_seq, const int32_t* tile_tok0,
                        const int32_t* tile_ntok, const int32_t* tile_pos0, int n_tiles, int max_tile_tokens, int H, int G, int dk, int dv,
                        float scale, int window, int P, int R, cudaStream_t stream) {
  const size_t smem = sizeof(float) * ((size_t)TW_KEYS * (dk + 1) + (size_t)TW_KEYS * dv + (size_t)TW_ROWS * dk + (size_t)TW_ROWS * TW_KEYS);
  auto kern = pooled_window_attn_tiled_kernel<T, NC>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    set_error("pooled_window_attn_tiled: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
    return -2;
  }
  const dim3 grid(n_tiles, G, (max_tile_tokens * (H / G) + TW_ROWS - 1) / TW_ROWS);
  kern<<<grid, TW_WARPS * 32, smem, stream>>>((const T*)q, (T*)out, (const T*)kc, (const T*)vc, pk, pv, page_table, table_stride, n_pages, tile_seq,
                                             tile_tok0, tile_ntok, tile_pos0, H, G, dk, dv, scale, window, P, R);
  return 0;
}

extern "C" int edgelm_pooled_window_attn_tiled(const void* q, void* out, const void* kcache, const void* vcache, int dtype, const float* pk,
                                               const float* pv, const int32_t* page_table, int table_stride, int n_pages,
                                               const int32_t* tile_seq, const int32_t* tile_tok0, const int32_t* tile_ntok,
                                               const int32_t* tile_pos0, int n_tiles, int max_tile_tokens, int H, int G, int dk, int dv,
                                               float scale, int window, int P, int R, cudaStream_t stream) {
  if (n_tiles == 0) return 0;
  EL_REFUSE(n_tiles > 0 && max_tile_tokens > 0 && H > 0 && G > 0 && H % G == 0, "pooled_window_attn_tiled: %d query heads over %d key/value heads", H, G);
  EL_REFUSE(dk >= 1 && dk <= 256 && dv >= 1 && dv <= 256, "pooled_window_attn_tiled: head sizes %d / %d are not taken (1 to 256)", dk, dv);
  EL_REFUSE(window >= 1 && P >= 0 && (P == 0 || R == (PAGE + P - 1) / P), "pooled_window_attn_tiled: window %d, block %d, rows a page %d", window, P, R);
  EL_REFUSE(dtype == DT_F32 || dtype == DT_BF16, "pooled_window_attn_tiled: unknown dtype code %d", dtype);
  int rc;
#define EL_TW(NC)                                                                                                                                  \
  rc = dtype == DT_F32 ? launch_tiled<float, NC>(q, out, kcache, vcache, pk, pv, page_table, table_stride, n_pages, tile_seq, tile_tok0, tile_ntok, \
                                                 tile_pos0, n_tiles, max_tile_tokens, H, G, dk, dv, scale, window, P, R, stream)                    \
                       : launch_tiled<__nv_bfloat16, NC>(q, out, kcache, vcache, pk, pv, page_table, table_stride, n_pages, tile_seq, tile_tok0,   \
                                                         tile_ntok, tile_pos0, n_tiles, max_tile_tokens, H, G, dk, dv, scale, window, P, R, stream)
  if (dv <= 32) { EL_TW(1); } else if (dv <= 64) { EL_TW(2); } else if (dv <= 128) { EL_TW(4); } else { EL_TW(8); }
#undef EL_TW
  if (rc != 0) return rc;
  EL_LAUNCH_CHECK("pooled_window_attn_tiled");
  return 0;
}

// 1 if the tensor-core kernel of prompt steps takes these head sizes, else 0.
extern "C" int edgelm_pooled_window_attn_mma_takes(int dk, int dv) { return dk == dv && (dk == 32 || dk == 64 || dk == 96 || dk == 128) ? 1 : 0; }

// `edgelm_pooled_window_attn_tiled` on the tensor cores: a bfloat16 cache, tiles of at most 64 consecutive tokens of one sequence.
extern "C" int edgelm_pooled_window_attn_mma(const void* q, void* out, const void* kcache, const void* vcache, const float* pk, const float* pv,
                                             const int32_t* page_table, int table_stride, int n_pages, const int32_t* tile_seq,
                                             const int32_t* tile_tok0, const int32_t* tile_ntok, const int32_t* tile_pos0, int n_tiles, int H,
                                             int G, int dk, int dv, float scale, int window, int P, int R, cudaStream_t stream) {
  if (n_tiles == 0) return 0;
  EL_REFUSE(n_tiles > 0 && H > 0 && H <= 65535 && G > 0 && H % G == 0, "pooled_window_attn_mma: %d query heads over %d key/value heads", H, G);
  EL_REFUSE(edgelm_pooled_window_attn_mma_takes(dk, dv), "pooled_window_attn_mma: head sizes %d / %d are not taken (32, 64, 96 or 128, both alike)", dk, dv);
  EL_REFUSE(window >= 1 && P >= 0 && (P == 0 || (R == (PAGE + P - 1) / P && pk != nullptr && pv != nullptr)), "pooled_window_attn_mma: window %d, block %d, rows a page %d", window, P, R);
  EL_REFUSE((uintptr_t)q % 4 == 0 && (uintptr_t)out % 4 == 0 && (uintptr_t)kcache % 16 == 0 && (uintptr_t)vcache % 16 == 0 && (uintptr_t)pk % 8 == 0 && (uintptr_t)pv % 8 == 0,
            "pooled_window_attn_mma: keys and values must be 16-byte aligned, pooled rows 8");
  const size_t smem = (size_t)2 * 2 * PAGE * (dk + 8) * 2;      // (more than the pooled rows' six terms of 32 rows)
#define EL_PM(HDT)                                                                                                                       \
  do {                                                                                                                                   \
    auto kern = pooled_window_attn_mma_kernel<HDT>;                                                                                      \
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                            \
    EL_REFUSE(e == cudaSuccess, "pooled_window_attn_mma: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));          \
    kern<<<dim3(n_tiles, H), PM_WARPS * 32, smem, stream>>>((const __nv_bfloat16*)q, (__nv_bfloat16*)out, (const __nv_bfloat16*)kcache,  \
                                                           (const __nv_bfloat16*)vcache, pk, pv, page_table, table_stride, n_pages,      \
                                                           tile_seq, tile_tok0, tile_ntok, tile_pos0, H, G, scale, window, P, R);        \
  } while (0)
  if (dk == 32) EL_PM(2);
  else if (dk == 64) EL_PM(4);
  else if (dk == 96) EL_PM(6);
  else EL_PM(8);
#undef EL_PM
  EL_LAUNCH_CHECK("pooled_window_attn_mma");
  return 0;
}
