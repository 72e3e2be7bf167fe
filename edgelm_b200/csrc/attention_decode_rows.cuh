// Decode attention on the CUDA cores with whole rows in registers: the variant of attn_decode_kernel for head sizes whose
// rows are 8, 16 or 32 pieces of 16 bytes (float32: 32, 64, 128; bfloat16: 64, 128).  Included by attention.cu, which owns
// the entry points, the split bookkeeping and the combine kernel.
//
// Same decomposition (grid (sequence, kv head, split), 4 warps, partials folded in shared memory and across splits by
// the combine kernel); what differs is how a warp goes over its keys.  attn_decode_kernel brings a tile of K and V to
// shared memory, waits, and then reads every key once a query head and every query once a key from there: it was bound by
// shared memory and by one tile in flight a warp.  Here LPR lanes hold a row, 16 bytes each, and a warp requests 8 rows a
// lane of K and of V (a chunk of 256 / LPR keys) straight into registers, the next chunk's keys as soon as the scores
// are done and its values as soon as they are added: nothing is staged, and 8 KB a warp are on their way all the time.
// A lane multiplies its dims of 8 keys by the queries it holds; the lanes' partial scores are summed by a reduction that
// halves the keys a lane holds at every step (8 shuffles a head for 8 keys, not 8 x log2 LPR), so that every key's weight
// is computed once (or by LPR / 8 lanes at once), and is handed to the row's lanes by shuffle.
// What bounds it now is a chunk's latency when a warp has only a few, and issue when it has many (float32, 24 sequences of
// 500 keys, head size 64: 31 MB in 9.9 us with the splits' fold, 3.1 TB/s; head size 64, 32 heads on 32, 64 sequences
// of 1,000: 6.3 TB/s).  Before and after, with the fold: launch_decode.
#pragma once

namespace edgelm {

template <typename T, int LPR, int R>   // R: query heads a pass (RW at most)
__global__ void __launch_bounds__(DEC_WARPS * 32, sizeof(T) == 4 ? 3 : 2)
attn_decode_rows_kernel(const T* __restrict__ q, int ldq, T* __restrict__ out, int ldo, T* kcache, T* vcache,
                        const int32_t* __restrict__ page_table, int table_stride, const int32_t* __restrict__ seq_slot,
                        const int32_t* __restrict__ seq_pos, int nh, int nkv, float scale, int n_splits,
                        float* __restrict__ part_o, float* __restrict__ part_ml, int* err, const float* __restrict__ cos_t,
                        const float* __restrict__ sin_t, int max_pos, int window, int meta_ready) {
  constexpr int VEC = KVec<T>::N, HD = LPR * VEC, G = 32 / LPR, KEYS = 8 * G, PER_PAGE = PAGE / KEYS, SAME = LPR / 8, WS = HD + 2;
  static_assert(LPR >= 8 && 32 % LPR == 0 && PAGE % KEYS == 0, "");
  __shared__ __align__(16) float Qs[R][HD];
  __shared__ __align__(16) T newkv[2][HD];              // the new token's rotated key and its value
  __shared__ __align__(16) float Wp[DEC_WARPS * R * WS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int seq = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
  const int g = nh / nkv;
  const int row_of = lane / LPR, dim0 = (lane % LPR) * VEC;        // which of a load's G rows, and the lane's dims of it
  const int my_key = (lane % LPR) / SAME * G + row_of;             // the key of the chunk whose score the lane ends up with
  pdl_launch_dependents();
  if (!meta_ready) pdl_wait();
  const int nkeys = seq_pos[seq] + 1;      // the new token's own key is the last one
  const int32_t* pages = page_table + (size_t)seq_slot[seq] * table_stride;
  const int first_key = window > 0 ? max(0, nkeys - window) : 0;
  const int page0 = first_key / PAGE;      // the first page that holds a key the token sees
  const int n_pages = (nkeys + PAGE - 1) / PAGE - page0;
  const int per_split = (n_pages + n_splits - 1) / n_splits;
  const int p_begin = page0 + split * per_split, p_end = min(page0 + n_pages, p_begin + per_split);
  const int end_key = min(nkeys, p_end * PAGE);
  const int pos = nkeys - 1, half = HD / 2;
  const bool fused = cos_t != nullptr;
  const int tpos = min(pos, max_pos - 1);
  const bool owner = fused && (pos / PAGE - page0) / per_split == split;   // this block's pages include the new token's
  const int new_page = owner ? pages[pos / PAGE] : -1;
  // the warp's chunks: every DEC_WARPS-th of the split's, from the first that reaches into the window on
  int key0 = p_begin * PAGE + warp * KEYS;
  while (key0 + KEYS <= first_key) key0 += DEC_WARPS * KEYS;       // (the window starts on the first page: a few steps at most)
  const int first = key0;
  int page = key0 < end_key ? pages[key0 / PAGE] : 0;
  if (meta_ready) pdl_wait();   // the queries, the new key and value and the cache rows of the step before are the earlier kernels'
  if (fused && pos >= max_pos && threadIdx.x == 0 && err) atomicOr(err, ERR_POSITION_RANGE);
  if (owner && new_page < 0 && threadIdx.x == 0 && err) atomicOr(err, ERR_PAGE_RANGE);

  auto rotated = [&](const T* row, int d) {   // element d of the rotated head `row`
    const int j = d < half ? d : d - half;
    const float c = cos_t[(size_t)tpos * half + j], sn = sin_t[(size_t)tpos * half + j];
    const float self = to_f32(row[d]), other = to_f32(row[d < half ? d + half : d - half]);
    const float y = d < half ? self * c - other * sn : self * c + other * sn;
    return to_f32(from_f32<T>(y));
  };
  // the rows of the chunk at `k0` on page `pg`, the lane's 16 bytes of each: keys outside what the token sees read as zeros
  // (what the page holds there is not the sequence's), and the new token's own row is put in later (it may not have
  // landed yet)
  auto request = [&](const T* cache, int k0, int pg, uint4 (&v)[8]) {
    const T* base = cache + (((size_t)pg * nkv + kvh) * PAGE + (k0 % PAGE)) * HD + dim0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int key = k0 + i * G + row_of;
      v[i] = make_uint4(0, 0, 0, 0);
      if (pg >= 0 && key >= first_key && key < end_key && !(fused && key == pos)) v[i] = *reinterpret_cast<const uint4*>(base + (size_t)(i * G + row_of) * HD);
    }
  };
  auto own_row = [&](const T* row, int k0, uint4 (&v)[8]) {
    if (!fused || pos < k0 || pos >= k0 + KEYS) return;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k0 + i * G + row_of == pos) v[i] = *reinterpret_cast<const uint4*>(row + dim0);
  };
  auto floats = [](const uint4& v, float (&f)[VEC]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (VEC == 4) {
        f[i] = __uint_as_float(w[i]);
      } else {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      }
    }
  };

  uint4 kr[8], vr[8];
  for (int h0 = 0; h0 < g; h0 += R) {     // passes of R query heads of this kv head
    const int rows = min(R, g - h0);
    key0 = first;
    if (key0 < end_key) {   // the first chunk is on its way while the queries are staged
      if (h0) page = pages[key0 / PAGE];
      request(kcache, key0, page, kr);
      request(vcache, key0, page, vr);
    }
    __syncthreads();
    if (owner && h0 == 0) {
      const T* krow = q + (size_t)seq * ldq + (size_t)(nh + kvh) * HD;
      const T* vrow = q + (size_t)seq * ldq + (size_t)(nh + nkv + kvh) * HD;
      for (int d = threadIdx.x; d < HD; d += DEC_WARPS * 32) {
        const T kd = from_f32<T>(rotated(krow, d));
        newkv[0][d] = kd;
        newkv[1][d] = vrow[d];
        if (new_page >= 0) {
          const size_t dst = (((size_t)new_page * nkv + kvh) * PAGE + pos % PAGE) * HD + d;
          kcache[dst] = kd;
          vcache[dst] = vrow[d];
        }
      }
    }
    for (int i = threadIdx.x; i < R * HD; i += DEC_WARPS * 32) {
      const int r = i / HD, d = i - r * HD;
      const T* qrow = q + (size_t)seq * ldq + (size_t)(kvh * g + h0 + r) * HD;
      Qs[r][d] = r >= rows ? 0.f : fused ? rotated(qrow, d) : to_f32(qrow[d]);
    }
    __syncthreads();
    float qv[R][VEC], acc[R][VEC], m[R], l[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      m[r] = -CUDART_INF_F;
      l[r] = 0.f;
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        qv[r][e] = Qs[r][dim0 + e];
        acc[r][e] = 0.f;
      }
    }
    while (key0 < end_key) {
      const int next = key0 + DEC_WARPS * KEYS;
      const int next_page = next < end_key ? pages[next / PAGE] : 0;
      own_row(newkv[0], key0, kr);
      float s[8][R];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float f[VEC];
        floats(kr[i], f);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          s[i][r] = 0.f;
#pragma unroll
          for (int e = 0; e < VEC; ++e) s[i][r] = fmaf(qv[r][e], f[e], s[i][r]);
        }
      }
      if (next < end_key) request(kcache, next, next_page, kr);
      // the sums over the row's lanes: every step hands half of the keys a lane holds to its partner
#pragma unroll
      for (int n = 4, mask = LPR / 2; n >= 1; n /= 2, mask /= 2) {
        const bool upper = (lane & mask) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float give = upper ? s[i][r] : s[i + n][r], keep = upper ? s[i + n][r] : s[i][r];
            s[i][r] = keep + __shfl_xor_sync(0xffffffffu, give, mask);
          }
      }
      const bool seen = key0 + my_key >= first_key && key0 + my_key < end_key;
      float p[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int mask = SAME / 2; mask >= 1; mask /= 2) s[0][r] += __shfl_xor_sync(0xffffffffu, s[0][r], mask);
        const float a = seen ? s[0][r] * scale : -CUDART_INF_F;
        float mx = a;
#pragma unroll
        for (int mask = 16; mask >= SAME; mask /= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, mask));
        mx = fmaxf(m[r], mx);
        const float ref = mx == -CUDART_INF_F ? 0.f : mx;     // (no score above minus infinity yet: weights of zero, not of no number)
        const float corr = expf(m[r] - ref);
        p[r] = expf(a - ref);
        l[r] = l[r] * corr + p[r];         // (the lane's own keys; summed over the lanes at the end)
        m[r] = mx;
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[r][e] *= corr;
      }
      own_row(newkv[1], key0, vr);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float f[VEC];
        floats(vr[i], f);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float w = __shfl_sync(0xffffffffu, p[r], row_of * LPR + i * SAME);
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[r][e] = fmaf(w, f[e], acc[r][e]);
        }
      }
      if (next < end_key) request(vcache, next, next_page, vr);
      key0 = next;
    }
    // the lanes' shares, then warps -> shared memory
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int mask = 16; mask >= SAME; mask /= 2) l[r] += __shfl_xor_sync(0xffffffffu, l[r], mask);
#pragma unroll
      for (int mask = 16; mask >= LPR; mask /= 2)
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[r][e] += __shfl_xor_sync(0xffffffffu, acc[r][e], mask);
      float* w = Wp + (warp * R + r) * WS;
      if (row_of == 0)
#pragma unroll
        for (int e = 0; e < VEC; ++e) w[dim0 + e] = acc[r][e];
      if (lane == 0) {
        w[HD] = m[r];
        w[HD + 1] = l[r];
      }
    }
    __syncthreads();
    decode_fold_warps<T, (HD + 63) / 64>(Wp, R, rows, HD, seq, kvh * g + h0, nh, split, n_splits, out, ldo, part_o, part_ml);
  }
}

}  // namespace edgelm
