// Attention of many new tokens of a float32 model over its paged float32 keys and values on the tensor cores: causal, grouped heads,
// float32 softmax, float32 output.  Every operand of a product goes as the sum of three bfloat16 terms (8 + 8 + 8 of its 24 mantissa bits)
// and six of the nine products of terms are computed, all but those under 2^-25 of the whole (mma_split.cuh, gemm_split.cu):
//
//   S = Q K^T, O = P V:   1.1 | 1.2 + 2.1 + 2.2 + 1.3 + 3.1      the cross terms first, while the sum they join is small
//
// The tensor cores cut sums off below their last place, so a sum never runs on: a score takes head size / 16 leading products, and a page's
// 64 weighted values are a sum of their own (4 leading products), which joins the running output rounded to nearest.
//
// grid (query tile, query head); a block of 4 warps times NG groups owns 64 consecutive new tokens of one sequence for one head, 16
// rows a warp; the groups take the pages in turn and are merged at the end, in order.  A group's threads bring a page by 16-byte cp.async
// while they multiply the one before, then write its terms into padded rows (ldmatrix) that all its warps read.  Bound by the longest tile's
// chain of pages (two warps a scheduler, 384 MMAs and 800 other instructions a page each; ncu, 1,500 tokens, 9 heads of 64: tensor pipe active 52 % of
// the time on the busiest SM, 30 on average).  On the CUDA cores and here, 9 heads of 64 over
// 3, us: prompts of 61, 381 and 701 tokens 125 and 40.6; one of 1,500 344 and 100; 8 heads of 128, 333 and 200 tokens 98 and 57; one of 17
// 15 and 15.  Distance from float64 (2-norm) 1.5e-7 against 3.6e-7 at 1,500 keys, 8.7e-8 against 1.3e-7 at 17.  Values that are mostly positive (mean
// 3, deviation 1) under scores of deviation 4, whose products are cut off in one direction: 2.2e-7 against 1.5e-7 at 64 keys, 3.2e-7 against 2.6e-7 at 300,
// 3.6e-7 against 9.1e-7 at 1,500.
// A key or value that is no finite number, or rounds to none in bfloat16, shows in its last term; a tile that met one is computed again in plain
// multiply-adds, so that it reaches the rows that see it as it does on the CUDA cores, and no others (looking takes 0 to 2 % of the time).
#include <math_constants.h>

#include "mma_split.cuh"

namespace edgelm {

constexpr int AF_WARPS = 4, AF_ROWS = 16 * AF_WARPS;

template <int HDT> constexpr int af_group_bytes() { return 2 * PAGE * HDT * 16 * 4 + 6 * PAGE * (HDT * 16 + 8) * 2; }

// c += the products of A's and B's terms: the cross terms only, or the leading one
__device__ __forceinline__ void af_cross(float* c, const uint32_t (*a)[4], const uint32_t (*b)[2]) {
  constexpr int TA[5] = {2, 0, 1, 1, 0}, TB[5] = {0, 2, 1, 0, 1};
#pragma unroll
  for (int p = 0; p < 5; ++p) sp_mma(c, a[TA[p]][0], a[TA[p]][1], a[TA[p]][2], a[TA[p]][3], b[TB[p]][0], b[TB[p]][1]);
}

// A tile whose keys or values hold a number without bfloat16 terms, in plain multiply-adds: a warp a row, a lane a key, then hd / 32 dimensions.
__device__ __noinline__ void af_plain_tile(const float* q, int ldq, float* out, int ldo, const float* kcache, const float* vcache, const int32_t* pages, int tok0,
                                           int ntok, int pos0, int nkv, int kvh, int head, int hd, float scale) {
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < ntok; r += blockDim.x >> 5) {
    const float* qr = q + (size_t)(tok0 + r) * ldq + head * hd;
    const int limit = pos0 + r;
    float m = -CUDART_INF_F, l = 0.f, o[4] = {};
    for (int key0 = 0; key0 <= limit; key0 += 32) {
      const int page = pages[key0 / PAGE], n = min(32, limit + 1 - key0);
      const size_t at = (((size_t)max(page, 0) * nkv + kvh) * PAGE + key0 % PAGE) * hd;
      float s = 0.f;
      if (lane < n && page >= 0)
        for (int d = 0; d < hd; ++d) s = fmaf(qr[d], kcache[at + lane * hd + d], s);
      s = lane < n ? s * scale : -CUDART_INF_F;
      const float mx = fmaxf(m, warp_max(s)), ref = mx == -CUDART_INF_F ? 0.f : mx, corr = expf(m - ref), p = expf(s - ref);
      l = l * corr + p;
      m = mx;
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] *= corr;
      for (int i = 0; i < n; ++i) {
        const float w = __shfl_sync(0xffffffffu, p, i);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (32 * c < hd) o[c] = fmaf(w, page >= 0 ? vcache[at + i * hd + 32 * c + lane] : 0.f, o[c]);
      }
    }
    l = warp_sum(l);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (32 * c < hd) out[(size_t)(tok0 + r) * ldo + head * hd + 32 * c + lane] = o[c] / l;
  }
}

template <int HDT, int NG>
__global__ void __launch_bounds__(AF_WARPS * 32 * NG)
attn_prefill_f32_kernel(const float* __restrict__ q, int ldq, float* __restrict__ out, int ldo, const float* __restrict__ kcache,
                        const float* __restrict__ vcache, const int32_t* __restrict__ page_table, int table_stride,
                        const int32_t* __restrict__ seq_slot, const int32_t* __restrict__ tile_seq, const int32_t* __restrict__ tile_tok0,
                        const int32_t* __restrict__ tile_ntok, const int32_t* __restrict__ tile_pos0, int nh, int nkv, float scale) {
  constexpr int HD = HDT * 16, PITCH = HD + 8, PLANE = PAGE * PITCH, PIECES = HD / 4;
  extern __shared__ __align__(16) uint8_t af_raw[];
  const int group = threadIdx.x / (AF_WARPS * 32), gtid = threadIdx.x % (AF_WARPS * 32);
  uint8_t* mine = af_raw + (size_t)group * af_group_bytes<HDT>();
  float* raw = reinterpret_cast<float*>(mine);                                          // [K: 64 x HD | V: 64 x HD]
  __nv_bfloat16* planes = reinterpret_cast<__nv_bfloat16*>(mine + 2 * PAGE * HD * 4);   // [K's three terms | V's three terms], 64 x PITCH each

  const int tile = gridDim.x - 1 - blockIdx.x, head = blockIdx.y, kvh = head / (nh / nkv);   // (the last tiles see the most keys: first)
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % AF_WARPS, gid = lane >> 2, tig = lane & 3;
  const int seq = tile_seq[tile], tok0 = tile_tok0[tile], ntok = tile_ntok[tile], pos0 = tile_pos0[tile];
  const int32_t* pages = page_table + (size_t)seq_slot[seq] * table_stride;
  const int nkeys = pos0 + ntok, n_pages = (nkeys + PAGE - 1) / PAGE;
  const int rowA = warp * 16 + gid, rowB = rowA + 8;
  const int limA = rowA < ntok ? pos0 + rowA : -1, limB = rowB < ntok ? pos0 + rowB : -1;    // the last key a row sees; -1: no such row
  const int warp_limit = warp * 16 < ntok ? pos0 + min(ntok - 1, warp * 16 + 15) : -1, warp_min_limit = warp * 16 < ntok ? pos0 + warp * 16 : -1;
  const float scale2 = scale * 1.4426950408889634f;

  auto load_page = [&](int pg) {
    const int page = max(pages[pg], 0), valid = pages[pg] >= 0 ? min(PAGE, nkeys - pg * PAGE) : 0;
    const float* kp = kcache + ((size_t)page * nkv + kvh) * PAGE * HD;
    const float* vp = vcache + ((size_t)page * nkv + kvh) * PAGE * HD;
    for (int i = gtid; i < PAGE * PIECES; i += AF_WARPS * 32) {
      const int bytes = i / PIECES < valid ? 16 : 0;   // (what lies behind the last key is not this sequence's: zeros)
      sp_cp16(sp_smem(raw + i * 4), kp + i * 4, bytes);
      sp_cp16(sp_smem(raw + PAGE * HD + i * 4), vp + i * 4, bytes);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto group_sync = [&]() {
    if (NG == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(AF_WARPS * 32) : "memory");
  };

  uint32_t qa[HDT][3][4];
  {
    const float* qA = q + (size_t)(tok0 + min(rowA, ntok - 1)) * ldq + head * HD;
    const float* qB = q + (size_t)(tok0 + min(rowB, ntok - 1)) * ldq + head * HD;
#pragma unroll
    for (int ks = 0; ks < HDT; ++ks)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 v = *reinterpret_cast<const float2*>((j & 1 ? qB : qA) + ks * 16 + tig * 2 + (j >> 1) * 8);
        sp_split(v.x, v.y, qa[ks][0][j], qa[ks][1][j], qa[ks][2][j]);
      }
  }
  float o[HD / 8][4];
#pragma unroll
  for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float mA = -CUDART_INF_F, mB = -CUDART_INF_F, lA = 0.f, lB = 0.f;     // (maxima of the scores as they come; sums of this lane's keys)

  uint32_t nothing = 0;      // the sum of 0 x the last terms: not a number from the first key or value on whose first term is none
  if (group < n_pages) load_page(group);
  for (int pg = group; pg < n_pages; pg += NG) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    group_sync();            // the page is there for all, the terms of the one before are read
    for (int i = gtid; i < 2 * PAGE * PIECES; i += AF_WARPS * 32) {
      const int r = i / PIECES, c = i % PIECES;        // rows 64 ..: V's
      const float4 v = *reinterpret_cast<const float4*>(raw + i * 4);
      uint2 t1, t2, t3;
      sp_split(v.x, v.y, t1.x, t2.x, t3.x);
      sp_split(v.z, v.w, t1.y, t2.y, t3.y);
      __nv_bfloat16* dst = planes + (r / PAGE) * 3 * PLANE + (r % PAGE) * PITCH + c * 4;
      *reinterpret_cast<uint2*>(dst) = t1;
      *reinterpret_cast<uint2*>(dst + PLANE) = t2;
      *reinterpret_cast<uint2*>(dst + 2 * PLANE) = t3;
      asm("{\n\tfma.rn.bf16x2 %0, %1, %3, %0;\n\tfma.rn.bf16x2 %0, %2, %3, %0;\n\t}" : "+r"(nothing) : "r"(t3.x), "r"(t3.y), "r"(0u));
    }
    group_sync();
    if (pg + NG < n_pages) load_page(pg + NG);
    if (pg * PAGE > warp_limit) continue;              // no row of this warp sees this page
    float s[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
      uint32_t kb[HDT][3][2];
#pragma unroll
      for (int ks = 0; ks < HDT; ks += 2)
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const int mi = lane >> 3;
          sp_ldmatrix_x4(sp_smem(planes + t * PLANE + (nt * 8 + (lane & 7)) * PITCH + (ks + (mi >> 1)) * 16 + (mi & 1) * 8), kb[ks][t][0], kb[ks][t][1],
                         kb[ks + 1][t][0], kb[ks + 1][t][1]);
        }
#pragma unroll
      for (int ks = 0; ks < HDT; ++ks) af_cross(s[nt], qa[ks], kb[ks]);
#pragma unroll
      for (int ks = 0; ks < HDT; ++ks) sp_mma(s[nt], qa[ks][0][0], qa[ks][0][1], qa[ks][0][2], qa[ks][0][3], kb[ks][0][0], kb[ks][0][1]);
    }
    if (pg * PAGE + PAGE - 1 > warp_min_limit) {
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const int key = pg * PAGE + nt * 8 + tig * 2;
        if (key > limA) s[nt][0] = -CUDART_INF_F;
        if (key + 1 > limA) s[nt][1] = -CUDART_INF_F;
        if (key > limB) s[nt][2] = -CUDART_INF_F;
        if (key + 1 > limB) s[nt][3] = -CUDART_INF_F;
      }
    }
    float nmA = mA, nmB = mB;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      nmA = fmaxf(nmA, fmaxf(s[nt][0], s[nt][1]));
      nmB = fmaxf(nmB, fmaxf(s[nt][2], s[nt][3]));
    }
    nmA = fmaxf(nmA, __shfl_xor_sync(0xffffffffu, nmA, 1));
    nmA = fmaxf(nmA, __shfl_xor_sync(0xffffffffu, nmA, 2));
    nmB = fmaxf(nmB, __shfl_xor_sync(0xffffffffu, nmB, 1));
    nmB = fmaxf(nmB, __shfl_xor_sync(0xffffffffu, nmB, 2));
    const float refA = nmA == -CUDART_INF_F ? 0.f : nmA, refB = nmB == -CUDART_INF_F ? 0.f : nmB;   // (a row that sees no key yet)
    const float corrA = exp2f((mA - refA) * scale2), corrB = exp2f((mB - refB) * scale2);
    mA = nmA;
    mB = nmB;
    float sumA = 0.f, sumB = 0.f;
    uint32_t pa[4][3][4];
#pragma unroll
    for (int kt = 0; kt < 4; ++kt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {                    // rows A, B of keys 2 tig, then of keys 2 tig + 8
        float* v = s[2 * kt + (j >> 1)] + (j & 1) * 2;
        v[0] = exp2f((v[0] - (j & 1 ? refB : refA)) * scale2);
        v[1] = exp2f((v[1] - (j & 1 ? refB : refA)) * scale2);
        if (j & 1) sumB += v[0] + v[1];
        else sumA += v[0] + v[1];
        sp_split(v[0], v[1], pa[kt][0][j], pa[kt][1][j], pa[kt][2][j]);
      }
    lA = lA * corrA + sumA;
    lB = lB * corrB + sumB;
    const __nv_bfloat16* vs = planes + 3 * PLANE;
#pragma unroll
    for (int dt = 0; dt < HD / 8; dt += 2) {
      float c[2][4] = {};
      uint32_t first[4][4];
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        uint32_t vb[2][3][2];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const int mi = lane >> 3;
          sp_ldmatrix_x4_trans(sp_smem(vs + t * PLANE + (kt * 16 + (mi & 1) * 8 + (lane & 7)) * PITCH + (dt + (mi >> 1)) * 8), vb[0][t][0], vb[0][t][1],
                               vb[1][t][0], vb[1][t][1]);
        }
        af_cross(c[0], pa[kt], vb[0]);
        af_cross(c[1], pa[kt], vb[1]);
        first[kt][0] = vb[0][0][0]; first[kt][1] = vb[0][0][1]; first[kt][2] = vb[1][0][0]; first[kt][3] = vb[1][0][1];
      }
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        sp_mma(c[0], pa[kt][0][0], pa[kt][0][1], pa[kt][0][2], pa[kt][0][3], first[kt][0], first[kt][1]);
        sp_mma(c[1], pa[kt][0][0], pa[kt][0][1], pa[kt][0][2], pa[kt][0][3], first[kt][2], first[kt][3]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        o[dt + h][0] = fmaf(o[dt + h][0], corrA, c[h][0]);
        o[dt + h][1] = fmaf(o[dt + h][1], corrA, c[h][1]);
        o[dt + h][2] = fmaf(o[dt + h][2], corrB, c[h][2]);
        o[dt + h][3] = fmaf(o[dt + h][3], corrB, c[h][3]);
      }
    }
  }
  if (__syncthreads_or((nothing & 0x7fffu) > 0x7f80u || (nothing & 0x7fff0000u) > 0x7f800000u)) {
    af_plain_tile(q, ldq, out, ldo, kcache, vcache, pages, tok0, ntok, pos0, nkv, kvh, head, HD, scale);
    return;
  }
  lA += __shfl_xor_sync(0xffffffffu, lA, 1);
  lA += __shfl_xor_sync(0xffffffffu, lA, 2);
  lB += __shfl_xor_sync(0xffffffffu, lB, 1);
  lB += __shfl_xor_sync(0xffffffffu, lB, 2);
  if (NG > 1) {
    constexpr int MP = HD + 2;
    float* mg = reinterpret_cast<float*>(af_raw);      // [NG - 1][64 rows][HD + 2]: groups 1 ..'s output, maximum, sum
    if (group > 0) {
      float* a = mg + ((size_t)(group - 1) * AF_ROWS + rowA) * MP;
      float* b = mg + ((size_t)(group - 1) * AF_ROWS + rowB) * MP;
#pragma unroll
      for (int dt = 0; dt < HD / 8; ++dt) {
        a[dt * 8 + tig * 2] = o[dt][0];
        a[dt * 8 + tig * 2 + 1] = o[dt][1];
        b[dt * 8 + tig * 2] = o[dt][2];
        b[dt * 8 + tig * 2 + 1] = o[dt][3];
      }
      if (tig == 0) {
        a[HD] = mA;
        a[HD + 1] = lA;
        b[HD] = mB;
        b[HD + 1] = lB;
      }
    }
    __syncthreads();
    if (group > 0) return;
    for (int g = 1; g < NG; ++g) {
      const float* a = mg + ((size_t)(g - 1) * AF_ROWS + rowA) * MP;
      const float* b = mg + ((size_t)(g - 1) * AF_ROWS + rowB) * MP;
      const float nmA = fmaxf(mA, a[HD]), nmB = fmaxf(mB, b[HD]);
      const float refA = nmA == -CUDART_INF_F ? 0.f : nmA, refB = nmB == -CUDART_INF_F ? 0.f : nmB;
      const float fA0 = exp2f((mA - refA) * scale2), fA1 = exp2f((a[HD] - refA) * scale2);
      const float fB0 = exp2f((mB - refB) * scale2), fB1 = exp2f((b[HD] - refB) * scale2);
      lA = lA * fA0 + a[HD + 1] * fA1;
      lB = lB * fB0 + b[HD + 1] * fB1;
      mA = nmA;
      mB = nmB;
#pragma unroll
      for (int dt = 0; dt < HD / 8; ++dt) {
        o[dt][0] = o[dt][0] * fA0 + a[dt * 8 + tig * 2] * fA1;
        o[dt][1] = o[dt][1] * fA0 + a[dt * 8 + tig * 2 + 1] * fA1;
        o[dt][2] = o[dt][2] * fB0 + b[dt * 8 + tig * 2] * fB1;
        o[dt][3] = o[dt][3] * fB0 + b[dt * 8 + tig * 2 + 1] * fB1;
      }
    }
  }
#pragma unroll
  for (int dt = 0; dt < HD / 8; ++dt) {
    const int d = head * HD + dt * 8 + tig * 2;
    if (rowA < ntok) *reinterpret_cast<float2*>(out + (size_t)(tok0 + rowA) * ldo + d) = make_float2(o[dt][0] / lA, o[dt][1] / lA);
    if (rowB < ntok) *reinterpret_cast<float2*>(out + (size_t)(tok0 + rowB) * ldo + d) = make_float2(o[dt][2] / lB, o[dt][3] / lB);
  }
}

template <int HDT, int NG>
static int launch_prefill_f32(const float* q, int ldq, float* out, int ldo, const float* kc, const float* vc, const int32_t* page_table, int table_stride,
                              const int32_t* seq_slot, const int32_t* tile_seq, const int32_t* tile_tok0, const int32_t* tile_ntok, const int32_t* tile_pos0,
                              int n_tiles, int nh, int nkv, float scale, cudaStream_t stream) {
  constexpr size_t pages = (size_t)NG * af_group_bytes<HDT>(), merge = (size_t)(NG - 1) * AF_ROWS * (HDT * 16 + 2) * 4, smem = pages > merge ? pages : merge;
  auto kern = attn_prefill_f32_kernel<HDT, NG>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  EL_REFUSE(e == cudaSuccess, "attn_prefill_f32: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
  kern<<<dim3(n_tiles, nh), AF_WARPS * 32 * NG, smem, stream>>>(q, ldq, out, ldo, kc, vc, page_table, table_stride, seq_slot, tile_seq, tile_tok0, tile_ntok,
                                                                tile_pos0, nh, nkv, scale);
  return 0;
}

}  // namespace edgelm

using namespace edgelm;

// Tokens per tile that the host must cut sequences into for this kernel.
extern "C" int edgelm_attn_prefill_f32_tile_tokens() { return AF_ROWS; }

extern "C" int edgelm_attn_prefill_f32_takes(int hd) { return hd == 32 || hd == 64 || hd == 96 || hd == 128 ? 1 : 0; }

// q [tokens][nh hd] (row pitch ldq), out [tokens][nh hd] (row pitch ldo), the cache's pages [page][kv head][64][hd], all float32; `seq_slot`
// maps a step's sequence to its row of the page table; tiles of at most 64 new tokens of one sequence each.  Two warp groups a block where
// both find room (head sizes up to 64).
extern "C" int edgelm_attn_prefill_f32(const float* q, int ldq, float* out, int ldo, const float* kcache, const float* vcache, const int32_t* page_table,
                                       int table_stride, const int32_t* seq_slot, const int32_t* tile_seq, const int32_t* tile_tok0, const int32_t* tile_ntok,
                                       const int32_t* tile_pos0, int n_tiles, int nh, int nkv, int hd, float scale, cudaStream_t stream) {
  if (n_tiles == 0) return 0;
  EL_REFUSE(n_tiles > 0 && nh > 0 && nkv > 0 && nh % nkv == 0 && nh <= 65535, "attn_prefill_f32: %d query heads over %d key/value heads", nh, nkv);
  EL_REFUSE(edgelm_attn_prefill_f32_takes(hd), "attn_prefill_f32: head size %d (takes 32, 64, 96, 128)", hd);
  EL_REFUSE(scale > 0.f, "attn_prefill_f32: the scale must be positive");
  EL_REFUSE(ldq % 2 == 0 && ldo % 2 == 0 && (uintptr_t)q % 8 == 0 && (uintptr_t)out % 8 == 0, "attn_prefill_f32: rows must be 8-byte aligned");
  EL_REFUSE((uintptr_t)kcache % 16 == 0 && (uintptr_t)vcache % 16 == 0, "attn_prefill_f32: keys and values must be 16-byte aligned");
  int rc = 0;
#define EL_AF(H, G) rc = launch_prefill_f32<H, G>(q, ldq, out, ldo, kcache, vcache, page_table, table_stride, seq_slot, tile_seq, tile_tok0, tile_ntok, tile_pos0, n_tiles, nh, nkv, scale, stream)
  if (hd == 32) EL_AF(2, 2);
  else if (hd == 64) EL_AF(4, 2);
  else if (hd == 96) EL_AF(6, 1);
  else EL_AF(8, 1);
#undef EL_AF
  if (rc) return rc;
  EL_LAUNCH_CHECK("attn_prefill_f32");
  return 0;
}
