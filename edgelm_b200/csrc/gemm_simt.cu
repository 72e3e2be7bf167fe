// y = a . W^T with float32 accumulation on the CUDA cores (FFMA): the whole of the true
// 32-bit path, and the any-size fallback of the bfloat16 path.
//
//   a   [M, K]  float or bfloat16, row stride lda
//   W   [N, K]  float or bfloat16, row-major as a checkpoint stores it (out, in)
// Epilogues:
//   EPI_STORE     out[M, N] (float or bfloat16)             = acc
//   EPI_RESIDUAL  out[M, N] (float) = residual[M, N] + acc   (out may be residual itself)
//   EPI_SWIGLU    out[M, N] = silu(acc_gate) * acc_up with a second weight W2 (up) of W's shape
//   EPI_RELU2     out[M, N] = max(acc, 0)^2
// Three kernels: register tiles of 8x8 outputs a thread for float32 operands in 16-byte pieces (the 32-bit path's products of
// more than 16 rows), a 64x64 tile for any size and alignment, and a one-warp-per-output-column kernel for a few
// rows (decode), which reads every weight once.  Each output element is summed over k in an
// order that depends on the sizes alone (in the last two: on K alone), never on the row's place in the batch.
#include <cooperative_groups.h>

#include "common.cuh"

namespace edgelm {

enum : int { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_SWIGLU = 2, EPI_RELU2 = 4 };

__device__ __forceinline__ float silu_f32(float z) { return z / (1.0f + expf(-z)); }

template <int EPI, typename TOut>
__device__ __forceinline__ void epilogue_store(TOut* out, const float* residual, size_t idx, float acc, float acc2) {
  if (EPI == EPI_STORE) out[idx] = from_f32<TOut>(acc);
  if (EPI == EPI_RESIDUAL) out[idx] = from_f32<TOut>(residual[idx] + acc);
  if (EPI == EPI_SWIGLU) out[idx] = from_f32<TOut>(silu_f32(acc) * acc2);
  if (EPI == EPI_RELU2) out[idx] = from_f32<TOut>(fmaxf(acc, 0.f) * fmaxf(acc, 0.f));
}

// ------------------------------------------------------------------ tiled kernel
constexpr int BM = 64, BN = 64, BK = 16, PADT = 4;

template <typename TA, typename TW, int EPI, typename TOut>
__global__ void __launch_bounds__(256)
gemm_tile_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, const TW* __restrict__ W2,
                 TOut* out, int ldo, const float* residual, int M, int N, int K) {
  __shared__ float As[BK][BM + PADT];
  __shared__ float Ws[BK][BN + PADT];
  __shared__ float Ws2[EPI == EPI_SWIGLU ? BK : 1][BN + PADT];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4] = {}, acc2[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * 256, r = e >> 4, k = e & 15;
      const int gk = k0 + k;
      As[k][r] = (m0 + r < M && gk < K) ? to_f32(A[(size_t)(m0 + r) * lda + gk]) : 0.f;
      const bool ok = (n0 + r < N && gk < K);
      Ws[k][r] = ok ? to_f32(W[(size_t)(n0 + r) * K + gk]) : 0.f;
      if (EPI == EPI_SWIGLU) Ws2[k][r] = ok ? to_f32(W2[(size_t)(n0 + r) * K + gk]) : 0.f;
    }
    __syncthreads();
    // a tile's products are summed on their own and then added to the running sums: the rounding error of a long
    // row of products grows with the number of tiles and the tile's length, not with their product
    float part[4][4] = {}, part2[4][4] = {};
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], b[4], b2[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[k][tx * 4 + j];
      if (EPI == EPI_SWIGLU) {
#pragma unroll
        for (int j = 0; j < 4; ++j) b2[j] = Ws2[k][tx * 4 + j];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          part[i][j] = fmaf(a[i], b[j], part[i][j]);
          if (EPI == EPI_SWIGLU) part2[i][j] = fmaf(a[i], b2[j], part2[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] += part[i][j];
        if (EPI == EPI_SWIGLU) acc2[i][j] += part2[i][j];
      }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) epilogue_store<EPI, TOut>(out, residual, (size_t)m * ldo + n, acc[i][j], acc2[i][j]);
    }
  }
}

// ------------------------------------------------------------------ float32 register tiles
// A block computes 8 TY x 8 TX outputs (a SwiGLU's gate and up columns side by side: 4 TX columns of either weight).  KG groups of
// TY TX threads share K, and a cluster of CS blocks shares it again; a thread keeps 8 x 8 sums, rows ty + TY i and columns
// tx + TX j, reading four k of a row at a time (16 reads of 16 bytes for 256 multiply-adds).  The multiply-adds are packed pairs
// (`fma.rn.f32x2`: even and odd k in sums of their own; single ones waited for register ports).  Both operands come by
// cp.async, S_STAGES stages of 16 k a group, a row's four pieces of 16 bytes exchanged by
// the row's number so that eight neighbouring rows' reads lie in different banks.  After S_FLUSH stages the pairs join running sums
// that lie in shared memory (a thread's own 64): the rounding error of a long row of products grows with the number of runs and the
// run's length, not with their product.  (Two stages, runs of 16 products a pair: 1.13e-7 of the result at K 576, 1.82e-7 at K 2560, the
// any-size kernel's 1.34e-7 and 2.41e-7; runs twice as long are 7 % faster and less exact than it at K under 300.)  The sums of groups and
// blocks are added in the order of K.  Measured beside the any-size kernel: 2,000 rows, N 1000, K 2560 680 -> 326 us; 300 rows, N 576,
// K 2560 173 -> 47 us; 24 rows, N 960, K 2560 169 -> 10 us.  Bound by the chains of two warps a scheduler, which is what 64
// pairs of sums leave room for (1,143 rows, N 1536, K 576: the multiply-adds' pipe active 52 %, issue slots 45 %, memory 1 %).
constexpr int SK = 16, S_STAGES = 3, S_FLUSH = 2;

__device__ __forceinline__ void cp_async16(unsigned dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

template <int THREADS>
__device__ __forceinline__ void group_sync(int group) {
  if (THREADS == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(THREADS) : "memory");
}

using pair_t = unsigned long long;       // two float32
__device__ __forceinline__ void fma_pair(pair_t& c, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ float pair_sum(pair_t c) { return __uint_as_float((uint32_t)c) + __uint_as_float((uint32_t)(c >> 32)); }

template <int EPI>
__device__ __forceinline__ void epilogue_put(float* out, float residual, float acc, float acc2) {
  if (EPI == EPI_STORE) *out = acc;
  if (EPI == EPI_RESIDUAL) *out = residual + acc;
  if (EPI == EPI_SWIGLU) *out = silu_f32(acc) * acc2;
  if (EPI == EPI_RELU2) *out = fmaxf(acc, 0.f) * fmaxf(acc, 0.f);
}

template <int TY, int TX, int KG> constexpr size_t sgemm_smem() {
  constexpr size_t ring = (size_t)KG * S_STAGES * 8 * (TY + TX) * SK * 4, sums = (size_t)TY * TX * KG * 64 * 4, red = (size_t)KG * 8 * TY * (8 * TX + 8) * 4;
  return ring + sums > red ? ring + sums : red;
}

template <int TY, int TX, int KG, int EPI>
__global__ void __launch_bounds__(TY * TX * KG)
sgemm_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, const float* __restrict__ W2, float* out, int ldo,
             const float* residual, int M, int N, int K, int CS) {
  extern __shared__ __align__(128) float sm[];
  constexpr int GT = TY * TX, BM = 8 * TY, BN = 8 * TX, NOUT = EPI == EPI_SWIGLU ? BN / 2 : BN, STAGE = (BM + BN) * SK;
  constexpr int PIECES = (BM + BN) * 4 / GT, RP = BN + 8;
  pdl_launch_dependents();
  pdl_wait();
  const int g = threadIdx.x / GT, t = threadIdx.x % GT, lane = t & 31, w = t >> 5;
  // (a read of 16 bytes a lane takes two clocks where neighbouring lanes share their row or two rows alternate, four elsewhere)
  const int tx = (w % (TX / 8)) * 8 + (lane >> 1 & 7), ty = (w / (TX / 8)) * 4 + (lane & 1) + (lane >> 4) * 2;
  const int rank = blockIdx.x % CS, m0 = blockIdx.y * BM, n0 = (blockIdx.x / CS) * NOUT;
  const int chunks = (K + SK - 1) / SK, parts = KG * CS, part_no = rank * KG + g;
  const int c_end = (int)((long long)chunks * (part_no + 1) / parts), c_begin = (int)((long long)chunks * part_no / parts);
  float* ring = sm + (size_t)g * S_STAGES * STAGE;
  float4* sums = reinterpret_cast<float4*>(sm + KG * S_STAGES * STAGE) + threadIdx.x;      // [16][threads]
  // this thread's pieces of a stage: row t / 4 + i GT / 4 of the tile's rows of A and then of W, 16 bytes t % 4 of its 64.
  // (rows beyond M or N: the last row again, whose sums are not stored)
  const int kp = (t & 3) * 4, k_end = K - kp;
  const float* src[PIECES];
  unsigned dst0 = (unsigned)__cvta_generic_to_shared(ring) + (t >> 2) * SK * 4;
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int r = (t >> 2) + i * (GT / 4);
    if (r < BM) {
      src[i] = A + (size_t)min(m0 + r, M - 1) * lda + kp + c_begin * SK;
    } else {
      const int c = r - BM;
      const bool up = EPI == EPI_SWIGLU && c >= NOUT;
      src[i] = (up ? W2 : W) + (size_t)min(n0 + (up ? c - NOUT : c), N - 1) * K + kp + c_begin * SK;
    }
  }
  // the next stage's pieces on their way (a stage beyond this group's last: nothing); `src` moves on
  int next = c_begin;
  auto load = [&](int slot) {
    if (next < c_end) {
      const bool there = next * SK < k_end;      // (K is a multiple of 4)
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        const int sw = (((t >> 2) + i * (GT / 4)) >> 1 & 3) * 4;
        cp_async16(dst0 + (slot * STAGE + i * (GT / 4) * SK + (kp ^ sw)) * 4, there ? src[i] : A, there);
        src[i] += SK;
      }
    }
    ++next;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < S_STAGES - 1; ++s) load(s);
  pair_t part[8][8] = {};
  int run = 0, slot = 0;                 // stages since the pairs last joined the sums
  bool kept = false;
  int oa[4], ow[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    oa[k] = ty * SK + (k * 4 ^ (ty >> 1 & 3) * 4);
    ow[k] = (BM + tx) * SK + (k * 4 ^ (tx >> 1 & 3) * 4);
  }
  for (int c = c_begin; c < c_end; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S_STAGES - 2) : "memory");
    group_sync<GT>(g);                   // the stage is there for all; the one computed last is free
    load(slot == 0 ? S_STAGES - 1 : slot - 1);
    if (run == S_FLUSH) {
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        float4 v = kept ? sums[q * GT * KG] : make_float4(0.f, 0.f, 0.f, 0.f);
        const int i = q >> 1, j = (q & 1) * 4;
        v.x += pair_sum(part[i][j]); v.y += pair_sum(part[i][j + 1]); v.z += pair_sum(part[i][j + 2]); v.w += pair_sum(part[i][j + 3]);
        part[i][j] = part[i][j + 1] = part[i][j + 2] = part[i][j + 3] = 0;
        sums[q * GT * KG] = v;
      }
      run = 0;
      kept = true;
    }
    ++run;
    const float* st = ring + slot * STAGE;
    slot = slot == S_STAGES - 1 ? 0 : slot + 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ulonglong2 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(st + oa[k ^ (TY * i / 2 & 3)] + i * TY * SK);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(st + ow[k] + j * TX * SK);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma_pair(part[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma_pair(part[i][j], a[i].y, b.y);
      }
    }
  }
  float acc[8][8];
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const float4 v = kept ? sums[q * GT * KG] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int i = q >> 1, j = (q & 1) * 4;
    acc[i][j] = v.x + pair_sum(part[i][j]);
    acc[i][j + 1] = v.y + pair_sum(part[i][j + 1]);
    acc[i][j + 2] = v.z + pair_sum(part[i][j + 2]);
    acc[i][j + 3] = v.w + pair_sum(part[i][j + 3]);
  }
  if (KG == 1 && CS == 1) {
    // (`out` may be the residual itself: a row's residuals are requested before the row ahead of it is stored, or every load would
    // wait for the store before it)
    float ahead[2][8] = {};
    auto fetch = [&](int i) {
      const int m = m0 + ty + TY * i;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (m < M && n0 + tx + TX * j < N) ahead[i & 1][j] = residual[(size_t)m * ldo + n0 + tx + TX * j];
    };
    if (EPI == EPI_RESIDUAL) fetch(0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + ty + TY * i;
      if (EPI == EPI_RESIDUAL && i < 7) fetch(i + 1);
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < (EPI == EPI_SWIGLU ? 4 : 8); ++j) {
        const int n = n0 + tx + TX * j;
        if (n < N) epilogue_put<EPI>(out + (size_t)m * ldo + n, ahead[i & 1][j], acc[i][j], EPI == EPI_SWIGLU ? acc[i][(j + 4) & 7] : 0.f);
      }
    }
    return;
  }
  // partial tiles into shared memory (over the rings and sums), the groups' added in every block, then the blocks'
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) sm[(g * BM + ty + TY * i) * RP + tx + TX * j] = acc[i][j];
  __syncthreads();
  if (KG > 1) {
    for (int e = threadIdx.x; e < BM * BN; e += GT * KG) {
      float* p = sm + e / BN * RP + e % BN;
      float v = p[0];
#pragma unroll
      for (int q = 1; q < KG; ++q) v += p[q * BM * RP];
      p[0] = v;
    }
    __syncthreads();
  }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  if (CS > 1) cluster.sync();
  const int r_begin = BM * rank / CS, r_end = BM * (rank + 1) / CS;
  constexpr int AHEAD = 4;               // (residuals requested together: `out` may be the residual itself)
  for (int e0 = r_begin * NOUT + threadIdx.x; e0 < r_end * NOUT; e0 += AHEAD * GT * KG) {
    float ahead[AHEAD] = {};
    auto at = [&](int e) { return (size_t)(m0 + e / NOUT) * ldo + n0 + e % NOUT; };
    auto there = [&](int e) { return e < r_end * NOUT && m0 + e / NOUT < M && n0 + e % NOUT < N; };
    if (EPI == EPI_RESIDUAL)
#pragma unroll
      for (int x = 0; x < AHEAD; ++x)
        if (there(e0 + x * GT * KG)) ahead[x] = residual[at(e0 + x * GT * KG)];
#pragma unroll
    for (int x = 0; x < AHEAD; ++x) {
      const int e = e0 + x * GT * KG;
      if (!there(e)) continue;
      float v = 0.f, v2 = 0.f;
      for (int q = 0; q < CS; ++q) {
        const float* p = (CS > 1 ? cluster.map_shared_rank(sm, q) : sm) + e / NOUT * RP + e % NOUT;
        v += p[0];
        if (EPI == EPI_SWIGLU) v2 += p[NOUT];
      }
      epilogue_put<EPI>(out + at(e), ahead[x], v, v2);
    }
  }
  if (CS > 1) cluster.sync();            // (no block leaves while another reads its sums)
}

template <int TY, int TX, int KG, int EPI>
int launch_sgemm(const float* a, int lda, const float* w, const float* w2, float* out, int ldo, const float* residual, int M, int N, int K,
                 int CS, cudaStream_t stream) {
  constexpr int NOUT = EPI == EPI_SWIGLU ? 4 * TX : 8 * TX;
  constexpr size_t smem = sgemm_smem<TY, TX, KG>();
  auto* kern = sgemm_kernel<TY, TX, KG, EPI>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  EL_REFUSE(e == cudaSuccess, "gemm_simt: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((N + NOUT - 1) / NOUT * CS), (unsigned)((M + 8 * TY - 1) / (8 * TY)));
  cfg.blockDim = dim3(TY * TX * KG);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)CS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (pdl_enabled() & 1) ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kern, a, lda, w, w2, out, ldo, residual, M, N, K, CS);
  return 0;
}

// The tile and the number of blocks that share K: what takes the least time by a count of waves of one block an SM (a block's
// registers and rings fill it; clusters of eight find room for 120 blocks).  The constants are measured: a stage of all of a block's
// groups takes 1.83, 1.95 and 2.1 us in the three tiles (one wave, K 960: 110, 31 and 18.6 us), a wave 2.5 us beside them, and 2.5 more
// where blocks exchange sums.  24 rows, N 960, K 960: 12.4, 9.2 and 6.5 us with the middle tile in clusters of 4, of 8, and the small
// one of 8; N 2560, K 960 (SwiGLU): 33, 19.5 and 23.7 us with the middle tile, the small one alone and in clusters of 4.
template <int EPI>
int launch_sgemm_best(const float* a, int lda, const float* w, const float* w2, float* out, int ldo, const float* residual, int M, int N,
                      int K, cudaStream_t stream) {
  const int chunks = (K + SK - 1) / SK;
  struct Tile { int rows, columns, groups; float stage_us; };
  constexpr Tile tiles[3] = {{128, 128, 1, 1.83f}, {64, 64, 4, 1.95f}, {32, 64, 8, 2.1f}};
  float best = 0.f;
  int best_t = -1, best_cs = 1;
  for (int t = 0; t < 3; ++t)
    for (int cs = 1; cs <= (t == 0 ? 1 : 8) && (cs == 1 || 2 * chunks >= tiles[t].groups * cs); cs *= 2) {
      const int columns = tiles[t].columns / (EPI == EPI_SWIGLU ? 2 : 1), room = cs == 8 ? 120 : cs == 4 ? 136 : 148;
      const long long blocks = (long long)((M + tiles[t].rows - 1) / tiles[t].rows) * ((N + columns - 1) / columns) * cs;
      const int stages = (chunks + tiles[t].groups * cs - 1) / (tiles[t].groups * cs);
      const float us = (float)((blocks + room - 1) / room) * ((float)stages * tiles[t].stage_us + 2.5f + (cs > 1 ? 2.5f : 0.f));
      if (best_t < 0 || us < best) { best = us; best_t = t; best_cs = cs; }
    }
  if (best_t == 0) return launch_sgemm<16, 16, 1, EPI>(a, lda, w, w2, out, ldo, residual, M, N, K, best_cs, stream);
  if (best_t == 1) return launch_sgemm<8, 8, 4, EPI>(a, lda, w, w2, out, ldo, residual, M, N, K, best_cs, stream);
  return launch_sgemm<4, 8, 8, EPI>(a, lda, w, w2, out, ldo, residual, M, N, K, best_cs, stream);
}

// ------------------------------------------------------------------ few-rows kernel
template <typename T, int VEC> struct VecLoad;
template <> struct VecLoad<float, 4> {
  static __device__ __forceinline__ void load(const float* p, float* o) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};
template <> struct VecLoad<float, 1> {
  static __device__ __forceinline__ void load(const float* p, float* o) { o[0] = *p; }
};
template <> struct VecLoad<__nv_bfloat16, 8> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* o) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};
template <> struct VecLoad<__nv_bfloat16, 1> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* o) { o[0] = __bfloat162float(*p); }
};

constexpr int GEMV_ROWS = 8;  // rows of `a` that one pass over a weight row serves

template <typename TA, typename TW, int EPI, typename TOut, int VA, int VW>
__global__ void __launch_bounds__(256)
gemv_rows_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, const TW* __restrict__ W2,
                 TOut* out, int ldo, const float* residual, int M, int N, int K) {
  static_assert(VA == VW, "one vector width for both operands");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * 8 + warp;
  const int m0 = blockIdx.y * GEMV_ROWS;
  if (n >= N) return;
  const int rows = min(GEMV_ROWS, M - m0);
  float acc[GEMV_ROWS] = {}, acc2[GEMV_ROWS] = {};
  const TW* wrow = W + (size_t)n * K;
  const TW* wrow2 = EPI == EPI_SWIGLU ? W2 + (size_t)n * K : nullptr;
  for (int k = lane * VW; k < K; k += 32 * VW) {
    float w[VW], w2[VW];
    VecLoad<TW, VW>::load(wrow + k, w);
    if (EPI == EPI_SWIGLU) VecLoad<TW, VW>::load(wrow2 + k, w2);
#pragma unroll
    for (int r = 0; r < GEMV_ROWS; ++r) {
      if (r < rows) {
        float a[VA];
        VecLoad<TA, VA>::load(A + (size_t)(m0 + r) * lda + k, a);
#pragma unroll
        for (int v = 0; v < VW; ++v) {
          acc[r] = fmaf(a[v], w[v], acc[r]);
          if (EPI == EPI_SWIGLU) acc2[r] = fmaf(a[v], w2[v], acc2[r]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < GEMV_ROWS; ++r) {
    if (r < rows) {  // uniform over the warp
      const float s = warp_sum(acc[r]);
      const float s2 = EPI == EPI_SWIGLU ? warp_sum(acc2[r]) : 0.f;
      if (lane == 0) epilogue_store<EPI, TOut>(out, residual, (size_t)(m0 + r) * ldo + n, s, s2);
    }
  }
}

template <typename TA, typename TW, int EPI, typename TOut>
int launch_gemm(const void* A, int lda, const void* W, const void* W2, void* out, int ldo, const float* residual,
                int M, int N, int K, int force_kernel, cudaStream_t stream) {
  const TA* a = (const TA*)A;
  const TW* w = (const TW*)W;
  const TW* w2 = (const TW*)W2;
  TOut* o = (TOut*)out;
  const bool few = force_kernel == 1 || (force_kernel == 0 && M <= 2 * GEMV_ROWS);
  if constexpr (sizeof(TA) == 4 && sizeof(TOut) == 4) {
    const bool pieces = K % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0 && (W2 == nullptr || (uintptr_t)W2 % 16 == 0);
    // (short K in one wave of the any-size kernel's blocks: that kernel has done before the other's stages are on their way; 100 rows,
    // N 200: 5.1 against 5.8 us at K 48, 6.3 against 5.9 at K 64, 8.4 against 5.3 at K 96)
    const bool short_k = K < 96 && (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN) <= 148;
    if (pieces && (force_kernel == 3 || (force_kernel == 0 && !few && !short_k)))
      return launch_sgemm_best<EPI>(a, lda, w, w2, o, ldo, residual, M, N, K, stream);
  }
  if (few) {
    constexpr int VEC = sizeof(TW) == 2 ? 8 : 4;
    const bool same_width = sizeof(TA) == sizeof(TW);
    const bool aligned = same_width && K % VEC == 0 && lda % VEC == 0 && ((uintptr_t)A % 16 == 0) &&
                         ((uintptr_t)W % 16 == 0) && (W2 == nullptr || (uintptr_t)W2 % 16 == 0);
    dim3 grid((N + 7) / 8, (M + GEMV_ROWS - 1) / GEMV_ROWS);
    if (aligned) {
      if constexpr (sizeof(TA) == sizeof(TW))
        gemv_rows_kernel<TA, TW, EPI, TOut, VEC, VEC><<<grid, 256, 0, stream>>>(a, lda, w, w2, o, ldo, residual, M, N, K);
    } else {
      gemv_rows_kernel<TA, TW, EPI, TOut, 1, 1><<<grid, 256, 0, stream>>>(a, lda, w, w2, o, ldo, residual, M, N, K);
    }
  } else {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    gemm_tile_kernel<TA, TW, EPI, TOut><<<grid, 256, 0, stream>>>(a, lda, w, w2, o, ldo, residual, M, N, K);
  }
  return 0;
}

}  // namespace edgelm

using namespace edgelm;

// a_dtype: dtype of `a` and of both weights; out_dtype: dtype of `out` (EPI_RESIDUAL: float).
// force_kernel: 0 choose by sizes and alignment, 1 the few-rows kernel, 2 the any-size tile kernel, 3 the float32 register tiles where
// the operands allow them, else 2 (tests call all).
extern "C" int edgelm_gemm_simt(const void* a, int lda, const void* w, const void* w2, void* out, int ldo,
                                const float* residual, int M, int N, int K, int a_dtype, int out_dtype, int epilogue,
                                int force_kernel, cudaStream_t stream) {
  if (M == 0) return 0;
  EL_REFUSE(M > 0 && N > 0 && K > 0 && lda >= K && ldo >= N, "gemm_simt: bad sizes M=%d N=%d K=%d lda=%d ldo=%d", M, N, K, lda, ldo);
  EL_REFUSE(epilogue != EPI_SWIGLU || w2 != nullptr, "gemm_simt: SwiGLU needs the second weight");
  EL_REFUSE(epilogue != EPI_RESIDUAL || (residual != nullptr && out_dtype == DT_F32), "gemm_simt: residual epilogue needs a float32 residual and output");
  EL_REFUSE((M + BM - 1) / BM <= 65535, "gemm_simt: too many rows (%d)", M);
  int rc = 0;
#define EL_GEMM_CASE(TA, TOUT)                                                                                      \
  switch (epilogue) {                                                                                                \
    case EPI_STORE: rc = launch_gemm<TA, TA, EPI_STORE, TOUT>(a, lda, w, w2, out, ldo, residual, M, N, K, force_kernel, stream); break;       \
    case EPI_RESIDUAL: rc = launch_gemm<TA, TA, EPI_RESIDUAL, float>(a, lda, w, w2, out, ldo, residual, M, N, K, force_kernel, stream); break; \
    case EPI_SWIGLU: rc = launch_gemm<TA, TA, EPI_SWIGLU, TOUT>(a, lda, w, w2, out, ldo, residual, M, N, K, force_kernel, stream); break;     \
    case EPI_RELU2: rc = launch_gemm<TA, TA, EPI_RELU2, TOUT>(a, lda, w, w2, out, ldo, residual, M, N, K, force_kernel, stream); break;       \
    default: EL_REFUSE(false, "gemm_simt: unknown epilogue %d", epilogue);                                           \
  }
  if (a_dtype == DT_F32 && out_dtype == DT_F32) {
    EL_GEMM_CASE(float, float)
  } else if (a_dtype == DT_BF16 && out_dtype == DT_BF16) {
    EL_GEMM_CASE(__nv_bfloat16, __nv_bfloat16)
  } else if (a_dtype == DT_BF16 && out_dtype == DT_F32) {
    EL_GEMM_CASE(__nv_bfloat16, float)
  } else {
    EL_REFUSE(false, "gemm_simt: unsupported dtypes a=%d out=%d", a_dtype, out_dtype);
  }
#undef EL_GEMM_CASE
  if (rc != 0) return rc;
  EL_LAUNCH_CHECK("gemm_simt");
  return 0;
}
