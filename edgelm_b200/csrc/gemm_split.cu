// out = a . W^T for float32 operands on the fifth-generation tensor cores (tcgen05), as exact as float32 sums: the 32-bit path's
// products of more rows than the few-rows kernels take.
//
//   a [M, K] float32 (row pitch lda), W [N, K] float32 row-major (out, in); out [M, N] float32.
//
// A float32 number is the sum of three bfloat16 numbers (8 + 8 + 8 significant bits, each the nearest to what the ones before it leave),
// and a product of two of them the sum of nine exact products.  Six are computed; the three left out (second by third, third by second,
// third by third) are under 2^-25 of the product, below what rounding one float32 product takes.  What rounds is the accumulation:
// the tensor cores cut a sum off below its last place, so the leading products (first by first) of 32 k's at a time go to an
// accumulator of their own, and these runs are added in registers, rounded to nearest, eight of them before they join the sum; the five
// cross products are 2^-8 of them and share an accumulator over all of K.  Distance from float64 (2-norm over the result's, normal
// operands) beside register tiles of float32 multiply-adds summed in runs of 32: K 16 3.6e-8 and 5.7e-8, K 576 7.7e-8 and 9.9e-8,
// K 2560 1.02e-7 and 1.12e-7 (one block a tile; less where blocks share K).  Cut-offs of one sign do not cancel: where all products are positive,
// sums are 3.8e-8 short on average at any K from 32 on, 5.6e-8 to 7.0e-8 off in all where the register tiles were 4.0e-8 to 5.3e-8.
//
// One CTA computes a tile of 128 rows of W (the lanes of tensor memory; for SwiGLU 64 gate rows and the 64 up rows of the same outputs)
// by BN rows of `a`.  A unit of work is 32 k's of the tile.  Warps:
//   0        TMA: 128 x 32 float32 of W and BN x 32 of `a` a slot, a ring of slots (deep: a decode step's products are a stream of
//            weights, and what is in flight is what its rate is made of);
//   1        one lane issues the MMAs (M 128, N BN or 2 BN, K 16): W's terms come out of tensor memory, `a`'s out of shared memory;
//   next     groups of four split: a thread takes a row of W (tcgen05.st, lane = row) and pieces of rows of `a` (swizzled K-major tiles);
//   last 8   add the runs (tcgen05.ld).
// Then all of them do the epilogue out of shared memory, a warp's lanes at neighbouring outputs of one row of `out`.
// Where the tiles leave SMs idle, K is shared by the blocks of a cluster, whose sums are folded out of shared memory.
//
// No unit is full (1,143 rows, SwiGLU N 1536, ncu: tensor pipe active 20 % of the time, issue slots half busy, shared memory's load/store path 34 %); the
// nearest by count is shared memory, to which TMA and the MMAs come as well: 64 k's of a tile of BN 64 are 48 KB written by TMA, 48 read, 24 written as terms and 48 read
// by the MMAs, 1,340 clocks of the 2,000 they take.  Both operands of the MMAs in shared memory would be
// 96 KB more; 128 rows of `a` a tile take 2,200 clocks, but half as many tiles fill fewer SMs (1,143 rows, N 576 to 1536: no gain), and
// twice the splitting threads 5 % longer at BN 64 (20 % shorter at BN 32).  Measured beside the register tiles that
// were here (a graph of launches over different weights): 1,143 rows, K 576, N 960 43.6 -> 17.8 us, SwiGLU N 1536 130 -> 50; K 1536, N 576
// 78 -> 34.7; 24 rows, K 960, N 49152 110 -> 50.5 (3.7 TB/s); SwiGLU N 2560 20.7 -> 10.9; 2,048 rows, K 2048, SwiGLU N 8192 3,668 -> 1,370.
//
// A value that is no finite number, or rounds to none in bfloat16, makes every sum it joins infinite or not a number; a sum under 1e-15 may
// have lost terms of its operands that are under 2^-126.  Such sums are computed again by one thread each as plain float32 multiply-adds, so they
// come out as the CUDA-core kernels give them.  What that leaves: K terms under 2^-126 times operands up to m are 2^-126 K m together, under
// 2^-24 of any sum from 1e-15 on while K m is up to 2^52 (K 65,536: operands up to 7e10).  Beside larger operands, ones under 2^-101 count
// with fewer digits, or as zero.  (The largest operand of every row gathered while splitting, and sums looked at by it, would leave nothing,
// and took 0.65 of 6.6 us at 24 rows, N 960, K 960 and 2 to 5 % of larger products.)
#include <cooperative_groups.h>

#include "mma_split.cuh"
#include "tc_common.cuh"

namespace edgelm {

enum : int { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_SWIGLU = 2, EPI_RELU2 = 4 };

constexpr int SP_ROWS = 128, SP_HALF = 32;   // rows of W a tile; k's a unit: a slot of the ring, half of a stage
constexpr int SP_W_BYTES = SP_ROWS * 128;
constexpr uint32_t SP_A_COLS = 96, SP_A_BASE = 512 - 2 * SP_A_COLS;   // W's three terms of a stage's 64 k's in tensor memory, two stages

template <int BN> constexpr int sp_slots() { return BN == 64 ? 6 : 8; }
template <int BN> constexpr int sp_split_groups() { return BN == 64 ? 2 : 4; }       // groups of four warps that split, a unit at a time
template <int BN> constexpr int sp_threads() { return 64 + 128 * sp_split_groups<BN>() + 256; }
template <int BN> constexpr int sp_slot_bytes() { return SP_W_BYTES + BN * 128; }
template <int BN> constexpr int sp_term_bytes() { return BN * 128; }
template <int BN> constexpr size_t split_smem() { return 1024 + 6 * sp_term_bytes<BN>() + sp_slots<BN>() * sp_slot_bytes<BN>() + 512; }

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ bool sum_stands(float v) {
  const float m = fabsf(v);
  return (m >= 1e-15f && m <= 3.402823466e38f) || v == 0.f;
}
__device__ __noinline__ float plain_dot(const float* a, const float* w, int K) {
  float sum = 0.f;
  for (int k0 = 0; k0 < K; k0 += 16) {
    float run = 0.f;
    for (int k = k0; k < min(K, k0 + 16); ++k) run = fmaf(a[k], w[k], run);
    sum += run;
  }
  return sum;
}

template <int EPI>
__device__ __forceinline__ float split_epilogue(float residual, float acc, float acc2) {
  if (EPI == EPI_RESIDUAL) return residual + acc;
  if (EPI == EPI_SWIGLU) return acc / (1.0f + expf(-acc)) * acc2;
  if (EPI == EPI_RELU2) return fmaxf(acc, 0.f) * fmaxf(acc, 0.f);
  return acc;
}

template <int BN, int EPI>
__global__ void __launch_bounds__(sp_threads<BN>(), 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_a,
                  const float* __restrict__ A, int lda, const float* __restrict__ W, const float* __restrict__ W2, float* out, int ldo,
                  const float* residual, int M, int N, int K, int CS, int* err) {
  constexpr int SP_THREADS = sp_threads<BN>(), GROUPS = sp_split_groups<BN>();
  constexpr int SLOTS = sp_slots<BN>(), SLOT = sp_slot_bytes<BN>(), TERM = sp_term_bytes<BN>();
  constexpr int NACC = 2;                      // accumulators of the leading products (tensor memory has room for)
  constexpr uint32_t CROSS = NACC * BN;                        // columns of the cross products' accumulator
  constexpr int NOUT = EPI == EPI_SWIGLU ? SP_ROWS / 2 : SP_ROWS;
  static_assert(CROSS + 2 * BN <= SP_A_BASE, "accumulators and W's terms share tensor memory");
  static_assert(BN * SP_ROWS * 4 <= 6 * TERM + SLOTS * SLOT, "a block's sums fit into its shared memory");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = smem + 6 * TERM;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + SLOTS * SLOT);
  uint64_t *ring_full = bars, *ring_empty = bars + SLOTS, *unit_full = bars + 2 * SLOTS, *unit_empty = unit_full + 4;
  uint64_t *acc_full = unit_empty + 4, *acc_empty = acc_full + 2, *all_done = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(all_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* sink = reinterpret_cast<int*>(tmem_slot + 2);           // where a wait that ran out is reported when the caller gave no error word
  if (err == nullptr) err = sink;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % CS, n0 = blockIdx.x / CS * NOUT, m0 = blockIdx.y * BN;
  const int chunks = (K + 2 * SP_HALF - 1) / (2 * SP_HALF);
  const int c_begin = (int)((long long)chunks * rank / CS), n_c = (int)((long long)chunks * (rank + 1) / CS) - c_begin;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(smem_u32(&ring_full[s]), 1);
      mbar_init(smem_u32(&ring_empty[s]), 4);                  // the warps that split a slot
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(smem_u32(&unit_full[s]), 4);
      mbar_init(smem_u32(&unit_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&acc_full[s]), 1);
      mbar_init(smem_u32(&acc_empty[s]), 8);
    }
    mbar_init(smem_u32(all_done), 1);
    *abort_flag = 0;
    *sink = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // (the weights of the first ring of slots are requested ahead of the wait for the kernel before this one)
  const int n_sub = 2 * n_c, n_ahead = n_sub < SLOTS ? n_sub : SLOTS;
  auto load_w = [&](int i) {
    const uint32_t bar = smem_u32(&ring_full[i % SLOTS]), dst = smem_u32(ring + i % SLOTS * SLOT);
    const int x = (2 * c_begin + i) * SP_HALF;
    mbar_expect_tx(bar, SLOT);
    tma_load_2d(dst, &map_w, bar, x, n0);
    if (EPI == EPI_SWIGLU) tma_load_2d(dst + SP_W_BYTES / 2, &map_w2, bar, x, n0);
  };
  auto load_a = [&](int i) {
    tma_load_2d(smem_u32(ring + i % SLOTS * SLOT + SP_W_BYTES), &map_a, smem_u32(&ring_full[i % SLOTS]), (2 * c_begin + i) * SP_HALF, m0);
  };
  if (warp == 0 && elect_one())
    for (int i = 0; i < n_ahead; ++i) load_w(i);
  __syncwarp();
  pdl_launch_dependents();
  pdl_wait();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint64_t* bar, int parity) { return __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), (uint32_t)parity, abort_flag, err)); };

  const int quarter = warp & 3, w_row = quarter * 32 + lane;   // a warp reaches the 32 lanes of tensor memory that its index modulo 4 selects
  const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
  if (warp == 0) {
    const bool leader = elect_one();
    for (int i = 0; i < n_sub; ++i) {
      if (i >= SLOTS && !wait(&ring_empty[i % SLOTS], (i / SLOTS & 1) ^ 1)) break;
      if (leader) {
        if (i >= n_ahead) load_w(i);
        load_a(i);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    // a step of 16 k's: W1 A1 | W1 [A2 A3] | W2 [A1 A2] | W3 A1, the bracketed terms of `a` one operand of 2 BN rows (as they lie)
    constexpr uint32_t one = umma_idesc(SP_ROWS, BN), two = umma_idesc(SP_ROWS, 2 * BN);
    const bool leader = elect_one();
    const uint64_t tiles = umma_desc(smem_u32(smem));
    const uint32_t a_lo = (uint32_t)tiles, a_hi = (uint32_t)(tiles >> 32);
    bool ok = true;
    for (int s0 = 0; s0 < n_sub && ok; s0 += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int st = u >> 1, h = u & 1;
        if (s0 + u >= n_sub || !ok) break;
        ok = wait(&unit_full[u], s0 >> 2 & 1) && wait(&acc_empty[h], (u >> 1) ^ 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (leader) {
          const uint32_t w = tmem + SP_A_BASE + st * SP_A_COLS + h * 16, a = a_lo + (st * 3 * TERM >> 4) + h * 4;
#pragma unroll
          for (int j = 0; j < 2; ++j) umma_f16_ts(tmem + h * BN, w + j * 8, a + j * 2, a_hi, one, j != 0);
          umma_commit(smem_u32(&acc_full[h]));
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            umma_f16_ts(tmem + CROSS, w + j * 8, a + (TERM >> 4) + j * 2, a_hi, two, j + u != 0 || s0 != 0);
            umma_f16_ts(tmem + CROSS, w + 32 + j * 8, a + j * 2, a_hi, two, true);
            umma_f16_ts(tmem + CROSS, w + 64 + j * 8, a + j * 2, a_hi, one, true);
          }
          umma_commit(smem_u32(&unit_empty[u]));
        }
        __syncwarp();
      }
    }
    if (leader) umma_commit(smem_u32(all_done));
    __syncwarp();
  } else if (warp < 2 + 4 * GROUPS) {
    // four warps a unit: while one unit's are at their barriers, others split
    for (int s = (warp - 2) >> 2; s < n_sub; s += GROUPS) {
      const int u = s & 3, st = u >> 1, half = u & 1;
      if (!wait(&ring_full[s % SLOTS], s / SLOTS & 1) || !wait(&unit_empty[u], (s >> 2 & 1) ^ 1)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint8_t* slot = ring + s % SLOTS * SLOT;
      const float4* row = reinterpret_cast<const float4*>(slot + w_row * 128);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t t[3][8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 v = row[(g * 4 + u) ^ (w_row & 7)];
          sp_split(v.x, v.y, t[0][2 * u], t[1][2 * u], t[2][2 * u]);
          sp_split(v.z, v.w, t[0][2 * u + 1], t[1][2 * u + 1], t[2][2 * u + 1]);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) tmem_st8(tmem + lanes + SP_A_BASE + st * SP_A_COLS + q * 32 + half * 16 + g * 8, t[q]);
      }
#pragma unroll
      for (int b = 0; b < BN / 32; ++b) {
        const int r = (lane & 7) + (quarter + b * 4) * 8, p = lane >> 3;     // eight k's of a row of `a`
        const float4* ar = reinterpret_cast<const float4*>(slot + SP_W_BYTES + r * 128);
        const float4 v = ar[(2 * p) ^ (r & 7)], w = ar[(2 * p + 1) ^ (r & 7)];
        uint4 t1, t2, t3;
        sp_split(v.x, v.y, t1.x, t2.x, t3.x);
        sp_split(v.z, v.w, t1.y, t2.y, t3.y);
        sp_split(w.x, w.y, t1.z, t2.z, t3.z);
        sp_split(w.z, w.w, t1.w, t2.w, t3.w);
        uint8_t* dst = smem + st * 3 * TERM + r * 128 + ((half * 4 + p) ^ (r & 7)) * 16;
        *reinterpret_cast<uint4*>(dst) = t1;
        *reinterpret_cast<uint4*>(dst + TERM) = t2;
        *reinterpret_cast<uint4*>(dst + 2 * TERM) = t3;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&unit_full[u]));
        mbar_arrive(smem_u32(&ring_empty[s % SLOTS]));
      }
    }
  } else {
    constexpr int COLS = BN / 2;                               // its share of the accumulators' columns: a lane's row of W, COLS rows of `a`
    const uint32_t col0 = (warp - 2 - 4 * GROUPS) / 4 * COLS;
    float sum[COLS] = {}, run[COLS] = {};
    auto add = [&](float* to, uint32_t from) {
#pragma unroll
      for (int c = 0; c < COLS; c += 8) {
        uint32_t r[8];
        tmem_ld8(tmem + lanes + from + col0 + c, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) to[c + j] += __uint_as_float(r[j]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    };
    bool ok = true;
    for (int f = 0; f < n_sub && ok; ++f) {
      const int b = f % NACC;
      ok = wait(&acc_full[b], f / NACC & 1);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      add(run, b * BN);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acc_empty[b]));
      if ((f & 7) == 7)
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
          sum[j] += run[j];
          run[j] = 0.f;
        }
    }
    if (ok) ok = wait(all_done, 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
      add(run, CROSS);
      add(run, CROSS + BN);
    }
    float* sums = reinterpret_cast<float*>(smem);              // [BN][128] (every MMA has read its tiles, every slot is split)
#pragma unroll
    for (int j = 0; j < COLS; ++j)                             // (a wait that ran out: nothing that could pass for a result)
      sums[(col0 + j) * SP_ROWS + w_row] = ok ? sum[j] + run[j] : __uint_as_float(0x7fc00000u);
  }
  // (also where a wait ran out: the block's own MMAs and copies in flight end before its memory is given back)
  if (warp == 1) {
    const long long t0 = clock64();
    while (!mbar_try(smem_u32(all_done), 0) && clock64() - t0 < TC_WAIT_CYCLES) {}
  }
  if (warp == 0 && *abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 100000) {}
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  const float* sums = reinterpret_cast<const float*>(smem);
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  if (CS > 1) cluster.sync();
  const bool whole = *abort_flag == 0;
  const int e_end = min(BN * (rank + 1) / CS, M - m0) * NOUT;
  constexpr int AHEAD = 4;               // (residuals requested together: `out` may be the residual itself)
  for (int e0 = BN * rank / CS * NOUT + threadIdx.x; e0 < e_end; e0 += AHEAD * SP_THREADS) {
    float ahead[AHEAD] = {};
    auto there = [&](int e) { return e < e_end && n0 + e % NOUT < N; };
    auto at = [&](int e) { return (size_t)(m0 + e / NOUT) * ldo + n0 + e % NOUT; };
    if (EPI == EPI_RESIDUAL)
#pragma unroll
      for (int x = 0; x < AHEAD; ++x)
        if (there(e0 + x * SP_THREADS)) ahead[x] = residual[at(e0 + x * SP_THREADS)];
#pragma unroll
    for (int x = 0; x < AHEAD; ++x) {
      const int e = e0 + x * SP_THREADS;
      if (!there(e)) continue;
      const int r = e / NOUT, n = e % NOUT;
      float v = 0.f, v2 = 0.f;
      for (int q = 0; q < CS; ++q) {
        const float* p = (CS > 1 ? cluster.map_shared_rank(sums, q) : sums) + r * SP_ROWS + n;
        v += p[0];
        if (EPI == EPI_SWIGLU) v2 += p[NOUT];
      }
      if (whole && !sum_stands(v)) v = plain_dot(A + (size_t)(m0 + r) * lda, W + (size_t)(n0 + n) * K, K);
      if (EPI == EPI_SWIGLU && whole && !sum_stands(v2)) v2 = plain_dot(A + (size_t)(m0 + r) * lda, W2 + (size_t)(n0 + n) * K, K);
      out[at(e)] = split_epilogue<EPI>(ahead[x], v, v2);
    }
  }
  if (CS > 1) cluster.sync();            // (no block leaves while another reads its sums)
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <int BN, int EPI>
int launch_split(const float* a, int lda, const float* w, const float* w2, float* out, int ldo, const float* residual, int M, int N, int K,
                 int CS, int* err, cudaStream_t stream) {
  constexpr int NOUT = EPI == EPI_SWIGLU ? SP_ROWS / 2 : SP_ROWS;
  constexpr size_t smem = split_smem<BN>();
  CUtensorMap mw, mw2, ma;
  if (tensor_map(w, N, K, K, NOUT, &mw, 4)) return -1;
  mw2 = mw;
  if (EPI == EPI_SWIGLU && tensor_map(w2, N, K, K, NOUT, &mw2, 4)) return -1;
  if (tensor_map(a, M, K, lda, BN, &ma, 4)) return -1;
  auto* kern = gemm_split_kernel<BN, EPI>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  EL_REFUSE(e == cudaSuccess, "gemm_split: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((N + NOUT - 1) / NOUT * CS), (unsigned)((M + BN - 1) / BN));
  cfg.blockDim = dim3(sp_threads<BN>());
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
  cudaLaunchKernelEx(&cfg, kern, mw, mw2, ma, a, lda, w, w2, out, ldo, residual, M, N, K, CS, err);
  return 0;
}

// The tile and the number of blocks that share K: what takes the least time by a count of waves of one block an SM (a block's tensor
// memory fills it; clusters of eight find room for 120 blocks, of six surely for 96).  Measured: 64 k's take a block 0.7 us with 32 rows of `a`, 1.08 with 64
// (TMA's writes, the splitting threads' reads and the MMAs' reads of shared memory: 116 and 168 KB at 128 bytes a clock), a block's
// start and end 5 to 8 us, a cluster's exchange one more.  K 2560, 24 rows, N 960, clusters of 1, 2, 4, 8: 32, 19.3, 12.4, 9.5 us.
template <int EPI>
int launch_split_best(const float* a, int lda, const float* w, const float* w2, float* out, int ldo, const float* residual, int M, int N, int K,
                      int form, int* err, cudaStream_t stream) {
  const int chunks = (K + 2 * SP_HALF - 1) / (2 * SP_HALF);
  int best_bn = form & 0xff, best_cs = form >> 8;
  if (form == 0) {
    struct Tile { int rows; float stage_us, block_us; };
    constexpr Tile tiles[2] = {{64, 1.08f, 7.f}, {32, 0.7f, 5.f}};
    const int tiles_n = (N + (EPI == EPI_SWIGLU ? 64 : 128) - 1) / (EPI == EPI_SWIGLU ? 64 : 128);
    float best = 0.f;
    for (const Tile& t : tiles) {
      const long long tiles_m = (M + t.rows - 1) / t.rows;
      if (tiles_m > 65535) continue;
      for (int cs : {1, 2, 3, 4, 6, 8}) {
        if (cs > chunks) break;
        const int room = cs == 8 ? 120 : cs == 6 ? 96 : cs > 2 ? 132 : 148;
        const float us = (float)((tiles_m * tiles_n * cs + room - 1) / room) * ((float)((chunks + cs - 1) / cs) * t.stage_us + t.block_us + (cs > 1 ? 1.f : 0.f));
        if (best_cs == 0 || us < best) { best = us; best_bn = t.rows; best_cs = cs; }
      }
    }
  }
  EL_REFUSE(best_cs >= 1 && best_cs <= 8 && best_cs <= chunks, "gemm_split: %d blocks do not share K=%d", best_cs, K);
  if (best_bn == 64) return launch_split<64, EPI>(a, lda, w, w2, out, ldo, residual, M, N, K, best_cs, err, stream);
  EL_REFUSE(best_bn == 32, "gemm_split: no tile of %d rows", best_bn);
  return launch_split<32, EPI>(a, lda, w, w2, out, ldo, residual, M, N, K, best_cs, err, stream);
}

}  // namespace edgelm

using namespace edgelm;

// 1 if the kernel takes these operands: rows in pieces of 16 bytes, as TMA wants them
extern "C" int edgelm_gemm_split_takes(const void* a, int lda, const void* w, const void* w2, int K) {
  return K > 0 && K % 4 == 0 && lda % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)w % 16 == 0 && (w2 == nullptr || (uintptr_t)w2 % 16 == 0) ? 1 : 0;
}

// `form`: 0 choose by sizes, else rows of the tile (32, 64) + 256 x the blocks that share K (tests and comparisons).  `err` may be
// null: sums behind a wait that ran out are then only not-a-numbers.
extern "C" int edgelm_gemm_split(const void* a, int lda, const void* w, const void* w2, void* out, int ldo, const float* residual, int M, int N,
                                 int K, int epilogue, int form, int* err, cudaStream_t stream) {
  if (M == 0) return 0;
  EL_REFUSE(M > 0 && N > 0 && K > 0 && lda >= K && ldo >= N, "gemm_split: bad sizes M=%d N=%d K=%d lda=%d ldo=%d", M, N, K, lda, ldo);
  EL_REFUSE(edgelm_gemm_split_takes(a, lda, w, w2, K), "gemm_split: K=%d and lda=%d must be multiples of 4 and the operands 16-byte aligned", K, lda);
  EL_REFUSE(epilogue != EPI_SWIGLU || w2 != nullptr, "gemm_split: SwiGLU needs the second weight");
  EL_REFUSE(epilogue != EPI_RESIDUAL || residual != nullptr, "gemm_split: the residual epilogue needs a residual");
  EL_REFUSE((M + 63) / 64 <= 65535, "gemm_split: too many rows (%d)", M);
  const float *fa = (const float*)a, *fw = (const float*)w, *fw2 = (const float*)w2;
  int rc = 0;
  switch (epilogue) {
    case EPI_STORE: rc = launch_split_best<EPI_STORE>(fa, lda, fw, fw2, (float*)out, ldo, residual, M, N, K, form, err, stream); break;
    case EPI_RESIDUAL: rc = launch_split_best<EPI_RESIDUAL>(fa, lda, fw, fw2, (float*)out, ldo, residual, M, N, K, form, err, stream); break;
    case EPI_SWIGLU: rc = launch_split_best<EPI_SWIGLU>(fa, lda, fw, fw2, (float*)out, ldo, residual, M, N, K, form, err, stream); break;
    case EPI_RELU2: rc = launch_split_best<EPI_RELU2>(fa, lda, fw, fw2, (float*)out, ldo, residual, M, N, K, form, err, stream); break;
    default: EL_REFUSE(false, "gemm_split: unknown epilogue %d", epilogue);
  }
  if (rc != 0) return rc;
  EL_LAUNCH_CHECK("gemm_split");
  return 0;
}
