// Small float32 matrix products out of shared memory, for recurrences that are worked off chunk by chunk: both operands lie with the
// summed index contiguous, in rows whose pitch is 4 floats times an odd number (eight neighbouring rows' pieces of 16 bytes then lie
// in different banks).
#pragma once
#include "common.cuh"

namespace edgelm {

constexpr int CHUNK = 64;      // tokens of a chunk (the step's tiles of that size)

__host__ __device__ constexpr int chunk_pitch(int n) { return ((n + 3) / 4 | 1) * 4; }

// Thread (ty, tx) of a block of 16 NY threads: rows m = ty + NY a, columns n = tx + 16 b.  (Neighbouring threads are two rows of one
// column: a read of 16 bytes a lane then takes two clocks for either operand.)
__device__ __forceinline__ int chunk_tx() { return threadIdx.x >> 1 & 15; }
__device__ __forceinline__ int chunk_ty() { return (threadIdx.x & 1) + (threadIdx.x >> 5) * 2; }

// acc[a][b] += sum over k < K of A[m][k] B[n][k]; K a multiple of 4; rows from M and columns from N on: the last one's again.
// Packed pairs of multiply-adds: even and odd k in sums of their own before they join `acc`.  (Four runs instead of two took the
// registers of a second block an SM, whose loads hide the first one's: the state-space outputs of state_chunks.cu 285 us against 126.)
template <int NY, int RM, int RN>
__device__ __forceinline__ void chunk_mm(float (&acc)[RM][RN], const float* A, int pa, int M, const float* B, int pb, int N, int K) {
  const int tx = chunk_tx(), ty = chunk_ty();
  const float* ar[RM];
  const float* br[RN];
  unsigned long long sum[RM][RN] = {};
#pragma unroll
  for (int a = 0; a < RM; ++a) ar[a] = A + min(ty + NY * a, M - 1) * pa;
#pragma unroll
  for (int b = 0; b < RN; ++b) br[b] = B + min(tx + 16 * b, N - 1) * pb;
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    ulonglong2 av[RM];
#pragma unroll
    for (int a = 0; a < RM; ++a) av[a] = *reinterpret_cast<const ulonglong2*>(ar[a] + k);
#pragma unroll
    for (int b = 0; b < RN; ++b) {
      const ulonglong2 bv = *reinterpret_cast<const ulonglong2*>(br[b] + k);
#pragma unroll
      for (int a = 0; a < RM; ++a) {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[a][b]) : "l"(av[a].x), "l"(bv.x));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[a][b]) : "l"(av[a].y), "l"(bv.y));
      }
    }
  }
#pragma unroll
  for (int a = 0; a < RM; ++a)
#pragma unroll
    for (int b = 0; b < RN; ++b) acc[a][b] += __uint_as_float((uint32_t)sum[a][b]) + __uint_as_float((uint32_t)(sum[a][b] >> 32));
}

// The logarithms of a chunk's decays: lg[t] = l_0 + .. + l_t, lane i of the calling warp bringing tokens 2 i and 2 i + 1.  No token's
// sum holds a later one's value, so that what is not finite stays at its token and behind.
__device__ __forceinline__ void chunk_log_sums(double* lg, double l0, double l1) {
  const int lane = threadIdx.x & 31;
  double sum = l0 + l1;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, sum, off);
    if (lane >= off) sum += up;
  }
  const double before = __shfl_up_sync(0xffffffffu, sum, 1);
  lg[2 * lane] = lane == 0 ? l0 : before + l0;
  lg[2 * lane + 1] = sum;
}

// An output that a product over all tokens of the chunk left not finite, over its own and the earlier ones alone: first . second + sum over
// s <= t of weights[s] values[s].  (A weight of zero times a later token's infinity is a NaN, where the walk has not met that token.)
__device__ __forceinline__ float chunk_causal(const float* first, const float* second, int K, float scale, const float* weights, const float* values, int t) {
  float v = 0.f;
  for (int k = 0; k < K; ++k) v = fmaf(first[k], second[k], v);
  v *= scale;
  for (int s = 0; s <= t; ++s) v = fmaf(weights[s], values[s], v);
  return v;
}

// acc[a][b] = the same sum in runs of eight products, which join in double.  (For products whose error travels on or whose terms largely
// cancel: scores between a chunk's tokens.  With sums as in `chunk_mm` they alone put the delta rule's and the state-space outputs further
// from float64 than a walk over the tokens is.)
template <int NY, int RM, int RN>
__device__ __forceinline__ void chunk_mm_runs(double (&acc)[RM][RN], const float* A, int pa, int M, const float* B, int pb, int N, int K) {
  const int tx = chunk_tx(), ty = chunk_ty();
#pragma unroll
  for (int a = 0; a < RM; ++a)
#pragma unroll
    for (int b = 0; b < RN; ++b) acc[a][b] = 0.0;
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 8) {
    unsigned long long sum[RM][RN] = {};
#pragma unroll
    for (int k = k0; k < k0 + 8; k += 4) {
      if (k >= K) break;
      ulonglong2 av[RM];
#pragma unroll
      for (int a = 0; a < RM; ++a) av[a] = *reinterpret_cast<const ulonglong2*>(A + min(ty + NY * a, M - 1) * pa + k);
#pragma unroll
      for (int b = 0; b < RN; ++b) {
        const ulonglong2 bv = *reinterpret_cast<const ulonglong2*>(B + min(tx + 16 * b, N - 1) * pb + k);
#pragma unroll
        for (int a = 0; a < RM; ++a) {
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[a][b]) : "l"(av[a].x), "l"(bv.x));
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[a][b]) : "l"(av[a].y), "l"(bv.y));
        }
      }
    }
#pragma unroll
    for (int a = 0; a < RM; ++a)
#pragma unroll
      for (int b = 0; b < RN; ++b) acc[a][b] += (double)(__uint_as_float((uint32_t)sum[a][b]) + __uint_as_float((uint32_t)(sum[a][b] >> 32)));
  }
}

__device__ __forceinline__ void chunk_cp16(float* dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// rows [rows][n] of `src` (row pitch ld, n a multiple of 4, 16-byte aligned) on their way into dst [..][pitch]; zeros for the rows from
// `valid` on
__device__ __forceinline__ void chunk_rows(float* dst, int pitch, const float* src, size_t ld, int rows, int valid, int n) {
  const int nv = n >> 2;
  for (int i = threadIdx.x; i < rows * nv; i += blockDim.x) {
    const int r = i / nv, c = (i - r * nv) * 4;
    chunk_cp16(dst + r * pitch + c, r < valid ? src + (size_t)r * ld + c : src, r < valid);
  }
}

}  // namespace edgelm
