// Attention of many new tokens over bfloat16 keys and values with float32 queries, scores and softmax weights on the fifth-generation
// tensor cores (tcgen05): what attention_mma_split.cu computes, for steps whose sequences bring enough tokens for tiles of 128.
//
//   S = (q1 + q2 + q3) K^T,  O += (p1 + p2 + p3) V      the float32 operand as the sum of three bfloat16 terms, exact products, float32 sums
//
// grid (head or head's map, query tile); a CTA takes up to 128 consecutive tokens of one sequence for one head and walks the keys that its
// rows see in blocks of two cache pages (or of the step's own rows).  Roles: warp 0 loads the keys by TMA, warp 1 the values, warp 2 issues
// S (A: the queries' terms, swizzled K-major tiles written once; B: the keys as they lie), warp 3 issues O (A: the weights' terms out
// of tensor memory; B: the values as they lie, MN-major), warps 4 to 19 are the softmax: four threads a row, half a page
// of the block each.  They exchange a row's maximum through shared memory, so that they share one reference; it moves only when the
// maximum has outgrown it by 2^8.  A thread's weights go back over the scores that they came from: its 32 columns hold terms 1 and 2,
// 16 further ones the third.  Tensor memory: two such buffers of 192 columns and O: 128 columns, or twice 64.
// So S of block j + 1 is computed beside the softmax of block j, and O of block j beside the softmax of block j + 1.
//
// The tensor cores cut a sum off below its last place at every MMA, and with one accumulator over all keys these add up: O's runs are two
// blocks long, and the softmax threads add a run to the row's output in registers, rounded to nearest (a quarter of the dimensions each; where
// the reference moves they scale that, and a run that has begun in place).  Heads of 64 value dimensions have two accumulators, so that a run
// waits a block long before it is added.  Distance from float64 in the float32 output of two maps of 64 over 128, of 256, 700, 2,000 and 5,000
// tokens (2-norm; scores of standard deviation 1): 2.3e-7, 3.4e-7, 4.1e-7, 4.6e-7; one run over all keys 2.3e-7, 6.6e-7, 1.9e-6, 4.2e-6 and
// 1 to 7 % less time; mma.sync 4.1e-7, 4.8e-7, 1.0e-6, 2.2e-6.
//
// A value that is no finite number makes that dimension of the rows that see it none, a key their whole output; rows that do not see it are as they were
// without it: in blocks that some row sees in part such values are taken out ahead of the MMAs by the loaders and given to their rows at the end
// (blocks that every row sees whole need none of it; windows and chunks of 1,024, two maps of 64 over 128, 256 tokens: 27.8 -> 30.8 us, else 1 to 3 %).
//
// Masks, sinks, gates, kept keys and maps as in attention_mma_split.cu.  Every wait is bounded; where one runs out the block reports it, writes
// not-a-numbers and waits for its own copies and MMAs before it gives its memory back.
// mma.sync takes a scheduler 16 clocks for an m16n8k16 here, four times what tcgen05 takes for as many multiply-adds, and bounds the other kernel.
// What bounds this one is the softmax: about 3,200 clocks a block, most of them the exponentials, the splitting and the stores into tensor memory (ncu,
// 4,000 tokens, 9 heads of 64: issue slots 57 % busy, tensor pipe active 36 %; in the form with one run, with a third of either product's MMAs it
// took 3 % less, without exponentials and splitting 17 %); 3 us a tile before the first block.
// mma.sync and here, us: 9 heads of 64 over 3, 1,000 and 2,000 tokens 26 and 21, 78 and 34; 512 behind 4,000 103 and 66; 16
// heads of two maps of 64 over values of 128, chunks of 1,024, 1,000 and 2,000 tokens 88 and 34, 158 and 64; 32 heads of 128, 2,000 tokens 373 and 115.
// Tiles of the most keys go first over all heads (a head's tiles next to each other left the last head's longest tile to the end).
#include <math_constants.h>

#include "mma_split.cuh"
#include "tc_common.cuh"

namespace edgelm {

enum : int { ST_MASK_CAUSAL = 0, ST_MASK_WINDOW = 1, ST_MASK_CHUNK = 2 };

constexpr int ST_ROWS = 128, ST_SOFT_WARPS = 16, ST_THREADS = 128 + ST_SOFT_WARPS * 32;
constexpr uint32_t ST_BUF_COLS = 192, ST_O_COL = 2 * ST_BUF_COLS;
constexpr float ST_LAZY = 8.f;
constexpr int ST_TILE = 128 * 128;             // bytes of 128 rows of 64 bfloat16

template <int DK, int DV> struct StSizes {
  static constexpr int KC = (DK + 63) / 64, VC = (DV + 63) / 64;      // tiles of 64 dimensions
  static constexpr int KS = 2, VS = KC == 2 && VC == 2 ? 1 : 2;       // stages of keys and values
  static constexpr int CLEANERS = VS;             // warps that clean the values
  static constexpr int smem = 1024 + (3 * KC + KS * KC + VS * VC) * ST_TILE + 12 * ST_ROWS * 4 + 256;
};

__device__ __forceinline__ int st_first_key(int pos, int mask, int size) {
  if (mask == ST_MASK_WINDOW) return max(0, pos - size + 1);
  if (mask == ST_MASK_CHUNK) return (pos / size) * size;
  return 0;
}
// O of the run (of two blocks) that block j belongs to: with room for two, the runs take turns
template <int DV> __device__ __forceinline__ uint32_t st_run_col(int j) { return ST_O_COL + (DV == 64 ? (j >> 1 & 1) * 64 : 0); }
// Two bfloat16 numbers: bits 15 and 31 where they are infinite or not a number; a mask of those that are numbers; these alone
__device__ __forceinline__ uint32_t st_no_number(uint32_t w) { return ((w & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }
__device__ __forceinline__ uint32_t st_numbers_mask(uint32_t w) { return ~((st_no_number(w) >> 15) * 0xffffu); }
__device__ __forceinline__ uint32_t st_numbers(uint32_t w) { return w & st_numbers_mask(w); }
__device__ __forceinline__ void st_add_nothing(const uint4& v, uint32_t& sum) {
  asm("{\n\tfma.rn.bf16x2 %0, %1, %5, %0;\n\tfma.rn.bf16x2 %0, %2, %5, %0;\n\tfma.rn.bf16x2 %0, %3, %5, %0;\n\tfma.rn.bf16x2 %0, %4, %5, %0;\n\t}"
      : "+r"(sum) : "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(0u));
}
__device__ __forceinline__ uint32_t st_low_bits(int n) { return n >= 32 ? ~0u : ~(~0u << max(n, 0)); }
__device__ __forceinline__ void st_tmem_st4(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// A block's last wait for what it has in flight, bounded and without a report (the wait that ran out before has made one)
__device__ __forceinline__ void st_drain(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try(bar, parity) && clock64() - t0 < TC_WAIT_CYCLES) {}
}

struct SplitTcArgs {
  const float* q;
  const __nv_bfloat16* values;
  int ldq;
  void* out;
  int ldo;
  const int32_t* page_table;       // null: the step's own rows
  int table_stride, n_pages;
  const int32_t *tile_seq, *tile_tok0, *tile_ntok, *tile_pos0;
  int n_tiles, nh, nkv, maps;
  float scale;
  const float* gate;
  int ldg, mask, mask_size;
  const float* sink;
  int keep, gate_ch;
  int* err;
};

template <int DK, int DV>
__global__ void __launch_bounds__(ST_THREADS, 1)
attn_prefill_split_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const SplitTcArgs a) {
  using Z = StSizes<DK, DV>;
  constexpr int KC = Z::KC, VC = Z::VC, KS = Z::KS, VS = Z::VS;
  extern __shared__ uint8_t st_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(st_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* q_s = smem;                             // [3 terms][KC][128 rows][128 bytes]
  uint8_t* k_s = q_s + 3 * KC * ST_TILE;           // [KS][KC][128 keys][128 bytes]
  uint8_t* v_s = k_s + KS * KC * ST_TILE;          // [VS][VC][128 keys][128 bytes]
  float* row_max = reinterpret_cast<float*>(v_s + VS * VC * ST_TILE);      // [block & 1][quarter of its keys][128 rows]
  float* row_sum = row_max + 8 * ST_ROWS;          // [quarter of the keys][128 rows]
  uint64_t* bars = reinterpret_cast<uint64_t*>(row_sum + 4 * ST_ROWS);
  uint64_t *q_ready = bars, *k_full = bars + 1, *k_empty = k_full + KS, *v_full = k_empty + KS, *v_empty = v_full + VS;
  uint64_t *v_clean = v_empty + VS, *s_ready = v_clean + VS, *p_ready = s_ready + 2, *o_done = p_ready + 2;
  uint64_t* all_done = o_done + 2;                 // both issuers' MMAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(all_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* taken_out = abort_flag + 1;        // some value that is no number was

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = a.n_tiles - 1 - (int)blockIdx.y, head = blockIdx.x, kvh = head / (a.nh / a.nkv * a.maps), map = head % a.maps;
  const int seq = a.tile_seq[tile], tok0 = a.tile_tok0[tile], ntok = a.tile_ntok[tile], pos0 = a.tile_pos0[tile];
  const int n_keys = pos0 + ntok, n_pg = (n_keys + PAGE - 1) / PAGE;
  // the pages to visit: those of the kept keys that lie ahead of the window's first, then the window's; two a block
  const int first_page = st_first_key(pos0, a.mask, a.mask_size) / PAGE, kept_pages = min(first_page, (a.keep + PAGE - 1) / PAGE);
  const int n_visit = kept_pages + n_pg - first_page, n_blk = (n_visit + 1) / 2;
  auto page_at = [&](int i) { return i < kept_pages ? i : first_page + i - kept_pages; };
  const int last_first = st_first_key(n_keys - 1, a.mask, a.mask_size);      // the first key of the tile's last row
  auto hidden = [&](int key0, int n) { return key0 + n - 1 > pos0 || (key0 < last_first && key0 + n > a.keep); };      // from some row: some of n keys
  auto some_hidden = [&](int j) {                  // some key of block j from some row (or it has no second page)
    return 2 * j + 1 >= n_visit || hidden(page_at(2 * j) * PAGE, PAGE) || hidden(page_at(2 * j + 1) * PAGE, PAGE);
  };

  if (threadIdx.x == 0) {
    for (uint64_t* b = bars; b < o_done + 2; ++b)
      mbar_init(smem_u32(b), b == q_ready || (b >= p_ready && b < o_done) ? ST_SOFT_WARPS : b >= v_clean && b < s_ready ? Z::CLEANERS : 1);
    mbar_init(smem_u32(all_done), 2);
    *abort_flag = *taken_out = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint64_t* bar, int parity) { return __all_sync(0xffffffffu, mbar_wait_parked(smem_u32(bar), (uint32_t)parity, abort_flag, a.err)); };

  if (warp < 2) {
    const bool keys = warp == 0;
    const CUtensorMap* m = keys ? &map_k : &map_v;
    const int stages = keys ? KS : VS, chunks = keys ? KC : VC, dim = keys ? DK : DV;
    uint64_t *full = keys ? k_full : v_full, *empty = keys ? k_empty : v_empty;
    uint8_t* dst = keys ? k_s : v_s;
    const int32_t* pages = a.page_table ? a.page_table + (size_t)seq * a.table_stride : nullptr;
    const bool leader = elect_one();
    // Values that some row of the tile must not see meet weights of zero: where there are such, rows behind the tile's last position (or of no page) become
    // zero, whatever lies there, and so do values that are no finite number (0 x inf would be none); the rows that see such a value get it at the end.
    // (both loaders, half of the rows each, with the next block's copies on their way; with one stage of values their loader alone)
    constexpr int CLEANERS = Z::CLEANERS, PIECES = 32 / CLEANERS;
    auto clean = [&](int j) {
      const int st = j % VS;
      if (!wait(&v_full[st], j / VS & 1)) return false;
      if (some_hidden(j)) {
        uint4* mine = reinterpret_cast<uint4*>(v_s + st * VC * ST_TILE) + (CLEANERS > 1 ? warp * PIECES : 0) * 32 + lane;      // four rows a warp and load
        const int row0 = (CLEANERS > 1 ? warp * PIECES : 0) * 4 + (lane >> 3);
        const int from0 = min(PAGE, n_keys - page_at(2 * j) * PAGE), from1 = 2 * j + 1 < n_visit ? min(PAGE, n_keys - page_at(2 * j + 1) * PAGE) : 0;
        bool written = false;
        if (from0 < PAGE || from1 < PAGE) {
          for (int x = 0; x < PIECES; ++x) {
            const int r = row0 + x * 4;
            if ((r & (PAGE - 1)) < (r < PAGE ? from0 : from1)) continue;
#pragma unroll
            for (int c = 0; c < VC; ++c) mine[c * (ST_TILE / 16) + x * 32] = make_uint4(0, 0, 0, 0);
            written = true;
          }
        }
        uint32_t sum = 0;                          // (0 x a value that is no number is none, and stays)
#pragma unroll 1
        for (int x = 0; x < PIECES * VC; x += 8) {
          uint4 v[8];
#pragma unroll
          for (int y = 0; y < 8; ++y) v[y] = mine[x / PIECES * (ST_TILE / 16) + (x % PIECES + y) * 32];
#pragma unroll
          for (int y = 0; y < 8; ++y) st_add_nothing(v[y], sum);
        }
        if (st_no_number(sum)) {
          for (int x = 0; x < PIECES * VC; ++x) {
            uint4* at = mine + x / PIECES * (ST_TILE / 16) + x % PIECES * 32;
            const uint4 v = *at;
            if ((st_no_number(v.x) | st_no_number(v.y) | st_no_number(v.z) | st_no_number(v.w)) == 0) continue;
            *at = make_uint4(st_numbers(v.x), st_numbers(v.y), st_numbers(v.z), st_numbers(v.w));
            written = true;
            *taken_out = 1;
          }
        }
        if (written) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&v_clean[st]));
      return true;
    };
    int issued = 0;
    for (int j = 0; j < n_blk; ++j) {
      const int st = j % stages;
      if (j >= stages && !wait(&empty[st], (j / stages & 1) ^ 1)) break;
      issued = j + 1;
      if (leader) {
        const uint32_t bar = smem_u32(&full[st]);
        mbar_expect_tx(bar, chunks * ST_TILE);
        for (int h = 0; h < 2; ++h) {
          const int pg = page_at(2 * j + h < n_visit ? 2 * j + h : 2 * j);      // (no second page: the first again, masked)
          int x, y;
          if (pages) {
            int page = pages[pg];
            if (page < 0 || page >= a.n_pages) {
              atomicOr(a.err, ERR_PAGE_RANGE);
              page = 0;
            }
            x = keys ? map * DK : 0;
            y = (page * a.nkv + kvh) * PAGE;
          } else {
            x = (keys ? kvh * a.maps + map : kvh) * dim;
            y = tok0 - pos0 + pg * PAGE;
          }
          for (int c = 0; c < chunks; ++c) tma_load_2d(smem_u32(dst + (st * chunks + c) * ST_TILE + h * (ST_TILE / 2)), m, bar, x + c * 64, y);
        }
      }
      __syncwarp();
      if ((!keys || CLEANERS > 1) && j >= VS - 1 && !clean(j - (VS - 1))) break;
    }
    if (VS > 1 && issued == n_blk) clean(n_blk - 1);
    // (also where a wait ran out: no copy may be on its way when the block's memory is given back)
    for (int i = max(0, issued - stages); i < issued; ++i) st_drain(smem_u32(&full[i % stages]), i / stages & 1);
  } else if (warp == 2) {
    constexpr uint32_t idesc = umma_idesc(ST_ROWS, 128);
    const bool leader = elect_one();
    const uint64_t dq = umma_desc(smem_u32(q_s));
    bool ok = wait(q_ready, 0);
    for (int j = 0; j < n_blk && ok; ++j) {
      const int b = j & 1, st = j % KS;
      if (j >= 2) ok = wait(&o_done[b], (j >> 1) - 1 & 1);            // (the block before last has left this buffer)
      if (ok) ok = wait(&k_full[st], j / KS & 1);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t dk = umma_desc(smem_u32(k_s + st * KC * ST_TILE));
      if (leader) {
#pragma unroll
        for (int t = 2; t >= 0; --t)                                  // (the small terms first)
#pragma unroll
          for (int s = 0; s < DK / 16; ++s)
            umma_f16(tmem + b * ST_BUF_COLS, dq + ((t * KC + s / 4) * ST_TILE >> 4) + 2 * (s % 4), dk + (s / 4 * ST_TILE >> 4) + 2 * (s % 4), idesc, t != 2 || s != 0);
        umma_commit(smem_u32(&s_ready[b]));
        umma_commit(smem_u32(&k_empty[st]));
      }
      __syncwarp();
    }
    if (leader) umma_commit(smem_u32(all_done));
    __syncwarp();
    st_drain(smem_u32(all_done), 0);
  } else if (warp == 3) {
    constexpr uint32_t idesc = umma_idesc(ST_ROWS, 64) | (1u << 16);  // B (the values) is MN-major
    const bool leader = elect_one();
    bool ok = true;
    for (int j = 0; j < n_blk && ok; ++j) {
      const int b = j & 1, st = j % VS;
      ok = wait(&p_ready[b], j >> 1 & 1) && wait(&v_clean[st], j / VS & 1);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t dv = umma_desc(smem_u32(v_s + st * VC * ST_TILE));
      if (leader) {
#pragma unroll
        for (int c = 0; c < VC; ++c)
#pragma unroll
          for (int t = 2; t >= 0; --t)
#pragma unroll
            for (int s = 0; s < 8; ++s) {                             // 16 keys: of the threads of quarter s / 2
              const uint32_t p = tmem + b * ST_BUF_COLS + (t == 2 ? 128 + s * 8 : s / 2 * 32 + t * 16 + s % 2 * 8);
              umma_f16_ts(tmem + st_run_col<DV>(j) + c * 64, p, (uint32_t)dv + (c * ST_TILE + s * 16 * 128 >> 4), (uint32_t)(dv >> 32), idesc, j & 1 || t != 2 || s != 0);
            }
        umma_commit(smem_u32(&o_done[b]));
        umma_commit(smem_u32(&v_empty[st]));
      }
      __syncwarp();
    }
    if (leader) umma_commit(smem_u32(all_done));
    __syncwarp();
    st_drain(smem_u32(all_done), 0);
  } else {
    const int sw = warp - 4, part = sw >> 2, half = part >> 1, quarter = warp & 3, row = quarter * 32 + lane, tid = threadIdx.x - 128;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    // scores in units of log 2; the scale's sign (or a scale of 0) goes to the queries, so that the largest score has the largest weight
    const float scale2 = a.scale == 0.f ? 1.f : fabsf(a.scale) * 1.4426950408889634f, turn = a.scale < 0.f ? -1.f : a.scale > 0.f ? 1.f : 0.f;
    for (int i = tid; i < ST_ROWS * (DK / 4); i += ST_SOFT_WARPS * 32) {
      const int r = i / (DK / 4), d = i % (DK / 4) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < ntok) v = *reinterpret_cast<const float4*>(a.q + (size_t)(tok0 + r) * a.ldq + head * DK + d);
      uint2 t[3];
      sp_split(turn * v.x, turn * v.y, t[0].x, t[1].x, t[2].x);
      sp_split(turn * v.z, turn * v.w, t[0].y, t[1].y, t[2].y);
      uint8_t* dst = q_s + d / 64 * ST_TILE + r * 128 + ((d % 64 / 8 ^ (r & 7)) << 4) + d % 8 * 2;
#pragma unroll
      for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(dst + k * KC * ST_TILE) = t[k];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(q_ready));
    const int pos = row < ntok ? pos0 + row : -1, first = st_first_key(max(pos, 0), a.mask, a.mask_size);
    float m = -CUDART_INF_F, l = 0.f;             // the row's reference (in units of log 2), this thread's keys' weights
    float acc[DV / 4] = {};                       // the row's output, this thread's dimensions
    auto gather = [&](int j) {                    // += the run that the MMAs of block j ended in tensor memory
      if (!wait(&o_done[j & 1], j >> 1 & 1)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < DV / 4; c += 16) {
        uint32_t o[16];
        tmem_ld8(tmem + lanes + st_run_col<DV>(j) + part * (DV / 4) + c, o);
        tmem_ld8(tmem + lanes + st_run_col<DV>(j) + part * (DV / 4) + c + 8, o + 8);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(o[i]);
      }
      return true;
    };
    bool ok = true, waiting = false;              // (a run is whole and not in `acc` yet)
    for (int j = 0; j < n_blk; ++j) {             // (also behind a wait that ran out: the row's other thread may be at the exchange)
      const int b = j & 1;
      const bool there = 2 * j + half < n_visit;
      const int page0 = page_at(there ? 2 * j + half : 2 * j) * PAGE, key0 = page0 + part % 2 * 32;
      const uint32_t s_addr = tmem + lanes + b * ST_BUF_COLS + part * 32;
      if (ok) ok = wait(&s_ready[b], j >> 1 & 1);
      uint32_t r[32];
      float mx = -CUDART_INF_F;
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_ld32(s_addr, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (!there || hidden(key0, 32)) {
          // (a bit a key: five instructions a score, with its place compared to each bound, made a masked block twice as long)
          const uint32_t seen = (there ? st_low_bits(pos - key0 + 1) : 0u) & (~st_low_bits(first - key0) | st_low_bits(a.keep - key0));
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (!(seen >> i & 1)) r[i] = __float_as_uint(-CUDART_INF_F);
        }
        float mx1 = -CUDART_INF_F;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          mx = fmaxf(mx, fmaxf(__uint_as_float(r[i]), __uint_as_float(r[i + 1])));
          mx1 = fmaxf(mx1, fmaxf(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])));
        }
        mx = fmaxf(mx, mx1);
      }
      row_max[(b * 4 + part) * ST_ROWS + row] = mx;
      asm volatile("bar.sync %0, 128;" ::"r"(quarter + 1) : "memory");      // the row's four threads (warps w, w + 4, w + 8, w + 12)
      if (!ok) continue;
#pragma unroll
      for (int k = 1; k < 4; ++k) mx = fmaxf(mx, row_max[(b * 4 + (part ^ k)) * ST_ROWS + row]);
      mx = mx == -CUDART_INF_F ? mx : mx * scale2;
      float rescale = 1.f;
      if (j == 0) {
        m = mx;
      } else if (mx > m + ST_LAZY) {
        rescale = sp_exp2(m - mx);                 // (0 if the row has seen no key so far)
        m = mx;
        l *= rescale;
      }
      if (j > 0 && !(j & 1)) waiting = true;       // the run before this block's is whole, or soon
      if (__any_sync(0xffffffffu, rescale != 1.f)) {       // (rare after the first blocks; all warps of the rows take it)
        if (waiting) ok = gather(j - 1 - (j & 1));
        waiting = false;
        if (ok && (j & 1)) {                       // the run's first block is in tensor memory
          ok = wait(&o_done[0], j >> 1 & 1);
          if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c = 0; c < DV / 4; c += 8) {
              uint32_t o[8];
              const uint32_t at = tmem + lanes + st_run_col<DV>(j) + part * (DV / 4) + c;
              tmem_ld8(at, o);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * rescale);
              st_tmem_st4(at, o);
              st_tmem_st4(at + 4, o + 4);
            }
          }
        }
        if (!ok) continue;
#pragma unroll
        for (int i = 0; i < DV / 4; ++i) acc[i] *= rescale;
      }
      const float ref = m == -CUDART_INF_F ? 0.f : m;
      float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {                // 8 keys: 4 columns of each term
        uint32_t t[3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float p0 = sp_exp2(fmaf(__uint_as_float(r[c * 8 + 2 * i]), scale2, -ref)), p1 = sp_exp2(fmaf(__uint_as_float(r[c * 8 + 2 * i + 1]), scale2, -ref));
          sum0 += p0;
          sum1 += p1;
          sp_split(p0, p1, t[0][i], t[1][i], t[2][i]);
        }
        st_tmem_st4(s_addr + c * 4, t[0]);
        st_tmem_st4(s_addr + 16 + c * 4, t[1]);
        st_tmem_st4(tmem + lanes + b * ST_BUF_COLS + 128 + part * 16 + c * 4, t[2]);
      }
      l += sum0 + sum1;
      if (waiting && (DV != 64 || (j & 1))) {      // before the next block's MMAs may take its columns
        waiting = false;
        ok = gather(j - 1 - (j & 1));
        if (!ok) continue;
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_ready[b]));
    }
    if (ok && waiting) ok = gather(n_blk - 2);     // (the last block has a run of its own)
    if (ok) ok = gather(n_blk - 1);
    if (ok && *taken_out && row < ntok) {         // (rare: values that were taken out above, to the rows that see them)
      for (int i = 0; i < n_visit; ++i) {
        if (!some_hidden(i / 2)) continue;
        const int pg = page_at(i), page = a.page_table ? a.page_table[(size_t)seq * a.table_stride + pg] : 0;
        const __nv_bfloat16* values = a.page_table ? a.values + ((size_t)(page < 0 || page >= a.n_pages ? 0 : page) * a.nkv + kvh) * PAGE * DV
                                                   : a.values + ((size_t)(tok0 - pos0 + pg * PAGE) * a.nkv + kvh) * DV;
        const size_t pitch = a.page_table ? DV : (size_t)a.nkv * DV;
#pragma unroll 1
        for (int k = 0; k < PAGE; ++k) {
          const int key = pg * PAGE + k;
          if (key > pos || (key < first && key >= a.keep)) continue;
          const uint2* at = reinterpret_cast<const uint2*>(values + k * pitch + part * (DV / 4));
#pragma unroll
          for (int c = 0; c < DV / 16; ++c) {
            const uint2 v = at[c];
            if ((st_no_number(v.x) | st_no_number(v.y)) == 0) continue;
            const uint32_t w[2] = {v.x & ~st_numbers_mask(v.x), v.y & ~st_numbers_mask(v.y)};
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[c * 4 + e] += __uint_as_float(e & 1 ? w[e / 2] & 0xffff0000u : w[e / 2] << 16);
          }
        }
      }
    }
    row_sum[part * ST_ROWS + row] = l;
    asm volatile("bar.sync %0, 128;" ::"r"(quarter + 1) : "memory");
    float den = (row_sum[row] + row_sum[ST_ROWS + row]) + (row_sum[2 * ST_ROWS + row] + row_sum[3 * ST_ROWS + row]), fix = 1.f;
    if (a.sink != nullptr) {                       // one more term of the denominator
      const float s2 = a.sink[head] * 1.4426950408889634f, nm = fmaxf(m, s2);
      fix = exp2f(m - nm);
      den = den * fix + exp2f(s2 - nm);
    }
    float inv = den > 0.f ? fix / den : 0.f;
    if (den != den) inv = den;                     // (not a number stays one)
    const bool mine = row < ntok;
    const size_t tok = (size_t)(tok0 + row);
    if (a.gate != nullptr && !a.gate_ch && mine) inv *= 1.0f / (1.0f + expf(-a.gate[tok * a.ldg + head]));
    if (!ok) inv = __uint_as_float(0x7fc00000u);   // a wait that ran out: nothing that could pass for a result
    if (mine) {
#pragma unroll
      for (int c = 0; c < DV / 4; c += 8) {
        const int d = part * (DV / 4) + c;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = acc[c + i] * inv;
        if (a.gate != nullptr && a.gate_ch) {
          const float* g = a.gate + tok * a.ldg + head * DV + d;
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] *= 1.0f / (1.0f + expf(-g[i]));
        }
        if (a.maps > 1) {
          float4* dst = reinterpret_cast<float4*>(static_cast<float*>(a.out) + tok * a.ldo + head * DV + d);
          dst[0] = make_float4(v[0], v[1], v[2], v[3]);
          dst[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
          __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.out) + tok * a.ldo + head * DV + d;
          store_piece(dst, make_float4(v[0], v[1], v[2], v[3]));
          store_piece(dst + 4, make_float4(v[4], v[5], v[6], v[7]));
        }
      }
    }
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <int DK, int DV>
static int launch_split_tc(const CUtensorMap& mk, const CUtensorMap& mv, const SplitTcArgs& a, cudaStream_t stream) {
  constexpr int smem = StSizes<DK, DV>::smem;
  static_assert(smem <= 227 * 1024, "shared memory");
  auto kern = attn_prefill_split_tc_kernel<DK, DV>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  EL_REFUSE(e == cudaSuccess, "attn_prefill_split_tc: %d bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
  kern<<<dim3(a.nh * a.maps, a.n_tiles), ST_THREADS, smem, stream>>>(mk, mv, a);
  return 0;
}

}  // namespace edgelm

using namespace edgelm;

// Tokens per tile that the host must cut sequences into for this kernel.
extern "C" int edgelm_attn_prefill_split_tc_tile_tokens() { return ST_ROWS; }

// 1 if the kernel takes these key and value head sizes and maps a head, else 0: value sizes of whole tiles of 64 dimensions, whose columns of tensor
// memory the softmax threads share out in pieces of 16, over key sizes from 64 on.  Value sizes of 32 and 96, and key sizes of 32, stay on mma.sync:
// they would need other pieces, and no form of them has been built or measured.
extern "C" int edgelm_attn_prefill_split_tc_takes(int dk, int dv, int maps) {
  if (maps == 2) return dk == 64 && (dv == 64 || dv == 128) ? 1 : 0;
  return maps == 1 && ((dv == 64 && (dk == 64 || dk == 96 || dk == 128)) || (dv == 128 && dk == 128)) ? 1 : 0;
}

// As `edgelm_attn_prefill_split`, over tiles of at most 128 tokens; `n_pages` of the cache, or, with `page_table` null, the step's rows of
// `kcache` and `vcache` ([rows][kv heads][...]).  `err`: the device error word (waits that run out, pages out of range).
extern "C" int edgelm_attn_prefill_split_tc(const float* q, int ldq, void* out, int ldo, const void* kcache, const void* vcache, int n_pages,
                                            const int32_t* page_table, int table_stride, const int32_t* tile_seq, const int32_t* tile_tok0,
                                            const int32_t* tile_ntok, const int32_t* tile_pos0, int n_tiles, int nh, int nkv, int dk, int dv, float scale,
                                            int mask, int mask_size, const float* sink, const float* gate, int ldg, int keep, int gate_ch, int maps,
                                            int* err, cudaStream_t stream) {
  if (n_tiles == 0) return 0;
  EL_REFUSE(nh > 0 && nkv > 0 && nh % nkv == 0, "attn_prefill_split_tc: %d query heads are not a multiple of %d key/value heads", nh, nkv);
  EL_REFUSE(edgelm_attn_prefill_split_tc_takes(dk, dv, maps), "attn_prefill_split_tc: head sizes %d / %d with %d maps", dk, dv, maps);
  EL_REFUSE(maps == 1 || (sink == nullptr && gate == nullptr), "attn_prefill_split_tc: two maps take no sink and no gate");
  EL_REFUSE(ldq % 4 == 0 && ldo % 4 == 0 && (uintptr_t)q % 16 == 0 && (uintptr_t)out % 16 == 0, "attn_prefill_split_tc: rows must be 16- and 8-byte aligned");
  EL_REFUSE((uintptr_t)kcache % 16 == 0 && (uintptr_t)vcache % 16 == 0, "attn_prefill_split_tc: keys and values must be 16-byte aligned");
  EL_REFUSE(mask == ST_MASK_CAUSAL || ((mask == ST_MASK_WINDOW || mask == ST_MASK_CHUNK) && mask_size >= 1), "attn_prefill_split_tc: mask %d of size %d", mask, mask_size);
  EL_REFUSE(keep >= 0 && (keep == 0 || mask == ST_MASK_WINDOW) && (gate_ch == 0 || gate_ch == dv), "attn_prefill_split_tc: %d kept keys, a gate of %d channels", keep, gate_ch);
  EL_REFUSE(err != nullptr && n_tiles > 0 && n_tiles <= 65535 && n_pages > 0 && (long long)n_pages * nkv * PAGE < (1LL << 31), "attn_prefill_split_tc: bad grid");
  CUtensorMap mk, mv;
  if (page_table) {
    if (tensor_map(kcache, n_pages * nkv * PAGE, dk * maps, dk * maps, PAGE, &mk)) return -1;
    if (tensor_map(vcache, n_pages * nkv * PAGE, dv, dv, PAGE, &mv)) return -1;
  } else {
    if (tensor_map(kcache, n_pages, nkv * maps * dk, nkv * maps * dk, PAGE, &mk)) return -1;
    if (tensor_map(vcache, n_pages, nkv * dv, nkv * dv, PAGE, &mv)) return -1;
  }
  const SplitTcArgs a{q, (const __nv_bfloat16*)vcache, ldq, out, ldo, page_table, table_stride, n_pages, tile_seq, tile_tok0, tile_ntok, tile_pos0, n_tiles, nh, nkv, maps, scale,
                      gate, ldg, mask, mask_size, sink, keep, gate_ch, err};
  int rc = 0;
  if (dk == 64 && dv == 64) rc = launch_split_tc<64, 64>(mk, mv, a, stream);
  else if (dk == 64) rc = launch_split_tc<64, 128>(mk, mv, a, stream);
  else if (dk == 96) rc = launch_split_tc<96, 64>(mk, mv, a, stream);
  else if (dv == 64) rc = launch_split_tc<128, 64>(mk, mv, a, stream);
  else rc = launch_split_tc<128, 128>(mk, mv, a, stream);
  if (rc) return rc;
  EL_LAUNCH_CHECK("attn_prefill_split_tc");
  return 0;
}
