// Error reporting and small queries of the kernel library.
#include <cstdarg>
#include <cstring>

#include "common.cuh"

namespace edgelm {

static thread_local char g_error[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

static int g_pdl = 57;   // the few-rows matrix products (bit 0), the tcgen05 products (bits 3 and 5), the tcgen05 prefill attention
                         // (bit 4), RMSNorm and the rotation (bit 5) start under the tail of the kernel before them
int pdl_enabled() { return g_pdl; }

}  // namespace edgelm

// Switch programmatic dependent launch of the decode kernels on (1, the default) or off (0).
extern "C" int edgelm_set_pdl(int on) {
  edgelm::g_pdl = on;
  return 0;
}

// Message of the last refused or failed call of this thread.
extern "C" const char* edgelm_last_error() { return edgelm::g_error; }

// Compute capability of the current device as major * 10 + minor, or a negative code.
extern "C" int edgelm_device_arch() {
  int dev = 0, major = 0, minor = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess) return -1;
  return major * 10 + minor;
}

// A step's metadata laid out in the host's staging buffer, section behind section, for the one copy that brings it to the device:
//   ids [T], position [T] and sequence [T] of every token; last position [B], first packed row [B + 1]; wanted rows [R]; slots [B]; every
//   table's rows of the slots [B stride]; and, in steps of more than one token a sequence, four columns of every tile size's tiles (sequence,
//   first packed token, tokens, first position), runs of at most so many consecutive tokens of one sequence.
// `first` [7 + tables + 4 tile sizes + 1] gets every section's first word and the end.  Host code only; refuses what does not fit
// into `capacity` words before anything is written.  (6,000 tokens: the same passes as NumPy calls took 100 to 150 us, with the GPU idle.)
extern "C" int edgelm_lay_out_step(int32_t* host, long long capacity, const int64_t* ids, long long T, const int64_t* ntok, const int64_t* pos0,
                                   const int64_t* slots, int B, const int64_t* want, int R, int n_tables, const int32_t* const* tables, const int* strides,
                                   const int* table_rows, int n_tile_sizes, const int* tile_sizes, int64_t* first) {
  EL_REFUSE(host && T >= 0 && B >= 0 && R >= 0 && n_tables >= 0 && n_tile_sizes >= 0, "lay_out_step: bad sizes");
  const bool tiled = T != B;
  long long words = 3 * T + 3LL * B + 1 + R, sum = 0;
  for (int b = 0; b < B; ++b) {
    EL_REFUSE(ntok[b] >= 0, "lay_out_step: %lld tokens", (long long)ntok[b]);
    sum += ntok[b];
    for (int g = 0; g < n_tables; ++g) EL_REFUSE(slots[b] >= 0 && slots[b] < table_rows[g], "lay_out_step: slot %lld of %d", (long long)slots[b], table_rows[g]);
    for (int i = 0; tiled && i < n_tile_sizes; ++i) words += 4 * ((ntok[b] + tile_sizes[i] - 1) / tile_sizes[i]);
  }
  EL_REFUSE(sum == T, "lay_out_step: %lld tokens in sequences of %lld", T, sum);
  for (int g = 0; g < n_tables; ++g) words += (long long)B * strides[g];
  EL_REFUSE(words <= capacity, "lay_out_step: %lld words into a buffer of %lld", words, capacity);
  int32_t* p = host;
  int section = 0;
  auto begin = [&]() { first[section++] = p - host; };
  begin();
  for (long long t = 0; t < T; ++t) *p++ = (int32_t)ids[t];
  begin();
  for (int b = 0; b < B; ++b)
    for (int64_t t = 0; t < ntok[b]; ++t) *p++ = (int32_t)(pos0[b] + t);
  begin();
  for (int b = 0; b < B; ++b)
    for (int64_t t = 0; t < ntok[b]; ++t) *p++ = b;
  begin();
  for (int b = 0; b < B; ++b) *p++ = (int32_t)(pos0[b] + ntok[b] - 1);
  begin();
  long long row = 0;
  for (int b = 0; b < B; ++b) {
    *p++ = (int32_t)row;
    row += ntok[b];
  }
  *p++ = (int32_t)T;
  begin();
  for (int r = 0; r < R; ++r) *p++ = (int32_t)want[r];
  begin();
  for (int b = 0; b < B; ++b) *p++ = (int32_t)slots[b];
  for (int g = 0; g < n_tables; ++g) {
    begin();
    for (int b = 0; b < B; ++b, p += strides[g]) memcpy(p, tables[g] + slots[b] * strides[g], (size_t)strides[g] * 4);
  }
  for (int i = 0; tiled && i < n_tile_sizes; ++i) {
    const int64_t size = tile_sizes[i];
    for (int column = 0; column < 4; ++column) {
      begin();
      int64_t t0 = 0;
      for (int b = 0; b < B; t0 += ntok[b++])
        for (int64_t a = 0; a < ntok[b]; a += size)
          *p++ = (int32_t)(column == 0 ? b : column == 1 ? t0 + a : column == 2 ? (ntok[b] - a < size ? ntok[b] - a : size) : pos0[b] + a);
    }
  }
  first[section] = p - host;
  return 0;
}
