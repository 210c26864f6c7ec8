// cof_search_chunk_static: search one genome chunk without allocating memory.
//
// Who needs this: callers that are not allowed to allocate device memory at
// the point where they search -- for example a host application that reserves
// all of its GPU memory up front in its own pool and forbids other
// allocations, or a latency-sensitive caller for whom the implicit device-wide
// synchronization of cudaMalloc/cudaFree would stall unrelated streams.  Such a
// caller owns the genome planes and the hit buffer (device memory it allocated
// earlier) and passes them in.  The direct count (direct.cuh) needs no other
// device memory: the pattern and the compare string travel as a kernel
// argument, and no candidate is stored.  One kernel after the counter's reset:
// 12.3 us of GPU time for 2^20 positions (28.3 for a finder, a comparer and
// the store of the compare masks).  A caller that then sorts its hits with
// torch (59 us alone) waits 73 us for both (79).
//
// Chunks longer than kStaticMaxPositions are rejected with COF_ERR_TOO_LARGE.
//
// The pattern and compare string are upper-cased first, as the reference does
// with its input file; every other byte keeps its meaning (IUPAC codes, 'N'
// and any byte outside the IUPAC set never mismatch).
#include <cuda_runtime.h>

#include <cstring>
#include <string>

#include "../../include/cof.h"
#include "cof_internal.h"
#include "direct.cuh"

namespace {

using namespace cof;

constexpr uint64_t kStaticMaxPositions = 1ull << 21;

// The reference upper-cases the pattern and every guide before it builds its
// compare strings (cas-offinder.cpp:625, :640); so does this entry point.
std::string upper_of(const char* s, uint32_t L) {
  std::string r(s, L);
  for (char& c : r)
    if (c >= 'a' && c <= 'z') c = (char)(c - 32);
  return r;
}

}  // namespace

extern "C" cof_status cof_search_chunk_static(const uint32_t* d_hi, const uint32_t* d_lo, const uint32_t* d_ot,
                                              uint64_t n, const char* pattern, const char* comp,
                                              uint32_t patternlen, uint16_t threshold, uint64_t* d_hits,
                                              uint64_t hit_cap, unsigned long long* d_hit_count, void* stream) {
  if (!d_hi || !d_lo || !d_ot || !pattern || !comp || !d_hits || !d_hit_count) return COF_ERR_ARG;
  if (patternlen == 0 || patternlen > (uint32_t)kMaxL) return COF_ERR_UNSUPPORTED;
  if (n > kStaticMaxPositions) return COF_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  // An unread error of the caller's own CUDA work is left for the caller:
  // nothing is queued, so every error this call reports after its launches
  // is its own.
  if (cudaPeekAtLastError() != cudaSuccess) return COF_ERR_CUDA;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return COF_ERR_CUDA;

  // The counter starts at zero on every call.
  if (cudaMemsetAsync(d_hit_count, 0, sizeof(unsigned long long), st) != cudaSuccess) return COF_ERR_CUDA;
  const uint64_t npos = n >= patternlen ? n - patternlen + 1 : 0;
  if (npos == 0) return COF_OK;

  const DirectVariant var{upper_of(comp, patternlen), 0, threshold};
  DirectParams params;
  if (!plan_direct(upper_of(pattern, patternlen), &var, 1, params)) return COF_ERR_UNSUPPORTED;
  GenomeView g;
  std::memset(&g, 0, sizeof g);
  g.hi = d_hi;
  g.lo = d_lo;
  g.ot = d_ot;
  g.n = n;
  launch_direct(g, 0, (npos + 31) / 32, params, nullptr, HitSink{d_hits, d_hit_count, hit_cap}, sms, st);
  return cudaGetLastError() == cudaSuccess ? COF_OK : COF_ERR_CUDA;
}
