// Direct bit-sliced count (see direct.cuh).
//
// A warp takes 64 plane words (2,048 starts) at a time.  For each kind of
// pattern byte in use it writes the mismatch row -- bit p set where genome
// byte p mismatches that kind -- to shared memory; pattern position k of all
// 32 starts of a word is then one funnel shift of two row words.  The PAM's
// positions are OR-ed into the candidate masks; a variant's are summed by
// carry-save adders (3 LOP3 per position and word) and compared with its
// limit, for 32 starts per word at once.  The work does not depend on how
// many starts match the PAM, so it suits patterns that nearly every start
// matches: 3 variants of 40 positions over 30 M starts of an all-N pattern
// take 0.12 ms (finder and popcount comparer 3.0 ms, finder and screen 0.70).
// Bound by issue (22 instructions per position and 64 words) and by the four
// shared loads among them: 185 SM clocks per 2,048 starts and 12.5 per
// position, so that one 20-nt variant costs as much as the scanning screen of
// an NRG pattern (450 to 530) and more than that of an NGG one (280).
#include <algorithm>

#include "cof_internal.h"
#include "direct.cuh"
#include "finder.cuh"

namespace cof {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kDirectThreads = 256;
constexpr int kDirectCtas = 5;  // per SM
constexpr uint32_t kRowWords = 68;  // 64 words, up to 3 that their windows reach, one for padding

__device__ __forceinline__ uint32_t maj3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0xE8>(a, b, c); }
__device__ __forceinline__ uint32_t xor3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0x96>(a, b, c); }

// The mismatch word of class bits `cls` (any value; warp-uniform).
__device__ __forceinline__ uint32_t class_word(uint32_t cls, uint32_t h, uint32_t l, uint32_t o) {
  const uint32_t t = 0u - (cls & 1u), c = 0u - (cls >> 1 & 1u), a = 0u - (cls >> 2 & 1u), g = 0u - (cls >> 3 & 1u),
                 x = 0u - (cls >> 4 & 1u);
  auto mux = [](uint32_t s, uint32_t p, uint32_t q) { return (s & p) | (~s & q); };
  return mux(o, x, mux(h, mux(l, g, a), mux(l, c, t)));
}

// NB: planes of the counts (positions < 2^NB).
template <int NB>
__global__ void __launch_bounds__(kDirectThreads, kDirectCtas)
    direct_kernel(const __grid_constant__ GenomeView g, uint64_t w_begin, uint32_t words, uint64_t pos_end,
                  const __grid_constant__ DirectParams P, unsigned long long* __restrict__ qcount,
                  const __grid_constant__ HitSink sink) {
  extern __shared__ uint32_t rows_all[];
  const unsigned lane = threadIdx.x & 31;
  uint32_t* rows = rows_all + (threadIdx.x >> 5) * P.rows * kRowWords;
  const char* mine = (const char*)(rows + lane);
  const uint32_t units = (words + 63) / 64;
  const uint32_t *hi = g.hi + w_begin, *lo = g.lo + w_begin, *ot = g.ot + w_begin;
  const uint32_t starts = pos_end > (w_begin << 5) ? (uint32_t)min(pos_end - (w_begin << 5), (uint64_t)words << 5) : 0u;
  uint32_t found = 0;
  for (uint32_t i = lane; i < kRowWords; i += 32) rows[i] = 0;
  // Position `e` of the starts of words lane and lane + 32.
  auto at = [&](uint32_t e, uint32_t& x0, uint32_t& x1) {
    const uint32_t* r = (const uint32_t*)(mine + (e >> 5) * 4);
    x0 = __funnelshift_r(r[0], r[1], e);
    x1 = __funnelshift_r(r[32], r[33], e);
  };
  for (uint32_t s = (blockIdx.x * kDirectThreads + threadIdx.x) / 32; s < units; s += gridDim.x * kDirectThreads / 32) {
    // Words past the end repeat the last ones (their starts are cut off
    // below); the planes hold two words past the last start's.
    __syncwarp();
    bool sep = false;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const uint32_t i = lane + 32 * j, w = min(s * 64 + i, words + 1);
      if (j == 2 && lane >= 3) continue;
      const uint32_t h = __ldg(hi + w), l = __ldg(lo + w), o = __ldg(ot + w);
      const uint32_t sw = o & l & ~h;
      rows[kRowWords + i] = sw;
      sep |= sw != 0;
      for (uint32_t r = 2; r < P.rows; ++r) rows[r * kRowWords + i] = class_word(P.row_class[r], h, l, o);
    }
    __syncwarp();
    uint32_t keep[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t w = s * 64 + lane + 32 * j, p = w << 5;
      keep[j] = w >= (starts + 31) / 32 ? 0u : starts - p >= 32 ? kFull : kFull >> (32 - (starts - p));
    }
    if (__any_sync(kFull, sep)) {
      // Drop windows holding a record separator.
      for (uint32_t q = 0; q < P.L; ++q) {
        uint32_t x0, x1;
        at((kRowWords + (q >> 5)) << 5 | (q & 31), x0, x1);
        keep[0] &= ~x0;
        keep[1] &= ~x1;
      }
    }
#pragma unroll 1
    for (uint32_t strand = 0; strand < 2; ++strand) {
      uint32_t bad0 = ~keep[0], bad1 = ~keep[1];
      for (uint32_t j = 0; j < P.pam_n[strand]; ++j) {
        uint32_t x0, x1;
        at(P.pam[strand][j], x0, x1);
        bad0 |= x0;
        bad1 |= x1;
      }
      if (!__any_sync(kFull, ~(bad0 & bad1))) continue;
      found += __popc(~bad0) + __popc(~bad1);
#pragma unroll 1
      for (uint32_t v = 0; v < P.variants; ++v) {
        uint32_t b[2][NB] = {};
        for (uint32_t k = 0; k < P.n[v]; k += 4) {
          uint32_t x[4][2];
          const uint2 e = *(const uint2*)&P.pos[v][strand][k];
          at(e.x & 0xFFFFu, x[0][0], x[0][1]);
          at(e.x >> 16, x[1][0], x[1][1]);
          at(e.y & 0xFFFFu, x[2][0], x[2][1]);
          at(e.y >> 16, x[3][0], x[3][1]);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint32_t* p = b[i];
            const uint32_t c0 = maj3(p[0], x[0][i], x[1][i]);
            p[0] = xor3(p[0], x[0][i], x[1][i]);
            const uint32_t c1 = maj3(p[0], x[2][i], x[3][i]);
            p[0] = xor3(p[0], x[2][i], x[3][i]);
            uint32_t t = maj3(p[1], c0, c1);
            p[1] = xor3(p[1], c0, c1);
#pragma unroll
            for (int n = 2; n < NB; ++n) {
              const uint32_t u = p[n] & t;
              p[n] ^= t;
              t = u;
            }
          }
        }
        // count + (2^NB - 1 - limit) carries out exactly where count > limit.
        const uint32_t bias = (1u << NB) - 1 - min(P.limit[v], (1u << NB) - 1);
        uint32_t over0 = 0, over1 = 0;
#pragma unroll
        for (int n = 0; n < NB; ++n) {
          const uint32_t k = 0u - (bias >> n & 1u);
          over0 = maj3(b[0][n], k, over0);
          over1 = maj3(b[1][n], k, over1);
        }
        if (!__any_sync(kFull, ~((over0 | bad0) & (over1 | bad1)))) continue;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          for (uint32_t hit = ~(i ? over1 | bad1 : over0 | bad0); hit; hit &= hit - 1) {
            const uint32_t c = __ffs(hit) - 1;
            uint32_t mm = 0;
#pragma unroll
            for (int n = 0; n < NB; ++n) mm |= (b[i][n] >> c & 1u) << n;
            const unsigned long long to = atomicAdd(sink.count, 1ull);
            if (to < sink.cap)
              sink.hits[to] = make_hit(P.id[v], ((w_begin + s * 64ull + lane + 32 * i) << 5) + c, strand, mm);
          }
      }
    }
  }
  if (qcount) {
    found = __reduce_add_sync(kFull, found);
    if (lane == 0 && found) atomicAdd(qcount, (unsigned long long)found);
  }
}

}  // namespace

bool plan_direct(const std::string& pattern, const DirectVariant* vars, size_t n, DirectParams& p) {
  p = DirectParams();
  const uint32_t L = (uint32_t)pattern.size();
  if (L == 0 || L > (uint32_t)kMaxL || n == 0 || n > (size_t)kDirectVariants) return false;
  p.L = L;
  p.variants = (uint32_t)n;
  p.rows = 2;
  // The place of pattern byte `c` at window position k; 0xFFFF: no row left.
  auto place = [&](unsigned char c, uint32_t k) -> uint32_t {
    const uint32_t cls = class_bits_of(c);
    uint32_t r = 2;
    while (r < p.rows && p.row_class[r] != cls) ++r;
    if (r == (uint32_t)kDirectRows) return 0xFFFFu;
    if (r == p.rows) p.row_class[p.rows++] = (uint8_t)cls;
    return (r * kRowWords + (k >> 5)) << 5 | (k & 31);
  };
  // Positions that can mismatch, of a string and of its reverse complement.
  auto list = [&](const std::string& s, uint32_t strand, uint16_t* out, uint32_t& count) {
    count = 0;
    for (uint32_t k = 0; k < L; ++k) {
      const unsigned char c = strand ? complement_byte((unsigned char)s[L - 1 - k]) : (unsigned char)s[k];
      if (!class_bits_of(c)) continue;
      const uint32_t e = place(c, k);
      if (e == 0xFFFFu) return false;
      out[count++] = (uint16_t)e;
    }
    return true;
  };
  for (uint32_t strand = 0; strand < 2; ++strand) {
    if (!list(pattern, strand, p.pam[strand], p.pam_n[strand])) return false;
    for (size_t v = 0; v < n; ++v) {
      if (vars[v].key.size() != L || !list(vars[v].key, strand, p.pos[v][strand], p.n[v])) return false;
      p.n[v] = (p.n[v] + 3) & ~3u;  // the rest of pos points at row 0
    }
  }
  for (size_t v = 0; v < n; ++v) {
    p.id[v] = vars[v].id;
    p.limit[v] = vars[v].limit;
  }
  return true;
}

double direct_cost(const DirectParams& p) {
  double c = 185.0;
  for (uint32_t v = 0; v < p.variants; ++v) c += 12.5 * p.n[v];
  return c;
}

void launch_direct(const GenomeView& g, uint64_t w_begin, uint64_t w_end, const DirectParams& p, unsigned long long* qcount,
                   const HitSink& sink, int sm_count, cudaStream_t stream) {
  uint32_t most = 0;
  for (uint32_t v = 0; v < p.variants; ++v) most = std::max(most, p.n[v]);
  const uint64_t pos_end = g.n >= p.L ? g.n - p.L + 1 : 0;
  const size_t smem = (size_t)kDirectThreads / 32 * p.rows * kRowWords * 4;
  auto kernel = most < 32 ? direct_kernel<5> : direct_kernel<7>;
  // At most 2^26 words at a time (starts are counted in 32 bits).
  for (uint64_t w0 = w_begin; w0 < w_end; w0 += 1ull << 26) {
    const uint32_t words = (uint32_t)std::min<uint64_t>(w_end - w0, 1ull << 26);
    const uint32_t ctas = ((words + 63) / 64 + kDirectThreads / 32 - 1) / (kDirectThreads / 32);
    kernel<<<std::min<uint32_t>(ctas, (uint32_t)sm_count * kDirectCtas), kDirectThreads, smem, stream>>>(
        g, w0, words, pos_end, p, qcount, sink);
  }
}

}  // namespace cof
