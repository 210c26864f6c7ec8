// Table screen: table construction and the screening kernel (see screen.cuh).
#include <algorithm>

#include "finder.cuh"
#include "screen.cuh"

namespace cof {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kScreenThreads = 1024;  // one CTA per SM shares one set of tables
constexpr int kPerLane = 2;           // candidates per lane and iteration

__device__ __forceinline__ uint32_t mux(uint32_t s, uint32_t a, uint32_t b) { return (s & a) | (~s & b); }

// Shared-memory accesses at byte addresses of the shared window (32-bit
// address arithmetic).
template <uint32_t IMM>
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(IMM));
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
template <uint32_t IMM>
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(IMM));
  return v;
}
__device__ __forceinline__ void sts16(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((uint16_t)v) : "memory");
}

// One record's class masks; bit k = oriented window position k.
template <int NW>
struct Record {
  uint32_t t[NW], c[NW], a[NW], g[NW], o[NW], meta;
  __device__ __forceinline__ explicit Record(const uint32_t* __restrict__ p) {
    const uint4 x = __ldg((const uint4*)p), y = __ldg((const uint4*)p + 1);
    t[0] = x.x, c[0] = x.y, a[0] = x.z, g[0] = x.w;
    o[0] = y.x, meta = y.y;
    if (NW == 2) {
      const uint4 z = __ldg((const uint4*)p + 2);
      o[NW - 1] = y.z;
      t[NW - 1] = z.x, c[NW - 1] = z.y, a[NW - 1] = z.z, g[NW - 1] = z.w;
    }
  }
};

// A thread takes one class of one table entry: the least mismatch count on
// the run over the class's variants, capped.  A warp's lanes take consecutive
// entries and read the same records (a broadcast), the CTA's warps the word's
// classes, whose fields are joined in shared memory.  (One thread per entry
// with all classes took 34 us for 217 variants, waiting on its record loads.)
template <int NW>
__global__ void __launch_bounds__(256) screen_tables_kernel(const __grid_constant__ ScreenGeom G,
                                                            const uint32_t* __restrict__ records,
                                                            const uint32_t* __restrict__ first,
                                                            uint32_t* __restrict__ tables) {
  __shared__ uint32_t field[8][32];
  const uint32_t entries = screen_entries(G.K), lane = threadIdx.x & 31, c = threadIdx.x >> 5;
  const uint32_t i = blockIdx.x * 32 + lane, word = blockIdx.y;
  uint32_t k = 0;
  while (k + 1 < G.K && i >= screen_base(k + 1)) ++k;
  const uint32_t x = i - screen_base(k), q = screen_run_len(G.K, k), m = (1u << q) - 1u, a = G.a0 + screen_run_at(k);
  const uint32_t h = x & m, l = x >> q;  // the run's plane bits
  const uint32_t* f = first + word * (G.fields + 1);
  int least = (int)G.cap[k];
  if (c < G.fields) {
    const uint32_t v1 = f[c + 1];
#pragma unroll 4
    for (uint32_t v = f[c]; v < v1; ++v) {
      const Record<NW> r(records + (size_t)v * screen_record_words(NW));
      auto run = [&](const uint32_t (&w)[NW]) {
        if (NW == 1) return a < 32 ? w[0] >> a : 0u;
        return a < 32 ? __funnelshift_r(w[0], w[NW - 1], a) : a < 64 ? w[NW - 1] >> (a - 32) : 0u;
      };
      int d = __popc(mux(h, mux(l, run(r.g), run(r.a)), mux(l, run(r.c), run(r.t))) & m);
      if (k == 0) d += (1 << (G.bits - 1)) - 1 - (int)(r.meta & 15u);
      least = min(least, d);
    }
  }
  field[c][lane] = c < G.fields ? (uint32_t)least << (c * G.bits) : 0u;
  __syncthreads();
  if (c == 0) {
    uint32_t out = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) out |= field[j][lane];
    tables[(size_t)word * entries + i] = out;
  }
}

template <int NW>
__device__ __forceinline__ void orient_plane(uint32_t (&w)[NW], bool minus, bool flip, uint32_t L) {
  if (NW == 1) {
    const uint32_t r = __brev(w[0]) >> (32 - L);
    w[0] = minus ? (flip ? ~r : r) : w[0];
  } else {
    const uint64_t x = __brevll(((uint64_t)w[NW - 1] << 32) | w[0]) >> (64 - L);
    const uint64_t y = flip ? ~x : x;
    w[0] = minus ? (uint32_t)y : w[0];
    w[NW - 1] = minus ? (uint32_t)(y >> 32) : w[NW - 1];
  }
}

template <int NW>
__device__ __forceinline__ void load_plane(uint32_t (&w)[NW], const uint32_t* __restrict__ plane, uint32_t at,
                                           uint32_t r) {
  uint32_t x[NW + 1];
#pragma unroll
  for (int i = 0; i <= NW; ++i) x[i] = __ldg(plane + at + i);
#pragma unroll
  for (int i = 0; i < NW; ++i) w[i] = __funnelshift_r(x[i], x[i + 1], r);
}

// The looked-up entry of run R: h, l hold the screen's first position in bit 0.
template <int K, int R>
__device__ __forceinline__ uint32_t run_entry(uint32_t tab_addr, uint32_t h, uint32_t l) {
  constexpr uint32_t at = screen_run_at(R), q = screen_run_len(K, R), m = ((1u << q) - 1u) << 2;
  // A run's hi bits go to bits 2.., its lo bits above them.
  const uint32_t x = at >= 2 ? h >> (at >= 2 ? at - 2 : 0) : h << (at < 2 ? 2 - at : 0);
  const uint32_t y = at >= 2 + q ? l >> (at >= 2 + q ? at - 2 - q : 0) : l << (at < 2 + q ? 2 + q - at : 0);
  return lds32<4 * screen_base(R)>(tab_addr + ((x & m) | (y & (m << q))));
}
// The sum of all runs' entries.
template <int K>
__device__ __forceinline__ uint32_t run_sum(uint32_t tab_addr, uint32_t h, uint32_t l) {
  uint32_t sum = run_entry<K, 0>(tab_addr, h, l) + run_entry<K, 1>(tab_addr, h, l) + run_entry<K, 2>(tab_addr, h, l);
  if constexpr (K == 4) sum += run_entry<K, 3>(tab_addr, h, l);
  return sum;
}

// Mismatches of an oriented window against one record.
template <int NW>
__device__ __forceinline__ uint32_t mismatches(const uint32_t (&h)[NW], const uint32_t (&l)[NW],
                                               const uint32_t (&o)[NW], const Record<NW>& r) {
  uint32_t mm = 0;
#pragma unroll
  for (int i = 0; i < NW; ++i)
    mm += __popc(mux(o[i], r.o[i], mux(h[i], mux(l[i], r.g[i], r.a[i]), mux(l[i], r.c[i], r.t[i]))));
  return mm;
}

__device__ __forceinline__ void append_hit(const HitSink& sink, uint32_t id, uint64_t pos0, uint32_t x, uint32_t mm) {
  const unsigned long long at = atomicAdd(sink.count, 1ull);
  if (at < sink.cap) sink.hits[at] = make_hit(id, pos0 + (x >> 1), x & 1, mm);
}

// The oriented window of item position x.
template <int NW>
__device__ __forceinline__ void load_window(uint32_t (&h)[NW], uint32_t (&l)[NW], uint32_t (&o)[NW],
                                            const GenomeView& g, uint32_t w0, uint32_t x, uint32_t L) {
  const uint32_t w = w0 + (x >> 6), r = (x >> 1) & 31;
  load_plane<NW>(h, g.hi, w, r);
  load_plane<NW>(l, g.lo, w, r);
  load_plane<NW>(o, g.ot, w, r);
  orient_plane<NW>(h, x & 1, true, L);
  orient_plane<NW>(l, x & 1, false, L);
  orient_plane<NW>(o, x & 1, false, L);
}

// Counts one candidate (one lane) against the classes whose top bits are set
// in `test`; only where a list is full.
template <int NW>
__device__ __noinline__ void count_now(const GenomeView& g, uint64_t pos0, uint32_t x, uint32_t test, uint32_t bits,
                                       const uint32_t* cls, const uint32_t* __restrict__ records, uint32_t L,
                                       const HitSink& sink) {
  uint32_t h[NW], l[NW], o[NW];
  load_window<NW>(h, l, o, g, (uint32_t)(pos0 >> 5), x, L);
  for (; test; test &= test - 1) {
    const uint32_t c = (uint32_t)(__ffs(test) - 1) / bits;
    for (uint32_t v = cls[c]; v < cls[c + 1]; ++v) {
      const Record<NW> r(records + (size_t)v * screen_record_words(NW));
      const uint32_t mm = mismatches<NW>(h, l, o, r);
      if (mm <= (r.meta & 15u)) append_hit(sink, r.meta >> 4, pos0, x, mm);
    }
  }
}

// A warp's list.
struct WarpList {
  uint4* items;
  uint32_t cap, used;
  __device__ __forceinline__ explicit WarpList(const ScreenList& list) : used(0) {
    const uint32_t warps = blockDim.x / 32;
    cap = (uint32_t)(list.room / (gridDim.x * warps));
    items = list.items + (size_t)(blockIdx.x * warps + threadIdx.x / 32) * cap;
  }
  // Appends the candidates of the lanes in `m` (all lanes call); false where
  // the lane's did not fit.
  __device__ __forceinline__ bool append(uint32_t m, uint32_t x, uint32_t test, uint32_t h, uint32_t l) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t at = used + __popc(m & ((1u << lane) - 1u));
    const bool mine = m >> lane & 1u, fits = at < cap;
    if (mine && fits) items[at] = make_uint4(x, test, h, l);
    used = min(used + __popc(m), cap);
    return !mine || fits;
  }
  __device__ __forceinline__ void close(const ScreenList& list) const {
    if ((threadIdx.x & 31) == 0) list.counts[blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32] = used;
  }
};

// Copies word `word`'s tables and class bounds into shared memory (whole CTA).
__device__ __forceinline__ void load_tables(const ScreenGeom& G, const ScreenTables& tb, uint32_t word, uint32_t* tab,
                                            uint32_t* cls) {
  __syncthreads();
  const uint4* src = (const uint4*)(tb.tables + (size_t)word * screen_entries(G.K));
  for (uint32_t i = threadIdx.x; i < screen_entries(G.K) / 4; i += blockDim.x) ((uint4*)tab)[i] = __ldg(src + i);
  if (threadIdx.x <= G.fields) cls[threadIdx.x] = tb.first[word * (G.fields + 1) + threadIdx.x];
  __syncthreads();
}

// Whether an item's window holds a non-base byte.
template <int NW>
__device__ __forceinline__ bool odd_window(const GenomeView& g, uint32_t seg_w0, uint32_t x, uint32_t L) {
  uint32_t o[NW], some = 0;
  load_plane<NW>(o, g.ot, seg_w0 + (x >> 6), (x >> 1) & 31);
#pragma unroll
  for (int i = 0; i < NW; ++i)
    some |= o[i] & (L >= 32u * (i + 1) ? kFull : L > 32u * i ? (1u << (L & 31)) - 1u : 0u);
  return some != 0;
}

// The oriented windows of a queue, for a screen that looks them up once per
// word; entries whose window holds a non-base byte get kOddEntry.
constexpr uint32_t kOddEntry = 1u << 31;
template <int NW>
__global__ void __launch_bounds__(256) windows_kernel(const __grid_constant__ GenomeView g, uint32_t* __restrict__ queue,
                                                      const uint32_t* __restrict__ qcount, uint64_t seg_pos0, uint32_t a0,
                                                      uint32_t L, const __grid_constant__ ScreenList list) {
  const uint32_t n = *qcount, seg_w0 = (uint32_t)(seg_pos0 >> 5);
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    const uint32_t e = queue[i], w = seg_w0 + (e >> 6), r = (e >> 1) & 31;
    uint32_t h[NW], l[NW];
    load_plane<NW>(h, g.hi, w, r);
    load_plane<NW>(l, g.lo, w, r);
    orient_plane<NW>(h, e & 1, true, L);
    orient_plane<NW>(l, e & 1, false, L);
    if (odd_window<NW>(g, seg_w0, e, L)) queue[i] = e | kOddEntry;
    list.windows[i] = NW == 1 ? make_uint2(h[0], l[0])
                      : a0 >= 32 ? make_uint2(h[NW - 1] >> (a0 & 31), l[NW - 1] >> (a0 & 31))
                                 : make_uint2(__funnelshift_r(h[0], h[NW - 1], a0), __funnelshift_r(l[0], l[NW - 1], a0));
  }
}

// The screen of a finder pass's queue.  One CTA per SM holds one word's
// tables in shared memory.  The work -- (word, chunk of candidates),
// word-major -- is cut into one contiguous share per CTA, so a CTA loads the
// tables of few words.  Candidates that pass are listed (a candidate counted
// on the spot would hold its warp up: 103 us for the plain search's segment
// of 2^26 starts, 64 + 18 us since) and counted by screen_count_kernel.
// Bound by issue and by the lookups: 32 lanes at random banks take about 3.5
// shared-memory wavefronts.  0.88 SM clocks per candidate and word.
// READY takes the windows from windows_kernel, an iteration ahead: the plain
// form waits for the entries and then for the planes in every word, three
// quarters of its warps' cycles.  Four sets of 256 guides on 0.8 Gbp (16 to 22
// words): 8.20 -> 6.82 ms; issue-bound since (71 % of slots).  With 3 or 4 words
// the extraction costs as much as it saves (272 us for 2^26 starts, 16.8 M
// candidates, either way).
template <int NW, int K, bool DEG, bool READY>
__global__ void __launch_bounds__(kScreenThreads, 1) screen_kernel(
    const __grid_constant__ GenomeView g, const uint32_t* __restrict__ queue, const uint32_t* __restrict__ qcount,
    uint64_t seg_pos0, const __grid_constant__ ScreenGeom G, const __grid_constant__ ScreenTables tb, uint32_t L,
    const __grid_constant__ ScreenList list, const __grid_constant__ HitSink sink) {
  extern __shared__ __align__(16) uint32_t tab[];
  __shared__ uint32_t cls[9];
  constexpr uint32_t kWarpSpan = 32 * kPerLane;
  const unsigned lane = threadIdx.x & 31;
  const uint32_t n = *qcount;
  const uint32_t seg_w0 = (uint32_t)(seg_pos0 >> 5);
  const uint64_t spans = (n + kWarpSpan - 1) / kWarpSpan;  // warp iterations per word
  const uint64_t total = spans * G.words;
  uint64_t u = total * blockIdx.x / gridDim.x;
  const uint64_t u_end = total * (blockIdx.x + 1) / gridDim.x;
  const uint32_t word0 = u < u_end ? (uint32_t)(u / spans) : 0u;
  const uint32_t tab_addr = (uint32_t)__cvta_generic_to_shared(tab);
  WarpList out(list);
  while (u < u_end) {
    const uint32_t word = (uint32_t)(u / spans);
    const uint64_t word_u = (uint64_t)word * spans, stop = min(u_end, word_u + spans);
    load_tables(G, tb, word, tab, cls);
    // The coming iteration's entries and windows (past the last: any).
    uint32_t next[kPerLane];
    uint2 next_win[kPerLane];
    auto fetch = [&](uint64_t s) {
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const uint32_t i = min((uint32_t)(s - word_u) * kWarpSpan + lane + 32 * j, n - 1);
        next[j] = __ldg(queue + i);
        next_win[j] = __ldg(list.windows + i);
      }
    };
    if (READY) fetch(u + (threadIdx.x >> 5));
    for (uint64_t s = u + (threadIdx.x >> 5); s < stop; s += kScreenThreads / 32) {
      const uint32_t i0 = (uint32_t)(s - word_u) * kWarpSpan + lane;
      uint32_t e[kPerLane], test[kPerLane], h0[kPerLane], l0[kPerLane], any = 0;
      if constexpr (READY) {
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
          e[j] = next[j];
          h0[j] = next_win[j].x;
          l0[j] = next_win[j].y;
        }
        fetch(s + kScreenThreads / 32);
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
          const uint32_t a0 = NW == 1 ? G.a0 : 0;
          test[j] = ~run_sum<K>(tab_addr, h0[j] >> a0, l0[j] >> a0) & G.top;
          if (DEG && e[j] >= kOddEntry) test[j] = G.top;
          if (i0 + 32 * j >= n) test[j] = 0;
          any |= test[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
          const uint32_t i = i0 + 32 * j;
          e[j] = i < n ? __ldg(queue + i) : 0xFFFFFFFFu;
        }
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
          const bool have = e[j] != 0xFFFFFFFFu;
          const uint32_t w = seg_w0 + (have ? e[j] >> 6 : 0u), r = (e[j] >> 1) & 31;
          uint32_t h[NW], l[NW];
          load_plane<NW>(h, g.hi, w, r);
          load_plane<NW>(l, g.lo, w, r);
          orient_plane<NW>(h, e[j] & 1, true, L);
          orient_plane<NW>(l, e[j] & 1, false, L);
          // The window from the screen's first position on (26 positions at most).
          const uint32_t hr = NW == 1 || G.a0 >= 32 ? h[NW - 1] >> (G.a0 & 31) : __funnelshift_r(h[0], h[NW - 1], G.a0);
          const uint32_t lr = NW == 1 || G.a0 >= 32 ? l[NW - 1] >> (G.a0 & 31) : __funnelshift_r(l[0], l[NW - 1], G.a0);
          test[j] = ~run_sum<K>(tab_addr, hr, lr) & G.top;
          if (DEG && have && odd_window<NW>(g, seg_w0, e[j], L)) test[j] = G.top;
          if (!have) test[j] = 0;
          any |= test[j];
          h0[j] = h[0];
          l0[j] = l[0];
        }
      }
      if (!__any_sync(kFull, any)) continue;
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const uint32_t m = __ballot_sync(kFull, test[j] != 0);
        if (!m) continue;
        const uint32_t flag =
            test[j] && (READY ? e[j] >= kOddEntry : odd_window<NW>(g, seg_w0, e[j], L)) ? kOddWindow : 0u;
        const uint32_t x = READY ? e[j] & ~kOddEntry : e[j];
        if (!out.append(m, x, test[j] | flag | (word - word0), h0[j], l0[j]))
          count_now<NW>(g, seg_pos0, x, test[j], G.bits, cls, tb.records, L, sink);
      }
    }
    u = stop;
  }
  out.close(list);
}

// The scanning screen.  A warp takes 64 plane words (2,048 starts) at a time,
// two per lane, tests the PAM bit-parallel, stages the candidates of one
// strand after the other in shared memory and looks them up 32 at a time.
// The words are staged in the strand's orientation -- the '-' strand's
// reversed and complemented, last word first -- so that a candidate is a
// place q in the staged planes from which its window's screened positions
// follow in ascending order: q's two words of both planes, one funnel shift
// per plane, the lookups.
// Bound by issue (2.6 instructions per clock): 770 instructions per 64 words
// at 166 candidates (NGG), 1,580 at 400 (NRG), of which the PAM test takes 80,
// staging 220 and 420, a lookup of 32 candidates 38.  0.4 Gbp take 189 us
// (NGG) and 359 us (NRG), against 155 + 137 and 181 + 270 us for finder_kernel
// and screen_kernel.  24 warps of 80 registers measured best (20: 201 / 382
// us, 28: 200 / 364 us).
constexpr int kScanThreads = 768;
constexpr uint32_t kScanStage = 320;  // staged candidates per warp (16 bits each)
constexpr uint32_t kScanPlaneBytes = 66 * 8;  // 64 words, the one their windows end in, one never used
constexpr uint32_t kScanWarpBytes = kScanPlaneBytes + kScanStage * 2;

// The PAM's positions that can mismatch, per strand and sorted by class.
struct ScanParams {
  uint32_t L, n[2];
  uint8_t pos[2][kMaxL], cls[2][kMaxL];
};

// The mismatch words of class `cls` for the lane's three words.
__device__ __forceinline__ void class_words(uint32_t cls, const uint32_t (&h)[3], const uint32_t (&l)[3],
                                            const uint32_t (&o)[3], uint32_t (&c)[3]) {
  switch (cls) {
#define COF_CLASS_CASE(V)                                                                            \
  case V:                                                                                            \
    _Pragma("unroll") for (int i = 0; i < 3; ++i) c[i] = lop3<class_lut(V)>(h[i], l[i], o[i]);       \
    break;
    COF_CLASS_CASE(0x1B) COF_CLASS_CASE(0x1D) COF_CLASS_CASE(0x17) COF_CLASS_CASE(0x1E) COF_CLASS_CASE(0x03)
    COF_CLASS_CASE(0x0C) COF_CLASS_CASE(0x06) COF_CLASS_CASE(0x09) COF_CLASS_CASE(0x0A) COF_CLASS_CASE(0x05)
    COF_CLASS_CASE(0x08) COF_CLASS_CASE(0x04) COF_CLASS_CASE(0x01) COF_CLASS_CASE(0x02)
#undef COF_CLASS_CASE
    default:  // class_bits_of has no other values
      break;
  }
}

template <int K, bool DEG>
__global__ void __launch_bounds__(kScanThreads, 1) scan_screen_kernel(
    const __grid_constant__ GenomeView g, uint64_t w_begin, uint32_t words, uint32_t skip, uint64_t pos_end,
    const __grid_constant__ ScanParams P, const __grid_constant__ ScreenGeom G,
    const __grid_constant__ ScreenTables tb, const __grid_constant__ ScreenList list,
    unsigned long long* __restrict__ qcount, const __grid_constant__ HitSink sink) {
  extern __shared__ __align__(16) uint32_t tab[];
  __shared__ uint32_t cls[9];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint2* planes = (uint2*)((char*)(tab + screen_entries(K)) + warp * kScanWarpBytes);
  const uint32_t tab_addr = (uint32_t)__cvta_generic_to_shared(tab);
  const uint32_t planes_addr = (uint32_t)__cvta_generic_to_shared(planes), staged_addr = planes_addr + kScanPlaneBytes;
  const uint32_t units = (words + 63) / 64;
  const uint64_t total = (uint64_t)units * G.words;
  uint64_t u = total * blockIdx.x / gridDim.x;
  const uint64_t u_end = total * (blockIdx.x + 1) / gridDim.x;
  const uint32_t word0 = u < u_end ? (uint32_t)(u / units) : 0u;
  WarpList out(list);
  uint32_t found = 0;
  const uint32_t *hi = g.hi + w_begin, *lo = g.lo + w_begin, *ot = g.ot + w_begin;
  // Starts of this launch that lie inside the genome.
  const uint32_t starts = pos_end > (w_begin << 5) ? (uint32_t)min(pos_end - (w_begin << 5), (uint64_t)words << 5) : 0u;
  while (u < u_end) {
    const uint32_t word = (uint32_t)(u / units);
    const uint64_t word_u = (uint64_t)word * units;
    const uint32_t stop = (uint32_t)(min(u_end, word_u + units) - word_u);
    load_tables(G, tb, word, tab, cls);
    // The next unit's plane words are loaded while the current is looked up.
    uint32_t nh[3], nl[3], no[3];
    auto fetch = [&](uint32_t s) {
      // Past the end lanes load the last words again (their starts are cut
      // off below).  The last start's window may end in word `words`, and the
      // planes hold at least three more.
      const uint32_t w = min(s * 64 + 2 * lane, (words + 1) & ~1u);
      const uint2 a = __ldg((const uint2*)(hi + w)), b = __ldg((const uint2*)(lo + w)), c = __ldg((const uint2*)(ot + w));
      nh[0] = a.x, nh[1] = a.y, nh[2] = __ldg(hi + w + 2);
      nl[0] = b.x, nl[1] = b.y, nl[2] = __ldg(lo + w + 2);
      no[0] = c.x, no[1] = c.y, no[2] = __ldg(ot + w + 2);
    };
    uint32_t s = (uint32_t)(u - word_u) + warp;
    fetch(s);
    for (; s < stop; s += kScanThreads / 32) {
      const uint32_t h[3] = {nh[0], nh[1], nh[2]}, l[3] = {nl[0], nl[1], nl[2]}, o[3] = {no[0], no[1], no[2]};
      fetch(s + kScanThreads / 32);
      uint32_t mask[2][2];  // [strand][word]: candidates
#pragma unroll
      for (int strand = 0; strand < 2; ++strand) {
        uint32_t bad0 = 0, bad1 = 0, c[3] = {0, 0, 0}, last = 0;
        for (uint32_t j = 0; j < P.n[strand]; ++j) {
          if (P.cls[strand][j] != last) {
            last = P.cls[strand][j];
            class_words(last, h, l, o, c);
          }
          const uint32_t q = P.pos[strand][j];
          bad0 |= __funnelshift_r(c[0], c[1], q);
          bad1 |= __funnelshift_r(c[1], c[2], q);
        }
        mask[strand][0] = ~bad0;
        mask[strand][1] = ~bad1;
      }
      // As finder_kernel: starts inside the genome, windows without a separator.
      const uint32_t p0 = (s * 64 + 2 * lane) << 5;
      if (s == 0 && lane == 0 && skip) mask[0][0] = mask[1][0] = 0;
      if (s * 64 + 64 > starts >> 5) {  // warp-uniform: the last units only
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t p = p0 + 32 * i;
          const bool past = (s * 64 + 2 * lane + i) >= (starts + 31) / 32;
          const uint32_t keep = past ? 0u : starts - p >= 32 ? kFull : kFull >> (32 - (starts - p));
          mask[0][i] &= keep;
          mask[1][i] &= keep;
        }
      }
      if (o[0] | o[1] | o[2]) {
        const uint32_t s0 = o[0] & l[0] & ~h[0], s1 = o[1] & l[1] & ~h[1], s2 = o[2] & l[2] & ~h[2];
        if (s0 | s1 | s2) {
          uint32_t near0 = 0, near1 = 0;
          for (unsigned q = 0; q < P.L; ++q) {
            near0 |= __funnelshift_r(s0, s1, q);
            near1 |= __funnelshift_r(s1, s2, q);
          }
          mask[0][0] &= ~near0, mask[1][0] &= ~near0;
          mask[0][1] &= ~near1, mask[1][1] &= ~near1;
        }
      }
      const bool any_odd = __any_sync(kFull, o[0] | o[1] | o[2]);
      // Places of the lane's candidates, both strands in one scan.
      const uint32_t own = (__popc(mask[0][0]) + __popc(mask[0][1])) |
                           (__popc(mask[1][0]) + __popc(mask[1][1])) << 16;
      uint32_t incl = own;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, d);
        if (lane >= (unsigned)d) incl += t;
      }
      const uint32_t all = __shfl_sync(kFull, incl, 31);
      if (!all) continue;
      if (word == 0) found += (all & 0xFFFFu) + (all >> 16);
#pragma unroll
      for (uint32_t strand = 0; strand < 2; ++strand) {
        const uint32_t count = strand ? all >> 16 : all & 0xFFFFu;
        if (!count) continue;
        // Start p of the unit is place a0 + p of the '+' strand's planes and
        // place 65 * 32 - L + a0 - p of the '-' strand's.
        const uint32_t origin = strand ? 65 * 32 - P.L + G.a0 : G.a0;
        if (strand) {
          planes[64 - 2 * lane] = make_uint2(~__brev(h[0]), __brev(l[0]));
          planes[63 - 2 * lane] = make_uint2(~__brev(h[1]), __brev(l[1]));
          if (lane == 31) planes[0] = make_uint2(~__brev(h[2]), __brev(l[2]));
        } else {
          *(uint4*)(planes + 2 * lane) = make_uint4(h[0], l[0], h[1], l[1]);
          if (lane == 31) planes[64] = make_uint2(h[2], l[2]);
        }
        const uint32_t end = strand ? incl >> 16 : incl & 0xFFFFu, begin = end - (strand ? own >> 16 : own & 0xFFFFu);
        // Dense units go through the stage in rounds of four lanes' candidates.
        const uint32_t rounds = count <= kScanStage ? 1 : 8;
        for (uint32_t round = 0; round < rounds; ++round) {
          uint32_t to = staged_addr + 2 * begin, here = count;
          bool mine = true;
          if (rounds > 1) {
            const uint32_t before = __shfl_sync(kFull, begin, 4 * round);
            here = __shfl_sync(kFull, end, 4 * round + 3) - before;
            mine = (lane >> 2) == round;
            to -= 2 * before;
          }
          if (mine) {
            // The highest and the lowest candidate left per trip.
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint32_t q0 = strand ? origin - 64 * lane - 32 * i : origin + 64 * lane + 32 * i;
              for (uint32_t left = mask[strand][i]; left;) {
                const uint32_t hb = 31 - __clz(left), lb = __ffs(left) - 1;
                sts16(to, strand ? q0 - hb : q0 + hb);
                if (lb != hb) sts16(to + 2, strand ? q0 - lb : q0 + lb);
                to += lb != hb ? 4 : 2;
                left &= ~((1u << hb) | (1u << lb));
              }
            }
          }
          __syncwarp();
          // The plane words from place q on.
          auto words_at = [&](uint32_t q, uint32_t& hw, uint32_t& lw) {
            const uint32_t at = planes_addr + (q >> 2 & 0x3F8u);
            const uint2 x = lds64<0>(at), y = lds64<8>(at);
            hw = __funnelshift_r(x.x, y.x, q);
            lw = __funnelshift_r(x.y, y.y, q);
          };
          // Whether the window at place q holds a non-base byte (units with some).
          auto odd = [&](uint32_t q) {
            const uint32_t p = (strand ? origin - q : q - origin) & 2047u, w = min(s * 64 + (p >> 5), words);
            return (__funnelshift_r(__ldg(ot + w), __ldg(ot + w + 1), p) & (kFull >> (32 - P.L))) != 0;
          };
          for (uint32_t i0 = 0; i0 < here; i0 += 32) {
            const uint32_t i = i0 + lane;
            const uint32_t q = i < here ? lds16(staged_addr + 2 * i) : 32u;
            uint32_t hw, lw;
            words_at(q, hw, lw);
            uint32_t test = ~run_sum<K>(tab_addr, hw, lw) & G.top;
            if (DEG && any_odd && odd(q)) test = G.top;
            const uint32_t m = __ballot_sync(kFull, test != 0 && i < here);
            if (m) {
              const uint32_t x = (s * 2048 + (strand ? origin - q : q - origin)) << 1 | strand;
              words_at(q - G.a0, hw, lw);
              const uint32_t flag = any_odd && odd(q) ? kOddWindow : 0u;
              if (!out.append(m, x, test | flag | (word - word0), hw, lw))
                count_now<1>(g, w_begin << 5, x, test, G.bits, cls, tb.records, P.L, sink);
            }
          }
          __syncwarp();
        }
      }
    }
    u = word_u + stop;
  }
  if (lane == 0 && found) atomicAdd(qcount, (unsigned long long)found);
  out.close(list);
}

// Counts the listed candidates exactly.  A warp takes 128 items of one
// screening CTA's lists at a time; class by class, its lanes hold a variant
// each (two where the class has more than 32) and the class's items pass by,
// gathered in shared memory and read by all lanes at once, so no warp waits
// for another.  Bound by issue: about 22 instructions per item of a 28-variant
// class.  101 us for 3.7 M items (sorting them by class in shared memory
// across a CTA took 167 us, 256 items at a time 112).
constexpr int kCountThreads = 128;
constexpr uint32_t kCountBlock = 128;  // items at a time
constexpr uint32_t kCountShare = 64;   // warps per screening CTA

// The gathered windows of one class against one variant (or two) per lane;
// `n` of them, `pos` their positions.
template <int NW, int V>
__device__ __forceinline__ void count_gathered(const uint2* got, const uint32_t* pos, uint32_t n,
                                               const uint32_t* __restrict__ records, uint32_t v0, uint32_t v1,
                                               uint64_t pos0, const HitSink& sink) {
  const unsigned lane = threadIdx.x & 31;
  uint32_t t[V][NW], c[V][NW], a[V][NW], g[V][NW], id[V];
  int limit[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const uint32_t v = v0 + 32 * i + lane;
    const Record<NW> r(records + (size_t)min(v, v1 - 1) * screen_record_words(NW));
#pragma unroll
    for (int k = 0; k < NW; ++k) t[i][k] = r.t[k], c[i][k] = r.c[k], a[i][k] = r.a[k], g[i][k] = r.g[k];
    id[i] = r.meta >> 4;
    limit[i] = v < v1 ? (int)(r.meta & 15u) : -1;
  }
  constexpr int kStep = V * NW == 1 ? 4 : 2;
  for (uint32_t at = 0; at < n; at += kStep) {  // items past n are stale: dropped where a hit is reported
    int mm[kStep][V] = {};
    bool any = false;
#pragma unroll
    for (int j = 0; j < kStep; ++j) {
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint2 w = got[(at + j) * NW + k];
#pragma unroll
        for (int i = 0; i < V; ++i)
          mm[j][i] += __popc(mux(w.x, mux(w.y, g[i][k], a[i][k]), mux(w.y, c[i][k], t[i][k])));
      }
#pragma unroll
      for (int i = 0; i < V; ++i) any |= mm[j][i] <= limit[i];
    }
    if (any) {
#pragma unroll
      for (int j = 0; j < kStep; ++j)
#pragma unroll
        for (int i = 0; i < V; ++i)
          if (at + j < n && mm[j][i] <= limit[i]) append_hit(sink, id[i], pos0, pos[at + j], mm[j][i]);
    }
  }
}

template <int NW>
__global__ void __launch_bounds__(kCountThreads) screen_count_kernel(
    const __grid_constant__ GenomeView g, uint64_t pos0, const __grid_constant__ ScreenGeom G,
    const __grid_constant__ ScreenTables tb, uint32_t L, const __grid_constant__ ScreenList list, uint32_t ctas,
    uint32_t warps, uint64_t spans, const uint32_t* __restrict__ qcount, uint32_t warp_span,
    const __grid_constant__ HitSink sink) {
  constexpr uint32_t kWarps = kCountThreads / 32;
  static_assert(kCountShare % kWarps == 0, "a CTA serves one screening CTA");
  __shared__ __align__(16) uint2 got_all[kWarps][(kCountBlock + 4) * NW];
  __shared__ uint32_t pos_all[kWarps][kCountBlock + 4];
  __shared__ uint32_t begin[33];  // first item of each of the screening CTA's lists
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint2* got = got_all[warp];
  uint32_t* at_pos = pos_all[warp];
  const uint32_t cta = blockIdx.x / (kCountShare / kWarps), cap = (uint32_t)(list.room / (ctas * warps));
  if (warp == 0) {
    const uint32_t own = lane < warps ? list.counts[cta * warps + lane] : 0u;
    uint32_t incl = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, incl, d);
      if (lane >= (unsigned)d) incl += t;
    }
    begin[lane] = incl - own;
    if (lane == 31) begin[32] = incl;
  }
  __syncthreads();
  const uint32_t n = begin[32];
  const uint32_t first_block = (blockIdx.x % (kCountShare / kWarps) * kWarps + warp) * kCountBlock;
  if (first_block >= n) return;
  // The first word of the screening CTA's share (as the screening kernels cut
  // them), and the classes its items may belong to.
  if (qcount) spans = (*qcount + warp_span - 1) / warp_span;
  const uint64_t total = spans * G.words;
  const uint32_t word0 = (uint32_t)(total * cta / ctas / spans), w0 = (uint32_t)(pos0 >> 5);
  const uint32_t classes = ((uint32_t)((total * (cta + 1) / ctas - 1) / spans) - word0 + 1) * G.fields;
  const uint4* src = list.items + (size_t)cta * warps * cap;
  for (uint32_t i0 = first_block; i0 < n; i0 += kCountShare * kCountBlock) {
    constexpr uint32_t kEach = kCountBlock / 32;
    uint32_t x[kEach], test[kEach], wh[kEach], wl[kEach];
#pragma unroll
    for (uint32_t j = 0; j < kEach; ++j) {
      const uint32_t i = i0 + 32 * j + lane;
      uint32_t r = 0;  // the last list starting at or before i (empty lists share starts)
#pragma unroll
      for (uint32_t step = 16; step; step >>= 1)
        if (begin[r + step] <= i) r += step;
      const uint4 it = i < n ? src[(size_t)r * cap + (i - begin[r])] : make_uint4(0, 0, 0, 0);
      x[j] = it.x, test[j] = it.y, wh[j] = it.z, wl[j] = it.w;
    }
    for (uint32_t c = 0; c < classes; ++c) {
      const uint32_t bit = 1u << (c % G.fields * G.bits + G.bits - 1);
      uint32_t m[kEach], any = 0;
#pragma unroll
      for (uint32_t j = 0; j < kEach; ++j) {
        m[j] = __ballot_sync(kFull, (test[j] & bit) && (test[j] & 7u) == c / G.fields);
        any |= m[j];
      }
      if (!any) continue;
      const uint32_t f = (word0 + c / G.fields) * (G.fields + 1) + c % G.fields;
      const uint32_t first = __ldg(tb.first + f), end = __ldg(tb.first + f + 1);
      // Windows with a non-base byte are left to the loop below.
      uint32_t at = 0;
      any = 0;
      __syncwarp();
#pragma unroll
      for (uint32_t j = 0; j < kEach; ++j) {
        const uint32_t plain = __ballot_sync(kFull, (m[j] >> lane & 1u) && !(test[j] & kOddWindow));
        if (plain >> lane & 1u) {
          const uint32_t to = at + __popc(plain & ((1u << lane) - 1u));
          uint32_t h[NW] = {wh[j]}, l[NW] = {wl[j]};
          if (NW > 1) {
            const uint32_t w = w0 + (x[j] >> 6), r = (x[j] >> 1) & 31;
            load_plane<NW>(h, g.hi, w, r);
            load_plane<NW>(l, g.lo, w, r);
            orient_plane<NW>(h, x[j] & 1, true, L);
            orient_plane<NW>(l, x[j] & 1, false, L);
          }
#pragma unroll
          for (int k = 0; k < NW; ++k) got[to * NW + k] = make_uint2(h[k], l[k]);
          at_pos[to] = x[j];
        }
        at += __popc(plain);
        m[j] &= ~plain;
        any |= m[j];
      }
      __syncwarp();
      for (uint32_t v0 = first; v0 < end; v0 += 64) {
        if (end - v0 > 32) count_gathered<NW, 2>(got, at_pos, at, tb.records, v0, end, pos0, sink);
        else count_gathered<NW, 1>(got, at_pos, at, tb.records, v0, end, pos0, sink);
      }
      if (!any) continue;
      for (uint32_t v0 = first; v0 < end; v0 += 32) {
#pragma unroll
        for (uint32_t j = 0; j < kEach; ++j)
          for (uint32_t left = m[j]; left; left &= left - 1) {
            const uint32_t at = __shfl_sync(kFull, x[j], __ffs(left) - 1);
            uint32_t h[NW], l[NW], o[NW];
            load_window<NW>(h, l, o, g, w0, at, L);
            if (v0 + lane < end) {
              const Record<NW> r(tb.records + (size_t)(v0 + lane) * screen_record_words(NW));
              const uint32_t mm = mismatches<NW>(h, l, o, r);
              if (mm <= (r.meta & 15u)) append_hit(sink, r.meta >> 4, pos0, at, mm);
            }
          }
      }
    }
  }
}

// The count of a screening launch of `ctas` x `warps` warps over `spans` warp
// shares per word (qcount: read there, in shares of warp_span candidates).
void launch_count(const GenomeView& g, uint64_t pos0, const ScreenGeom& geom, int nw, const ScreenTables& tb, uint32_t L,
                  const ScreenList& list, uint32_t ctas, uint32_t warps, uint64_t spans, const uint32_t* qcount,
                  uint32_t warp_span, const HitSink& sink, cudaStream_t stream) {
  auto kernel = nw == 1 ? screen_count_kernel<1> : screen_count_kernel<2>;
  kernel<<<ctas * (kCountShare * 32 / kCountThreads), kCountThreads, 0, stream>>>(g, pos0, geom, tb, L, list, ctas, warps,
                                                                                 spans, qcount, warp_span, sink);
}

template <int NW, int K, bool DEG>
void run_screen(const GenomeView& g, uint32_t* queue, const uint32_t* qcount, uint64_t seg_pos0,
                const ScreenGeom& geom, const ScreenTables& tb, uint32_t L, const ScreenList& list, const HitSink& sink,
                int sm_count, cudaStream_t stream) {
  const size_t smem = (size_t)screen_entries(K) * 4;
  const bool ready = geom.words >= kWindowWords && list.windows;
  auto kernel = ready ? screen_kernel<NW, K, DEG, true> : screen_kernel<NW, K, DEG, false>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (ready) windows_kernel<NW><<<8 * sm_count, 256, 0, stream>>>(g, queue, qcount, seg_pos0, geom.a0, L, list);
  kernel<<<sm_count, kScreenThreads, smem, stream>>>(g, queue, qcount, seg_pos0, geom, tb, L, list, sink);
  launch_count(g, seg_pos0, geom, NW, tb, L, list, sm_count, kScreenThreads / 32, 0, qcount, 32 * kPerLane, sink,
               stream);
}

template <int K, bool DEG>
void run_scan_screen(const GenomeView& g, uint64_t w_begin, uint64_t w_end, const FinderPattern& pat,
                     const ScreenGeom& geom, const ScreenTables& tb, const ScreenList& list,
                     unsigned long long* qcount, const HitSink& sink, int sm_count, cudaStream_t stream) {
  const size_t smem = (size_t)screen_entries(K) * 4 + kScanThreads / 32 * kScanWarpBytes;
  const uint64_t pos_end = g.n >= pat.L ? g.n - pat.L + 1 : 0;
  cudaFuncSetAttribute(scan_screen_kernel<K, DEG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  ScanParams P{};
  P.L = pat.L;
  for (int strand = 0; strand < 2; ++strand)
    for (uint32_t c = 1; c < 32; ++c)
      for (uint32_t j = 0; j < (strand ? pat.nr : pat.nf); ++j)
        if (((strand ? pat.rm[j] : pat.fm[j]) & 31u) == c) {
          P.pos[strand][P.n[strand]] = strand ? pat.rk[j] : pat.fk[j];
          P.cls[strand][P.n[strand]++] = (uint8_t)c;
        }
  // The kernel loads pairs of words: an odd range begins a word early, with
  // that word's starts left out.
  const uint32_t skip = (uint32_t)(w_begin & 1);
  w_begin -= skip;
  scan_screen_kernel<K, DEG><<<sm_count, kScanThreads, smem, stream>>>(
      g, w_begin, (uint32_t)(w_end - w_begin), skip, pos_end, P, geom, tb, list, qcount, sink);
  launch_count(g, w_begin << 5, geom, 1, tb, pat.L, list, sm_count, kScanThreads / 32, (w_end - w_begin + 63) / 64,
               nullptr, 1, sink, stream);
}

}  // namespace

uint32_t screen_lists(int sm_count) { return (uint32_t)sm_count * (kScreenThreads / 32); }

uint64_t screen_list_items(uint64_t positions) {
  return std::min<uint64_t>(1ull << 25, std::max<uint64_t>(1ull << 18, positions / 2));
}

void launch_screen_tables(const ScreenGeom& geom, int nw, const uint32_t* records, const uint32_t* first,
                          uint32_t* tables, cudaStream_t stream) {
  const dim3 grid(screen_entries(geom.K) / 32, geom.words);
  if (nw == 1) screen_tables_kernel<1><<<grid, 256, 0, stream>>>(geom, records, first, tables);
  else screen_tables_kernel<2><<<grid, 256, 0, stream>>>(geom, records, first, tables);
}

void launch_screen(const GenomeView& g, uint32_t* queue, const uint32_t* qcount, uint64_t seg_pos0,
                   const ScreenGeom& geom, int nw, const ScreenTables& tb, uint32_t L, const ScreenList& list,
                   const HitSink& sink, int sm_count, cudaStream_t stream) {
  auto run = nw == 1 ? (geom.K == 3 ? (geom.degenerate ? run_screen<1, 3, true> : run_screen<1, 3, false>)
                                    : (geom.degenerate ? run_screen<1, 4, true> : run_screen<1, 4, false>))
                     : (geom.K == 3 ? (geom.degenerate ? run_screen<2, 3, true> : run_screen<2, 3, false>)
                                    : (geom.degenerate ? run_screen<2, 4, true> : run_screen<2, 4, false>));
  run(g, queue, qcount, seg_pos0, geom, tb, L, list, sink, sm_count, stream);
}

void launch_scan_screen(const GenomeView& g, uint64_t w_begin, uint64_t w_end, const FinderPattern& pat,
                        const ScreenGeom& geom, const ScreenTables& tb, const ScreenList& list,
                        unsigned long long* qcount, const HitSink& sink, int sm_count, cudaStream_t stream) {
  auto run = geom.K == 3 ? (geom.degenerate ? run_scan_screen<3, true> : run_scan_screen<3, false>)
                         : (geom.degenerate ? run_scan_screen<4, true> : run_scan_screen<4, false>);
  run(g, w_begin, w_end, pat, geom, tb, list, qcount, sink, sm_count, stream);
}

}  // namespace cof
