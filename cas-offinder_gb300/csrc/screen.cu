// Table screen: table construction and the screening kernel (see screen.cuh).
#include <algorithm>

#include "screen.cuh"

namespace cof {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kScreenThreads = 1024;  // one CTA per SM shares one set of tables
constexpr int kPerLane = 2;           // candidates per lane and iteration

__device__ __forceinline__ uint32_t mux(uint32_t s, uint32_t a, uint32_t b) { return (s & a) | (~s & b); }

__device__ __forceinline__ uint32_t rotl(uint32_t x, uint32_t r) { return __funnelshift_l(x, x, r); }

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

// One table entry per thread: the least mismatch count on the run over each
// class's variants, capped, in the class's field.  Every thread of a warp
// reads the same record at a time (a broadcast).
template <int NW>
__global__ void __launch_bounds__(256) screen_tables_kernel(const __grid_constant__ ScreenGeom G,
                                                            const uint32_t* __restrict__ records,
                                                            const uint32_t* __restrict__ first,
                                                            uint32_t* __restrict__ tables) {
  constexpr uint32_t kRec = screen_record_words(NW);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, word = blockIdx.y;
  if (i >= G.entries) return;
  uint32_t k = 0;
  while (k + 1 < G.K && i >= G.base[k + 1]) ++k;
  const uint32_t x = i - G.base[k], q = G.q[k], m = (1u << q) - 1u, a = G.a[k];
  const uint32_t h = x & m, l = x >> q;  // the run's plane bits
  const uint32_t T = 1u << (G.bits - 1);
  const uint32_t* f = first + word * (G.fields + 1);
  uint32_t out = 0;
  for (uint32_t c = 0; c < G.fields; ++c) {
    int least = (int)G.cap[k];
    for (uint32_t v = f[c]; v < f[c + 1]; ++v) {
      const Record<NW> r(records + (size_t)v * kRec);
      auto run = [&](const uint32_t (&w)[NW]) {
        return NW == 1 ? w[0] >> a : __funnelshift_rc(w[0], w[NW - 1], a < 32 ? a : 32) >> (a < 32 ? 0 : a - 32);
      };
      int d = __popc(mux(h, mux(l, run(r.g), run(r.a)), mux(l, run(r.c), run(r.t))) & m);
      if (k == 0) d += (int)T - 1 - (int)(r.meta & 15u);
      least = min(least, d);
    }
    out |= (uint32_t)least << (c * G.bits);
  }
  tables[(size_t)word * G.entries + i] = out;
}

// A candidate's oriented window planes.
template <int NW>
struct Window {
  uint32_t h[NW], l[NW], o[NW];
};

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

// Byte offset within a run's table of the window's plane bits there: hi bits
// below lo bits, q each.
template <int NW>
__device__ __forceinline__ uint32_t run_offset(const uint32_t (&h)[NW], const uint32_t (&l)[NW], uint32_t a,
                                               uint32_t q) {
  const uint32_t m = ((1u << q) - 1u) << 2;
  if (NW == 1) {
    return (rotl(h[0], (34 - a) & 31) & m) | ((rotl(l[0], (34 - a + q) & 31)) & (m << q));
  } else {
    const uint64_t H = ((uint64_t)h[NW - 1] << 32) | h[0], Lo = ((uint64_t)l[NW - 1] << 32) | l[0];
    return (((uint32_t)(H >> a) << 2) & m) | (((uint32_t)(Lo >> a) << (2 + q)) & (m << q));
  }
}

// Counts the window of queue entry `e` (lane-uniform) against the records
// [v0, v1), one variant per lane, and appends the hits.
template <int NW>
__device__ __forceinline__ void count_class(const Window<NW>& w, uint32_t v0, uint32_t v1, unsigned lane, uint32_t e,
                                            uint64_t seg_pos0, const uint32_t* __restrict__ records,
                                            uint64_t* __restrict__ hits, unsigned long long* __restrict__ hit_count,
                                            uint64_t hit_cap) {
  for (uint32_t v = v0 + lane; v < v1; v += 32) {
    const Record<NW> r(records + (size_t)v * screen_record_words(NW));
    uint32_t mm = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i)
      mm += __popc(mux(w.o[i], r.o[i], mux(w.h[i], mux(w.l[i], r.g[i], r.a[i]), mux(w.l[i], r.c[i], r.t[i]))));
    if (mm <= (r.meta & 15u)) {
      const unsigned long long at = atomicAdd(hit_count, 1ull);
      if (at < hit_cap) hits[at] = make_hit(r.meta >> 4, seg_pos0 + (e >> 1), e & 1, mm);
    }
  }
}

// One CTA per SM holds one word's tables in shared memory.  The work --
// (word, chunk of candidates), word-major -- is cut into one contiguous
// share per CTA, so a CTA loads the tables of few words.
// Bound by the shared-memory lookups (32 lanes at random banks: about 3.5
// wavefronts each) and by the latency of counting the candidates that pass.
// A segment of 2^26 starts, against the bit-sliced comparer: 12.8 M
// candidates x 217 variants (NRG, bulges 2/1, limit 5) 103 us (was 164); 5.3
// M x 1 23 us (was 65); 5.4 M x 1,000 179 us (was 1,000).
template <int NW, int K, bool DEG>
__global__ void __launch_bounds__(kScreenThreads, 1) screen_kernel(
    const uint32_t* __restrict__ hi, const uint32_t* __restrict__ lo, const uint32_t* __restrict__ ot,
    const uint32_t* __restrict__ queue, const uint32_t* __restrict__ qcount, uint64_t seg_pos0,
    const __grid_constant__ ScreenGeom G, const uint32_t* __restrict__ records, const uint32_t* __restrict__ first,
    const uint32_t* __restrict__ tables, uint32_t L, uint64_t* __restrict__ hits,
    unsigned long long* __restrict__ hit_count, uint64_t hit_cap) {
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
  while (u < u_end) {
    const uint32_t word = (uint32_t)(u / spans);
    const uint64_t word_u = (uint64_t)word * spans, stop = min(u_end, word_u + spans);
    __syncthreads();
    {
      const uint4* src = (const uint4*)(tables + (size_t)word * G.entries);
      for (uint32_t i = threadIdx.x; i < G.entries / 4; i += kScreenThreads) ((uint4*)tab)[i] = __ldg(src + i);
      if (threadIdx.x <= G.fields) cls[threadIdx.x] = first[word * (G.fields + 1) + threadIdx.x];
    }
    __syncthreads();
    for (uint64_t s = u + (threadIdx.x >> 5); s < stop; s += kScreenThreads / 32) {
      const uint32_t i0 = (uint32_t)(s - word_u) * kWarpSpan + lane;
      uint32_t e[kPerLane], test[kPerLane], any = 0;
      uint32_t h[kPerLane][NW], l[kPerLane][NW];
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const uint32_t i = i0 + 32 * j;
        e[j] = i < n ? __ldg(queue + i) : 0xFFFFFFFFu;
      }
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const bool have = e[j] != 0xFFFFFFFFu;
        const uint32_t w = seg_w0 + (have ? e[j] >> 6 : 0u), r = (e[j] >> 1) & 31;
        load_plane<NW>(h[j], hi, w, r);
        load_plane<NW>(l[j], lo, w, r);
        orient_plane<NW>(h[j], e[j] & 1, true, L);
        orient_plane<NW>(l[j], e[j] & 1, false, L);
        uint32_t sum = 0;
#pragma unroll
        for (int k = 0; k < K; ++k)
          sum += *(const uint32_t*)((const char*)(tab + G.base[k]) + run_offset<NW>(h[j], l[j], G.a[k], G.q[k]));
        test[j] = ~sum & G.top;
        if (DEG) {
          uint32_t o[NW], some = 0;
          load_plane<NW>(o, ot, w, r);
#pragma unroll
          for (int i = 0; i < NW; ++i) {
            const uint32_t in = L >= 32u * (i + 1) ? kFull : (1u << (L & 31)) - 1u;
            some |= o[i] & (L > 32u * i ? in : 0u);
          }
          if (some) test[j] = G.top;
        }
        if (!have) test[j] = 0;
        any |= test[j];
      }
      if (!__any_sync(kFull, any)) continue;
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        uint32_t left = __ballot_sync(kFull, test[j] != 0);
        while (left) {
          const int src = __ffs(left) - 1;
          left &= left - 1;
          const uint32_t es = __shfl_sync(kFull, e[j], src);
          uint32_t t = __shfl_sync(kFull, test[j], src);
          Window<NW> w;
#pragma unroll
          for (int i = 0; i < NW; ++i) {
            w.h[i] = __shfl_sync(kFull, h[j][i], src);
            w.l[i] = __shfl_sync(kFull, l[j][i], src);
          }
          load_plane<NW>(w.o, ot, seg_w0 + (es >> 6), (es >> 1) & 31);
          orient_plane<NW>(w.o, es & 1, false, L);
          while (t) {
            const uint32_t c = (uint32_t)(__ffs(t) - 1) / G.bits;
            t &= t - 1;
            count_class<NW>(w, cls[c], cls[c + 1], lane, es, seg_pos0, records, hits, hit_count, hit_cap);
          }
        }
      }
    }
    u = stop;
  }
}

template <int NW, int K, bool DEG>
void run_screen(const GenomeView& g, const uint32_t* queue, const uint32_t* qcount, uint64_t seg_pos0,
                const ScreenGeom& geom, const uint32_t* records, const uint32_t* first, const uint32_t* tables,
                uint32_t L, uint64_t* hits, unsigned long long* hit_count, uint64_t hit_cap, int sm_count,
                cudaStream_t stream) {
  const size_t smem = (size_t)geom.entries * 4;
  cudaFuncSetAttribute(screen_kernel<NW, K, DEG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  screen_kernel<NW, K, DEG><<<sm_count, kScreenThreads, smem, stream>>>(
      g.hi, g.lo, g.ot, queue, qcount, seg_pos0, geom, records, first, tables, L, hits, hit_count, hit_cap);
}

}  // namespace

void launch_screen_tables(const ScreenGeom& geom, int nw, const uint32_t* records, const uint32_t* first,
                          uint32_t* tables, cudaStream_t stream) {
  const dim3 grid((geom.entries + 255) / 256, geom.words);
  if (nw == 1) screen_tables_kernel<1><<<grid, 256, 0, stream>>>(geom, records, first, tables);
  else screen_tables_kernel<2><<<grid, 256, 0, stream>>>(geom, records, first, tables);
}

void launch_screen(const GenomeView& g, const uint32_t* queue, const uint32_t* qcount, uint64_t seg_pos0,
                   const ScreenGeom& geom, int nw, const uint32_t* records, const uint32_t* first,
                   const uint32_t* tables, uint32_t L, uint64_t* hits, unsigned long long* hit_count,
                   uint64_t hit_cap, int sm_count, cudaStream_t stream) {
  auto run = nw == 1 ? (geom.K == 3 ? (geom.degenerate ? run_screen<1, 3, true> : run_screen<1, 3, false>)
                                    : (geom.degenerate ? run_screen<1, 4, true> : run_screen<1, 4, false>))
                     : (geom.K == 3 ? (geom.degenerate ? run_screen<2, 3, true> : run_screen<2, 3, false>)
                                    : (geom.degenerate ? run_screen<2, 4, true> : run_screen<2, 4, false>));
  run(g, queue, qcount, seg_pos0, geom, records, first, tables, L, hits, hit_count, hit_cap, sm_count, stream);
}

}  // namespace cof
