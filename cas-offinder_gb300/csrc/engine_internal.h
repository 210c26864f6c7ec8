// Internal types of libcasoff.so shared by engine.cu and server.cu: device
// buffers, the resident genome, pattern groups and the handle.  Not part of
// the public ABI.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/cof.h"
#include "cof_internal.h"
#include "direct.cuh"
#include "kernels.cuh"
#include "screen.cuh"

namespace cof {
namespace eng {

constexpr uint64_t kSegPositions = 1ull << 26;  // start positions per finder/comparer pass
constexpr uint64_t kSegWords = kSegPositions / 32;

struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  // With a stream set, allocation and release are stream-ordered
  // (cudaMallocAsync / cudaFreeAsync on it): no device-wide synchronisation.
  cudaStream_t st = nullptr;
  DevBuf() = default;
  explicit DevBuf(cudaStream_t s) : st(s) {}
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), cap(o.cap), st(o.st) { o.p = nullptr, o.cap = 0; }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p, cap = o.cap, st = o.st;
      o.p = nullptr, o.cap = 0;
    }
    return *this;
  }
  ~DevBuf() { release(); }
  void release() {
    if (p) st ? cudaFreeAsync(p, st) : cudaFree(p);
    p = nullptr;
    cap = 0;
  }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    release();
    cudaError_t e = st ? cudaMallocAsync(&p, bytes ? bytes : 1, st) : cudaMalloc(&p, bytes ? bytes : 1);
    if (e == cudaSuccess) cap = bytes;
    else p = nullptr;
    return e;
  }
  template <typename T>
  T* as() const {
    return (T*)p;
  }
};

struct HostPinned {
  void* p = nullptr;
  size_t cap = 0;
  ~HostPinned() {
    if (p) cudaFreeHost(p);
  }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    if (p) cudaFreeHost(p);
    p = nullptr;
    cap = 0;
    cudaError_t e = cudaMallocHost(&p, bytes ? bytes : 1);
    if (e == cudaSuccess) cap = bytes;
    return e;
  }
};

// A genome resident on the device.
struct DevGenome {
  uint64_t n = 0;
  uint32_t n_rec = 0;
  uint64_t n_exc = 0;
  DevBuf hi, lo, ot, exc_pos, exc_byte, rec_start, rec_name_off, rec_name_len, rec_names;
  bool loaded = false;
  GenomeView view() const {
    GenomeView g;
    g.hi = hi.as<uint32_t>();
    g.lo = lo.as<uint32_t>();
    g.ot = ot.as<uint32_t>();
    g.exc_pos = exc_pos.as<uint64_t>();
    g.exc_byte = exc_byte.as<uint8_t>();
    g.n_exc = n_exc;
    g.n = n;
    g.rec_start = rec_start.as<uint64_t>();
    g.rec_name_off = rec_name_off.as<uint32_t>();
    g.rec_name_len = rec_name_len.as<uint32_t>();
    g.rec_names = rec_names.as<char>();
    g.n_rec = n_rec;
    return g;
  }
};

// cof_handle::qcounts for `passes` passes (segment, group): a 64-bit candidate
// count each -- a scanning group counts a whole genome in one pass, two
// candidates a start; a finder pass fills its queue's count, at most 2^27, in
// the low half -- and then a 32-bit tile counter each.
struct PassCounts {
  unsigned long long* counts;
  uint32_t* tiles;
  PassCounts(const DevBuf& b, uint64_t passes) : counts(b.as<unsigned long long>()), tiles((uint32_t*)(counts + passes)) {}
  uint32_t* queue(uint64_t pass) const { return (uint32_t*)(counts + pass); }
  static size_t bytes(uint64_t passes) { return passes * 12; }
};

struct KernelStat {
  uint64_t launches = 0;
  double ms = 0;
  double units = 0;
};

// Compare variants (of one or more jobs) that share one padded pattern.
struct PatternGroup {
  std::string pattern;
  uint32_t L = 0;
  FinderPattern fpat{};
  int nw = 1;                  // 32-bit words per window (popcount comparer)
  int bs_slots = 0;            // bit-sliced slot count, 0 = popcount comparer
  bool concrete_only = true;   // no variant uses a degenerate IUPAC code
  bool bs_narrow = false;      // bit-sliced counts fit bit_width(bs_slots) planes (bs_narrow_ok)
  std::vector<uint32_t> gids;  // global variant ids, ascending
  double nonN_sum = 0;         // sum of non-N positions over the group's variants
  // Bit-sliced comparer programs (layout in kernels.cuh): bs_chunks chunks of
  // 32 lane programs, each a first variant and bs_m - 1 update steps.
  uint32_t bs_chunks = 0, bs_m = 1;
  std::vector<uint32_t> bs_candidates;             // lengths m worth timing (cost model's best first)
  std::vector<std::pair<uint32_t, float>> bs_tuned;  // (m, comparer µs per segment) measured by the autotuner
  DevBuf vmask, bs_prog, bs_pgid;
  // Table screen (screen.cuh); where it runs, bs_slots is 0.
  bool screen_on = false;
  ScreenGeom screen;
  uint32_t screen_level = 0;
  std::vector<uint32_t> screen_levels;                  // partitions worth timing (cost model's best first)
  std::vector<std::pair<uint32_t, float>> screen_tuned;  // (partition, µs per segment) measured by the autotuner
  DevBuf screen_records, screen_first, screen_tables;
  uint64_t screen_from = 0;  // the choice between screen and popcount comparer changes at this many positions (0: nowhere)
  uint64_t scan_words = kScanWords;  // words of a scanning launch: its list holds what passes
  bool screen_scans = false;  // the screen scans the planes itself: no finder pass, no candidate queue
  bool direct_on = false;     // direct count (direct.cuh): no tables, no candidates
  DirectParams direct;
  bool scans() const { return screen_scans || direct_on; }
  int comparer() const { return direct_on ? 4 : screen_on ? 3 : bs_slots ? 2 : 1; }  // as cof_comparer_info
  // The screen extracts the queue's windows first.
  bool windows() const { return screen_on && !screen_scans && screen.words >= kWindowWords; }
  ScreenTables screen_tb() const {
    return ScreenTables{screen_records.as<uint32_t>(), screen_first.as<uint32_t>(), screen_tables.as<uint32_t>()};
  }
};

}  // namespace eng
}  // namespace cof

using namespace cof;
using namespace cof::eng;

struct cof_handle {
  int device = 0;
  int sm_count = 0;
  cudaStream_t stream = nullptr;   // comparer, formatting, copies
  cudaStream_t stream2 = nullptr;  // finder passes, one segment ahead of the comparer
  cudaEvent_t ev_start = nullptr, ev_found[2] = {nullptr, nullptr}, ev_used[2] = {nullptr, nullptr};
  // Streamed upload (cof_search_planes).  From page-locked planes every copy
  // is queued at once on stream3, which runs ahead at the link's rate, in the
  // chunks upload_ends; upload_ev[c] marks chunk c as copied.  From pageable
  // planes the copies go on stream2, one segment ahead of the finders.
  cudaStream_t stream3 = nullptr;
  std::vector<cudaEvent_t> upload_ev;
  std::vector<uint64_t> upload_ends;  // words
  size_t upload_pending = 0;  // segments of the current streamed upload (0: none)
  size_t upload_issued = 0;   // segments whose copies are queued so far
  bool upload_pinned = false;  // the host planes are page-locked
  const uint32_t* upload_src[3] = {nullptr, nullptr, nullptr};  // host planes (valid during the call)
  uint64_t upload_words = 0;
  std::string err;

  // The batch: one or more parsed input files ("jobs").  Variant ids are
  // global and job-major (job j owns [job_gid0[j], job_gid0[j+1])), so one
  // sort of the hit keys yields every job's rows contiguously, in job order.
  std::vector<Job> jobs;
  std::vector<uint32_t> job_gid0;
  bool jobs_on_device = false;
  uint64_t planned_positions = 0;  // the genome's when the groups' comparers were chosen
  int comparer_kind = 0;  // cof_set_comparer
  std::vector<PatternGroup> groups;  // jobs sharing a padded pattern share finder + comparer passes
  DevBuf vfmt, sfmt, pool;           // row formatting tables over all variants
  DevGenome genome, scratch;

  // An allocation has failed: screens take no more memory than they hold until
  // a genome is loaded (a try for each search would free, fail and wait for the
  // device each time, and change the captured passes).
  bool memory_short = false;
  DevBuf screen_windows;  // windows of a queue's candidates (ScreenList), used on `stream`
  DevBuf screen_items, screen_counts;  // candidates that passed a screen (ScreenList), used on `stream`
  DevBuf queue[2], qcounts, hits, hits_sorted, summary_counts, hit_count, sort_tmp, row_bytes, row_offsets, row_count, text, small,
      job_start, job_bytes;
  DevBuf tune_bufs[3];  // a screen's records, classes and tables while its partitions are timed
  HostPinned stage;  // page-locked source of the batch's tables (Upload)
  HostPinned host_text, small_out;  // small_out: SmallOut of the latest search
  DevBuf stream_dev[2];  // cof_search_stream: row chunks on the device / in pinned memory
  HostPinned stream_host[2];
  cudaEvent_t stream_ev[2] = {nullptr, nullptr};
  std::string summary_text;
  std::vector<std::map<std::string, unsigned long long>> summaries;  // per job
  bool summary_on = false;
  uint64_t last_hits = 0, last_rows = 0;
  std::vector<uint64_t> job_byte0;  // row text of job j: [job_byte0[j], job_byte0[j+1]) of host_text

  bool profiling = false;
  // Pinned host buffers for served results, reused across requests.
  std::mutex pinned_mu;
  std::multimap<size_t, void*> pinned_free;
  size_t pinned_pooled = 0;
  // CUDA graph of the finder / comparer passes of a search, replayed while
  // everything its launches depend on (pass_key) is unchanged.
  cudaGraphExec_t pass_graph = nullptr;
  std::string pass_key;
  uint64_t pass_nseg = 0;
  bool use_graphs = true;
  bool autotune = true;  // time the lane-program lengths on the first search of a job set
  std::map<std::string, KernelStat> stats;
  std::vector<cudaEvent_t> event_pool;  // reused timing events (profiling)
  cudaEvent_t timer_a = nullptr, timer_b = nullptr;
};


namespace cof {
namespace eng {

cof_status fail(cof_handle* h, cof_status st, const std::string& msg);

#define COF_CUDA(h, call)                                                                           \
  do {                                                                                              \
    cudaError_t e_ = (call);                                                                        \
    if (e_ != cudaSuccess)                                                                          \
      return ::cof::eng::fail(h, e_ == cudaErrorMemoryAllocation ? COF_ERR_NOMEM : COF_ERR_CUDA,    \
                              std::string(#call) + ": " + cudaGetErrorString(e_));                  \
  } while (0)

// PAM-scan pattern from the forward pattern and its reverse complement.
bool make_finder_pattern(const std::string& fwd, const std::string& rev, FinderPattern& fp);
std::string revcomp(const std::string& s);
// Initialises g (pattern, L, word count, finder pattern) for a padded pattern.
void init_group(PatternGroup& g, const std::string& pattern);
// Pool of pinned host buffers kept by the handle: acquire returns a buffer of
// at least `bytes` (its size in *cap), or nullptr; release gives it back.
// Thread-safe.
void* pinned_acquire(cof_handle* h, size_t bytes, size_t* cap);
void pinned_release(cof_handle* h, void* p, size_t cap);

// Host side of a pattern group's comparer tables (built without the GPU).
struct GroupHost {
  std::vector<unsigned char> masks;  // popcount comparer (only when the bit-sliced one cannot run)
  std::vector<uint32_t> prog, pgid;  // bit-sliced lane programs
  ScreenPlan screen;                 // table screen (then the others stay empty)
};
// Fills g's host-side fields (slots, chunks, m, screen, ...) and `gh` for
// `vars` (ids g.gids); `kind` as cof_set_comparer, `sm_count` the SMs the
// launches get, `positions` the genome's.  Thread-safe: touches only its
// arguments.
void build_group_host(int kind, int sm_count, uint64_t positions, PatternGroup& g, const std::vector<const Variant*>& vars, GroupHost& gh);
// Host-to-device copies gathered into one page-locked buffer, so that they are
// queued without waiting.  The sources may go once `run` returns.
struct Upload {
  struct Part {
    DevBuf* dst;
    const void* src;
    size_t bytes;
  };
  std::vector<Part> parts;
  void add(DevBuf& dst, const void* src, size_t bytes) { parts.push_back(Part{&dst, src, bytes}); }
  // Copies every part on `st` by way of `stage`, whose earlier copies are done.
  cof_status run(cof_handle* h, HostPinned& stage, cudaStream_t st);
};
// Copies `gh` into g's device buffers on `st`; gh must stay alive until the
// copies are done.
cof_status upload_group(cof_handle* h, PatternGroup& g, const GroupHost& gh, cudaStream_t st);
// Compares the candidates of one finder pass (queue `q`, count `qc`, segment
// starting at `pos0`) with g's variants: screen, bit-sliced or popcount
// comparer.  `tile_ctr`: a zeroed u32 of this launch.  Runs on h->stream.
void launch_group_compare(const cof_handle* h, const PatternGroup& g, uint32_t* q, const uint32_t* qc,
                          uint32_t* tile_ctr, uint64_t pos0, const HitSink& sink);
// Scans plane words [w0, w1) for g (scans()) on h->stream; candidates are
// added to *qc.
void launch_group_scan(const cof_handle* h, const PatternGroup& g, uint64_t w0, uint64_t w1, unsigned long long* qc,
                       const HitSink& sink);
// b.ensure(bytes) for memory that a call cannot do without: where there is not
// enough, once more after give_back.  On the thread that launches the screens.
cudaError_t need(cof_handle* h, DevBuf& b, size_t bytes);
// Frees the buffers of ensure_screen_list that only speed depends on (false:
// there are none).  Launches queued so far are waited for.
bool give_back(cof_handle* h);
// The list buffers of the screens of launches over up to `positions` starts
// (with `windows`, those of a queue's windows too).
cof_status ensure_screen_list(cof_handle* h, uint64_t positions, bool windows);
// Lane programs of the bit-sliced comparer for `vars` (ids `gids`), `S` slots,
// class rows of `row` words; layout in kernels.cuh.
// force_m (1-24) replaces the cost model's choice of m; `ranked` (may be
// null) receives the model's best m and up to two runners-up.
void build_bs_programs(const std::vector<const Variant*>& vars, const std::vector<uint32_t>& gids, int S,
                       uint32_t row, std::vector<uint32_t>& prog, std::vector<uint32_t>& pgid, uint32_t& chunks,
                       uint32_t& m, uint32_t force_m, std::vector<uint32_t>* ranked);
// Row shapes of `vars` (variant i gets id first_gid + i) appended to the
// formatting tables vf (indexed by id), sf and pool.
void append_format_tables(const Job& job, std::vector<VariantFmt>& vf, std::vector<ShapeFmt>& sf, std::string& pool);

}  // namespace eng
}  // namespace cof
