// Table screen: finds the hits of a pattern group by looking parts of each
// candidate window up in tables of least mismatch counts, and counting only
// the candidates that the tables cannot rule out.
//
// A screen splits (part of) the window into K disjoint runs of 6 or 7
// positions.  For a class of compare variants, table k holds for each of the
// 4^q words that run k of a window can spell the least mismatch count of any
// variant of the class on that run.  The sum over the runs is a lower bound
// of every variant's mismatch count, so a candidate whose sum exceeds the
// limit holds no hit of the class; the rest (a few per cent) are counted
// exactly against the class's variants.  Non-base bytes read as some base in
// the lookups, which can only lower the bound for the variants' concrete
// bases; a degenerate code may match a non-base byte, so groups with such
// codes count every window that holds one.
//
// Classes are fields of F bits of one 32-bit table word: one lookup per run
// serves all classes of the word, and the K looked-up words are added.  Run
// 0's entries carry the bias T - 1 - limit (T = 2^(F-1)), so a field's top
// bit is set exactly where its sum exceeds the limit; entries are capped so
// that no field overflows (a cap only lowers the bound).
#pragma once

#include <cstdint>
#include <vector>

#include "cof_internal.h"
#include "kernels.cuh"

namespace cof {

// Runs of a screen, from its first position `a0` on: three of 7 positions, or
// four of 7, 7, 6 and 6.  The layout is fixed so that a run's bits are reached
// by immediate shifts and masks; positions past the window or outside the
// variants' span mismatch nobody.
constexpr int kScreenRuns = 4;
constexpr uint32_t screen_run_at(uint32_t k) { return k < 3 ? 7u * k : 20u; }
constexpr uint32_t screen_run_len(uint32_t K, uint32_t k) { return K == 4 && k >= 2 ? 6u : 7u; }
// First entry of each run's table within a word's tables, and their size.
constexpr uint32_t screen_base(uint32_t k) { return k == 0 ? 0u : k == 1 ? 16384u : k == 2 ? 32768u : 36864u; }
constexpr uint32_t screen_entries(uint32_t K) { return K == 4 ? 40960u : 49152u; }
constexpr uint32_t kScreenMaxLimit = 15;  // largest mismatch limit (5-bit fields)
// Most table words of a screen launched as `sm_count` CTAs.  A list item holds
// its word in 3 bits, relative to the first word of its CTA's share; a share
// of 7 words' candidates touches 8 words.
constexpr uint32_t screen_max_words(uint32_t sm_count) { return 7 * sm_count < 768 ? 7 * sm_count : 768; }

// Geometry of a group's screen (kernel argument).
struct ScreenGeom {
  uint32_t K = 0;                  // runs (3 or 4)
  uint32_t a0 = 0;                 // first position of the runs in the oriented window
  uint32_t cap[kScreenRuns] = {};  // largest entry of each run's table
  uint32_t bits = 4;             // field width F
  uint32_t fields = 8;           // classes per word
  uint32_t top = 0x88888888u;    // the fields' top bits
  uint32_t words = 0;            // table words (sets of `fields` classes)
  uint32_t degenerate = 0;       // some variant uses an IUPAC code other than N
};

// Uint32 words of one variant record: class masks t, c, a, g, o and
// meta = id << 4 | limit (NW = 2: the second mask words too).
constexpr uint32_t screen_record_words(int nw) { return nw == 1 ? 8 : 12; }

// A planned screen on the host: variants sorted by class.
struct ScreenPlan {
  bool on = false;
  bool scans = false;  // the scanning kernel rather than the finder and the screen of its queue
  double listed = 0;    // candidates expected in the list, per start
  double cost = 0;          // SM clocks per 2,048 starts of the screen ...
  double counted = 0;       // ... and of the comparer that runs without one
  uint64_t from = 0;        // the screen pays for genomes of this many positions or more
  double start_candidates = 0;  // candidates expected per 2,048 starts
  uint32_t most = 0;            // positions that can mismatch, of one variant
  ScreenGeom geom;
  std::vector<uint32_t> records;  // screen_record_words(nw) per variant
  std::vector<uint32_t> first;    // words * (fields + 1): first record of each class of a word, then the word's end
  uint32_t level = 0;             // the partition taken (screen_level_name)
  std::vector<uint32_t> candidates;  // levels worth timing, the model's best first
  bool windows() const;  // it extracts the queue's windows first
};

// Plans the screen of a pattern group (PAM scan `pat`) over `vars` (ids
// `gids`) for launches on `sm_count` SMs.  `on` stays false where the screen
// cannot run (a limit above 15, more than screen_max_words) or its cost model
// puts the comparer that would run without it (bit-sliced, or popcount for
// variants of more than 32 counted positions) ahead.  `force_level` >= 0 takes that partition.
void plan_screen(const std::vector<const Variant*>& vars, const std::vector<uint32_t>& gids, const FinderPattern& pat,
                 uint32_t sm_count, int force_level, ScreenPlan& plan);
// What writing the hits that random windows give adds to the direct count and
// to the comparer that runs without a screen, in clocks per 2,048 starts, for
// a few variants; `plan` as plan_screen left it.
struct HitCosts {
  double direct, counted;
};
HitCosts hit_costs(const std::vector<const Variant*>& vars, const ScreenPlan& plan);
// Text of a partition ("2 classes/guide", "4 guides/class", ...).
const char* screen_level_name(uint32_t level);

// Candidates that passed a class, listed per warp of the screening launch: an
// item is {position relative to the launch's base << 1 | strand, the passed
// classes' top bits | kOddWindow | the word relative to the first of its CTA,
// first word of the oriented window's hi and lo planes}.
struct ScreenList {
  uint4* items = nullptr;      // `room` of them, shared out evenly over the warps
  uint32_t* counts = nullptr;  // items of each warp
  uint64_t room = 0;
  // Windows of a queue's candidates, for screens of kWindowWords words or more:
  // the oriented window's first word of the hi and lo planes (two-word windows:
  // 32 positions from the screen's first on).  Room for a full queue.
  uint2* windows = nullptr;
};
// Words from which on a queue's windows are extracted once, ahead of the
// lookups (measured: a gain at 16, none at 4).
constexpr uint32_t kWindowWords = 8;
inline bool ScreenPlan::windows() const { return on && !scans && geom.words >= kWindowWords; }
// Set in an item whose window may hold a non-base byte (a bit that is neither
// a field's top bit nor part of the relative word).
constexpr uint32_t kOddWindow = 1u << 5;
// Most warps of a launch on a device of `sm_count` SMs, and the items
// `positions` start positions should have room for.  A warp whose list is
// full counts its further candidates on the spot, so the size only affects
// the speed.
// Half an item per start of a segment (2^26 starts), of which 0.25 leaves room
// for uneven shares.  A listed item costs up to 20 SM clocks, one counted on
// the spot 95 (64 guides with 2 DNA and 2 RNA bulges, limit 6, on 2^26 starts:
// 15.9 ms with room for 0.19 items a start, 12.2 ms with 0.5).
constexpr double kScreenListed = 0.25;
uint32_t screen_lists(int sm_count);
uint64_t screen_list_items(uint64_t positions);

// Device side of a group's screen.
struct ScreenTables {
  const uint32_t *records, *first, *tables;
};
// Where hits go (as launch_comparer).
struct HitSink {
  uint64_t* hits;
  unsigned long long* count;
  uint64_t cap;
};

// Fills the tables of a planned screen from its records (device pointers):
// geom.words * screen_entries(geom.K) words at `tables`.
void launch_screen_tables(const ScreenGeom& geom, int nw, const uint32_t* records, const uint32_t* first,
                          uint32_t* tables, cudaStream_t stream);
// Tests every entry of `queue` (count read on the device) against the
// screen's variants; appends hit keys as launch_comparer does.  May mark
// entries of the queue.
void launch_screen(const GenomeView& g, uint32_t* queue, const uint32_t* qcount, uint64_t seg_pos0,
                   const ScreenGeom& geom, int nw, const ScreenTables& tb, uint32_t L, const ScreenList& list,
                   const HitSink& sink, int sm_count, cudaStream_t stream);
// PAM scan and screen in one kernel, without a candidate queue, for windows
// of up to 32 positions: plane words [w_begin, w_end), at most
// kScanWords of them; adds the candidates found to *qcount.
constexpr uint64_t kScanWords = 1ull << 24;
void launch_scan_screen(const GenomeView& g, uint64_t w_begin, uint64_t w_end, const FinderPattern& pat,
                        const ScreenGeom& geom, const ScreenTables& tb, const ScreenList& list,
                        unsigned long long* qcount, const HitSink& sink, int sm_count, cudaStream_t stream);

}  // namespace cof
