// Table screen: finds the hits of a pattern group by looking parts of each
// candidate window up in tables of least mismatch counts, and counting only
// the candidates that the tables cannot rule out.
//
// A screen splits (part of) the window into K disjoint runs of at most 7
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

constexpr int kScreenRuns = 4;       // most runs of a screen
constexpr int kScreenRunMax = 7;     // positions per run at most (4^7 entries of 4 bytes = 64 KiB)
constexpr uint32_t kScreenMaxLimit = 15;  // largest mismatch limit (5-bit fields)
constexpr uint32_t kScreenMaxWords = 2048;

// Geometry of a group's screen (kernel argument).
struct ScreenGeom {
  uint32_t K = 0;                // runs (3 or 4)
  uint32_t a[kScreenRuns] = {};  // first position of each run in the oriented window
  uint32_t q[kScreenRuns] = {};  // its positions
  uint32_t base[kScreenRuns] = {};  // first entry of its table within a word's tables
  uint32_t cap[kScreenRuns] = {};   // largest entry of its table
  uint32_t entries = 0;          // 32-bit entries of one word's tables
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
  ScreenGeom geom;
  std::vector<uint32_t> records;  // screen_record_words(nw) per variant
  std::vector<uint32_t> first;    // words * (fields + 1): first record of each class of a word, then the word's end
  uint32_t level = 0;             // the partition taken (index of screen_levels)
  std::vector<uint32_t> candidates;  // levels worth timing, the model's best first
};

// Plans the screen of a pattern group of windows of L positions over `vars`
// (ids `gids`).  `on` stays false where the screen cannot run (a limit above
// 15) or its cost model puts the bit-sliced comparer ahead.  `force_level`
// >= 0 takes that partition.
void plan_screen(const std::vector<const Variant*>& vars, const std::vector<uint32_t>& gids, uint32_t L,
                 int force_level, ScreenPlan& plan);
// Text of a partition ("2/guide", "4 guides", ...).
const char* screen_level_name(uint32_t level);

// Fills the tables of a planned screen from its records (device pointers):
// geom.words * geom.entries words at `tables`.
void launch_screen_tables(const ScreenGeom& geom, int nw, const uint32_t* records, const uint32_t* first,
                          uint32_t* tables, cudaStream_t stream);
// Tests every entry of `queue` (count read on the device) against the
// screen's variants; appends hit keys as launch_comparer does.
void launch_screen(const GenomeView& g, const uint32_t* queue, const uint32_t* qcount, uint64_t seg_pos0,
                   const ScreenGeom& geom, int nw, const uint32_t* records, const uint32_t* first,
                   const uint32_t* tables, uint32_t L, uint64_t* hits, unsigned long long* hit_count,
                   uint64_t hit_cap, int sm_count, cudaStream_t stream);

}  // namespace cof
