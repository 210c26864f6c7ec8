// Direct count: every start of the genome against a few compare variants,
// bit-sliced over the starts, without candidates.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "kernels.cuh"
#include "screen.cuh"

namespace cof {

constexpr int kDirectVariants = 8;  // variants per launch
constexpr int kDirectRows = 16;     // mismatch rows: kinds of pattern byte in use, a zero row, the separators

// A place in a unit's mismatch rows: row and word offset in bits 5-15, bit
// offset in bits 0-4.
struct DirectParams {
  uint32_t L = 0, variants = 0, rows = 0;
  uint8_t row_class[kDirectRows] = {};     // class bits; row 0 stays zero, row 1 holds the separators
  uint32_t pam_n[2] = {};                  // per strand: the PAM's positions ...
  uint16_t pam[2][kMaxL] = {};
  uint32_t id[kDirectVariants] = {}, limit[kDirectVariants] = {};
  uint32_t n[kDirectVariants] = {};        // ... and each variant's, padded to a multiple of 4 with row 0
  alignas(8) uint16_t pos[kDirectVariants][2][kMaxL] = {};
};

// A compare string with its id and mismatch limit.
struct DirectVariant {
  std::string key;
  uint32_t id, limit;
};
// Fills the parameters for `pattern` (L <= 64 bytes) and up to
// kDirectVariants variants; false where the kinds of pattern byte do not fit
// the rows.
bool plan_direct(const std::string& pattern, const DirectVariant* vars, size_t n, DirectParams& out);
// SM clocks the kernel takes per 2,048 starts.
double direct_cost(const DirectParams& p);
// Counts starts [32 * w_begin, 32 * w_end) below g.n - L + 1 and appends hit
// keys; adds the candidates (starts that match the PAM, per strand) to
// *qcount (may be null).
void launch_direct(const GenomeView& g, uint64_t w_begin, uint64_t w_end, const DirectParams& p, unsigned long long* qcount,
                   const HitSink& sink, int sm_count, cudaStream_t stream);

}  // namespace cof
