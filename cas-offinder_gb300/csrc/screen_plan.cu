// Host side of the table screen (see screen.cuh): where its runs lie, how the
// variants are split into classes, and whether it pays.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>

#include "screen.cuh"

namespace cof {

namespace {

// Partitions of the variants into classes, from few large classes to many
// small ones: `guides` whole guides per class, or each guide's variants cut
// into `parts` by where their bulge lies.  A class's bound is the least over
// its variants on each run separately, so variants that agree on most runs
// belong together: those of one guide whose bulges lie close to each other.
struct Level {
  uint32_t guides, parts;
  const char* name;
};
constexpr Level kLevels[] = {{64, 1, "64 guides/class"}, {32, 1, "32 guides/class"}, {16, 1, "16 guides/class"},
                             {8, 1, "8 guides/class"},   {4, 1, "4 guides/class"},   {2, 1, "2 guides/class"},
                             {1, 1, "1 class/guide"},    {1, 2, "2 classes/guide"},  {1, 3, "3 classes/guide"}};
constexpr uint32_t kLevelCount = sizeof(kLevels) / sizeof(kLevels[0]);

// Random windows to estimate pass rates with: base[r][b][w] has bit j set
// where position j of run r of window w is base b.
constexpr uint32_t kWindows = 256;
constexpr size_t kSampled = 32;
struct Windows {
  uint8_t base[4][4][kWindows];
};
const Windows& windows() {
  static const Windows win = [] {
    Windows x;
    uint64_t s = 0x9E3779B97F4A7C15ull;
    for (auto& run : x.base)
      for (uint32_t w = 0; w < kWindows; ++w) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        const uint32_t hi = (uint32_t)(s >> 40) & 127u, lo = (uint32_t)(s >> 50) & 127u;
        for (uint32_t b = 0; b < 4; ++b) run[b][w] = (uint8_t)((b & 2 ? hi : ~hi) & (b & 1 ? lo : ~lo) & 127u);
      }
    return x;
  }();
  return win;
}

// least[w] = min(least[w], positions j of run r where window w's base b has
// bit j of m[b] set).
void least_counts(const Windows& win, uint32_t r, const uint8_t (&m)[4], uint8_t* least) {
  const auto& base = win.base[r];
  for (uint32_t w = 0; w < kWindows; ++w) {
    uint8_t x = (uint8_t)((m[0] & base[0][w]) | (m[1] & base[1][w]) | (m[2] & base[2][w]) | (m[3] & base[3][w]));
    x = (uint8_t)(x - ((x >> 1) & 0x55));
    x = (uint8_t)((x & 0x33) + ((x >> 2) & 0x33));
    x = (uint8_t)((x + (x >> 4)) & 0x0f);
    least[w] = std::min(least[w], x);
  }
}

// Class row of a pattern byte (bs_class_of), by table.
uint32_t class_of(char c) {
  static const std::array<uint8_t, 256> table = [] {
    std::array<uint8_t, 256> t{};
    for (int i = 0; i < 256; ++i) t[i] = (uint8_t)bs_class_of((unsigned char)i);
    return t;
  }();
  return table[(unsigned char)c];
}

// A guide: a run of variants in generation order.
struct Guide {
  size_t begin, end;
  int lo, hi;  // bulge positions in use
  uint32_t limit;
};

}  // namespace

const char* screen_level_name(uint32_t level) { return level < kLevelCount ? kLevels[level].name : "?"; }

namespace {

// Costs in SM clocks per 2,048 starts, of which `c` are candidates (measured
// at 0.08 and 0.2 candidates per start: 280 and 533 for one scanning word,
// 227 and 265 for the finder, 0.88 per candidate and word of the queue, 0.65
// where its windows are extracted first).
double scan_cost(double c, double words) { return words * (100.0 + 1.08 * c); }
double finder_cost(double c) { return 182.0 + 0.22 * c; }
double queue_cost(double c, double words) {
  return finder_cost(c) + (words < kWindowWords ? words * (15.0 + 0.88 * c) : 0.3 * c + words * (15.0 + 0.65 * c));
}

// The comparer that runs where no screen does, finder included.  Bit-sliced,
// in clocks per 32 candidates: its table build and the count (measured: 108 up
// to 32 variants; with bulges 131 for 224 and 1,231 for 3,554; without 363 for
// 256 and 1,250 for 1,000).  Variants of more than 32 counted positions run in
// the popcount comparer (measured per candidate, finder included: 16 up to 32
// variants, 30 for 96, 63 for 200 and 247 for 1,000).
double counted_cost(double c, size_t V, bool chained, uint32_t most_positions) {
  if (!bs_slots_for((int)most_positions)) return finder_cost(c) + c * (8.0 + 7.5 * (double)((V + 31) / 32));
  return finder_cost(c) + c / 32 * std::max(108.0, 60.0 + (chained ? 0.36 : 1.2) * (double)V);
}

// Starts from which on a screen of cost `best` is taken instead of the popcount
// comparer of cost `counted` (0: for any number).  Where counting the whole
// genome takes less than 0.1 ms of 152 SMs, launches and short lists weigh more
// than the counts: 100 40-nt NGG guides at limit 12, half the popcount
// comparer's time on 150 Mbp (1.05 against 2.14 ms), take 68 against 62 us on
// 3 Mbp and 41 against 26 on 100 kbp; 9 pairs of 2 x 20 nt at limit 8 take 115
// against 322 us on 3 Mbp and 47 against 43 on 100 kbp.  There the screen runs
// where it costs a fifth.
uint64_t screen_from(double best, double counted) {
  return 5.0 * best <= counted ? 0 : (uint64_t)(31.5e6 * 2048.0 / counted);
}

// The scanning kernel stages up to 320 of 2,048 starts' candidates at a time
// and takes one-word windows.
bool can_scan(const FinderPattern& pat, double plus, double minus) {
  return pat.L <= 32 && std::max(plus, minus) <= 0.14;
}

}  // namespace

void plan_screen(const std::vector<const Variant*>& vars, const std::vector<uint32_t>& gids, const FinderPattern& pat,
                 uint32_t sm_count, int force_level, ScreenPlan& plan) {
  plan = ScreenPlan();
  const size_t V = vars.size();
  const uint32_t L = pat.L;
  if (V == 0 || L == 0 || L > (uint32_t)kMaxL) return;
  ScreenGeom& G = plan.geom;
  uint32_t limit = 0;

  // Positions: how many variants can mismatch there.
  std::vector<uint32_t> cover(L, 0);
  uint32_t most = 0;  // positions that can mismatch, of one variant
  for (const Variant* v : vars) {
    limit = std::max<uint32_t>(limit, v->threshold);
    uint32_t positions = 0;
    for (uint32_t k = 0; k < L; ++k) {
      const uint32_t cl = class_of(v->key[k]);
      cover[k] += cl != 0;
      positions += cl != 0;
      if (cl > 4) G.degenerate = 1;
    }
    most = std::max(most, positions);
  }
  // Share of random windows that match the PAM, per strand.
  double share[2] = {1.0, 1.0};
  for (uint32_t st = 0; st < 2; ++st)
    for (uint32_t j = 0; j < (st ? pat.nr : pat.nf); ++j)
      share[st] *= (4 - __builtin_popcount((st ? pat.rm[j] : pat.fm[j]) & 15u)) / 4.0;
  const double c = (share[0] + share[1]) * 2048.0;
  const bool may_scan = can_scan(pat, share[0], share[1]);
  plan.counted = counted_cost(c, V, false, most);  // also where no screen can run
  plan.start_candidates = c;
  plan.most = most;
  if (limit > kScreenMaxLimit) return;
  uint32_t p0 = 0, p1 = L;
  while (p0 < p1 && !cover[p0]) ++p0;
  while (p1 > p0 && !cover[p1 - 1]) --p1;
  const uint32_t span = p1 - p0;
  if (span < 9) return;
  // Three runs of 7 positions (192 KiB of tables) for spans up to 23, four
  // of 7, 7, 6, 6 (160 KiB) beyond; of a longer span, the stretch that the
  // most variants use.
  G.K = span <= 23 ? 3 : 4;
  const uint32_t take = std::min<uint32_t>(span, G.K == 3 ? 21 : 26);
  uint32_t best_s = p0;
  uint64_t best_c = 0;
  for (uint32_t s = p0; s + take <= p1; ++s) {
    uint64_t c = 0;
    for (uint32_t k = s; k < s + take; ++k) c += cover[k];
    if (c > best_c) best_c = c, best_s = s;
  }
  G.a0 = best_s;
  // Fields of 4 bits (8 classes a word) hold three runs for limits up to 7;
  // otherwise 5 bits (6 classes).  Run 0's entries reach the top bit by
  // themselves; the other runs' caps keep the sum within the field.
  if (G.K == 3 && limit <= 7) {
    G.bits = 4, G.fields = 8, G.top = 0x88888888u;
    G.cap[0] = 7, G.cap[1] = 4, G.cap[2] = 4;
  } else {
    G.bits = 5, G.fields = 6, G.top = 0x21084210u;
    if (G.K == 3) G.cap[0] = 16, G.cap[1] = 7, G.cap[2] = 7;
    else G.cap[0] = 16, G.cap[1] = G.cap[2] = G.cap[3] = 5;
  }

  // Generation order (job by job, then by first insertion), cut into guides.
  std::vector<uint32_t> ord(V);
  {
    std::vector<uint64_t> rank(V);
    uint64_t job = 0;
    for (size_t i = 0; i < V; ++i) {
      if (i && vars[i] != vars[i - 1] + 1) ++job;
      rank[i] = (job << 32) | vars[i]->order;
      ord[i] = (uint32_t)i;
    }
    std::sort(ord.begin(), ord.end(), [&](uint32_t a, uint32_t b) { return rank[a] < rank[b]; });
    // A new job or another id starts a guide.
    std::vector<Guide> guides;
    std::vector<int> at_bulge(V);  // in generation order
    for (size_t i = 0; i < V; ++i) {
      const uint32_t v = ord[i];
      if (i == 0 || (rank[v] >> 32) != (rank[ord[i - 1]] >> 32) || vars[v]->id != vars[ord[i - 1]]->id)
        guides.push_back(Guide{i, i, 1 << 30, -1, 0});
      Guide& g = guides.back();
      g.end = i + 1;
      g.limit = std::max<uint32_t>(g.limit, vars[v]->threshold);
      at_bulge[i] = vars[v]->bulges.empty() ? 0 : std::abs(vars[v]->bulges.front().index);
      g.lo = std::min(g.lo, at_bulge[i]);
      g.hi = std::max(g.hi, at_bulge[i]);
    }

    // Each variant's rank by bulge position within its guide.
    std::vector<uint32_t> by_place(V);
    std::vector<uint32_t> at_count;
    for (const Guide& g : guides) {
      at_count.assign((size_t)(g.hi - g.lo + 2), 0);
      for (size_t i = g.begin; i < g.end; ++i) ++at_count[at_bulge[i] - g.lo + 1];
      for (size_t k = 1; k < at_count.size(); ++k) at_count[k] += at_count[k - 1];
      for (size_t i = g.begin; i < g.end; ++i) by_place[i] = at_count[at_bulge[i] - g.lo]++;
    }

    // Guides of like limits share classes: a class passes what its largest
    // limit passes.
    std::stable_sort(guides.begin(), guides.end(), [](const Guide& a, const Guide& b) { return a.limit < b.limit; });

    // The guide's variants in equal shares by bulge position.
    auto part_of = [&](const Level& lv, const Guide& g, size_t i) {
      return lv.parts > 1 ? by_place[i] * lv.parts / (uint32_t)(g.end - g.begin) : 0u;
    };
    // The class of each variant (in generation order) at a level.
    auto classes_of = [&](const Level& lv, std::vector<uint32_t>& cls) {
      cls.assign(V, 0);
      for (size_t gi = 0; gi < guides.size(); ++gi) {
        const Guide& g = guides[gi];
        for (size_t i = g.begin; i < g.end; ++i) cls[i] = (uint32_t)(gi / lv.guides) * lv.parts + part_of(lv, g, i);
      }
      return (uint32_t)((guides.size() + lv.guides - 1) / lv.guides) * lv.parts;
    };
    // Sampled guides stand for the rest: up to kSampled, evenly spaced.
    // bound[r][p][w] is the least mismatch count on run r of random window w
    // over the sample's variants whose bulge lies in sixth p of the guide; a
    // part of any level is a union of sixths.
    struct Sample {
      uint32_t limit;
      size_t variants[6];
      std::vector<uint8_t> bound;
    };
    std::vector<Sample> samples;
    {
      const size_t ns = std::min<size_t>(guides.size(), kSampled);
      const Windows& win = windows();
      samples.resize(ns);
      for (size_t k = 0; k < ns; ++k) {
        const Guide& g = guides[(2 * k + 1) * guides.size() / (2 * ns)];
        Sample& s = samples[k];
        s.limit = g.limit;
        s.bound.assign(G.K * 6 * kWindows, 8);
        std::fill(s.variants, s.variants + 6, 0);
        for (size_t i = g.begin; i < g.end; ++i) {
          const uint32_t part = by_place[i] * 6 / (uint32_t)(g.end - g.begin);
          ++s.variants[part];
          for (uint32_t r = 0; r < G.K; ++r) {
            const uint32_t q = screen_run_len(G.K, r), at = G.a0 + screen_run_at(r);
            uint8_t m[4] = {};
            for (uint32_t j = 0; j < q && at + j < L; ++j) {
              const uint32_t bits = class_bits_of((unsigned char)vars[ord[i]]->key[at + j]);
              for (int b = 0; b < 4; ++b) m[b] |= (uint8_t)((bits >> b & 1u) << j);
            }
            least_counts(win, r, m, s.bound.data() + (r * 6 + part) * kWindows);
          }
        }
      }
    }
    // What listing and counting the passing candidates costs at level lv with n
    // classes: SM clocks per candidate, and items listed per candidate.
    auto count_work = [&](const Level& lv, uint32_t n, double* items) {
      const size_t ns = samples.size(), whole = (guides.size() + lv.guides - 1) / lv.guides, span = 6 / lv.parts;
      const size_t groups = std::min(ns, whole), t = ns / groups;
      const double more = std::max(1.0, (double)std::min<size_t>(lv.guides, guides.size()) / (double)t);
      double pass = 0, counts = 0;  // sums of P[class passes], and times its counting steps
      uint32_t classes = 0;
      std::vector<uint8_t> least(kWindows);
      for (size_t k = 0; k < groups; ++k)
        for (uint32_t p = 0; p < lv.parts; ++p) {
          // t samples (and `more` - 1 times as many like them) in one class.
          // A random window's runs are independent, so the bound's
          // distribution is that of the runs' counts convolved.
          uint32_t limit = 0;
          size_t members = 0;
          std::vector<double> dist(1, 1.0);
          for (uint32_t r = 0; r < G.K; ++r) {
            std::fill(least.begin(), least.end(), 8);
            for (size_t j = 0; j < t; ++j) {
              const Sample& s = samples[k * t + j];
              for (size_t x = p * span; x < (p + 1) * span; ++x) {
                const uint8_t* b = s.bound.data() + (r * 6 + x) * kWindows;
                for (uint32_t w = 0; w < kWindows; ++w) least[w] = std::min(least[w], b[w]);
                if (r == 0) members += s.variants[x];
              }
              limit = std::max(limit, s.limit);
            }
            uint32_t hist[9] = {};
            for (uint32_t w = 0; w < kWindows; ++w) ++hist[std::min<uint32_t>(least[w], G.cap[r])];
            std::vector<double> next(dist.size() + 8, 0.0);
            double at_least = 1.0;
            uint32_t below = 0;
            for (uint32_t d = 0; d <= 8; ++d) {
              below += hist[d];
              const double left = (double)(kWindows - below) / kWindows, beyond = more > 1.0 ? std::pow(left, more) : left;
              for (size_t j = 0; j < dist.size(); ++j) next[j + d] += dist[j] * (at_least - beyond);
              at_least = beyond;
            }
            dist.swap(next);
          }
          if (!members) continue;
          double passes = 0;
          for (size_t j = 0; j < dist.size() && j <= limit; ++j) passes += dist[j];
          pass += passes;
          counts += passes * std::ceil((double)members * more / 32);
          ++classes;
        }
      if (!classes) return 0.0;
      const double words = (double)((n + G.fields - 1) / G.fields);
      const double q = 1.0 - std::pow(std::max(0.0, 1.0 - pass / classes), n / words);  // an item, per candidate and word
      *items = q * words;
      return words * (0.5 * (1.0 - std::pow(1.0 - q, 32.0)) + 4.3 * q) + 3.4 * counts / classes * n;
    };
    double best = 1e300;
    uint32_t best_level = 0;
    std::vector<std::pair<double, uint32_t>> costs;
    std::vector<uint32_t> cls;
    for (uint32_t li = 0; li < kLevelCount; ++li) {
      const Level& lv = kLevels[li];
      if (force_level >= 0 && (uint32_t)force_level != li) continue;
      if (force_level < 0 && lv.guides > 1 && lv.guides >= 2 * guides.size()) continue;
      if (force_level < 0 && lv.parts > 1 && V < 4 * guides.size()) continue;
      const uint32_t n = (uint32_t)((guides.size() + lv.guides - 1) / lv.guides) * lv.parts;
      if ((n + G.fields - 1) / G.fields > screen_max_words(sm_count)) continue;
      const double words = (double)((n + G.fields - 1) / G.fields), queue = queue_cost(c, words);
      double items = 0;
      const double work = c * count_work(lv, n, &items), listed = c / 2048.0 * items;
      const double cost = (may_scan ? std::min(queue, scan_cost(c, words)) : queue) + work +
                          95.0 * 2048.0 * std::max(0.0, listed - kScreenListed);
      costs.emplace_back(cost, li);
      if (cost < best) best = cost, best_level = li, plan.listed = listed;
    }
    if (costs.empty()) return;
    const bool chained = V >= 4 * guides.size();
    plan.cost = best;
    plan.counted = counted_cost(c, V, chained, most);
    if (force_level < 0 && best >= plan.counted) return;
    if (!bs_slots_for((int)most)) plan.from = screen_from(best, plan.counted);
    std::stable_sort(costs.begin(), costs.end());
    for (const auto& c : costs)
      if (plan.candidates.size() < 2 && c.first <= 1.8 * best) plan.candidates.push_back(c.second);
    if (!chained) plan.candidates.resize(1);  // whole guides only: the model is close, and timing costs as much as it gains
    plan.level = best_level;

    // Records by class, class by class.  The classes are dealt out to the words
    // in turn, each round one word further on (parts of a guide differ), so
    // that candidates pass all words alike: each CTA's list is an equal share
    // of the room.
    const uint32_t n = classes_of(kLevels[best_level], cls);
    G.words = (n + G.fields - 1) / G.fields;
    for (uint32_t& x : cls) x = (x + x / G.words) % G.words * G.fields + x / G.words;
    plan.scans = may_scan && scan_cost(c, G.words) < queue_cost(c, G.words);
    std::vector<uint32_t> start((size_t)G.words * G.fields + 1, 0);
    for (size_t i = 0; i < V; ++i) ++start[cls[i] + 1];
    for (size_t c = 1; c < start.size(); ++c) start[c] += start[c - 1];
    plan.first.resize((size_t)G.words * (G.fields + 1));
    for (uint32_t w = 0; w < G.words; ++w)
      for (uint32_t c = 0; c <= G.fields; ++c) plan.first[w * (G.fields + 1) + c] = start[w * G.fields + c];
    const int nw = L <= 32 ? 1 : 2;
    const uint32_t rec = screen_record_words(nw);
    plan.records.assign(V * rec, 0);
    for (size_t i = 0; i < V; ++i) {
      const Variant& v = *vars[ord[i]];
      uint32_t* r = &plan.records[(size_t)start[cls[i]]++ * rec];
      for (uint32_t k = 0; k < L; ++k) {
        const uint32_t m = class_bits_of((unsigned char)v.key[k]);
        if (k < 32) {
          for (int b = 0; b < 5; ++b) r[b] |= (m >> b & 1u) << k;
        } else {
          for (int b = 0; b < 4; ++b) r[8 + b] |= (m >> b & 1u) << (k - 32);
          r[6] |= (m >> 4 & 1u) << (k - 32);
        }
      }
      r[5] = gids[ord[i]] << 4 | v.threshold;
    }
  }
  plan.on = true;
}

// The comparers write a 32-candidate group's hits one candidate after the
// other, so that the bit-sliced one waits for the variant with the most
// (measured: 210 clocks a turn) and the popcount one for each candidate with
// some (190).  The direct count writes the hits of a word of 32 starts one
// after the other, a warp's 32 words in step: 47 clocks a turn and 15 a hit
// (8 40-nt NGG guides at limit 24, 24 hits in 1,000 windows: 6,665 clocks
// measured, 6,743 by this sum; one at limit 40, all windows hits: 5,615 and
// 5,583).
HitCosts hit_costs(const std::vector<const Variant*>& vars, const ScreenPlan& plan) {
  const double c = plan.start_candidates;
  double none = 1.0, top = 0.0, direct = 0.0;
  for (const Variant* v : vars) {
    // P[a random window has at most the limit's mismatches].
    std::vector<double> mm(1, 1.0);
    for (char ch : v->key) {
      const double q = __builtin_popcount(class_bits_of((unsigned char)ch) & 15u) / 4.0;
      if (q == 0) continue;
      mm.push_back(0.0);
      for (size_t k = mm.size() - 1; k; --k) mm[k] = mm[k] * (1 - q) + mm[k - 1] * q;
      mm[0] *= 1 - q;
    }
    double p = 0;
    for (size_t k = 0; k < mm.size() && k <= v->threshold; ++k) p += mm[k];
    none *= 1 - std::min(p, 1.0);
    top = std::max(top, p);
    const double word = c * p / 128;  // hits expected of 32 starts on one strand
    const double turns = std::min(32.0, std::min(1.0, 32 * word) * (word + 2.07 * std::sqrt(word) + 0.7));
    direct += 4 * 47.0 * turns + 15.0 * c * p;
  }
  if (!bs_slots_for((int)plan.most)) return HitCosts{direct, 190.0 * c * (1 - none)};
  // The largest of V binomials of 32 candidates.
  const double spread = std::sqrt(std::log((double)vars.size()) * 32 * top * (1 - std::min(top, 1.0)));
  return HitCosts{direct, 210.0 * c / 32 * std::min(32.0, 32 * top + spread)};
}

}  // namespace cof
