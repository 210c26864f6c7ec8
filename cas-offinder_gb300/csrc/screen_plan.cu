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

// P[mismatches of a random window against c concrete positions <= d].
double binomial_cdf(double c, int d) {
  const int n = (int)std::lround(c);
  double p = std::pow(0.25, n), s = 0;
  for (int k = 0; k <= std::min(d, n); ++k) {
    s += p;
    p *= 3.0 * (n - k) / (k + 1);
  }
  return std::min(1.0, s);
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
};

}  // namespace

const char* screen_level_name(uint32_t level) { return level < kLevelCount ? kLevels[level].name : "?"; }

namespace {

// Costs in SM clocks per 2,048 starts, of which `c` are candidates (measured
// at 0.08 and 0.2 candidates per start: 280 and 533 for one scanning word,
// 227 and 265 for the finder, 0.88 per candidate and word of the queue).
double scan_cost(double c, double words) { return words * (100.0 + 1.08 * c); }
double finder_cost(double c) { return 182.0 + 0.22 * c; }
double queue_cost(double c, double words) { return finder_cost(c) + words * (15.0 + 0.88 * c); }

// The scanning kernel stages up to 320 of 2,048 starts' candidates at a time
// and takes one-word windows.
bool can_scan(const FinderPattern& pat, double plus, double minus) {
  return pat.L <= 32 && std::max(plus, minus) <= 0.14;
}

}  // namespace

void plan_screen(const std::vector<const Variant*>& vars, const std::vector<uint32_t>& gids, const FinderPattern& pat,
                 int force_level, ScreenPlan& plan) {
  plan = ScreenPlan();
  const size_t V = vars.size();
  const uint32_t L = pat.L;
  if (V == 0 || L == 0 || L > (uint32_t)kMaxL) return;
  uint32_t limit = 0;
  for (const Variant* v : vars) limit = std::max<uint32_t>(limit, v->threshold);
  if (limit > kScreenMaxLimit) return;
  ScreenGeom& G = plan.geom;

  // Positions: how many variants can mismatch there.
  std::vector<uint32_t> cover(L, 0);
  for (const Variant* v : vars)
    for (uint32_t k = 0; k < L; ++k) {
      const uint32_t cl = class_of(v->key[k]);
      cover[k] += cl != 0;
      if (cl > 4) G.degenerate = 1;
    }
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
        guides.push_back(Guide{i, i, 1 << 30, -1});
      Guide& g = guides.back();
      g.end = i + 1;
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
    // Chance that a random candidate passes a class that holds `times` guides'
    // worth of the variants `members` (generation-order indexes): distinct
    // spellings on each run, each run's least count taken as that of
    // independent spellings.
    std::vector<uint32_t> spell;
    auto pass_rate = [&](const std::vector<size_t>& members, double times) {
      std::vector<double> dist(1, 1.0);  // distribution of the bound
      uint32_t lim = 0;
      for (size_t i : members) lim = std::max<uint32_t>(lim, vars[ord[i]]->threshold);
      for (uint32_t k = 0; k < G.K; ++k) {
        const uint32_t q = screen_run_len(G.K, k), at = G.a0 + screen_run_at(k);
        spell.clear();
        for (size_t i : members) {
          uint32_t s = 0;  // the class of each position, 4 bits
          for (uint32_t j = 0; j < q && at + j < L; ++j) s = s << 4 | class_of(vars[ord[i]]->key[at + j]);
          spell.push_back(s);
        }
        std::sort(spell.begin(), spell.end());
        spell.erase(std::unique(spell.begin(), spell.end()), spell.end());
        double concrete = 0;
        for (uint32_t s : spell)
          for (; s; s >>= 4) concrete += (s & 15) == 0 ? 0.0 : (s & 15) <= 4 ? 1.0 : (s & 15) <= 8 ? 0.3 : 0.6;
        concrete /= (double)spell.size();
        std::vector<double> next(dist.size() + q, 0.0);
        double before = 0;
        for (uint32_t d = 0; d <= q; ++d) {
          const double cdf =
              d == q ? 1.0 : 1.0 - std::pow(1.0 - binomial_cdf(concrete, (int)d), times * (double)spell.size());
          for (size_t j = 0; j < dist.size(); ++j) next[j + d] += dist[j] * (cdf - before);
          before = cdf;
        }
        dist.swap(next);
      }
      double p = 0;
      for (size_t j = 0; j < dist.size() && j <= lim; ++j) p += dist[j];
      return p;
    };
    // Share of random windows that match the PAM, per strand.
    double share[2] = {1.0, 1.0};
    for (uint32_t st = 0; st < 2; ++st)
      for (uint32_t j = 0; j < (st ? pat.nr : pat.nf); ++j)
        share[st] *= (4 - __builtin_popcount((st ? pat.rm[j] : pat.fm[j]) & 15u)) / 4.0;
    const double c = (share[0] + share[1]) * 2048.0;
    const bool may_scan = can_scan(pat, share[0], share[1]);
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
      if ((n + G.fields - 1) / G.fields > kScreenMaxWords) continue;
      if (force_level >= 0) {
        best_level = li;
        costs.emplace_back(0.0, li);
        break;
      }
      // Up to 4 guides, spread over all, stand for the rest.
      const size_t step = std::max<size_t>(1, guides.size() / 4);
      double work = 0;
      uint32_t sampled = 0;
      for (size_t gi = step / 2; gi < guides.size(); gi += step)
        for (uint32_t part = 0; part < lv.parts; ++part) {
          const Guide& g = guides[gi];
          std::vector<size_t> members;
          for (size_t i = g.begin; i < g.end; ++i)
            if (part_of(lv, g, i) == part) members.push_back(i);
          if (members.empty()) continue;
          const double times = (double)std::min<size_t>(lv.guides, guides.size());
          // Clocks to count a passing candidate.
          work += pass_rate(members, times) * (5.0 + 9.0 * std::ceil((double)members.size() * times / 32));
          ++sampled;
        }
      if (!sampled) continue;
      const double words = (double)((n + G.fields - 1) / G.fields), queue = queue_cost(c, words);
      const double cost = (may_scan ? std::min(queue, scan_cost(c, words)) : queue) + c * work / sampled * n;
      costs.emplace_back(cost, li);
      if (cost < best) best = cost, best_level = li;
    }
    if (costs.empty()) return;
    // The bit-sliced comparer, in clocks per 32 candidates: its table build
    // and the count (measured: 100 for 1 variant, 104 for 217 and 1,650 for
    // 1,000 without bulges).
    const bool chained = V >= 4 * guides.size();
    const double sliced = finder_cost(c) + c / 32 * (60.0 + (chained ? 0.5 : 1.6) * (double)std::max<size_t>(V, 32));
    plan.cost = std::min(best, sliced);
    if (force_level < 0 && best >= sliced) return;
    std::stable_sort(costs.begin(), costs.end());
    for (const auto& c : costs)
      if (plan.candidates.size() < 2 && c.first <= 1.8 * best) plan.candidates.push_back(c.second);
    if (!chained) plan.candidates.resize(1);  // whole guides only: the model is close, and timing costs as much as it gains
    plan.level = best_level;

    // Records by class, class by class.
    const uint32_t n = classes_of(kLevels[best_level], cls);
    G.words = (n + G.fields - 1) / G.fields;
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

}  // namespace cof
