// Replays the planner of nb_accelerations_noalloc (csrc/noalloc_plan.hpp) on the host.
// Arguments: threads, i-particles per thread and j-tile of its kNaCount shapes, then SMs and
// the CTAs per SM of each shape, then the sizes from, to and step.  Prints the first plan
// that is refused, does not fit, leaves SMs idle or does not cover every block once.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "noalloc_plan.hpp"

using namespace nbg;

namespace {

NaPlan plan;
alignas(256) unsigned char image[kNaMaxImage];

const char* check(const SystemDesc& sd, const SymCandidate& c) {
  const NaLayout& at = plan.at;
  const int bi = c.shape.bi(), bj = c.shape.bj, njt = (sd.npad + bj - 1) / bj;
  if (!(at.segs < at.tiles && at.tiles < at.partials && at.partials < at.rows &&
        at.rows + 12 * static_cast<size_t>(plan.row_values) <= (at.copy ? at.copy : at.end) &&
        at.end <= kNaScratchBytes && at.partials <= kNaMaxImage))
    return "layout";
  if (plan.bands[0].grid != c.max_grid) return "idle CTAs";
  const SymSegment* segs = reinterpret_cast<const SymSegment*>(image + at.segs);
  const SymTile* tiles = reinterpret_cast<const SymTile*>(image + at.tiles);
  std::vector<char> seen(static_cast<size_t>(njt));
  for (int b = 0; b < static_cast<int>(plan.bands.size()); ++b) {
    const SymBand& band = plan.bands[b];
    const int end = b + 1 < static_cast<int>(plan.bands.size())
                        ? plan.bands[b + 1].seg0 : static_cast<int>(plan.segs.size());
    const int count = end - band.seg0;
    std::vector<std::vector<const SymSegment*>> of(band.tile1 - band.tile0);
    std::vector<char> slot(plan.slots);
    int met = 0;
    for (int p = 0; p < band.grid; ++p)
      for (int q = p + 1; q > 0; q = segs[band.seg0 + q - 1].next) {
        if (q > count || ++met > count) return "list";
        const SymSegment& s = segs[band.seg0 + q - 1];
        if (s.itile < band.tile0 || s.itile >= band.tile1 || s.n != sd.n) return "segment";
        if (s.slot < 0 || s.slot >= plan.slots || slot[s.slot]++) return "slot";
        of[s.itile - band.tile0].push_back(&s);
      }
    if (met != count) return "list";
    for (int t = band.tile0; t < band.tile1; ++t) {
      seen.assign(njt, 0);
      const SymTile& tile = tiles[t];
      if (tile.itile != t || static_cast<int>(of[t - band.tile0].size()) != tile.nslots)
        return "i-tile";
      for (const SymSegment* s : of[t - band.tile0]) {
        if (s->row != tile.row || s->slot < tile.slot0 || s->slot >= tile.slot0 + tile.nslots)
          return "i-tile's parts";
        for (int jt = s->jt0; jt < s->jt1; ++jt)
          if (jt >= njt || seen[jt]++) return "block";
      }
      for (int jt = t * (bi / bj); jt < njt; ++jt)
        if (!seen[jt]) return "block left out";
      const int64_t first = tile.row + static_cast<int64_t>(t + 1) * bi;
      if (static_cast<int64_t>(t + 1) * bi < sd.npad &&
          (first < 0 || tile.row + sd.npad > plan.row_values))
        return "row";
    }
  }
  return nullptr;
}

}  // namespace

int main(int argc, char** argv) {
  std::vector<int> v;
  for (int k = 1; k < argc; ++k) v.push_back(std::atoi(argv[k]));
  if (v.size() != 4 * kNaCount + 4) return 2;
  const int sms = v[3 * kNaCount];
  SymCandidate c[kNaCount];
  for (int k = 0; k < kNaCount; ++k)
    c[k] = SymCandidate{{v[3 * k], v[3 * k + 1], v[3 * k + 2], 0}, kNaRates[k][0], kNaRates[k][1],
                        std::min(v[3 * kNaCount + 1 + k] * sms, kNaMaxGrid)};
  const int* range = &v[4 * kNaCount + 1];
  int plans = 0;
  for (int64_t n = range[0]; n <= range[1]; n += range[2])
    for (int copied = 0; copied < 2; ++copied, ++plans) {
      const SystemDesc sd = na_system(n, 1.f);
      const int k = na_plan(sd, c, sms, copied, plan, image);
      const char* wrong = k < 0 ? "refused" : check(sd, c[k]);
      if (wrong) {
        std::printf("%d particles%s: %s\n", sd.n, copied ? ", one buffer" : "", wrong);
        return 1;
      }
    }
  std::printf("%d plans\n", plans);
  return 0;
}
