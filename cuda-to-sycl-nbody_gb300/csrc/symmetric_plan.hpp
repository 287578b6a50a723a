// The planner behind symmetric.hpp, writing to tables that grow (plan_symmetric) or to
// fixed ones (nb_accelerations_noalloc) by one rule.
//
// Plan has the members of SymPlanHost; its tables provide the std::vector operations
// used here, and fixed ones drop what does not fit (their owner checks).
#pragma once

#include <algorithm>
#include <cstdint>

#include "symmetric.hpp"

namespace nbg {

// Charges of one i-tile's units: the j-tiles from t0 (diagonal) over td (behind the
// i-tile) to t1, each bj particles of the diagonal or the pair cost.
struct SymTileCharge {
  int32_t t0, td, t1;
  int64_t diag, pair;
  int64_t upto(int32_t t) const {
    const int64_t d = std::min(t, td) - t0, p = std::max(0, t - td);
    return d * diag + p * pair;
  }
  // Smallest t in [t0, t1] with upto(t) >= c.
  int32_t reach(int64_t c) const {
    if (c <= 0) return t0;
    const int64_t whole = upto(td);
    const int64_t t = c <= whole ? t0 + (c + diag - 1) / diag
                                 : td + (c - whole + pair - 1) / pair;
    return static_cast<int32_t>(std::min<int64_t>(t, t1));
  }
};

template <class Plan>
void plan_symmetric_into(const SystemDesc* sys, int32_t first, int32_t count, int32_t bi,
                         int32_t bj, int32_t max_grid, int64_t max_row_values,
                         int64_t max_band_tiles, int diag_cost, int pair_cost, Plan& plan) {
  // The i-tiles, their rows and the bands they fall into.
  plan.sys_tile0.assign(first + count + 1, 0);
  int64_t values = 0;
  for (int32_t s = first; s < first + count; ++s) {
    plan.sys_tile0[s] = static_cast<int32_t>(plan.tiles.size());
    const int32_t nit = (sys[s].n + bi - 1) / bi;
    for (int32_t it = 0; it < nit; ++it) {
      const int32_t t = static_cast<int32_t>(plan.tiles.size());
      const int64_t behind = static_cast<int64_t>(it + 1) * bi;
      const int64_t len = std::max<int64_t>(0, sys[s].npad - behind);
      if (plan.bands.empty() || values + len > max_row_values ||
          t - plan.bands.back().tile0 >= max_band_tiles) {
        SymBand b;
        b.tile0 = t;
        plan.bands.push_back(b);
        values = 0;
      }
      plan.tiles.push_back(SymTile{values - behind, sys[s].offset, sys[s].n, s, it, 0, 0, 0});
      values += len;
      plan.row_values = std::max(plan.row_values, values);
      plan.bands.back().tile1 = t + 1;
    }
  }
  plan.sys_tile0[first + count] = static_cast<int32_t>(plan.tiles.size());

  auto charge_of = [&](const SymTile& t) {
    const SystemDesc& d = sys[t.sys];
    SymTileCharge c;
    c.t0 = t.itile * (bi / bj);
    c.t1 = (d.npad + bj - 1) / bj;
    c.td = std::min(c.t1, c.t0 + bi / bj);
    c.diag = static_cast<int64_t>(bj) * diag_cost;
    c.pair = static_cast<int64_t>(bj) * pair_cost;
    return c;
  };
  for (SymBand& b : plan.bands) {
    b.end = plan.sys_tile0[plan.tiles[b.tile1 - 1].sys + 1];
    int64_t total = 0, units = 0;
    for (int32_t t = b.tile0; t < b.tile1; ++t) {
      const SymTileCharge c = charge_of(plan.tiles[t]);
      total += c.upto(c.t1);
      units += c.t1 - c.t0;
    }
    b.grid = static_cast<int32_t>(std::max<int64_t>(1, std::min<int64_t>(max_grid, units)));
    b.begin0 = static_cast<int32_t>(plan.seg_begin.size());
    // CTA k takes the units whose starting charge is in [k, k + 1) * total / grid: `bound`
    // is (k + 1) * total / grid rounded up, kept as quotient and remainder, as a division
    // per segment (two, of 128 bits) took most of the planning.
    const int64_t share = total / b.grid, rest = total % b.grid;
    int64_t k = 0, quot = share, rem = rest;
    int64_t bound = quot + (rem > 0);
    auto next_bound = [&] {
      ++k;
      quot += share;
      rem += rest;
      if (rem >= b.grid) rem -= b.grid, ++quot;
      bound = quot + (rem > 0);
    };
    int64_t c0 = 0;
    int32_t next_cta = 0, slot = 0;
    b.seg0 = static_cast<int32_t>(plan.segs.size());
    for (int32_t t = b.tile0; t < b.tile1; ++t) {
      SymTile& tile = plan.tiles[t];
      const SymTileCharge c = charge_of(tile);
      tile.slot0 = slot;
      int32_t jt = c.t0;
      while (jt < c.t1) {
        const int64_t at = c0 + c.upto(jt);
        while (k + 1 < b.grid && at >= bound) next_bound();
        int32_t end = c.t1;
        if (k + 1 < b.grid) end = std::max(jt + 1, c.reach(bound - c0));
        while (next_cta <= k) {
          plan.seg_begin.push_back(static_cast<int32_t>(plan.segs.size()));
          ++next_cta;
        }
        plan.segs.push_back(SymSegment{tile.sys, tile.itile, jt, end, tile.row,
                                       sys[tile.sys].offset, sys[tile.sys].n, slot++, -1, 0});
        jt = end;
      }
      tile.nslots = slot - tile.slot0;
      if (tile.nslots > 1) ++plan.split_tiles;
      c0 += c.upto(c.t1);
    }
    while (next_cta <= b.grid) {
      plan.seg_begin.push_back(static_cast<int32_t>(plan.segs.size()));
      ++next_cta;
    }
    // A CTA whose share holds no unit's start (a unit can charge more than a share)
    // drops out.
    const auto begin = plan.seg_begin.begin() + b.begin0;
    plan.seg_begin.erase(std::unique(begin, plan.seg_begin.end()), plan.seg_begin.end());
    b.grid = static_cast<int32_t>(plan.seg_begin.size()) - b.begin0 - 1;
    plan.slots = std::max(plan.slots, static_cast<int32_t>(plan.segs.size()) - b.seg0);
  }
}

// Largest grid that link_segments_into orders (it sorts on the stack).
constexpr int32_t kSymMaxOrdered = 8192;

// `order` receives the indices of `charge` (n of them), the lightest first and of equal
// ones the last first.  Charges are the same to within a unit or two, so they are counted
// where their range allows (1,216 of them: 4 us, 31 with std::sort).
inline void order_by_charge(const uint32_t* charge, int32_t n, int32_t* order) {
  constexpr uint32_t kBins = 2048;
  uint32_t lo = charge[0], hi = charge[0];
  for (int32_t k = 1; k < n; ++k) {
    lo = std::min(lo, charge[k]);
    hi = std::max(hi, charge[k]);
  }
  if (hi - lo < kBins) {
    int32_t at[kBins + 1] = {};
    for (int32_t k = 0; k < n; ++k) ++at[charge[k] - lo + 1];
    for (uint32_t c = 0; c <= hi - lo; ++c) at[c + 1] += at[c];
    for (int32_t k = n - 1; k >= 0; --k) order[at[charge[k] - lo]++] = k;
    return;
  }
  for (int32_t k = 0; k < n; ++k) order[k] = k;
  std::sort(order, order + n, [charge](int32_t a, int32_t b) {
    return charge[a] != charge[b] ? charge[a] < charge[b] : a > b;
  });
}

// `out` holds plan.segs.size() segments.  The rest as link_segments.
template <class Plan, class Out>
void link_segments_into(const Plan& plan, int32_t tiles_per_i, int32_t schedulers, int diag_cost,
                        int pair_cost, Out& out) {
  uint32_t charge[kSymMaxOrdered];
  int32_t order[kSymMaxOrdered];
  for (const SymBand& b : plan.bands) {
    const auto first = plan.seg_begin.begin() + b.begin0;
    const bool ordered = schedulers > 0 && b.grid > schedulers && b.grid <= kSymMaxOrdered;
    for (int32_t k = 0; ordered && k < b.grid; ++k) {
      uint64_t sum = 0;
      for (int32_t q = first[k]; q < first[k + 1]; ++q) {
        const SymSegment& sg = plan.segs[q];
        const int32_t td = std::max(sg.jt0, std::min(sg.jt1, (sg.itile + 1) * tiles_per_i));
        sum += static_cast<uint64_t>(td - sg.jt0) * diag_cost +
               static_cast<uint64_t>(sg.jt1 - td) * pair_cost + pair_cost / 5;
      }
      charge[k] = static_cast<uint32_t>(std::min<uint64_t>(sum, UINT32_MAX));
    }
    if (ordered) order_by_charge(charge, b.grid, order);
    int32_t more = b.grid;  // the next free place behind the first segments
    for (int32_t p = 0; p < b.grid; ++p) {
      int32_t k = p;
      if (ordered) {
        // Heaviest round first, its heaviest CTA last; every other round the other way about.
        const int32_t round = p / schedulers, p0 = round * schedulers;
        const int32_t len = std::min(schedulers, b.grid - p0);
        const int32_t rank = round % 2 == 1 ? p : p0 + len - 1 - (p - p0);
        k = order[b.grid - 1 - rank];
      }
      int32_t at = p;
      for (int32_t q = first[k]; q < first[k + 1]; ++q) {
        SymSegment sg = plan.segs[q];
        const bool last = q + 1 == first[k + 1];
        sg.next = last ? 0 : ++more;
        out[b.seg0 + at] = sg;
        at = sg.next - 1;
      }
    }
  }
}

}  // namespace nbg
