// Work-list planner of the symmetric force kernel (the rule is in symmetric.hpp).
#include "symmetric_plan.hpp"

#include <algorithm>
#include <cfloat>

namespace nbg {

int choose_symmetric(const SystemDesc* sys, int32_t first, int32_t count, const SymCandidate* c,
                     int count_c, int diag_cost, int pair_cost) {
  int best = count_c - 1;
  double best_time = DBL_MAX;
  for (int k = 0; k < count_c; ++k) {
    const KernelShape& sh = c[k].shape;
    double charge = 0, blocks = 0;
    for (int32_t q = first; q < first + count; ++q) {
      const double npad = sys[q].npad, bi = sh.bi();
      const double tiles = (sys[q].n + sh.bi() - 1) / sh.bi();
      const double last = npad - (tiles - 1) * bi;  // columns of the last i-tile
      const double cols = tiles * npad - bi * tiles * (tiles - 1) / 2;
      const double diag = (tiles - 1) * bi + last;
      charge += bi * (diag_cost * diag + pair_cost * (cols - diag));
      blocks += cols / sh.bj;
    }
    const double time = charge / c[k].rate;
    if (time < best_time &&
        (k + 1 == count_c || blocks >= c[k].blocks_per_cta * c[k].max_grid)) {
      best = k;
      best_time = time;
    }
  }
  return best;
}

SymPlanHost plan_symmetric(const SystemDesc* sys, int32_t first, int32_t count, int32_t bi,
                           int32_t bj, int32_t max_grid, int64_t max_row_values, int diag_cost,
                           int pair_cost) {
  SymPlanHost plan;
  plan_symmetric_into(sys, first, count, bi, bj, max_grid, max_row_values, INT64_MAX, diag_cost,
                      pair_cost, plan);
  return plan;
}

std::vector<SymSegment> link_segments(const SymPlanHost& plan, int32_t tiles_per_i,
                                      int32_t schedulers, int diag_cost, int pair_cost) {
  std::vector<SymSegment> out(plan.segs.size());
  link_segments_into(plan, tiles_per_i, schedulers, diag_cost, pair_cost, out);
  return out;
}

}  // namespace nbg
