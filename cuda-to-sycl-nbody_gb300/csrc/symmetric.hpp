// Work lists of the symmetric force kernel (symmetric_kernel.cuh) and their planner.
//
// The unit of work is one (system, i-tile, j-tile) block on or above the diagonal: an
// i-tile I of bi particles meets the j-tiles from its own first particle to the end of
// its system, so every unordered pair of particles in different i-tiles is in exactly
// one block.  The j-tiles inside the i-tile (the diagonal block) are summed for the i
// side only, over all ordered pairs; the others for both sides.
//
// Units are laid out in (system, i-tile, j-tile) order and charged their particles
// times the pair loop's lane operations (kSymDiagCost, kSymPairCost), and cut into one
// contiguous run per CTA of the same charge to within one unit, as in worklist.hpp.
//
// The j-side sums of i-tile I are one row of scratch, a value per component and
// particle behind the tile; the rows of a system of n particles take about n^2 / (2 bi)
// values.  Where all rows together pass the scratch's bound, the i-tiles are cut into
// bands that are run (and their rows added up) one after another in the same scratch.
#pragma once

#include <cstdint>
#include <vector>

#include "nb_internal.hpp"

namespace nbg {

// Lane operations per pair on the FMA pipe (symmetric_kernel.cuh): one side, both sides.
constexpr int kSymDiagCost = 11;
constexpr int kSymPairCost = 14;
// The same of the adjoint (adjoint_kernel.cu).
constexpr int kAdjDiagCost = 22;
constexpr int kAdjPairCost = 25;
constexpr int64_t kSymRowBytes = 3 * sizeof(float);  // scratch per row value
constexpr int64_t kSymScratchBytes = int64_t{1} << 28;

// One entry of a CTA's list: i-tile `itile` of system `sys` against j-tiles [jt0, jt1).
// The j-side sum of particle j goes to value row + j of each plane of the row scratch,
// the i-side sums to slot `slot` of the partial sums.
struct SymSegment {
  int32_t sys;
  int32_t itile;
  int32_t jt0;
  int32_t jt1;
  int64_t row;
  int64_t offset;  // first particle of the system, and its particles
  int32_t n;
  int32_t slot;
  int32_t next;    // 1 + the CTA's next segment, 0 for none; CTA k starts with segment k
  int32_t pad_;
};

// One i-tile: its row, and its first slot (its slots run to the next i-tile's first).
struct SymTile {
  int64_t row;
  int64_t offset;  // first particle of the system, and its particles
  int32_t n;
  int32_t sys;
  int32_t itile;
  int32_t slot0;
  int32_t nslots;
  int32_t pad_;
};

// A band of i-tiles [tile0, tile1): its work list and what the adding pass covers.
struct SymBand {
  int32_t tile0 = 0, tile1 = 0;
  int32_t end = 0;       // one past the last i-tile of the last system it touches
  int32_t grid = 0;
  int32_t begin0 = 0;    // first of its grid + 1 entries of seg_begin
  int32_t seg0 = 0;      // its first segment
};

struct SymPlanHost {
  std::vector<SymSegment> segs;
  std::vector<int32_t> seg_begin;
  std::vector<SymTile> tiles;
  std::vector<int32_t> sys_tile0;  // first i-tile of each planned system, by its index
  std::vector<SymBand> bands;
  int64_t row_values = 0;          // largest band's row values (per plane)
  int32_t slots = 0;               // largest band's slots
  int32_t split_tiles = 0;
};

// Rows and parts per particle of the first band, on average.
template <class Plan>
float terms_per_particle(const Plan& plan, int bi) {
  const double particles = static_cast<double>(plan.bands[0].tile1 - plan.bands[0].tile0) * bi;
  return static_cast<float>(
      (static_cast<double>(plan.row_values) + static_cast<double>(plan.slots) * bi) / particles);
}

// The segments in the order the kernel wants them: per band, the first of every CTA and
// then the others, linked by `next` (counted from the band's seg0).
//
// `schedulers` > 0: CTAs of one warp, more of them than the GPU's warp schedulers.  CTA b
// then shares its scheduler with b + schedulers and so on (to within a few places, as
// the clocks at which the warps end show), and of the two the older runs at nearly its
// full rate, so what counts is the charge per scheduler.  Its units are coarse (N =
// 8,192: 3 or 4 per CTA, 6.8 per scheduler), so the CTAs are given out by charge,
// heaviest round first and every other round the other way about (us per step, in list
// order / by charge: 8,192 25.4 / 23.8, 12,800 50.5 / 47.9, 20,000 107.5 / 103.4; the
// adjoint at 16,384 133 / 127; 25,600, where 34 units meet 33.2 on average, 163 either
// way; measured before the sums' chains were shortened).  `tiles_per_i`: j-tiles per i-tile.
std::vector<SymSegment> link_segments(const SymPlanHost& plan, int32_t tiles_per_i,
                                      int32_t schedulers, int diag_cost = kSymDiagCost,
                                      int pair_cost = kSymPairCost);

// Plan systems [first, first + count) (whole systems, no shards) for i-tiles of bi and
// j-tiles of bj particles (bi % bj == 0) on at most max_grid CTAs, with at most
// max_row_values row values per band (one i-tile at least); diag_cost and pair_cost: the
// charges per particle of a diagonal and of another j-tile.
SymPlanHost plan_symmetric(const SystemDesc* sys, int32_t first, int32_t count, int32_t bi,
                           int32_t bj, int32_t max_grid, int64_t max_row_values,
                           int diag_cost = kSymDiagCost, int pair_cost = kSymPairCost);

// A shape to choose from: its relative rate where it is balanced, the blocks per CTA
// from which it is, and its largest grid.
struct SymCandidate {
  KernelShape shape;
  double rate;
  double blocks_per_cta;
  int max_grid;
};

// Index of the best of `count_c` shapes for systems [first, first + count): the lowest
// charge over rate among those with enough blocks per CTA (the last always counts).
// Larger i-tiles run their pairs at a higher rate but leave more of them on the diagonal
// and in a system's last tile, and make fewer blocks to balance.
int choose_symmetric(const SystemDesc* sys, int32_t first, int32_t count, const SymCandidate* c,
                     int count_c, int diag_cost, int pair_cost);

}  // namespace nbg
