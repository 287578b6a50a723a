// The work list of nb_accelerations_noalloc (noalloc.cu): planned into tables of fixed size
// and laid out in its fixed scratch, without an allocation.  Host code only.
//
// A caller whose particle count changes plans in every call, while the GPU waits, so a plan
// is made once: how many i-tiles a band may have, and on how many CTAs, follows from
// bounds on what the plan will take.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "symmetric_plan.hpp"

namespace nbg {

constexpr int64_t kNaMaxParticles = 1 << 18;  // 262,144
// What the largest plans take on a full grid: 262,144 particles in one buffer for input and
// output, 10 MB of parts (152 CTAs), 3.1 MB for an i-tile's row, 4.2 MB for the copy of the
// positions, 0.5 MB for the list.  13 MiB left them 83 CTAs (us per call: 30,900 and 18,930
// now; one i-tile per band either way), and put 20,000 particles into two bands (131 / 126).
constexpr size_t kNaScratchBytes = 18u << 20;

// Bounds: at most 64 i-tiles of 4,096 particles, each a band of its own on up to 152
// CTAs; the smaller shapes are chosen for at most about 128 i-tiles, in a few bands on
// at most kNaMaxGrid CTAs.  A plan that passes them is refused for the next shape.
constexpr int kNaMaxGrid = 2432;
constexpr int kNaMaxTiles = 512;
constexpr int kNaMaxSegments = 10240;
constexpr int kNaMaxBands = 64;

// Candidate shapes by index of the symmetric kernel (i-tiles of 4,096, 256 and 64
// particles), largest first, and choose_symmetric's rates for them.  512-particle
// i-tiles would need 10 MB for the parts and as much for the rows at their sizes.
constexpr int kNaShapes[] = {0, 2, 3};
constexpr double kNaRates[][2] = {{1.0, 6.0}, {0.86, 0.8}, {0.617, 0.0}};
constexpr int kNaCount = 3;

// A table of fixed size with the vector operations the planner uses; what does not fit
// is dropped and remembered.
template <class T, int N>
struct FixedTable {
  T data[N];
  int n = 0;
  bool full = false;
  void push_back(const T& v) {
    if (n < N)
      data[n++] = v;
    else
      full = true;
  }
  void clear() {
    n = 0;
    full = false;
  }
  void assign(size_t count, const T& v) {
    clear();
    for (size_t k = 0; k < count; ++k) push_back(v);
  }
  void erase(T* from, T* to) {
    (void)to;  // the planner erases the tail
    n = static_cast<int>(from - data);
  }
  size_t size() const { return n; }
  bool empty() const { return n == 0; }
  T& operator[](size_t i) { return data[i]; }
  const T& operator[](size_t i) const { return data[i]; }
  T& back() { return data[n - 1]; }
  T* begin() { return data; }
  T* end() { return data + n; }
  const T* begin() const { return data; }
  const T* end() const { return data + n; }
};

// Where the parts lie in the scratch: the system record, the segments and the i-tiles (up
// to `partials` the image that is uploaded), the partial sums, the rows, and a copy of the
// caller's positions (0 where they are read in place).
struct NaLayout {
  size_t sys = 0, segs = 256, tiles = 0, partials = 0, rows = 0, copy = 0, end = 0;
};

constexpr size_t na_align(size_t x) { return (x + 255) / 256 * 256; }

inline NaLayout na_layout(int64_t segs, int64_t tiles, int64_t slots, int64_t row_values, int bi,
                          size_t copy) {
  NaLayout at;
  at.tiles = na_align(at.segs + segs * sizeof(SymSegment));
  at.partials = na_align(at.tiles + tiles * sizeof(SymTile));
  at.rows = na_align(at.partials + slots * static_cast<size_t>(bi) * 4 * sizeof(float));
  const size_t end = na_align(at.rows + 3 * sizeof(float) * static_cast<size_t>(row_values));
  at.copy = copy ? end : 0;
  at.end = end + copy;
  return at;
}

constexpr size_t kNaMaxImage = 256 + na_align(kNaMaxSegments * sizeof(SymSegment)) +
                               na_align(kNaMaxTiles * sizeof(SymTile));

struct NaPlan {
  FixedTable<SymSegment, kNaMaxSegments> segs;
  FixedTable<int32_t, kNaMaxSegments + kNaMaxBands + 1> seg_begin;
  FixedTable<SymTile, kNaMaxTiles> tiles;
  FixedTable<int32_t, 2> sys_tile0;
  FixedTable<SymBand, kNaMaxBands> bands;
  int64_t row_values = 0;
  int32_t slots = 0;
  int32_t split_tiles = 0;
  NaLayout at;
  void clear() {
    segs.clear();
    seg_begin.clear();
    tiles.clear();
    sys_tile0.clear();
    bands.clear();
    row_values = 0;
    slots = split_tiles = 0;
    at = NaLayout{};
  }
  bool fits() const {
    return !segs.full && !seg_begin.full && !tiles.full && !bands.full &&
           at.end <= kNaScratchBytes;
  }
};

inline SystemDesc na_system(uint64_t n, float G) {
  SystemDesc sd{};
  sd.n = static_cast<int32_t>(n);
  sd.npad = (sd.n + kPadQuantum - 1) / kPadQuantum * kPadQuantum;
  sd.gscale = G;  // per-pair masses: each pair term carries m_j
  return sd;
}

// Whether bands of `per` i-tiles on `grid` CTAs fit the tables and the scratch, by upper
// bounds: a band's segments are at most its CTAs and its i-tiles less one, and at most its
// (i-tile, j-tile) blocks.
inline bool na_fits(const SystemDesc& sd, const KernelShape& sh, int64_t tiles, int64_t per,
                    int64_t grid, size_t copy) {
  const int64_t bi = sh.bi(), jper = bi / sh.bj, njt = (sd.npad + sh.bj - 1) / sh.bj;
  if (tiles > kNaMaxTiles || (tiles + per - 1) / per > kNaMaxBands) return false;
  int64_t segs = 0, slots = 0;
  for (int64_t t = 0; t < tiles; t += per) {
    const int64_t count = std::min(per, tiles - t);
    const int64_t units = count * njt - jper * (t * count + count * (count - 1) / 2);
    const int64_t most = std::min(units, std::min(units, grid) + count - 1);
    segs += most;
    slots = std::max(slots, most);
  }
  if (segs > kNaMaxSegments) return false;
  int64_t rows = 0;  // of the first band, the longest
  for (int64_t t = 0; t < std::min(per, tiles); ++t)
    rows += std::max<int64_t>(0, sd.npad - (t + 1) * bi);
  return na_layout(segs, tiles, slots, rows, sh.bi(), copy).end <= kNaScratchBytes;
}

// Plan the system for shape `c`: as large bands as fit, on the shape's full grid, or on a
// smaller one where even one i-tile's row and parts are too much.  False if none fits.
inline bool na_plan_shape(const SystemDesc& sd, const SymCandidate& c, int sms, size_t copy,
                          NaPlan& plan, unsigned char* image) {
  const KernelShape& sh = c.shape;
  const int64_t tiles = (sd.n + sh.bi() - 1) / sh.bi();
  int64_t per = tiles, grid = c.max_grid;
  while (!na_fits(sd, sh, tiles, per, grid, copy)) {
    if (per > 1)
      per = (per + 1) / 2;
    else if ((grid -= 8) < 1)
      return false;
  }
  const int64_t longest = std::max<int64_t>(0, sd.npad - sh.bi());  // values of the first row
  plan.clear();
  plan_symmetric_into(&sd, 0, 1, sh.bi(), sh.bj, static_cast<int32_t>(grid),
                      std::max<int64_t>(1, per * longest), per, kSymDiagCost, kSymPairCost, plan);
  plan.at = na_layout(plan.segs.size(), plan.tiles.size(), plan.slots, plan.row_values, sh.bi(),
                      copy);
  if (!plan.fits()) return false;
  std::memcpy(image + plan.at.sys, &sd, sizeof(sd));
  std::memcpy(image + plan.at.tiles, plan.tiles.data, plan.tiles.size() * sizeof(SymTile));
  SymSegment* linked = reinterpret_cast<SymSegment*>(image + plan.at.segs);
  link_segments_into(plan, sh.bi() / sh.bj, sh.threads == 32 ? 4 * sms : 0, kSymDiagCost,
                     kSymPairCost, linked);
  return true;
}

// Plan the system for the best of the kNaCount candidates, or, where that does not fit, for the
// first; `copied`: with room for a copy of the positions.  The index of the candidate, -1
// if neither fits.  `image` (kNaMaxImage bytes) receives what goes to the scratch.
inline int na_plan(const SystemDesc& sd, const SymCandidate* c, int sms, bool copied, NaPlan& plan,
                   unsigned char* image) {
  const size_t copy = copied ? static_cast<size_t>(sd.n) * 16 : 0;
  const int k = choose_symmetric(&sd, 0, 1, c, kNaCount, kSymDiagCost, kSymPairCost);
  if (na_plan_shape(sd, c[k], sms, copy, plan, image)) return k;
  return na_plan_shape(sd, c[0], sms, copy, plan, image) ? 0 : -1;
}

}  // namespace nbg
