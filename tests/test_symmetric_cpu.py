"""Work lists of the symmetric force kernel (csrc/symmetric.hpp), planned on the host."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb


def symmetric_configs():
    """The symmetric shapes: the configs without a tile ring."""
    return [c for c in range(nb.num_kernel_configs()) if nb.kernel_config_info(c)["stages"] == 0]


@pytest.mark.parametrize("cfg", symmetric_configs())
@pytest.mark.parametrize("sizes,grid", [
    ([1], 152), ([17], 8), ([512], 152), ([513], 152), ([4096], 152), ([4097], 152),
    ([25600], 304), ([70001], 1216), ([262144], 152),
    ([64, 100, 8192, 3, 700, 4097], 300), ([1000] * 50, 1216), ([300000], 1)])
def test_every_pair_of_particles_is_in_exactly_one_block(cfg, sizes, grid):
    # Each i-tile meets the j-tiles from its own first particle to the end of its
    # system once; CTAs get one contiguous run each, balanced to within one block.
    info = nb.kernel_config_info(cfg)
    bi, bj = info["threads_per_block"] * info["particles_per_thread"], info["j_tile"]
    assert bi % bj == 0
    g, segs, begin, nfix, slots = nb.plan_work(sizes, cfg, grid)
    assert 1 <= g <= grid and slots == len(segs)
    assert begin[0] == 0 and begin[-1] == len(segs) and np.all(np.diff(begin) >= 0)
    npad = [(n + 15) // 16 * 16 for n in sizes]
    seen, parts = {}, {}
    cost = np.zeros(g)
    for c in range(g):
        for s, it, j0, j1, fix, part in segs[begin[c]:begin[c + 1]]:
            assert j0 < j1
            assert j0 == seen.get((s, it), it * bi // bj)      # runs join in j order
            seen[s, it] = j1
            parts.setdefault((s, it), []).append(part)
            diag = min(j1, (it + 1) * bi // bj) - min(j0, (it + 1) * bi // bj)
            cost[c] += bj * (11 * diag + 14 * (j1 - j0 - diag))
    for s, n in enumerate(sizes):
        for it in range((n + bi - 1) // bi):
            assert seen.pop((s, it)) == (npad[s] + bj - 1) // bj
            assert parts[s, it] == list(range(len(parts[s, it])))
    assert not seen
    assert nfix == sum(len(p) > 1 for p in parts.values())
    assert cost.max() - cost.min() <= 2 * 14 * bj or g == 1
