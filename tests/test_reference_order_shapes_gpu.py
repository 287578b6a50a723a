"""Every shape of the reference-order kernel (csrc/reference_order_kernel.cu) gives the
same words: each particle's sum is one sequence of roundings whatever the tiling.  Shape
0 (two i-particles per packed register pair) is pinned to the reference kernel by the
golden fixtures; here the j-pair shape, its masked and remaining loops and its grids
(one CTA per i-tile, and shared i-tiles) are compared with it, BRANCH and PREDICATED."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

pytestmark = pytest.mark.gpu


def words(sim, pos, vel, steps):
    sim.set_state(pos, vel)
    sim.advance(steps)
    return [a.view(np.uint32) for a in sim.get_state()]


# 128-particle i-tiles and 512-particle j-tiles, 64 j-particles per pipelined round:
# edges of each, odd sizes, sizes whose i-tiles share 152 or 304 CTAs.
@pytest.mark.parametrize("n", [1, 2, 31, 33, 63, 64, 65, 127, 128, 129, 191, 511, 512, 513, 640,
                               1025, 4099, 19457, 22001, 45001])
@pytest.mark.parametrize("method,eps", [(nb.BRANCH, 1e-3), (nb.BRANCH, 0.0), (nb.PREDICATED, 1e-3)])
def test_shapes_give_the_same_words(n, method, eps):
    pos, vel, _ = disk_case(n, seed=n)
    steps = 2 if n < 10000 else 1
    p = params(n, eps=eps, method=method, acc=nb.ACC_REFERENCE_ORDER)
    with nb.Simulation(p, pos, vel, None) as sim:
        default = words(sim, pos, vel, steps)
        sim.set_kernel_config(0)
        want = words(sim, pos, vel, steps)
        sim.set_kernel_config(3)
        got = words(sim, pos, vel, steps)
    for d, g, w in zip(default, got, want):
        assert np.array_equal(g, w) and np.array_equal(d, w)


def test_ensemble_and_coincident_particles_give_the_same_words():
    sizes = [1, 513, 64, 2000, 130]
    parts = [disk_case(s, seed=s) for s in sizes]
    pos, vel = ([np.concatenate([p[q][c] for p in parts]) for c in range(3)] for q in (0, 1))
    for a in pos:
        a[700] = a[600]                     # NaN in both without softening
    p = params(sum(sizes), eps=0.0, acc=nb.ACC_REFERENCE_ORDER)
    out = []
    for shape in (0, 3):
        with nb.Simulation(p, pos, vel, None, sizes=sizes) as sim:
            sim.set_kernel_config(shape)
            out.append(words(sim, pos, vel, 1))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
