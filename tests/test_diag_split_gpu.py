"""The potential's pair kernels (csrc/diag_kernels.cu): terms as sums of two floats for
large systems, FP64 for small ones, tiny softenings and values out of the split's range.
Against FP64 terms added exactly (math.fsum), on the host.

Tolerance: a term's error is below 1e-14 either way, and sums over at least 4,000 x
4,000 / 2 pairs average it out; 2e-15 also covers the blocks' partial sums."""
from __future__ import annotations

import math

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

pytestmark = pytest.mark.gpu


def exact_potential(pos, m, eps):
    x = [a.astype(np.float64) for a in pos]
    mm = m.astype(np.float64)
    rows = []
    for i in range(len(mm) - 1):
        d2 = sum((a[i + 1:] - a[i]) ** 2 for a in x) + float(np.float32(eps))
        with np.errstate(divide="ignore"):
            rows.append(mm[i] * math.fsum(mm[i + 1:] / np.sqrt(d2)))
    return -math.fsum(rows)


def potential(pos, vel, m, eps):
    with nb.Simulation(params(len(m), eps=eps), pos, vel, m) as sim:
        return sim.diagnostics()["potential"]


# 4,096 is the first size of the split kernel; 256 its tile.
@pytest.mark.parametrize("n", [4095, 4096, 4097, 4351, 4353, 6000])
@pytest.mark.parametrize("mass", ["equal", "random", "with_zeros"])
def test_potential_matches_exact_sum(n, mass):
    pos, vel, m = disk_case(n, seed=n)
    if mass != "equal":
        m = (m * np.random.default_rng(n).uniform(0.5, 1.5, n)).astype(np.float32)
    if mass == "with_zeros":
        m[::7] = 0.0
    want = exact_potential(pos, m, 1e-3)
    assert abs(potential(pos, vel, m, 1e-3) - want) <= 2e-15 * abs(want)


@pytest.mark.parametrize("change", ["tiny_softening", "far", "heavy", "clustered"])
def test_potential_out_of_the_split_range(change):
    n, eps = 4200, 1e-3
    pos, vel, m = disk_case(n, seed=3)
    if change == "tiny_softening":
        eps = 1e-14
    elif change == "far":                       # squares overflow FP32
        pos = [(a * np.float32(1e21)).astype(np.float32) for a in pos]
    elif change == "heavy":
        m = (np.random.default_rng(1).uniform(1e29, 2e30, n)).astype(np.float32)
    else:                                       # differences far below the coordinates
        pos = [(a * np.float32(1e-4) + np.float32(900.0)).astype(np.float32) for a in pos]
    want = exact_potential(pos, m, eps)
    assert abs(potential(pos, vel, m, eps) - want) <= 2e-15 * abs(want)


def test_coincident_particles_without_softening():
    pos, vel, m = disk_case(4200, seed=4)
    for a in pos:
        a[4000] = a[17]
    assert potential(pos, vel, m, 0.0) == -math.inf


def test_ensemble_mixes_both_kernels():
    sizes = [1, 5000, 300, 4096]
    parts = [disk_case(s, seed=90 + k) for k, s in enumerate(sizes)]
    pos, vel = ([np.concatenate([p[q][c] for p in parts]) for c in range(3)] for q in (0, 1))
    m = np.concatenate([p[2] for p in parts])
    with nb.Simulation(params(sum(sizes)), pos, vel, m, sizes=sizes) as sim:
        per = [sim.diagnostics(k)["potential"] for k in range(len(sizes))]
        total = sim.diagnostics(-1)["potential"]
        again = sim.diagnostics(1)["potential"]
    for got, (p, _, ms) in zip(per, parts):
        want = exact_potential(p, ms, 1e-3)
        assert abs(got - want) <= 2e-15 * abs(want)
    assert abs(total - math.fsum(per)) <= 2e-15 * abs(total) and again == per[1]
