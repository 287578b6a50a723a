"""The potential where few distinct distances dominate, so that the rounding errors of its
terms repeat instead of averaging out: the particles of two points, listed alternately.
The exact value has a closed form (three distinct terms).

Tolerance: terms as exact as FP64's leave the sums' own rounding.  The terms of a row have
one sign, and a partial sum of the k-th of 32 parts (128 terms each) is rounded by at most
2^-53 of k / 32 of the row: 16.5 2^-53 = 1.8e-15 in all, with the trees behind it 2e-15."""
from __future__ import annotations

from fractions import Fraction
from math import isqrt

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import params

pytestmark = pytest.mark.gpu

N = 4096  # the first size of the split kernel


def inverse_root(d2: Fraction) -> Fraction:
    """1 / sqrt(d2) to 60 digits."""
    scale = 10 ** 60
    return Fraction(isqrt(d2.denominator * scale ** 2 // d2.numerator), scale)


def two_points(a, b, ma, mb, eps):
    pos = [np.where(np.arange(N) % 2 == 0, a[c], b[c]).astype(np.float32) for c in range(3)]
    m = np.where(np.arange(N) % 2 == 0, ma, mb).astype(np.float32)
    e = Fraction(float(np.float32(eps)))
    d2 = sum((Fraction(float(p)) - Fraction(float(q))) ** 2 for p, q in zip(a, b)) + e
    h = N // 2
    fa, fb = Fraction(float(np.float32(ma))), Fraction(float(np.float32(mb)))
    want = -((fa * fa + fb * fb) * (h * (h - 1) // 2) * inverse_root(e)
             + fa * fb * h * h * inverse_root(d2))
    return pos, m, want


@pytest.mark.parametrize("masses", ["equal", "own"])
def test_two_points_listed_alternately(masses):
    rng = np.random.default_rng(5)
    vel = [np.zeros(N, np.float32)] * 3
    worst = 0.0
    for _ in range(96):
        a, b = rng.uniform(-3.0, 3.0, (2, 3)).astype(np.float32)
        eps = float(np.exp(rng.uniform(np.log(0.1), np.log(2.0))))
        ma, mb = (1.0, 1.0) if masses == "equal" else rng.uniform(0.5, 1.5, 2)
        pos, m, want = two_points(a, b, ma, mb, eps)
        with nb.Simulation(params(N, eps=eps), pos, vel, m) as sim:
            got = sim.diagnostics()["potential"]
        worst = max(worst, float(abs(Fraction(got) - want) / abs(want)))
    assert worst <= 2e-15, worst
