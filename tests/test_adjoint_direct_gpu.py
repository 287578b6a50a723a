"""The adjoint's direct kernel (csrc/adjoint_kernel.cu) for small systems at the edges of
its i-tiles and passes and where its shapes change, and the pair kernel just above the
line between them, against FP64 torch autograd (test_adjoint_symmetric_gpu.py, whose
bound this takes over)."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params
from test_adjoint_symmetric_gpu import DAMP, DT, check, reference

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 7, 9, 15, 17, 255, 257, 511, 512, 513, 1025, 2431, 2434, 2549,
                               2550, 2561, 2593])
@pytest.mark.parametrize("mass,eps", [("equal", 1e-3), ("random", 1e-3), ("random", 0.0)])
def test_gradients_at_edges(n, mass, eps):
    pos, vel, m = disk_case(n, seed=n)
    rng = np.random.default_rng(n)
    if eps == 0.0:  # apart from each other: no softening bounds the force
        pos = [(8 * rng.permutation(n) + rng.uniform(0, 1, n)).astype(np.float32) for _ in range(3)]
    if mass == "random":
        m = (m * rng.uniform(0.5, 1.5, n)).astype(np.float32)
    gx, gv = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    with nb.Simulation(params(n, dt=DT, damping=DAMP, eps=eps), pos, vel, m) as sim:
        sim.adjoint_forward(3, 2)
        got = sim.adjoint_backward(gx.astype(np.float32), gv.astype(np.float32))
    check(got, reference(pos, vel, m, gx, gv, eps, 3))


@pytest.mark.parametrize("sizes", [[1, 300, 17, 256], [64, 700] * 12, [1100, 130] * 3 + [90] * 300,
                                   [40, 500, 16] * 30, [300] * 30, [100] * 130 + [150] * 20])
def test_gradients_of_ensembles(sizes):
    parts = [disk_case(s, seed=70 + k) for k, s in enumerate(sizes)]
    pos, vel = ([np.concatenate([p[q][c] for p in parts]) for c in range(3)] for q in (0, 1))
    m = np.concatenate([p[2] for p in parts])
    n = sum(sizes)
    rng = np.random.default_rng(3)
    gx, gv = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    with nb.Simulation(params(n, dt=DT, damping=DAMP), pos, vel, m, sizes=sizes) as sim:
        sim.adjoint_forward(2, 1)
        gx0, gv0 = sim.adjoint_backward(gx.astype(np.float32), gv.astype(np.float32))
    off = 0
    for k, (s, (p, v, ms)) in enumerate(zip(sizes, parts)):
        sl = slice(off, off + s)
        off += s
        if s > 1 and k % 7 in (0, 1):
            check((gx0[sl], gv0[sl]), reference(p, v, ms, gx[sl], gv[sl], 1e-3, 2))
