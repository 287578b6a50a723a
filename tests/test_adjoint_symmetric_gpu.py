"""The adjoint's pair kernel (csrc/adjoint_kernel.cu) at the edges of its tiles, against
FP64 torch autograd of the same map (src/simulator.cu:197-228): one and several i-tiles
of each shape, ragged sizes, no softening, an ensemble.  The vector-Jacobian product of
one step is a sum of n FP32 terms per particle, so the relative error of a gradient is
of the order of 1e-6; the bound is that of the other adjoint tests, 1e-4."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DT, DAMP = 1e-3, 0.999


def reference(pos, vel, m, gx, gv, eps, steps):
    x, v = (torch.from_numpy(np.stack(a, 1).astype(np.float64)).cuda().requires_grad_(True)
            for a in (pos, vel))
    mass = torch.from_numpy(m.astype(np.float64)).cuda()
    eye = torch.eye(len(m), dtype=torch.float64, device="cuda")
    xt, vt = x, v
    for _ in range(steps):
        r = xt[None] - xt[:, None]
        s = ((r * r).sum(-1) + float(np.float32(eps)) + eye).pow(-1.5) * (1 - eye) * mass[None]
        vt = float(np.float32(DAMP)) * vt + float(np.float32(DT)) * (r * s[..., None]).sum(1)
        xt = xt + float(np.float32(DT)) * vt
    ((xt * torch.from_numpy(gx).cuda()).sum() + (vt * torch.from_numpy(gv).cuda()).sum()).backward()
    return x.grad.cpu().numpy(), v.grad.cpu().numpy()


def check(got, want):
    for g, r in zip(got, want):
        rel = np.linalg.norm(g - r) / np.linalg.norm(r)
        assert rel <= 1e-4, rel


@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 97, 127, 130, 1000, 2049])
@pytest.mark.parametrize("mass,eps", [("equal", 1e-3), ("random", 1e-3), ("equal", 0.0)])
def test_gradients_at_tile_edges(n, mass, eps):
    pos, vel, m = disk_case(n, seed=n)
    rng = np.random.default_rng(n)
    if eps == 0.0:  # apart from each other: no softening bounds the force
        pos = [(8 * rng.permutation(n) + rng.uniform(0, 1, n)).astype(np.float32) for _ in range(3)]
    if mass == "random":
        m = (m * rng.uniform(0.5, 1.5, n)).astype(np.float32)
    gx, gv = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    with nb.Simulation(params(n, dt=DT, damping=DAMP, eps=eps), pos, vel, m) as sim:
        sim.adjoint_forward(2, 1)
        got = sim.adjoint_backward(gx.astype(np.float32), gv.astype(np.float32))
    check(got, reference(pos, vel, m, gx, gv, eps, 2))


@pytest.mark.parametrize("sizes,steps", [
    # About 5,300 blocks choose 256-particle i-tiles, systems of one to 18 of them.
    ([4500, 1, 4500, 256, 257, 3000, 4500, 600], 2),
    # Six systems of 11 i-tiles are enough blocks for the 768-particle i-tiles.
    ([8192, 8192, 8195, 8192, 8192, 8192], 1)])
def test_gradients_of_ensembles_with_larger_tiles(sizes, steps):
    parts = [disk_case(s, seed=70 + k) for k, s in enumerate(sizes)]
    pos, vel = ([np.concatenate([p[q][c] for p in parts]) for c in range(3)] for q in (0, 1))
    m = np.concatenate([p[2] for p in parts])
    n = sum(sizes)
    rng = np.random.default_rng(3)
    gx, gv = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    with nb.Simulation(params(n, dt=DT, damping=DAMP), pos, vel, m, sizes=sizes) as sim:
        sim.adjoint_forward(steps, 2)
        gx0, gv0 = sim.adjoint_backward(gx.astype(np.float32), gv.astype(np.float32))
    off = 0
    for s, (p, v, ms) in zip(sizes, parts):
        sl = slice(off, off + s)
        off += s
        check((gx0[sl], gv0[sl]), reference(p, v, ms, gx[sl], gv[sl], 1e-3, steps))
