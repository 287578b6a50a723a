"""Images of every small height: the blur's columns take more shared memory the lower the
image is, from under a kernel's default to over it.  Highest first: the limit that an image
raises stays raised for the next."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_every_small_height():
    n, w = 200, 48
    pos, vel, m = disk_case(n, seed=14)
    vel = [v * 20 for v in vel]
    off, wt, flare = nb.render_tables()
    for h in range(79, 15, -1):
        view, proj = nb.camera_matrices(0.3, 0.5, 4.0, w, h)
        with nb.Simulation(params(n), pos, vel, m) as sim:
            out = torch.full((h, w, 4), float("nan"), dtype=torch.float32, device="cuda")
            sim.render(view, proj, w, h, out.data_ptr())
            sim.synchronize()
        pv = (proj.reshape(4, 4).T @ view.reshape(4, 4).T).T.reshape(-1).astype(np.float32)
        ref = orc.render(pos, vel, pv, w, h, off, wt, flare)
        diff = np.abs(out.cpu().numpy() - ref)
        assert diff.max() < 2e-3 and diff.mean() < 1e-5, (h, diff.max(), diff.mean())
