"""The renderer's kernels (csrc/render_kernels.cu) at the sizes where they branch: odd and
even images (the blur's fixed and general taps), sprites wider than the lanes' 8 x 16
pixels (small images), few particles (fewer per warp), particles across the image's
edges, against the CPU restatement (oracle/render_oracle.c).  Tolerances are those of
tests/test_render_gpu.py: float reduction order, exp and pow ulps."""
from __future__ import annotations

import math

import numpy as np
import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 1000, 40000])
@pytest.mark.parametrize("w,h,dist", [(16, 16, 4.0), (17, 40, 3.0), (120, 90, 2.0), (301, 201, 1.2),
                                      (640, 361, 4.0)])
def test_image_matches_cpu_restatement(n, w, h, dist):
    pos, vel, m = disk_case(n, seed=n + w)
    vel = [v * 20 for v in vel]
    view, proj = nb.camera_matrices(0.3, math.pi / 4, dist, w, h)
    with nb.Simulation(params(n), pos, vel, m) as sim:
        out = torch.full((h, w, 4), float("nan"), dtype=torch.float32, device="cuda")
        sim.render(view, proj, w, h, out.data_ptr())
        sim.synchronize()
    img = out.cpu().numpy()
    pv = (proj.reshape(4, 4).T @ view.reshape(4, 4).T).T.reshape(-1).astype(np.float32)
    off, wt, flare = nb.render_tables()
    ref = orc.render(pos, vel, pv, w, h, off, wt, flare)
    assert np.all(img[..., 3] == 1.0)
    diff = np.abs(img - ref)
    assert diff.max() < 2e-3 and diff.mean() < 1e-5, (diff.max(), diff.mean())
