"""Threads render images of different small heights, each with a simulation of its own.
Low images need more shared memory than a kernel has by default, the lower the more, and
that limit belongs to the kernel on the device: no thread may take it back."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


HEIGHTS = (16, 18, 32, 40)


def test_small_heights_in_several_threads():
    n, w, frames = 40, 16, 12000
    pos, vel, m = disk_case(n, seed=12)
    errors, images = [], {}

    def render(h):
        try:
            view, proj = nb.camera_matrices(0.3, 0.5, 4.0, w, h)
            out = torch.empty((h, w, 4), dtype=torch.float32, device="cuda")
            with nb.Simulation(params(n), pos, vel, m) as sim:
                for _ in range(frames):
                    sim.render(view, proj, w, h, out.data_ptr())
                sim.synchronize()
            images[h] = out.cpu().numpy()
        except nb.NbError as e:
            errors.append((h, str(e)))

    threads = [threading.Thread(target=render, args=(h,)) for h in HEIGHTS]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert sorted(images) == list(HEIGHTS) and all(np.isfinite(i).all() for i in images.values())
