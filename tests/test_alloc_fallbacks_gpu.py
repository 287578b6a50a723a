"""What runs without an allocation that failed: the tuned kernel where the symmetric
kernel's scratch cannot be had, one copy of the HDR buffer, the autotuner's other
candidates.  A failure leaves the runtime's last error set; the next launches must not
report it (a step that did had updated the velocities but not the positions)."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, displacement_errors, g_eff, params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class failing_allocation:
    """The k-th device allocation inside the block fails."""

    def __init__(self, k):
        self.k = k

    def __enter__(self):
        nb.inject_alloc_failure(self.k)

    def __exit__(self, *exc):
        nb.inject_alloc_failure(0)


def check_steps(sim, pos, vel, m):
    sim.advance(1)
    sim.synchronize()
    sim.advance(2)
    got = sim.get_state()
    ref = orc.run_fp32(pos, vel, None, g_eff(1.0, m[0]), 1e-3, 0.999, 1e-3, iters=3)
    rms, mx = displacement_errors(got[:3], ref[:3], pos)
    assert rms <= 1e-4 and mx <= 1e-2, (rms, mx)


def test_creation_falls_back_to_the_tuned_kernel_and_steps():
    n = 6000
    pos, vel, m = disk_case(n, seed=5)
    fell_back = 0
    for k in range(1, 40):
        with failing_allocation(k):
            try:
                sim = nb.Simulation(params(n, acc=nb.ACC_COMPENSATED), pos, vel, m)
            except nb.NbError as e:
                assert e.status == nb.NB_ERR_OUT_OF_MEMORY
                continue
        with sim:
            stages = sim.kernel_info()["stages"]
            check_steps(sim, pos, vel, m)
        if stages == 0:
            break                       # past the last allocation: the symmetric kernel
        fell_back += 1
    assert fell_back >= 3               # segments, i-tiles, rows, parts


def test_autotune_goes_on_without_a_candidate():
    n = 6000
    pos, vel, m = disk_case(n, seed=6)
    tuned = 0
    for k in (10, 45, 60, 61, 62, 63, 64, 65):
        with nb.Simulation(params(n, acc=nb.ACC_COMPENSATED), pos, vel, m) as sim:
            with failing_allocation(k):
                try:
                    sim.autotune()
                    tuned += 1
                except nb.NbError as e:
                    assert e.status == nb.NB_ERR_OUT_OF_MEMORY
            check_steps(sim, pos, vel, m)
    assert tuned


def test_render_with_one_copy_of_the_hdr_buffer():
    n, w, h = 60000, 64, 64
    pos, vel, m = disk_case(n, seed=7)
    view, proj = nb.camera_matrices(0.3, 0.5, 4.0, w, h)
    images = []
    for k in (0, 1):
        with nb.Simulation(params(n), pos, vel, m) as sim:
            out = torch.full((h, w, 4), float("nan"), dtype=torch.float32, device="cuda")
            with failing_allocation(k):
                sim.render(view, proj, w, h, out.data_ptr())
            sim.synchronize()
            images.append(out.cpu().numpy())
    # Sums of the same non-negative terms in another order: up to thousands of them at a
    # pixel of the middle, each rounded by 2^-24 of its sum, through exp and a root.
    assert np.abs(images[0] - images[1]).max() <= 1e-3
