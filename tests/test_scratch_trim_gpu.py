"""Device memory that a simulation holds: the symmetric kernel's scratch goes when nothing
runs that kernel any more (a shard, another shape selected), and no part of it stays
behind where its creation failed half-way."""
from __future__ import annotations

import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 120000                 # rows: about n * n / (2 * 4096) values of 12 bytes, 21 MB
ROWS = 12 * N * N // (2 * 4096) - 12 * N
SLACK = 6 << 20            # allocations come in pages of 2 MiB: lists, parts


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def case():
    pos, vel, m = disk_case(N, seed=15)
    with nb.Simulation(params(N, acc=nb.ACC_COMPENSATED), pos, vel, m) as sim:
        for config in (-1, 9):             # their kernels are loaded
            sim.set_kernel_config(config)
            check_step(sim, pos, vel, m)
    return pos, vel, m


def check_step(sim, pos, vel, m):
    rows = range(0, 9600, 400)
    sim.set_state(pos, vel)
    got = sim.accelerations()
    ref = orc.accel_fp64(pos, m, 1.0, 1e-3, rows=list(rows))
    for g, r in zip(got, ref):
        assert max(abs(g[i] - x) for i, x in zip(rows, r)) <= 1e-4 * max(abs(r))


@pytest.mark.parametrize("how", ["shard", "config"])
def test_scratch_goes_with_the_symmetric_kernel(case, how):
    pos, vel, m = case
    with nb.Simulation(params(N, acc=nb.ACC_COMPENSATED), pos, vel, m) as sim:
        sim.advance(1)
        sim.advance_per_system(1)
        if how == "shard":
            sim.adjoint_forward(1, 1)
        sim.synchronize()
        before = free_bytes()
        if how == "shard":
            sim.set_shard(0, 60000 // 16 * 16)
        else:
            sim.set_kernel_config(9)
            sim.advance_per_system(1)          # its own list is the symmetric kernel's
            assert free_bytes() - before <= SLACK
            return
        assert free_bytes() - before >= ROWS - SLACK
        check_step(sim, pos, vel, m)
        sim.set_shard(0, 0)
        assert sim.kernel_info()["stages"] == 0
        check_step(sim, pos, vel, m)


def test_scratch_goes_with_another_shape(case):
    pos, vel, m = case
    with nb.Simulation(params(N, acc=nb.ACC_COMPENSATED), pos, vel, m) as sim:
        sim.graph_capture(1)
        before = free_bytes()
        sim.set_kernel_config(9)
        assert free_bytes() - before >= ROWS - SLACK
        check_step(sim, pos, vel, m)
        sim.set_kernel_config(-1)
        check_step(sim, pos, vel, m)


def test_nothing_stays_of_a_scratch_that_failed(case):
    pos, vel, m = case
    held = []
    for k in range(1, 40):
        start = free_bytes()
        nb.inject_alloc_failure(k)
        try:
            sim = nb.Simulation(params(N, acc=nb.ACC_COMPENSATED), pos, vel, m)
        except nb.NbError as e:
            assert e.status == nb.NB_ERR_OUT_OF_MEMORY
            continue
        finally:
            nb.inject_alloc_failure(0)
        with sim:
            if sim.kernel_info()["stages"] == 0:
                break
            held.append(start - free_bytes())
            check_step(sim, pos, vel, m)
    assert len(held) >= 3 and max(held) - min(held) <= SLACK, held


def test_predicated_holds_no_scratch(case):
    # Its kernels need a list of work and, for the i-pair shapes, 32 bytes per particle.
    pos, vel, _ = case
    held = []
    for method in (nb.PREDICATED, nb.BRANCH):
        start = free_bytes()
        with nb.Simulation(params(N, method=method, acc=nb.ACC_COMPENSATED), pos, vel, None) as sim:
            held.append(start - free_bytes())
            sim.advance(1)
            sim.synchronize()
    assert held[0] + ROWS - SLACK <= held[1], held
