"""The failure hook (nb_sim_inject_failure) whatever kernel shape is selected when it is
armed and when the hooked launch is made: it runs the tuned kernel, whose bounded wait
runs out, over the systems of that launch and no others."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

pytestmark = pytest.mark.gpu

SIZES = [20000, 700, 5000]


def ensemble():
    parts = [disk_case(s, seed=60 + k) for k, s in enumerate(SIZES)]
    pos, vel = ([np.concatenate([p[q][c] for p in parts]) for c in range(3)] for q in (0, 1))
    m = np.concatenate([np.full(s, 1.0 / s, np.float32) for s in SIZES])
    return pos, vel, m


def timed_out(sim):
    with pytest.raises(nb.NbError) as e:
        sim.synchronize()
    return e.value.status == nb.NB_ERR_DEVICE_TIMEOUT


def test_per_system_pass_with_a_tuned_shape_selected():
    pos, vel, m = ensemble()
    p = params(sum(SIZES), acc=nb.ACC_COMPENSATED)
    with nb.Simulation(p, pos, vel, m, sizes=SIZES) as sim:
        sim.advance_per_system(1)
        want = sim.get_state()
    for config in (4, -1):
        with nb.Simulation(p, pos, vel, m, sizes=SIZES) as sim:
            sim.set_kernel_config(config)
            sim.inject_wait_timeout()
            sim.advance_per_system(1)
            assert timed_out(sim)
            got = sim.get_state()
            for g, w in zip(got, want):       # the other systems: one step, the usual one
                assert np.array_equal(g[SIZES[0]:], w[SIZES[0]:])
            sim.set_state(pos, vel)
            sim.advance_per_system(1)
            for g, w in zip(sim.get_state(), want):
                assert np.array_equal(g, w)


@pytest.mark.parametrize("armed,launched", [(4, -1), (-1, 4), (-1, 13), (9, 13)])
def test_shape_selected_after_arming(armed, launched):
    n = 20000
    pos, vel, m = disk_case(n, seed=64)
    with nb.Simulation(params(n), pos, vel, m) as sim:
        sim.set_kernel_config(armed)
        sim.inject_wait_timeout()
        sim.set_kernel_config(launched)
        sim.advance(1)
        assert timed_out(sim)
        sim.set_state(pos, vel)
        sim.advance(1)
        sim.synchronize()


def test_whole_system_again_after_arming_a_shard():
    n = 20000
    pos, vel, m = disk_case(n, seed=65)
    with nb.Simulation(params(n), pos, vel, m) as sim:
        sim.set_shard(0, 9600)
        sim.inject_wait_timeout()
        sim.set_shard(0, 0)
        sim.advance(1)
        assert timed_out(sim)
        sim.set_state(pos, vel)
        sim.advance(1)
        sim.synchronize()
