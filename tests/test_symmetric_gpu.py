"""The symmetric force kernel (csrc/symmetric_kernel.cuh): each unordered pair once,
applied to both particles.  Every shape against the CPU oracle (reference semantics:
src/simulator.cu:193-228) at the edges of its tiles, and the ways its launches differ
from the tuned kernel's: bands, ensembles, masks, graphs, shards, failure hooks.

Tolerances are those of the other parity tests: FP32 pair arithmetic, accelerations to
1e-5 relative RMS and 1e-4 per particle."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, g_eff, params, vec_errors
from test_symmetric_cpu import symmetric_configs

pytestmark = pytest.mark.gpu

ACC_RMS, ACC_MAX = 1e-5, 1e-4
EPS32 = float(np.float32(1e-3))


def _case(n, mass="equal", seed=5):
    pos, vel, m = disk_case(n, seed=seed + n)
    if mass == "random":
        m = (m * np.random.default_rng(n).uniform(0.5, 1.5, n)).astype(np.float32)
    return pos, vel, m


@pytest.mark.parametrize("cfg", symmetric_configs())
@pytest.mark.parametrize("mass", ["equal", "random"])
@pytest.mark.parametrize("acc", [nb.ACC_PLAIN, nb.ACC_COMPENSATED])
def test_tile_edges_match_fp64(cfg, mass, acc):
    info = nb.kernel_config_info(cfg)
    bi, bj = info["threads_per_block"] * info["particles_per_thread"], info["j_tile"]
    for n in (2, 31, 33, bj + 1, bi - 1, bi, bi + 1, bi + 17, 2 * bi, 2 * bi + bj + 5):
        pos, vel, m = _case(n, mass)
        with nb.Simulation(params(n, acc=acc), pos, vel, m) as sim:
            sim.set_kernel_config(cfg)
            got = sim.accelerations()
            sim.advance(2)
            st = sim.get_state()
        rms, mx = vec_errors(got, orc.accel_fp64(pos, m, 1.0, EPS32))
        assert rms <= ACC_RMS and mx <= ACC_MAX, (n, rms, mx)
        om, G = (m, 1.0) if mass == "random" else (None, g_eff(1.0, m[0]))
        ref = orc.run_fp32(pos, vel, om, G, 1e-3, 0.999, 1e-3, iters=2)
        for g, r in zip(st, ref):
            assert np.max(np.abs(g - r)) <= 1e-5 * max(1.0, np.max(np.abs(r))), n


@pytest.mark.parametrize("acc", [nb.ACC_PLAIN, nb.ACC_COMPENSATED])
@pytest.mark.parametrize("cfg", symmetric_configs())
def test_zero_softening_and_coincident_particles(cfg, acc):
    # eps = 0: the self pair is left out by index; coincident particles get NaN, and
    # only they (0 * rsqrt(0), as in the reference).  Pairs of one tile and of two.
    n = 5000
    pos, vel, m = _case(n)
    with nb.Simulation(params(n, eps=0.0, acc=acc), pos, vel, m) as sim:
        sim.set_kernel_config(cfg)
        got = sim.accelerations()
    rms, mx = vec_errors(got, orc.accel_fp32(pos, None, g_eff(1.0, m[0]), 0.0))
    assert rms <= ACC_RMS and mx <= ACC_MAX
    same = [(3, 4), (10, 600), (100, 4999)]
    for a in pos:
        for i, j in same:
            a[j] = a[i]
    with nb.Simulation(params(n, eps=0.0, acc=acc), pos, vel, m) as sim:
        sim.set_kernel_config(cfg)
        got = sim.accelerations()
    want = np.zeros(n, bool)
    want[[k for p in same for k in p]] = True
    for g in got:
        assert np.array_equal(np.isnan(g), want)


@pytest.mark.parametrize("cfg", symmetric_configs())
def test_uneven_ensemble_matches_fp64(cfg):
    sizes = [1, 5000, 64, 513, 16, 2049, 4100]
    parts = [_case(s, seed=50 + k) for k, s in enumerate(sizes)]
    pos, vel = ([np.concatenate([p[q][c] for p in parts]) for c in range(3)] for q in (0, 1))
    m = np.concatenate([p[2] for p in parts])
    with nb.Simulation(params(sum(sizes), acc=nb.ACC_COMPENSATED), pos, vel, m, sizes=sizes) as sim:
        sim.set_kernel_config(cfg)
        got = sim.accelerations()
    off = 0
    for s, (p, _, ms) in zip(sizes, parts):
        g = [a[off:off + s] for a in got]
        off += s
        if s == 1:
            assert all(a[0] == 0 for a in g)
            continue
        rms, mx = vec_errors(g, orc.accel_fp64(p, ms, 1.0, EPS32))
        assert rms <= ACC_RMS and mx <= ACC_MAX, (s, rms, mx)


def test_bands_match_the_tuned_kernel():
    # At 512-particle i-tiles the rows of 300,001 particles take 1 GB: several bands,
    # with the running sums carried from one to the next.
    n = 300001
    pos, vel, m = _case(n)
    small = symmetric_configs()[-1]
    with nb.Simulation(params(n, acc=nb.ACC_COMPENSATED), pos, vel, m) as sim:
        sim.set_kernel_config(9)
        want = sim.accelerations()
        sim.set_kernel_config(small)
        got = sim.accelerations()
        again = sim.accelerations()
    rms, mx = vec_errors(got, want)
    assert rms <= 1e-6 and mx <= 1e-5, (rms, mx)
    for a, b in zip(got, again):
        assert np.array_equal(a, b)


def test_graph_failure_hook_and_shard():
    n = 30000
    pos, vel, m = _case(n)
    cfg = symmetric_configs()[1]
    with nb.Simulation(params(n, acc=nb.ACC_COMPENSATED), pos, vel, m) as sim:
        sim.set_kernel_config(cfg)
        assert sim.kernel_info()["config_index"] == cfg
        sim.advance(3)
        want = sim.get_state()
        sim.set_state(pos, vel)
        sim.graph_capture(3)
        sim.graph_launch()
        for a, b in zip(sim.get_state(), want):
            assert np.array_equal(a, b)
        # The hook's bounded wait belongs to the tuned kernel, which takes that launch.
        sim.inject_wait_timeout()
        sim.advance(1)
        with pytest.raises(nb.NbError) as e:
            sim.synchronize()
        assert e.value.status == nb.NB_ERR_DEVICE_TIMEOUT
        sim.set_state(pos, vel)
        sim.advance(3)
        for a, b in zip(sim.get_state(), want):
            assert np.array_equal(a, b)
        # A shard integrates part of the system: the tuned kernel.
        sim.set_shard(0, 16000)
        assert sim.kernel_info()["stages"] > 0
        with pytest.raises(nb.NbError) as e:
            sim.set_kernel_config(cfg)
        assert e.value.status == nb.NB_ERR_INVALID_ARGUMENT
        sim.set_shard(0, 0)
        sim.set_kernel_config(cfg)
        sim.set_state(pos, vel)
        sim.advance(3)
        for a, b in zip(sim.get_state(), want):
            assert np.array_equal(a, b)
