"""The direct force kernel (csrc/direct_kernel.cu): every shape against the CPU oracle
(reference semantics: src/simulator.cu:193-228) at the edges of its i-tiles, its passes
over the j-particles and the folds of its sums; masks, ensembles, graphs, shards, and the
small no-allocation calls that run it.

Tolerances are those of the other parity tests: FP32 pair arithmetic, accelerations to
1e-5 relative RMS and 1e-4 per particle."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, g_eff, params, vec_errors

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ACC_RMS, ACC_MAX = 1e-5, 1e-4
EPS32 = float(np.float32(1e-3))


def direct_configs():
    """The direct shapes: the last configs, of one stage."""
    return [c for c in range(13, nb.num_kernel_configs())
            if nb.kernel_config_info(c)["stages"] == 1]


def _case(n, mass="equal"):
    pos, vel, m = disk_case(n, seed=5 + n)
    if mass == "random":
        m = (m * np.random.default_rng(n).uniform(0.5, 1.5, n)).astype(np.float32)
    return pos, vel, m


@pytest.mark.parametrize("cfg", direct_configs())
@pytest.mark.parametrize("mass", ["equal", "random"])
@pytest.mark.parametrize("acc", [nb.ACC_PLAIN, nb.ACC_COMPENSATED])
def test_edges_match_fp64(cfg, mass, acc):
    info = nb.kernel_config_info(cfg)
    r, per_pass = info["particles_per_thread"], info["j_tile"]
    for n in (1, 2, 3, r - 1, r, r + 1, 15, 17, per_pass - 1, per_pass + 1, 3 * per_pass + 5,
              64 * per_pass - 16, 64 * per_pass + 2):
        pos, vel, m = _case(n, mass)
        rows = np.unique(np.linspace(0, n - 1, 600).astype(np.int64))
        with nb.Simulation(params(n, acc=acc), pos, vel, m) as sim:
            sim.set_kernel_config(cfg)
            got = sim.accelerations()
            sim.advance(2)
            st = sim.get_state()
        if n == 1:
            assert all(g[0] == 0 for g in got)
            continue
        rms, mx = vec_errors([g[rows] for g in got],
                             orc.accel_fp64(pos, m, 1.0, EPS32, rows=rows))
        assert rms <= ACC_RMS and mx <= ACC_MAX, (n, rms, mx)
        if n <= 4200:
            om, G = (m, 1.0) if mass == "random" else (None, g_eff(1.0, m[0]))
            ref = orc.run_fp32(pos, vel, om, G, 1e-3, 0.999, 1e-3, iters=2)
            for g, w in zip(st, ref):
                assert np.max(np.abs(g - w)) <= 1e-5 * max(1.0, np.max(np.abs(w))), n


@pytest.mark.parametrize("acc", [nb.ACC_PLAIN, nb.ACC_COMPENSATED])
@pytest.mark.parametrize("cfg", direct_configs())
def test_zero_softening_and_coincident_particles(cfg, acc):
    # eps = 0: the self pair is left out by index; coincident particles get NaN, and
    # only they (0 * rsqrt(0), as in the reference).
    n = 3001
    pos, vel, m = _case(n)
    with nb.Simulation(params(n, eps=0.0, acc=acc), pos, vel, m) as sim:
        sim.set_kernel_config(cfg)
        got = sim.accelerations()
    rms, mx = vec_errors(got, orc.accel_fp32(pos, None, g_eff(1.0, m[0]), 0.0))
    assert rms <= ACC_RMS and mx <= ACC_MAX
    same = [(3, 4), (10, 600), (100, 3000)]
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


@pytest.mark.parametrize("cfg", direct_configs())
def test_uneven_ensemble_in_a_graph(cfg):
    sizes = [1, 3000, 64, 513, 16, 2049, 7]
    parts = [_case(s) for s in sizes]
    pos = [np.concatenate([p[0][c] for p in parts]) for c in range(3)]
    vel = [np.concatenate([p[1][c] for p in parts]) for c in range(3)]
    m = np.concatenate([p[2] for p in parts])
    n = sum(sizes)
    stream = torch.cuda.Stream()
    with nb.Simulation(params(n, acc=nb.ACC_COMPENSATED), pos, vel, m, sizes=sizes) as sim:
        sim.set_stream(stream.cuda_stream)
        sim.set_kernel_config(cfg)
        got = sim.accelerations()
        sim.advance(3)
        want = sim.get_state()
        sim.set_state(pos, vel)
        sim.graph_capture(3)
        sim.graph_launch()
        for a, b in zip(sim.get_state(), want):
            assert np.array_equal(a, b)
    at = 0
    for s, p in zip(sizes, parts):
        if s > 1:
            rms, mx = vec_errors([g[at:at + s] for g in got],
                                 orc.accel_fp64(p[0], p[2], 1.0, EPS32))
            assert rms <= ACC_RMS and mx <= ACC_MAX, (s, rms, mx)
        at += s


def test_defaults_hook_and_shard():
    n = 2048
    pos, vel, m = _case(n)
    with nb.Simulation(params(n, acc=nb.ACC_COMPENSATED), pos, vel, m) as sim:
        cfg = sim.kernel_info()["config_index"]
        assert cfg in direct_configs()
        sim.advance(3)
        want = sim.get_state()
        sim.set_state(pos, vel)
        sim.inject_wait_timeout()  # belongs to the tuned kernel, which takes that launch
        sim.advance(1)
        with pytest.raises(nb.NbError) as e:
            sim.synchronize()
        assert e.value.status == nb.NB_ERR_DEVICE_TIMEOUT
        sim.set_shard(0, 1008)
        assert sim.kernel_info()["config_index"] < 13
        with pytest.raises(nb.NbError) as e:
            sim.set_kernel_config(cfg)
        assert e.value.status == nb.NB_ERR_INVALID_ARGUMENT
        sim.set_shard(0, 0)
        sim.set_state(pos, vel)
        sim.advance(3)
        for a, b in zip(sim.get_state(), want):
            assert np.array_equal(a, b)
    pos, vel, m = _case(8192)
    with nb.Simulation(params(8192), pos, vel, m) as sim:
        assert sim.kernel_info()["stages"] == 0


@pytest.mark.parametrize("n", [1, 2, 7, 255, 511, 513, 2433, 4257, 4690])
@pytest.mark.parametrize("eps", [1e-3, 0.0])
def test_no_allocation_call(n, eps):
    pos, _, m = _case(n, "random")
    xyzm = torch.from_numpy(np.stack([*pos, m], 1)).cuda()
    out = torch.full((n, 4), float("nan"), device="cuda")
    nb.accelerations_noalloc(xyzm.data_ptr(), n, 1.0, eps, out.data_ptr())
    got = [out[:, c].cpu().numpy() for c in range(4)]
    assert np.all(got[3] == 0.0)
    if n == 1:
        assert all(g[0] == 0 for g in got)
        return
    want = (orc.accel_fp64(pos, m, 1.0, EPS32) if eps else
            orc.accel_fp32(pos, m, 1.0, 0.0))
    rms, mx = vec_errors(got[:3], want)
    assert rms <= ACC_RMS and mx <= ACC_MAX, (n, rms, mx)


def test_no_allocation_copy_over_a_kept_plan():
    # A large call's plan stays in the scratch; a small in-place call copies its input there.
    big = torch.from_numpy(np.stack([*_case(20000)[0], _case(20000)[2]], 1)).cuda()
    small = torch.from_numpy(np.stack([*_case(1000)[0], _case(1000)[2]], 1)).cuda()
    out = [torch.empty_like(big) for _ in range(2)]
    apart = torch.empty_like(small)
    nb.accelerations_noalloc(big.data_ptr(), 20000, 1.0, 1e-3, out[0].data_ptr())
    nb.accelerations_noalloc(small.data_ptr(), 1000, 1.0, 1e-3, apart.data_ptr())
    nb.accelerations_noalloc(small.data_ptr(), 1000, 1.0, 1e-3, small.data_ptr())
    nb.accelerations_noalloc(big.data_ptr(), 20000, 1.0, 1e-3, out[1].data_ptr())
    assert torch.equal(small, apart) and torch.equal(out[0], out[1])
