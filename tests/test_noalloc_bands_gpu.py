"""nb_accelerations_noalloc (csrc/noalloc.cu) over its shapes and bands: sizes at the
edges of i-tiles and of the fixed scratch, one buffer for input and output, and calls of
different sizes in turn (the work list stays in the scratch for the next call of the
same size).  Tolerances are those of the other parity tests."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, vec_errors

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS32 = float(np.float32(1e-3))


def case(n):
    pos, _, m = disk_case(n, seed=n)
    m = (m * np.random.default_rng(n).uniform(0.5, 1.5, n)).astype(np.float32)
    return pos, m, torch.from_numpy(np.stack([*pos, m], 1)).cuda()


def check(got, pos, m, rows=None):
    g = [got[:, c].cpu().numpy() for c in range(4)]
    assert np.all(g[3] == 0.0)
    rows = np.arange(len(m)) if rows is None else rows
    rms, mx = vec_errors([a[rows] for a in g[:3]], orc.accel_fp64(pos, m, 1.0, EPS32, rows=rows))
    assert rms <= 1e-5 and mx <= 1e-4, (len(m), rms, mx)


@pytest.mark.parametrize("n", [2, 63, 64, 65, 2000, 4095, 4097, 9000, 16385, 25000, 60001, 150000,
                               262143])
@pytest.mark.parametrize("in_place", [False, True])
def test_sizes_bands_and_one_buffer(n, in_place):
    pos, m, xyzm = case(n)
    out = xyzm if in_place else torch.full((n, 4), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    nb.accelerations_noalloc(xyzm.data_ptr(), n, 1.0, 1e-3, out.data_ptr(), stream)
    check(out, pos, m, None if n <= 9000 else np.linspace(0, n - 1, 384).astype(np.int64))


def test_sizes_in_turn_and_other_parameters():
    cases = {n: case(n) for n in (300, 5000, 20000)}
    first = {}
    for n in (300, 5000, 300, 20000, 5000, 20000):
        pos, m, xyzm = cases[n]
        out = torch.empty((n, 4), device="cuda")
        nb.accelerations_noalloc(xyzm.data_ptr(), n, 1.0, 1e-3, out.data_ptr())
        check(out, pos, m, np.arange(0, n, 7))
        assert torch.equal(out, first.setdefault(n, out.clone()))
    pos, m, xyzm = cases[5000]
    out = torch.empty((5000, 4), device="cuda")
    nb.accelerations_noalloc(xyzm.data_ptr(), 5000, 2.0, 1e-3, out.data_ptr())
    assert torch.allclose(out, 2 * first[5000], rtol=1e-6, atol=0)


def test_no_plan_is_refused_up_to_the_limit():
    # The largest plans of every i-tile count of the largest shape, planned but small in
    # work: any status other than NB_OK fails.
    for n in range(4096, 262145, 8192 + 4096 + 17):
        xyzm = torch.zeros((n, 4), device="cuda")
        xyzm[:, 0] = torch.arange(n, device="cuda")
        for out in (torch.empty_like(xyzm), xyzm):
            rc = nb.lib.nb_accelerations_noalloc(C.c_void_p(xyzm.data_ptr()), n, 1.0, 1e-3,
                                                 C.c_void_p(out.data_ptr()), None)
            assert rc == nb.NB_OK, (n, nb.lib.nb_last_error())
