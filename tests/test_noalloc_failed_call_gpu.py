"""nb_accelerations_noalloc after a call that failed on the way: on a stream that is being
captured the call cannot wait, so it ends with an error, and the work list that it was
to upload is not in the scratch.  The next calls must not take it for granted."""
from __future__ import annotations

import ctypes as C

import pytest

import nbody_gb300 as nb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

THREAD_LOCAL = 1  # CU_STREAM_CAPTURE_MODE_THREAD_LOCAL


def particles(n):
    g = torch.Generator().manual_seed(n)
    return torch.randn((n, 4), generator=g).abs().cuda()


def call(xyzm, out, stream=0):
    n = xyzm.shape[0]
    return nb.lib.nb_accelerations_noalloc(C.c_void_p(xyzm.data_ptr()), n, 1.0, 1e-3,
                                           C.c_void_p(out.data_ptr()), C.c_void_p(stream))


@pytest.mark.parametrize("n", [300, 6000, 20000])  # direct, one band, several
@pytest.mark.parametrize("in_place", [False, True])
def test_calls_after_a_call_under_capture(n, in_place):
    cu = C.CDLL("libcuda.so.1")
    xyzm, other = particles(n), particles(9000)
    want, scrap = torch.empty_like(xyzm), torch.empty_like(other)
    assert call(xyzm.clone() if in_place else xyzm, want) == nb.NB_OK
    if in_place:
        want = xyzm.clone()
        assert call(want, want) == nb.NB_OK
    assert call(other, scrap) == nb.NB_OK      # another plan in the scratch
    torch.cuda.synchronize()

    buf = xyzm.clone()
    out = buf if in_place else torch.empty_like(xyzm)
    stream = torch.cuda.Stream()
    handle, graph = C.c_void_p(stream.cuda_stream), C.c_void_p()
    assert cu.cuStreamBeginCapture_v2(handle, THREAD_LOCAL) == 0
    status = call(buf, out, stream.cuda_stream)
    cu.cuStreamEndCapture(handle, C.byref(graph))
    assert status == nb.NB_ERR_CUDA

    buf = xyzm.clone()
    out = buf if in_place else torch.empty_like(xyzm)
    assert call(buf, out) == nb.NB_OK
    assert torch.equal(out, want)
    assert call(other, other.clone()) == nb.NB_OK
