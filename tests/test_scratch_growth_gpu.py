"""Per-system launches whose lists need more scratch than the all-systems list had: the
launches use the scratch as it is after the lists were planned."""
from __future__ import annotations

import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, displacement_errors, g_eff, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["advance_per_system", "time_iterations"])
def test_per_system_lists_outgrow_the_scratch(method):
    n = 6000
    pos, vel, m = disk_case(n, seed=8)
    ref = orc.run_fp32(pos, vel, None, g_eff(1.0, m[0]), 1e-3, 0.999, 1e-3, iters=2)
    small = 0
    for k in range(1, 40):
        # Creation without one of the symmetric kernel's allocations: the tuned kernel's
        # list, and its smaller scratch.
        nb.inject_alloc_failure(k)
        try:
            sim = nb.Simulation(params(n, acc=nb.ACC_COMPENSATED), pos, vel, m)
        except nb.NbError as e:
            assert e.status == nb.NB_ERR_OUT_OF_MEMORY
            continue
        finally:
            nb.inject_alloc_failure(0)
        with sim:
            done = sim.kernel_info()["stages"] == 0
            if method == "advance_per_system":
                sim.advance_per_system(2)
            else:
                sim.time_iterations(2, per_system=1)
            got = sim.get_state()
        rms, mx = displacement_errors(got[:3], ref[:3], pos)
        assert rms <= 1e-4 and mx <= 1e-2, (k, rms, mx)
        if done:
            break
        small += 1
    assert small
