"""The planner of nb_accelerations_noalloc (csrc/noalloc_plan.hpp), replayed on the host over
its whole range: no plan is refused, each fits the fixed tables and the scratch on the
full grid, and covers every (i-tile, j-tile) block once."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

import pytest

import nbody_gb300 as nb

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "cuda-to-sycl-nbody_gb300" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
LARGEST = 262144


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    exe = tmp_path_factory.mktemp("noalloc") / "replay"
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-I", str(CSRC), "-I",
                    str(CUDA / "include"), str(ROOT / "tests" / "noalloc_plan_replay.cpp"),
                    str(CSRC / "symmetric.cpp"), "-o", str(exe)], check=True)
    symmetric = [i for i in map(nb.kernel_config_info, range(nb.num_kernel_configs()))
                 if i["stages"] == 0]
    shapes = [str(symmetric[k][key]) for k in (0, 2, 3)
              for key in ("threads_per_block", "particles_per_thread", "j_tile")]

    def run(sms, per_sm, first, last, step):
        r = subprocess.run([str(exe), *shapes, *map(str, (sms, *per_sm, first, last, step))],
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr

    return run


# CTAs per SM: what the kernels' launch bounds grant at least, and twice that.  Sizes from the
# smallest that plans (smaller ones run the direct kernel) to the largest.
@pytest.mark.parametrize("sms,per_sm", [(152, (1, 8, 8)), (152, (1, 8, 16)), (152, (1, 9, 16)),
                                        (160, (1, 8, 16)), (148, (1, 8, 12))])
def test_every_plan_fits_on_the_full_grid(replay, sms, per_sm):
    replay(sms, per_sm, 4690, 32768, 61)
    replay(sms, per_sm, 32768, LARGEST, 1021)
    replay(sms, per_sm, LARGEST - 1, LARGEST, 1)
