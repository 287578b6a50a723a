"""Work lists of the direct force kernel (csrc/direct_kernel.cu): a CTA per i-tile."""
from __future__ import annotations

import pytest

import nbody_gb300 as nb


@pytest.mark.parametrize("cfg", [c for c in range(13, nb.num_kernel_configs())
                                 if nb.kernel_config_info(c)["stages"] == 1])
def test_one_cta_per_i_tile(cfg):
    info = nb.kernel_config_info(cfg)
    r, bj = info["particles_per_thread"], info["j_tile"]
    assert 16 % r == 0  # a tile never reaches past the padding
    sizes = [1, r, r + 1, 2049]
    want = [(s, t, 0, -(-(-(-n // 16) * 16) // bj), -1, 0)
            for s, n in enumerate(sizes) for t in range(-(-n // r))]
    g, segs, begin, nfix, slots = nb.plan_work(sizes, cfg, len(want))
    assert [tuple(s) for s in segs] == want
    assert g == len(want) and list(begin) == list(range(g + 1)) and nfix == slots == 0
    with pytest.raises(nb.NbError) as e:
        nb.plan_work(sizes, cfg, len(want) - 1)
    assert e.value.status == nb.NB_ERR_INVALID_ARGUMENT
