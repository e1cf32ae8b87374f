"""Image lists beyond their memory limit leave nothing allocated."""
import numpy as np
import pytest

from conftest import packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu

_STEP = 2 ** 25  # the pool grows by 32 MiB


def _many_types():
    # 144 potential types of one term: a range per unit and type, 90 MB of them
    s = configs.graphite_cell(reps=(6, 6, 1), kmesh=(1, 1, 1), jitter=0.02)
    p = s.pot_types[0]
    s.pot_types = [configs.PotType(element=1 + i, label=f"c{i}", nuc_charge=6.0,
                                   nuc_alpha=20.0, alphas=p.alphas[[8]].copy())
                   for i in range(len(s.site_pos))]
    s.pot_site_type = np.arange(1, len(s.site_pos) + 1, dtype=np.int32)
    return s


SYSTEMS = {"ranges": (_many_types, "lists=64"),
           "lists": (lambda: configs.graphite_cell(reps=(6, 6, 1), kmesh=(1, 1, 1), jitter=0.02),
                     "lists=48")}


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_limit_covers_ranges_and_lists(imago_lib, monkeypatch, name):
    import torch
    make, limit = SYSTEMS[name]
    s = make()
    used, mats = {}, {}
    for tuning in ("lists=off", limit, ""):
        monkeypatch.setenv("IMAGO_TUNING", tuning)
        intg.trim_memory(0)
        free0 = torch.cuda.mem_get_info()[0]
        with intg.IntegralSetup(s) as g:
            intg.trim_memory(0)
            used[tuning] = free0 - torch.cuda.mem_get_info()[0]
            g.gauss_overlap_ol()
            mats[tuning] = g.elec_pot_gauss_overlap_range(0, 1)
    assert used[""] > used["lists=off"] + 2 * _STEP  # the limit is below what they need
    assert used[limit] <= used["lists=off"] + _STEP
    for m in mats.values():
        assert packed_mismatch(m, mats[""])[1] == 0
