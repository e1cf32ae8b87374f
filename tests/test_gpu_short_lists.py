"""Image lists of many potential types: short ones, ranked by a warp, and the
longer ones beside them.

A type of several sites against the same sites with a type each, whose
matrices add up to it; the nuclear term, which runs over every type, against
itself.
"""
import numpy as np
import pytest

from conftest import packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu


def _own_types(s, alphas):
    p = s.pot_types[0]
    n = len(s.pot_site_pos)
    s.pot_types = [configs.PotType(element=1, label=f"c{i}", nuc_charge=p.nuc_charge,
                                   nuc_alpha=p.nuc_alpha, alphas=alphas.copy()) for i in range(n)]
    s.pot_site_type = np.arange(1, n + 1, dtype=np.int32)
    return s


# cells of 6.7 bohr by 6.7 by 6.7 to 33.7: lists of a site's images from some
# 150 down to some 25, those of the most diffuse pairs on either side of 32
@pytest.mark.parametrize("reps", [(1, 1, 1), (1, 1, 2), (1, 1, 4), (1, 1, 5), (2, 2, 2)])
def test_types_per_site_add_up_to_the_shared_type(imago_lib, reps):
    make = lambda: configs.cubic_supercell("diamond", reps=reps, kmesh=(1, 1, 1))
    s = make()
    alphas = s.pot_types[0].alphas[[0, 9]]
    s.pot_types[0].alphas = alphas.copy()
    with intg.IntegralSetup(s) as g:
        g.gauss_overlap_ol()
        nuc, ep = g.gauss_overlap_np(), g.elec_pot_gauss_overlap()
    own = _own_types(make(), alphas)
    n = len(own.pot_types)
    with intg.IntegralSetup(own) as g:
        g.gauss_overlap_ol()
        assert packed_mismatch(g.gauss_overlap_np(), nuc)[1] == 0
        each = g.elec_pot_gauss_overlap().reshape((n, 2) + ep.shape[1:])
    # every matrix zeroes its own elements below 1e-10
    assert np.abs(each.sum(axis=0) - ep).max() <= 1e-10 * (n + 1)
