"""Builds over k-point lists that hold nothing but Gamma points.

Every matrix is real then, but there are as many of them as points, and up to
eight points share the register phase sum with a single Gamma point.
"""
import numpy as np
import pytest

from conftest import packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu

_AXIS = {"ol_packed": 0, "ol_cv_re": 0, "ol_cv_im": 0, "ke_packed": 0, "np_packed": 0,
         "mv_packed": 0, "ep_packed": 1, "ep_range": 1, "mm": 1, "dm": 1, "ham": 1, "kov": 2}


def _all(s):
    with intg.IntegralSetup(s) as g:
        out = g.build(intg.IMAGO_OL | intg.IMAGO_KE | intg.IMAGO_NP | intg.IMAGO_EP |
                      intg.IMAGO_MV)
        out["ep_range"] = g.elec_pot_gauss_overlap_range(1, 2)
        out["mm"] = g.gauss_overlap_mm()
        out["dm"] = g.gauss_overlap_dm([0.3, 0.1, -0.2])
        out["kov"] = np.stack(g.gauss_koverlap(np.diag([0.2, 0.1, 0.3])))
        out["ham"] = g.ham_pscf(np.linspace(-1.0, 1.0, 2 * g.pot_dim).reshape(-1, 2), rel=True)
    return out


@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("make", [configs.small_test_system, configs.no_core_test_system])
def test_every_gamma_point_of_a_list_is_written(imago_lib, make, n):
    s = make()
    s.kmesh = None
    s.kpoints_abc = np.zeros((1, 3))
    one = _all(s)
    s.kpoints_abc = np.zeros((n, 3))
    got = _all(s)
    for key, axis in _AXIS.items():
        if make is configs.no_core_test_system and key.startswith("ol_cv"):
            continue
        assert np.any(np.take(one[key], 0, axis=axis)) or key == "ol_cv_im"
        for k in range(n):
            # the same real sums, in another order from nine points on: a
            # hundred images at most, elements below 1e2
            a, b = np.take(got[key], k, axis=axis), np.take(one[key], 0, axis=axis)
            assert packed_mismatch(a, b, atol=2e-12)[1] == 0, (key, k)
