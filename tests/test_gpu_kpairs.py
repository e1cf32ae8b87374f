"""Builds over k-point lists that hold each other's negatives.

Of two k-points k and -k (up to a reciprocal lattice vector) only one is
summed and orthogonalised, the other's matrices being its conjugates.  Every
matrix is compared here with the build of each k-point alone, where nothing
is paired, on lists with paired, self-negative, unpaired and repeated points.
"""
import numpy as np
import pytest

from conftest import packed_mismatch
from imago_b200 import configs, intg
from imago_b200.system import kpoint_mesh

pytestmark = pytest.mark.gpu

_R = np.random.default_rng(3).uniform(-0.5, 0.5, size=(5, 3))
LISTS = {
    "mesh_2x2x2_shifted": kpoint_mesh((2, 2, 2), (0.5, 0.5, 0.5)),
    "mesh_3x3x1_shifted": kpoint_mesh((3, 3, 1), (0.5, 0.5, 0.5)),
    "mesh_4x3x1_centred": kpoint_mesh((4, 3, 1)),
    "mesh_5x7x1_shifted": kpoint_mesh((5, 7, 1), (0.5, 0.5, 0.0)),
    "no_pairs": np.abs(_R) * 0.9 + 0.01,
    "pairs_out_of_order": np.concatenate([_R, -_R[::-1]]),
    "pairs_up_to_a_lattice_vector": np.concatenate([_R, [1.0, 0.0, -2.0] - _R]),
    # two equal points share one negative; Gamma and 1/2 are their own
    "repeated_and_self_negative": np.concatenate(
        [_R[:1], _R[:1], -_R[:1], np.zeros((2, 3)), [[0.5, 0.5, 0.5], [-0.5, 0.5, 0.0]]]),
}


def _all(s):
    with intg.IntegralSetup(s) as g:
        out = g.build(intg.IMAGO_OL | intg.IMAGO_KE | intg.IMAGO_NP | intg.IMAGO_EP |
                      intg.IMAGO_MV)
        out["mm"] = g.gauss_overlap_mm()
        out["dm"] = g.gauss_overlap_dm([0.3, 0.1, -0.2])
        out["kov"] = np.stack(g.gauss_koverlap(np.diag([0.2, 0.1, 0.3])))
        out["ham"] = g.ham_pscf(np.linspace(-1.0, 1.0, 2 * g.pot_dim).reshape(-1, 2), rel=True)
    return out


_AXIS = {"ol_packed": 0, "ol_cv_re": 0, "ol_cv_im": 0, "ke_packed": 0, "np_packed": 0,
         "mv_packed": 0, "ep_packed": 1, "mm": 1, "dm": 1, "ham": 1, "kov": 2}


@pytest.mark.parametrize("name", sorted(LISTS))
@pytest.mark.parametrize("make", [configs.small_test_system, configs.no_core_test_system])
def test_paired_k_points_equal_the_build_of_each_alone(imago_lib, name, make):
    s = make()
    s.kmesh = None
    s.kpoints_abc = LISTS[name]
    got = _all(s)
    for k, f in enumerate(LISTS[name]):
        s.kpoints_abc = f[None]
        one = _all(s)
        for key, axis in _AXIS.items():
            if make is configs.no_core_test_system and key.startswith("ol_cv"):
                continue
            a = np.take(got[key], k, axis=axis)
            b = np.take(one[key], 0, axis=axis)
            # k and -k + G differ by the rounding of k.R (|k.R| < 100: 100 ulp
            # of 1, 2e-14) on matrix elements below 1e2
            assert packed_mismatch(a, b, atol=2e-12)[1] == 0, (key, k)
