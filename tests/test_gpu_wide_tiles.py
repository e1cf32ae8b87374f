"""The 64 x 64 tiles of the tiled orthogonalisation (valence dimensions from
512) in every form a build uses: several terms in one launch, the form with a
Hermitian core block and the general one (momentum, dipole), complex matrices
at Gamma (momentum) and the whole matrix (plane-wave overlap); and, just below,
the same with 32 x 32 tiles."""
import numpy as np
import pytest

import oracle
from conftest import ATOL, packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu


def _diamond(reps, atoms, kmesh):
    s = configs.cubic_supercell("diamond", reps=reps, kmesh=kmesh or (1, 1, 1))
    s.site_type, s.site_pos = s.site_type[:atoms], s.site_pos[:atoms]
    s.pot_site_type, s.pot_site_pos = s.pot_site_type[:atoms], s.pot_site_pos[:atoms]
    if kmesh is None:
        s.kmesh = None
        s.kpoints_abc = np.zeros((1, 3))
    return s


@pytest.mark.parametrize("reps,atoms,kmesh", [((4, 4, 1), 127, None), ((4, 4, 1), 128, None),
                                              ((3, 3, 2), 143, None), ((3, 3, 2), 143, (1, 1, 2))])
def test_all_forms_match_oracle(imago_lib, reps, atoms, kmesh):
    s = _diamond(reps, atoms, kmesh)
    center, dk = [0.3, 0.1, -0.2], np.diag([0.2, 0.1, 0.3])
    ob = oracle.OracleBuild(s)
    ob.overlap()
    with intg.IntegralSetup(s) as g:
        assert g.vale_dim == 4 * atoms
        g.gauss_overlap_ol()
        last = g.pot_dim - 3
        pairs = {"ep": (g.elec_pot_gauss_overlap_range(last, 3), ob.elec_pot(last, last + 3)),
                 "np": (g.gauss_overlap_np(), ob.nuclear()),
                 "mm": (g.gauss_overlap_mm(), ob.momentum()),
                 "dm": (g.gauss_overlap_dm(center), ob.dipole(center))}
        re, im = g.gauss_koverlap(dk)
        kov = ob.koverlap(dk).transpose(0, 1, 3, 2)  # [axis, k, col, row]
    for key, (a, b) in pairs.items():
        assert packed_mismatch(a, b)[1] == 0, key
    # nothing of these is zeroed
    assert max(np.abs(re - kov.real).max(), np.abs(im - kov.imag).max()) <= ATOL
