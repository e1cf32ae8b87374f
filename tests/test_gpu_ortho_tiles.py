"""The tiled orthogonalisation at the edges of its two tile sizes: 32 x 32 up
to a valence dimension of 511, 64 x 64 from there, with core dimensions that
end inside a stage and matrices that end inside a tile."""
import numpy as np
import pytest

import oracle
from conftest import packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu


def _diamond(reps, atoms, kmesh):
    """The first `atoms` sites of a diamond supercell (4 valence and 1 core
    state each)."""
    s = configs.cubic_supercell("diamond", reps=reps, kmesh=kmesh or (1, 1, 1))
    s.site_type, s.site_pos = s.site_type[:atoms], s.site_pos[:atoms]
    s.pot_site_type, s.pot_site_pos = s.pot_site_type[:atoms], s.pot_site_pos[:atoms]
    if kmesh is None:
        s.kpoints_abc = np.zeros((1, 3))
    return s


@pytest.mark.parametrize("kmesh", [None, (1, 1, 2)])
@pytest.mark.parametrize("reps,atoms", [((3, 2, 1), 41), ((4, 4, 1), 127), ((4, 4, 1), 128),
                                        ((3, 3, 2), 143)])
def test_two_centre_builds_match_oracle(imago_lib, reps, atoms, kmesh):
    s = _diamond(reps, atoms, kmesh)
    assert s.vale_dim == 4 * atoms and s.core_dim == atoms
    ob = oracle.OracleBuild(s)
    ref_ol, ref_re, ref_im = ob.overlap()
    ref_ke = ob.kinetic()
    with intg.IntegralSetup(s) as g:
        ol, re, im = g.gauss_overlap_ol()
        ke = g.gauss_overlap_ke()
    for a, b in ((ol, ref_ol), (re, ref_re), (im, ref_im), (ke, ref_ke)):
        assert packed_mismatch(a, b)[1] == 0
