"""Three-centre sums cut off by the lattice cell list.

The reference enumerates the images of a potential site from a list of lattice
vectors whose extent follows from the first exponent of each atom and
potential type (lattice.f90:310-469) and, along each axis, from the length of
the lattice vector.  Where another exponent reaches further (a very diffuse
nuclear exponent, potential exponents that do not ascend) or the cell is
skewed, its sums end with the list, and so must every kernel's.
"""
import numpy as np
import pytest

import oracle
from conftest import packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu


def _nuclear(alpha):
    s = configs.no_core_test_system()
    for p in s.pot_types:
        p.nuc_alpha = alpha
    return s


def _neutral():
    # neutral sites have no nuclear term, whatever their exponent
    s = configs.small_test_system()
    s.pot_types[1].nuc_charge = 0.0
    s.pot_types[1].nuc_alpha = 1e-12
    return s


def _descending():
    s = configs.small_test_system()
    for p in s.pot_types:
        p.alphas = np.sort(p.alphas)[::-1].copy()
        p.alphas[-1] = 0.03
    return s


def _skewed(make):
    # 17 degrees between the first two vectors: the list's box along them
    # leaves out vectors within its own radius
    s = make()
    a, b, c = s.real_vectors
    s.real_vectors = np.array([a, a + 0.3 * b, c])
    return s


def _flat():
    # a skewed cell whose list is long enough all the same: half its longest
    # diagonal overstates the distance to the nearest lattice point
    s = configs.no_core_test_system()
    a, b, c = s.real_vectors
    s.real_vectors = np.array([a, b + 1.25 * a, c])
    return s


SYSTEMS = {"nuclear": lambda: _nuclear(0.05), "far_nuclear": lambda: _nuclear(1e-7),
           "neutral": _neutral, "descending": _descending, "flat": _flat,
           "skewed": lambda: _skewed(configs.small_test_system),
           "skewed_f": lambda: _skewed(configs.f_test_system)}


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_sums_end_with_the_cell_list(imago_lib, name):
    s = SYSTEMS[name]()
    # sites off the atoms: halfway between an atom and its own image two images
    # of the atom's site are equally close, and rounding says from which of them
    # the list is walked
    s.pot_site_pos = s.pot_site_pos + np.random.default_rng(8).normal(
        0.0, 0.1, size=np.shape(s.pot_site_pos))
    ob = oracle.OracleBuild(s)
    ob.overlap()
    ref_np = ob.nuclear()
    count_np = ob.last_counts()[2]
    ref_ep = ob.elec_pot()
    count_ep = ob.last_counts()[2]
    coeffs = np.stack([np.sin(1.0 + np.arange(ob.pot_dim)), np.cos(np.arange(ob.pot_dim))], 1)
    ref_ham = ob.ham_pscf(coeffs)
    for schedule in ("per_class", "pairs", "queue"):
        with intg.IntegralSetup(s) as g:
            g.set_schedule(schedule)
            g.gauss_overlap_ol()
            assert packed_mismatch(g.gauss_overlap_np(), ref_np)[1] == 0
            assert packed_mismatch(g.elec_pot_gauss_overlap(), ref_ep)[1] == 0
            for mode in ("auto", "blocks"):
                g.set_ham_mode(mode)
                assert packed_mismatch(g.ham_pscf(coeffs), ref_ham)[1] == 0
            if not name.endswith("_f"):  # f classes are not counted
                assert int(g.count_triples(intg.IMAGO_NP).sum()) == count_np
            # the reference leaves out pairs that the term before did not reach
            if not name.endswith("_f") and name != "descending":
                assert int(g.count_triples(intg.IMAGO_EP).sum()) == count_ep
