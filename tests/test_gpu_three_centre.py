"""The three-centre stage's walks over image lists.

The term-group kernel ("pairs" schedule) against one (shell pair, term) per
thread, the nuclear and Hamiltonian kernels' shared walks, and all of them
without the lists, on systems that reach each branch: potential exponents
that do not ascend, several potential types, more term groups than one
launch takes, images in plenty and hardly any, f classes.
"""
import numpy as np
import pytest

import oracle
from conftest import packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu


def _si_gamma():
    return configs.silicon_cubic8(kmesh=(1, 1, 1))


def _descending():
    s = configs.small_test_system()
    for p in s.pot_types:
        p.alphas = p.alphas[::-1].copy()
    return s


def _shuffled():
    s = configs.silicon_cubic8(kmesh=(1, 1, 1), npot=7)
    for p in s.pot_types:
        p.alphas = p.alphas[[3, 0, 6, 1, 5, 2, 4]].copy()
    return s


def _type_per_site():
    # 40 potential types of two terms: more groups than one launch's 64
    s = configs.cubic_supercell("diamond", reps=(1, 1, 5), kmesh=(1, 1, 1))
    p = s.pot_types[0]
    s.pot_types = [configs.PotType(element=1 + i, label=f"c{i}", nuc_charge=6.0,
                                   nuc_alpha=15.0 + i, alphas=p.alphas[[i % 7, 9]].copy())
                   for i in range(len(s.site_pos))]
    s.pot_site_type = np.arange(1, len(s.site_pos) + 1, dtype=np.int32)
    return s


SYSTEMS = {"small": configs.small_test_system, "f": configs.f_test_system, "si8": _si_gamma,
           "diamond2": lambda: configs.diamond_primitive(kmesh=(2, 1, 1)),
           "descending": _descending, "shuffled": _shuffled, "type_per_site": _type_per_site,
           "quartz9": lambda: configs.quartz_supercell(reps=(1, 1, 1), gamma=True)}


def _build(s, schedule):
    with intg.IntegralSetup(s) as g:
        g.set_schedule(schedule)
        g.gauss_overlap_ol()
        ke = g.gauss_overlap_ke()
        coeffs = np.sin(1.0 + np.arange(g.pot_dim))
        return {"ep": g.elec_pot_gauss_overlap(), "np": g.gauss_overlap_np(), "ke": ke,
                "ham": g.ham_pscf(coeffs), "coeffs": coeffs}


def _close(a, b, scale):
    # the same triples in another order, matrix elements zeroed below 1e-10
    # on one side only aside: rounding of the largest element
    d = np.abs(a - b)
    d[(np.abs(a) < 1.1e-10) & (np.abs(b) < 1.1e-10)] = 0.0
    assert d.max() <= 2e-14 * scale, d.max() / scale


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_term_groups_equal_one_term_per_thread(imago_lib, name):
    s = SYSTEMS[name]()
    a, b = _build(s, "pairs"), _build(s, "per_class")
    _close(a["ep"], b["ep"], np.abs(b["ep"]).max())
    assert np.array_equal(a["np"], b["np"])
    # the Hamiltonian's summed terms against the sum of the matrices
    w = a["coeffs"]
    ham = a["ke"] + a["np"] + np.tensordot(w, a["ep"], axes=1)
    scale = np.abs(a["ke"]).max() + np.abs(a["np"]).max() + \
        (np.abs(w) * np.abs(a["ep"]).max(axis=(1, 2, 3))).sum()
    # each matrix zeroes its own elements below 1e-10
    assert np.abs(a["ham"][0] - ham).max() <= 2e-14 * scale + 1e-10 * (len(w) + 3)


@pytest.mark.parametrize("schedule", ["pairs", "per_class", "queue"])
@pytest.mark.parametrize("name", ["small", "f", "si8"])
def test_without_image_lists(imago_lib, monkeypatch, name, schedule):
    # beyond the lists' memory limit every image of a type is tested, in
    # another order: against the oracle, within the builds' 1e-10 bar
    s = SYSTEMS[name]()
    monkeypatch.setenv("IMAGO_TUNING", "lists=off")
    got = _build(s, schedule)
    ob = oracle.OracleBuild(s)
    ob.overlap()
    assert packed_mismatch(got["np"], ob.nuclear())[1] == 0
    assert packed_mismatch(got["ep"], ob.elec_pot())[1] == 0


@pytest.mark.parametrize("schedule", ["per_item", "piped", "auto"])
def test_odd_valence_dimension_runs_under_every_orthogonalisation_schedule(imago_lib, schedule):
    # V = 87: the TMA-fed kernel's boxes would start off their 128 bytes, so
    # it does not take the system; the other one serves every schedule
    s = SYSTEMS["quartz9"]()
    assert s.vale_dim % 2 == 1
    ob = oracle.OracleBuild(s)
    ob.overlap()
    ref = ob.elec_pot()
    with intg.IntegralSetup(s) as g:
        g.set_ortho_schedule(schedule)
        g.gauss_overlap_ol()
        ep = g.elec_pot_gauss_overlap()
    assert packed_mismatch(ep, ref)[1] == 0
