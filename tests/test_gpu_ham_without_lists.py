"""The PSCF Hamiltonian's walk without image lists, against the oracle."""
import numpy as np
import pytest

import oracle
from conftest import packed_mismatch
from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu

SYSTEMS = {"small": configs.small_test_system, "f": configs.f_test_system,
           "si8": lambda: configs.silicon_cubic8(kmesh=(1, 1, 1))}


@pytest.mark.parametrize("spin", [1, 2])
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_hamiltonian_without_image_lists_matches_oracle(imago_lib, monkeypatch, name, spin):
    s = SYSTEMS[name]()
    ob = oracle.OracleBuild(s)
    ob.overlap()
    coeffs = np.random.default_rng(11).normal(scale=0.5, size=(ob.pot_dim, spin))
    ref = ob.ham_pscf(coeffs, rel=True)
    monkeypatch.setenv("IMAGO_TUNING", "lists=off")
    with intg.IntegralSetup(s) as g:
        g.gauss_overlap_ol()
        for mode in ("fused", "fused1", "blocks"):
            g.set_ham_mode(mode)
            assert packed_mismatch(g.ham_pscf(coeffs, rel=True), ref)[1] == 0, mode
