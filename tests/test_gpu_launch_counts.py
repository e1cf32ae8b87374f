"""kernel_stats() counts the kernels a call launches, whichever routes it takes.

Si8 has shell pairs of four classes (p-p, p-d, d-p, d-d): a launch each of the
two-centre, nuclear and Hamiltonian kernels, one of the merged EP kernel or the
work queue; then one contraction, one phase sum and one fused
orthogonalisation per kind.
"""
import numpy as np
import pytest

from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu


def _matrices(torch, g):
    P = lambda *n: torch.empty(n + (g.nk, g.npacked, 2), dtype=torch.float64, device="cuda")
    return {"ol_packed": P(), "ke_packed": P(), "np_packed": P(), "ep_packed": P(g.pot_dim)}


@pytest.mark.parametrize("schedule,ep", [("pairs", 1), ("queue", 1), ("per_class", 4)])
def test_launches_of_a_silicon_build(imago_lib, schedule, ep):
    import torch
    s = configs.silicon_cubic8(kmesh=(2, 2, 2))
    with intg.IntegralSetup(s, outputs_on_device=True) as g:
        g.set_schedule(schedule)
        g.set_ortho_schedule("per_item")
        out = _matrices(torch, g)
        g.build(out=out)  # measures the contraction
        for which, prim in ((intg.IMAGO_OL, 4), (intg.IMAGO_KE, 4), (intg.IMAGO_NP, 4),
                            (intg.IMAGO_EP, ep)):
            g.build(which, out=out)
            assert g.kernel_stats()[1] == prim + 3
        for _ in range(2):  # captured, then replayed
            g.build_graph(out)
        assert g.kernel_stats()[1] == 12 + ep + 4 * 3
        ham = torch.empty((2,) + out["ol_packed"].shape, dtype=torch.float64, device="cuda")
        for spin in (1, 2):
            for rel in (False, True):
                g.ham_pscf(np.ones((g.pot_dim, spin)), rel=rel, out=ham[:spin])
                # kinetic, nuclear and potential blocks, their sum, then as above
                assert g.kernel_stats()[1] == 12 + 4 * rel + 1 + 3


def test_f_classes_of_the_nuclear_term_are_one_launch(imago_lib):
    # classes of p, d and f exponents: four without f, five with
    import torch
    s = configs.f_test_system()
    with intg.IntegralSetup(s, outputs_on_device=True) as g:
        g.set_ortho_schedule("per_item")
        out = _matrices(torch, g)
        g.build(intg.IMAGO_OL, out=out)
        g.build(intg.IMAGO_NP, out=out)
        assert g.kernel_stats()[1] == 4 + 1 + 3
