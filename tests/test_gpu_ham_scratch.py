"""The PSCF Hamiltonian works in the scratch of the EP lane."""
import numpy as np
import pytest

from imago_b200 import configs, intg

pytestmark = pytest.mark.gpu


def _used(torch):
    intg.trim_memory(0)
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("spin", [1, 2])
def test_hamiltonian_needs_only_its_summed_blocks_beside_the_ep_scratch(imago_lib, spin):
    import torch
    s = configs.silicon_cubic8()
    with intg.IntegralSetup(s, outputs_on_device=True) as g:
        coeffs = np.ones((g.pot_dim, spin))
        mats = torch.empty((spin, g.nk, g.npacked, 2), dtype=torch.float64, device="cuda")
        g.build(intg.IMAGO_OL, out={"ol_packed": mats[0]})
        g.elec_pot_gauss_overlap_range(0, spin, out=mats)  # the EP lane's scratch
        before = _used(torch)
        g.ham_pscf(coeffs, rel=True, out=mats)
        grown = _used(torch) - before
        # a shell pair's block has at most 84 doubles; the pool grows in steps
        # of 32 MiB
        assert grown <= spin * g.num_shell_pairs * 84 * 8 + 2 ** 25 + 2 ** 20

