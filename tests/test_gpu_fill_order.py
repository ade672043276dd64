"""The CRS fill that generates rows in column order, against the one that
sorts them."""
import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed

pytestmark = pytest.mark.gpu


def build(N, norb, lz, pp, upper):
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(N, norb, twoLz=lz)
    H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb, pp), store_upper=upper)
    return H.m_crsSparseMatrix.to_host()


# 32 and 33 orbitals (the word types), the most orbitals, one pair, a nearly
# and a wholly full shell, fewer than 32 and more than 32 x 8 pairs of orbitals
@pytest.mark.parametrize("case", [(4, 32, 0), (4, 33, 0), (3, 40, 1), (2, 9, 0), (20, 22, 1), (5, 5, 0), (3, 8, 1), (16, 20, 0)])
@pytest.mark.parametrize("zeros", [False, True])
def test_ordered_rows_are_the_sorted_rows(cuda, monkeypatch, case, zeros):
    N, norb, lz = case
    lz += (N * (norb - 1) - lz) % 2
    pp = ed.odd_coulomb_list(norb)
    if zeros:
        pp = [0.0] * len(pp)      # every weight zero: the rows keep what the threshold leaves
    for upper in (False, True):
        monkeypatch.delenv("ED_FILL_SORT", raising=False)
        a = build(N, norb, lz, pp, upper)
        monkeypatch.setenv("ED_FILL_SORT", "smem")
        b = build(N, norb, lz, pp, upper)
        for u, v in zip(a, b):
            assert np.array_equal(u.view(np.uint8), v.view(np.uint8))
        for r in range(len(a[0]) - 1):
            assert np.all(np.diff(a[1][a[0][r]:a[0][r + 1]]) > 0)
