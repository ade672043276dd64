"""ed_kernel_launches counts each launch once."""
import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed
from hamiltonian_diagonalization_gb300 import _capi as C

pytestmark = pytest.mark.gpu


def test_first_and_later_fixed_point_products(cuda):
    torch = cuda
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(8, 22, twoLz=0)
    H.Add_CdCdCC_Terms(ed.QuarticTermTables(22, ed.odd_coulomb_list(22)))
    x = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, H.GetDimension())).cuda()
    y = torch.empty_like(x)
    counts = []
    for _ in range(2):
        before = C.lib().ed_kernel_launches()
        H.m_crsSparseMatrix.multiply(x, y, kernel=6)
        counts.append(C.lib().ed_kernel_launches() - before)
    torch.cuda.synchronize()
    # the values' exponents, their bound and their copy; then x's copy and the product
    assert counts == [3 + 2, 2]
