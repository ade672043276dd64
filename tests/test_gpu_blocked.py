"""The row-blocked stored product (long rows, 2^16 rows and more, below the
split product's line): the row kernel's bits, whatever ran before it."""
import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed

pytestmark = pytest.mark.gpu


def one_level(N, norb, lz):
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(N, norb, twoLz=lz)
    H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb, ed.odd_coulomb_list(norb)))
    return H


# just past the line (one row in the last block of eight), seven rows in the
# last block, and the smallest long-row sector that is split instead
@pytest.mark.parametrize("case", [(9, 26, 1), (9, 27, 0), (10, 26, 0), (11, 32, 1)])
def test_default_product_gives_the_row_kernels_bits(cuda, case):
    torch = cuda
    H = one_level(*case)
    n = H.GetDimension()
    assert n >= 1 << 16
    rng = np.random.default_rng(n)
    for x in (rng.uniform(-1, 1, n), rng.standard_normal(n) * 10.0 ** rng.integers(-8, 3, n), np.eye(1, n, n - 1)[0]):
        xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        y, rows, again = (torch.full_like(xd, 7.0) for _ in range(3))
        product = ed.MatrixVectorFunction(H)
        product.Simple(xd, y)
        H.m_crsSparseMatrix.multiply(xd, rows, kernel=6)
        product.Simple(xd, again)
        torch.cuda.synchronize()
        assert torch.equal(y.view(torch.int64), rows.view(torch.int64))
        assert torch.equal(again.view(torch.int64), rows.view(torch.int64))
    xd[n // 2] = float("nan")
    product.Simple(xd, y)
    H.m_crsSparseMatrix.multiply(xd, rows, kernel=6)
    torch.cuda.synchronize()
    assert torch.isnan(y).all() and torch.isnan(rows).all()
