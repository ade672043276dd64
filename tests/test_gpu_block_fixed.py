"""The integer block product: exact sums of fixed-point weights and vectors,
so each column has the bits of its Hamiltonian's own fixed-point product."""
import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed

pytestmark = pytest.mark.gpu


def lists(K, count):
    out = []
    for v1 in np.linspace(0.5, 3.0, count):
        v = ed.odd_coulomb_list(K)
        v[1] = v1
        out.append(v)
    return out


# every tile (4, 8, 16, 32 Hamiltonians a row) full, partial and more than
# one, rows that start and end at any offset in a block of eight, a row count
# below a block's
@pytest.mark.parametrize("case,count", [((4, 10, 0), 1), ((5, 13, 2), 3), ((6, 16, 0), 4), ((6, 16, 4), 5), ((7, 19, 0), 8),
                                        ((7, 18, 1), 9), ((8, 20, 0), 16), ((8, 21, 2), 17), ((6, 16, 2), 32), ((7, 18, 3), 45),
                                        ((5, 13, 0), 256)])
def test_block_product_gives_the_single_products_bits(cuda, case, count):
    torch = cuda
    N, norb, lz = case
    basis = ed.FermionFockBasis()
    assert not basis.GenerateFockSpace(N, norb, lz)
    n = basis.GetStoredDimension()
    vs = lists(norb, count)
    batch = ed.HamiltonianBatch(basis, vs, autotune=False)
    rng = np.random.default_rng(count)
    X = torch.from_numpy(rng.standard_normal((n, count)) * 10.0 ** rng.integers(-6, 3, (1, count))).cuda()
    Y = torch.full_like(X, 7.0)
    batch.spmm(X, Y)
    torch.cuda.synchronize()
    for b in sorted({0, count // 3, count - 1}):
        H = ed.SpinlessFermionHamiltonian()
        H.Initialize(N, norb, twoLz=lz)
        H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb, vs[b]))
        x = X[:, b].contiguous()
        y = torch.empty_like(x)
        H.m_crsSparseMatrix.multiply(x, y, kernel=6)
        torch.cuda.synchronize()
        got, want = Y[:, b].contiguous().cpu().numpy(), y.cpu().numpy()
        assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), b


def test_non_finite_entries_stay_in_the_rows_they_meet(cuda):
    torch = cuda
    basis = ed.FermionFockBasis()
    basis.GenerateFockSpace(6, 16, 0)
    n = basis.GetStoredDimension()
    batch = ed.HamiltonianBatch(basis, lists(16, 6), autotune=False)
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(6, 16, twoLz=0)
    H.Add_CdCdCC_Terms(ed.QuarticTermTables(16, lists(16, 6)[2]))
    rowptr, col, _ = H.m_crsSparseMatrix.to_host()
    X = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, (n, 6))).cuda()
    Y = torch.empty_like(X)
    X[7, 2] = float("nan")
    batch.spmm(X, Y)
    torch.cuda.synchronize()
    bad = ~np.isfinite(Y.cpu().numpy())
    hit = np.zeros(n, bool)
    hit[np.repeat(np.arange(n), np.diff(rowptr))[col == 7]] = True
    assert np.array_equal(bad[:, 2], hit)
    assert not bad[:, [0, 1, 3, 4, 5]].any()
