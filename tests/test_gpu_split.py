"""The split products (matrix-free of every sector, stored ones of large
sectors): both sum the same fixed-point weights exactly and round once, so
they give the stored fixed-point kernels' bits."""
import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed

pytestmark = pytest.mark.gpu


def one_level(N, norb, lz, **kw):
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(N, norb, twoLz=lz)
    H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb, ed.odd_coulomb_list(norb)), **kw)
    return H


def two_level(N, norb0, lz, **kw):
    H = ed.TwoLevelSpinlessFermionHamiltonian()
    H.Initialize(N, 2 * norb0 + 2, twoLz=lz)
    H.Add_CdC_Terms(np.linspace(0.5, 1.0, norb0 + 2), 1, 1)
    for lv in (0, 1):
        H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb0 + 2 * lv, ed.odd_coulomb_list(norb0 + 2 * lv)), lv, lv, lv, lv, **kw)
    H.Build()
    return H


def product(torch, H, x):
    y = torch.full_like(x, 7.0)
    ed.MatrixVectorFunction(H).Simple(x, y)
    torch.cuda.synchronize()
    return y


def bits(t):
    return t.view(-1).cpu().numpy().view(np.uint64)


# segments of one row (4, 10), odd and even splits, off-centre sectors, fewer
# than 32 rows, more than 256 rows a segment (10, 32 and 9, 33), many holes
# (4, 40) and many particles (11, 16)
@pytest.mark.parametrize("case", [(4, 10, 0), (5, 13, 8), (6, 16, 4), (6, 16, 0), (7, 19, -6), (8, 22, 0), (11, 16, 5),
                                  (4, 40, 6), (9, 27, 40), (9, 33, 0), (10, 32, 0)])
def test_matrix_free_gives_the_stored_bits(cuda, case):
    torch = cuda
    N, norb, lz = case
    lz += (N * (norb - 1) - lz) % 2
    stored = one_level(N, norb, lz)
    free = one_level(N, norb, lz, matrix_free=True)
    n = stored.GetDimension()
    rng = np.random.default_rng(N * norb)
    for x in (rng.uniform(-1, 1, n), rng.standard_normal(n) * 10.0 ** rng.integers(-8, 3, n), np.eye(1, n, n // 2)[0]):
        xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        y = torch.empty_like(xd)
        stored.m_crsSparseMatrix.multiply(xd, y, kernel=6)
        torch.cuda.synchronize()
        assert np.array_equal(bits(product(torch, free, xd)), bits(y))


def test_matrix_free_keeps_non_finite_entries_to_their_rows(cuda):
    torch = cuda
    stored = one_level(7, 19, 0)
    free = one_level(7, 19, 0, matrix_free=True)
    rowptr, col, _ = stored.m_crsSparseMatrix.to_host()
    n = len(rowptr) - 1
    x = np.random.default_rng(3).uniform(-1, 1, n)
    clean = product(torch, free, torch.from_numpy(x).cuda()).cpu().numpy()
    bad = [5, n // 3]
    x[bad] = [np.nan, np.inf]
    y = product(torch, free, torch.from_numpy(x).cuda()).cpu().numpy()
    rows = np.repeat(np.arange(n), np.diff(rowptr))
    hit = np.zeros(n, bool)
    hit[rows[np.isin(col, bad)]] = True
    assert np.array_equal(~np.isfinite(y), hit)
    # the others as the row kernel's FP64 sums: at most nnz/row roundings of the row's magnitude
    assert np.max(np.abs(y[~hit] - clean[~hit])) <= 1e-13 * np.abs(clean).max()


# the smallest sectors past the line from which stored products are split
@pytest.mark.parametrize("make,case,kernel", [(one_level, (11, 31, 0), 6), (one_level, (12, 30, 0), 6), (two_level, (8, 18, 2), 8),
                                              (two_level, (9, 16, 3), 8)])
def test_large_stored_products_give_the_row_kernels_bits(cuda, make, case, kernel):
    torch = cuda
    H = make(*case)
    n = H.GetDimension()
    assert n >= 1 << 20
    x = torch.from_numpy(np.random.default_rng(n).uniform(-1, 1, n)).cuda()
    y = torch.empty_like(x)
    split = product(torch, H, x)
    H.m_crsSparseMatrix.multiply(x, y, kernel=kernel)
    torch.cuda.synchronize()
    assert np.array_equal(bits(split), bits(y))
    x[n // 5] = float("inf")
    assert bool(torch.isnan(product(torch, H, x)).all())
    x[n // 5] = 0.25
    if make is two_level:      # upper-triangle storage: the same operator
        U = make(*case, store_upper=True)
        H.m_crsSparseMatrix.multiply(x, y, kernel=kernel)
        torch.cuda.synchronize()
        assert np.array_equal(bits(product(torch, U, x)), bits(y))


def test_split_products_on_two_streams_and_in_a_solve(cuda):
    torch = cuda
    free = one_level(8, 22, 0, matrix_free=True)
    stored = one_level(8, 22, 0)
    n = free.GetDimension()
    xs = [torch.from_numpy(np.random.default_rng(i).uniform(-1, 1, n)).cuda() for i in range(2)]
    ys = [torch.empty_like(x) for x in xs]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for s, x, y in zip(streams, xs, ys):
        ed.MatrixVectorFunction(free).Simple(x, y, stream=s.cuda_stream)
    torch.cuda.synchronize()
    for x, y in zip(xs, ys):
        z = torch.empty_like(x)
        stored.m_crsSparseMatrix.multiply(x, z, kernel=6)
        torch.cuda.synchronize()
        assert np.array_equal(bits(y), bits(z))
    v0 = np.random.default_rng(9).uniform(-1, 1, n)
    assert free.LanczosDiagonalize(3, tol=1e-10, v0=v0) and stored.LanczosDiagonalize(3, tol=1e-10, v0=v0)
    assert np.array_equal(free.m_eigenvalues, stored.m_eigenvalues)


# what took FP64 sums before they were fixed point still keeps a NaN to the
# rows that meet it: the upper triangle of a large sector, short rows of a small one
@pytest.mark.parametrize("make,case,kw", [(two_level, (8, 18, 2), dict(store_upper=True)), (two_level, (6, 13, 0), {})])
def test_products_keep_a_nan_to_its_rows(cuda, make, case, kw):
    torch = cuda
    H = make(*case, **kw)
    rowptr, col, _ = H.m_crsSparseMatrix.to_host()
    n = len(rowptr) - 1
    x = torch.from_numpy(np.random.default_rng(5).uniform(-1, 1, n)).cuda()
    clean = product(torch, H, x).cpu().numpy()
    x[n // 2] = float("nan")
    y = product(torch, H, x).cpu().numpy()
    rows = np.repeat(np.arange(n), np.diff(rowptr))
    hit = np.zeros(n, bool)
    hit[rows[col == n // 2]] = True
    if kw:
        hit[col[rows == n // 2]] = True
    assert np.array_equal(np.isnan(y), hit)
    assert np.max(np.abs(y[~hit] - clean[~hit])) <= 1e-13 * np.abs(clean).max()
