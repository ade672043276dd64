"""Vectors with entries far below their largest one.  Products that ran in FP64
before they were fixed point (matrix-free, block products, the upper triangle
of large sectors, short rows of small ones) lose no entry: where fixed point
would make one zero the FP64 kernel runs, and every row, however small, is as
accurate as its own FP64 sum."""
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


class _Array:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def csr(torch, H):
    """The full-storage matrix of H and its rows' lengths, in torch."""
    n, nnz, upper = H.m_crsSparseMatrix.info()
    assert not upper
    r, c, v = H.m_crsSparseMatrix.device_arrays()
    r, c, v = (torch.as_tensor(_Array(p, k, t), device="cuda").clone() for p, k, t in ((r, n + 1, "<i8"), (c, nnz, "<i4"), (v, nnz, "<f8")))
    return torch.sparse_csr_tensor(r, c.to(torch.int64), v, (n, n)), torch.diff(r)


def graded(n, seed, floor):
    """Entries of about the floor, one of 1."""
    x = np.random.default_rng(seed).uniform(-floor, floor, n)
    x[n // 2] = 1.0
    return x


def assert_rows(torch, A, lengths, x, y):
    """Each row within the bound of an FP64 sum of its elements, in any order (both sides' twice)."""
    scale = torch.sparse_csr_tensor(A.crow_indices(), A.col_indices(), A.values().abs(), A.shape) @ x.abs()
    err = (y - A @ x).abs()
    assert bool((err <= 2.0 * (lengths + 2) * 2.0 ** -52 * scale).all()), float((err / scale).max())


def product(torch, H, x):
    y = torch.full_like(x, 7.0)
    ed.MatrixVectorFunction(H).Simple(x, y)
    torch.cuda.synchronize()
    return y


# 2^-58 is 3.5e-18: all but one entry are lost, or every other one is
@pytest.mark.parametrize("floor", [1e-22, 2e-18])
@pytest.mark.parametrize("make,case,kw", [(one_level, (8, 22, 0), dict(matrix_free=True)), (one_level, (9, 26, 1), dict(matrix_free=True)),
                                          (one_level, (8, 22, 0), {}), (two_level, (6, 13, 0), {}),
                                          (two_level, (8, 18, 2), dict(store_upper=True))])
def test_products_lose_no_entry(cuda, make, case, kw, floor):
    torch = cuda
    full = make(*case)
    A, lengths = csr(torch, full)
    x = torch.from_numpy(graded(len(lengths), 1, floor)).cuda()
    H = make(*case, **kw) if kw else full
    assert_rows(torch, A, lengths, x, product(torch, H, x))
    x = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, len(lengths))).cuda()
    assert_rows(torch, A, lengths, x, product(torch, H, x))      # nothing of it stays


@pytest.mark.parametrize("count", [1, 5])
def test_block_product_loses_no_entry(cuda, count):
    torch = cuda
    N, norb = 8, 20
    basis = ed.FermionFockBasis()
    basis.GenerateFockSpace(N, norb, 0)
    vs = [ed.odd_coulomb_list(norb) for _ in range(count)]
    for v, v1 in zip(vs, np.linspace(0.5, 3.0, count)):
        v[1] = v1
    bt = ed.HamiltonianBatch(basis, vs, autotune=False)
    X = np.random.default_rng(3).uniform(-1, 1, (bt.n, count))
    X[:, count - 1] = graded(bt.n, 4, 1e-22)
    X = torch.from_numpy(X).cuda()
    Y = torch.empty_like(X)
    bt.spmm(X, Y)
    torch.cuda.synchronize()
    for b in {0, count - 1}:
        H = ed.SpinlessFermionHamiltonian()
        H.Initialize(N, norb, twoLz=0)
        H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb, vs[b]))
        A, lengths = csr(torch, H)
        assert_rows(torch, A, lengths, X[:, b].contiguous(), Y[:, b].contiguous())


def test_a_solve_from_a_graded_vector(cuda):
    H = one_level(8, 22, 0)
    n = H.GetDimension()
    assert H.LanczosDiagonalize(3, tol=1e-10, v0=np.random.default_rng(5).uniform(-1, 1, n))
    want = H.m_eigenvalues
    assert H.LanczosDiagonalize(3, tol=1e-10, v0=graded(n, 6, 1e-22))
    assert np.max(np.abs(H.m_eigenvalues - want)) <= 1e-10 * np.abs(want).max()


def assert_default_bound(torch, A, lengths, x, y):
    """The bound that ed_capi.h states for the fixed-point products, beside the comparison's own FP64 sums."""
    a, ones = torch.sparse_csr_tensor(A.crow_indices(), A.col_indices(), A.values().abs(), A.shape), torch.ones_like(x)
    pattern = torch.sparse_csr_tensor(A.crow_indices(), A.col_indices(), torch.ones_like(A.values()), A.shape)
    scale = a @ x.abs()
    bound = 2.0 ** -58 * (x.abs().max() * (a @ ones) + A.values().abs().max() * (pattern @ x.abs())) + 2.0 ** -53 * y.abs()
    assert bool(((y - A @ x).abs() <= bound + (lengths + 2) * 2.0 ** -52 * scale).all())


def levelled(n, seed, level):
    """Entries of the level to within a factor of two, one of 1: none is lost, all keep few bits."""
    r = np.random.default_rng(seed)
    x = level * r.uniform(0.5, 1.0, n) * r.choice([-1.0, 1.0], n)
    x[n // 2] = 1.0
    return x


# entries that fixed point keeps to a few bits: the handles' FP64 choice keeps all of them
@pytest.mark.parametrize("make,case,kw", [(one_level, (8, 22, 0), dict(matrix_free=True)), (one_level, (9, 26, 1), {}),
                                          (two_level, (6, 13, 0), {}), (two_level, (7, 15, 0), {}),
                                          (two_level, (8, 18, 2), {}), (two_level, (8, 18, 2), dict(store_upper=True))])
def test_products_in_fp64_by_choice(cuda, make, case, kw):
    torch = cuda
    full = make(*case)
    A, lengths = csr(torch, full)
    x = torch.from_numpy(levelled(len(lengths), 7, 1e-15)).cuda()
    H = make(*case, **kw) if kw else full
    handle = H.m_terms if H.m_crsSparseMatrix is None else H.m_crsSparseMatrix
    default = product(torch, H, x)
    assert_default_bound(torch, A, lengths, x, default)
    handle.set_fp64()
    assert_rows(torch, A, lengths, x, product(torch, H, x))
    handle.set_fp64(False)
    assert torch.equal(product(torch, H, x).view(torch.int64), default.view(torch.int64))


def test_solves_in_fp64_by_choice(cuda):
    for kw in ({}, dict(matrix_free=True)):
        H = one_level(8, 22, 0, **kw)
        v0 = np.random.default_rng(8).uniform(-1, 1, H.GetDimension())
        assert H.LanczosDiagonalize(3, tol=1e-10, v0=v0)
        want = H.m_eigenvalues
        (H.m_terms if kw else H.m_crsSparseMatrix).set_fp64()
        assert H.LanczosDiagonalize(3, tol=1e-10, v0=v0)
        assert np.max(np.abs(H.m_eigenvalues - want)) <= 1e-11 * np.abs(want).max()


def test_block_product_in_fp64_by_choice(cuda):
    torch = cuda
    N, norb = 8, 20
    basis = ed.FermionFockBasis()
    basis.GenerateFockSpace(N, norb, 0)
    v = ed.odd_coulomb_list(norb)
    bt = ed.HamiltonianBatch(basis, [v, v, v], autotune=False)
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(N, norb, twoLz=0)
    H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb, v))
    A, lengths = csr(torch, H)
    X = torch.from_numpy(np.stack([levelled(bt.n, i, 1e-15) for i in range(3)], 1)).cuda()
    Y = torch.empty_like(X)
    bt.spmm(X, Y)
    torch.cuda.synchronize()
    assert_default_bound(torch, A, lengths, X[:, 1].contiguous(), Y[:, 1].contiguous())
    bt.set_fp64()
    bt.spmm(X, Y)
    torch.cuda.synchronize()
    assert_rows(torch, A, lengths, X[:, 1].contiguous(), Y[:, 1].contiguous())
    want, _, _ = bt.solve(2, V0=X)
    bt.set_fp64(False)
    got, _, _ = bt.solve(2, V0=X)
    assert np.max(np.abs(got - want)) <= 1e-11 * np.abs(want).max()
