"""Where device memory is short a product or solve takes the kernels that need
none instead of failing (ed_memory_limit stands in for a full device)."""
import contextlib

import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed
from hamiltonian_diagonalization_gb300 import _capi as C

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def memory(nbytes):
    C.lib().ed_memory_limit(int(nbytes))
    try:
        yield
    finally:
        C.lib().ed_memory_limit(-1)


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


def product(torch, H, x, stream=None):
    y = torch.full_like(x, 7.0)
    ed.MatrixVectorFunction(H).Simple(x, y, stream=stream)
    torch.cuda.synchronize()
    return y


def close(torch, a, b):
    # two orders of FP64 sums of a few hundred elements, or one and the exact sum
    return float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())


def vector(torch, H, seed):
    x = torch.from_numpy(np.random.default_rng(seed).uniform(-1, 1, H.GetDimension())).cuda()
    torch.cuda.synchronize()
    return x


def test_matrix_free_without_room_for_the_plan(cuda):
    torch = cuda
    H = one_level(8, 22, 0, matrix_free=True)
    x = vector(torch, H, 1)
    with memory(1 << 20):     # the diagonal and the row kernel's tables fit
        y = product(torch, H, x)
        again = product(torch, H, x)
    want = product(torch, one_level(8, 22, 0, matrix_free=True), x)
    assert close(torch, y, want) and torch.equal(y, again)


def test_matrix_free_without_room_for_a_streams_scratch(cuda):
    torch = cuda
    H = one_level(8, 22, 0, matrix_free=True)
    x = vector(torch, H, 2)
    want = product(torch, H, x)
    s = torch.cuda.Stream()
    with memory(0):
        y = product(torch, H, x, stream=s.cuda_stream)
        assert torch.equal(product(torch, H, x), want)       # this stream has its scratch
    assert close(torch, y, want)
    assert torch.equal(product(torch, H, x, stream=s.cuda_stream), want)


# a sector of the row-blocked copy, short rows of a small one, the upper triangle of one that is split
@pytest.mark.parametrize("make,case,kw", [(one_level, (9, 26, 1), {}), (two_level, (6, 13, 0), {}),
                                          (two_level, (8, 18, 2), dict(store_upper=True)), (two_level, (8, 18, 2), {})])
def test_stored_products_without_room(cuda, make, case, kw):
    torch = cuda
    H = make(*case, **kw)
    x = vector(torch, H, 3)
    with memory(1 << 10):
        y = product(torch, H, x)
    want = product(torch, make(*case, **kw), x)
    assert close(torch, y, want)
    assert close(torch, product(torch, H, x), want)


# the plan is made after the basis vectors, which filled the device before there was one
@pytest.mark.parametrize("kw", [dict(matrix_free=True)])
def test_a_solve_that_fills_the_device(cuda, kw):
    torch = cuda
    H = one_level(10, 28, 0, **kw)
    n, nev = H.GetDimension(), 14
    m = 2 * nev + 21
    v0 = np.random.default_rng(5).uniform(-1, 1, n)
    assert H.LanczosDiagonalize(nev, tol=1e-10, v0=v0)
    want = H.m_eigenvalues
    K = one_level(10, 28, 0, **kw)
    basis = 2 * (m + 1) * n * 8
    # the diagonal, start vector, eigenvectors and a residual's product beside it, and 8 MB of tables
    with memory(basis + (3 + nev) * n * 8 + (8 << 20)):
        assert K.LanczosDiagonalize(nev, tol=1e-10, v0=v0)
    assert np.max(np.abs(K.m_eigenvalues - want)) <= 1e-11 * np.abs(want).max()


def sweep(N, norb, count):
    basis = ed.FermionFockBasis()
    basis.GenerateFockSpace(N, norb, 0)
    vs = []
    for v1 in np.linspace(0.5, 3.0, count):
        v = ed.odd_coulomb_list(norb)
        v[1] = v1
        vs.append(v)
    return ed.HamiltonianBatch(basis, vs, autotune=False)


def block(torch, bt, seed):
    X = torch.from_numpy(np.random.default_rng(seed).uniform(-1, 1, (bt.n, bt.nham))).cuda()
    torch.cuda.synchronize()
    return X


def test_block_product_without_room(cuda):
    torch = cuda
    X = block(torch, sweep(7, 19, 6), 6)
    Y, want = torch.empty_like(X), torch.empty_like(X)
    bt = sweep(7, 19, 6)
    with memory(1 << 12):
        bt.spmm(X, Y)
    sweep(7, 19, 6).spmm(X, want)
    torch.cuda.synchronize()
    assert close(torch, Y, want)
    first = sweep(7, 19, 6)
    first.spmm(X, Y)
    with memory(1 << 12):       # the operands are there, another stream's scratch is not
        first.spmm(X, Y, stream=torch.cuda.Stream().cuda_stream)
    torch.cuda.synchronize()
    assert close(torch, Y, want)


# the solve's own vectors, a second set of operands, and a residual's product: all that the FP64 products need
def test_a_batched_solve_that_fills_the_device(cuda):
    torch = cuda
    N, norb, count, nev = 9, 25, 16, 2
    bt = sweep(N, norb, count)
    X = block(torch, bt, 7)
    want, _, _ = bt.solve(nev, V0=X)
    m, vs = 2 * nev + 21, bt.n * count
    short = sweep(N, norb, count)
    with memory((2 * (m + 1) + nev + 3) * vs * 8 + (4 << 20)):
        got, _, info = short.solve(nev, V0=X)
    assert info["converged"] == count and np.max(np.abs(got - want)) <= 1e-11 * np.abs(want).max()


def held(torch):
    torch.cuda.synchronize()
    return -torch.cuda.mem_get_info()[0]


def test_solves_and_streams_leave_one_set_of_operands(cuda):
    torch = cuda
    N, norb, count = 9, 25, 16
    X = block(torch, sweep(N, norb, count), 8)
    Y = torch.empty_like(X)
    warm = sweep(N, norb, count)      # modules and the like
    warm.solve(2, V0=X)
    warm.spmm(X, Y)
    bt = sweep(N, norb, count)
    one, slack = bt.n * count * 8, 2 << 20      # a block of vectors; the allocator's granularity
    before = held(torch)
    for _ in range(3):
        bt.solve(2, V0=X)
    assert held(torch) - before <= slack
    bt.spmm(X, Y)
    torch.cuda.synchronize()
    first = held(torch)
    streams = [torch.cuda.Stream() for _ in range(3)]
    for s in streams:
        bt.spmm(X, Y, stream=s.cuda_stream)
        torch.cuda.synchronize()
    assert held(torch) - first <= len(streams) * (one + slack)
