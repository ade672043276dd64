"""Hamiltonians that the split product's plan or the block product's fixed-point
operands do not take: the FP64 kernels answer."""
import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed

pytestmark = pytest.mark.gpu


def tables(K, diagonal=True):
    t = ed.QuarticTermTables(K, ed.odd_coulomb_list(K))
    if diagonal:
        return t
    # no direct or exchange terms: the weights are the largest entries, and a
    # row of 64 and more of them could overflow the high limbs' sum
    k4, k3, k2 = np.indices((K, K, K))
    v = t.m_vTable.reshape(K, K, K).copy()
    v[(k2 == k3) | (k2 == k4)] = 0.0
    return ed.QuarticTermTables(K, ktable=t.m_kTable, vtable=v.ravel())


# rows of up to 30 * 29 / 2 * 17 + 1 > 2,048 elements by the plan's bound; weights above the diagonal
@pytest.mark.parametrize("N,norb,diagonal", [(30, 34, True), (8, 20, False)])
def test_matrix_free_without_a_plan(cuda, N, norb, diagonal):
    torch = cuda
    t = tables(norb, diagonal)
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(N, norb, twoLz=0)
    H.Add_CdCdCC_Terms(t)
    n = H.GetDimension()
    x = torch.from_numpy(np.random.default_rng(N).uniform(-1, 1, n)).cuda()
    want, y = torch.empty_like(x), torch.empty_like(x)
    H.m_crsSparseMatrix.multiply(x, want, kernel=1)
    F = ed.SpinlessFermionHamiltonian()
    F.Initialize(N, norb, twoLz=0)
    F.Add_CdCdCC_Terms(t, matrix_free=True)
    ed.MatrixVectorFunction(F).Simple(x, y)
    torch.cuda.synchronize()
    assert n > 100 and float((y - want).abs().max()) <= 1e-13 * float(want.abs().max())
    # FP64 it was: a choice of FP64 changes no bit
    z = torch.empty_like(x)
    t.set_fp64()
    ed.MatrixVectorFunction(F).Simple(x, z)
    torch.cuda.synchronize()
    assert torch.equal(y.view(torch.int64), z.view(torch.int64))
