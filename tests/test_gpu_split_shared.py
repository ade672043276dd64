"""Operators on one set of term tables share the split product's plan and a
stream's scratch: products that two threads enqueue on one stream, or on their
own per-thread default streams, keep to their own vectors."""
import threading

import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed

pytestmark = pytest.mark.gpu

PER_THREAD = 2      # cudaStreamPerThread: one handle, a stream for each thread


@pytest.mark.parametrize("per_thread", [False, True])
def test_two_threads_on_one_set_of_terms(cuda, per_thread):
    torch = cuda
    N, norb = 8, 22
    tables = ed.QuarticTermTables(norb, ed.odd_coulomb_list(norb))
    hams, xs, ys, wanted = [], [], [], []
    for i in range(2):
        H = ed.SpinlessFermionHamiltonian()
        H.Initialize(N, norb, twoLz=0)
        H.Add_CdCdCC_Terms(tables, matrix_free=True)
        n = H.GetDimension()
        x = torch.from_numpy(np.random.default_rng(i).uniform(-1, 1, n)).cuda()
        y = torch.empty_like(x)
        ed.MatrixVectorFunction(H).Simple(x, y)
        torch.cuda.synchronize()
        hams.append(H)
        xs.append(x)
        wanted.append(y.clone())
        ys.append([torch.empty_like(x) for _ in range(100)])
    stream = PER_THREAD if per_thread else torch.cuda.Stream().cuda_stream
    torch.cuda.synchronize()
    start = threading.Barrier(2)

    def products(i):
        start.wait(30)
        for y in ys[i]:
            ed.MatrixVectorFunction(hams[i]).Simple(xs[i], y, stream=stream)

    threads = [threading.Thread(target=products, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
        assert not t.is_alive()
    torch.cuda.synchronize()
    for want, got in zip(wanted, ys):
        for y in got:
            assert torch.equal(y.view(torch.int64), want.view(torch.int64))
