"""Products captured by the caller: a graph may be replayed on any stream, so
what keeps a scratch per stream outside a capture (block products, short rows
of small sectors, upper-triangle storage of large ones) keeps none inside."""
import numpy as np
import pytest

import hamiltonian_diagonalization_gb300 as ed

pytestmark = pytest.mark.gpu


def two_level(N, norb0, lz, **kw):
    H = ed.TwoLevelSpinlessFermionHamiltonian()
    H.Initialize(N, 2 * norb0 + 2, twoLz=lz)
    H.Add_CdC_Terms(np.linspace(0.5, 1.0, norb0 + 2), 1, 1)
    for lv in (0, 1):
        H.Add_CdCdCC_Terms(ed.QuarticTermTables(norb0 + 2 * lv, ed.odd_coulomb_list(norb0 + 2 * lv)), lv, lv, lv, lv, **kw)
    H.Build()
    return H


def batch(N, norb, count):
    basis = ed.FermionFockBasis()
    basis.GenerateFockSpace(N, norb, 0)
    vs = []
    for v1 in np.linspace(0.5, 3.0, count):
        v = ed.odd_coulomb_list(norb)
        v[1] = v1
        vs.append(v)
    return ed.HamiltonianBatch(basis, vs, autotune=False)


def make(kind):
    if kind == "batch":
        bt = batch(7, 19, 6)
        return bt, (bt.n, 6), lambda x, y, s: bt.spmm(x, y, stream=s)
    H = two_level(8, 18, 2, store_upper=True) if kind == "upper" else two_level(6, 13, 0)
    n = H.GetDimension()
    assert n >= 1 << 20 if kind == "upper" else 4096 <= n < 32768
    f = ed.MatrixVectorFunction(H)
    return H, (n,), lambda x, y, s: f.Simple(x, y, stream=s)


@pytest.mark.parametrize("kind", ["batch", "short", "upper"])
@pytest.mark.parametrize("scratch", [False, True])
def test_graphs_of_one_stream_replay_side_by_side(cuda, kind, scratch):
    torch = cuda
    owner, shape, product = make(kind)
    rng = np.random.default_rng(11)
    xs = [torch.from_numpy(rng.uniform(-1, 1, shape)).cuda() for _ in range(2)]
    ys = [torch.zeros_like(x) for x in xs]
    capture = torch.cuda.Stream()
    torch.cuda.synchronize()
    if scratch:      # an ordinary product of the same stream before the capture
        product(xs[0], ys[0], capture.cuda_stream)
        torch.cuda.synchronize()
    graphs = []
    for x, y in zip(xs, ys):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=capture):
            product(x, y, capture.cuda_stream)
        graphs.append(g)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(5):
        for y in ys:
            y.fill_(7.0)
        torch.cuda.synchronize()
        for _ in range(4):
            for s, g in zip(streams, graphs):
                with torch.cuda.stream(s):
                    g.replay()
        torch.cuda.synchronize()
    for x, y in zip(xs, ys):
        want = torch.empty_like(x)
        product(x, want, None)
        torch.cuda.synchronize()
        # FP64 sums of up to 300 elements against the fixed-point ones
        assert float((y - want).abs().max()) <= 1e-13 * float(want.abs().max())
    del owner
