"""The measured cases: calls that programs using this package make, over the
sizes of its configurations.  listed() is the fixed list, draw() gives further
cases of the same ranges, prepare() makes a call's inputs on the GPU, run()
makes the call, work() says what it has to move and compute, and exact() gives
its result by plain 64-bit torch without the package.

A case names its kind, the sector and the options of the call:

  product   y = H x with a stored matrix (model sphere: one level; two: two
            Landau levels; ofl: complex momentum sector); upper: the
            reference's upper-triangle storage
  matfree   y = H x with the elements regenerated from the term tables
  build     sector basis and full CRS from the term tables
  spmm      one block product of a pseudopotential sweep's Hamiltonians
  program   a small whole program: tables, basis, CRS, lowest eigenpairs to
            host arrays, pair correlations of the ground state
  solve     the same solve with start vector and eigenvectors in device memory
            (sphere), or through the complex model class (ofl)
  sweep     the lowest eigenpairs of every Hamiltonian of a sweep, in one batch

Vectors are determined up to their sign (phase): run() fixes it, as a program
that compares states does, by their overlap with the start vector.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

# The reference calls ARPACK with this tolerance, and so do the solves here.
TOL = 1e-12


def listed():
    return [
        # the smallest configuration's product: 8,512 states, launch latency
        dict(name="product-n8", kind="product", model="sphere", N=8, norb=22, lz=0, upper=False),
        # the stored-CRS configuration's product: 4.2 GB of matrix per call
        dict(name="product-n11", kind="product", model="sphere", N=11, norb=31, lz=0, upper=False),
        # the reference's own storage, an odd sector of the sweep's size
        dict(name="product-upper-n10", kind="product", model="sphere", N=10, norb=28, lz=2, upper=True),
        # two Landau levels: short rows, 2.0 million states
        dict(name="product-two-level", kind="product", model="two", N=8, norb=19, lz=0, upper=False),
        # optical flux lattice: complex elements
        dict(name="product-ofl", kind="product", model="ofl", N=10, dx=5, dy=6, kx=0, ky=0, upper=False),
        # matrix-free product at the stored configuration's size
        dict(name="matfree-n11", kind="matfree", model="sphere", N=11, norb=31, lz=0),
        # basis and CRS of one sector of the sweep configuration
        dict(name="build-n10", kind="build", model="sphere", N=10, norb=28, lz=4),
        # the sweep's block product, half its 64 Hamiltonians
        dict(name="spmm-n10-b32", kind="spmm", model="sphere", N=10, norb=28, lz=0, nham=32),
        # the smallest configuration as a whole program
        dict(name="program-n8", kind="program", model="sphere", N=8, norb=22, lz=0, nev=5),
        # the headline: time to 10 eigenpairs of the stored-CRS configuration
        dict(name="solve-n11", kind="solve", model="sphere", N=11, norb=31, lz=0, nev=10),
        # a complex sector's solve
        dict(name="solve-ofl", kind="solve", model="ofl", N=9, dx=4, dy=6, kx=0, ky=0, nev=4),
        # a batch of a sweep: 16 Hamiltonians of one sector
        dict(name="sweep-n9-b16", kind="sweep", model="sphere", N=9, norb=25, lz=0, nham=16, nev=4),
    ]


# (N, norb) of one-level sectors between a few hundred and 1.4 million states
_SPHERE = [(6, 16), (7, 18), (7, 19), (7, 21), (8, 20), (8, 21), (8, 22), (8, 23), (9, 23), (9, 24), (9, 25), (9, 26),
           (10, 26), (10, 27), (10, 28), (11, 28), (11, 29), (11, 30), (11, 31)]
# (N, norb0) of two-level sectors up to 2 million states
_TWO = [(5, 9), (5, 14), (6, 11), (6, 13), (6, 16), (7, 13), (7, 15), (7, 17), (8, 16), (8, 17), (8, 18)]
# (N, dimX, dimY) of complex sectors up to 1 million states
_OFL = [(6, 3, 5), (6, 4, 5), (7, 4, 5), (8, 4, 5), (8, 4, 6), (9, 4, 6), (8, 5, 5), (9, 5, 5), (10, 5, 5), (9, 5, 6)]


def draw(rng):
    case = _draw(rng)
    while any(case == {k: v for k, v in c.items() if k != "name"} for c in listed()):
        case = _draw(rng)
    return case


def _draw(rng):
    kind = rng.choice(["product"] * 5 + ["matfree", "build", "spmm", "program", "solve", "solve", "sweep"])
    model = "sphere"
    if kind == "product":
        model = rng.choice(["sphere", "sphere", "two", "ofl"])
    elif kind == "solve":
        model = rng.choice(["sphere", "ofl"])
    c = dict(kind=kind, model=model)
    if model == "ofl":
        N, dx, dy = rng.choice(_OFL[:6] if kind == "solve" else _OFL)
        c.update(N=N, dx=dx, dy=dy, kx=rng.randrange(dx), ky=rng.randrange(dy))
    else:
        sizes = _TWO if model == "two" else _SPHERE
        if kind == "program":
            sizes = _SPHERE[:10]
        elif kind in ("spmm", "sweep"):
            sizes = _SPHERE[4:12]
        N, norb = rng.choice(sizes)
        # 2 Lz has the parity of N * (norb - 1)
        c.update(N=N, norb=norb, lz=2 * rng.randrange(9) + (N * (norb - 1)) % 2)
    if kind == "product":
        c["upper"] = rng.random() < 0.2
    if kind in ("spmm", "sweep"):
        c["nham"] = rng.choice([2, 5, 8, 11, 16, 23, 32])
    if kind in ("program", "solve"):
        c["nev"] = rng.randrange(2, 6)
    if kind == "sweep":
        c["nev"] = rng.randrange(2, 5)
    return c


# ------------------------------------------------------------------ inputs

def _coulomb(norb):
    """Odd-m Coulomb pseudopotentials on the sphere, m = 0..norb-2."""
    q = norb - 1
    den = math.comb(2 * q + 2, q + 1) ** 2
    v = np.zeros(norb)
    for L in range(q + 1):
        num = math.comb(2 * q - 2 * L, q - L) * math.comb(2 * q + 2 * L + 2, q + L + 1)
        v[q - L] = 2.0 / math.sqrt(q / 2.0) * (num / den)
    v = v[:norb - 1]
    v[0::2] = 0.0
    return v


def _potentials(norb, seed):
    """The Coulomb list with V_1 and V_3 moved by the seed, as a scan over interactions has them."""
    v = _coulomb(norb)
    r = np.random.default_rng([seed, norb])
    v[1] *= 1.0 + 0.2 * r.random()
    v[3] *= 1.0 + 0.1 * r.random()
    return v


def _sweep_lists(case, seed):
    out = []
    for v1 in np.linspace(0.5, 3.0, case["nham"]) + 0.01 * np.random.default_rng(seed).random():
        v = _coulomb(case["norb"])
        v[1] = v1
        out.append(v)
    return out


def _ofl_tables(dx, dy, seed):
    """Momentum-conserving complex tables with the model's layout and rule:
    entry (t1 K + t2 - t1 (t1 + 1) / 2) K + k, values uniform in the unit
    square, real where the diagonal reads them."""
    K = dx * dy
    t1, t2 = np.triu_indices(K)
    k2 = np.arange(K)
    kx = (t1[:, None] // dy + t2[:, None] // dy - k2[None, :] // dy) % dx
    ky = (t1[:, None] % dy + t2[:, None] % dy - k2[None, :] % dy) % dy
    ktab = np.zeros(((K + 1) * K // 2, K), dtype=np.uint16)
    vtab = np.zeros(((K + 1) * K // 2, K), dtype=np.complex128)
    r = np.random.default_rng(seed)
    row = t1 * K + t2 - t1 * (t1 + 1) // 2
    ktab[row] = (kx * dy + ky).astype(np.uint16)
    vtab[row] = r.uniform(-1, 1, (len(t1), K)) + 1j * r.uniform(-1, 1, (len(t1), K))
    vtab[row, t1] = vtab[row, t1].real
    vtab[row, t2] = vtab[row, t2].real
    return ktab.ravel(), vtab.ravel()


def _energies(K):
    return np.linspace(-0.5, 0.5, K)


def _vector(n, seed, dtype=torch.float64):
    """A unit vector, as every product inside a solver gets one."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = 2.0 * torch.rand(n * (2 if dtype == torch.complex128 else 1), generator=g, dtype=torch.float64, device="cuda") - 1.0
    x /= torch.linalg.vector_norm(x)
    return torch.view_as_complex(x.view(n, 2)) if dtype == torch.complex128 else x


class _DeviceArray:
    """A library-owned device array for torch, keeping its owner alive."""

    def __init__(self, ptr, n, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _two_level(ed, case, seed):
    K = case["norb"]
    H = ed.TwoLevelSpinlessFermionHamiltonian()
    H.Initialize(case["N"], 2 * K + 2, twoLz=case["lz"])
    H.Add_CdC_Terms(np.ones(K + 2), 1, 1)
    for lv in (0, 1):
        t = ed.QuarticTermTables(K + 2 * lv, _potentials(K + 2 * lv, seed))
        H.Add_CdCdCC_Terms(t, lv, lv, lv, lv, store_upper=case["upper"])
    H.Build()
    return H


def _ofl_model(ed, case, seed):
    kt, vt = _ofl_tables(case["dx"], case["dy"], seed)
    K = case["dx"] * case["dy"]
    m = ed.InteractingOflModel(case["N"], case["dx"], case["dy"], ed.ComplexQuarticTermTables(case["dx"], case["dy"], kt, vt),
                               _energies(K), case.get("nev", 1))
    m.SetSector(case["kx"], case["ky"])
    return m


def prepare(case, seed):
    import hamiltonian_diagonalization_gb300 as ed
    kind, model = case["kind"], case["model"]
    s = dict(case=case, ed=ed)
    if kind == "product" and model == "ofl":
        m = _ofl_model(ed, case, seed)
        m.BuildFockBasis()
        m.BuildHamiltonian(store_upper=case["upper"])
        s["H"] = m.hamiltonian
        s["x"] = _vector(m.hamiltonian.GetDimension(), seed, torch.complex128)
        s["y"] = torch.empty_like(s["x"])
    elif kind in ("product", "matfree"):
        if model == "two":
            H = _two_level(ed, case, seed)
        else:
            H = ed.SpinlessFermionHamiltonian()
            H.Initialize(case["N"], case["norb"], twoLz=case["lz"])
            tables = ed.QuarticTermTables(case["norb"], _potentials(case["norb"], seed))
            H.Add_CdCdCC_Terms(tables, store_upper=case.get("upper", False), matrix_free=kind == "matfree")
        s["product"] = ed.MatrixVectorFunction(H)
        s["x"] = _vector(H.GetDimension(), seed)
        s["y"] = torch.empty_like(s["x"])
    elif kind == "build":
        s["tables"] = ed.QuarticTermTables(case["norb"], _potentials(case["norb"], seed))
    elif kind in ("spmm", "sweep"):
        basis = ed.FermionFockBasis()
        basis.GenerateFockSpace(case["N"], case["norb"], case["lz"])
        s["batch"] = ed.HamiltonianBatch(basis, _sweep_lists(case, seed))
        n = basis.GetStoredDimension()
        s["X"] = _vector(n * case["nham"], seed).view(n, case["nham"])
        if kind == "spmm":
            s["Y"] = torch.empty_like(s["X"])
    elif kind == "program" or (kind == "solve" and model == "sphere"):
        n = len(_words_of(case))
        s["v"] = _coulomb(case["norb"])
        s["v0"] = _vector(n, seed)
        if kind == "program":
            s["v0"] = s["v0"].cpu().numpy()
        else:
            s["vectors"] = torch.empty((case["nev"], n), dtype=torch.float64, device="cuda")
    elif kind == "solve":
        s["model"] = _ofl_model(ed, case, seed)
        s["v0"] = _vector(len(_words_of(case)), seed, torch.complex128).cpu().numpy()
    else:
        raise ValueError(kind)
    return s


def run(s):
    case, ed = s["case"], s["ed"]
    kind, model = case["kind"], case["model"]
    if kind == "product" and model == "ofl":
        s["H"].apply(s["x"], s["y"])
        return s["y"]
    if kind in ("product", "matfree"):
        s["product"].Simple(s["x"], s["y"])
        return s["y"]
    if kind == "build":
        H = ed.SpinlessFermionHamiltonian()
        H.Initialize(case["N"], case["norb"], twoLz=case["lz"])
        H.Add_CdCdCC_Terms(s["tables"])
        n, nnz, _ = H.m_crsSparseMatrix.info()
        rowptr, col, val = H.m_crsSparseMatrix.device_arrays()
        parts = dict(words=(H.m_fockBasis.words_device_ptr(), n, "<i8"), rowptr=(rowptr, n + 1, "<i8"), col=(col, nnz, "<i4"),
                     val=(val, nnz, "<f8"))
        return {k: torch.as_tensor(_DeviceArray(*p, H), device="cuda") for k, p in parts.items()}
    if kind == "spmm":
        s["batch"].spmm(s["X"], s["Y"])
        return s["Y"]
    if kind == "sweep":
        evals, vecs, _ = s["batch"].solve(case["nev"], tol=TOL, V0=s["X"], want_vectors=True)
        return evals, vecs * torch.sign((vecs * s["X"]).sum(1, keepdim=True))
    if kind == "program":
        m = ed.SpherePseudopotentialModel(case["N"], case["norb"], s["v"], case["nev"])
        m.SetSector(case["lz"])
        m.BuildTermTables()
        m.BuildFockBasis()
        m.BuildHamiltonian()
        if not m.Diagonalize(tol=TOL, v0=s["v0"]):
            raise RuntimeError("not converged")
        H = m.hamiltonian
        vecs = H.m_eigenvectors * np.sign(H.m_eigenvectors @ s["v0"])[:, None]
        return H.m_eigenvalues, vecs, ed.Observables().DensityDensityFunction(H, 0)
    if model == "ofl":
        m = s["model"]
        m.BuildFockBasis()
        m.BuildHamiltonian()
        if not m.Diagonalize(tol=TOL, v0=s["v0"]):
            raise RuntimeError("not converged")
        H = m.hamiltonian
        phase = H.m_eigenvectors.conj() @ s["v0"]
        return H.m_eigenvalues, H.m_eigenvectors * (phase / np.abs(phase))[:, None]
    H = ed.SpinlessFermionHamiltonian()
    H.Initialize(case["N"], case["norb"], twoLz=case["lz"])
    H.Add_CdCdCC_Terms(ed.QuarticTermTables(case["norb"], s["v"]))
    op = H.operator_handle()
    try:
        evals = np.empty(case["nev"])
        p = ed.LanczosParams(nev=case["nev"], tol=TOL, want_vectors=1, verify=1)
        st = ed.lib().ed_lanczos_device(op, ctypes.byref(p), ctypes.c_void_p(s["v0"].data_ptr()),
                                        evals.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                        ctypes.c_void_p(s["vectors"].data_ptr()), None)
    finally:
        ed.lib().ed_op_free(op)
    if st != 0:
        raise RuntimeError(ed.lib().ed_last_error().decode())
    vecs = s["vectors"]
    return evals, vecs * torch.sign(vecs @ s["v0"])[:, None]


# -------------------------------------------- the sectors in plain torch

def _words(weights, N, target, mod):
    """Ascending words of N set bits whose weights sum to target (modulo mod,
    componentwise, where mod is given)."""
    memo = {}

    def red(t):
        return tuple(v % m for v, m in zip(t, mod)) if mod else t

    def get(k, left, t):
        if left < 0 or left > k or (not mod and t[0] < 0):
            return np.zeros(0, dtype=np.int64)
        if left == 0:
            return np.zeros(1 if not any(red(t)) else 0, dtype=np.int64)
        key = (k, left, t)
        if key not in memo:
            w = weights[k - 1]
            low = get(k - 1, left, t)
            high = get(k - 1, left - 1, red(tuple(a - b for a, b in zip(t, w))))
            memo[key] = np.concatenate([low, high | (1 << (k - 1))])
        return memo[key]

    return get(len(weights), N, red(target))


def _words_of(case):
    N = case["N"]
    if case["model"] == "ofl":
        dx, dy = case["dx"], case["dy"]
        return _words([(k // dy, k % dy) for k in range(dx * dy)], N, (case["kx"], case["ky"]), (dx, dy))
    K = case["norb"]
    if case["model"] == "two":
        return _words([(j,) for j in range(K + 2)] + [(i + 1,) for i in range(K)], N, ((case["lz"] + N * (K + 1)) // 2,), None)
    return _words([(k,) for k in range(K)], N, ((case["lz"] + N * (K - 1)) // 2,), None)


def _pair_matrix(norb, v):
    """P[k1, k2, k3, k4] = sum_L V_L <k1 k2|J M><J M|k3 k4>, J = 2S - L, from
    the eigenvectors of J^2 at each total M."""
    q, j = norb - 1, (norb - 1) / 2.0
    P = np.zeros((norb,) * 4)
    m = np.arange(norb) - j
    for s in range(2 * norb - 1):
        a = np.arange(max(0, s - q), min(q, s) + 1)
        b = s - a
        J2 = np.diag(2 * j * (j + 1) + 2 * m[a] * m[b])
        up = np.sqrt((j * (j + 1) - m[a[:-1]] * (m[a[:-1]] + 1)) * (j * (j + 1) - m[b[:-1]] * (m[b[:-1]] - 1)))
        J2 += np.diag(up, 1) + np.diag(up, -1)
        _, U = np.linalg.eigh(J2)
        U = U[:, ::-1]                      # column L has J = 2 S - L
        d = np.array([v[L] if L < len(v) else 0.0 for L in range(len(a))])
        block = (U * d) @ U.T
        P[a[:, None], b[:, None], a[None, :], b[None, :]] = block
    return P


def _sphere_hops(norb, v):
    """Hops (a, b, c, d, weight) that raise the word, and the diagonal weights
    of the occupied pairs; v: one list, or several of as many Hamiltonians."""
    Ps = [_pair_matrix(norb, u) for u in v]
    hops = []
    for a in range(norb):
        for b in range(a + 1, norb):
            for c in range(max(0, a + b - norb + 1), a):
                d = a + b - c
                w = [-(P[d, c, b, a] - P[c, d, b, a] - P[d, c, a, b] + P[c, d, a, b]) for P in Ps]
                hops.append((a, b, c, d, w))
    diag = [[P[a, b, a, b] + P[b, a, b, a] - P[a, b, b, a] - P[b, a, a, b] for P in Ps]
            for a in range(norb) for b in range(a + 1, norb)]
    return hops, diag


def _ofl_hops(dx, dy, vtab):
    K = dx * dy
    T = vtab.reshape(-1, K)

    def V(k1, k2, k3, k4):
        lo, hi = min(k3, k4), max(k3, k4)
        return T[lo * K + hi - lo * (lo + 1) // 2, k1 if k4 > k3 else k2]

    def fold(a, b, c, d):      # c+_k1 c+_k2 c_k3 c_k4 over the four orders of {c, d} and {a, b}
        return V(d, c, b, a) - V(c, d, b, a) - V(d, c, a, b) + V(c, d, a, b)

    cls = {}
    for a in range(K):
        for b in range(a + 1, K):
            cls.setdefault(((a // dy + b // dy) % dx, (a % dy + b % dy) % dy), []).append((a, b))
    hops = [(a, b, c, d, [fold(a, b, c, d)]) for ps in cls.values() for a, b in ps for c, d in ps if (1 << c) + (1 << d) > (1 << a) + (1 << b)]
    diag = [[-fold(a, b, a, b)] for a in range(K) for b in range(a + 1, K)]
    return hops, diag


def _terms(case, seed):
    """[(bit shift, orbitals, hops, diagonal pair weights, orbital energies)] of each level."""
    if case["model"] == "ofl":
        K = case["dx"] * case["dy"]
        return [(0, K, *_ofl_hops(case["dx"], case["dy"], _ofl_tables(case["dx"], case["dy"], seed)[1]), _energies(K))]
    K = case["norb"]
    if case["model"] == "two":
        return [(K + 2, K, *_sphere_hops(K, [_potentials(K, seed)]), np.zeros(K)),
                (0, K + 2, *_sphere_hops(K + 2, [_potentials(K + 2, seed)]), np.ones(K + 2))]
    if case["kind"] in ("program", "solve"):
        lists = [_coulomb(K)]      # the configured interaction; the seed gives the start vector
    else:
        lists = _sweep_lists(case, seed) if "nham" in case else [_potentials(K, seed)]
    return [(0, K, *_sphere_hops(K, lists), np.zeros(K))]


def _parity(v):
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> s)
    return v & 1


def _elements(case, seed, words):
    """Every element above the diagonal, hop by hop: (rows, columns, value of each Hamiltonian)."""
    cplx = case["model"] == "ofl"
    for shift, K, hops, _, _ in _terms(case, seed):
        lev = (words >> shift) & ((1 << K) - 1)
        held = {}
        for a, b, c, d, w in hops:
            if max(abs(x) for x in w) < 1e-14:
                continue
            if (a, b) not in held:
                ab = (1 << a) | (1 << b)
                held = {(a, b): torch.nonzero((lev & ab) == ab).ravel()}
            r = held[(a, b)]
            rest = lev[r] ^ ((1 << a) | (1 << b))
            keep = (rest & ((1 << c) | (1 << d))) == 0
            r, rest = r[keep], rest[keep]
            if not len(r):
                continue
            between = (((1 << b) - 1) & ~((2 << a) - 1)) ^ (((1 << d) - 1) & ~((2 << c) - 1))
            # operators passed by c_a, c_b and then by c+_c, c+_d; one more swap orders them
            sign = 1 - 2 * (1 ^ _parity(rest & between)).to(torch.float64)
            out = words[r] + (((1 << c) + (1 << d) - (1 << a) - (1 << b)) << shift)
            col = torch.searchsorted(words, out)
            yield r, col, sign, torch.tensor(w, dtype=torch.complex128 if cplx else torch.float64, device=words.device)


def _diagonal(case, seed, words):
    total = 0
    for shift, K, _, pairs, energies in _terms(case, seed):
        bits = torch.stack([((words >> (shift + k)) & 1).to(torch.float64) for k in range(K)])
        i = 0
        w = np.array(pairs)
        cplx = np.iscomplexobj(w)
        acc = torch.zeros((len(words), w.shape[1]), dtype=torch.complex128 if cplx else torch.float64, device=words.device)
        for a in range(K):
            acc += energies[a] * bits[a][:, None]
            for b in range(a + 1, K):
                acc += (bits[a] * bits[b])[:, None] * torch.tensor(w[i], device=words.device)
                i += 1
        total = total + acc
    return total


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _apply(case, seed, X):
    words = torch.from_numpy(_words_of(case)).to(X.device)
    Y = _diagonal(case, seed, words) * X
    for r, c, sign, w in _elements(case, seed, words):
        v = sign[:, None] * w[None, :]
        Y[r] += v * X[c]
        Y[c] += v.conj() * X[r]
    return Y


def _dense(case, seed):
    words = torch.from_numpy(_words_of(case))
    d = _diagonal(case, seed, words)[:, 0]
    A = torch.diag(d)
    for r, c, sign, w in _elements(case, seed, words):
        A[r, c] += sign * w[0]
        A[c, r] += (sign * w[0]).conj()
    return words, A


def exact(case, seed):
    kind = case["kind"]
    if kind in ("product", "matfree"):
        n = len(_words_of(case))
        x = _vector(n, seed, torch.complex128 if case["model"] == "ofl" else torch.float64)
        return _apply(case, seed, x[:, None])[:, 0]
    if kind == "spmm":
        n = len(_words_of(case))
        return _apply(case, seed, _vector(n * case["nham"], seed).view(n, case["nham"]))
    if kind == "build":
        words = torch.from_numpy(_words_of(case)).to(_device())
        n = len(words)
        d = _diagonal(case, seed, words)[:, 0]
        i = torch.arange(n, device=words.device)
        key, val = [i * n + i], [d]
        for r, c, sign, w in _elements(case, seed, words):
            key += [r * n + c, c * n + r]
            val += [sign * w[0]] * 2
        key, order = torch.sort(torch.cat(key))
        val = torch.cat(val)[order]
        keep = val.abs() > 1e-14
        key, val = key[keep], val[keep]
        rowptr = torch.searchsorted(key, torch.arange(n + 1, device=words.device) * n)
        return dict(words=words, rowptr=rowptr, col=(key % n).to(torch.int32), val=val)
    n = len(_words_of(case))
    if kind == "sweep" or n > 2500:
        return None
    words, A = _dense(case, seed)
    ev, U = torch.linalg.eigh(A)
    vecs = U[:, :case["nev"]].T
    v0 = _vector(n, seed, A.dtype).cpu()
    phase = vecs.conj() @ v0
    vecs = vecs * (phase / phase.abs())[:, None]
    ev = ev[:case["nev"]]
    if kind == "solve":
        return ev, vecs
    bits = torch.stack([((words >> k) & 1).to(torch.float64) for k in range(case["norb"])])
    return ev, vecs, (bits * vecs[0] ** 2) @ bits.T


# ------------------------------------------------------------------- work

def _counts(case):
    """States and stored elements (both triangles and the diagonal)."""
    words = torch.from_numpy(_words_of(case)).to(_device())
    nnz = len(words)
    one = {k: v for k, v in case.items() if k != "nham"}
    for shift, K, hops, _, _ in _terms(one, 1):
        lev = (words >> shift) & ((1 << K) - 1)
        for a, b, c, d, w in hops:
            if abs(w[0]) < 1e-14:
                continue
            ab, cd = (1 << a) | (1 << b), (1 << c) | (1 << d)
            nnz = nnz + 2 * ((lev & (ab | cd)) == ab).sum() if ab & cd == 0 else nnz
    return len(words), int(nnz)


def work(case):
    """Bytes and FP64 operations of one pass.  A stored product reads each
    stored element (8- or 16-byte value, 4-byte column), the row pointers and x,
    and writes y; a regenerated one reads x and the words; a build writes the
    matrix; the solves make at least about 30 products for each pair (ARPACK
    needs 334 for the headline's ten)."""
    kind = case["kind"]
    n, nnz = _counts(case)
    cplx = case["model"] == "ofl"
    vb, fl = (16, 8) if cplx else (8, 2)
    stored = (nnz + n) // 2 if case.get("upper") else nnz
    product = dict(bytes=stored * (vb + 4) + (n + 1) * 8 + 2 * n * vb, flops=nnz * fl)
    if kind == "product":
        return product
    if kind == "matfree":
        return dict(bytes=3 * n * 8, flops=nnz * fl)
    if kind == "build":
        return dict(bytes=nnz * 12 + (n + 1) * 8 + n * 8, flops=0)
    if kind == "spmm":
        B = case["nham"]
        return dict(bytes=nnz * 6 + (n + 1) * 8 + 2 * n * B * 8, flops=nnz * fl * B)
    steps = 30 * case["nev"]
    if kind == "sweep":
        B = case["nham"]
        return dict(bytes=steps * (nnz * 6 + 2 * n * B * 8) + n * B * case["nev"] * 8, flops=steps * nnz * fl * B)
    return dict(bytes=steps * product["bytes"] + nnz * (vb + 4) + n * case["nev"] * vb, flops=steps * product["flops"])
