"""The work that users of this framework have it do, as measurable cases.

Almost all of a solve is the block filter Y = p(A_hat) Q (a Clenshaw recurrence of K fused
sparse steps over an n x b block), so most cases are filters: one per matrix family, block
width and element type that the solvers meet, from the smallest matrices of the tests to the
widest blocks of the benchmark configurations.  The others are the dense products that
orthogonalize a filtered block against the stored basis, the KPM moments that place windows
and feed the planner, and one whole POLFED solve.

Matrices, vectors and coefficients are made here from the seed with numpy and torch alone, so
that ``exact`` can evaluate the same inputs in 64 bits without the library.
"""
import math

import numpy as np
import scipy.sparse as sp
import torch

import sparse_matrix_algorithms_b200 as S
from sparse_matrix_algorithms_b200 import _lib as L
from sparse_matrix_algorithms_b200 import api

ANDERSON_W = 16.5  # disorder strength of the Anderson configurations
XXZ_H = 3.0        # random-field strength of the XXZ configurations


def listed():
    return [
        # The smallest test chains, degree 80 (the solvers' default): the recurrence is a row of
        # kernels of a few microseconds each, so launches and latency are the time.
        dict(name="filter_xxz14_b8_f64", kind="filter", model="xxz", size=14, b=8, K=80, precision="fp64"),
        # Chebyshev iteration on the 8000-site lattice with its m0 = 64 block.
        dict(name="filter_anderson20_b64_f64", kind="filter", model="anderson", size=20, b=64, K=200, precision="fp64"),
        # POLFED blocks of the L = 18 chain (s = 32): the blocks fit in the L2 cache.
        dict(name="filter_xxz18_b32_f64", kind="filter", model="xxz", size=18, b=32, K=200, precision="fp64"),
        # A block whose rank dropped to an odd width: no two columns share an aligned access.
        dict(name="filter_anderson30_b37_f64", kind="filter", model="anderson", size=30, b=37, K=100, precision="fp64"),
        # The benchmark's plain FP64 arm: n = 262144, s = 64.
        dict(name="filter_anderson64_b64_f64", kind="filter", model="anderson", size=64, b=64, K=64, precision="fp64"),
        # The benchmark's mixed-precision arm builds its basis with this filter.
        dict(name="filter_anderson64_b64_f32", kind="filter", model="anderson", size=64, b=64, K=96, precision="fp32"),
        # Chebyshev iteration on the same lattice with m0 = 768: the widest block.
        dict(name="filter_anderson64_b768_f32", kind="filter", model="anderson", size=64, b=768, K=16, precision="fp32"),
        # The mixed-precision polish: one polynomial per column over the in-window candidates
        # (the same segmented step also runs batched windows).
        dict(name="percol_anderson64_b496_f32", kind="percol", model="anderson", size=64, b=496, K=24, precision="fp32"),
        # The matrix-free signatures on the device stencil.
        dict(name="stencil_anderson48_b64_f64", kind="stencil", model="anderson", size=48, b=64, K=64, precision="fp64"),
        # A block orthogonalized against a mid-run basis of 1024 columns.
        dict(name="reorth_n262144_m1024_p64", kind="reorth", n=262144, m=1024, p=64),
        # The spectral density of the L = 20 chain, as the planner asks for it.
        dict(name="kpm_xxz20_M256_R16", kind="kpm", model="xxz", size=20, M=256, R=16),
        # A whole solve: an interior window of the 1D Laplacian, mixed precision.
        dict(name="polfed_lap1d_20000_mixed", kind="polfed", n=20000, nev=160, s=32, precision="mixed"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["filter"] * 6 + ["percol", "stencil", "reorth", "reorth", "kpm", "polfed"])
    if kind == "reorth":
        return dict(kind=kind, n=log(3000, 262144), m=log(16, 1024), p=rng.choice([log(1, 64), 8, 16, 32, 64]))
    if kind == "polfed":
        n = log(4000, 30000)
        return dict(kind=kind, n=n, nev=max(40, n // rng.randint(80, 160)), s=rng.choice([16, 32, 48, 64]),
                    precision=rng.choice(["fp64", "mixed"]))
    model = rng.choice(["anderson", "xxz"])
    size = log(12, 64) if model == "anderson" else 2 * rng.randint(6, 10)
    if kind == "kpm":
        return dict(kind=kind, model=model, size=size, M=log(32, 256), R=rng.choice([4, 8, 13, 16, 32]))
    n = _dimension(model, size)
    precision = rng.choice(["fp64", "fp64", "fp32"])
    words = 8 if precision == "fp64" else 4
    widest = max(8, min(768, int(262144 * 768 * 4 / (n * words)), n // 4))
    b = rng.choice([log(3, widest), 8 * max(1, log(8, widest) // 8)])
    steps = 262144 * 768 * 4 * 16 / (n * b * words)  # no more work than the widest listed block
    return dict(kind=kind, model=model, size=size, b=b, K=max(4, min(log(16, 256), int(steps))), precision=precision)


# ------------------------------------------------------------------ inputs
def _dimension(model, size):
    return size ** 3 if model == "anderson" else math.comb(size, size // 2)


def _mix64(x):
    """SplitMix64's output function, the random stream of the stencils and the KPM vectors."""
    with np.errstate(over="ignore"):
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _stream(seed, count):
    with np.errstate(over="ignore"):
        return _mix64(np.uint64(seed) + np.arange(1, count + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15))


def _uniform(seed, count):
    return (_stream(seed, count) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _anderson(size, seed):
    """Periodic L^3 lattice, hopping -1, on-site energies uniform in [-W/2, W/2]."""
    n = size ** 3
    i = np.arange(n)
    x, y, z = i % size, i // size % size, i // size ** 2
    cols = np.stack([i] + [((x + a) % size) + size * ((y + b) % size) + size ** 2 * ((z + c) % size)
                           for a, b, c in ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))], axis=1)
    vals = np.full((n, 7), -1.0)
    vals[:, 0] = ANDERSON_W * (_uniform(seed, n) - 0.5)
    order = np.argsort(cols, axis=1)
    return sp.csr_matrix((np.take_along_axis(vals, order, 1).ravel(), np.take_along_axis(cols, order, 1).astype(np.int32).ravel(),
                          np.arange(0, 7 * n + 1, 7, dtype=np.int32)), shape=(n, n))


def _xxz(size, seed):
    """Periodic random-field XXZ chain (J = Delta = 1) in its Sz = 0 sector."""
    every = np.arange(1 << size, dtype=np.int64)
    bits = sum((every >> i) & 1 for i in range(size))
    states = every[bits == size // 2]
    n = states.size
    rank = np.empty(1 << size, dtype=np.int64)
    rank[states] = np.arange(n)
    spin = [((states >> i) & 1) - 0.5 for i in range(size)]
    field = XXZ_H * (2.0 * _uniform(seed, size) - 1.0)
    diag = sum(spin[i] * spin[(i + 1) % size] + field[i] * spin[i] for i in range(size))
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [diag]
    for i in range(size):
        j = (i + 1) % size
        r = np.nonzero(spin[i] != spin[j])[0]
        rows.append(r)
        cols.append(rank[states[r] ^ ((1 << i) | (1 << j))])
        vals.append(np.full(r.size, 0.5))
    A = sp.coo_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), shape=(n, n)).tocsr()
    A.sort_indices()
    return A


def _laplacian(n, seed):
    """v + t tridiag(-1, 2, -1), its spectrum and its scale (v, t from the seed)."""
    v, t = _uniform(seed, 2) - 0.5
    t += 1.5
    A = sp.diags([np.full(n - 1, -t), np.full(n, v + 2.0 * t), np.full(n - 1, -t)], [-1, 0, 1], format="csr")
    return A, v + t * (2.0 - 2.0 * np.cos(np.pi * np.arange(1, n + 1) / (n + 1))), (v, v + 4.0 * t)


def _target(case, spectrum):
    """nev interior eigenvalues and a window that ends between them and their neighbours.  Off
    centre: the filter must not map the two sides of a symmetric spectrum onto each other."""
    lo = int(0.45 * case["n"]) - case["nev"] // 2
    hi = lo + case["nev"]
    return spectrum[lo:hi], 0.5 * (spectrum[lo - 1] + spectrum[lo]), 0.5 * (spectrum[hi - 1] + spectrum[hi])


def _matrix(case, seed):
    if case["kind"] == "polfed":
        return _laplacian(case["n"], seed)[0]
    return (_anderson if case["model"] == "anderson" else _xxz)(case["size"], seed)


def _bounds(case):
    """An interval that holds every such matrix's spectrum (Gershgorin, worst disorder)."""
    r = 0.5 * ANDERSON_W + 6.0 if case["model"] == "anderson" else case["size"] * (0.25 + 0.5 * XXZ_H + 0.5)
    return -r, r


def _jackson(K):
    k, N = np.arange(K + 1), K + 1
    a = math.pi / (N + 1)
    return ((N - k + 1) * np.cos(a * k) + np.sin(a * k) / math.tan(a)) / (N + 1)


def _coefficients(K, centre=0.1):
    """Jackson-damped delta filter at `centre` of [-1, 1] (an array gives one column each),
    scaled to 1 there."""
    t = np.arccos(np.atleast_1d(centre))
    c = 2.0 * np.cos(np.outer(np.arange(K + 1), t)) * _jackson(K)[:, None]
    c[0] *= 0.5
    c /= (c * np.cos(np.outer(np.arange(K + 1), t))).sum(axis=0)
    return np.ascontiguousarray(c if np.ndim(centre) else c[:, 0])


def _block(n, b, seed, dtype=torch.float64):
    g = torch.Generator("cuda").manual_seed(seed)
    return torch.randn(n, b, generator=g, device="cuda", dtype=torch.float64).to(dtype)


def _centres(case):
    return 0.1 + 0.002 * (np.arange(case["b"]) / case["b"] - 0.5)


def _polfed_size(case):
    """The harness's rule: degree 4 n / nev (12 half-widths of the spectrum per window), a basis
    of three times the wanted pairs."""
    return 4 * case["n"] // case["nev"], math.ceil(3 * case["nev"] / case["s"])


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    kind = case["kind"]
    state = dict(case)
    if kind == "reorth":
        n, m, p = case["n"], case["m"], case["p"]
        state.update(ctx=api.context(), V=_block(n, m, seed).mul_(n ** -0.5), W=_block(n, p, seed + 1000003),
                     C=torch.empty(p, m, device="cuda", dtype=torch.float64))
    elif kind == "stencil":
        state.update(op=S.AndersonOperator(case["size"], ANDERSON_W, seed) if case["model"] == "anderson"
                     else S.XXZOperator(case["size"], XXZ_H, seed))
    else:
        state.update(op=S.SparseOperator(_matrix(case, seed)))
    state["seed"] = seed
    if kind == "polfed":
        _, spectrum, state["bounds"] = _laplacian(case["n"], seed)
        _, state["emin"], state["emax"] = _target(case, spectrum)
    if kind in ("filter", "percol", "stencil"):
        Q = _block(state["op"].n, case["b"], seed, torch.float64 if case["precision"] == "fp64" else torch.float32)
        c = _coefficients(case["K"], _centres(case) if kind == "percol" else 0.1)
        state.update(Q=Q, Y=torch.empty_like(Q), coeffs=c)
    torch.cuda.synchronize()  # the library runs on its own stream
    return state


def run(state):
    kind = state["kind"]
    if kind == "reorth":
        h, V, W, C, n, m, p = (state[k] for k in ("ctx", "V", "W", "C", "n", "m", "p"))
        lib = L.load()
        # C = V' W (column-major m x p), W -= V C
        L.check(lib.sma_dense_gram_dev(h.handle, n, m, p, V.data_ptr(), m, W.data_ptr(), p, C.data_ptr(), m, 1.0, 0.0))
        L.check(lib.sma_dense_update_dev(h.handle, n, m, p, V.data_ptr(), m, C.data_ptr(), m, 0, W.data_ptr(), p, -1.0, 1.0))
        return {"C": C, "W": W}
    op = state["op"]
    if kind == "polfed":
        degree, mmax = _polfed_size(state)
        (smin, smax), emin, emax = state["bounds"], state["emin"], state["emax"]
        lam, _, res = S.polfed(op, state["nev"], degree, s=state["s"], smin=smin, smax=smax, sigma=0.5 * (emin + emax),
                               emin=emin, emax=emax, tol=1e-10, window_type="delta", mmax=mmax, seed=state["seed"],
                               precision=state["precision"], vectors=False)
        order = np.argsort(lam)
        return {"lam": lam[order], "lam_res": np.stack([lam[order], res[order]])}
    smin, smax = _bounds(state)
    if kind == "kpm":
        mu, vectors = api.kpm_moments(op, state["M"], state["R"], smin=smin, smax=smax, seed=state["seed"], per_vector=True)
        return {"mu": mu, "vectors": vectors}
    Q, Y, c = state["Q"], state["Y"], state["coeffs"]
    b, precision = state["b"], L.PRECISIONS[state["precision"]]
    if kind == "percol":
        L.check(L.load().sma_apply_poly_block_percol_dev(op.handle, c.ctypes.data, state["K"], smin, smax, Q.data_ptr(),
                                                         Y.data_ptr(), b, precision))
    else:
        L.check(L.load().sma_apply_poly_block_dev(op.handle, c.ctypes.data, state["K"], smin, smax, Q.data_ptr(), b,
                                                  Y.data_ptr(), b, b, precision))
    return Y


def work(case):
    """Inputs and outputs once each; a filter's flops are its K products and recurrence steps."""
    kind = case["kind"]
    if kind == "reorth":
        n, m, p = case["n"], case["m"], case["p"]
        return {"bytes": 8.0 * (n * m + 2 * n * p + m * p), "flops": 4.0 * n * m * p}
    if kind == "polfed":
        degree, mmax = _polfed_size(case)
        return {"bytes": 36.0 * case["n"], "flops": mmax * case["s"] * degree * 12.0 * case["n"]}
    n = _dimension(case["model"], case["size"])
    row = 7 if case["model"] == "anderson" else 1 + 0.5 * case["size"] * case["size"] / (case["size"] - 1)
    nnz = row * n
    if kind == "kpm":
        return {"bytes": 12.0 * nnz + 8.0 * case["M"] * case["R"], "flops": (case["M"] / 2 * (2 * nnz + 4.0 * n) + 2.0 * case["M"] * n) * case["R"]}
    words = 8 if case["precision"] == "fp64" else 4
    matrix = 8.0 * n if kind == "stencil" else nnz * (words + 4) + 4 * (n + 1)
    return {"bytes": matrix + 2.0 * words * n * case["b"], "flops": case["K"] * case["b"] * (2 * nnz + 6.0 * n)}


# ------------------------------------------------------------------ the same in 64 bits
def _device_csr(A):
    return torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)), torch.from_numpy(A.indices.astype(np.int64)),
                                   torch.from_numpy(A.data), size=A.shape, device="cuda", check_invariants=False)


def exact(case, seed):
    kind = case["kind"]
    if kind == "reorth":
        V, W = _block(case["n"], case["m"], seed).mul_(case["n"] ** -0.5), _block(case["n"], case["p"], seed + 1000003)
        C = V.T @ W
        return {"C": C.T.contiguous(), "W": W - V @ C}
    if kind == "polfed":
        return {"lam": _target(case, _laplacian(case["n"], seed)[1])[0], "lam_res": None}
    A = _matrix(case, seed)
    n = A.shape[0]
    smin, smax = _bounds(case)
    centre, half = 0.5 * (smin + smax), 0.5 * (smax - smin)
    M = _device_csr(((A - centre * sp.identity(n, format="csr")) / half).tocsr())
    if kind == "kpm":
        signs = _stream((seed ^ 0x2545F4914F6CDD1D) & (2 ** 64 - 1), n * case["R"]) >> np.uint64(63)
        z = torch.from_numpy(np.where(signs == 0, 1.0, -1.0).reshape(case["R"], n).T.copy()).cuda()
        t0, t1, mu = z, M @ z, [(z * z).sum(0)]
        for _ in range(1, case["M"]):
            mu.append((z * t1).sum(0))
            t0, t1 = t1, 2.0 * (M @ t1) - t0
        vectors = (torch.stack(mu) / n).cpu().numpy()
        return {"mu": vectors.mean(axis=1), "vectors": vectors}
    c = torch.from_numpy(_coefficients(case["K"], _centres(case) if kind == "percol" else 0.1)).cuda()
    # the rounded FP32 block is the input there is
    Q = _block(n, case["b"], seed, torch.float64 if case["precision"] == "fp64" else torch.float32).double()
    b1, b2 = torch.zeros_like(Q), torch.zeros_like(Q)
    for k in range(case["K"], 0, -1):
        b1, b2 = c[k] * Q + 2.0 * (M @ b1) - b2, b1
    return c[0] * Q + M @ b1 - b2
