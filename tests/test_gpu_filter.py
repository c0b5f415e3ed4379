"""GPU parity of the hot path: the block Clenshaw filter (apply_poly_block!) and the
sparse block product, through the C ABI, against the CPU oracle on identical inputs.

Tolerances: FP64 results agree with the oracle to 1e-12 relative to the block's
magnitude (the GPU fuses multiply-adds, the oracle rounds twice, and the recurrence
runs K steps).  The FP32 filter is compared with the FP64 oracle at 2e-4 relative.
"""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

import sma_oracle as O
from sparse_matrix_algorithms_b200 import matrices as M

pytestmark = pytest.mark.gpu


def _ragged(n, seed):
    """Symmetric matrix with empty, short and long rows (ragged CSR)."""
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for i in range(n):
        k = [0, 1, 2, 5, 13][i % 5]
        js = rng.integers(0, n, size=k)
        rows += [i] * k
        cols += list(js)
    A = sp.coo_matrix((rng.uniform(-1, 1, len(rows)), (rows, cols)), shape=(n, n)).tocsr()
    A = A + A.T
    A.setdiag(np.where(np.arange(n) % 7 == 3, 0.0, rng.uniform(-2, 2, n)))
    A.eliminate_zeros()
    return M._canonical(A)


MATRICES = {
    "lap1d": lambda: M.lap1d(700),
    "anderson_L8": lambda: M.anderson3d(8, 16.5, 2),
    "xxz_L12": lambda: M.xxz_sz0(12, 5.0, 1),
    "ragged": lambda: _ragged(333, 4),
}


def _bounds(A):
    return O.gershgorin_bounds(A)


@pytest.mark.parametrize("name", sorted(MATRICES))
@pytest.mark.parametrize("b", [1, 2, 3, 8, 17, 32, 64, 100])
def test_filter_fp64_matches_oracle(lib_built, name, b):
    import sparse_matrix_algorithms_b200 as S

    A = MATRICES[name]()
    smin, smax = _bounds(A)
    Q = M.splitmix_normal(b, A.shape[0], b)
    for K, window in [(0, "step"), (1, "delta"), (2, "step"), (37, "smooth"), (160, "step")]:
        c = O.build_coeffs(K, smin, smax, 0.1, -0.4, 0.3, window, True)
        ref = O.apply_poly_block(A, Q, c, smin, smax)
        got = S.apply_poly_block(A, Q, c, smin, smax)
        scale = max(np.abs(ref).max(), np.abs(Q).max())
        assert np.abs(got - ref).max() <= 1e-12 * scale, (K, window)


@pytest.mark.parametrize("name,b", [("anderson_L28", 8), ("anderson_L28", 32), ("xxz_L18", 32),
                                    ("xxz_L18", 48), ("xxz_L18", 6)])
def test_filter_all_autotuner_candidates_match_oracle(lib_built, name, b):
    """Operators with n >= 20000 are autotuned online: the first 2 x (candidates) steps of
    the recurrence each run a different kernel configuration (all three families), so
    the result checks every configuration on real work."""
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(28, 16.5, 9) if name == "anderson_L28" else M.xxz_sz0(18, 5.0, 1)
    smin, smax = _bounds(A)
    op = S.SparseOperator(A)
    Q = M.splitmix_normal(5, A.shape[0], b)
    c = O.build_coeffs(90, smin, smax, 0.0, -0.3, 0.3, "step", True)
    ref = O.apply_poly_block(A, Q, c, smin, smax)
    for _ in range(2):  # tuning run, then the chosen configuration
        got = S.apply_poly_block(op, Q, c, smin, smax)
        assert np.abs(got - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Q).max())
    got32 = S.apply_poly_block(op, Q, c, smin, smax, precision="fp32")
    got32 = S.apply_poly_block(op, Q, c, smin, smax, precision="fp32")
    assert np.abs(got32 - ref).max() <= 2e-4 * np.abs(ref).max()


@pytest.mark.parametrize("b", [1, 4, 6, 32, 96])
def test_filter_fp32_close_to_oracle(lib_built, b):
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(8, 16.5, 2)
    smin, smax = _bounds(A)
    Q = M.splitmix_normal(7, A.shape[0], b)
    c = O.build_coeffs(120, smin, smax, 0.0, -0.5, 0.5, "step", True)
    ref = O.apply_poly_block(A, Q, c, smin, smax)
    got = S.apply_poly_block(A, Q, c, smin, smax, precision="fp32")
    assert np.abs(got - ref).max() <= 2e-4 * np.abs(ref).max()


def test_identity_filter_returns_q(lib_built):
    import sparse_matrix_algorithms_b200 as S

    A = M.xxz_sz0(10, 3.0, 5)
    Q = M.splitmix_normal(1, A.shape[0], 16)
    c = O.cheb_window_coeffs(-1.0, 1.0, 80, jackson=True)
    Y = S.apply_poly_block(A, Q, c, *_bounds(A))
    assert np.abs(Y - Q).max() < 1e-12 * np.abs(Q).max()


def test_lap1d_stencil_operator_matches_csr_oracle(lib_built):
    import sparse_matrix_algorithms_b200 as S

    n = 1234
    op = S.Lap1dOperator(n)
    Q = M.splitmix_normal(9, n, 24)
    for K in [0, 1, 5, 200]:
        c = O.build_coeffs(K, 0.0, 4.0, 2.0, 1.9, 2.2, "delta", True)
        ref = O.apply_poly_block(M.lap1d(n), Q, c, 0.0, 4.0)
        got = S.apply_poly_block(op, Q, c, 0.0, 4.0)
        assert np.abs(got - ref).max() <= 1e-12 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("Lsz", [5, 9, 28])
def test_anderson_stencil_matches_csr_kernel_and_oracle(lib_built, Lsz):
    """Matrix-free Anderson stencil: same terms in the same order as the CSR kernel."""
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(Lsz, 16.5, 3)
    st = S.AndersonOperator(Lsz, 16.5, 3)
    csr = S.SparseOperator(A)
    smin, smax = _bounds(A)
    for b, K in [(1, 7), (8, 60), (32, 130)]:
        Q = M.splitmix_normal(b, A.shape[0], b)
        c = O.build_coeffs(K, smin, smax, 0.0, -0.4, 0.4, "step", True)
        y_st = S.apply_poly_block(st, Q, c, smin, smax)
        y_csr = S.apply_poly_block(csr, Q, c, smin, smax)
        scale = max(np.abs(y_csr).max(), 1.0)
        assert np.abs(y_st - y_csr).max() <= 1e-15 * scale
        ref = O.apply_poly_block(A, Q, c, smin, smax)
        assert np.abs(y_st - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Q).max())


@pytest.mark.parametrize("Lc", [4, 10, 14, 18])
def test_xxz_stencil_matches_oracle(lib_built, Lc):
    import sparse_matrix_algorithms_b200 as S

    A = M.xxz_sz0(Lc, 5.0, 1)
    st = S.XXZOperator(Lc, 5.0, 1)
    assert st.n == A.shape[0]
    smin, smax = _bounds(A)
    for b, K in [(2, 9), (16, 80)]:
        Q = M.splitmix_normal(b + 1, A.shape[0], b)
        c = O.build_coeffs(K, smin, smax, 0.0, -0.4, 0.4, "delta", True)
        ref = O.apply_poly_block(A, Q, c, smin, smax)
        got = S.apply_poly_block(st, Q, c, smin, smax)
        assert np.abs(got - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Q).max())


def _device(arr):
    import torch

    return torch.as_tensor(np.ascontiguousarray(arr), device="cuda")


def test_device_entry_with_padded_leading_dimension(lib_built):
    """sma_apply_poly_block_dev on row-major device blocks with ld > b."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    A = M.anderson3d(7, 16.5, 1)
    n, b, ldq, ldy = A.shape[0], 10, 13, 16
    smin, smax = _bounds(A)
    op = S.SparseOperator(A)
    Q = M.splitmix_normal(4, n, b)
    Qpad = np.zeros((n, ldq))
    Qpad[:, :b] = Q
    dQ = _device(Qpad)
    dY = torch.full((n, ldy), 7.0, dtype=torch.float64, device="cuda")
    c = np.ascontiguousarray(O.build_coeffs(45, smin, smax, 0.0, -1.0, 1.5, "step", True))
    torch.cuda.synchronize()
    L.check(L.load().sma_apply_poly_block_dev(op.handle, c.ctypes.data, len(c) - 1, smin, smax,
                                              dQ.data_ptr(), ldq, dY.data_ptr(), ldy, b, 0))
    Y = dY.cpu().numpy()
    ref = O.apply_poly_block(A, Q, c, smin, smax)
    assert np.abs(Y[:, :b] - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.all(Y[:, b:] == 7.0)  # padding untouched


def test_spmm_dev_matches_scipy(lib_built):
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    A = _ragged(500, 9)
    op = S.SparseOperator(A)
    X = M.splitmix_normal(2, 500, 33)
    dX = _device(X)
    dY = torch.empty((500, 33), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    L.check(L.load().sma_spmm_dev(op.handle, dX.data_ptr(), 33, dY.data_ptr(), 33, 33))
    assert np.abs(dY.cpu().numpy() - A @ X).max() < 1e-13 * np.abs(A @ X).max()


def test_empty_block_and_empty_matrix(lib_built):
    import sparse_matrix_algorithms_b200 as S

    A = M.lap1d(50)
    Y = S.apply_poly_block(A, np.zeros((50, 0)), [1.0, 0.5], 0.0, 4.0)
    assert Y.shape == (50, 0)
    E = sp.csr_matrix((0, 0))
    Y = S.apply_poly_block(E, np.zeros((0, 3)), [1.0, 0.5], 0.0, 4.0)
    assert Y.shape == (0, 3)


def test_invalid_csr_is_rejected_before_upload(lib_built):
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    ctx = S.context()
    colptr = np.array([0, 2, 3], dtype=np.int64)
    rowval = np.array([1, 0, 5], dtype=np.int64)  # unsorted and out of range
    nzval = np.ones(3)
    h = ctypes.c_void_p()
    rc = L.load().sma_op_create_csc(ctx.handle, 2, 3, colptr.ctypes.data, rowval.ctypes.data,
                                    nzval.ctypes.data, 0, 0, ctypes.byref(h))
    assert rc == L.SMA_ERR_ARG
    with pytest.raises(S.ArgumentError):
        S.SparseOperator(sp.csr_matrix(np.array([[1.0, 2.0], [0.0, 1.0]])), check_symmetric=True)


@pytest.mark.parametrize("precision,b", [("fp64", 32), ("fp64", 64), ("fp32", 64), ("fp32", 128)])
def test_autotuned_filter_bit_identical_to_untuned(lib_built, monkeypatch, capfd, precision, b):
    """The autotuner's trial steps run every candidate family on real recurrence steps --
    DIRECT, STAGED, ASYNC and BULK (rows staged by bulk copies onto an mbarrier) -- so a tuned
    filter equals an untuned one bit for bit only if every family computes the same bits.
    The BULK family must have been among the candidates."""
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(30, 16.5, 9)  # n = 27000: autotuned
    smin, smax = _bounds(A)
    Q = M.splitmix_normal(3, A.shape[0], b)
    c = O.build_coeffs(120, smin, smax, 0.0, -0.3, 0.3, "step", True)
    monkeypatch.setenv("SMA_AUTOTUNE_VERBOSE", "1")
    tuned = S.apply_poly_block(S.SparseOperator(A, S.Context(0)), Q, c, smin, smax, precision=precision)
    err = capfd.readouterr().err
    assert "bulk/" in err, err
    monkeypatch.setenv("SMA_AUTOTUNE", "0")
    plain = S.apply_poly_block(S.SparseOperator(A, S.Context(0)), Q, c, smin, smax, precision=precision)
    np.testing.assert_array_equal(tuned, plain)


@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-12), ("fp32", 2e-4)])
@pytest.mark.parametrize("b,ldq,shift", [
    (1, 1, 0), (3, 3, 0), (5, 7, 1), (9, 9, 0), (13, 16, 0), (31, 31, 0), (33, 40, 1),
    (64, 65, 0), (64, 64, 1), (66, 66, 0), (127, 128, 0), (260, 260, 0), (517, 517, 0)])
def test_filter_ragged_widths_and_strides(lib_built, precision, rtol, b, ldq, shift):
    """Widths around the vector, CTA and panel edges of the step kernel (1, 2, 4 or 8 columns a
    thread, panels beyond 64 vectors), strides and addresses that forbid wide accesses, degrees on
    both sides of the staging threshold; every column equal to the filter of that column alone at
    the oracle's tolerance, and nothing written past the block."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    A = _ragged(333, 4)
    n = A.shape[0]
    smin, smax = _bounds(A)
    dt = torch.float64 if precision == "fp64" else torch.float32
    Qh = M.splitmix_normal(b, n, b)
    store = torch.full((n * ldq + shift + 8,), 7.0, dtype=dt, device="cuda")
    Q = store[shift:shift + n * ldq].view(n, ldq)
    Q[:, :b] = torch.as_tensor(Qh, device="cuda").to(dt)
    op = S.SparseOperator(A)
    for K in (1, 3, 4, 45):
        c = np.ascontiguousarray(O.build_coeffs(K, smin, smax, 0.1, -0.4, 0.3, "step", True))
        Y = torch.full((n, b + 3), 3.0, dtype=dt, device="cuda")
        torch.cuda.synchronize()
        L.check(L.load().sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, smin, smax, Q.data_ptr(),
                                                  ldq, Y.data_ptr(), b + 3, b, L.PRECISIONS[precision]))
        ref = O.apply_poly_block(A, Qh, c, smin, smax)
        got = Y.cpu().numpy()
        assert np.abs(got[:, :b] - ref).max() <= rtol * max(np.abs(ref).max(), np.abs(Qh).max())
        assert np.all(got[:, b:] == 3.0)


@pytest.mark.parametrize("stencil", ["lap1d", "anderson", "xxz"])
@pytest.mark.parametrize("b", [1, 3, 8, 31, 200])
def test_model_steps_equal_the_stored_matrix(lib_built, stencil, b):
    """The models' entries are built per CTA: first and last rows, wrapped neighbours and the
    periodic bond, at one and at many rows a CTA.  Bit for bit for the models whose entries are
    accumulated in the stored matrix's order."""
    import sparse_matrix_algorithms_b200 as S

    if stencil == "lap1d":
        op, A = S.Lap1dOperator(1001), M.lap1d(1001)
    elif stencil == "anderson":
        op, A = S.AndersonOperator(7, 16.5, 5), M.anderson3d(7, 16.5, 5)
    else:
        op, A = S.XXZOperator(10, 5.0, 1), M.xxz_sz0(10, 5.0, 1)
    smin, smax = _bounds(A)
    c = O.build_coeffs(40, smin, smax, 0.1, -0.4, 0.3, "step", True)
    Q = M.splitmix_normal(b, A.shape[0], b)
    got, ref = S.apply_poly_block(op, Q, c, smin, smax), S.apply_poly_block(A, Q, c, smin, smax)
    if stencil == "xxz":
        assert np.abs(got - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Q).max())
    else:
        np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("rows", ["equal", "short", "ragged"])
@pytest.mark.parametrize("b", [32, 64])
@pytest.mark.parametrize("threads", [9472, 40000, 303104, 909312])
def test_filter_at_the_edges_of_the_step_rule(lib_built, rows, b, threads):
    """The step's gathers in flight and columns a thread follow the number of threads (n b / 4 and
    n b / 2 for FP64): one row below and exactly at each line of the rule, for rows of one length,
    of at most four entries and of all lengths, against the oracle."""
    import sparse_matrix_algorithms_b200 as S

    at = threads * (2 if threads == 9472 else 4) // b
    for n in (at - 1, at):
        if rows == "ragged":
            d = np.where(np.arange(n) % 3 == 0, 1.0, 0.0)  # a third of the rows has far entries
            off = [sp.diags([d[:n - k] * d[k:] * 0.1], [k]) for k in (3, 6, 9, 12, 15)]
            A = M._canonical((sum(off) + sum(off).T + 0.5 * M.lap1d(n)).tocsr())
        elif rows == "equal":
            off = [sp.diags([np.full(n - k, -1.0 / k)], [k]) for k in (1, 7, 50)]
            A = M._canonical((sum(off) + sum(off).T + sp.diags([np.cos(np.arange(n))], [0])).tocsr())
        else:
            A = M.lap1d(n)
        smin, smax = _bounds(A)
        Q = M.splitmix_normal(b, n, b)
        c = O.build_coeffs(5, smin, smax, 0.1, -0.4, 0.3, "step", True)
        ref = O.apply_poly_block(A, Q, c, smin, smax)
        got = S.apply_poly_block(A, Q, c, smin, smax)
        assert np.abs(got - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Q).max())


@pytest.mark.parametrize("kind", ["csr", "anderson", "xxz"])
@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("b", [1, 5, 24])
def test_first_steps_of_every_recurrence(lib_built, kind, K, b):
    """The block c_K Q is folded into the first two steps: the degrees at which those are also the
    last, in place (Y = Q) and not, through the block, the allocation-free and the per-column
    entry."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    op, A = {"csr": lambda: (S.SparseOperator(_ragged(333, 4)), _ragged(333, 4)),
             "anderson": lambda: (S.AndersonOperator(7, 16.5, 5), M.anderson3d(7, 16.5, 5)),
             "xxz": lambda: (S.XXZOperator(10, 5.0, 1), M.xxz_sz0(10, 5.0, 1))}[kind]()
    n = A.shape[0]
    smin, smax = _bounds(A)
    Q = M.splitmix_normal(K, n, b)
    c = np.ascontiguousarray(O.build_coeffs(K, smin, smax, 0.1, -0.4, 0.3, "step", True))
    ref = O.apply_poly_block(A, Q, c, smin, smax)
    table = np.ascontiguousarray(np.repeat(c[:, None], b, axis=1))
    lib, scale = L.load(), max(np.abs(ref).max(), np.abs(Q).max())
    for in_place in (False, True):
        for entry in ("block", "noalloc", "percol"):
            dQ = _device(Q)
            dY = dQ if in_place else torch.full_like(dQ, 7.0)
            torch.cuda.synchronize()
            if entry == "block":
                rc = lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, smin, smax, dQ.data_ptr(), b,
                                                  dY.data_ptr(), b, b, 0)
            elif entry == "noalloc":
                rc = lib.sma_apply_poly_block_noalloc(op.handle, c.ctypes.data, K, smin, smax,
                                                      dQ.data_ptr(), b, dY.data_ptr(), b, b)
            else:
                rc = lib.sma_apply_poly_block_percol_dev(op.handle, table.ctypes.data, K, smin, smax,
                                                         dQ.data_ptr(), dY.data_ptr(), b, 0)
            L.check(rc)
            assert np.abs(dY.cpu().numpy() - ref).max() <= 1e-12 * scale, (entry, in_place)


def _band(n, w, seed):
    rng = np.random.default_rng(seed)
    off = [sp.diags([rng.uniform(0.5, 1.0, n - k)], [k]) for k in range(1, w + 1)]
    return M._canonical((sum(off) + sum(off).T + sp.diags([rng.uniform(-1, 1, n)], [0])).tocsr())


@pytest.mark.parametrize("w,n", [(1, 3), (1, 257), (1, 1500), (2, 5), (2, 130), (2, 1111)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("b", [1, 7, 8, 9, 40])
def test_banded_filter_equals_the_step_by_step_one(lib_built, w, n, precision, b):
    """Operators with a full narrow band take many steps a launch, halo rows recomputed; in place
    they take one (other CTAs still read Q).  Bit for bit the same, for numbers of steps around
    those of a launch, and equal to the oracle; so is the per-column filter, whose columns differ."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    A = _band(n, w, n + b)
    smin, smax = _bounds(A)
    op, lib = S.SparseOperator(A), L.load()
    dt = torch.float64 if precision == "fp64" else torch.float32
    rtol = 1e-12 if precision == "fp64" else 2e-4
    Q = torch.zeros((n, b + 3), dtype=dt, device="cuda")
    Q[:, :b] = torch.as_tensor(M.splitmix_normal(b, n, b), device="cuda").to(dt)
    Qh = Q[:, :b].double().cpu().numpy()
    for K in (1, 2, 7, 8, 9, 16, 33, 70):
        c = np.ascontiguousarray(O.build_coeffs(K, smin, smax, 0.1, -0.4, 0.3, "step", True))
        ref = O.apply_poly_block(A, Qh, c, smin, smax)
        Y = torch.full((n, b + 1), 3.0, dtype=dt, device="cuda")
        Z = Q.clone()
        P, R = Q[:, :b].contiguous(), torch.empty((n, b), dtype=dt, device="cuda")
        torch.cuda.synchronize()
        for src, out in ((Q, Y), (Z, Z)):
            L.check(lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, smin, smax, src.data_ptr(),
                                                 b + 3, out.data_ptr(), out.shape[1], b,
                                                 L.PRECISIONS[precision]))
        table = np.ascontiguousarray(c[:, None] * np.linspace(1.0, 2.0, b)[None, :])
        L.check(lib.sma_apply_poly_block_percol_dev(op.handle, table.ctypes.data, K, smin, smax,
                                                    P.data_ptr(), R.data_ptr(), b, L.PRECISIONS[precision]))
        scale = max(np.abs(ref).max(), np.abs(Qh).max())
        assert torch.equal(Y[:, :b], Z[:, :b]), K
        assert bool((Y[:, b:] == 3.0).all())
        assert np.abs(Y[:, :b].double().cpu().numpy() - ref).max() <= rtol * scale
        assert np.abs(R.double().cpu().numpy() / np.linspace(1.0, 2.0, b) - ref).max() <= rtol * scale


def test_band_of_the_laplacian_stencil_and_of_other_matrices(lib_built):
    """The 1D Laplacian stencil equals its stored matrix; a periodic chain, a band with a missing
    entry and a wider one keep the step kernel."""
    import sparse_matrix_algorithms_b200 as S

    n = 700
    ring = sp.lil_matrix(M.lap1d(n))
    ring[0, n - 1] = ring[n - 1, 0] = -1.0
    hole = sp.lil_matrix(M.lap1d(n))
    hole[350, 351] = hole[351, 350] = 0.0
    for op, A in ((S.Lap1dOperator(n), M.lap1d(n)), (None, ring), (None, hole), (None, _band(n, 3, 1))):
        A = M._canonical(sp.csr_matrix(A))
        A.eliminate_zeros()
        smin, smax = _bounds(A)
        c = O.build_coeffs(50, smin, smax, 0.1, -0.4, 0.3, "step", True)
        Q = M.splitmix_normal(3, n, 12)
        ref = O.apply_poly_block(A, Q, c, smin, smax)
        got = S.apply_poly_block(A if op is None else op, Q, c, smin, smax)
        assert np.abs(got - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Q).max())


@pytest.mark.parametrize("n,b", [(30011, 52), (75001, 52), (45013, 88), (75001, 172)])
@pytest.mark.parametrize("rows", ["equal", "ragged"])
def test_filter_where_ctas_end_within_rows(lib_built, n, b, rows):
    """Thread counts a row that do not divide a CTA's (13, 22, 43): large blocks go on in the next
    row, the last CTA beyond the last; against the oracle."""
    import sparse_matrix_algorithms_b200 as S

    d = np.where(np.arange(n) % 3 == 0, 1.0, 0.0) if rows == "ragged" else np.ones(n)
    off = [sp.diags([d[:n - k] * d[k:] * 0.1], [k]) for k in (3, 6, 9, 12)]
    A = M._canonical((sum(off) + sum(off).T + 0.5 * M.lap1d(n)).tocsr())
    A.eliminate_zeros()
    smin, smax = _bounds(A)
    Q = M.splitmix_normal(b, n, b)
    c = np.ascontiguousarray(O.build_coeffs(4, smin, smax, 0.1, -0.4, 0.3, "step", True))
    ref = O.apply_poly_block(A, Q, c, smin, smax)
    got = S.apply_poly_block(A, Q, c, smin, smax)
    assert np.abs(got - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Q).max())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,b", [(600, 8), (20000, 8), (20000, 64)])
def test_banded_launches_wait_for_the_one_before(lib_built, precision, n, b):
    """Many launches of the banded filter in a row, each started while the one before still runs: its
    blocks may be read only after the wait.  The same bits, over and over, as the step kernel's, which
    an in-place call takes, for the stored matrix and the stencil."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    lib, K = L.load(), 400
    c = np.ascontiguousarray(O.build_coeffs(K, 0.0, 4.0, 1.7, 1.6, 1.8, "step", True))
    Q = _device(M.splitmix_normal(3, n, b))
    Q = Q.to(torch.float64 if precision == "fp64" else torch.float32)

    def run(op, q, y):
        torch.cuda.synchronize()
        L.check(lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, 0.0, 4.0, q.data_ptr(), b, y.data_ptr(),
                                             b, b, L.PRECISIONS[precision]))
        return y

    ops = S.SparseOperator(M.lap1d(n)), S.Lap1dOperator(n)
    Z = Q.clone()
    ref = run(ops[0], Z, Z)
    Z = Q.clone()
    assert torch.equal(run(ops[1], Z, Z), ref)
    for _ in range(5):
        for op in ops:
            assert torch.equal(run(op, Q, torch.empty_like(Q)), ref)


@pytest.mark.parametrize("b", [32, 64])
@pytest.mark.parametrize("threads", [9472, 40000, 303104, 909312])
def test_step_rule_for_short_rows_that_are_no_band(lib_built, b, threads):
    """The rule's line for rows of at most four entries, on a ring, which the banded filter does not
    take: one launch a step, one row below and exactly at each line, against the oracle."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    lib, K = L.load(), 5
    at = threads * (2 if threads == 9472 else 4) // b
    for n in (at - 1, at):
        far = sp.coo_matrix((np.ones(1), ([0], [n - 1])), shape=(n, n))
        A = M._canonical((M.lap1d(n) - far - far.T).tocsr())
        op = S.SparseOperator(A)
        smin, smax = _bounds(A)
        Qh = M.splitmix_normal(b, n, b)
        Q = _device(Qh)
        Y = torch.empty_like(Q)
        c = np.ascontiguousarray(O.build_coeffs(K, smin, smax, 0.1, -0.4, 0.3, "step", True))
        torch.cuda.synchronize()
        before = lib.sma_kernel_launch_count()
        L.check(lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, smin, smax, Q.data_ptr(), b, Y.data_ptr(),
                                             b, b, 0))
        assert lib.sma_kernel_launch_count() - before == K
        ref = O.apply_poly_block(A, Qh, c, smin, smax)
        assert np.abs(Y.cpu().numpy() - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Qh).max())


@pytest.mark.parametrize("n", [2, 3, 130, 1001])
@pytest.mark.parametrize("b", [1, 3, 8, 31, 200])
def test_lap1d_stencil_on_the_step_kernel(lib_built, n, b):
    """The 1D Laplacian's rows as the step kernel builds them, which in-place calls take (one launch a
    step): against the oracle, and bit for bit the stored matrix's and, for n >= 3, the banded filter's."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    lib, K = L.load(), 20
    A = M.lap1d(n)
    c = np.ascontiguousarray(O.build_coeffs(K, 0.0, 4.0, 1.7, 1.3, 2.1, "step", True))
    Qh = M.splitmix_normal(b, n, b)
    ref = O.apply_poly_block(A, Qh, c, 0.0, 4.0)
    out = []
    for op in (S.Lap1dOperator(n), S.SparseOperator(A)):
        for in_place in (True, False):
            Q = _device(Qh)
            Y = Q if in_place else torch.empty_like(Q)
            torch.cuda.synchronize()
            before = lib.sma_kernel_launch_count()
            L.check(lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, 0.0, 4.0, Q.data_ptr(), b,
                                                 Y.data_ptr(), b, b, 0))
            launches = lib.sma_kernel_launch_count() - before
            assert launches >= K if in_place or n < 3 else launches < K
            out.append(Y.cpu().numpy())
    assert np.abs(out[0] - ref).max() <= 1e-12 * max(np.abs(ref).max(), np.abs(Qh).max())
    for got in out[1:]:
        np.testing.assert_array_equal(got, out[0])


@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-12), ("fp32", 2e-4)])
@pytest.mark.parametrize("L_", [4, 10, 14, 16])
def test_xxz_rows_walked_and_in_shared_memory(lib_built, L_, precision, rtol):
    """XXZ rows of few threads are walked by each of them, the others' entries go through shared
    memory: every column has the same bits at every width, on both sides of the rule's lines (6 and 16
    threads a row, a wave of threads), by the block and the per-column entry; against the oracle."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    op, A = S.XXZOperator(L_, 5.0, 1), M.xxz_sz0(L_, 5.0, 1)
    n, K, lib = A.shape[0], 5, L.load()
    smin, smax = _bounds(A)
    c = np.ascontiguousarray(O.build_coeffs(K, smin, smax, 0.1, -0.4, 0.3, "step", True))
    dt = torch.float64 if precision == "fp64" else torch.float32
    Qh = M.splitmix_normal(L_, n, 128)
    ref = O.apply_poly_block(A, Qh, c, smin, smax)
    full = None
    for b in (128, 64, 52, 32, 24, 16, 8, 6, 5, 3, 2, 1):
        Q = _device(Qh[:, :b]).to(dt)
        Y, P = torch.empty_like(Q), torch.empty_like(Q)
        table = np.ascontiguousarray(np.repeat(c[:, None], b, axis=1))
        torch.cuda.synchronize()
        L.check(lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, smin, smax, Q.data_ptr(), b, Y.data_ptr(), b,
                                             b, L.PRECISIONS[precision]))
        L.check(lib.sma_apply_poly_block_percol_dev(op.handle, table.ctypes.data, K, smin, smax, Q.data_ptr(),
                                                    P.data_ptr(), b, L.PRECISIONS[precision]))
        if full is None:
            full = Y
            assert np.abs(Y.double().cpu().numpy() - ref).max() <= rtol * max(np.abs(ref).max(), np.abs(Qh).max())
        assert torch.equal(Y, full[:, :b]) and torch.equal(P, Y), b


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind,n,widths", [("csr", 50653, (3, 5, 13, 15, 17, 19, 31)), ("anderson", 50653, (5, 13, 31)),
                                           ("ring", 3100, (61, 253, 257, 261)), ("ragged", 6100, (29, 31, 61))])
def test_filter_of_columns_a_row_apart(lib_built, precision, kind, n, widths):
    """Blocks that allow accesses of one element only, wide enough for four columns a thread: at every
    remainder of the columns, over one panel and two, every column has the bits of the aligned block's,
    by the block entry in place and not, the per-column and the allocation-free one, and nothing is
    written past the block."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    A = {"csr": lambda: M.anderson3d(37, 16.5, 5), "anderson": lambda: M.anderson3d(37, 16.5, 5),
         "ring": lambda: M._canonical((M.lap1d(n) - sp.coo_matrix(([1.0, 1.0], ([0, n - 1], [n - 1, 0])), shape=(n, n))).tocsr()),
         "ragged": lambda: _ragged(n, 4)}[kind]()
    op = S.AndersonOperator(37, 16.5, 5) if kind == "anderson" else S.SparseOperator(A)
    smin, smax = _bounds(A)
    dt = torch.float64 if precision == "fp64" else torch.float32
    lib, P = L.load(), L.PRECISIONS[precision]
    wide = -(-max(widths) // 8) * 8
    full = _device(M.splitmix_normal(n, n, wide)).to(dt)
    for K in (1, 2, 3):
        c = np.ascontiguousarray(O.build_coeffs(K, smin, smax, 0.1, -0.4, 0.3, "step", True))
        ref = torch.empty_like(full)
        torch.cuda.synchronize()
        L.check(lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, smin, smax, full.data_ptr(), wide,
                                             ref.data_ptr(), wide, wide, P))
        for b in widths:
            table = np.ascontiguousarray(np.repeat(c[:, None], b, axis=1))
            for entry in ("block", "in place", "percol", "noalloc"):
                if entry == "noalloc" and (precision == "fp32" or n * b > 2 ** 21):
                    continue
                Q = full[:, :b].contiguous()
                store = torch.full((n * b + 9,), 7.0, dtype=dt, device="cuda")
                Y = Q if entry == "in place" else store[1:1 + n * b].view(n, b)
                torch.cuda.synchronize()
                if entry == "percol":
                    rc = lib.sma_apply_poly_block_percol_dev(op.handle, table.ctypes.data, K, smin, smax, Q.data_ptr(),
                                                             Y.data_ptr(), b, P)
                elif entry == "noalloc":
                    rc = lib.sma_apply_poly_block_noalloc(op.handle, c.ctypes.data, K, smin, smax, Q.data_ptr(), b,
                                                          Y.data_ptr(), b, b)
                else:
                    rc = lib.sma_apply_poly_block_dev(op.handle, c.ctypes.data, K, smin, smax, Q.data_ptr(), b,
                                                      Y.data_ptr(), b, b, P)
                L.check(rc)
                assert torch.equal(Y, ref[:, :b]), (K, b, entry)
                assert bool((store[0] == 7.0) & (store[1 + n * b:] == 7.0).all())
    ref0 = O.apply_poly_block(A, full[:, :3].double().cpu().numpy(), c, smin, smax)
    assert np.abs(ref[:, :3].double().cpu().numpy() - ref0).max() <= (1e-12 if precision == "fp64" else 2e-4) * 5
