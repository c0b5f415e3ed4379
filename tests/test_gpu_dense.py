"""This library's FP64 tensor-core (DMMA) products, through the C ABI, against numpy in FP64:
the Gram X^T Y (split-n reduction) and the block update Y = alpha X B + beta Y, at the
shapes of the solvers -- tall skinny, ragged sizes (not multiples of the 64 x 64 / 128 x 64
tiles), odd leading dimensions and offsets (the 8-byte copy path) -- plus the in-place
X <- X B of CholQR.  Tolerance: 1e-13 relative to the product's scale (sum |x||y| over n).
The Gram is deterministic: two runs give the same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch

    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _gram(ctx, X, Y, m, k, C0=None, alpha=1.0, beta=0.0, ldc=None):
    import torch
    from sparse_matrix_algorithms_b200 import _lib as L

    n = X.shape[0]
    ldc = ldc or m
    Cd = _dev(np.zeros((k, ldc)) if C0 is None else C0)
    Xd, Yd = _dev(X), _dev(Y)
    torch.cuda.synchronize()
    L.check(L.load().sma_dense_gram_dev(ctx.handle, n, m, k, Xd.data_ptr(), X.shape[1],
                                        Yd.data_ptr(), Y.shape[1], Cd.data_ptr(), ldc, alpha, beta))
    return Cd.cpu().numpy()  # row j of this (k x ldc) array is column j of C


@pytest.mark.parametrize("n,m,k", [(262144, 64, 64), (50000, 200, 64), (9999, 37, 5),
                                   (3001, 130, 130), (100, 64, 64), (0, 8, 8)])
def test_gram_matches_numpy(lib_built, n, m, k):
    import sparse_matrix_algorithms_b200 as S

    ctx = S.context()
    rng = np.random.default_rng(n + m + k)
    ldx, ldy = m + (3 if m % 2 else 0), k
    X = rng.standard_normal((n, ldx))
    Y = rng.standard_normal((n, ldy))
    C = _gram(ctx, X, Y, m, k)
    ref = X[:, :m].T @ Y[:, :k]
    scale = (np.abs(X[:, :m]).T @ np.abs(Y[:, :k])).max() if n else 1.0
    assert np.abs(C[:, :m].T - ref).max() <= 1e-13 * max(scale, 1.0)
    assert np.array_equal(C, _gram(ctx, X, Y, m, k))  # deterministic


def test_gram_alpha_beta(lib_built):
    import sparse_matrix_algorithms_b200 as S

    ctx = S.context()
    rng = np.random.default_rng(1)
    n, m, k = 7000, 70, 40
    X, Y = rng.standard_normal((n, m)), rng.standard_normal((n, k))
    C0 = rng.standard_normal((k, m))
    C = _gram(ctx, X, Y, m, k, C0=C0, alpha=-0.5, beta=2.0)
    ref = -0.5 * (X.T @ Y) + 2.0 * C0.T
    assert np.abs(C.T - ref).max() <= 1e-12 * np.abs(ref).max()


def _update(ctx, X, Cm, p, transC, Y0, alpha, beta, m):
    import torch
    from sparse_matrix_algorithms_b200 import _lib as L

    n = X.shape[0]
    Xd, Cd, Yd = _dev(X), _dev(Cm), _dev(Y0)
    torch.cuda.synchronize()
    L.check(L.load().sma_dense_update_dev(ctx.handle, n, m, p, Xd.data_ptr(), X.shape[1],
                                          Cd.data_ptr(), max(Cm.shape[1], 1), int(transC),
                                          Yd.data_ptr(),
                                          Y0.shape[1], alpha, beta))
    return Yd.cpu().numpy()


@pytest.mark.parametrize("n,m,p", [(262144, 512, 64), (40000, 64, 64), (12345, 33, 70),
                                   (5000, 0, 16), (777, 1000, 200)])
@pytest.mark.parametrize("transC", [False, True])
def test_update_matches_numpy(lib_built, n, m, p, transC):
    import sparse_matrix_algorithms_b200 as S

    ctx = S.context()
    rng = np.random.default_rng(n + m + p + transC)
    X = rng.standard_normal((n, m + 1))  # ld = m + 1 (odd for even m: the 8-byte path)
    B = rng.standard_normal((m, p))
    if transC:  # C is p x m column-major: row i of the array = column i of C = row i of B
        Cm = np.ascontiguousarray(B)
    else:       # C is m x p column-major: row j of the array = column j of C
        Cm = np.ascontiguousarray(B.T)
    Y0 = rng.standard_normal((n, p + 2))
    Y = _update(ctx, X, Cm, p, transC, Y0, -1.0, 1.0, m)
    ref = Y0[:, :p] - X[:, :m] @ B
    scale = (np.abs(X[:, :m]) @ np.abs(B)).max() if m else 1.0
    assert np.abs(Y[:, :p] - ref).max() <= 1e-13 * max(scale, 1.0)
    assert np.array_equal(Y[:, p:], Y0[:, p:])  # columns beyond p untouched


def test_update_in_place_triangular_inverse(lib_built):
    """X <- X R^-1 in place (k <= 64, beta = 0: Y aliases X), the product that replaces the
    triangular solve of CholQR, against numpy."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    ctx = S.context()
    rng = np.random.default_rng(7)
    n, k = 100000, 48
    X = rng.standard_normal((n, k))
    R = np.triu(rng.standard_normal((k, k))) + 5 * np.eye(k)
    Rinv = np.linalg.inv(R)
    Xd = _dev(X)
    Cd = _dev(np.ascontiguousarray(Rinv.T))  # column-major k x k
    torch.cuda.synchronize()
    L.check(L.load().sma_dense_update_dev(ctx.handle, n, k, k, Xd.data_ptr(), k, Cd.data_ptr(), k,
                                          0, Xd.data_ptr(), k, 1.0, 0.0))
    got = Xd.cpu().numpy()
    ref = X @ Rinv
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("m,p", [(1, 1), (31, 32), (33, 31), (128, 33), (129, 64), (127, 32), (200, 65)])
def test_products_at_the_edges_of_their_tiles(lib_built, m, p):
    """Tile choices change at 32 columns and at 128 summands: both sides, with an aligned and an
    odd leading dimension, n one off a multiple of the tile; tolerances as above."""
    import sparse_matrix_algorithms_b200 as S

    ctx = S.context()
    rng = np.random.default_rng(m + p)
    for n in (63, 64, 4097):
        for pad in (m % 2, 1 - m % 2):
            X, B = rng.standard_normal((n, m + pad)), rng.standard_normal((m, p))
            Y0 = rng.standard_normal((n, p + pad))
            Y = _update(ctx, X, np.ascontiguousarray(B.T), p, False, Y0, 0.5, -2.0, m)
            ref = 0.5 * X[:, :m] @ B - 2.0 * Y0[:, :p]
            assert np.abs(Y[:, :p] - ref).max() <= 1e-13 * max((np.abs(X[:, :m]) @ np.abs(B)).max(), 8.0)
            assert np.array_equal(Y[:, p:], Y0[:, p:])
            C = _gram(ctx, X, Y0, m, p)
            scale = (np.abs(X[:, :m]).T @ np.abs(Y0[:, :p])).max()
            assert np.abs(C.T - X[:, :m].T @ Y0[:, :p]).max() <= 1e-13 * max(scale, 1.0)


@pytest.mark.parametrize("k", [1, 31, 32, 33, 64])
def test_update_in_place_of_every_width(lib_built, k):
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    rng = np.random.default_rng(k)
    n = 1000
    X, B = rng.standard_normal((n, k)), rng.standard_normal((k, k))
    Xd, Cd = _dev(X), _dev(B.T)
    torch.cuda.synchronize()
    L.check(L.load().sma_dense_update_dev(S.context().handle, n, k, k, Xd.data_ptr(), k, Cd.data_ptr(),
                                          k, 0, Xd.data_ptr(), k, 1.0, 0.0))
    assert np.abs(Xd.cpu().numpy() - X @ B).max() <= 1e-13 * max((np.abs(X) @ np.abs(B)).max(), 1.0)


def _gram_of_ones_in_order(x, m, k):
    """X^T 1 as the Gram sums it: rows in order within a split, the splits one after the other; the
    splits follow from the shape as the kernel states it (148 SMs)."""
    n = x.shape[0]
    splits = max(1, min(2 * 148 // (-(-m // 64) * -(-k // 64)), -(-n // 256)))
    rows = -(-n // splits)
    total = np.zeros(x.shape[1])
    for r in range(0, n, rows):
        total = total + np.add.accumulate(x[r:r + rows], axis=0)[-1]
    return total, rows


@pytest.mark.parametrize("n,m,k", [(20000, 32, 32), (262144, 16, 8), (9999, 100, 64), (3000, 300, 13), (5001, 17, 17),
                                   (100000, 15, 1), (40000, 130, 130), (262144, 192, 64), (200, 3, 3)])
def test_gram_sums_in_the_order_of_the_shape(lib_built, n, m, k):
    """The order of a Gram's sums is part of its result (an unconverged pair of a solve shows it): ones
    and, in every column, pairs of +-2^70 that swallow the ones summed between them, so that the total
    tells which rows were summed with which.  Exact, whatever the tile: the 2^70 go first and last in a
    group of four rows, within which the order does not matter then."""
    import sparse_matrix_algorithms_b200 as S

    rng = np.random.default_rng(n + m)
    x = np.ones((n, m))
    _, rows = _gram_of_ones_in_order(x[:, :1], m, k)
    for c in range(m):
        a, b = np.sort(rng.choice(n // 8 - 1, 2, replace=False)) * 8 if n >= 64 else (0, 8)
        a, b = [r // rows * rows + r % rows // 4 * 4 for r in (int(a), int(b))]  # groups start with their split
        b = min(b + 3, b // rows * rows + rows - 1, n - 1)
        if b % rows % 4 == 3 and b > a:
            x[a, c], x[b, c] = 2.0 ** 70, -(2.0 ** 70)
    ref, _ = _gram_of_ones_in_order(x, m, k)
    assert n < 1000 or np.unique(ref).size > min(m, 8)
    C = _gram(S.context(), x, np.ones((n, k)), m, k)
    np.testing.assert_array_equal(C, np.broadcast_to(ref, (k, m)))


def test_gram_of_a_wide_block_with_little_memory_left(lib_built):
    """The workspace of the partial products stays small where the tiles alone fill the GPU: 1896
    columns with 1.5 GB of device memory left."""
    import torch
    import sparse_matrix_algorithms_b200 as S
    from sparse_matrix_algorithms_b200 import _lib as L

    n, k = 131072, 1896
    ctx = S.context()
    X = torch.randn(n, k, dtype=torch.float64, device="cuda")
    C = torch.empty(k, k, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - 3 * 2 ** 29, dtype=torch.uint8, device="cuda")
    try:
        L.check(L.load().sma_dense_gram_dev(ctx.handle, n, k, k, X.data_ptr(), k, X.data_ptr(), k, C.data_ptr(), k,
                                            1.0, 0.0))
    finally:
        del held
        torch.cuda.empty_cache()
    assert (C - X.T @ X).abs().max().item() <= 1e-13 * n


@pytest.mark.parametrize("p", [1, 2, 33, 64])
@pytest.mark.parametrize("odd", [0, 1])
def test_update_rounds_its_epilogue_once(lib_built, p, odd):
    """alpha acc + beta Y is one fused multiply-add on the rounded product beta Y, by the 16-byte path
    and the 8-byte one (an odd leading dimension): one product of one summand, exactly."""
    from fractions import Fraction
    import sparse_matrix_algorithms_b200 as S

    rng = np.random.default_rng(p)
    n, alpha, beta = 130, 0.37, 1.3
    X, B, Y = rng.standard_normal((n, 1)), rng.standard_normal((p, 1)), rng.standard_normal((n, p + odd))
    got = _update(S.context(), X, B, p, False, Y, alpha, beta, 1)
    acc, by = X * B.T, beta * Y[:, :p]
    ref = [[float(Fraction(alpha) * Fraction(a) + Fraction(b)) for a, b in zip(*r)] for r in zip(acc, by)]
    np.testing.assert_array_equal(got[:, :p], np.array(ref))
    np.testing.assert_array_equal(got[:, p:], Y[:, p:])
