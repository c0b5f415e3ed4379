"""KPM moments on the GPU against the oracle (same seeded Rademacher vectors)."""
import os
import sys

import numpy as np
import pytest
import scipy.sparse as sp

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

import sma_oracle as O  # noqa: E402
from sparse_matrix_algorithms_b200 import matrices as M  # noqa: E402

pytestmark = pytest.mark.gpu


def test_kpm_moments_match_oracle(lib_built):
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(10, 16.5, 0)
    smin, smax = O.gershgorin_bounds(A)
    mu, pv = S.kpm_moments(A, 64, 8, smin=smin, smax=smax, seed=4, per_vector=True)
    mo, pvo = O.kpm_moments(A, 64, 8, 4, smin, smax, per_vector=True)
    assert mu[0] == 1.0
    np.testing.assert_allclose(pv, pvo, rtol=0, atol=1e-11)
    np.testing.assert_allclose(mu, pv.mean(axis=1), rtol=0, atol=1e-15)
    for a, b in [(-1.0, 1.0), (2.0, 6.0)]:
        assert abs(S.kpm_count(mu, A.shape[0], smin, smax, a, b) -
                   O.kpm_count(mu, A.shape[0], smin, smax, a, b)) <= 1e-9 * A.shape[0]


@pytest.mark.parametrize("M_", [1, 2, 7, 8])
def test_kpm_moments_diagonal_exact(lib_built, M_):
    import sparse_matrix_algorithms_b200 as S

    lam = np.linspace(-2.0, 3.0, 513)
    A = sp.diags(lam).tocsr()
    mu = S.kpm_moments(A, M_, 5, smin=-2.5, smax=3.5, seed=1)
    x = (lam - 0.5) / 3.0
    exact = np.array([np.mean(np.cos(k * np.arccos(x))) for k in range(M_)])
    np.testing.assert_allclose(mu, exact, rtol=0, atol=1e-12)


def test_kpm_stencil_equals_csr(lib_built):
    """The Anderson stencil's products are bit-identical to the CSR matrix's."""
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(16, 16.5, 2)
    smin, smax = O.gershgorin_bounds(A)
    m1 = S.kpm_moments(A, 128, 4, smin=smin, smax=smax)
    m2 = S.kpm_moments(S.AndersonOperator(16, 16.5, 2), 128, 4, smin=smin, smax=smax)
    np.testing.assert_array_equal(m1, m2)


def test_kpm_count_tracks_dense_count(lib_built):
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(12, 16.5, 0)
    lam = np.linalg.eigvalsh(A.toarray())
    smin, smax = O.gershgorin_bounds(A)
    mu = S.kpm_moments(A, 512, 64, smin=smin, smax=smax)
    for a, b in [(-0.5, 0.5), (-4.0, -2.0)]:
        exact = int(np.sum((lam >= a) & (lam <= b)))
        est = S.kpm_count(mu, A.shape[0], smin, smax, a, b)
        assert abs(est - exact) <= 0.1 * exact + 4, (a, b, est, exact)


@pytest.mark.parametrize("n", [64, 1331])
@pytest.mark.parametrize("R", [1, 3, 16, 33])
@pytest.mark.parametrize("M_", [3, 34])
def test_kpm_moments_of_ragged_blocks(lib_built, n, R, M_):
    """Blocks of odd widths (the recurrence runs on padded rows), few rows and odd moment counts."""
    import sparse_matrix_algorithms_b200 as S

    A = M.lap1d(n) if n == 64 else M.anderson3d(11, 16.5, 1)
    smin, smax = O.gershgorin_bounds(A)
    _, pv = S.kpm_moments(A, M_, R, smin=smin, smax=smax, seed=2, per_vector=True)
    _, pvo = O.kpm_moments(A, M_, R, 2, smin, smax, per_vector=True)
    np.testing.assert_allclose(pv, pvo, rtol=0, atol=1e-11)


@pytest.mark.parametrize("R", [2, 12, 20, 40, 64, 72])
@pytest.mark.parametrize("kind", ["csr", "anderson", "xxz"])
def test_kpm_dots_of_every_row_layout(lib_built, kind, R):
    """The step sums its own dots per CTA where 16 or fewer threads make a row (in shuffles, or a
    tree for other counts than powers of two), else a pass of its own does: a last CTA with rows
    missing, more CTAs than one group of the second stage, an odd number of moments."""
    import sparse_matrix_algorithms_b200 as S

    A = M.xxz_sz0(14, 5.0, 1) if kind == "xxz" else M.anderson3d(15, 16.5, 1)
    op = {"csr": lambda: S.SparseOperator(A), "anderson": lambda: S.AndersonOperator(15, 16.5, 1),
          "xxz": lambda: S.XXZOperator(14, 5.0, 1)}[kind]()
    smin, smax = O.gershgorin_bounds(A)
    _, pv = S.kpm_moments(op, 21, R, smin=smin, smax=smax, seed=3, per_vector=True)
    _, pvo = O.kpm_moments(A, 21, R, 3, smin, smax, per_vector=True)
    np.testing.assert_allclose(pv, pvo, rtol=0, atol=1e-11)


@pytest.mark.parametrize("L,M_,R", [(84, 32, 16), (24, 279, 80)])
def test_kpm_partials_in_many_batches(lib_built, L, M_, R):
    """More steps than the partials of one batch, which their number does not divide: the step's own
    sums (six steps a batch) and the pass over the blocks (132), an even and an odd number of moments."""
    import sparse_matrix_algorithms_b200 as S

    A = M.anderson3d(L, 16.5, 1)
    smin, smax = O.gershgorin_bounds(A)
    _, pv = S.kpm_moments(A, M_, R, smin=smin, smax=smax, seed=3, per_vector=True)
    _, pvo = O.kpm_moments(A, M_, R, 3, smin, smax, per_vector=True)
    np.testing.assert_allclose(pv, pvo, rtol=0, atol=1e-11)


def test_kpm_with_little_memory_left(lib_built):
    """Three unpadded blocks and the sums of one step are all that a call needs: 13 columns, which run
    padded to 16 where there is room for them (1.04 GB of blocks, 0.85 GB unpadded).  In a process of
    its own: the library keeps the memory that it has had."""
    import subprocess

    code = """if True:
        import sys, numpy as np, torch
        import sparse_matrix_algorithms_b200 as S
        op = S.AndersonOperator(140, 16.5, 1)
        moments = lambda: S.kpm_moments(op, 9, 13, smin=-15.0, smax=15.0, seed=3, per_vector=True)[1]
        torch.cuda.init()
        held = torch.empty(torch.cuda.mem_get_info()[0] - 960 * 10 ** 6, dtype=torch.uint8, device="cuda")
        got = moments()
        del held
        torch.cuda.empty_cache()
        np.testing.assert_allclose(got, moments(), rtol=0, atol=1e-13)
    """
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, cwd=ROOT, timeout=300)
    assert out.returncode == 0, out.stderr.decode()[-2000:]
