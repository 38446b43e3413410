"""The tridiagonal eigen-solvers of the quadrature on the GPU, at the sizes where a warp's rows per lane change."""
import numpy as np
import pytest

import ftlm_extended_hubbard_b200 as F

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129, 159, 160]


def jacobi_rotations(a, b, rotations):
    """Classical Jacobi with a full pivot search (largest |A_ij|, i < j, first in row-major order)."""
    n = a.size
    A = np.diag(a) + np.diag(b[:n - 1], 1) + np.diag(b[:n - 1], -1)
    v = np.zeros(n)
    v[0] = 1.0
    for _ in range(rotations):
        U = np.abs(np.triu(A, 1))
        p, q = divmod(int(np.argmax(U)), n)
        if U[p, q] < 1e-14:
            break
        phi = 0.5 * np.arctan2(2.0 * A[p, q], A[q, q] - A[p, p])
        c, s = np.cos(phi), np.sin(phi)
        J = np.eye(n)
        J[p, p], J[q, q], J[p, q], J[q, p] = c, c, s, -s
        A = J.T @ A @ J
        A[p, q] = A[q, p] = 0.0
        v = v @ J
    return np.diag(A), v ** 2


@pytest.mark.parametrize("n", SIZES)
def test_capped_jacobi_follows_the_full_pivot_search(gpu, n):
    """After a few rotations the diagonal depends on every pivot taken: rounding of R rotations of a matrix of
    norm 40 is below R * 8 * 2.2e-16 * 40, so 1e-10 separates it from another pivot order."""
    rng = np.random.default_rng(n)
    a, b = 20 + 6 * rng.random((1, n)), 8 + rng.random((1, n))
    for rotations in (1, 40, 200):
        lam, w = F.tridiag_eig(a, b, np.array([n]), max_rot=rotations)
        lam0, w0 = jacobi_rotations(a[0], b[0], rotations)
        assert np.abs(lam[0] - lam0).max() <= 1e-10
        assert np.abs(w[0] - w0).max() <= 1e-10


def test_jacobi_with_equal_and_zero_entries(gpu):
    """Equal off-diagonal entries (every pivot a tie) and zero ones (split and diagonal matrices), with rotations
    enough to converge (the default cap of 120 n is not, from n of about 100)."""
    for n in (2, 33, 64, 130):
        a = np.stack([np.full(n, 3.0), np.arange(n) * 0.25, np.linspace(1, 2, n)])
        b = np.stack([np.full(n, 1.5), np.zeros(n), np.where(np.arange(n) % 3 == 0, 0.0, 1.0)])
        lam, w = F.tridiag_eig(a, b, np.full(3, n), max_rot=20 * n * n)
        for i in range(3):
            T = np.diag(a[i]) + np.diag(b[i, :n - 1], 1) + np.diag(b[i, :n - 1], -1)
            assert np.abs(np.sort(lam[i]) - np.linalg.eigvalsh(T)).max() <= 1e-11
            assert abs(w[i].sum() - 1.0) <= 1e-11


@pytest.mark.parametrize("n", [1, *SIZES])
def test_converged_quadrature_against_eigh(gpu, n):
    """log sum_k w_k exp(-b lam_k) and its energy from the converged solver: five chains (one past a block of four),
    one of them shorter, one scaled far from 1, one of a split matrix.  lam is good to a few n eps ||T|| (1e-12 of the
    norm), so the logarithm to b times that."""
    rng = np.random.default_rng(n)
    a, b = 20 + 6 * rng.random((5, n)), 8 + rng.random((5, n))
    b[3, ::3] = 0.0
    scale = np.array([1.0, 1.0, 1e-160, 1.0, 1.0])
    a, b = a * scale[:, None], b * scale[:, None]
    size = np.array([n, max(1, n - 1), n, n, n])
    for beta in (0.01, 1.0, 10.0):
        lq, e = quadrature_exact(a, b, size, beta)
        for c in range(5):
            m = size[c]
            T = np.diag(a[c, :m]) + np.diag(b[c, :m - 1], 1) + np.diag(b[c, :m - 1], -1)
            lam, z = np.linalg.eigh(T / scale[c])
            lam *= scale[c]
            w = z[0] ** 2
            x = np.log(np.maximum(w, 1e-300)) - beta * lam
            ref = x.max() + np.log(np.exp(x - x.max()).sum())
            tol = 1e-12 * (1.0 + beta * np.abs(lam).max())
            assert abs(lq[c] - ref) <= tol
            p = np.exp(x - ref)
            assert abs(e[c] - (p * lam).sum()) <= 1e-11 * np.abs(lam).max()


def quadrature_exact(a, b, n, beta):
    import ctypes as C

    from ftlm_extended_hubbard_b200._lib import call
    n = np.ascontiguousarray(n, np.int32)
    bt = np.array([beta])
    lq, e = np.zeros(len(n)), np.zeros(len(n))
    call("ftlm_gpu_tridiag_quadrature_exact", *[x.ctypes.data_as(C.c_void_p) for x in (a, b, n)], a.shape[0],
         a.shape[1], bt.ctypes.data_as(C.c_void_p), 1, lq.ctypes.data_as(C.c_void_p), e.ctypes.data_as(C.c_void_p))
    return lq, e
