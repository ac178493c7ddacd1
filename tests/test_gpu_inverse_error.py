"""GPU test of the inverse's error at a block size without a panel form, against
64 bits: no larger than the unblocked Gauss-Jordan elimination's (numpy, one
rank-1 update a column, the reference's partial pivoting) on the same
matrices.  A chain of decoupled blocks at E = 0 has G^R_ll = (-H_ll)^-1.  The
two errors' log ratio scatters by 0.5 a matrix between such algorithms, so the
geometric mean over 64 matrices is within 1.2 (three standard deviations) of
the true ratio; panels of 48 columns summed as one give 1.4."""
import numpy as np
import pytest

from test_gpu_cms import rgf  # noqa: F401

pytestmark = pytest.mark.gpu


def _gauss_jordan(A):
    X, n, perm = A.copy(), len(A), []
    for k in range(n):
        q = k + int(np.argmax(np.abs(X[k:, k].real) + np.abs(X[k:, k].imag)))
        perm.append(q)
        X[[k, q]] = X[[q, k]]
        p, f = 1 / X[k, k], X[:, k].copy()
        f[k] = 0
        r = X[k] * p
        r[k] = p
        X[:, k] = 0
        X[k] = 0
        X -= np.outer(f, r)
        X[k] = r
    for k in range(n - 1, -1, -1):
        X[:, [k, perm[k]]] = X[:, [perm[k], k]]
    return X


def _error(A, X):
    A, Y, one = A.astype(np.clongdouble), X.astype(np.clongdouble), np.eye(len(A), dtype=np.clongdouble)
    for _ in range(2):
        Y = Y + Y @ (one - A @ Y)
    return float(np.linalg.norm((X - Y).astype(complex)) / np.linalg.norm(Y.astype(complex)))


def test_error_of_the_inverse(rgf):  # noqa: F811
    nm, nx = 136, 64
    rng = np.random.default_rng(136)
    A = rng.normal(size=(nx, nm, nm)) + 1j * rng.normal(size=(nx, nm, nm))
    B = (A + np.conj(np.swapaxes(A, -1, -2))) / (2 * np.sqrt(nm))   # Hermitian, with a small broadening
    A[::2] = (B + (0.1 + 1e-3j) * np.eye(nm))[::2]
    H = np.ascontiguousarray(np.swapaxes(-A, -1, -2))
    G = np.zeros((1, nx, nm, nm), complex)
    with rgf.Context(rgf.Options()) as ctx:
        ctx.solve_energies(H, np.zeros_like(H), np.zeros(1), (0.1, -0.1), (300.0, 300.0), ldos=G)
    ratio = [np.log(_error(a, g.T) / _error(a, _gauss_jordan(a))) for a, g in zip(A, G[0])]
    assert np.exp(np.mean(ratio)) <= 1.2
