"""Selected inverse of one large front (several 64-column blocks) whose triangular factor is ill-conditioned:
the products with the explicit inverse of the whole front's factor must not lose more than a backward stable
inversion may. Reference: LDL^T and inverse in extended precision."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import GpuSolver, _lib

pytestmark = pytest.mark.gpu


def _inverse_diagonal(a):
    """diag(A^-1) by LDL^T without pivoting in long double (64-bit mantissa)."""
    n = len(a)
    w = a.astype(np.longdouble)
    low = np.eye(n, dtype=np.longdouble)
    for j in range(n):
        low[j + 1:, j] = w[j + 1:, j] / w[j, j]
        w[j + 1:, j + 1:] -= np.outer(low[j + 1:, j], w[j, j + 1:])
    x = np.eye(n, dtype=np.longdouble)
    for i in range(1, n):
        x[i, :i] -= low[i, :i] @ x[:i, :i]
    return np.sum(x * x / np.diag(w)[:, None], axis=0)


def _matrix(kind, n):
    rng = np.random.default_rng(n)
    if kind == "kahan":  # condition of L grows like (1 + c)^n
        low = np.eye(n) - 0.02 * np.tril(np.ones((n, n)), -1)
        return low @ low.T
    if kind == "kernel":
        t = np.sort(rng.uniform(0.0, 1.0, n))
        return np.exp(-0.5 * ((t[:, None] - t) / 0.05) ** 2) + 1e-6 * np.eye(n)
    if kind == "rw2":  # second differences plus a small ridge, permuted
        d = np.diff(np.eye(n), 2, axis=0)
        p = rng.permutation(n)
        return (d.T @ d + 1e-6 * np.eye(n))[np.ix_(p, p)]
    b = rng.uniform(-1.0, 1.0, (n, n))  # random L, pivots over six orders of magnitude
    low = np.eye(n) + np.tril(b, -1) * (2.7 / np.sqrt(n))
    return low @ np.diag(10.0 ** rng.uniform(-3.0, 3.0, n)) @ low.T


@pytest.mark.parametrize("kind", ["kahan", "kernel", "rw2", "random"])
@pytest.mark.parametrize("n", [129, 300])
def test_diagonal_of_the_inverse(kind, n):
    a = _matrix(kind, n)
    a = np.tril(a) + np.tril(a, -1).T
    a[a == 0.0] = np.finfo(float).tiny  # one dense front
    want = _inverse_diagonal(a).astype(float)
    sv = GpuSolver(_lib.ORDER_NATURAL)
    sv.factorize(sp.csc_matrix(a))
    err = np.max(np.abs(sv.diag_inv() - want)) / np.max(want)
    # a backward stable inversion errs by up to a few n u cond of the largest entry
    assert err <= 4.0 * n * np.finfo(float).eps * np.linalg.cond(a)
