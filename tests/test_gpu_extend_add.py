"""Extend-add of large fronts from lists of the children's columns: a dense block whose front has from one to
some hundred children, each touching from one to all of its rows (around the 32-row pieces, eight of them in
flight, and the 32 list entries read at a time), by level launches and by the persistent schedule."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import GpuSolver, _lib

pytestmark = pytest.mark.gpu

HUB = 300


def _arrow(nleaf, width, seed):
    """Leaves (single unknowns) coupled to `width` rows each of a dense block of HUB unknowns."""
    rng = np.random.default_rng(seed)
    n = nleaf + HUB
    a = np.zeros((n, n))
    b = rng.uniform(-1.0, 1.0, size=(HUB, HUB))
    a[nleaf:, nleaf:] = 0.5 * (b + b.T)
    for i in range(nleaf):
        w = width if width > 0 else int(rng.integers(1, HUB + 1))
        rows = nleaf + np.sort(rng.choice(HUB, size=w, replace=False))
        a[i, rows] = rng.uniform(-1.0, 1.0, size=w)
        a[rows, i] = a[i, rows]
    np.fill_diagonal(a, 0.0)
    np.fill_diagonal(a, 1.0 + 2.0 * np.abs(a).sum(axis=1))
    return a


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("nleaf,width", [(1, HUB), (7, 256), (8, 257), (9, 33), (31, 32), (32, 31), (33, 1), (65, 64),
                                         (65, 65), (200, 5), (130, 0)])
def test_arrow(nleaf, width, mode):
    a = _arrow(nleaf, width, 100 * nleaf + width)
    n = a.shape[0]
    _lib.check(_lib.lib().inla_set_persistent_schedule(mode))
    try:
        sv = GpuSolver()
        sv.factorize(sp.csc_matrix(a))
    finally:
        _lib.check(_lib.lib().inla_set_persistent_schedule(1))
    # dominance by a factor of two: LDL^T is backward stable with growth of at most two
    tol = 20.0 * n * np.finfo(float).eps * np.linalg.cond(a)
    inv = np.linalg.inv(a)
    b = np.random.default_rng(n).standard_normal(n)
    assert np.max(np.abs(sv.solve(b) - inv @ b)) <= tol * np.max(np.abs(inv @ b))
    ld = np.linalg.slogdet(a)[1]
    assert abs(sv.log_abs_det() - ld) <= tol * max(1.0, abs(ld))
    assert np.max(np.abs(sv.diag_inv() - np.diag(inv))) <= tol * np.max(np.abs(inv))
