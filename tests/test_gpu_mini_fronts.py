"""Forests whose fronts have at most eight rows (eight lanes per front, a few levels per launch): chains,
hubs with more children than lanes, trees, cliques of up to eight, and single unknowns, against dense
linear algebra."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import GpuSolver, _lib

pytestmark = pytest.mark.gpu


def _edges(kind, n):
    if kind == "chain":
        return [(i, i + 1) for i in range(n - 1)]
    if kind == "hub":
        return [(0, i) for i in range(1, n)]
    if kind == "tree":
        return [((i - 1) // 3, i) for i in range(1, n)]
    if kind == "wide chain":
        return [(i, j) for i in range(n) for j in range(i + 1, min(i + 4, n))]
    return [(i, j) for i in range(n) for j in range(i)]  # clique


def _forest(parts, signs, seed):
    rng = np.random.default_rng(seed)
    n = sum(m for _, m in parts)
    a, off = np.zeros((n, n)), 0
    for kind, m in parts:
        for i, j in _edges(kind, m):
            a[off + i, off + j] = a[off + j, off + i] = rng.uniform(-1.0, 1.0)
        off += m
    s = np.where(rng.uniform(size=n) < 0.4, -1.0, 1.0) if signs else np.ones(n)
    np.fill_diagonal(a, s * (1.0 + 2.0 * np.abs(a).sum(axis=1)))
    return a


FORESTS = {
    "chains": [("chain", m) for m in (1, 2, 3, 7, 8, 9, 33, 64, 150)],
    "hubs": [("hub", m) for m in (2, 8, 9, 10, 17, 18, 40)],
    "trees": [("tree", m) for m in (4, 13, 40, 121)],
    "wide chains": [("wide chain", m) for m in (4, 8, 9, 31, 100)],
    "cliques": [("clique", m) for m in range(1, 9)],
    "all": [("chain", 21), ("hub", 30), ("tree", 50), ("wide chain", 40), ("clique", 8), ("chain", 1)] * 5,
}


@pytest.mark.parametrize("name", list(FORESTS))
@pytest.mark.parametrize("signs", [False, True])
def test_forest(name, signs):
    a = _forest(FORESTS[name], signs, len(name))
    n = a.shape[0]
    q = sp.csc_matrix(a)
    _lib.check(_lib.lib().inla_set_persistent_schedule(0))  # level launches
    try:
        sv = GpuSolver()
        sv.factorize(q)
    finally:
        _lib.check(_lib.lib().inla_set_persistent_schedule(1))
    # dominance by a factor of two: LDL^T without pivoting is backward stable with growth of at most two,
    # so relative errors stay within a few n u cond
    tol = 20.0 * n * np.finfo(float).eps * np.linalg.cond(a)
    inv = np.linalg.inv(a)
    b = np.random.default_rng(n).standard_normal(n)
    x = sv.solve(b)
    assert np.max(np.abs(x - inv @ b)) <= tol * np.max(np.abs(inv @ b))
    ld = np.linalg.slogdet(a)[1]
    assert abs(sv.log_abs_det() - ld) <= tol * max(1.0, abs(ld))
    d = sv.diag_inv()
    assert np.max(np.abs(d - np.diag(inv))) <= tol * np.max(np.abs(inv))
