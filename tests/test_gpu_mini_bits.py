"""The eight-lane kernels of the bands of small fronts against the one-warp kernels, bit for bit: the same
forest alone (its levels form bands) and beside a path of larger fronts as deep as the forest (no level has
small fronts only, so every front takes the one-warp kernels), and in the persistent schedule, which knows no
bands. Batches of one and three problems."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import BatchSolver, GpuSolver, _lib

NATURAL = _lib.ORDER_NATURAL


def cliques_on_separators(groups, per, size, sep):
    """``groups`` separators of ``sep`` unknowns with ``per`` cliques of ``size`` each, joined in pairs above."""
    edges, n, roots = [], 0, []

    def clique(ids):
        edges.extend((i, j) for i in ids for j in ids if i < j)

    for _ in range(groups):
        members = []
        for _ in range(per):
            members.append(list(range(n, n + size)))
            n += size
        s = list(range(n, n + sep))
        n += sep
        for m in members:
            clique(m + s)
        roots.append(s)
    while len(roots) > 1:
        nxt = []
        for a in range(0, len(roots) - 1, 2):
            s = list(range(n, n + sep))
            n += sep
            clique(roots[a] + s)
            clique(roots[a + 1] + s)
            nxt.append(s)
        if len(roots) % 2:
            nxt.append(roots[-1])
        roots = nxt
    return n, edges


def tree(n, ary):
    """Complete ``ary`` tree, children before parents."""
    return n, [(n - 1 - i, n - 1 - (i - 1) // ary) for i in range(1, n)]


FORESTS = {
    "cliques 4 on 2": cliques_on_separators(13, 3, 4, 2),
    "cliques 5 on 3": cliques_on_separators(16, 2, 5, 3),
    "cliques 1 on 1": cliques_on_separators(40, 4, 1, 1),
    "binary": tree(300, 2),
    "ternary": tree(200, 3),
    "8-ary": tree(200, 8),
}


def matrix(n, edges, signs, seed):
    rng = np.random.default_rng(seed)
    i, j = np.array(edges).T
    a = sp.coo_matrix((rng.uniform(-1.0, 1.0, len(i)), (i, j)), shape=(n, n)).tocsc()
    a = a + a.T
    s = np.where(rng.uniform(size=n) < 0.4, -1.0, 1.0) if signs else np.ones(n)
    q = (a + sp.diags(s * (1.0 + 2.0 * np.asarray(abs(a).sum(axis=0)).ravel()))).tocsc()
    q.sort_indices()
    return q


def larger_fronts(levels):
    """A path of dense 12-column blocks, each coupled to the next: one front of 24 rows per level."""
    k = 12
    a = np.zeros((k * levels, k * levels))
    for b in range(levels):
        e = min(k * (b + 2), k * levels)
        a[k * b:e, k * b:e] = 0.1
    np.fill_diagonal(a, 2.0 * k)
    return sp.csc_matrix(a)


def bands(q):
    s = GpuSolver(NATURAL)
    s.analyze(q)
    info = np.zeros(3, dtype=np.int64)
    assert _lib.lib().inla_solver_check_bands(s._h, _lib.lptr(info)) == _lib.INLA_OK
    return int(info[0]), s.info()


def outputs(q, B, mode, rhs):
    _lib.check(_lib.lib().inla_set_persistent_schedule(mode))
    try:
        sv = BatchSolver(q, max_batch=B, ordering=NATURAL)
        ld, st = sv.factorize(np.stack([q.data * (1.0 + 0.25 * b) for b in range(B)]))
    finally:
        _lib.check(_lib.lib().inla_set_persistent_schedule(1))
    assert (st == 0).all()
    return sv.solve(rhs), sv.diag_inv()


@pytest.mark.parametrize("name", list(FORESTS))
def test_patterns_take_both_routes(name):
    n, edges = FORESTS[name]
    q = matrix(n, edges, False, 1)
    nb, info = bands(q)
    assert nb >= 1
    both = sp.block_diag([q, larger_fronts(info["nlevels"] + 2)]).tocsc()
    assert bands(both)[0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(FORESTS))
@pytest.mark.parametrize("signs", [False, True])
@pytest.mark.parametrize("B", [1, 3])
def test_same_bits(name, signs, B):
    n, edges = FORESTS[name]
    q = matrix(n, edges, signs, 17 * B)
    both = sp.block_diag([q, larger_fronts(bands(q)[1]["nlevels"] + 2)]).tocsc()
    both.sort_indices()
    rhs = np.random.default_rng(n).standard_normal((B, both.shape[0]))
    x, d = outputs(q, B, 0, rhs[:, :n])
    xb, db = outputs(both, B, 0, rhs)
    assert np.array_equal(x, xb[:, :n])
    assert np.array_equal(d, db[:, :n])
    xp, _ = outputs(q, B, 2, rhs[:, :n])
    assert np.array_equal(x, xp)
    # and right: dominance by a factor of two, see the dense comparison of the same kernels
    dense = q.toarray()
    tol = 20.0 * n * np.finfo(float).eps * np.linalg.cond(dense)
    assert np.max(np.abs(d[0] - np.diag(np.linalg.inv(dense)))) <= tol * np.max(np.abs(np.linalg.inv(dense)))
