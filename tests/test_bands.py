"""Host check of the bands of small fronts (no GPU): tasks cover every front of a band once, children first,
and stay short whatever the tree -- a hub with thousands of leaves, nested groups and k-ary trees are one
connected component each, and a task runs its fronts one after the other."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import GpuSolver, _lib

LONGEST = 16  # fronts of a task


def pattern(n, i, j):
    a = sp.coo_matrix((np.ones(len(i)), (i, j)), shape=(n, n))
    return (a + a.T + 8.0 * sp.identity(n)).tocsc()


def star(leaves, hubs=1):
    i = np.concatenate([np.repeat(np.arange(hubs), leaves), np.tril_indices(hubs, -1)[0]])
    j = np.concatenate([hubs + np.tile(np.arange(leaves), hubs), np.tril_indices(hubs, -1)[1]])
    return pattern(hubs + leaves, i, j)


def nested(groups, per):
    g = 1 + np.arange(groups)
    return pattern(1 + groups + groups * per, np.concatenate([np.zeros(groups, int), np.repeat(g, per)]),
                   np.concatenate([g, 1 + groups + np.arange(groups * per)]))


def tree(n, ary):
    i = np.arange(1, n)
    return pattern(n, (i - 1) // ary, i)


def chain(n, width):
    d = [np.ones(n - k) for k in range(1, width + 1)]
    return sp.diags(d + d + [8.0 * np.ones(n)], [*range(1, width + 1), *range(-1, -width - 1, -1), 0]).tocsc()


PATTERNS = {
    "star": star(24000), "three hubs": star(24000, 3), "short star": star(LONGEST + 4), "nested": nested(480, 49),
    "nested, small groups": nested(500, 7), "binary tree": tree(4000, 2), "ternary tree": tree(4000, 3),
    "16-ary tree": tree(4000, 16), "chain": chain(5000, 1), "wide chain": chain(3000, 3),
    "stars and chains": sp.block_diag([star(60), chain(400, 1), star(5)] * 3).tocsc(),
}


@pytest.mark.parametrize("ordering", [_lib.ORDER_ND, _lib.ORDER_AMD])
@pytest.mark.parametrize("name", list(PATTERNS))
def test_tasks_are_short(name, ordering):
    s = GpuSolver(ordering)
    s.analyze(PATTERNS[name])
    info = np.zeros(3, dtype=np.int64)
    assert _lib.lib().inla_solver_check_bands(s._h, _lib.lptr(info)) == _lib.INLA_OK, _lib.lib().inla_last_error()
    assert info[2] <= LONGEST
    if name == "binary tree":  # what the bands are for
        assert info[0] >= 1 and info[1] > 100


def test_no_band_without_small_fronts():
    s = GpuSolver(_lib.ORDER_ND)
    s.analyze(sp.csc_matrix(np.ones((40, 40))))
    info = np.zeros(3, dtype=np.int64)
    assert _lib.lib().inla_solver_check_bands(s._h, _lib.lptr(info)) == _lib.INLA_OK
    assert list(info) == [0, 0, 0]
