"""The host check of the persistent factorization queue sees a wait that is too short (no GPU): every count
that a task of a large front waits for is lowered by one in turn, and every one must be reported -- on the
GPU such a task would read what the step before is still writing."""
import numpy as np
import pytest
import scipy.sparse as sp

from fixtures import grid_laplacian
from inla_b200 import GpuSolver, _lib

DIAG, NEXT, ROWS, UPDATE = 3, 4, 5, 6
NEED, ARG = 3, 5


def edit(s, task, field, delta):
    e = np.zeros(6, dtype=np.int32)
    rc = _lib.lib().inla_solver_check_schedule_edit(s._h, task, field, delta, _lib.iptr(e))
    return rc, e


def dense(n):
    return sp.csc_matrix(np.ones((n, n)) + n * np.eye(n))


def coupled_blocks(k, sep):
    """Two dense blocks of k, each coupled to a dense separator."""
    a = np.ones((2 * k + sep, 2 * k + sep))
    a[:k, k:2 * k] = a[k:2 * k, :k] = 0.0
    return sp.csc_matrix(a + 2.0 * len(a) * np.eye(len(a)))


@pytest.mark.parametrize("q, several", [(dense(97), False), (dense(128), False), (dense(129), False),
                                           (dense(330), True), (coupled_blocks(100, 150), True),
                                           (coupled_blocks(130, 64), True), (grid_laplacian(80, 80, ridge=0.3), False)],
                         ids=["97", "128", "129", "330", "blocks100", "blocks130", "grid"])
def test_every_wait_is_checked(q, several):
    s = GpuSolver(_lib.ORDER_ND)
    s.analyze(sp.csc_matrix(q))
    info = np.zeros(3, dtype=np.int64)
    assert _lib.lib().inla_solver_check_schedule(s._h, _lib.lptr(info)) == _lib.INLA_OK
    seen = set()
    for t in range(int(info[0])):
        rc, e = edit(s, t, NEED, 0)
        assert rc == _lib.INLA_OK
        if e[0] not in (DIAG, NEXT, ROWS, UPDATE):
            continue
        for field in (NEED, ARG):
            if e[field] == 0:
                continue
            seen.add((int(e[0]), field))
            rc, _ = edit(s, t, field, -1)
            assert rc == _lib.INLA_ERR_INTERNAL, (t, list(e), field)
            rc, _ = edit(s, t, field, 10 ** 6)  # a wait that nothing can end
            assert rc == _lib.INLA_ERR_INTERNAL, (t, list(e), field)
    assert (DIAG, NEED) in seen  # a block waits for its extend-add
    if several:  # several blocks: every kind of wait occurs
        assert {(NEXT, NEED), (NEXT, ARG), (ROWS, NEED), (ROWS, ARG), (UPDATE, NEED)} <= seen


def test_bad_edits_are_refused():
    s = GpuSolver(_lib.ORDER_ND)
    s.analyze(dense(128))
    for task, field in ((-1, 3), (10 ** 6, 3), (0, 6), (0, -1)):
        assert edit(s, task, field, 0)[0] == _lib.INLA_ERR_INVALID
