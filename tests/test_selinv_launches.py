"""Launches of the selected inverse over the large fronts. A matrix whose hub is eliminated first fills in to
one dense front of n pivots, so fronts of any size come from a pattern of 3 n entries; grid meshes have fronts
with rows below their pivots. On the host: grids within the device's limits and every tile computed once. On
the GPU: a front of more than 16 384 pivots (more than 256 blocks) against the closed form."""
import numpy as np
import pytest
import scipy.sparse as sp

from fixtures import grid_laplacian
from inla_b200 import GpuSolver, _lib


def hub_first(n, v=None, d=None, a=None):
    """[[a, v'], [v, diag(d)]], the hub first."""
    v = np.ones(n - 1) if v is None else v
    d = np.full(n - 1, float(n)) if d is None else d
    j = np.arange(1, n)
    i0 = np.zeros(n - 1, dtype=np.int64)
    rows = np.concatenate([i0, j, j, [0]])
    cols = np.concatenate([j, i0, j, [0]])
    return sp.csc_matrix((np.concatenate([v, v, d, [float(n) if a is None else a]]), (rows, cols)), shape=(n, n))


def check(q, ordering, batch):
    s = GpuSolver(ordering)
    s.analyze(q)
    info = np.zeros(3, dtype=np.int64)
    rc = _lib.lib().inla_solver_check_selinv(s._h, batch, _lib.lptr(info))
    assert rc == _lib.INLA_OK, _lib.lib().inla_last_error()
    return info


@pytest.mark.parametrize("n", [130, 192, 193, 1087, 1088, 1089, 16384, 16385, 16449, 23168, 25600])
@pytest.mark.parametrize("batch", [1, 10])
def test_one_dense_front(n, batch):
    info = check(hub_first(n), _lib.ORDER_NATURAL, batch)
    nblk = -(-n // 64)
    joins = int(np.ceil(np.log2(nblk)))
    products = 2 * joins + 1  # T and X per join, then Sigma_KK
    assert info[0] >= products and info[1] <= 65535
    # every tile that is launched exists (T and X: all pairs of blocks once; Sigma_KK: the lower triangle),
    # whole or as two halves
    tiles = nblk * (nblk - 1) + nblk * (nblk + 1) // 2
    assert tiles <= info[2] <= 2 * tiles


@pytest.mark.parametrize("q", [grid_laplacian(90, 70, ridge=0.3), grid_laplacian(40, 200, ridge=0.3)], ids=["90x70", "40x200"])
@pytest.mark.parametrize("ordering", [_lib.ORDER_ND, _lib.ORDER_AMD])
@pytest.mark.parametrize("batch", [1, 7, 30])
def test_fronts_with_rows_below(q, ordering, batch):
    check(sp.csc_matrix(q), ordering, batch)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16449])
def test_front_of_more_than_256_blocks(n):
    rng = np.random.default_rng(n)
    v = rng.uniform(-1.0, 1.0, n - 1)
    d = rng.uniform(2.0, 3.0, n - 1)
    a = 2.0 * np.sum(v * v / d)
    q = hub_first(n, v, d, a)
    sv = GpuSolver(_lib.ORDER_NATURAL)
    sv.factorize(q)
    schur = a - np.sum(v * v / d)
    want = np.concatenate([[1.0 / schur], 1.0 / d + (v / d) ** 2 / schur])
    # scaled to a unit diagonal the eigenvalues are 1 and 1 +- sqrt(sum v^2 / (a d)) = 1 +- sqrt(1 / 2); a
    # backward stable inverse errs by a few n u cond of its largest entry
    scale = np.concatenate([[a], d])
    cond = (1.0 + np.sqrt(0.5)) / (1.0 - np.sqrt(0.5))
    tol = 20.0 * n * np.finfo(float).eps * cond
    err = np.abs(sv.diag_inv() - want) * scale
    assert np.max(err) <= tol * np.max(want * scale)
    ld = np.log(schur) + np.sum(np.log(d))
    assert abs(sv.log_abs_det() - ld) <= tol * abs(ld)
