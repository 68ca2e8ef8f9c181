"""The blocked dense LDL^T inside the fronts, on dense matrices (one front): orders around the 8-wide
pivot blocks and the front size classes, negative pivots, and entries scaled by powers of two far from
one (the reciprocal of a pivot has a plain-division path outside 2^+-964)."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import GpuSolver, InlaError

pytestmark = pytest.mark.gpu


def _matrix(n, seed, signs):
    """Diagonally dominant, so that LDL^T without pivoting is stable for either sign pattern."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1.0, 1.0, size=(n, n))
    a = 0.5 * (a + a.T)
    s = np.where(rng.uniform(size=n) < 0.4, -1.0, 1.0) if signs else np.ones(n)
    np.fill_diagonal(a, s * (n + 1.0 + rng.uniform(0.0, 5.0, size=n)))
    return a


@pytest.mark.parametrize("n", [33, 39, 40, 41, 63, 64, 65, 71, 95, 96, 97, 103, 128, 129, 200])
@pytest.mark.parametrize("signs", [False, True])
@pytest.mark.parametrize("shift", [0, 600, -600, 980])
def test_dense_front(n, signs, shift):
    a = _matrix(n, 1000 + n, signs)
    sv = GpuSolver()
    if shift < 0:  # every pivot is below the gate |D| < 1e-14
        with pytest.raises(InlaError):
            sv.factorize(sp.csc_matrix(np.ldexp(a, shift)))
        return
    sv.factorize(sp.csc_matrix(np.ldexp(a, shift)))
    b = np.random.default_rng(n).standard_normal(n)
    # condition number below 10 (off-diagonal row sums below n / 2 against n + 1): a backward stable
    # solve errs by at most a few n u
    tol = 50.0 * n * np.finfo(float).eps
    inv = np.linalg.inv(a)
    x = sv.solve(np.ldexp(b, shift))
    assert np.max(np.abs(x - inv @ b)) <= tol * np.max(np.abs(inv @ b))
    d = np.ldexp(sv.diag_inv(), shift)
    assert np.max(np.abs(d - np.diag(inv))) <= tol * np.max(np.abs(np.diag(inv)))
    ld = np.linalg.slogdet(a)[1] + n * shift * np.log(2.0)
    assert abs(sv.log_abs_det() - ld) <= tol * max(1.0, abs(ld))
