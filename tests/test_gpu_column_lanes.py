"""Lanes per column in the Newton right-hand side and A^T v: banded models with column lengths on both sides of
the line between eight lanes and a warp, at several orders (the line rises with the order), against dense
numpy."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import models
from inla_b200.laplace import LaplaceModel

pytestmark = pytest.mark.gpu


def _band(n, w, rng):
    d = [rng.uniform(-1.0, 1.0, n - k) for k in range(1, w + 1)]
    return (sp.diags(d + d, [*range(1, w + 1), *range(-1, -w - 1, -1)]) + (2 * w + 2) * sp.identity(n)).tocsc()


# 2 w + 2 entries per column with the observation's: lines at 16 (n = 300), 18 (900) and 40 (2000)
@pytest.mark.parametrize("n,w", [(300, 6), (300, 7), (300, 8), (300, 70), (900, 8), (900, 9), (2000, 19), (2000, 20)])
@pytest.mark.parametrize("B", [1, 6])
def test_banded_poisson(n, w, B):
    rng = np.random.default_rng(n + w)
    m0, m1 = _band(n, w, rng), _band(n, w, rng)
    y = rng.poisson(np.exp(0.3 * rng.standard_normal(n))).astype(float)
    m = LaplaceModel(models.build_latent(n, [m0, m1], "band"), family="poisson", y=y, max_batch=B)
    coefs = np.array([[1.0 + 0.1 * b, 0.5] for b in range(B)])
    out = m.eval(coefs, variances=True, gradient=True)
    assert (out["status"] == 0).all()
    for b in (0, B - 1):
        q = (coefs[b, 0] * m0 + coefs[b, 1] * m1).toarray()
        x = np.zeros(n)
        for _ in range(50):
            mu = np.exp(x)
            step = np.linalg.solve(q + np.diag(mu), y - mu - q @ x)
            x += step
            if np.abs(step).max() < 1e-13:
                break
        mu = np.exp(x)
        s = np.linalg.inv(q + np.diag(mu))
        z = s @ (mu * np.diag(s))
        # the Newton loop stops at a step below 1e-5 and converges quadratically: the mode is within about
        # 1e-10; the other quantities are smooth functions of it
        for got, want in ((out["x"][b], x), (out["var"][b], np.diag(s)), (out["quad"][b], x @ q @ x),
                          (out["zMx"][b][:2], np.array([z @ (m0 @ x), z @ (m1 @ x)]))):
            assert np.max(np.abs(got - want)) <= 1e-8 * max(1.0, np.max(np.abs(want)))
