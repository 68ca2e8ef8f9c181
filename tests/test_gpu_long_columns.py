"""Columns that every observation touches (intercepts) in the Newton right-hand side, the quadratic
forms, the traces, A^T v and the value fill, against dense numpy: sizes on both sides of the limits
at which a whole CTA takes a column over, batches that are no multiple of the problems per CTA, and
all-dense patterns."""
import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import models
from inla_b200.laplace import LaplaceModel
from inla_b200.multi import MultiModel

pytestmark = pytest.mark.gpu


def _problem(k, seed, dense=False):
    """Poisson counts of [intercept | k iid effects] (optionally on an all-dense pattern)."""
    rng = np.random.default_rng(seed)
    n = k + 1
    a = sp.hstack([sp.csr_matrix(np.ones((k, 1))), sp.identity(k)]).tocsr()
    m0 = sp.diags(np.r_[0.5, np.zeros(k)]).tocsc()
    m1 = sp.diags(np.r_[0.0, np.ones(k)]).tocsc()
    extra = [sp.csc_matrix(np.ones((n, n)))] if dense else [(a.T @ a).tocsc()]
    y = rng.poisson(np.exp(0.3 + 0.5 * rng.standard_normal(k))).astype(float)
    return models.build_latent(n, [m0, m1], "iid", extra_pattern=extra), a, y


def _reference(a, y, tau):
    """Mode, variances and trace pieces of the Poisson model by dense Newton iterations."""
    A, n = np.asarray(a.todense()), a.shape[1]
    d = np.r_[0.5, np.full(n - 1, tau)]
    x = np.zeros(n)
    for _ in range(50):
        mu = np.exp(A @ x)
        step = np.linalg.solve(np.diag(d) + A.T @ (mu[:, None] * A), A.T @ (y - mu) - d * x)
        x += step
        if np.abs(step).max() < 1e-12:
            break
    mu = np.exp(A @ x)
    H = np.diag(d) + A.T @ (mu[:, None] * A)
    S = np.linalg.inv(H)
    v = np.einsum("ij,jk,ik->i", A, S, A)
    z = S @ (A.T @ (mu * v))
    e0 = np.r_[0.5, np.zeros(n - 1)]
    e1 = np.r_[0.0, np.ones(n - 1)]
    return {"x": x, "var": np.diag(S), "logdet_post": np.linalg.slogdet(H)[1], "quad": x @ (d * x),
            "trQ": np.r_[(e0 * np.diag(S)).sum(), (e1 * np.diag(S)).sum(), (mu * v).sum()],
            "zMx": np.r_[(z * e0 * x).sum(), (z * e1 * x).sum()]}


def _check(out, ref, where):
    # the Newton loop stops at a step below 1e-5 and converges quadratically: the mode is within
    # about 1e-10; the other quantities are smooth functions of it
    for key in ("x", "var", "logdet_post", "quad", "trQ"):
        got = np.asarray(out[key])[where]
        assert np.max(np.abs(got - ref[key])) <= 1e-8 * max(1.0, np.max(np.abs(ref[key]))), key
    got = np.asarray(out["zMx"])[where][:2]
    assert np.max(np.abs(got - ref["zMx"])) <= 1e-8 * max(1.0, np.max(np.abs(ref["zMx"])))


# 2 k + 1 entries in the intercept's column of Q and A^T (limit 128, or 1024 on a dense pattern), k
# contributions to its diagonal entry (limit 128 in the fill, 32 in the traces)
@pytest.mark.parametrize("k,dense", [(31, False), (33, False), (63, False), (64, False), (128, False), (129, False),
                                     (1500, False), (511, True), (512, True), (1030, True)])
@pytest.mark.parametrize("B", [1, 5])
def test_intercept_column(k, dense, B):
    model, a, y = _problem(k, 100 + k, dense)
    m = LaplaceModel(model, a=a, family="poisson", y=y, max_batch=B)
    taus = 3.0 + 0.5 * np.arange(B)
    out = m.eval(np.array([[1.0, t] for t in taus]), variances=True, gradient=True)
    assert (out["status"] == 0).all()
    for b in range(B):
        _check(out, _reference(a, y, taus[b]), b)


def test_intercept_columns_of_many_models():
    ks = [40, 511, 512, 900]
    parts = [_problem(k, 7 + k) for k in ks]
    m = MultiModel([p[0] for p in parts], [p[1] for p in parts], [p[2] for p in parts], max_batch=2)
    taus = np.array([[2.0 + g for g in range(4)], [4.0 - 0.5 * g for g in range(4)]])
    out = m.eval(np.array([[[1.0, t] for t in row] for row in taus]), variances=True, gradient=True)
    assert (out["status"] == 0).all()
    for b in range(2):
        for g, (_, a, y) in enumerate(parts):
            one = {k: out[k][b, g] for k in ("logdet_post", "quad", "trQ", "zMx")}
            one.update({k: m.split(out[k])[g][b] for k in ("x", "var")})
            _check(one, _reference(a, y, taus[b, g]), ...)
