"""Workloads of the framework's public entry points at the sizes its users meet.

``listed`` names twelve: the drop-in solver seam at the smallest and an ordinary size, the batched
device solver at one and at ten problems, Laplace evaluations of every latent model and family
(with gradients or with marginal variances), many uneven models at once, a whole fit and the
mesh tools. ``draw`` gives more of the same kinds over the same ranges. A case is a dict of plain
values; ``prepare`` builds what a program holds before the call, ``run`` is one pass, ``work`` the
bytes and operations one pass cannot do without, ``exact`` the outputs by dense 64-bit algebra.
"""
import ctypes
import math
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path.cwd() / "rust-inla_b200"))

from inla_b200 import BatchSolver, GpuSolver, _lib, models  # noqa: E402
from inla_b200.autograd import log_posterior  # noqa: E402
from inla_b200.laplace import LaplaceModel  # noqa: E402
from inla_b200.mesh import Mesh, SpdePlan  # noqa: E402
from inla_b200.multi import MultiModel  # noqa: E402

KAPPA = 3.059023205018258e6  # weight of the hard constraints in the working prior


def listed():
    return [
        # the InlaSolver seam of a host program on a small mesh: latency and host path only
        {"name": "seam-30", "kind": "seam", "nx": 30},
        # the same seam on an ordinary mesh (n = 10 000)
        {"name": "seam-100", "kind": "seam", "nx": 100},
        # one theta-point at a time on the headline mesh (a Nelder-Mead search): n = 40 000, B = 1
        {"name": "batch-200-b1", "kind": "batch", "nx": 200, "B": 1},
        # the batch of one Newton iteration of the headline fit: 7 stencil points + 3 priors
        {"name": "batch-200-b10", "kind": "batch", "nx": 200, "B": 10},
        # value and gradient of log pi(theta | y) through autograd, the stencil of one Newton step
        {"name": "grad-200-b7", "kind": "grad", "nx": 200, "B": 7},
        # the CCD stage of the headline fit: 15 nodes with every marginal variance
        {"name": "ccd-200-b15", "kind": "ccd", "nx": 200, "B": 15},
        # non-Gaussian SPDE (negative-binomial counts) on a larger mesh (n = 90 000), gradient stencil
        {"name": "nb-300-b5", "kind": "nb", "nx": 300, "B": 5},
        # Besag GLMM on the 30 x 30 lattice, sum-to-zero, Poisson: small dense-ish constrained model
        {"name": "besag-30-b3", "kind": "besag", "nr": 30, "nc": 30, "B": 3},
        # Besag x AR1 + iid + intercept, binomial, one constraint per time (bordered), gradient
        {"name": "group-24x24x14-b2", "kind": "group", "nr": 24, "nc": 24, "T": 14, "B": 2},
        # uneven independent AR1 + iid Poisson models in lockstep (200 to 5000 observations each)
        {"name": "multi-96-b2", "kind": "multi", "G": 96, "B": 2},
        # a whole fit: Newton mode search, FD Hessian, CCD, mixture moments
        {"name": "fit-45", "kind": "fit", "nx": 45},
        # setting an SPDE model up on the device: FEM blocks, components, projector (odd mesh)
        {"name": "mesh-301", "kind": "mesh", "nx": 301, "npts": 50000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["seam", "seam", "batch", "batch", "grad", "ccd", "nb", "besag", "group", "multi", "fit", "mesh"])
    if kind == "seam":
        return {"kind": kind, "nx": _log_int(rng, 25, 150)}
    if kind == "batch":
        nx = _log_int(rng, 40, 200)
        return {"kind": kind, "nx": nx, "B": _log_int(rng, 1, 21 if nx <= 150 else 12)}
    if kind == "grad":
        return {"kind": kind, "nx": _log_int(rng, 40, 200), "B": rng.choice([1, 4, 7])}
    if kind == "ccd":
        return {"kind": kind, "nx": _log_int(rng, 40, 200), "B": rng.choice([9, 15])}
    if kind == "nb":
        return {"kind": kind, "nx": _log_int(rng, 50, 250), "B": rng.choice([1, 3, 5])}
    if kind == "besag":
        return {"kind": kind, "nr": rng.randint(12, 36), "nc": rng.randint(12, 36), "B": rng.choice([1, 2, 3, 5])}
    if kind == "group":
        return {"kind": kind, "nr": rng.randint(24, 30), "nc": rng.randint(24, 30), "T": rng.randint(13, 18),
                "B": rng.choice([1, 2])}
    if kind == "multi":
        return {"kind": kind, "G": _log_int(rng, 8, 110), "B": rng.choice([1, 2])}
    if kind == "fit":
        return {"kind": kind, "nx": _log_int(rng, 20, 60)}
    return {"kind": kind, "nx": _log_int(rng, 60, 300), "npts": _log_int(rng, 1000, 50000)}


# ---------------------------------------------------------------------------
# inputs (host arrays from the seed alone)
# ---------------------------------------------------------------------------

def _field(rng, pts, corr_range=0.2):
    """A smooth random field of unit variance at ``pts``: 96 random Fourier features."""
    w = rng.standard_normal((2, 96)) * (2.0 / corr_range)
    return np.cos(pts @ w + rng.uniform(0.0, 2.0 * math.pi, 96)) @ (rng.standard_normal(96) * math.sqrt(2.0 / 96))


def _spde(nx, n_obs, seed, family="gaussian"):
    """SPDE model on a jittered nx x nx mesh with n_obs observations of a smooth field."""
    rng = np.random.default_rng([seed, nx])
    verts, tris = models.grid_mesh(nx, rng)
    c0, g = models.fem_matrices(verts, tris)
    pts = rng.uniform(0.0, 1.0, size=(n_obs, 2))
    a = models.grid_projector(verts, tris, nx, pts)
    f = _field(rng, pts)
    if family == "nbinomial":
        mu = np.exp(f)
        y = rng.negative_binomial(5.0, 5.0 / (5.0 + mu)).astype(float)
    else:
        y = f + 0.1 * rng.standard_normal(n_obs)
    model = models.build_latent(len(verts), models.spde_components(c0, g), "spde", extra_pattern=[(a.T @ a).tocsc()])
    return model, a, y, rng


LOG_KAPPA = math.log(math.sqrt(8.0) / 0.2)
LOG_TAU = -math.log(2.0 * math.sqrt(math.pi)) - LOG_KAPPA


def _spde_thetas(rng, B, h=1e-3):
    """B points [log prec, log tau, log kappa] near the generating values: the centre and its
    central-difference points in batches of up to 7, a spread design beyond that."""
    c = np.array([math.log(100.0), LOG_TAU, LOG_KAPPA]) + 0.1 * rng.standard_normal(3)
    if B > 7:
        return c + 0.15 * rng.standard_normal((B, 3))
    th = np.tile(c, (B, 1))
    for b in range(1, B):
        th[b, (b - 1) // 2] += h if b % 2 else -h
    return th


def _posterior_matrix(model, a, theta):
    """Q(theta) + prec A'A on the model's pattern."""
    q = (model.matrix(models.spde_coefs(theta[1], theta[2])[0]) + math.exp(theta[0]) * (a.T @ a)).tocsc()
    q.sort_indices()
    return q


def _inputs(case, seed):
    """Host inputs of a case: a dict of arrays, sparse matrices and models."""
    kind = case["kind"]
    if kind in ("seam", "batch"):
        B = case.get("B", 1)
        model, a, y, rng = _spde(case["nx"], case["nx"] ** 2 // 2, seed)
        q = [_posterior_matrix(model, a, t) for t in _spde_thetas(rng, B)]
        return {"q": q, "rhs": rng.standard_normal((B, model.n))}
    if kind in ("grad", "ccd"):
        model, a, y, rng = _spde(case["nx"], case["nx"] ** 2 // 2, seed)
        th = _spde_thetas(rng, case["B"])
        return {"model": model, "a": a, "y": y, "theta": th, "family": "gaussian", "p1": None, "c": None,
                "coefs": np.stack([models.spde_coefs(t[1], t[2])[0] for t in th]), "p1scale": np.exp(th[:, 0])}
    if kind == "nb":
        model, a, y, rng = _spde(case["nx"], case["nx"] ** 2 // 4, seed, "nbinomial")
        th = _spde_thetas(rng, case["B"])
        th[:, 1:] = np.array([LOG_TAU, LOG_KAPPA]) + 0.1 * rng.standard_normal(2)
        for b in range(1, case["B"]):
            th[b, 1 + (b - 1) // 2] += 1e-3 if b % 2 else -1e-3
        return {"model": model, "a": a, "y": y, "family": "nbinomial", "p1": 5.0, "c": None, "p1scale": None,
                "coefs": np.stack([models.spde_coefs(t[1], t[2])[0] for t in th])}
    if kind == "besag":
        p = models.make_besag_problem(case["nr"], case["nc"], seed=seed)
        rng = np.random.default_rng([seed, 1])
        lt = math.log(2.0) + 0.2 * rng.standard_normal() + np.array([0.0, 1e-3, -1e-3, 0.3, -0.3])[:case["B"]]
        return {"model": p.model, "a": p.a, "y": p.y, "family": "poisson", "p1": 1.0, "c": p.constraint, "p1scale": None,
                "coefs": np.stack([models.besag_coefs(t)[0] for t in lt])}
    if kind == "group":
        p = models.make_group_problem(case["nr"], case["nc"], case["T"], seed=seed)
        rng = np.random.default_rng([seed, 1])
        th = np.array([0.0, 0.0, 2.2, 1.4]) + 0.1 * rng.standard_normal(4)
        th = np.tile(th, (case["B"], 1))
        th[1:, 2] += 1e-3
        return {"model": p.model, "a": p.a, "y": p.y, "family": "binomial", "p1": p.ntrials, "c": p.constraint,
                "p1scale": None, "coefs": np.stack([models.group_coefs(t)[0] for t in th])}
    if kind == "multi":
        rng = np.random.default_rng([seed, case["G"]])
        ms, As, ys = [], [], []
        for g in range(case["G"]):  # sizes log-uniform over [200, 5000), fixed by G; paths and counts by the seed
            nk = int(200.0 * 25.0 ** ((g * 0.6180339887498949) % 1.0))
            model, a = models.ar1_iid_model(nk)
            e = rng.standard_normal(nk)
            rho = rng.uniform(0.3, 0.95)
            f = np.convolve(e, rho ** np.arange(200.0))[:nk]
            ms.append(model)
            As.append(a)
            ys.append(rng.poisson(np.exp(0.5 + f * rng.lognormal(-0.25, 0.25) + rng.standard_normal(nk) / math.sqrt(10.0))).astype(float))
        th = np.array([0.0, 1.3, 2.3]) + 0.2 * rng.standard_normal((1, case["G"], 3))
        th = np.tile(th, (case["B"], 1, 1))
        th[1:, :, 0] += 1e-3
        return {"models": ms, "a": As, "y": ys,
                "coefs": np.stack([[models.ar1_iid_coefs(t)[0] for t in row] for row in th])}
    if kind == "fit":
        model, a, y, rng = _spde(case["nx"], case["nx"] ** 2 // 2, seed)
        return {"model": model, "a": a, "y": y}
    rng = np.random.default_rng([seed, 7])
    verts, tris = models.grid_mesh(case["nx"], rng)
    return {"verts": verts, "tris": tris, "pts": rng.uniform(0.0, 1.0, size=(case["npts"], 2))}


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

def prepare(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "seam":
        s["solver"] = GpuSolver()
        s["solver"].analyze(x["q"][0])
        s["q"], s["rhs"] = x["q"][0], x["rhs"][0]
    elif kind == "batch":
        B = case["B"]
        s["solver"] = BatchSolver(x["q"][0], max_batch=B)
        s["vals"] = torch.tensor(np.stack([q.data for q in x["q"]]), device="cuda")
        s["rhs"] = torch.tensor(x["rhs"], device="cuda")
        s["logdet"] = torch.zeros(B, dtype=torch.float64, device="cuda")
        s["status"] = torch.zeros(B, dtype=torch.int32, device="cuda")
        s["x"] = torch.empty_like(s["rhs"])
        s["diag"] = torch.empty_like(s["rhs"])
    elif kind in ("grad", "ccd", "nb", "besag", "group"):
        m = LaplaceModel(x["model"], a=x["a"], family=x["family"], y=x["y"], p1=x["p1"], max_batch=case["B"])
        if x["c"] is not None:
            m.set_constraints(*x["c"])
        s["model"], s["coefs"], s["p1scale"] = m, x["coefs"], x["p1scale"]
        if kind == "grad":
            s["theta"] = torch.tensor(x["theta"])
    elif kind == "multi":
        s["model"] = MultiModel(x["models"], x["a"], x["y"], max_batch=case["B"])
        s["coefs"] = x["coefs"]
    elif kind == "fit":
        s["model"] = LaplaceModel(x["model"], a=x["a"], family="gaussian", y=x["y"], max_batch=15)
    else:
        m = Mesh(x["verts"], x["tris"])
        s["mesh"] = m
        s["plan"] = SpdePlan(m.nv, *m.fem_pattern("g1"))
        s["pts"] = torch.tensor(x["pts"], device="cuda")
    return s


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    kind = state["case"]["kind"]
    if kind == "seam":
        sv = state["solver"]
        sv.factorize(state["q"])
        return {"logdet": sv.log_abs_det(), "x": sv.solve(state["rhs"]), "diag": sv.diag_inv()}
    if kind == "batch":
        B, h = state["case"]["B"], state["solver"]._h
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        lib = _lib.lib()
        state["x"].copy_(state["rhs"])
        _lib.check(lib.inla_batch_factorize_dev(h, B, _ptr(state["vals"]), _ptr(state["logdet"]), _ptr(state["status"]),
                                                stream))
        _lib.check(lib.inla_batch_solve_dev(h, B, _ptr(state["x"]), stream))
        _lib.check(lib.inla_batch_diag_inv_dev(h, B, _ptr(state["diag"]), stream))
        return {k: state[k] for k in ("logdet", "status", "x", "diag")}
    if kind == "grad":
        theta = state["theta"].clone().requires_grad_(True)
        value = log_posterior(theta, state["model"])
        value.sum().backward()
        return {"value": value.detach(), "grad": theta.grad}
    if kind == "ccd":
        r = state["model"].eval(state["coefs"], state["p1scale"], variances=True)
        del r["dll"]  # d loglik / d log precision: written with the gradient only
        return r
    if kind in ("nb", "besag", "group", "multi"):
        r = state["model"].eval(state["coefs"], variances=True, gradient=True)
        # written for the Gaussian family only: d loglik / d log precision; z' M x has the components'
        # columns and no observation term
        del r["dll"]
        r["zMx"] = r["zMx"][..., :-1]
        return r
    if kind == "fit":
        r = state["model"].fit(np.zeros(3), mode_search="newton", batched=True)
        return {k: r[k] for k in ("mode", "mean", "var", "mlik", "node_theta", "node_weight", "pred_mean", "pred_var")}
    out = state["mesh"].fem_device()
    out["comp"] = state["plan"].components(out["c0"], out["g1"])
    out["rowptr"], out["colidx"], out["weights"] = state["mesh"].projector_device(state["pts"])
    return out


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------

def _sparse_cost(pattern):
    """(nnz(L), LDL' operations, selected-inverse operations) of a pattern under nested dissection."""
    s = GpuSolver(ordering=_lib.ORDER_ND)
    s.analyze(pattern)
    c = s.colcounts().astype(float) - 1.0  # below the diagonal
    return float(np.sum(c + 1.0)), float(np.sum(c * c + 2.0 * c)), float(np.sum(2.0 * c * c + 2.0 * c))


def work(case):
    """One factorization, solve and selected inverse per problem at the least (one more of each for
    the prior of a Laplace gradient, four Newton factorizations for a non-Gaussian family, 80
    evaluations for a fit); every input and the outputs once."""
    x = _inputs(case, 0)
    kind, B = case["kind"], case.get("B", 1)
    if kind == "mesh":
        nv, nt = len(x["verts"]), len(x["tris"])
        values = nv + 3 * 7 * nv + 3 * 19 * nv  # c0; c1, g1, b1 at most; components
        return {"bytes": 8.0 * (2 * nv + 3 * nt + values + 2 * case["npts"] + 7 * case["npts"]), "flops": 60.0 * nt}
    if kind in ("seam", "batch"):
        n, nnz = x["q"][0].shape[0], x["q"][0].nnz
        nl, f, t = _sparse_cost(x["q"][0])
        return {"bytes": 8.0 * B * (nnz + 3 * n), "flops": B * (f + t + 4.0 * nl)}
    if kind == "multi":
        n = nobs = nnz = nl = f = t = 0.0
        for m, y in zip(x["models"], x["y"]):
            a, b, c = _sparse_cost(m.pattern)
            nl, f, t = nl + a, f + b, t + c
            n, nobs, nnz = n + m.n, nobs + len(y), nnz + m.pattern.nnz
        T = 5
    else:
        m = x["model"]
        nl, f, t = _sparse_cost(m.pattern)
        n, nobs, nnz, T = m.n, len(x["y"]), m.pattern.nnz, m.n_comp
    inputs, outputs = 8.0 * (T * nnz + 6 * nobs), 16.0 * B * n
    if kind == "fit":
        return {"bytes": inputs + 16.0 * n, "flops": 80.0 * (2.0 * f + 4.0 * nl) + 15.0 * t}
    if kind == "grad":
        return {"bytes": inputs, "flops": B * (f + t + 4.0 * nl) + min(B, 5) * (f + t)}
    if kind == "ccd":
        return {"bytes": inputs + outputs, "flops": B * (2.0 * f + t + 4.0 * nl)}
    return {"bytes": inputs + outputs, "flops": B * (5.0 * f + 2.0 * t + 20.0 * nl)}


# ---------------------------------------------------------------------------
# the outputs by dense 64-bit algebra
# ---------------------------------------------------------------------------

def _dense(q):
    q = q.tocoo()
    d = torch.zeros(q.shape, dtype=torch.float64, device="cuda")
    d.index_put_((torch.tensor(q.row, device="cuda").long(), torch.tensor(q.col, device="cuda").long()),
                 torch.tensor(q.data, device="cuda"), accumulate=True)
    return d


def _logdet(ch):
    return float(2.0 * torch.log(torch.diagonal(ch)).sum())


def _solve(ch, b):
    return torch.cholesky_solve(b[:, None], ch)[:, 0]


def _likelihood(family, eta, y, p1):
    """(log p, d/d eta, weight, d weight / d eta) per observation."""
    if family == "gaussian":
        r = y - eta
        return 0.5 * math.log(p1 / (2.0 * math.pi)) - 0.5 * p1 * r * r, p1 * r, torch.full_like(eta, p1), torch.zeros_like(eta)
    if family == "poisson":
        mu = p1 * torch.exp(eta)
        return y * torch.log(mu) - mu - torch.lgamma(y + 1.0), y - mu, mu, mu
    if family == "binomial":
        p = torch.sigmoid(eta)
        n = torch.full_like(y, p1)
        lc = torch.lgamma(n + 1.0) - torch.lgamma(y + 1.0) - torch.lgamma(n - y + 1.0)
        w = n * p * (1.0 - p)
        return lc + y * torch.nn.functional.logsigmoid(eta) + (n - y) * torch.nn.functional.logsigmoid(-eta), y - n * p, w, w * (1.0 - 2.0 * p)
    r, mu = p1, torch.exp(eta)
    lp = (torch.lgamma(y + r) - math.lgamma(r) - torch.lgamma(y + 1.0) + r * torch.log(r / (mu + r)) + y * torch.log(mu / (mu + r)))
    w = (y + r) * r * mu / (mu + r) ** 2
    return lp, y - (y + r) * mu / (mu + r), w, w * (r - mu) / (mu + r)


def _laplace(model, a, y, family, p1, coefs, c=None):
    """One Laplace evaluation with its trace pieces, dense."""
    n = model.n
    pat = model.pattern.tocoo()
    ri, ci = torch.tensor(pat.row, device="cuda").long(), torch.tensor(pat.col, device="cuda").long()
    comp = torch.tensor(model.comp_values, device="cuda")
    A, y = _dense(a), torch.tensor(y, device="cuda")
    q = _dense(model.matrix(coefs))
    cons = None
    if c is not None:
        cm, e = torch.tensor(np.atleast_2d(c[0]), device="cuda"), torch.tensor(np.atleast_1d(c[1]), device="cuda")
        q += KAPPA * (cm.T @ cm)
        cons = (cm, e, torch.linalg.inv(cm @ cm.T))
    else:
        q.diagonal().add_(1e-12)
    ch = torch.linalg.cholesky(q)
    ld_prior = _logdet(ch)
    inv = torch.cholesky_inverse(ch)
    trP = (comp * inv[ri, ci]).sum(1)
    del ch, inv
    if c is None:
        q.diagonal().sub_(1e-12)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    for _ in range(60):
        lp, g, w, dw = _likelihood(family, A @ x, y, p1)
        chp = torch.linalg.cholesky(q + A.T @ (w[:, None] * A))
        rhs = A.T @ g - q @ x
        step = _solve(chp, rhs)
        biggest = float(step.abs().max())
        x = x + step * min(1.0, 10.0 / max(biggest, 1e-300))
        if cons:
            x = x - cons[0].T @ (cons[2] @ (cons[0] @ x - cons[1]))
        if family == "gaussian" or biggest < 1e-11:
            break
    eta = A @ x
    lp, g, w, dw = _likelihood(family, eta, y, p1)
    chp = torch.linalg.cholesky(q + A.T @ (w[:, None] * A))
    inv = torch.cholesky_inverse(chp)
    ld_post, loglik = _logdet(chp), float(lp.sum())
    M = comp * x[ri] * x[ci]
    quad = float(x @ (q @ x))
    v = ((A @ inv) * A).sum(1)
    z = _solve(chp, A.T @ (dw * v))
    T1 = len(comp) + 1
    tr = {k: np.zeros(T1) for k in ("trP", "trQ", "xMx", "zMx")}
    tr["trP"][:-1] = trP.cpu().numpy()
    tr["trQ"][:-1] = (comp * inv[ri, ci]).sum(1).cpu().numpy()
    tr["trQ"][-1] = float((w * v).sum())
    tr["xMx"][:-1] = M.sum(1).cpu().numpy()
    if family != "gaussian":
        tr["zMx"][:-1] = (comp * z[ri] * x[ci]).sum(1).cpu().numpy()
    dll = float((0.5 - 0.5 * p1 * (y - eta) ** 2).sum()) if family == "gaussian" else 0.0
    return {"mlik": loglik - 0.5 * quad + 0.5 * ld_prior - 0.5 * ld_post, "logdet_prior": ld_prior, "logdet_post": ld_post,
            "loglik": loglik, "quad": quad, "dll": dll, "x": x.cpu().numpy(), "var": torch.diagonal(inv).cpu().numpy(), **tr}


def _spde_log_prior(t):
    """The default hyperpriors of an SPDE model and their gradient: log-gamma(1, 5e-5) on the log
    noise precision, the PC prior P(range < 1) = 0.05, P(sd > 1) = 0.01 on (log tau, log kappa)."""
    lam1, lam2 = -math.log(0.05), -math.log(0.01)
    log_rho, log_sd = 0.5 * math.log(8.0) - t[2], -0.5 * math.log(4.0 * math.pi) - t[1] - t[2]
    er, es = math.exp(-log_rho), math.exp(log_sd)
    value = math.log(5e-5) + t[0] - 5e-5 * math.exp(t[0])
    value += math.log(lam1) - log_rho - lam1 * er + math.log(lam2) + log_sd - lam2 * es
    d_rho, d_sd = lam1 * er - 1.0, 1.0 - lam2 * es
    return value, np.array([1.0 - 5e-5 * math.exp(t[0]), -d_sd, -d_rho - d_sd])


def _value_and_gradient(r, theta, coefs):
    """log pi(theta | y) and its gradient from one dense evaluation of the Gaussian SPDE model."""
    dc = np.zeros((3, 3))
    dc[1] = 2.0 * coefs
    dc[2] = [4.0 * coefs[0], 2.0 * coefs[1], 0.0]
    lp, g = _spde_log_prior(theta)
    g = g + dc @ (0.5 * (r["trP"] - r["trQ"] - r["xMx"])[:3])
    g[0] += r["dll"] - 0.5 * r["trQ"][3]
    return r["mlik"] + lp, g


#: Dense operations exact() may spend (about 15 s at the dense rate of this GPU).
DENSE_LIMIT = 1.2e14


def exact(case, seed):
    kind = case["kind"]
    if kind == "fit":
        return None  # a mode search has no closed form (its evaluations are the grad and ccd cases)
    if kind == "mesh":
        return _exact_mesh(case, seed)
    n = case.get("nx", 0) ** 2 or {"besag": case.get("nr", 0) * case.get("nc", 0),
         "group": 2 * case.get("nr", 0) * case.get("nc", 0) * case.get("T", 0) + 1,
                                  "multi": 3000}[kind]
    per = {"seam": 1.4, "batch": 1.4, "grad": 4.0, "ccd": 4.0, "nb": 15.0, "besag": 15.0, "group": 8.0, "multi": 45.0}[kind]
    if case.get("B", 1) * case.get("G", 1) * per * float(n) ** 3 > DENSE_LIMIT or n > 45000:
        return None
    x = _inputs(case, seed)
    if kind in ("seam", "batch"):
        out = {"logdet": [], "x": [], "diag": []}
        for q, b in zip(x["q"], x["rhs"]):
            ch = torch.linalg.cholesky(_dense(q))
            out["logdet"].append(_logdet(ch))
            out["x"].append(_solve(ch, torch.tensor(b, device="cuda")).cpu().numpy())
            out["diag"].append(torch.diagonal(torch.cholesky_inverse(ch)).cpu().numpy())
            del ch
        if kind == "seam":
            return {k: v[0] for k, v in out.items()}
        return {**{k: np.array(v) for k, v in out.items()}, "status": None}
    if kind == "multi":
        rows = [[_laplace(m, a, y, "poisson", 1.0, c) for m, a, y, c in zip(x["models"], x["a"], x["y"], row)]
                for row in x["coefs"]]
        out = {k: np.array([[r[k] for r in row] for row in rows]) for k in rows[0][0] if k not in ("x", "var")}
        out.update({k: np.stack([np.concatenate([r[k] for r in row]) for row in rows]) for k in ("x", "var")})
    else:
        s = x["p1scale"] if x["p1scale"] is not None else [x["p1"]] * case["B"]
        rows = [_laplace(x["model"], x["a"], x["y"], x["family"], float(p), c, x["c"]) for p, c in zip(s, x["coefs"])]
        out = {k: np.array([r[k] for r in rows]) for k in rows[0]}
        if kind == "grad":
            vg = [_value_and_gradient(r, t, c) for r, t, c in zip(rows, x["theta"], x["coefs"])]
            return {"value": np.array([v for v, _ in vg]), "grad": np.stack([g for _, g in vg])}
        if kind == "ccd":
            out = {k: v for k, v in out.items() if k not in ("trP", "trQ", "xMx", "zMx", "dll")}
    if kind in ("nb", "besag", "group", "multi"):
        del out["dll"]
        out["zMx"] = out["zMx"][..., :-1]
    return {**out, "iters": None, "status": None}


def _exact_mesh(case, seed):
    """Areas, masses and stiffness of linear elements by numpy on the vertices' coordinates."""
    x = _inputs(case, seed)
    v, t = x["verts"], x["tris"]
    n = len(v)
    p = [v[t[:, i]] for i in range(3)]
    e = [p[2] - p[1], p[0] - p[2], p[1] - p[0]]
    area = 0.5 * np.abs(e[0][:, 0] * e[1][:, 1] - e[0][:, 1] * e[1][:, 0])
    keys, mass, stiff = [], [], []
    for i in range(3):
        for j in range(3):
            keys.append(t[:, j] * n + t[:, i])
            mass.append(area / (6.0 if i == j else 12.0))
            stiff.append((e[i] * e[j]).sum(1) / (4.0 * area))
    uniq, inv = np.unique(np.concatenate(keys), return_inverse=True)
    c0 = np.bincount(t.ravel(), weights=np.repeat(area / 3.0, 3), minlength=n)
    return {"areas": area, "c0": c0, "c1": np.bincount(inv, weights=np.concatenate(mass)),
            "g1": np.bincount(inv, weights=np.concatenate(stiff)), "b1": None, "comp": None, "rowptr": None,
            "colidx": None, "weights": None}
