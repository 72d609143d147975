"""The calls whose speed is followed from change to change: exact and sparse
GP objectives, predictions, online updates, batches and new models, through
the package's public entry points, over the sizes users run them at.

A case is a dict of plain values; `kind` says which call it stands for:

  eval     FittedGpr.value_and_gradient: one step of a hyperparameter search
  hessian  FittedGpr.value_gradient_hessian: one step of a trust-region search
  predict  FittedGpr.predict on a resident model: a serving request
  online   OnlineGpr sliding window: predict the next points, insert one, drop the oldest
  model    Gpr.factor on host data, then a prediction: a new model from scratch
  batch    GprBatch.value_and_gradient: one round over many ragged problems
  sgpr     FittedSgpr.value_and_gradient: one step of a sparse (VFE) search

Points are column-major (x[i + f·n]); every input is made from the seed.
"""

import math

import numpy as np
import torch

import gprx_b200 as gx

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
LISTED = [
    # the smallest search step: a few dozen points, where launches and latency are all there is
    {"name": "eval_n64", "kind": "eval", "tree": "rbf", "n": 64, "d": 1, "precision": "fp64"},
    # the benchmark's small exact fit: RBF, n = 512, d = 2
    {"name": "eval_n512", "kind": "eval", "tree": "rbf", "n": 512, "d": 2, "precision": "fp64"},
    # an ordinary data set of a ragged size, ARD lengthscales
    {"name": "eval_n1537", "kind": "eval", "tree": "const_ard", "n": 1537, "d": 8, "precision": "fp64"},
    # the benchmark's large exact objective: Constant · RbfArd, n = 8192, d = 8, plain FP64 ...
    {"name": "eval_n8192", "kind": "eval", "tree": "const_ard", "n": 8192, "d": 8, "precision": "fp64"},
    # ... and with the mixed-precision option
    {"name": "eval_n8192_mixed", "kind": "eval", "tree": "const_ard", "n": 8192, "d": 8, "precision": "mixed"},
    # value, gradient and Hessian of an ordinary model
    {"name": "hessian_n2048", "kind": "hessian", "tree": "const_ard", "n": 2048, "d": 8, "precision": "fp64"},
    # one query point against a resident model: the latency of a serving request
    {"name": "predict_n1000_q1", "kind": "predict", "tree": "rbf_ard", "n": 1000, "d": 4, "q": 1},
    # the largest serving request: 10 000 points against a 4096-point model
    {"name": "predict_n4096_q10000", "kind": "predict", "tree": "rbf_ard", "n": 4096, "d": 4, "q": 10000},
    # a stream: a window of 2000 points that moves on by one
    {"name": "online_n2000", "kind": "online", "tree": "rbf_ard", "n": 2000, "d": 4, "q": 4},
    # a new model from host data: creation, factor and a first prediction
    {"name": "model_n1024_q256", "kind": "model", "tree": "rbf_ard", "n": 1024, "d": 4, "q": 256},
    # thousands of ragged problems in one round, RBF + periodic, d = 3
    {"name": "batch_4096", "kind": "batch", "tree": "rbf_periodic", "count": 4096, "n_lo": 32, "n_hi": 1024, "d": 3},
    # the benchmark's sparse objective: a million points, 1024 inducing inputs
    {"name": "sgpr_n1e6_m1024", "kind": "sgpr", "tree": "rbf_ard", "n": 1000000, "m": 1024, "d": 4,
     "precision": "fp64"},
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["eval", "eval", "eval", "hessian", "predict", "predict", "online", "model", "batch", "sgpr"])
    if kind == "eval":
        if rng.random() < 0.25:  # the mixed form's own range
            return {"kind": kind, "tree": "const_ard", "n": _log_int(rng, 1024, 8192), "d": 8, "precision": "mixed"}
        tree = rng.choice(["rbf", "rbf_ard", "const_ard", "rbf_periodic"])
        return {"kind": kind, "tree": tree, "n": _log_int(rng, 16, 8192),
                "d": rng.choice([1, 2, 3, 4, 8]) if tree != "rbf_periodic" else 1, "precision": "fp64"}
    if kind == "hessian":
        return {"kind": kind, "tree": rng.choice(["rbf_ard", "const_ard"]), "n": _log_int(rng, 64, 3000),
                "d": rng.choice([2, 4, 8]), "precision": "fp64"}
    if kind == "predict":
        return {"kind": kind, "tree": rng.choice(["rbf", "rbf_ard", "const_ard"]), "n": _log_int(rng, 64, 4096),
                "d": rng.choice([2, 4, 8]), "q": _log_int(rng, 1, 10000)}
    if kind == "online":
        return {"kind": kind, "tree": rng.choice(["rbf", "rbf_ard"]), "n": _log_int(rng, 64, 4096),
                "d": rng.choice([2, 4]), "q": rng.randint(1, 16)}
    if kind == "model":
        return {"kind": kind, "tree": rng.choice(["rbf", "rbf_ard", "const_ard"]), "n": _log_int(rng, 64, 4096),
                "d": rng.choice([2, 4, 8]), "q": _log_int(rng, 1, 2000)}
    if kind == "batch":
        lo = _log_int(rng, 16, 128)
        return {"kind": kind, "tree": rng.choice(["rbf_periodic", "rbf", "rbf_ard"]),
                "count": _log_int(rng, 16, 2048), "n_lo": lo, "n_hi": _log_int(rng, 2 * lo, 1024), "d": 3}
    return {"kind": "sgpr", "tree": "rbf_ard", "n": _log_int(rng, 2000, 250000), "m": _log_int(rng, 64, 1024),
            "d": rng.choice([3, 4]), "precision": "fp64"}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _noise(case):
    return 0.1 if case["kind"] in ("batch", "sgpr") else 0.05


def _theta(case, rs):
    """log θ of the tree (depth first), then log σn²."""
    d, tree = case["d"], case["tree"]
    if tree == "rbf":
        th = [math.log(0.9)]
    elif tree == "rbf_ard":
        th = list(rs.uniform(math.log(0.5), math.log(2.0), size=d))
    elif tree == "const_ard":
        th = [math.log(2.0)] + list(rs.uniform(math.log(0.3), math.log(3.0), size=d))
    else:  # RBF + periodic
        th = [0.0, 0.0, math.log(rs.uniform(10.0, 20.0) if case["kind"] == "batch" else 2.0)]
    return np.array(th + [math.log(_noise(case))])


def _kernel(case, theta):
    v = [math.exp(t) for t in theta[:-1]]
    if case["tree"] == "rbf":
        return gx.RbfKernel(v[0])
    if case["tree"] == "rbf_ard":
        return gx.RbfArdKernel(v)
    if case["tree"] == "const_ard":
        return gx.ConstantKernel(v[0]) * gx.RbfArdKernel(v[1:])
    return gx.RbfKernel(v[0]) + gx.PeriodicKernel(v[1], v[2])


def _points(case, rs, n):
    d = case["d"]
    if case["kind"] == "batch":
        return rs.uniform(0.0, 5.0, size=n * d)
    if case["tree"] in ("rbf", "rbf_periodic"):
        return rs.uniform(0.0, 10.0, size=n * d)
    return rs.standard_normal(n * d)


def _targets(rs, x, n, d):
    y = np.sin(x[:n])
    if d > 1:
        y = y + 0.5 * np.cos(x[n:2 * n])
    return y + 0.1 * rs.standard_normal(n)


def _exact_data(case, seed):
    rs = np.random.RandomState(seed % (1 << 31))
    theta = _theta(case, rs)
    n = case["n"]
    x = _points(case, rs, n)
    y = _targets(rs, x, n, case["d"])
    out = {"theta": theta, "x": x, "y": y, "at": theta + 0.1 * rs.standard_normal(theta.size)}
    if "q" in case:
        out["xs"] = _points(case, rs, case["q"])
    if case["kind"] == "online":
        out["pool_x"] = _points(case, rs, POOL).reshape(case["d"], POOL).T.copy()
        out["pool_y"] = np.sin(out["pool_x"][:, 0]) + 0.1 * rs.standard_normal(POOL)
    return out


POOL = 8192  # points that a stream brings before it starts over


def _batch_data(case, seed):
    rs = np.random.RandomState(seed % (1 << 31))
    u = rs.uniform(size=case["count"])
    sizes = np.floor(np.exp(math.log(case["n_lo"]) + u * math.log(case["n_hi"] / case["n_lo"]))).astype(int)
    xs, ys, params = [], [], []
    for n in sizes:
        params.append(_theta(case, rs))
        xs.append(_points(case, rs, int(n)))
        ys.append(_targets(rs, xs[-1], int(n), case["d"]))
    return {"xs": xs, "ys": ys, "params": np.stack(params)}


def _sgpr_data(case, seed):
    """Inducing inputs on a jittered grid 1.6 lengthscales apart, points
    uniform over the grid's box."""
    rs = np.random.RandomState(seed % (1 << 31))
    theta = _theta(case, rs)
    n, m, d = case["n"], case["m"], case["d"]
    ls = np.exp(theta[:d])
    k = int(math.ceil(m ** (1.0 / d) - 1e-9))
    at = np.indices((k,) * d).reshape(d, -1)[:, :m].T
    z = (at + 0.05 * rs.uniform(-1, 1, size=(m, d))) * (1.6 * ls)
    hi = z.max(axis=0) + 0.5 * ls
    x = np.stack([h * rs.uniform(size=n) for h in hi])  # d × n: column-major n × d
    y = np.sin(6.0 * x[0] / hi[0]) + np.cos(4.0 * x[1] / hi[1]) + 0.1 * rs.standard_normal(n)
    return {"theta": theta, "x": x.reshape(-1), "y": y, "z": z.T.reshape(-1).copy(),
            "at": theta + 0.05 * rs.standard_normal(theta.size)}


def _trainer(case, theta):
    precision = gx.Precision.Mixed if case.get("precision") == "mixed" else gx.Precision.Fp64
    cls = gx.Sgpr if case["kind"] == "sgpr" else gx.Gpr
    return cls(_kernel(case, theta), gx.GaussianLikelihood(math.exp(theta[-1])),
               precision=precision).with_optimizer(gx.Fixed())


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind, d = case["kind"], case["d"]
    if kind == "batch":
        data = _batch_data(case, seed)
        k = _kernel(case, data["params"][0])
        return {"case": case, "model": gx.GprBatch(k, data["xs"], data["ys"], d), "params": data["params"]}
    if kind == "sgpr":
        data = _sgpr_data(case, seed)
        m = _trainer(case, data["theta"]).factor(data["x"], case["n"], d, data["y"], data["z"], case["m"])
        return {"case": case, "model": m, "at": data["at"]}
    data = _exact_data(case, seed)
    s = {"case": case, "at": data["at"], "xs": data.get("xs")}
    if kind == "model":
        return dict(s, trainer=_trainer(case, data["theta"]), x=data["x"], y=data["y"])
    m = _trainer(case, data["theta"]).factor(data["x"], case["n"], d, data["y"])
    if kind == "online":
        m = m.into_online()
        s.update(pool_x=data["pool_x"], pool_y=data["pool_y"], next=0, ids=[int(i) for i in m.point_ids()])
    return dict(s, model=m)


def run(state):
    case = state["case"]
    kind, d = case["kind"], case["d"]
    if kind == "batch":
        nlml, grad, status = state["model"].value_and_gradient(state["params"])
        return {"nlml": nlml, "grad": grad, "status": status}
    if kind in ("eval", "sgpr"):
        nlml, grad = state["model"].value_and_gradient(state["at"])
        return {"nlml": nlml, "grad": grad}
    if kind == "hessian":
        nlml, grad, hess = state["model"].value_gradient_hessian(state["at"])
        return {"nlml": nlml, "grad": grad, "hess": hess}
    if kind == "predict":
        p = state["model"].predict(state["xs"], case["q"], d)
        return {"mean": p.mean, "variance": p.variance}
    if kind == "model":
        m = state["trainer"].factor(state["x"], case["n"], d, state["y"])
        p = m.predict(state["xs"], case["q"], d)
        return {"mean": p.mean, "variance": p.variance}
    m, k = state["model"], state["next"] % POOL
    p = m.predict(state["xs"], case["q"], d)
    state["ids"].append(m.insert(state["pool_x"][k], state["pool_y"][k]))
    m.delete(state["ids"].pop(0))
    state["next"] += 1
    return {"mean": p.mean, "variance": p.variance, "alpha": m.alpha()}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Each input read once and each output written once; the flops of the
    dense algebra (n³/3 for a factor, as much for a triangular inverse and
    for its product with itself, n² per solved right-hand side)."""
    kind, d = case["kind"], case["d"]
    p = {"rbf": 2, "rbf_ard": d + 1, "const_ard": d + 2, "rbf_periodic": 4}[case["tree"]]
    if kind == "batch":
        u = [(i + 0.5) / 256 for i in range(256)]
        ns = [case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** v for v in u]
        per = case["count"] / 256.0
        return {"bytes": per * sum(8 * (n * (d + 1) + 2 * p + 1) for n in ns),
                "flops": per * sum(n ** 3 + 2 * n * n for n in ns)}
    n = float(case["n"])
    if kind == "sgpr":
        m = float(case["m"])
        return {"bytes": 8 * (n * (d + 1) + m * d + 2 * p + 1), "flops": 7 * m * m * n + 2 * m ** 3 / 3}
    if kind == "eval":
        return {"bytes": 8 * (n * (d + 1) + 2 * p + 1), "flops": n ** 3 + 2 * n * n}
    if kind == "hessian":
        return {"bytes": 8 * (n * (d + 1) + p * p + 2 * p + 1), "flops": n ** 3 + (p - 1) * 4 * n ** 3 / 3}
    q = float(case["q"])
    if kind == "predict":
        return {"bytes": 8 * (n * (n + 1) / 2 + n * (d + 1) + q * (d + 2)), "flops": q * (n * n + 2 * n)}
    if kind == "model":
        return {"bytes": 8 * (n * (d + 1) + q * (d + 2)), "flops": n ** 3 / 3 + q * n * n + 2 * n * n}
    # online: the factor is read and written once; solves of q + 1 columns, a rank-one update, α
    return {"bytes": 8 * (n * (n + 1) + n * (d + 2) + q * (d + 2)), "flops": (q + 1) * n * n + 2 * n * n + 2 * n * n}


# ---------------------------------------------------------------------------
# the same results from plain torch in 64 bits
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=_dev())


def _cols(x, n, d):
    return _t(x).reshape(d, n)


def _k(tree, th, a, b):
    """k(a, b) of points given feature by feature (d × n), θ as a tensor."""
    d = a.shape[-2]

    def sq(inv):
        r = None
        for f in range(d):
            e = (a[..., f, :].unsqueeze(-1) - b[..., f, :].unsqueeze(-2)) ** 2
            e = e if inv is None else e * inv[..., f, None, None]
            r = e if r is None else r + e
        return r

    def at(i):
        return torch.exp(th[..., i, None, None])

    if tree == "rbf":
        return torch.exp(-0.5 * sq(None) / at(0) ** 2)
    if tree == "rbf_ard":
        return torch.exp(-0.5 * sq(torch.exp(-2.0 * th[..., :d])))
    if tree == "const_ard":
        return at(0) * torch.exp(-0.5 * sq(torch.exp(-2.0 * th[..., 1:1 + d])))
    r2 = sq(None)
    r = torch.sqrt(torch.where(r2 > 0, r2, torch.ones_like(r2))) * (r2 > 0)
    return (torch.exp(-0.5 * r2 / at(0) ** 2)
            + torch.exp(-2.0 * (torch.sin(math.pi * r / at(2)) / at(1)) ** 2))


def _dk(tree, th, x):
    """∂K/∂θ_i for every kernel parameter, one at a time."""
    d = x.shape[-2]

    def diff2(f):
        return (x[..., f, :].unsqueeze(-1) - x[..., f, :].unsqueeze(-2)) ** 2

    def at(i):
        return torch.exp(th[..., i, None, None])

    if tree in ("rbf_ard", "const_ard"):
        k = _k(tree, th, x, x)
        if tree == "const_ard":
            yield k
        for f in range(d):
            yield k * diff2(f) * at(f + (1 if tree == "const_ard" else 0)) ** -2
        return
    r2 = sum(diff2(f) for f in range(d))
    yield torch.exp(-0.5 * r2 / at(0) ** 2) * r2 / at(0) ** 2
    if tree == "rbf":
        return
    a = math.pi * torch.sqrt(r2) / at(2)
    s = torch.sin(a)
    kp = torch.exp(-2.0 * (s / at(1)) ** 2)
    yield kp * 4.0 * s * s / at(1) ** 2
    yield kp * 4.0 * s * torch.cos(a) * a / at(1) ** 2


def _objective(tree, th, x, y, live=None):
    """NLML and gradient of a stack of problems (padded rows: live = 0)."""
    n = x.shape[-1]
    k = _k(tree, th, x, x)
    noise = torch.exp(th[..., -1])[..., None, None]
    eye = torch.eye(n, dtype=k.dtype, device=k.device)
    if live is not None:
        pair = live.unsqueeze(-1) * live.unsqueeze(-2)
        k = k * pair + noise * eye * live.unsqueeze(-1) + eye * (1.0 - live).unsqueeze(-1)
        count = live.sum(-1)
    else:
        k = k + noise * eye
        count = float(n)
    c = torch.linalg.cholesky(k)
    del k
    alpha = torch.cholesky_solve(y.unsqueeze(-1), c)
    nlml = 0.5 * ((y.unsqueeze(-1) * alpha).sum((-1, -2))
                  + 2.0 * torch.log(torch.diagonal(c, dim1=-2, dim2=-1)).sum(-1) + count * math.log(2 * math.pi))
    w = alpha @ alpha.mT - torch.cholesky_inverse(c)
    if live is not None:
        w = w * pair
    g = [-0.5 * (w * dk).sum((-1, -2)) for dk in _dk(tree, th, x)]
    g.append(-0.5 * torch.exp(th[..., -1]) * torch.diagonal(w, dim1=-2, dim2=-1).sum(-1))
    return nlml, torch.stack(g, -1), c, alpha


def _posterior(case, th, x, y, xs):
    n = x.shape[1]
    k = _k(case["tree"], th, x, x)
    k.diagonal().add_(torch.exp(th[-1]))
    c = torch.linalg.cholesky(k)
    alpha = torch.cholesky_solve(y.reshape(n, 1), c)
    ks = _k(case["tree"], th, x, xs)
    v = torch.linalg.solve_triangular(c, ks, upper=False)
    kss = float(_k(case["tree"], th, x[:, :1], x[:, :1]))
    var = torch.clamp(kss - (v * v).sum(0), min=0.0) + torch.exp(th[-1])
    return (ks.T @ alpha).reshape(-1), var, alpha.reshape(-1)


def _hessian(case, th, x, y):
    """By differentiating the gradient −½⟨ααᵀ − K⁻¹, ∂K/∂θ⟩ in closed form."""
    tree, d = case["tree"], case["d"]
    n = x.shape[1]
    nlml, grad, c, alpha = _objective(tree, th, x, y)
    kinv = torch.cholesky_inverse(c)
    w = alpha @ alpha.T - kinv
    noise = torch.exp(th[-1])
    dks = list(_dk(tree, th, x))
    k = _k(tree, th, x, x)
    off = 1 if tree == "const_ard" else 0
    p = len(dks) + 1
    diff = [(x[f].unsqueeze(1) - x[f].unsqueeze(0)) ** 2 * torch.exp(-2.0 * th[off + f]) for f in range(d)]
    h = torch.zeros(p, p, dtype=k.dtype, device=k.device)
    t = [kinv @ dk for dk in dks] + [kinv * noise]
    v = [dk @ alpha for dk in dks] + [noise * alpha]
    for i in range(p):
        for j in range(i + 1):
            if i == p - 1 and j < p - 1:
                second = 0.0
            elif i == p - 1:
                second = noise * torch.diagonal(w).sum()
            elif j < off:  # ∂²/∂log c ∂θ_i
                second = (w * dks[i]).sum()
            else:
                q = k * diff[i - off] * diff[j - off]
                if i == j:
                    q = q - 2.0 * dks[i]
                second = (w * q).sum()
            e = -0.5 * second - 0.5 * (t[i] * t[j].T).sum() + (v[i].T @ (kinv @ v[j])).sum()
            h[i, j] = h[j, i] = e
    del n
    return nlml, grad, h


def _vfe(case, data):
    """The collapsed bound and its gradient by reverse differentiation, the
    cross covariance rebuilt part by part."""
    from torch.utils.checkpoint import checkpoint

    n, m, d = case["n"], case["m"], case["d"]
    th = _t(data["at"]).requires_grad_(True)
    x, y, z = _cols(data["x"], n, d), _t(data["y"]), _cols(data["z"], m, d)
    tree = case["tree"]
    kmm = _k(tree, th, z, z)
    noise = torch.exp(th[-1])
    c = torch.linalg.cholesky(kmm)

    def part(th, c, xp, yp):
        a = torch.linalg.solve_triangular(c, _k(tree, th, z, xp), upper=False)
        return a @ a.T, a @ yp, (1.0 - (a * a).sum(0)).sum()

    aat, ay, residual = 0.0, 0.0, 0.0
    for s in range(0, n, 65536):
        g, v, r = checkpoint(part, th, c, x[:, s:s + 65536], y[s:s + 65536], use_reentrant=False)
        aat, ay, residual = aat + g, ay + v, residual + r
    eye = torch.eye(m, dtype=torch.float64, device=x.device)
    lb = torch.linalg.cholesky(eye + aat / noise)
    w = torch.linalg.solve_triangular(lb, ay.unsqueeze(1) / noise, upper=False)
    nlml = 0.5 * (n * math.log(2 * math.pi) + n * torch.log(noise) + 2.0 * torch.log(torch.diagonal(lb)).sum()
                  + (y * y).sum() / noise - (w * w).sum() + residual / noise)
    grad, = torch.autograd.grad(nlml, th)
    return nlml.detach(), grad


def _batch(case, data):
    """The problems in groups of like size, padded to one."""
    ns = [y.size for y in data["ys"]]
    d, count = case["d"], len(ns)
    nlml = torch.zeros(count, dtype=torch.float64, device=_dev())
    grad = torch.zeros(count, data["params"].shape[1], dtype=torch.float64, device=_dev())
    order = sorted(range(count), key=lambda i: ns[i])
    while order:
        top = ns[order[-1]]
        take = max(1, min(len(order), int(6e8 / (top * top * 40))))
        group = [i for i in order[-take:] if ns[i] > top - max(16, top // 8)]
        order = order[:len(order) - len(group)]
        x, y, live = np.zeros((len(group), d, top)), np.zeros((len(group), top)), np.zeros((len(group), top))
        for r, i in enumerate(group):
            x[r, :, :ns[i]] = data["xs"][i].reshape(d, ns[i])
            x[r, :, ns[i]:] = data["xs"][i].reshape(d, ns[i])[:, :1]
            y[r, :ns[i]] = data["ys"][i]
            live[r, :ns[i]] = 1.0
        v, g, _, _ = _objective(case["tree"], _t(data["params"][group]), _t(x), _t(y), _t(live))
        nlml[group], grad[group] = v, g
    return nlml, grad


def exact(case, seed):
    kind, d = case["kind"], case["d"]
    if kind == "batch":
        nlml, grad = _batch(case, _batch_data(case, seed))
        return {"nlml": nlml, "grad": grad, "status": None}
    if kind == "sgpr":
        nlml, grad = _vfe(case, _sgpr_data(case, seed))
        return {"nlml": float(nlml), "grad": grad}
    data = _exact_data(case, seed)
    n = case["n"]
    x, y = _cols(data["x"], n, d), _t(data["y"])
    if kind == "eval":
        nlml, grad, _, _ = _objective(case["tree"], _t(data["at"]), x, y)
        return {"nlml": float(nlml), "grad": grad}
    if kind == "hessian":
        nlml, grad, hess = _hessian(case, _t(data["at"]), x, y)
        return {"nlml": float(nlml), "grad": grad, "hess": hess}
    th = _t(data["theta"])
    mean, var, alpha = _posterior(case, th, x, y, _cols(data["xs"], case["q"], d))
    if kind != "online":
        return {"mean": mean, "variance": var}
    # the window after its first move: the first point gone, the pool's first point last
    x1 = torch.cat([x[:, 1:], _t(data["pool_x"][0]).reshape(d, 1)], 1)
    y1 = torch.cat([y[1:], _t(data["pool_y"][:1])])
    return {"mean": mean, "variance": var, "alpha": _posterior(case, th, x1, y1, x1[:, :1])[2]}
