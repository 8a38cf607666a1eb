"""Performance cases of the likelihood engine: what a hyperparameter search
asks of it, through the package's public entry points.

* ``plain``: ``Engine.loglik``, one particle per call (the drop-in for the
  reference's likelihood call), optionally with alpha, the model file's weights;
* ``swarm``: ``Plan.run``, a whole swarm per call with host theta in and host
  log-likelihoods out, or ``Plan.run_device`` with theta resident on the GPU;
* ``grad``: ``Engine.grad``, the log-likelihood and its gradient (the polish of
  a swarm's global best).

Data are seeded stand-ins for molecular training sets: bond lengths and angles
scattered about an equilibrium, dihedrals uniform on the circle, and a smooth
random-Fourier-feature target.  Nuggets are the default 1e-10 where dihedrals
keep the kernel matrix well conditioned; the families without that (``water``,
``methanol``) carry a nugget of the size of their targets' noise, so that two
FP64 evaluations of one likelihood agree.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "ferebus-v7_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import fgpu  # noqa: E402
from fgpu.gpr import mean_vector  # noqa: E402

NOISE = {"water": 1e-5, "methanol": 1e-4, "glycine": 1e-10, "cyclic": 1e-10}


def _case(name, entry, family, n, d, s=1, likelihood="marginal", mean="constant", optimise_noise=False, alpha=False,
          op="+", atoms=1, n_min=0, device=False):
    case = {"entry": entry, "family": family, "n": n, "d": d, "s": s, "likelihood": likelihood,
            "mean": mean, "optimise_noise": optimise_noise, "alpha": alpha, "op": op, "atoms": atoms, "n_min": n_min,
            "device": device}
    return {"name": name, **case} if name else case


def listed():
    return [
        # one call on a small hand-made training set, the product of an rbf
        # and a periodic kernel: launches and latency alone
        _case("plain_59", "plain", "water", 59, 3, op="*"),
        # one call on a first training set of a few hundred geometries
        _case("plain_500", "plain", "methanol", 500, 12),
        # one call at the headline training-set size
        _case("plain_4000", "plain", "glycine", 4000, 24, likelihood="concentrated"),
        # the model writer's call: likelihood and weights, at an odd size
        _case("alpha_1501", "plain", "glycine", 1501, 24, alpha=True),
        # one iteration of a small molecule's swarm
        _case("swarm_500x20", "swarm", "water", 500, 3, s=20),
        # one iteration of a mid-sized swarm
        _case("swarm_2000x50", "swarm", "methanol", 2000, 12, s=50),
        # one iteration of the headline swarm, theta kept on the GPU
        _case("swarm_4000x40", "swarm", "glycine", 4000, 24, s=40, likelihood="concentrated", device=True),
        # one iteration on a large training set, noise optimised
        _case("swarm_10000x16", "swarm", "glycine", 10000, 30, s=16, mean="quadratic", optimise_noise=True),
        # one iteration over the atoms of a molecule, each with a training set of its own size
        _case("atoms_16x10", "swarm", "glycine", 6000, 93, s=10, mean="linear", atoms=16, n_min=500),
        # the wrapped-difference kernel, which takes the FP64 kernel-matrix build
        _case("cyclic_1000x20", "swarm", "cyclic", 1000, 24, s=20),
        # one gradient during the polish of a small model, noise optimised, odd size
        _case("grad_1003", "grad", "glycine", 1003, 24, optimise_noise=True),
        # one gradient at the headline training-set size
        _case("grad_4000", "grad", "glycine", 4000, 24, likelihood="concentrated"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: an entry point, a kernel family and sizes spread over their range."""
    entry = rng.choice(["plain", "plain", "swarm", "swarm", "swarm", "grad", "atoms"])
    if entry == "atoms":
        return _case("", "swarm", "glycine", _log_uniform(rng, 1500, 6000), 3 * rng.randint(8, 31),
                     s=rng.randint(3, 10), mean=rng.choice(["constant", "linear"]), atoms=rng.randint(2, 16),
                     n_min=rng.randint(100, 900))
    family = rng.choice(["water", "methanol", "glycine", "glycine", "cyclic"])
    top = {"water": 500, "methanol": 2500, "glycine": 10000, "cyclic": 2000}[family]
    if entry == "grad":
        family, top = "glycine", 4500
    n = _log_uniform(rng, 50, top)
    # enough dihedrals for the size that the default nugget leaves the kernel matrix well conditioned
    d = {"water": 3, "methanol": 12}.get(family) or 3 * rng.randint(6 if n < 3000 and family == "glycine" else 8, 10)
    s = 1
    if entry == "swarm":
        # no more than the largest listed case's work, and at most 60 particles
        s = max(2, min(rng.randint(8, 60), int(16e12 / float(n) ** 3)))
    means = ["constant", "linear", "quadratic"] if family == "glycine" else ["zero", "constant"]
    return _case("", entry, family, n, d, s=s, likelihood=rng.choice(["marginal", "concentrated"]),
                 mean=rng.choice(means), optimise_noise=family == "glycine" and rng.random() < 0.4,
                 alpha=entry == "plain" and family != "water" and rng.random() < 0.4,
                 op=rng.choice(["+", "+", "*"]), device=entry == "swarm" and rng.random() < 0.5)


def _dihedrals(d):
    return [j for j in range(d) if j >= 5 and j % 3 == 2]


def _features(rng, family, n, d):
    X = np.empty((n, d))
    if family == "water":
        X[:, :2] = rng.normal(1.81, 0.05, size=(n, 2))
        X[:, 2] = rng.normal(1.82, 0.08, size=n)
        return X, [2]
    if family == "methanol":
        X[:, :6] = rng.normal(2.0, 0.1, size=(n, 6))
        X[:, 6:9] = rng.uniform(1.7, 2.1, size=(n, 3))
        X[:, 9:] = rng.uniform(-np.pi, np.pi, size=(n, d - 9))
        return X, list(range(9, d))
    dih = _dihedrals(d)
    for j in range(d):
        X[:, j] = rng.uniform(-np.pi, np.pi, size=n) if j in dih else rng.normal(2.2, 0.15, size=n)
    return X, dih


def _target(rng, family, X):
    n, d = X.shape
    if family == "water":
        return (-75.4 + 0.3 * np.sin(2.0 * X[:, 0]) + 0.2 * (X[:, 1] - 1.81) ** 2
                + 0.1 * np.sin(X[:, 2]) * np.cos(X[:, 0]) + rng.normal(0.0, math.sqrt(1e-5), n))
    w = rng.normal(0.0, 1.0, size=(64, d))
    b = rng.uniform(0.0, 2 * np.pi, size=64)
    a = rng.normal(0.0, 1.0 / 8.0, size=64)
    return np.cos(X @ w.T + b) @ a + rng.normal(0.0, math.sqrt(1e-5), n)


def _problems(case, seed):
    """The training sets of a case and their particles, on the host."""
    rng = np.random.default_rng([seed, case["n"], case["d"], case["s"], case["atoms"]])
    fam, d = case["family"], case["d"]
    sizes = [case["n"]] if case["atoms"] == 1 else list(rng.integers(case["n_min"], case["n"] + 1, size=case["atoms"]))
    out = []
    for n in sizes:
        X, dih = _features(rng, fam, int(n), d)
        y = _target(rng, fam, X)
        rest = [j for j in range(d) if j not in dih]
        if fam == "cyclic":
            leaves = [("cyclic", list(range(d)))]
            kspec = [fgpu.RBF_CYCLIC, d] + [j + 1 for j in range(d)]
        else:
            leaves = [("rbf", rest), ("periodic", dih)]
            kspec = ([fgpu.RBF, len(rest)] + [j + 1 for j in rest] + [fgpu.PERIODIC, len(dih)] + [j + 1 for j in dih]
                     + [fgpu.SUM if case["op"] == "+" else fgpu.PROD])
        th = rng.uniform(1e-3, 1.0, size=(case["s"], d))
        if case["optimise_noise"]:
            th = np.concatenate([th, 10.0 ** rng.uniform(-12.0, -6.0, size=(case["s"], 1))], axis=1)
        out.append({"X": X, "y": y, "mu": mean_vector(case["mean"], X, y), "kspec": kspec, "leaves": leaves,
                    "theta": th})
    return out


_stream = None


def _shared_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def prepare(case, seed):
    lik = fgpu.CONCENTRATED if case["likelihood"] == "concentrated" else fgpu.MARGINAL
    probs = _problems(case, seed)
    engines = [fgpu.Engine(p["X"], p["y"], p["mu"], p["kspec"], lik, NOISE[case["family"]], case["optimise_noise"])
               for p in probs]
    state = {"entry": case["entry"], "alpha": case["alpha"], "device": case["device"], "engines": engines}
    if case["entry"] != "swarm":
        state["theta"] = probs[0]["theta"][0]
        return state
    state["theta"] = np.concatenate([p["theta"] for p in probs])
    state["plan"] = fgpu.Plan([e for e in engines for _ in range(case["s"])])
    if case["device"]:
        state["stream"] = _shared_stream()
        state["theta_dev"] = torch.tensor(state["theta"], dtype=torch.float64, device="cuda")
        state["ll"] = torch.empty(len(state["theta"]), dtype=torch.float64, device="cuda")
        state["info"] = torch.empty(len(state["theta"]), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
    return state


def run(state):
    if state["entry"] == "plain":
        return state["engines"][0].loglik(state["theta"], want_alpha=state["alpha"])
    if state["entry"] == "grad":
        return state["engines"][0].grad(state["theta"])
    if state["device"]:
        state["plan"].run_device(state["theta_dev"].data_ptr(), state["ll"].data_ptr(), state["info"].data_ptr(),
                                 state["stream"].cuda_stream)
        return state["ll"], state["info"]
    return state["plan"].run(state["theta"])


def work(case):
    """One evaluation: the features and targets in, a kernel value per pair
    (about 3 operations a feature, 20 an exponential), N^3 / 3 for the
    Cholesky factor, two triangular solves; the gradient adds the inverse and
    a pass over the kernel's derivatives."""
    mid = (case["n_min"] + case["n"]) / 2.0
    spread = (case["n"] - case["n_min"]) if case["atoms"] > 1 else 0.0
    n1 = float(case["n"]) if case["atoms"] == 1 else mid
    n2 = n1 * n1 + spread * spread / 12.0          # the mean of N^2 and N^3 over the atoms' sizes
    n3 = n1 ** 3 + n1 * spread * spread / 4.0
    evals = case["s"] * case["atoms"]
    d = case["d"]
    flops = n3 / 3.0 + n2 / 2.0 * (3.0 * d + 40.0) + 2.0 * n2
    if case["entry"] == "grad":
        flops += 2.0 * n3 / 3.0 + n2 / 2.0 * 4.0 * d
    nbytes = 8.0 * (case["atoms"] * n1 * (d + 2) + evals * (d + 2))
    if case["alpha"]:
        nbytes += 8.0 * n1
    return {"bytes": nbytes, "flops": flops * evals}


def _exact_one(p, th, case, noise):
    """Log-likelihood, alpha, the factor and the pieces of dK/dtheta, in 64-bit torch."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = torch.tensor(p["X"], dtype=torch.float64, device=dev)
    y = torch.tensor(p["y"], dtype=torch.float64, device=dev)
    n = X.shape[0]
    vals, o = [], 0
    for kind, dims in p["leaves"]:
        e = torch.zeros(n, n, dtype=torch.float64, device=dev)
        for k, j in enumerate(dims):
            diff = X[:, j, None] - X[None, :, j]
            if kind == "periodic":
                e.addcmul_(diff.div_(2).sin_(), diff, value=-2.0 * math.exp(-2.0 * th[o + k]))
            else:
                if kind == "cyclic" and (j + 1) % 3 == 0:
                    diff = torch.sign(diff) * (torch.remainder(diff.abs() + math.pi, 2 * math.pi) - math.pi)
                e.addcmul_(diff, diff, value=-0.5 * math.exp(th[o + k]))
        vals.append(e.exp_())
        o += len(dims)
    K = vals[0].clone() if len(vals) == 1 else (vals[0] + vals[1] if case["op"] == "+" else vals[0] * vals[1])
    K.diagonal().add_(th[-1] if case["optimise_noise"] else noise)
    L = torch.linalg.cholesky(K)
    del K
    logdet = 2.0 * L.diagonal().log().sum()
    if case["likelihood"] == "concentrated":
        one = torch.ones(n, 1, dtype=torch.float64, device=dev)
        z = torch.linalg.solve_triangular(L, torch.cat([y[:, None], one], 1), upper=False)
        mean = (z[:, 0] @ z[:, 1]) / (z[:, 1] @ z[:, 1])
        w = z[:, 0] - mean * z[:, 1]
        s2 = (w @ w) / n
        ll = -0.5 * n * torch.log(s2) - 0.5 * logdet
    else:
        w = torch.linalg.solve_triangular(L, (y - torch.tensor(p["mu"], device=dev))[:, None], upper=False)[:, 0]
        s2 = torch.ones((), dtype=torch.float64, device=dev)
        ll = -0.5 * (w @ w) - 0.5 * logdet - 0.5 * n * math.log(2.0 * math.pi)
    return X, L, w, s2, ll, vals


def exact(case, seed):
    """What ``run`` returns, by torch's FP64 elementwise operations, Cholesky and triangular solves."""
    probs = _problems(case, seed)
    noise = NOISE[case["family"]]
    if case["entry"] == "swarm":
        ll = [float(_exact_one(p, th, case, noise)[4]) for p in probs for th in p["theta"]]
        return (torch.tensor(ll, dtype=torch.float64) if case["device"] else np.asarray(ll)), None
    p, th = probs[0], probs[0]["theta"][0]
    X, L, w, s2, ll, vals = _exact_one(p, th, case, noise)
    if case["entry"] == "plain" and not case["alpha"]:
        return float(ll), None
    alpha = torch.linalg.solve_triangular(L.T, w[:, None], upper=True)[:, 0]
    if case["entry"] == "plain":
        return float(ll), None, alpha.cpu().numpy()
    W = alpha[:, None] * alpha[None, :] / s2 - torch.cholesky_inverse(L)
    g, o = [], 0
    for t, (kind, dims) in enumerate(p["leaves"]):
        V = W * vals[t]
        if case["op"] == "*" and len(vals) == 2:
            V = V * vals[1 - t]
        for k, j in enumerate(dims):
            diff = X[:, j, None] - X[None, :, j]
            if kind == "periodic":
                g.append(0.5 * 4.0 * math.exp(-2.0 * th[o + k]) * float((V * torch.sin(diff / 2) ** 2).sum()))
            else:
                g.append(-0.5 * 0.5 * math.exp(th[o + k]) * float((V * diff ** 2).sum()))
        o += len(dims)
    if case["optimise_noise"]:
        g.append(0.5 * float(W.diagonal().sum()))
    return float(ll), np.asarray(g), None
