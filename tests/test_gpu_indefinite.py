"""Nuggets below zero: K_ii = 1 + nugget is far smaller than the kernel values.
Where K is still positive definite the likelihood is the oracle's (1e-9 relative,
the well conditioned cases' tolerance), and where it is not, ``info`` is the first
leading minor that fails, as dpotrf has it."""
import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu


def _grid(n, step, dims=3):
    """n points of a cubic grid, far from one another."""
    side = int(np.ceil(n ** (1.0 / dims)))
    g = np.stack(np.meshgrid(*[np.arange(side) * step] * dims, indexing="ij"), axis=-1).reshape(-1, dims)
    return g[:n].astype(float)


@pytest.mark.parametrize("nugget", [-0.6, -0.8, -0.9, -0.96])
@pytest.mark.parametrize("spec", ["rbf", "rbf_plus_const", "cyclic"])
def test_small_diagonal_positive_definite(nugget, spec, lib):
    from fgpu import Engine, loglik_batch
    n = 150
    rng = np.random.default_rng(7)
    X = _grid(n, 7.0) + rng.uniform(-0.2, 0.2, size=(n, 3))
    if spec == "cyclic":
        X[:, 2] = rng.uniform(-1.0, 1.0, size=n)
        X[:, 0] += 50.0 * np.arange(n)
    y = rng.normal(size=n)
    ks = {"rbf": [O.RBF, 3, 1, 2, 3], "rbf_plus_const": [O.RBF, 3, 1, 2, 3, O.CONSTANT, 0, O.SUM],
          "cyclic": [O.RBF_CYCLIC, 3, 1, 2, 3]}[spec]
    th = np.array([0.1, 0.2, 0.05] + ([1e-6] if spec == "rbf_plus_const" else []))
    mu = np.zeros(n)
    ref, rinfo = O.loglik(ks, th, X, y, mu, 0, nugget, False)
    e = Engine(X, y, mu, ks, 0, nugget, False)
    ll, info = e.loglik(th)
    assert info == rinfo == 0
    assert abs(ll - ref) <= 1e-9 * abs(ref), (ll, ref)
    lb, ib = loglik_batch([e, e], [th, th])
    assert ib[0] == 0 and lb[0] == lb[1] == ll
