"""Leaf values of the gradient's dK (integer distances) for heavily weighted features:
30 pairs of a periodic leaf at E = |f_i - f_j|^2 = 1, weight e^8 (features up to 55),
under a nugget that makes the gradient sum_pairs y_i y_j dK_ij up to 10^-3 of it.

Tolerance: sin(d / 2) = 0.009 of a pair carries two roundings of 10^-16, its square
2 10^-14 (rms 1e-14), the features' units 5e-15 in E; over 30 pairs 2e-15 rms, allowed
seven times that."""
import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu


def test_heavily_weighted_periodic_leaf(lib):
    from fgpu import Engine
    n, theta, nugget = 60, -4.0, 1e3
    rng = np.random.default_rng(11)
    w = np.exp(-theta)
    X = np.empty((n, 1))
    X[::2, 0] = -3.0 + 0.2 * np.arange(n // 2) + rng.uniform(0.0, 0.01, size=n // 2)
    X[1::2, 0] = X[::2, 0] + 2.0 * np.arcsin(rng.uniform(0.45, 0.55, size=n // 2) / w)
    y = rng.uniform(10.0, 20.0, size=n)
    ks, th = [O.PERIODIC, 1, 1], np.array([theta])
    ll, g, info = Engine(X, y, np.zeros(n), ks, 0, nugget, False).grad(th)
    ld = np.longdouble
    x = X[:, 0].astype(ld)
    q = np.exp(ld(-2 * theta)) * np.sin((x[:, None] - x[None]) / 2) ** 2
    V = np.exp(-2 * q)
    K = V + np.eye(n, dtype=ld) * nugget
    # K^-1 = (I + V / nugget)^-1 / nugget by its series: ||V / nugget|| < 2e-3
    Kinv = term = np.eye(n, dtype=ld)
    for _ in range(12):
        term = -(V @ term) / nugget
        Kinv = Kinv + term
    Kinv = Kinv / nugget
    assert np.abs(K @ Kinv - np.eye(n)).max() < 1e-17
    a = Kinv @ y.astype(ld)
    want = float(((np.outer(a, a) - Kinv) * V * 4 * q).sum() / 2)
    assert info == 0
    assert abs(g[0] - want) <= 1.5e-14 * abs(want), (g[0], want, abs(g[0] / want - 1))
