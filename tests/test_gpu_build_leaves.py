"""Sums and products of two distance leaves in the tensor-core build's fixed point,
at the edges of its tiles, and with one leaf whose scale lies outside the
exponential's common form (features that do not vary, vary by 1e-15 or by 1e9): both
leaves then combine in FP64.  Against the oracle (1e-9 relative, the well conditioned
cases' tolerance) and the FP64 build (2e-9)."""
import os

import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu


def _engine(X, y, ks, lik, build):
    from fgpu import Engine
    old = os.environ.get("FGPU_BUILD")
    os.environ["FGPU_BUILD"] = build
    try:
        return Engine(X, y, O.mean_vector("constant", X, y), ks, lik, 1e-3, False)
    finally:
        if old is None:
            del os.environ["FGPU_BUILD"]
        else:
            os.environ["FGPU_BUILD"] = old


def _check(X, y, ks, lik):
    th = np.random.default_rng(4).uniform(0.2, 0.9, size=O.kernel_nparams(ks))
    ll, info = _engine(X, y, ks, lik, "tc").loglik(th)
    fp, i_fp = _engine(X, y, ks, lik, "fp64").loglik(th)
    ref, rinfo = O.loglik(ks, th, X, y, O.mean_vector("constant", X, y), lik, 1e-3, False)
    assert info == i_fp == rinfo == 0
    assert abs(ll - ref) <= 1e-9 * abs(ref), (ll, ref)
    assert abs(ll - fp) <= 2e-9 * abs(ref), (ll, fp)


def _data(n, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(1.0, 0.4, size=(n, 5))
    X[:, 4] = rng.uniform(-np.pi, np.pi, size=n)
    y = np.sin(X[:, 0]) + 0.3 * np.cos(X[:, 4]) + 0.03 * rng.normal(size=n)
    return X, y


@pytest.mark.parametrize("n", [3, 63, 64, 65, 127, 128, 129, 300])
@pytest.mark.parametrize("op", ["sum", "prod"])
def test_two_leaves(n, op, lib):
    X, y = _data(n, n)
    ks = [O.RBF, 4, 1, 2, 3, 4, O.PERIODIC, 1, 5, O.SUM if op == "sum" else O.PROD]
    _check(X, y, ks, n % 2)


# 30, 42 and 90 tiles: a CTA takes a quarter, half and the whole of one
@pytest.mark.parametrize("n", [600, 700, 1100])
@pytest.mark.parametrize("op", ["sum", "prod"])
def test_parts_of_tiles(n, op, lib):
    X, y = _data(n, n)
    ks = [O.RBF, 4, 1, 2, 3, 4, O.PERIODIC, 1, 5, O.SUM if op == "sum" else O.PROD]
    _check(X, y, ks, 1)


@pytest.mark.parametrize("spread", [0.0, 1e-15, 1e9])
@pytest.mark.parametrize("op", ["sum", "prod"])
@pytest.mark.parametrize("first", [True, False])
def test_one_leaf_out_of_scale(spread, op, first, lib):
    X, y = _data(150, 7)
    X[:, :2] = spread * (X[:, :2] - 1.0)
    odd, per = [O.RBF, 2, 1, 2], [O.PERIODIC, 1, 5]
    ks = (odd + per if first else per + odd) + [O.SUM if op == "sum" else O.PROD]
    _check(X, y, ks, 0)
