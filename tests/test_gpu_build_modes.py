"""The two kernel-matrix builds of the tensor-core mode, each really chosen
(set_build_mode; FGPU_BUILD is read once per process), over the kernels that both
serve and those that only the dot-product build does (more than two distance leaves,
an rbf-cyclic one): the oracle's likelihood to 1e-9, the well conditioned cases'
tolerance, and the two builds to 2e-9 of each other but not the same bits."""
import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu

RBF2, PER1 = [O.RBF, 2, 1, 2], [O.PERIODIC, 1, 5]
CYC = [O.RBF_CYCLIC, 5, 1, 2, 3, 4, 5]
BOTH = {
    "rbf": [O.RBF, 4, 1, 2, 3, 4],
    "periodic": [O.PERIODIC, 2, 4, 5],
    "sum": RBF2 + PER1 + [O.SUM],
    "prod": PER1 + RBF2 + [O.PROD],
    "prod_plus_const": RBF2 + PER1 + [O.PROD, O.CONSTANT, 0, O.SUM],
    "linear_times_periodic_plus_rbf": [O.LINEAR, 1, 1] + PER1 + [O.PROD] + RBF2 + [O.SUM],
}
DOT_ONLY = {
    "three_leaves": RBF2 + PER1 + [O.SUM, O.RBF, 2, 3, 4, O.PROD],
    "four_leaves": RBF2 + PER1 + [O.PROD, O.RBF, 1, 3, O.SUM, O.PERIODIC, 1, 4, O.PROD],
    "cyclic_plus_periodic": CYC + PER1 + [O.SUM],
    "cyclic_times_rbf_plus_periodic": CYC + RBF2 + [O.PROD] + PER1 + [O.SUM],
}


def _run(ks, n, build):
    from fgpu import Engine, loglik_batch
    from fgpu.gpr import set_build_mode
    rng = np.random.default_rng(n + len(ks))
    X = rng.normal(1.0, 0.4, size=(n, 5))
    X[:, 4] = rng.uniform(-np.pi, np.pi, size=n)
    y = np.sin(X[:, 0]) + 0.3 * np.cos(X[:, 4]) + 0.03 * rng.normal(size=n)
    mu, lik = O.mean_vector("constant", X, y), n % 2
    th = np.random.default_rng(4).uniform(0.2, 0.9, size=O.kernel_nparams(ks))
    prev = set_build_mode(build)
    try:
        e = Engine(X, y, mu, ks, lik, 1e-3, False)
    finally:
        set_build_mode(prev)
    ll, info = e.loglik(th)
    ref, rinfo = O.loglik(ks, th, X, y, mu, lik, 1e-3, False)
    assert info == rinfo == 0
    assert abs(ll - ref) <= 1e-9 * abs(ref), (build, ll, ref)
    lb, ib = loglik_batch([e, e, e], [th, th + 0.01, th])
    assert np.all(ib == 0) and lb[0] == lb[2] == ll
    return ll


@pytest.mark.parametrize("n", [2, 63, 65, 128, 129, 300])
@pytest.mark.parametrize("spec", sorted(BOTH))
def test_both_builds(spec, n, lib):
    tc, dot = _run(BOTH[spec], n, "tc"), _run(BOTH[spec], n, "fp64")
    assert abs(tc - dot) <= 2e-9 * abs(tc)
    assert n < 300 or tc != dot  # two builds, not one


@pytest.mark.parametrize("n", [2, 63, 65, 128, 129, 300])
@pytest.mark.parametrize("spec", sorted(DOT_ONLY))
def test_dot_product_build_alone(spec, n, lib):
    assert _run(DOT_ONLY[spec], n, "tc") == _run(DOT_ONLY[spec], n, "fp64")
