"""Batches whose panels have more row tiles than the GPU has SMs: their diagonal
tiles go first (beside the previous panel's update, where it has enough tiles) and
the rows follow two tiles to an SM.  The arithmetic is the one of the single
launch, so every problem's value is bit-identical to its own lone
evaluation; the oracle's tolerance is the well conditioned cases' 1e-9 relative."""
import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu


def _engine(n, lik, noise=1e-3, repeat=0):
    from fgpu import Engine
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 4))
    y = np.sin(X[:, 0]) + 0.3 * X[:, 1] ** 2
    if repeat:  # equal points without noise: K is singular
        X[-repeat:], y[-repeat:] = X[:repeat], y[:repeat]
    mu = O.mean_vector("constant", X, y)
    ks = [O.RBF, 4, 1, 2, 3, 4]
    return Engine(X, y, mu, ks, lik, noise, False), lambda th: O.loglik(ks, th, X, y, mu, lik, noise, False)


# one row tile under the diagonal one, ragged last tiles, several full panels
@pytest.mark.parametrize("n,s", [(129, 400), (200, 400), (256, 400), (257, 250), (385, 150), (640, 100), (1000, 60)])
@pytest.mark.parametrize("lik", [0, 1])
def test_batch_equals_lone_evaluations(n, s, lik, lib):
    from fgpu import loglik_batch
    e, ref = _engine(n, lik)
    th = np.random.default_rng(2).uniform(0.2, 0.9, size=(s, 4))
    ll, info = loglik_batch([e] * s, list(th))
    assert np.all(info == 0)
    for k in (0, 1, s // 2, s - 1):
        one, i1 = e.loglik(th[k])
        assert i1 == 0 and ll[k] == one, (k, ll[k], one)
    want, _ = ref(th[0])
    assert abs(ll[0] - want) <= 1e-9 * abs(want), (ll[0], want)


def test_failed_problem_leaves_the_others_alone(lib):
    from fgpu import loglik_batch
    good, _ = _engine(385, 0)
    bad, _ = _engine(300, 0, noise=0.0, repeat=140)
    th = np.full(4, 0.4)
    one, _ = good.loglik(th)
    bad_one, bad_info = bad.loglik(np.full(4, 1.0))
    assert bad_info > 0 and np.isnan(bad_one)
    es = [good] * 150
    ts = [th] * 150
    for k in (0, 77, 149):
        es[k], ts[k] = bad, np.full(4, 1.0)
    ll, info = loglik_batch(es, ts)
    for k in range(150):
        if k in (0, 77, 149):
            assert info[k] == bad_info and np.isnan(ll[k])
        else:
            assert info[k] == 0 and ll[k] == one
