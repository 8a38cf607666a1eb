"""alpha = K^-1 (y - mu) from the one-launch back-substitution (csrc/engine.cu,
k_backsolve) at the edges of its 64-row blocks, in both engine modes: backward
residual ||K alpha - r|| <= 1e-12 ||K|| ||alpha|| on the oracle's K, and the same
bits on a second call (the blocks are handed from CTA to CTA)."""
import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 128, 129, 200, 1000])
@pytest.mark.parametrize("mode", ["tcgen05", "fp64"])
def test_alpha_at_block_edges(n, mode, lib):
    from fgpu import Engine
    from fgpu.gpr import set_trailing_update
    rng = np.random.default_rng(n)
    X = rng.normal(2.0, 0.3, size=(n, 4))
    X[:, 3] = rng.uniform(-np.pi, np.pi, size=n)
    y = np.cos(X[:, 0]) + 0.3 * np.sin(X[:, 3]) + 1e-3 * rng.normal(size=n)
    ks = [O.RBF, 3, 1, 2, 3, O.PERIODIC, 1, 4, O.SUM]
    mu = O.mean_vector("constant", X, y)
    th = np.array([0.4, 0.7, 0.2, 0.5])
    prev = set_trailing_update(mode)
    try:
        e = Engine(X, y, mu, ks, 0, 1e-4, False)
    finally:
        set_trailing_update(prev)
    ll, info, alpha = e.loglik(th, want_alpha=True)
    K = O.compute_R(ks, th, 1e-4, O.Tensors(X))
    K = np.tril(K) + np.tril(K, -1).T  # dpotrf reads the lower triangle, which is what the oracle fills
    r = y - mu
    assert info == 0
    assert np.linalg.norm(K @ alpha - r) <= 1e-12 * np.linalg.norm(K, 2) * np.linalg.norm(alpha) + 1e-300
    _, _, again = e.loglik(th, want_alpha=True)
    assert np.array_equal(alpha, again)
