"""The adjoint's K^-1 on the tensor cores (csrc/inv.cu) at the edges of its
block recursion: one tile, one column past it, block counts that are not a
power of two; the last three around the size from which the dK/dtheta pass runs two
CTAs per SM.  Same tolerance as the other gradient tests: 1e-6 relative to
the oracle's FP64 gradient, 1e-9 of its largest component for those that
cancel."""
import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [127, 128, 129, 257, 385, 640, 897, 1024, 1025, 1200])
@pytest.mark.parametrize("lik", [0, 1])
def test_gradient_at_block_edges(n, lik, lib):
    from fgpu import Engine
    rng = np.random.default_rng(n)
    X = rng.normal(2.0, 0.3, size=(n, 4))
    X[:, 2:] = rng.uniform(-np.pi, np.pi, size=(n, 2))
    y = np.cos(X[:, 0]) + 0.3 * np.sin(X[:, 2]) + 1e-3 * rng.normal(size=n)
    ks = [O.RBF, 2, 1, 2, O.PERIODIC, 2, 3, 4, O.SUM]
    mu = O.mean_vector("constant", X, y)
    th = np.array([0.4, 0.7, 0.2, 0.5, 1e-3])
    e = Engine(X, y, mu, ks, lik, 1e-3, True)
    ll, g, info = e.grad(th)
    rll, rg, rinfo = O.loglik_grad(ks, th, X, y, mu, lik, 1e-3, True)
    assert info == rinfo == 0
    assert abs(ll - rll) <= 1e-9 * abs(rll)
    assert np.all(np.abs(g - rg) <= 1e-6 * np.abs(rg) + 1e-9 * np.max(np.abs(rg))), (g, rg)
    # the workspace is reused as it is: a second call gives the same bits
    ll2, g2, _ = e.grad(th)
    assert ll2 == ll and np.array_equal(g2, g)
