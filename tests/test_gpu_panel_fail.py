"""A pivot that fails in any piece of a panel: the diagonal tile marks the counters that
its problem's other CTAs wait on while its own warps may still publish earlier
pieces there.  Every call returns ``info`` = the failing column (of a pair of equal
points under a small negative nugget), alone and in a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(n, col):
    from fgpu import RBF, Engine
    side = int(np.ceil(n ** (1 / 3)))
    X = np.stack(np.meshgrid(*[np.arange(side) * 8.0] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n].copy()
    X[col - 1] = X[col // 2 - 1]
    return Engine(X, np.ones(n), np.zeros(n), [RBF, 3, 1, 2, 3], 0, -1e-6, False)


@pytest.mark.parametrize("n", [128, 300, 1000])
def test_failure_in_every_piece(n, lib):
    from fgpu import loglik_batch
    th = np.zeros(3)
    cols = list(range(3, n + 1, 7 if n < 1000 else 61)) + [n]
    es = [_engine(n, c) for c in cols]
    for e, c in zip(es, cols):
        for _ in range(3):
            ll, info = e.loglik(th)
            assert info == c and np.isnan(ll)
    ll, info = loglik_batch(es, [th] * len(es))
    assert list(info) == cols and np.all(np.isnan(ll))
