"""The rbf-cyclic leaf's fixed-point distances (the tensor-core mode's
dot-product build) against the oracle: dihedrals wrapped across +-pi, far outside
[-pi, pi] and at exactly opposite angles, sizes at the edges of its 64-row tiles,
alone and combined with other leaves.  Tolerance: the well conditioned cases'
1e-9 relative.  A point that is not finite fails the evaluation, as it does in
the FP64 mode."""
import numpy as np
import pytest

from oracle import gpr_oracle as O

pytestmark = pytest.mark.gpu


def _data(n, d, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(2.0, 0.3, size=(n, d))
    X[:, 2::3] = rng.uniform(-np.pi, np.pi, size=X[:, 2::3].shape)
    X[: n // 3, 2] += 4 * np.pi          # whole turns away
    X[n // 2, 2::3] = np.pi              # opposite to the next point's 0
    X[n // 2 - 1, 2::3] = 0.0
    y = np.cos(X[:, 0]) + 0.2 * np.sin(X[:, 2]) + 1e-3 * rng.normal(size=n)
    return X, y


@pytest.mark.parametrize("n", [3, 63, 64, 65, 129, 300])
@pytest.mark.parametrize("spec", ["cyclic", "cyclic_plus_rbf", "cyclic_times_const_plus_linear"])
def test_cyclic_against_oracle(n, spec, lib):
    from fgpu import Engine
    d = 9
    X, y = _data(n, d, n)
    cyc = [O.RBF_CYCLIC, d, *range(1, d + 1)]
    ks = {"cyclic": cyc, "cyclic_plus_rbf": cyc + [O.RBF, 2, 1, 2, O.SUM],
          "cyclic_times_const_plus_linear": cyc + [O.CONSTANT, 0, O.PROD, O.LINEAR, 1, 2, O.SUM]}[spec]
    mu = O.mean_vector("constant", X, y)
    th = np.random.default_rng(1).uniform(0.2, 0.9, size=O.kernel_nparams(ks))
    e = Engine(X, y, mu, ks, 0, 1e-3, False)
    ll, info = e.loglik(th)
    ref, rinfo = O.loglik(ks, th, X, y, mu, 0, 1e-3, False)
    assert info == rinfo == 0
    assert abs(ll - ref) <= 1e-9 * abs(ref), (ll, ref)


@pytest.mark.parametrize("col", [0, 2])  # a plain and a wrapped feature
def test_point_that_is_not_finite(col, lib):
    from fgpu import Engine
    from fgpu._lib import FgpuError
    X, y = _data(80, 9, 5)
    X[40, col] = np.nan
    e = Engine(X, y, np.zeros(80), [O.RBF_CYCLIC, 9, *range(1, 10)], 0, 1e-3, False)
    try:
        ll, info = e.loglik(np.full(9, 0.5))
    except FgpuError:
        return
    assert info > 0 and np.isnan(ll)


def test_squared_distance_beyond_63_bits(lib):
    """192 features at the opposite ends of their scale: the sum of the squares takes
    64 bits."""
    from fgpu import Engine
    d, n = 192, 70
    rng = np.random.default_rng(3)
    X = np.where(np.arange(n)[:, None] % 2, 0.9999, -0.9999) * np.ones((n, d))
    X[:, 2::3] = np.where(np.arange(n)[:, None] % 2, np.pi, 0.0)
    X[:, 0] = rng.uniform(-0.9, 0.9, size=n)
    y = rng.normal(size=n)
    ks = [O.RBF_CYCLIC, d, *range(1, d + 1)]
    for t in (0.0, -0.91, -8.0):  # -0.91: the wrapped differences fill their scale
        th = np.full(d, t)
        ll, info = Engine(X, y, np.zeros(n), ks, 0, 1e-2, False).loglik(th)
        ref, rinfo = O.loglik(ks, th, X, y, np.zeros(n), 0, 1e-2, False)
        assert info == rinfo == 0
        assert abs(ll - ref) <= 1e-9 * abs(ref), (t, ll, ref)


@pytest.mark.parametrize("value", [np.nan, np.inf, 2000.0])
@pytest.mark.parametrize("col", [0, 2])
def test_weight_that_is_not_usable(col, value, lib):
    """A plan takes theta as it is: NaN and weights beyond any scale fail the problem they belong to,
    whichever feature they are of."""
    from fgpu import Engine, Plan
    from fgpu._lib import FgpuError
    X, y = _data(80, 9, 5)
    e = Engine(X, y, np.zeros(80), [O.RBF_CYCLIC, 9, *range(1, 10)], 0, 1e-3, False)
    th = np.full((2, 9), 0.5)
    th[1, col] = value
    try:
        ll, info = Plan([e, e]).run(th)
    except FgpuError:
        return
    assert info[1] > 0 and np.isnan(ll[1])
    assert info[0] == 0 and ll[0] == e.loglik(th[0])[0]


def _exact_loglik(E, nugget):
    """logL at y = mu = 0 from the squared distances E, in extended precision."""
    K = np.exp(-E / 2) + np.eye(len(E), dtype=np.longdouble) * np.longdouble(nugget)
    ld, n = np.longdouble(0), len(E)
    for j in range(n):  # outer-product Cholesky
        ld += np.log(K[j, j])
        K[j + 1:, j + 1:] -= np.outer(K[j + 1:, j], K[j + 1:, j]) / K[j, j]
    return -ld / 2 - np.longdouble(n) / 2 * np.log(2 * np.longdouble(np.pi))


@pytest.mark.parametrize("theta", [0.5, 3.0, 5.5, 8.0])
@pytest.mark.parametrize("wrapped", [False, True])
def test_precision_of_close_points(theta, wrapped, lib):
    """Pairs at E = 1e-4 (K_ij = 1 - 5e-5) among points far apart: log(1 - K_ij^2) shows
    E's absolute error.  Allowed: E to 3e-16 relative and 6e-17 (the weight and the
    units of the distances), K_ij to 2^-53 + 2^-61 (its rounding, and the matrix's),
    over a pair's 1 - K_ij^2 = 1e-4; the conversions' few ulps of logL."""
    from fgpu import Engine
    n, d = 60, 3
    rng = np.random.default_rng(int(10 * theta))
    step = 12.0 / np.sqrt(np.exp(theta))  # one pair from the next
    X = np.zeros((n, d))
    X[:, 0] = 0.3 + (np.arange(n) // 2) * step
    X[:, 2] = 2.0
    col = 2 if wrapped else 1
    if wrapped:
        X[::4, 2] = np.pi - 0.001 * np.arange(len(X[::4]))
    else:
        X[::2, 1] = rng.uniform(-1.5, 1.5, size=n // 2)
    gap = np.sqrt(1e-4 / np.exp(theta))
    X[1::2, col] = X[::2, col] + gap * rng.uniform(0.9, 1.1, size=n // 2)
    ks, th = [O.RBF_CYCLIC, d, 1, 2, 3], np.full(d, theta)
    ld = np.longdouble
    D = X.astype(ld)[:, None] - X.astype(ld)[None]
    C, P = ld(2.0 * np.pi), ld(np.pi)  # the doubles the reference wraps by
    D[..., 2] = np.abs(D[..., 2]) + P
    D[..., 2] = np.fmod(D[..., 2], C) - P
    want = _exact_loglik((np.exp(ld(theta)) * D * D).sum(-1), 0.0)
    ll, info = Engine(X, np.zeros(n), np.zeros(n), ks, 0, 0.0, False).loglik(th)
    tol = n // 2 * ((3e-16 * 1e-4 + 6e-17) / 2 + 2.0 ** -53 + 2.0 ** -61) / 1e-4 / 0.8 + 4 * np.spacing(abs(float(want)))
    assert info == 0
    assert abs(ll - want) <= tol, (ll, float(want), float(abs(ll - want)), tol)


def test_angles_far_beyond_the_integers(lib):
    """Wrapped features around 1e17: their differences are exact, and so is the wrap."""
    from fgpu import Engine
    n = 40
    rng = np.random.default_rng(8)
    X = rng.normal(2.0, 0.3, size=(n, 3))
    X[:, 2] = 1e17 + 16.0 * np.arange(n)
    y = rng.normal(size=n)
    ks, th = [O.RBF_CYCLIC, 3, 1, 2, 3], np.full(3, 0.3)
    ll, info = Engine(X, y, np.zeros(n), ks, 0, 1e-2, False).loglik(th)
    ref, _ = O.loglik(ks, th, X, y, np.zeros(n), 0, 1e-2, False)
    assert info == 0 and abs(ll - ref) <= 1e-9 * abs(ref), (ll, ref)
