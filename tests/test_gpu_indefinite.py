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


def _star(m, r2, pos, n, scale):
    """n points in m dimensions: m of them at right angles, each at squared distance
    ``r2`` from one more, whose row is ``pos``; the others far from everything.
    Row ``pos`` alone is what the leading minors fail at, if they do."""
    d = max(m, 3)
    X = np.zeros((n, d))
    X[:, :3] = _grid(n, 14.0) + 60.0
    rows = [q for q in scale if q < pos]
    X[pos] = 0.0
    for k in range(m):
        X[rows[k]] = 0.0
        X[rows[k], k] = np.sqrt(r2)
    return X


# the star's centre in the first 16 columns, in the first panel, and in a later one
# with its neighbours in one panel or spread over two
LAYOUTS = {"block": (15, 40, range(15)), "panel": (120, 130, range(3, 120, 3)), "next": (200, 260, range(2, 128, 3)),
           "spread": (300, 330, range(1, 300, 7)), "far": (700, 720, range(5, 700, 17))}


def _cases(layout):
    for r2 in (4.0, 4.6) if layout == "far" else (2.5, 4.0, 4.6, 5.5):
        for nugget in (-0.9, -0.93) if layout == "far" else (-0.76, -0.8, -0.9, -0.93, -0.96):
            yield r2, nugget


@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("m", [2, 4, 6, 8, 10, 12, 14, 16, 20, 24, 32])
def test_row_beyond_its_diagonal(layout, m, lib):
    """A row whose factor entries' squares add up beyond K_ii, to several times the
    fixed point's range: each entry alone may be unremarkable."""
    from fgpu import Engine, loglik_batch
    pos, n, rows = LAYOUTS[layout]
    if m > len(rows):
        pytest.skip("more neighbours than rows")
    ks = [O.RBF, max(m, 3), *range(1, max(m, 3) + 1)]
    th = np.zeros(max(m, 3))
    y = np.random.default_rng(m).normal(size=n)
    es, want = [], []
    for r2, nugget in _cases(layout):
        X = _star(m, r2, pos, n, rows)
        ll, info = O.loglik(ks, th, X, y, np.zeros(n), 0, nugget, False)
        e = Engine(X, y, np.zeros(n), ks, 0, nugget, False)
        got, ginfo = e.loglik(th)
        assert ginfo == info, (r2, nugget, info, ginfo, got)
        if info == 0:
            assert abs(got - ll) <= 1e-9 * abs(ll), (r2, nugget, got, ll)
        es.append(e)
        want.append((got, info))
    assert any(info for _, info in want)
    reps = 10 if layout == "far" else 1  # as many row tiles as take the split panels
    lb, ib = loglik_batch(es * reps, [th] * (len(es) * reps))
    for k, (got, info) in enumerate(want * reps):
        assert ib[k] == info
        assert lb[k] == got or (info and np.isnan(lb[k]))


@pytest.mark.parametrize("nugget", [1e200, 1e299, 1e301, 1.5e308])
@pytest.mark.parametrize("n", [20, 150])
def test_huge_diagonal(nugget, n, lib):
    """The scale follows K_ii through the whole range of doubles; an infinite K_ii fails."""
    from fgpu import Engine
    from fgpu._lib import FgpuError
    rng = np.random.default_rng(3)
    X, y = rng.normal(size=(n, 3)), rng.normal(size=n)
    ks, th = [O.RBF, 3, 1, 2, 3], np.zeros(3)
    ref, _ = O.loglik(ks, th, X, y, np.zeros(n), 0, nugget, False)
    ll, info = Engine(X, y, np.zeros(n), ks, 0, nugget, False).loglik(th)
    assert info == 0
    assert abs(ll - ref) <= 1e-9 * abs(ref), (ll, ref)
    try:
        ll, info = Engine(X, y, np.zeros(n), ks, 0, np.inf, False).loglik(th)
    except FgpuError:
        return
    assert info > 0 and np.isnan(ll)
