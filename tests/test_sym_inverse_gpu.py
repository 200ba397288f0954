"""The symmetric sweep inverse against numpy: tile edges, orders past one
tile, indefinite matrices, and matrices whose leading block is (nearly)
singular although they are not, which need Newton steps or the pivoted
elimination."""
import numpy as np
import pytest

from scatt_b200 import _lib

pytestmark = pytest.mark.gpu


def symmetric(rng, count, n):
    """Indefinite, kappa of a few tens: a scaled random symmetric part (norm
    about 0.9) on a diagonal of 2 with every fifth sign turned."""
    M = rng.standard_normal((count, n, n))
    M = (M + np.swapaxes(M, 1, 2)) * (0.9 / (2.0 * np.sqrt(2.0 * n)))
    M[:, np.arange(n), np.arange(n)] += np.where(np.arange(n) % 5 == 0, -2.0, 2.0)
    return M


@pytest.mark.parametrize("n,count", [(1, 3), (2, 1), (17, 5), (63, 2), (64, 2), (65, 3), (100, 20), (127, 1), (128, 2),
                                     (129, 1), (162, 4), (193, 2), (324, 3), (441, 9), (774, 2), (1046, 2), (1314, 1)])
def test_matches_numpy(n, count):
    A = symmetric(np.random.default_rng(n), count, n)
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert np.all(st == 0) and np.all(mode == 0)
    assert np.array_equal(X, np.swapaxes(X, 1, 2))
    for a, x in zip(A, X):
        ref = np.linalg.inv(a)
        # kappa <= 2.9 / 1.1 up to the random part's spread: rounding of n-term sums, with room for growth below 10
        assert np.max(np.abs(x - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_pivots_inside_a_tile():
    n = 64
    A = np.zeros((1, n, n))
    i = np.arange(0, n, 2)
    A[0, i, i + 1] = A[0, i + 1, i] = 1.0 + i / n          # zero diagonal: 2 x 2 pivots only
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert st[0, 0] == 0 and mode[0] == 0
    assert np.max(np.abs(X[0] @ A[0] - np.eye(n))) <= 1e-15


@pytest.mark.parametrize("n", [128, 200, 450])
@pytest.mark.parametrize("delta,want", [(0.02, 1), (2e-3, 1), (1e-5, 2), (0.0, 3)])
def test_nearly_singular_leading_block(n, delta, want):
    """[[delta I, I], [I, A22]] on the first two tiles: |D| of the first pivot
    tile is 1 / delta, |X| about 2.  The sweep's error is delta^-2 eps (up to
    6e-11 and 2e-6); one Newton step, or two, square it away, leaving
    rounding; delta = 0 leaves no first pivot at all."""
    rng = np.random.default_rng(5)
    A = symmetric(rng, 2, n)
    A[1, :64, :64] = delta * np.eye(64)
    A[1, :64, 64:128] = A[1, 64:128, :64] = np.eye(64)
    A[1, :64, 128:] = A[1, 128:, :64] = 0.0
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert np.all(st[:, 0] == 0) and mode[0] == 0 and mode[1] == want
    for a, x in zip(A, X):
        ref = np.linalg.inv(a)
        kappa = np.linalg.cond(a)
        assert np.max(np.abs(x - ref)) <= 1e-13 * max(10.0, kappa) * np.max(np.abs(ref))
        assert np.array_equal(x, x.T)


def test_singular_and_nonfinite_are_reported():
    A = symmetric(np.random.default_rng(1), 3, 100)
    A[0, 70, :] = A[0, :, 70] = 0.0
    A[2, 5, 5] = np.nan
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert st[0, 0] == 1 and st[1, 0] == 0 and st[2, 0] == 2
    ref = np.linalg.inv(A[1])
    assert np.max(np.abs(X[1] - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_statuses_of_a_long_batch():
    """More matrices than one pass of the rescue looks at (256): slow pivoted
    eliminations in the first pass, failing matrices in both."""
    n, count = 200, 600
    A = np.repeat(symmetric(np.random.default_rng(3), 1, n), count, axis=0)
    rescued = [0, 148, 255, 300]                    # leading block zero, as in the test above: regular
    for b in rescued:
        A[b, :64, :64] = 0.0
        A[b, :64, 64:128] = A[b, 64:128, :64] = np.eye(64)
        A[b, :64, 128:] = A[b, 128:, :64] = 0.0
    singular, bad = [3, 149, 256, 297, 440, 599], [5, 254, 258, 400, 513]
    for b in singular:
        A[b, 70, :] = A[b, :, 70] = 0.0
    for b in bad:
        A[b, 5, 5] = np.nan
    want = np.zeros(count, dtype=int)
    want[singular], want[bad] = 1, 2
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert np.array_equal(st[:, 0], want)
    assert np.all(mode[rescued + singular + bad] == 3) and np.count_nonzero(mode) == len(rescued + singular + bad)
    good = np.linalg.inv(A[1])
    for b in range(count):
        if want[b] == 0 and b not in rescued:
            assert np.max(np.abs(X[b] - good)) <= 1e-12 * np.max(np.abs(good))
    for b in rescued:
        ref = np.linalg.inv(A[b])
        assert np.max(np.abs(X[b] - ref)) <= 1e-13 * max(10.0, np.linalg.cond(A[b])) * np.max(np.abs(ref))


def _solutions(A, X, b):
    """A^-1 b to 64-bit rounding: a few refinements with extended residuals."""
    Al, x = A.astype(np.longdouble), (X @ b).astype(np.longdouble)
    for _ in range(5):
        x = x + X @ (b - Al @ x).astype(np.float64)
    return x.astype(np.float64)


@pytest.mark.parametrize("n", [130, 196, 452, 1046])
@pytest.mark.parametrize("kind", ["one", "four", "graded"])
def test_dominant_directions(n, kind):
    """A part of norm c, which every tile has a share of, beside the family
    above: the pivot tiles' condition grows with c without any growth of the
    intermediate inverses.  The error is held to ten times the general
    inverse's (whose pivots run down the whole matrix); a sweep that takes D
    at its word loses log10(c) digits more, 1e3 times that bound at c = 1e6."""
    cs = [1.0, 1e1, 1e2, 1e3, 1e4, 1e5, 1e6]
    rng = np.random.default_rng(n)
    B = symmetric(rng, 1, n)[0]
    v = rng.standard_normal((n, 4 if kind == "four" else 1))
    if kind == "graded":
        v *= 10.0 ** (-2.0 * np.arange(n) / n)[:, None]
    sign = np.array([1.0, -1.0, 1.0, -1.0])[: v.shape[1]]
    A = np.stack([B + c / n * (v * sign) @ v.T for c in cs])
    A = 0.5 * (A + np.swapaxes(A, 1, 2))
    X, st, _ = _lib.inverse_symmetric_batched(A)
    G, _ = _lib.inverse_batched(A, symmetrize=True)
    assert np.all(st == 0)
    b = rng.standard_normal((n, 4))
    for a, x, g, c in zip(A, X, G, cs):
        t = _solutions(a, np.linalg.inv(a), b)
        err = lambda y: np.linalg.norm(y @ b - t) / np.linalg.norm(t)  # noqa: E731
        # the floor: rounding of the products X b themselves
        assert err(x) <= 10.0 * err(g) + 1e-15, (c, err(x), err(g))


@pytest.mark.parametrize("n", [256, 300])
@pytest.mark.parametrize("delta,want", [(1e-2, 1), (1e-4, 2), (1e-6, 2)])
def test_growth_in_one_block_only(n, delta, want):
    """The nearly singular leading block beside uncoupled blocks delta I and
    I / delta: these hold the largest element of A and of its inverse, so that
    only a record per tile row sees the first block's growth.  Its own part of
    the inverse is held to rounding (the sweep alone leaves eps / delta)."""
    rng = np.random.default_rng(9)
    A = np.zeros((1, n, n))
    A[0, :128, :128] = symmetric(rng, 1, 128)[0]
    A[0, :64, :64] = delta * np.diag(1.0 + rng.random(64))
    A[0, :64, 64:128] = np.linalg.qr(rng.standard_normal((64, 64)))[0]
    A[0, 64:128, :64] = A[0, :64, 64:128].T
    i = np.arange(128, n)
    A[0, i, i] = np.where(i < 192, delta, 1.0 / delta)
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert st[0, 0] == 0 and mode[0] == want
    ref = np.linalg.inv(A[0, :128, :128])
    kappa = np.linalg.cond(A[0, :128, :128])
    assert np.max(np.abs(X[0, :128, :128] - ref)) <= 1e-13 * max(10.0, kappa) * np.max(np.abs(ref))
    assert np.max(np.abs(X[0, i, i] * A[0, i, i] - 1.0)) <= 1e-14


@pytest.mark.parametrize("lam", [1e-6, 1e-8, 1e-9, 1e-10, 1e-11])
def test_newton_steps_that_do_not_converge(lam):
    """A nearly singular leading block (growth 2e5) in a matrix of condition
    about 5 / lam: past 1e9 the Newton steps run away, and the entry has to end
    in the pivoted elimination.  Held to ten times what rounding of A does to
    the inverse, kappa eps."""
    n = 200
    rng = np.random.default_rng(5)
    A = symmetric(rng, 1, n)
    A[0, :64, :64] = 2e-6 * np.eye(64)
    A[0, :64, 64:128] = A[0, 64:128, :64] = np.eye(64)
    A[0, :64, 128:] = A[0, 128:, :64] = 0.0
    A[0, 64:128, 128:] = 0.5 / 8.0 * rng.standard_normal((64, n - 128))
    A[0, 128:, 64:128] = A[0, 64:128, 128:].T
    v = np.zeros(n)
    v[128:] = rng.standard_normal(n - 128)
    v /= np.linalg.norm(v)
    # A + t v v^T is singular at t = -1 / (v^T A^-1 v)
    A[0] -= (1.0 + lam) / (v @ np.linalg.solve(A[0], v)) * np.outer(v, v)
    A[0] = 0.5 * (A[0] + A[0].T)
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert st[0, 0] == 0
    b = rng.standard_normal((n, 4))
    t = _solutions(A[0], np.linalg.inv(A[0]), b)
    kappa = np.linalg.cond(A[0])
    assert np.linalg.norm(X[0] @ b - t) <= 10.0 * kappa * 2.2e-16 * np.linalg.norm(t), (mode[0], kappa)


@pytest.mark.parametrize("n", [1, 64, 200])
def test_reciprocals_of_pivots(n):
    """Diagonal matrices: the inverse is the pivots' reciprocals, to half an
    ulp (and the 2^-27 of one that the Newton steps leave)."""
    rng = np.random.default_rng(n)
    d = np.ldexp(1.0 + rng.random((40, n)), rng.integers(-4, 5, size=(40, n)) + rng.integers(-900, 900, size=(40, 1)))
    d *= np.where(rng.random((40, n)) < 0.5, -1.0, 1.0)
    A = np.zeros((40, n, n))
    i = np.arange(n)
    A[:, i, i] = d
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert np.all(st == 0) and np.all(mode == 0)
    y = X[:, i, i].astype(np.longdouble)
    assert np.max(np.abs(y * d.astype(np.longdouble) - 1)) <= np.longdouble(2.0) ** -53 * (1 + 2.0 ** -9)
    assert np.count_nonzero(X) == d.size


@pytest.mark.parametrize("value", [2.0 ** -1023, 1.5 * 2.0 ** -1023, 2.0 ** 1022, 1.25 * 2.0 ** 1022, 1.7 * 2.0 ** 1023])
@pytest.mark.parametrize("at", [0, 40, 120])
def test_pivots_outside_the_reciprocal(value, at):
    A = np.eye(130)[None].copy()
    A[0, at, at] = value
    X, st, _ = _lib.inverse_symmetric_batched(A)
    assert st[0, 0] == 0
    want = np.eye(130)
    want[at, at] = 1.0 / value                      # a subnormal number for the last two
    assert np.all(np.abs(X[0] - want) <= np.where(want == 1.0 / value, np.spacing(want), 0.0))


def test_rescued_entries_share_their_scratch():
    """One, two and no Newton steps and eliminations side by side in a batch."""
    n, want = 200, [1, 2, 0, 1, 3, 2, 1, 0, 2, 3]
    A = symmetric(np.random.default_rng(21), len(want), n)
    for a, m in zip(A, want):
        if m:
            a[:64, :64] = {1: 2e-3, 2: 1e-5, 3: 0.0}[m] * np.eye(64)
            a[:64, 64:128] = a[64:128, :64] = np.eye(64)
            a[:64, 128:] = a[128:, :64] = 0.0
    X, st, mode = _lib.inverse_symmetric_batched(A)
    assert np.all(st == 0) and np.array_equal(mode, want)
    for a, x in zip(A, X):
        ref = np.linalg.inv(a)
        assert np.max(np.abs(x - ref)) <= 1e-13 * max(10.0, np.linalg.cond(a)) * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [2049, 5317, 8192])
def test_large_orders(n):
    """Up to the largest order accepted, by the residual on a few vectors
    (kappa as in the family above: rounding of n-term sums)."""
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    M += M.T.copy()
    M *= 0.9 / (2.0 * np.sqrt(2.0 * n))
    i = np.arange(n)
    M[i, i] += np.where(i % 5 == 0, -2.0, 2.0)
    X, st, mode = _lib.inverse_symmetric_batched(M[None])
    assert st[0, 0] == 0 and mode[0] == 0
    x = rng.standard_normal((n, 3))
    assert np.linalg.norm(X[0] @ (M @ x) - x) <= 1e-13 * np.linalg.norm(x)
    assert np.linalg.norm(X[0].T @ x - X[0] @ x) <= 1e-14 * np.linalg.norm(X[0] @ x)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("at", [(0, 0), (70, 3), (99, 99)])
def test_nonfinite_elements(value, at):
    A = symmetric(np.random.default_rng(2), 3, 100)
    A[1, at[0], at[1]] = A[1, at[1], at[0]] = value
    X, st, _ = _lib.inverse_symmetric_batched(A)
    assert list(st[:, 0]) == [0, 2, 0]
    for b in (0, 2):
        ref = np.linalg.inv(A[b])
        assert np.max(np.abs(X[b] - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_orders_and_batches_refused():
    with pytest.raises(_lib.ScattError):
        _lib.inverse_symmetric_batched(np.zeros((1, 8193, 8193)))
