"""GPU: the FP64 arbiter drops pairs by their partial sums.  Its counts equal the
oracle's whatever share of a tile's pairs drops out and when: none, all at the
first coordinates, only at the last, around the list's size; at ties, with
non-finite values, and at the extremes of the radius."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(ej, oracle_mod, x, eps, rows):
    ref, total = oracle_mod.self_join(x, eps)
    c, t, _ = ej.self_join(x, eps, precision="fp64_direct")
    assert t == total and np.array_equal(c, ref)
    assert np.array_equal(ej.query_counts(x, eps, rows), ref[rows])
    off_ref, nb_ref = oracle_mod.neighbor_lists(x, eps)
    off, nb, _ = ej.neighbor_lists(x, eps, precision="fp64_direct")
    assert np.array_equal(off, off_ref) and np.array_equal(nb, nb_ref)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 200, 700])
@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 15, 16, 17, 33, 100])
@pytest.mark.parametrize("share", [0.0, 0.004, 0.2, 0.26, 0.7, 1.0])
def test_shares(ej, oracle_mod, n, d, share):
    rng = np.random.default_rng(n * 131 + d)
    c = 3.0 * rng.random((5, d))
    x = c[rng.integers(0, 5, n)] + 0.3 * rng.standard_normal((n, d))
    i, j = rng.integers(0, n, 4000), rng.integers(0, n, 4000)
    eps = float(np.quantile(np.sqrt(((x[i] - x[j]) ** 2).sum(1)), share))
    check(ej, oracle_mod, x, eps, np.unique(rng.integers(0, n, 70)))


@pytest.mark.parametrize("d", [3, 20, 64])
@pytest.mark.parametrize("last", [False, True])
def test_where_the_distance_comes_from(ej, oracle_mod, d, last):
    # the coordinates that tell points apart come first, or last
    rng = np.random.default_rng(d)
    scale = np.geomspace(1.0, 1e-3, d)
    x = rng.standard_normal((500, d)) * (scale[::-1] if last else scale)
    for eps in (0.0, 0.05, 0.5, 2.0):
        check(ej, oracle_mod, x, eps, np.arange(0, 500, 7))


def test_ties_and_special_values(ej, oracle_mod):
    rng = np.random.default_rng(9)
    x = rng.integers(-2, 3, (400, 9)) / 8.0  # many d2 exactly eps^2
    x[5] = x[9]
    for eps in (0.125, 0.25, float(np.sqrt(0.125)), 0.5):
        check(ej, oracle_mod, x, eps, np.arange(400))
    y = rng.standard_normal((300, 21))
    y[3, 0], y[4, 20], y[5, 7], y[6, 0] = np.nan, np.nan, np.inf, -np.inf
    y[7] = np.inf
    y[8, 20] = 1e200
    y[9, 0] = -1e200
    for eps in (1.0, 1e150, 1e300, np.inf):
        ref, total = oracle_mod.self_join(y, eps)
        c, t, _ = ej.self_join(y, eps, precision="fp64_direct")
        assert t == total and np.array_equal(c, ref)
    z = y[20:120] * 1e-160  # squares underflow
    for eps in (0.0, 1e-161, 1e-159):
        check(ej, oracle_mod, z, eps, np.arange(50))
