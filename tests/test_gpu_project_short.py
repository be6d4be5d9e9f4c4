"""GPU: the projection of rows of at most 64 coordinates at the edges of its tiles
(128 rows) and of its copies (rows a multiple of four long or not), with many
tiles per block: pruned counts against the unpruned join's, for points whose
distances are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,d", [(1, 4), (8, 60), (8, 62), (8, 64), (9, 8), (16, 64)])
@pytest.mark.parametrize("n", [1, 127, 129, 4000, 130_003])
def test_pruned_counts(ej, k, d, n):
    rng = np.random.default_rng(100 * k + d + n)
    groups = max(1, n // 40)
    x = rng.integers(-500, 500, (groups, d))[rng.integers(0, groups, n)] + rng.integers(-1, 2, (n, d))
    x = x.astype(np.float64)
    eps = float(np.sqrt(np.floor(4.0 * d / 3.0) + 0.5))
    P = (rng.standard_normal((k, d)) / (3 * np.sqrt(d))).astype(np.float32)
    base, total, _ = ej.self_join(x, eps, proj_k=0)
    for order in (0, 1):
        got, t, st = ej.self_join(x, eps, proj_k=k, projection=P, order=order)
        assert np.array_equal(got, base) and t == total, st
