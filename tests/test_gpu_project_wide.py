"""GPU: the projection of rows longer than 64 coordinates, at the edges of its
tiles (256 rows x 64 coordinates), of its weights in shared memory and of the
alignment it needs: pruned counts against distances computed in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,d", [(1, 68), (8, 66), (8, 128), (8, 132), (9, 192), (16, 1020), (16, 1344), (16, 1348),
                                 (8, 2688), (8, 2692)])
@pytest.mark.parametrize("n", [1, 255, 257, 1409])
def test_pruned_counts(ej, k, d, n):
    rng = np.random.default_rng(1000 * k + d + n)
    # integer grid points in well-separated groups: every squared distance is an
    # exact integer, and eps^2 lies half-way between two of them
    groups = max(1, n // 40)
    x = 64.0 * rng.integers(0, 4, (groups, d))[rng.integers(0, groups, n)] + rng.integers(-1, 2, (n, d))
    eps = np.sqrt(np.floor(4.0 * d / 3.0) + 0.5)
    P = (rng.standard_normal((k, d)) / np.sqrt(d)).astype(np.float32)
    g = (x * x).sum(1)
    d2 = g[:, None] + g[None, :] - 2.0 * (x @ x.T)
    want = (d2 <= eps * eps).sum(1)
    for order in (0, 1):
        got, total, _ = ej.self_join(x, eps, proj_k=k, projection=P, order=order)
        assert np.array_equal(got.astype(np.int64), want) and total == int(want.sum())
