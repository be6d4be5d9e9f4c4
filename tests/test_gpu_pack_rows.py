"""GPU: the 16-bit packing with 8 and with 32 rows per warp, on both sides of the
size that separates them (2^20 padded rows), with rows that are not finite: counts
of sampled rows equal to the exact recount's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp16", "bf16_split"])
@pytest.mark.parametrize("n,d", [(1, 3), (31, 70), (33, 64), (1000, 18), (77_700, 12), (1_048_200, 7),
                                 (1_048_577, 6)])
def test_counts(ej, mode, n, d):
    rng = np.random.default_rng(n)
    x = rng.random((n, d))
    x[rng.random(n) < 0.01, d // 2] = np.nan
    eps = 0.5 * (min(n, 1000) / n) ** (1.0 / d)
    rows = np.unique(np.concatenate([rng.integers(0, n, 200), [0, n - 1, n // 32 * 32 % n]])).astype(np.uint64)
    ref = ej.query_counts(x, eps, rows)
    c, t, st = ej.self_join(x, eps, precision=mode)
    assert t == int(c.astype(np.int64).sum()) and np.array_equal(c[rows.astype(np.int64)], ref), st
