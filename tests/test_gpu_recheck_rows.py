"""GPU: the band recheck at every row length where its kernel or its loads change
(a thread, eight lanes or a warp per pair; rows padded to eight coordinates), on
lattices whose distances often equal the radius, so that the band is large and
the exact chain decides many pairs.  Counts equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp16", "bf16_split", "fp8_e4m3"])
@pytest.mark.parametrize("d", [1, 7, 8, 9, 55, 56, 57, 63, 64, 65, 127, 130, 200, 255, 256, 257, 264, 512, 1000])
def test_lattice(ej, oracle_mod, mode, d):
    rng = np.random.default_rng(d)
    n = 900
    x = np.zeros((n, d))
    k = min(d, 12)
    x[:, rng.permutation(d)[:k]] = rng.integers(0, 2, (n, k))
    x += rng.standard_normal(d)  # an offset: centring rounds, differences do not
    x[:, :] = np.round(x * 1024) / 1024
    eps = float(np.sqrt(max(1, k // 3)))
    ref, total = oracle_mod.self_join(x, eps)
    c, t, st = ej.self_join(x, eps, precision=mode)
    assert t == total and np.array_equal(c, ref), st
    assert st["band_pairs"] > 0 and st["exact_rechecks"] > 0
    q = x[rng.permutation(n)[:130]]
    got, _, _ = ej.join_counts(q, x, eps, precision=mode)
    assert np.array_equal(got, oracle_mod.cross_counts(q, x, eps))
