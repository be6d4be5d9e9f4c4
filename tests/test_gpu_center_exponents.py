"""GPU: the centring pass at the exponents where its ways of splitting a coordinate
meet (2^-126, 2^-74, and both signs of each), beside zeros and ordinary values:
counts equal to the oracle's at radii that are distances of the data, for an even
and an odd dimension."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp16", "bf16_split", "fp8_e4m3"])
@pytest.mark.parametrize("d", [9, 16])
def test_exponents(ej, oracle_mod, mode, d):
    rng = np.random.default_rng(d)
    n = 600
    x = rng.integers(-8, 9, (n, d)) / 8.0  # exact distances, many ties
    tiny = np.array([0.0, 2.0 ** -74, 2.0 ** -75, 2.0 ** -73, 2.0 ** -126, 2.0 ** -127, 2.0 ** -1074, 2.0 ** -51])
    for c in range(d // 2):
        x[:, c] = rng.choice(np.concatenate([tiny, -tiny]), n) * (1.0 + rng.integers(0, 2, n) * 2.0 ** -30)
    x[:, -1] += rng.integers(0, 2, n) * 2.0 ** -40  # beyond 24 bits
    for t in (0, 1):
        i, j = rng.integers(0, n, 2)
        eps = float(np.sqrt(((x[i] - x[j]) ** 2).sum())) * 0.7 ** t
        ref, total = oracle_mod.self_join(x, eps)
        c, tot, st = ej.self_join(x, eps, precision=mode)
        assert tot == total and np.array_equal(c, ref), st
