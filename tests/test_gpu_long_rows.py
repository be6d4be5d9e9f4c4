"""GPU: rows longer than a launch's y and z dimensions reach (65,535 groups of the
centring sample's 64 columns)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp16", "bf16", "bf16_split", "fp64_dmma"])
def test_rows_of_four_million_coordinates(ej, oracle_mod, mode):
    d = 65_535 * 64 + 1
    x = np.random.default_rng(1).standard_normal((5, d))
    x[3] = x[2]
    x[3, d - 1] += 1.0  # on the radius, by the last coordinate alone
    x[4] = x[2]
    x[4, d - 1] += 1.5
    ref, total = oracle_mod.self_join(x, 1.0)
    counts, got, st = ej.self_join(x, 1.0, precision=mode)
    assert got == total and np.array_equal(counts, ref), st
    assert ref.tolist() == [1, 1, 2, 3, 2]
