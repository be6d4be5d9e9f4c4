"""GPU: single rows whose squared norm exceeds the FP64 range, among ordinary ones.  The
products of such a row with others may overflow to +inf as well."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = ["fp64_direct", "fp64_dmma", "bf16_split", "fp16", "fp8_e4m3"]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("scale", [1.0, 1e9, -1e12])
@pytest.mark.parametrize("big", [1e300, -1e300, 1e155])
def test_outlying_rows(ej, oracle_mod, mode, scale, big):
    rng = np.random.default_rng(3)
    x = scale * (1.0 + rng.random((300, 20)))
    x[7, 3] = x[150, 3] = x[299, 19] = big
    x[151] = x[150]
    eps = 0.8 * abs(scale)
    ref, total = oracle_mod.self_join(x, eps)
    counts, got, st = ej.self_join(x, eps, precision=mode)
    assert got == total and np.array_equal(counts, ref), st
    off_ref, nb_ref = oracle_mod.neighbor_lists(x, eps)
    off, nb, _ = ej.neighbor_lists(x, eps, precision=mode)
    assert np.array_equal(off, off_ref) and np.array_equal(nb, nb_ref)
    got, _, _ = ej.join_counts(x[::3].copy(), x, eps, precision=mode)
    assert np.array_equal(got, oracle_mod.cross_counts(x[::3].copy(), x, eps))
