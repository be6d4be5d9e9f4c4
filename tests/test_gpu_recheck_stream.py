"""GPU: the FP8 join's recheck streamed through per-warp queues, at
the row lengths where its variants begin and end: all pairs of a row, single
pairs, rows shorter than the lanes' share.  Counts equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [257, 264, 504, 512, 513, 760, 1023, 1024])
@pytest.mark.parametrize("share", [0.02, 1.0])
def test_lattice_rows(ej, oracle_mod, d, share):
    rng = np.random.default_rng(d)
    n, k = 700, 12
    x = np.zeros((n, d))
    x[:, rng.permutation(d)[:k]] = rng.integers(0, 2, (n, k))
    # the others lie too far out for a band with anything but themselves
    far = rng.random(n) >= share
    x[far, rng.integers(0, d, int(far.sum()))] += 64.0 * (1 + np.arange(int(far.sum())))
    eps = 2.0
    ref, total = oracle_mod.self_join(x, eps)
    c, t, st = ej.self_join(x, eps, precision="fp8_e4m3")
    assert t == total and np.array_equal(c, ref), st
    q = x[rng.permutation(n)[:130]]
    got, _, _ = ej.join_counts(q, x, eps, precision="fp8_e4m3")
    assert np.array_equal(got, oracle_mod.cross_counts(q, x, eps))
