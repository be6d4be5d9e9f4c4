"""GPU: first size of the band queue of long joins whose band sits where a sample of
the blocks sees little of it.  (A queue that is too small costs a second screen.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def far_points(rng, n, d):
    """Uniform in a cube so large that no two lie within 2 of one another."""
    return 100.0 * rng.random((n, d))


def lattice_counts(x, bits, radius2):
    """Neighbours of 0/1 rows: Hamming distance at most radius2."""
    from itertools import combinations

    v = x[:, :bits].astype(np.int64) @ (1 << np.arange(bits))
    hist = np.bincount(v, minlength=1 << bits)
    out = np.zeros(v.size, dtype=np.int64)
    for r in range(radius2 + 1):
        for c in combinations(range(bits), r):
            out += hist[v ^ sum(1 << b for b in c)]
    return out


@pytest.mark.parametrize("mode", ["fp16", "bf16_split"])
def test_one_dense_cluster_of_a_long_file(ej, mode):
    # 10,240 of 300,032 points, one after the other, carry the whole band (1.6 M
    # records, in 820 of 687,378 blocks)
    rng = np.random.default_rng(1)
    x = far_points(rng, 300_032, 16)
    lo, m = 116 * 256, 10_240
    lat = np.zeros((m, 16))
    lat[:, :12] = rng.integers(0, 2, (m, 12))
    x[lo: lo + m] = 200.0 + lat
    ref = np.ones(300_032, dtype=np.int64)
    ref[lo: lo + m] = lattice_counts(lat, 12, 4)
    counts, total, st = ej.self_join(x, 2.0, precision=mode)
    assert total == ref.sum() and np.array_equal(counts, ref), st
    assert 1_000_000 < st["band_records"] < 1 << 22
    assert st["band_overflows"] == 0, st


@pytest.mark.parametrize("mode", ["fp16", "bf16_split"])
def test_far_points_at_every_eighth_block(ej, mode):
    # batches of 2,048 points, the first 256 of each far from everything: the blocks of
    # every eighth column pair hold no band, the others 9 M records
    rng = np.random.default_rng(2)
    n, bits = 150_016, 20
    x = far_points(rng, n, bits)
    keep = np.arange(n) % 2048 >= 256
    lat = rng.integers(0, 2, (n, bits)).astype(np.float64)
    x[keep] = 200.0 + lat[keep]
    ref = np.ones(n, dtype=np.int64)
    ref[keep] = lattice_counts(lat[keep], bits, 3)
    counts, total, st = ej.self_join(x, float(np.sqrt(3.0)), precision=mode)
    assert total == ref.sum() and np.array_equal(counts, ref), st
    assert st["band_records"] > 9_000_000
    assert st["band_overflows"] == 0, st
