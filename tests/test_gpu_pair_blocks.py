"""GPU: the blocks of CTA pairs at their edges -- a lone row or column tile, odd
tile counts, a last tile with one row -- and the epilogue's two ways of counting
a 32 x 32 chunk: rows put down one by one (few hits), bit masks (many hits, up
to every pair), and both in one join.  Counts are whole numbers: equal to the
oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = ["bf16", "bf16_split", "fp16", "fp8_e4m3"]


def radius(q, x, share, rng):
    """The radius that `share` of the sampled pairs lie within."""
    i, j = rng.integers(0, q.shape[0], 6000), rng.integers(0, x.shape[0], 6000)
    return float(np.quantile(np.sqrt(((q[i] - x[j]) ** 2).sum(1)), share))


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n,d", [(127, 64), (129, 64), (257, 65), (385, 128), (2049, 64), (2177, 129),
                                 (4225, 40)])
@pytest.mark.parametrize("share", [0.002, 0.03, 0.4, 1.0])
def test_self_join_edges(ej, oracle_mod, mode, n, d, share):
    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d))
    # clusters of very different density, so that chunks of both kinds meet
    x[: n // 3] *= 0.2
    x[n // 2] = x[n // 2 - 1]
    eps = radius(x, x, share, rng)
    ref, total = oracle_mod.self_join(x, eps)
    counts, tot, st = ej.self_join(x, eps, precision=mode)
    assert tot == total, st
    assert np.array_equal(counts, ref), st


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("nq,n", [(1, 129), (128, 128), (129, 1), (257, 385), (2177, 640), (300, 4353)])
@pytest.mark.parametrize("share", [0.01, 0.6])
def test_cross_edges(ej, oracle_mod, mode, nq, n, share):
    rng = np.random.default_rng(nq + n)
    x, q = rng.standard_normal((n, 72)), rng.standard_normal((nq, 72))
    eps = radius(q, x, share, rng)
    ref = oracle_mod.cross_counts(q, x, eps)
    got, tot, st = ej.join_counts(q, x, eps, precision=mode)
    assert np.array_equal(got, ref), st
    assert tot == int(ref.sum())


@pytest.mark.parametrize("n,k", [(4096, 8), (20_001, 8), (33_333, 3)])
def test_pruned_rows_paired(ej, oracle_mod, n, k):
    # few tile pairs survive, so row tiles that are not neighbours share blocks
    rng = np.random.default_rng(n)
    c = rng.random((60, 8))
    e = np.linalg.qr(rng.standard_normal((48, 8)))[0]
    x = (c[rng.integers(0, 60, n)] + 0.02 * rng.standard_normal((n, 8))) @ e.T
    x += 0.005 * rng.standard_normal(x.shape)
    eps = 0.06
    ref, total = oracle_mod.self_join(x, eps)
    for mode in ("fp16", "bf16_split"):
        counts, tot, st = ej.self_join(x, eps, precision=mode, proj_k=k)
        assert st["tile_pairs_run"] < st["tile_pairs_total"]
        assert st["gram_blocks"] * 2 >= st["tile_pairs_run"]
        assert tot == total and np.array_equal(counts, ref), st


@pytest.mark.parametrize("mode", ["fp16", "bf16_split"])
@pytest.mark.parametrize("n,share", [(129, 0.5), (1300, 0.004), (1300, 0.3)])
def test_lists_from_both_kinds(ej, oracle_mod, mode, n, share):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 64))
    x[: n // 3] *= 0.2
    eps = radius(x, x, share, rng)
    off_ref, nb_ref = oracle_mod.neighbor_lists(x, eps)
    off, nb, _ = ej.neighbor_lists(x, eps, precision=mode)
    assert np.array_equal(off, off_ref) and np.array_equal(nb, nb_ref)
