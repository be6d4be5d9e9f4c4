"""GPU: the screens that size their queues themselves, made to size them too small: the
screen runs again after a band overflow, the whole join after an overflow of the emitted
in-records, and the results are the same (short joins, whose queues come from the number
of pairs, and long ones, sized by a sample; with and without a learned order)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = ["bf16_split", "bf16", "fp16", "fp8_e4m3"]
FITS = 0xffffffff


def clusters(n, d, rng):
    """Groups with certain neighbours and, on a lattice of steps, pairs at the radius."""
    c = rng.integers(0, 2, (24, d)).astype(np.float64) * 8.0
    x = c[rng.integers(0, 24, n)] + 0.02 * rng.standard_normal((n, d))
    x[: n // 4] = c[0] + rng.integers(0, 2, (n // 4, d)) * (np.arange(d) < 10)
    return x[rng.permutation(n)]


@pytest.fixture(scope="module")
def short(oracle_mod):
    x = clusters(3000, 40, np.random.default_rng(1))
    return x, 2.0, oracle_mod.neighbor_lists(x, 2.0)


@pytest.fixture(scope="module")
def long(oracle_mod):
    x = clusters(20_000, 40, np.random.default_rng(2))
    return x, 2.0, oracle_mod.neighbor_lists(x, 2.0)


def lists(ej, x, eps, mode, k, total):
    """One call with buffers of the right size."""
    lib = ej.load_library()
    o = ej._options(precision=mode, proj_k=k)
    off = np.zeros(x.shape[0] + 1, dtype=np.uint64)
    nb = np.zeros(total, dtype=np.uint32)
    t, st = ctypes.c_uint64(0), ej.Stats()
    rc = lib.ejoin_neighbor_lists(x.ctypes.data, x.shape[0], x.shape[1], eps, ctypes.byref(o),
                                  off.ctypes.data, nb.ctypes.data, total, ctypes.byref(t),
                                  ctypes.byref(st))
    assert rc == 0
    return off, nb, st.as_dict()


@pytest.mark.parametrize("k", [0, 8])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("size", ["short", "long"])
def test_repeats(ej, request, size, mode, k):
    x, eps, (off_ref, nb_ref) = request.getfixturevalue(size)
    total = int(off_ref[-1])

    def call(band, emitted):
        if band < FITS or emitted < FITS:
            ej.testing_inject(ej.TESTING_FIRST_QUEUES, (band << 32) | emitted)
        off, nb, st = lists(ej, x, eps, mode, k, total)
        assert np.array_equal(off, off_ref) and np.array_equal(nb, nb_ref), st
        return st

    one = call(FITS, FITS)
    assert one["band_overflows"] == 0 and one["band_records"] > 1024
    band = call(1024, FITS)        # the screen twice
    emitted = call(FITS, 1024)     # the join twice
    both = call(64, 64)
    assert band["band_overflows"] >= 1 and emitted["band_overflows"] == 0
    assert both["band_overflows"] >= 1
    assert emitted["kernel_launches"] > band["kernel_launches"] > one["kernel_launches"]
    assert both["kernel_launches"] > emitted["kernel_launches"]
    # (the repeat of a join with a learned order trains nothing again)
    assert emitted["kernel_launches"] - one["kernel_launches"] < 40

    ej.testing_inject(ej.TESTING_FIRST_QUEUES, (1024 << 32) | FITS)
    counts, got, st = ej.self_join(x, eps, precision=mode, proj_k=k)
    assert st["band_overflows"] >= 1 and got == total
    assert np.array_equal(counts, np.diff(off_ref.astype(np.int64)))


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("nq,n", [(700, 3000), (6000, 20_000)])
def test_repeats_of_two_sets(ej, oracle_mod, mode, nq, n):
    rng = np.random.default_rng(n)
    x = clusters(n, 40, rng)
    q = x[rng.permutation(n)[:nq]].copy()
    ref = oracle_mod.cross_counts(q, x, 2.0)
    ej.testing_inject(ej.TESTING_FIRST_QUEUES, (1024 << 32) | FITS)
    counts, total, st = ej.join_counts(q, x, 2.0, precision=mode)
    assert st["band_overflows"] >= 1
    assert np.array_equal(counts, ref) and total == ref.sum()
