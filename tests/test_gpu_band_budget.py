"""GPU: a band queue that has to grow where device memory allows little more than the
band needs (the limit is a hook's: no memory is filled)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENOMEM = -3


@pytest.mark.parametrize("mode", ["fp16", "bf16_split"])
def test_queue_grows_into_what_memory_allows(ej, oracle_mod, mode):
    # a lattice: 6 M records of several pairs each, 24 M pairs at the radius
    x = np.random.default_rng(5).integers(0, 2, (20_000, 12)).astype(np.float64)
    ref, _ = oracle_mod.self_join(x, 2.0)
    counts, total, st = ej.self_join(x, 2.0, precision=mode)
    assert np.array_equal(counts, ref)
    records = st["band_records"]
    assert st["band_pairs"] > 2 * records > 8_000_000
    try:
        # 17/16 of the records and a warp's padding fit, 5/4 of them do not
        ej.testing_inject(ej.TESTING_BAND_BUDGET, int(2 * 1.17 * records))
        counts, total, st = ej.self_join(x, 2.0, precision=mode, band_capacity=1024)
        assert np.array_equal(counts, ref) and st["band_overflows"] >= 1
        ej.testing_inject(ej.TESTING_BAND_BUDGET, int(2 * 0.9 * records))
        with pytest.raises(ej.EjoinError) as e:
            ej.self_join(x, 2.0, precision=mode, band_capacity=1024)
        assert e.value.status == ENOMEM
    finally:
        ej.testing_inject(ej.TESTING_BAND_BUDGET, 0)
    counts, total, st = ej.self_join(x, 2.0, precision=mode, band_capacity=1024)
    assert np.array_equal(counts, ref)
