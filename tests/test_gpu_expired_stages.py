"""GPU: bounded waits that expire in the middle of a block, at every place of the slab
loop of the Gram kernel's issuing warp (the first slab's wait is covered by
test_gpu_failures.py).  The producer withholds one stage; every role gives up, the call
returns EJOIN_ETIMEOUT and the next one is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ETIMEOUT = -6


@pytest.fixture(scope="module")
def case(oracle_mod):
    rng = np.random.default_rng(17)
    x = rng.standard_normal((6000, 250))
    x[3000:] = x[:3000] + 0.01 * rng.standard_normal((3000, 250))
    ref, total = oracle_mod.self_join(x, 1.0)
    return x, ref, total


# stages per block at d = 250: 8 (hi+lo), 4 (16-bit), 2 (FP8); places in the first round
# of the ring of four, in later rounds, the hi and lo slab, the last slab of a block
@pytest.mark.parametrize("mode,stage", [("bf16_split", w) for w in (2, 3, 4, 5, 8, 9, 14, 16)] +
                         [("fp16", w) for w in (2, 4, 5, 7)] + [("fp8_e4m3", w) for w in (2, 3, 6)])
def test_withheld_stage(ej, case, mode, stage):
    x, ref, total = case
    ej.testing_inject(ej.TESTING_GRAM_STAGE, stage)
    ej.testing_inject(ej.TESTING_GRAM_TIMEOUT, 1_000_000)  # 1 ms
    with pytest.raises(ej.EjoinError) as e:
        ej.self_join(x, 1.0, precision=mode)
    assert e.value.status == ETIMEOUT
    counts, got, _ = ej.self_join(x, 1.0, precision=mode)
    assert got == total and np.array_equal(counts, ref)


@pytest.mark.parametrize("mode,d,stage", [("bf16_split", 32, 1), ("fp16", 32, 1), ("fp8_e4m3", 250, 3),
                                          ("fp8_e4m3", 250, 6), ("bf16_split", 250, 5)])
def test_the_call_returns_soon_after_the_deadline(ej, case, mode, d, stage):
    # (no role goes on waiting, up to the two seconds of the drains, for arrivals that
    # cannot come any more: some 6 s for a deadline of 1 ms)
    import time

    x = np.ascontiguousarray(case[0][:, :d])
    ej.self_join(x, 1.0, precision=mode)
    ej.testing_inject(ej.TESTING_GRAM_STAGE, stage)
    ej.testing_inject(ej.TESTING_GRAM_TIMEOUT, 1_000_000)
    t = time.monotonic()
    with pytest.raises(ej.EjoinError):
        ej.self_join(x, 1.0, precision=mode)
    assert time.monotonic() - t < 1.0
