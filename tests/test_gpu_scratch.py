"""GPU: the band queue's first size and the scratch that stays between calls."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_small_calls_retain_little_and_give_it_back(ej):
    rng = np.random.default_rng(0)
    # (the first call on a device also loads the kernels' code, 2 MiB that no call
    # gives back: not scratch)
    ej.self_join(rng.standard_normal((10, 18)), 0.5)
    ej.release_scratch(0)
    free0 = free_bytes()
    for n in (10, 1000, 9000):
        ej.self_join(rng.standard_normal((n, 18)), 0.5)
        assert free0 - free_bytes() <= 33 << 20
    ej.release_scratch(0)
    assert free0 - free_bytes() <= 1 << 20


@pytest.mark.parametrize("mode", ["fp16", "fp8_e4m3"])
@pytest.mark.parametrize("n,nq", [(900, 0), (5000, 0), (20_000, 0), (20_000, 6000)])
def test_queue_of_data_whose_pairs_all_lie_in_the_band(ej, oracle_mod, mode, n, nq):
    # points on a lattice of two values per column: many pairs at exactly the
    # radius, far more records than the first queue holds; the screen runs again
    rng = np.random.default_rng(n)
    x = rng.integers(0, 2, (n, 12)).astype(np.float64)
    eps = 2.0
    if nq:
        q = rng.integers(0, 2, (nq, 12)).astype(np.float64)
        got, total, st = ej.join_counts(q, x, eps, precision=mode)
        ref = oracle_mod.cross_counts(q, x, eps)
    else:
        got, total, st = ej.self_join(x, eps, precision=mode)
        ref, _ = oracle_mod.self_join(x, eps)
    assert np.array_equal(got, ref) and total == int(ref.sum())
    assert st["band_pairs"] > 0


def test_threads_share_the_pool(ej, oracle_mod):
    rng = np.random.default_rng(1)
    xs = [rng.standard_normal((1500 + 100 * t, 24)) for t in range(6)]
    refs = [oracle_mod.self_join(x, 4.0)[0] for x in xs]
    bad = []

    def work(t):
        for _ in range(5):
            c, _, _ = ej.self_join(xs[t], 4.0, precision="fp16" if t % 2 else "bf16_split")
            if not np.array_equal(c, refs[t]):
                bad.append(t)

    th = [threading.Thread(target=work, args=(t,)) for t in range(len(xs))]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad
