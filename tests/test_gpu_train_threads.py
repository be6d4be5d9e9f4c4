"""GPU: projections of different sizes trained and used by several threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_train_projections_of_different_sizes(ej):
    # sizes of every training and projection kernel, small and large shared memory each
    cases = [(24, 4), (64, 8), (130, 8), (250, 16), (400, 5), (1000, 8), (1000, 16), (1300, 8)]
    xs = [np.random.default_rng(d + k).random((1500, d)) for d, k in cases]
    kw = dict(train_steps=6, train_pairs=4096)

    def call(i):
        (d, k), x = cases[i], xs[i]
        eps = 0.4 * np.sqrt(d / 6.0)
        P, sigma, _ = ej.train_projection(x, eps, k=k, **kw)
        counts, total, _ = ej.self_join(x, eps, precision="bf16_split", proj_k=k, **kw)
        return P.tobytes(), sigma, total

    alone = [call(i) for i in range(len(cases))]
    failed = []

    def work(i):
        for _ in range(12):
            try:
                if call(i) != alone[i]:
                    failed.append((cases[i], "differs"))
            except ej.EjoinError as e:
                failed.append((cases[i], str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not failed, failed[:3]
