"""GPU: the training step at the edges of its two kernels (a thread per pair up
to 256 columns; columns in registers beyond), and the state that steps hand on."""
import ctypes

import numpy as np
import pytest

from oracle import learned

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


@pytest.mark.parametrize("k,d", [(8, 256), (1, 260), (8, 512), (9, 516), (16, 300), (16, 1020), (16, 1024),
                                 (16, 1030)])
@pytest.mark.parametrize("m", [1, 16, 17, 1500])
def test_gradient_within_its_rounding_bound(ej, k, d, m):
    rng = np.random.default_rng(k * d + m)
    V = rng.standard_normal((m, d)).astype(np.float32)
    P = (rng.standard_normal((k, d)) / np.sqrt(d)).astype(np.float32)
    V64, P64 = V.astype(np.float64), P.astype(np.float64)
    r = np.sqrt(((V64 @ P64.T) ** 2).sum(1))
    # targets well away from r: no pair's activity depends on rounding
    f = np.where(rng.random(m) < 0.7, rng.uniform(1.1, 2.0, m), rng.uniform(0.5, 0.9, m))
    tgt = np.where(rng.random(m) < 0.9, r * f, 0.0).astype(np.float32)
    G = np.zeros((k, d), dtype=np.float32)
    loss = ctypes.c_float(0)
    rc = ej.load_library().ejoin_testing_projection_grad(V.ctypes.data, tgt.ctypes.data, m,
                                                         P.ctypes.data, k, d, G.ctypes.data,
                                                         ctypes.byref(loss))
    assert rc == 0
    ref_loss, ref = learned.loss_and_grad(V, tgt, P)
    # FP32 sums of d (projection) and at most m (gradient) terms, each rounding
    # charged with the sum of magnitudes; a few more for r, the coefficient and the
    # 2^-40 fixed point of the accumulators (36 blocks at most add to an element)
    act = (tgt > 0) & (r < tgt)
    w = np.where(act, 1.0 / (m * np.where(tgt > 0, tgt, 1.0).astype(np.float64) * r), 0.0)
    mag = (w[:, None] * (np.abs(V64) @ np.abs(P64).T)).T @ np.abs(V64)
    bound = 2.0 * (d + m + 64) * U * mag + 64 * 2.0 ** -40
    assert np.all(np.abs(G - ref) <= bound)
    assert abs(loss.value - ref_loss) <= 2.0 * (d + m + 64) * U * max(1.0, ref_loss)


@pytest.mark.parametrize("k,d", [(8, 64), (5, 40), (16, 1024)])
def test_training_is_reproducible(ej, k, d):
    rng = np.random.default_rng(d)
    x = rng.random((20, d))[rng.integers(0, 20, 6000)] + 0.05 * rng.standard_normal((6000, d))
    runs = [ej.train_projection(x, 0.3, k=k, train_pairs=70_000, train_steps=9, seed=5) for _ in range(3)]
    for P, sigma, _ in runs[1:]:
        assert np.array_equal(P, runs[0][0]) and sigma == runs[0][1]
    assert np.all(np.isfinite(runs[0][0])) and runs[0][1] <= 1.0


@pytest.mark.parametrize("steps", [1, 2, 3])
def test_few_steps(ej, steps):
    # rounds of one step, and a single round
    rng = np.random.default_rng(steps)
    x = rng.standard_normal((500, 24))
    P, sigma, info = ej.train_projection(x, 1.0, k=4, train_pairs=300, train_steps=steps, seed=1)
    assert P.shape == (4, 24) and np.all(np.isfinite(P)) and 0 < sigma <= 1.0
