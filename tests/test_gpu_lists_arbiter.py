"""GPU: neighbour lists on the FP64 arbiter run it once where points have some hundred
neighbours (a first queue for 64 a point repeats it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64_direct", "fp64_dmma"])
@pytest.mark.parametrize("n,d,m", [(4000, 64, 200), (6001, 33, 300)])
def test_one_pass(ej, oracle_mod, mode, n, d, m):
    # groups of m points, neighbours of one another
    rng = np.random.default_rng(n)
    x = 50.0 * rng.random((n // m + 1, d))[rng.permutation(n) // m] + 1e-3 * rng.random((n, d))
    launches = []
    for eps in (1e-9, 1.0):
        off_ref, nb_ref = oracle_mod.neighbor_lists(x, eps)
        off, nb, st = ej.neighbor_lists(x, eps, precision=mode)
        assert np.array_equal(off, off_ref) and np.array_equal(nb, nb_ref)
        launches.append(st["kernel_launches"])
    assert off[-1] > 130 * n
    assert launches[0] == launches[1], launches
