"""GPU: neighbour lists around the block sort's bounds (128 and 1024 entries), on
its own and next to longer ones, and a list in every block of its grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[128, 129, 255, 256, 257, 258], [1, 511, 512, 513, 1023, 1024],
                                   [3, 1024, 1025, 1500], [130] * 20])
def test_list_lengths(ej, oracle_mod, sizes):
    rng = np.random.default_rng(len(sizes) + sizes[-1])
    place = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    x = 50.0 * rng.random((len(sizes), 20))[place] + 1e-3 * rng.random((place.size, 20))
    off_ref, nb_ref = oracle_mod.neighbor_lists(x, 0.5)
    for mode in ("fp64_direct", "fp16"):
        off, nb, st = ej.neighbor_lists(x, 0.5, precision=mode)
        assert np.array_equal(off, off_ref) and np.array_equal(nb, nb_ref), st
