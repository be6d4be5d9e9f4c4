"""GPU: neighbour lists emitted with the counts.  Lists of every length around
the warp's sort (0, 1, 32, 127 .. 129 and longer), queues that the first guess
makes too small, with a band overflow on top, and host or device buffers."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = ["fp64_direct", "fp64_dmma", "bf16_split", "fp16", "fp8_e4m3"]


def equal(ej, oracle_mod, x, eps, mode, **kw):
    off_ref, nb_ref = oracle_mod.neighbor_lists(x, eps)
    off, nb, st = ej.neighbor_lists(x, eps, precision=mode, **kw)
    assert np.array_equal(off, off_ref) and np.array_equal(nb, nb_ref), st
    return off_ref


@pytest.mark.parametrize("mode", MODES)
def test_list_lengths(ej, oracle_mod, mode):
    # groups of m points at one place each, far from one another: lists of length m
    rng = np.random.default_rng(1)
    sizes = [1, 2, 31, 32, 33, 64, 96, 127, 128, 129, 130, 257, 700]
    place = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    x = 50.0 * rng.random((len(sizes), 20))[place] + 1e-3 * rng.random((place.size, 20))
    x[place == 0] = np.nan  # a list of length 0
    off = equal(ej, oracle_mod, x, 0.5, mode)
    assert set(np.diff(off.astype(np.int64))) == {0, *sizes[1:]}


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n", [2, 129, 3000])
def test_every_pair_is_a_neighbour(ej, oracle_mod, mode, n):
    # n entries a list: more than the arbiter's guess of 64 a point
    x = np.random.default_rng(n).random((n, 8))
    equal(ej, oracle_mod, x, 10.0, mode)


@pytest.mark.parametrize("mode", ["fp16", "fp8_e4m3"])
def test_many_neighbours_and_a_band_overflow(ej, oracle_mod, mode):
    # a lattice: many certain neighbours and many pairs at the radius; the given
    # queue is too small for the band, so the screen emits twice
    x = np.random.default_rng(3).integers(0, 2, (4000, 11)).astype(np.float64)
    for cap in (0, 64):
        equal(ej, oracle_mod, x, 2.0, mode, band_capacity=cap)


def test_long_join_whose_sample_guesses_low(ej, oracle_mod):
    # 20,000 points whose neighbours all sit in a few blocks: a systematic sample
    # of the blocks may miss them all
    rng = np.random.default_rng(4)
    x = 100.0 * rng.random((20_000, 16))
    x[9000:9900] = 0.01 * rng.random((900, 16))
    equal(ej, oracle_mod, x, 1.0, "fp16")


def test_device_buffers_and_a_small_one(ej, oracle_mod):
    import torch

    rng = np.random.default_rng(5)
    x = rng.standard_normal((2500, 12))
    eps = 2.0
    off_ref, nb_ref = oracle_mod.neighbor_lists(x, eps)
    total = int(off_ref[-1])
    xd = torch.from_numpy(x).cuda()
    lib = ej.load_library()
    opt = ej.Options()
    lib.ejoin_default_options(ctypes.byref(opt))
    for cap in (total - 1, total, 3 * total):
        off = torch.zeros(2501, dtype=torch.int64, device="cuda")
        nb = torch.full((3 * total,), -7, dtype=torch.int32, device="cuda")
        t = ctypes.c_uint64(0)
        rc = lib.ejoin_neighbor_lists(xd.data_ptr(), 2500, 12, eps, ctypes.byref(opt), off.data_ptr(),
                                      nb.data_ptr(), cap, ctypes.byref(t), None)
        assert rc == (-3 if cap < total else 0) and t.value == total
        assert np.array_equal(off.cpu().numpy().astype(np.uint64), off_ref)
        got = nb.cpu().numpy()
        if cap >= total:
            assert np.array_equal(got[:total].astype(np.uint32), nb_ref)
            assert np.all(got[total:] == -7)
        else:
            assert np.all(got == -7)
