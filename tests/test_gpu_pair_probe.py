"""GPU: the MMAs that the join issues -- two CTAs, M = N = 256, aug tiles in store_aug's
order -- through a probe of one tile, against numpy: the products and the layout of
their operands and results, and the error of the accumulation against the model behind
the screen's margins (screen_params in api.cu)."""
import ctypes
import os

import numpy as np
import pytest

from conftest import ROOT
from test_gpu_probe import (bf16_bits_to_f64, e4m3_decode, f32_to_bf16_bits, magnitude_pattern,
                            random_e4m3)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(ej):
    lib = ctypes.CDLL(os.path.join(ROOT, "tests", "csrc", "libumma_pair_probe.so"))
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    lib.umma_pair_probe.argtypes = [vp, vp, i32, i32, i32, vp, vp, ctypes.POINTER(ctypes.c_uint)]
    lib.umma_pair_probe.restype = i32

    def run(A, B, fmt, split=0, aug=None):
        A, B = np.ascontiguousarray(A), np.ascontiguousarray(B)
        row = A.shape[1] * A.itemsize
        assert A.shape == B.shape and A.shape[0] == 256 and row % 128 == 0
        aug = None if aug is None else np.ascontiguousarray(aug, dtype=np.uint16)
        assert aug is None or aug.shape == (256, 32)
        D = np.zeros((256, 256), dtype=np.float32)
        to = ctypes.c_uint(0)
        rc = lib.umma_pair_probe(A.ctypes.data, B.ctypes.data, row // 128, fmt, split,
                                 None if aug is None else aug.ctypes.data, D.ctypes.data,
                                 ctypes.byref(to))
        assert rc == 0, (rc, to.value)
        return D.astype(np.float64)

    return run


def encode(x, fmt):
    """16-bit operands of float values: bits and their float64 values; the packer's
    operands hold no subnormals."""
    x = np.asarray(x, dtype=np.float32)
    if fmt == 1:
        b = f32_to_bf16_bits(x)
        return b, bf16_bits_to_f64(b)
    h = x.astype(np.float16)
    h[np.abs(h) < 2.0 ** -14] = 0
    return h.view(np.uint16), h.astype(np.float64)


def model(instructions):
    """Exact result and error bound of MMAs issued one after the other: instruction t of
    K_t products errs by at most K_t 2^-22 of the magnitudes accumulated up to its end;
    16 2^-22 of the total for the final value."""
    shape = (instructions[0][0].shape[0], instructions[0][1].shape[0])
    exact, prefix, total = np.zeros(shape), np.zeros(shape), np.zeros(shape)
    for a, b in instructions:
        exact += a @ b.T
        prefix += np.abs(a) @ np.abs(b).T
        total += a.shape[1] * prefix
    return exact, (total + 16 * prefix) * 2.0 ** -22


def steps(af, bf, k):
    return [(af[:, c: c + k], bf[:, c: c + k]) for c in range(0, af.shape[1], k)]


def check(D, instructions, what):
    exact, bound = model(instructions)
    worst = float((np.abs(D - exact) / bound).max())
    print(f"{what}: max error / model bound = {worst:.3e}")
    assert worst * 4 <= 1.0


def aug_values(rng, fmt, scale):
    """[256][32] values with the packer's zeros: A side 0..5, B side 16..21."""
    v = np.zeros((256, 32))
    v[:, 0:3] = scale * rng.standard_normal((256, 3)) * [1.0, 2.0 ** -9, 2.0 ** -18]
    v[:, 3:6] = -1.0
    v[:, 16:19] = -1.0
    v[:, 19:22] = scale * rng.standard_normal((256, 3)) * [1.0, 2.0 ** -9, 2.0 ** -18]
    return encode(v, fmt)


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("slabs", [1, 2, 6])
def test_tile_of_a_pair(probe, slabs, fmt):
    rng = np.random.default_rng(10 * slabs + fmt)
    A, af = encode(rng.standard_normal((256, 64 * slabs)), fmt)
    B, bf = encode(rng.standard_normal((256, 64 * slabs)), fmt)
    check(probe(A, B, fmt), steps(af, bf, 16), f"tile, {slabs} slabs, fmt {fmt}")


@pytest.mark.parametrize("fmt", [0, 1])
def test_every_row_and_column_has_its_place(probe, fmt):
    # one product per entry, exact in FP32: row i holds i + 1 in column 0, row j of B
    # holds 1 and j + 1 in different columns
    A = np.zeros((256, 64))
    B = np.zeros((256, 64))
    A[:, 0] = np.arange(256) + 1
    A[:, 33] = 1.0
    B[:, 0] = np.where(np.arange(256) % 2, 1.0, 2.0)
    B[:, 33] = np.arange(256) * 0.25
    D = probe(encode(A, fmt)[0], encode(B, fmt)[0], fmt)
    assert np.array_equal(D, encode(A, fmt)[1] @ encode(B, fmt)[1].T)


@pytest.mark.parametrize("fmt", [0, 1])
def test_aug_tiles_of_store_aug(probe, fmt):
    rng = np.random.default_rng(30 + fmt)
    v, vf = aug_values(rng, fmt, 8.0)
    # all 32 values of a row, also those that the packer leaves zero
    w, wf = encode(rng.standard_normal((256, 32)), fmt)
    Z = np.zeros((256, 64), dtype=np.uint16)
    for bits, val in ((v, vf), (w, wf)):
        check(probe(Z, Z, fmt, aug=bits), [(val[:, :16], val[:, 16:])], f"aug, fmt {fmt}")


@pytest.mark.parametrize("pattern", ["small_then_large", "large_last", "ramp", "large_first"])
@pytest.mark.parametrize("fmt", [0, 1])
def test_accumulation_of_a_pair(probe, fmt, pattern):
    rng = np.random.default_rng(100 + fmt * 10 + len(pattern))
    K = 256
    m = magnitude_pattern(rng, pattern, K)
    a, b = rng.standard_normal((256, K)) * m, rng.standard_normal((256, K)) * m
    # rows 128..: the last instruction of pair (j, j) only subtracts
    b[128:, K - 16:] = -a[128:, K - 16:]
    A, af = encode(a, fmt)
    B, bf = encode(b, fmt)
    check(probe(A, B, fmt), steps(af, bf, 16), f"{pattern}, fmt {fmt}")


@pytest.mark.parametrize("slabs", [1, 2, 3])
def test_split_products_and_aug_in_the_joins_order(probe, slabs):
    # centred rows, hi + lo in BF16; alpha about half the squared norm, as in a join
    rng = np.random.default_rng(50 + slabs)
    K = 64 * slabs
    a = rng.standard_normal((256, K)) / np.sqrt(K)
    b = a[rng.permutation(256)] + 2.0 ** -6 * rng.standard_normal((256, K)) / np.sqrt(K)
    ah, ahf = encode(a, 1)
    bh, bhf = encode(b, 1)
    al, alf = encode(a - ahf, 1)
    bl, blf = encode(b - bhf, 1)
    v, vf = aug_values(rng, 1, 0.5)
    seq = []
    for c in range(slabs):
        hi = [slice(64 * c + 16 * k, 64 * c + 16 * k + 16) for k in range(4)]
        for s in hi:
            seq += [(ahf[:, s], blf[:, s]), (alf[:, s], bhf[:, s])]
        seq += [(ahf[:, s], bhf[:, s]) for s in hi]
    seq.append((vf[:, :16], vf[:, 16:]))
    D = probe(np.concatenate([ah, al], 1), np.concatenate([bh, bl], 1), 1, split=1, aug=v)
    check(D, seq, f"hi+lo, {slabs} slabs")


@pytest.mark.parametrize("pattern", ["small_then_large", "large_last", "ramp"])
def test_fp8_accumulation_of_a_pair(probe, pattern):
    rng = np.random.default_rng(200 + len(pattern))
    span = {"small_then_large": [(-6, -4)] * 4 + [(2, 5)] * 4,
            "large_last": [(-6, -5)] * 7 + [(5, 7)],
            "ramp": [(-6 + i, -5 + i) for i in range(8)]}[pattern]
    A = np.concatenate([random_e4m3(rng, (256, 32), lo, hi) for lo, hi in span], axis=1)
    B = np.concatenate([random_e4m3(rng, (256, 32), lo, hi) for lo, hi in span], axis=1)
    af, bf = e4m3_decode(A), e4m3_decode(B)
    check(probe(A, B, 2), steps(af, bf, 32), f"FP8 {pattern}")
    # with BF16 aug operands on top, as in the join
    v, vf = aug_values(rng, 1, 64.0)
    check(probe(A, B, 2, aug=v), steps(af, bf, 32) + [(vf[:, :16], vf[:, 16:])],
          f"FP8 {pattern} and aug")
