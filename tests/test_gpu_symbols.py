"""Coefficient symbols and models made on the GPU against the host coder (which the oracle pins):
the same bytes at the edges of its parts (8 macroblocks), warps, rANS batches (16386 symbols) and
model chunks, and the hand-over to the host coder."""
import numpy as np
import pytest

from riv2_b200 import encoder as E

pytestmark = pytest.mark.gpu


def _blocks(n, density, big, seed, lo=0):
    """n blocks whose coefficients thin out towards high frequencies."""
    r = np.random.default_rng(seed)
    pos = np.concatenate([np.arange(256) / 256, np.arange(64) / 64, np.arange(64) / 64])
    keep = r.random((n, 384)) < density * np.exp(-3.0 * pos)[None]
    mag = 1 + np.floor(r.exponential(big, (n, 384))).astype(np.int64)
    b = np.where(keep, np.clip(mag, 1, 8192) * r.choice((-1, 1), (n, 384)), 0)
    b[:lo] = 0
    return b.astype(np.int16)


@pytest.mark.parametrize("intra", [False, True])
@pytest.mark.parametrize("n,density,big", [(1, 0.3, 1.0), (7, 1.0, 2.0), (8, 0.02, 0.3), (9, 0.5, 40.0), (33, 1.0, 900.0),
                                           (129, 0.2, 1.0), (1000, 0.05, 0.5), (2500, 0.6, 3.0)])
def test_matches_host_coder(n, density, big, intra):
    b = _blocks(n, density, big, n)
    skip = None if intra else (np.random.default_rng(n + 1).random(n) < 0.4).astype(np.uint8)
    coded = b if intra else b[skip == 0]
    want = E.dct_encode_host(coded, intra) if len(coded) else b""
    got, on_gpu = E.dct_encode_gpu(b, intra, skip, max_symbols=n * 384 * 27)
    assert on_gpu and got == want


@pytest.mark.parametrize("case", ["none_coded", "all_zero", "long_zero_runs", "long_one_runs", "alternating"])
def test_model_extremes(case):
    n = 3000
    b = np.zeros((n, 384), np.int16)
    skip = np.zeros(n, np.uint8)
    if case == "none_coded":
        skip[:] = 1
    elif case == "long_zero_runs":  # counts at 255 against 1, broken now and then
        b[:, 255] = 1
        b[::700, 3] = -2
        b[1::701, 3:5] = 1
    elif case == "long_one_runs":
        b[:, :256] = 3
        b[::611, 7] = 0
    elif case == "alternating":
        b[::2, :200] = -1
        b[:, 255] = 1
    got, on_gpu = E.dct_encode_gpu(b, False, skip, max_symbols=n * 384 * 27)
    assert on_gpu and got == (E.dct_encode_host(b, False) if case != "none_coded" else b"")


@pytest.mark.parametrize("mag", [4096, 4097, 8191, 8192])
def test_highest_classes(mag):
    b = _blocks(40, 0.1, 1.0, 3)
    b[17, 5], b[21, 270], b[39, 0] = mag, -mag, mag
    got, on_gpu = E.dct_encode_gpu(b, False)
    assert on_gpu and got == E.dct_encode_host(b, False)


def test_refused_class_and_full_stacks_go_to_the_host_coder():
    b = _blocks(300, 0.5, 3.0, 5)
    skip = (np.arange(300) % 3 == 0).astype(np.uint8)
    want = E.dct_encode_host(b[skip == 0], False)
    got, on_gpu = E.dct_encode_gpu(b, False, skip, max_symbols=16386)
    assert not on_gpu and got == want
    b[1, 40] = 8193
    with pytest.raises(E.EncodingFailed):
        E.dct_encode_gpu(b, False, skip)
    skip[1] = 1  # not coded: nothing to refuse
    got, on_gpu = E.dct_encode_gpu(b, False, skip)
    assert on_gpu and got == E.dct_encode_host(b[skip == 0], False)


@pytest.mark.parametrize("intra", [False, True])
@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 31, 32, 33, 47, 49])
def test_part_and_cta_edges(n, intra):
    """A part is two macroblocks (a warp's), a CTA eight parts."""
    b = _blocks(n, 0.4, 2.0, 100 + n)
    skip = None if intra else (np.random.default_rng(n).random(n) < 0.3).astype(np.uint8)
    coded = b if intra else b[skip == 0]
    want = E.dct_encode_host(coded, intra) if len(coded) else b""
    got, on_gpu = E.dct_encode_gpu(b, intra, skip, max_symbols=n * 384 * 27)
    assert on_gpu and got == want
