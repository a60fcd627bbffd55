"""The residual path with a warp for two macroblocks (frames of 592 and more) against the oracle, at
the smallest such frame and at an odd number of macroblocks, over the stage tests' inputs."""
import zlib

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_stages import CASES, _planes


def test_basis_symmetry():
    """The identities that the halved transforms use."""
    import ctypes as C

    from riv2_b200 import encoder as E
    t16, t8 = np.zeros(256, np.int32), np.zeros(64, np.int32)
    E.lib().riv_dct_tables(t16.ctypes.data_as(C.POINTER(C.c_int32)), t8.ctypes.data_as(C.POINTER(C.c_int32)))
    for t in (t16.reshape(16, 16), t8.reshape(8, 8)):
        while t.shape[0] >= 4:
            sign = np.where(np.arange(t.shape[1]) % 2, -1, 1)
            assert np.array_equal(t, t[::-1] * sign)
            t = t[: t.shape[0] // 2, ::2]


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(256, 592), (656, 368)])
@pytest.mark.parametrize("cur_kind,pred_kind,q,scale,dz", CASES)
def test_matches_oracle(w, h, cur_kind, pred_kind, q, scale, dz):
    from riv2_b200 import encoder as E
    n = (w // 16) * (h // 16)
    rng = np.random.default_rng(zlib.crc32(repr((w, cur_kind, pred_kind, q, scale, dz)).encode()))
    cur, pred = _planes(cur_kind, w, h, rng), _planes(pred_kind, w, h, rng)
    base = float(np.float32(O.lib().oracle_quant_step(q)))
    qs = (O.aq_steps(pred[: w * h].reshape(h, w), w, h, base) * np.float32(scale)).astype(np.float32)
    skip = (rng.random(n) < 0.2).astype(np.uint8)
    coded = np.zeros((n, 4), np.int8)
    coded[:, 0] = rng.integers(-2, 3, n)
    got = E.stage_residual(cur, pred, qs, skip, w, h, dz, coded)
    want = O.residual_inter(cur, pred, w, h, skip, qs, dz)
    for g, e in zip(got, want):
        assert np.array_equal(g, e)
    assert np.array_equal(got[3], np.where(want[1] == 0, 1, coded.any(axis=1)))
