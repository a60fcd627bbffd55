"""Frames with more symbols than usual, against the oracle: stacks beyond the pinned buffer of a
single encoder (384 symbols a macroblock), and frames that the GPU hands over to the host coder (512,
rounded up to whole batches of 16386), alone and in a step beside ordinary clips."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_search_direct import _configs, _frames

W, H = 352, 288
MBS = (W // 16) * (H // 16)
ROOM = -(-MBS * 512 // 16386) * 16386  # symbols of a frame that the GPU codes


def _noise(n, amplitude, seed):
    r = np.random.default_rng(seed)
    return [np.clip(128 + amplitude * r.standard_normal((H, W, 3)), 0, 255).astype(np.uint8) for _ in range(n)]


def _symbols(c, intra):
    """Symbols of a frame's coefficient stream (res/rans.rs:195-330) from its quantised blocks."""
    c = c.astype(np.int64)
    if not intra:
        c = c[c.any(axis=1)]
    length = lambda v: np.frexp(v.astype(np.float64))[1]  # noqa: E731  (bits of v >= 0)
    code = lambda k, top: k + (k < top) + np.maximum(k - 1, 0)  # noqa: E731
    total = 0
    for a, b, top in ((0, 256, 8), (256, 320, 6), (320, 384, 6)):
        v = c[:, a:b].copy()
        first = 1 if intra else 0
        i = np.arange(b - a)
        last = np.where((v != 0) & (i >= first), i, 0).max(axis=1)
        if intra:
            v[1:, 0] -= c[:-1, a]
        total += int(code(length(last), top).sum())
        used = i <= last[:, None]
        some = used & (v != 0)
        total += int(used.sum()) + int((1 + code(length(np.abs(v[some]) - 1), 12)).sum())
    return total


def _oracle(frames, iq, pq, sr):
    """The stream, and each frame's symbols."""
    _, oc = _configs(W, H, sr, 0, iq, pq)
    o, n = O.OracleEncoder(oc), []
    for t, f in enumerate(frames):
        assert o.encode_rgb(f, 20 * t) == 0
        n.append(_symbols(o.last_coeffs(), t == 0))
    return o.finish(), n


# amplitude of the noise, qualities: what the frames of each clip hold
CLIPS = {"stacks": (12, 95, 90), "host": (60, 100, 100)}


def _clip(kind, n=3):
    amplitude, iq, pq = CLIPS[kind]
    return _noise(n, amplitude, 5), iq, pq


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [0, 4])
@pytest.mark.parametrize("kind,sr", [("stacks", 16), ("stacks", 12), ("host", 16)])
def test_single_encoder(kind, sr, depth):
    from riv2_b200 import encoder as E
    frames, iq, pq = _clip(kind)
    want, n = _oracle(frames, iq, pq, sr)
    lo, hi = (384 * MBS, 512 * MBS) if kind == "stacks" else (ROOM, 1 << 30)
    assert all(lo < k <= hi for k in n), n
    wr = E.VecWriter()
    enc = E.Encoder.new(_configs(W, H, sr, depth, iq, pq)[0], wr)
    for t, f in enumerate(frames):
        enc.encode_frame(E.Frame(f, W, H, 20 * t))
    enc.finish()
    enc.close()
    assert wr.into_inner() == want


@pytest.mark.gpu
@pytest.mark.parametrize("table", [0, 1])
def test_batch(table):
    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    clips = [(_frames(W, H, 3, 9), 85, 80), _clip("host"), _clip("stacks"), (_frames(W, H, 3, 4), 75, 70)]
    want = [_oracle(f, iq, pq, 12) for f, iq, pq in clips]
    assert all(k > ROOM for k in want[1][1]) and all(k <= ROOM for _, n in want[2:] for k in n)
    writers = [E.VecWriter() for _ in clips]
    b = Batch.new([_configs(W, H, 12, 2, iq, pq)[0] for _, iq, pq in clips], writers)
    b.set_tune(100, 4, 128, table)
    for t in range(3):
        b.encode_step([f[t] for f, _, _ in clips], [20 * t] * len(clips))
    b.finish()
    b.close()
    for wr, (stream, _) in zip(writers, want):
        assert wr.into_inner() == stream
