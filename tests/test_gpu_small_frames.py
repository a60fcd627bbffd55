"""Frames of few macroblocks: which coder lists and models their coefficients, at both sides of each line
(40 with nothing in flight, 128 with frames in flight, 320 for key frames only), streams against the
oracle."""
import pytest

from test_gpu_search_direct import _configs, _frames, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,depth,interval,on_gpu", [
    (16, 16, 0, 1000, False), (208, 48, 0, 1000, False), (160, 64, 0, 1000, True), (208, 48, 1, 1, False),
    (160, 64, 1, 1, True), (2032, 16, 4, 1000, False), (256, 128, 4, 1000, True), (464, 176, 4, 1, False),
    (320, 256, 4, 1, True), (64, 48, 8, 3, False)])
def test_route_and_stream(w, h, depth, interval, on_gpu):
    from riv2_b200 import encoder as E
    gc, oc = _configs(w, h, 16, depth)
    gc = gc.with_keyframe_interval(E.KeyframeInterval.fixed(interval))
    oc.keyframe_interval = interval
    frames = _frames(w, h, 7, w + h)
    wr = E.VecWriter()
    enc = E.Encoder.new(gc, wr)
    for t, f in enumerate(frames):
        enc.encode_frame(E.Frame(f, w, h, 20 * t))
    enc.finish()
    launches = enc.counters()["launches"]
    enc.close()
    assert wr.into_inner() == _oracle(oc, frames)
    # conversion, residual, deblock; a search; the five symbol kernels, or three that pack the blocks
    keys = -(-7 // interval)
    assert launches == 7 * (8 if on_gpu else 6) + (7 - keys)


def test_frames_beyond_the_stacks_are_packed_at_once():
    """Key frames of noise at quality 100 (more symbols than the GPU's stacks hold) and of a still picture:
    the first of the noise runs all the symbol kernels, the others only those that pack, and so does the
    first still one."""
    import numpy as np

    from riv2_b200 import encoder as E
    w, h = 352, 288
    r = np.random.default_rng(8)
    noise = [r.integers(0, 256, (h, w, 3), dtype=np.uint8) for _ in range(3)]
    still = [np.full((h, w, 3), 90, np.uint8)] * 3
    gc, oc = _configs(w, h, 12, 0, 100, 100)
    gc = gc.with_keyframe_interval(E.KeyframeInterval.fixed(1))
    oc.keyframe_interval = 1
    wr = E.VecWriter()
    enc = E.Encoder.new(gc, wr)
    launches = [0]
    for t, f in enumerate(noise + still):
        enc.encode_frame(E.Frame(f, w, h, 20 * t))
        launches.append(enc.counters()["launches"])
    enc.finish()
    enc.close()
    assert wr.into_inner() == _oracle(oc, noise + still)
    steps = np.diff(launches)
    assert list(steps - steps[1]) == [2, 0, 0, 0, 2, 2]
