"""The symbol kernels on small frames."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _symbol_us(w, h):
    """GPU time of the symbol stage of a key frame at depth 0, the least of twelve."""
    from riv2_b200 import encoder as E
    cfg = (E.EncoderConfig.new(w, h, 30).with_intra_quality(85).with_keyframe_interval(E.KeyframeInterval.fixed(1))
           .with_pipeline_depth(0))
    enc = E.Encoder.new(cfg, E.VecWriter())
    r = np.random.default_rng(3)
    frame = np.clip(128 + 12 * r.standard_normal((h, w, 3)), 0, 255).astype(np.uint8)
    us = []
    for t in range(12):
        enc.encode_frame(E.Frame(frame, w, h, 20 * t))
        us.append(float(enc.last_kernel_times_us()[7]))
    enc.finish()
    enc.close()
    return min(us)


def test_a_small_frame_takes_no_longer_than_a_large_one():
    """12 macroblocks against 920."""
    small, large = _symbol_us(64, 48), _symbol_us(640, 368)
    assert small <= large, (small, large)
