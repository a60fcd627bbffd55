"""The search without an exhaustive SAD table (search ranges above 15, frames too tall for the fused
table launch, batches that compute their SADs on the way) against the oracle: streams byte for
byte, at both sides of the window and band limits, where search windows cross every frame edge,
and with frames in flight (the reconstruction then runs inside the search launch)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _frames(w, h, n, seed):
    """Textured blocks that move by up to 20 pixels a frame over a drifting gradient."""
    r = np.random.default_rng(seed)
    tex = r.integers(0, 256, (h + 80, w + 80, 3)).astype(np.float32)
    for _ in range(2):
        tex = (tex + np.roll(tex, 1, 0) + np.roll(tex, 1, 1) + np.roll(tex, (1, 1), (0, 1))) / 4
    blocks = [(int(x), int(y), int(vx), int(vy)) for x, y, vx, vy in
              zip(r.integers(0, w, 12), r.integers(0, h, 12), r.integers(-20, 21, 12), r.integers(-20, 21, 12))]
    out = []
    for t in range(n):
        f = tex[40 + t:40 + t + h, 40 + 2 * t:40 + 2 * t + w].copy()
        for k, (x, y, vx, vy) in enumerate(blocks):
            px, py = (x + vx * t) % w, (y + vy * t) % h
            bw, bh = min(24, w - px), min(40, h - py)
            f[py:py + bh, px:px + bw] = tex[10 + k:10 + k + bh, 5:5 + bw]
        f += r.normal(0, 2, f.shape)
        out.append(np.clip(f, 0, 255).astype(np.uint8))
    return out


def _configs(w, h, sr, depth, iq=85, pq=80):
    from riv2_b200 import encoder as E
    gc = (E.EncoderConfig.new(w, h, 30).with_intra_quality(iq).with_inter_quality(pq).with_search_range(sr)
          .with_keyframe_interval(E.KeyframeInterval.fixed(1000)).with_pipeline_depth(depth))
    oc = O.default_config(w, h, 30)
    oc.intra_quality, oc.inter_quality, oc.search_range = iq, pq, sr
    oc.keyframe_mode, oc.keyframe_interval = gc.keyframe_interval.mode, gc.keyframe_interval.interval
    return gc, oc


def _oracle(oc, frames):
    o = O.OracleEncoder(oc)
    for t, f in enumerate(frames):
        assert o.encode_rgb(f, 20 * t) == 0
    return o.finish()


@pytest.mark.parametrize("depth", [0, 4])
@pytest.mark.parametrize("w,h,sr", [(16, 16, 16), (48, 100, 16), (352, 288, 16), (352, 288, 31), (357, 131, 32), (208, 48, 63),
                                    (160, 208, 127), (3840, 48, 31), (3856, 32, 12), (32, 2384, 12), (64, 2240, 24)])
def test_encode(w, h, sr, depth):
    from riv2_b200 import encoder as E
    frames = _frames(w, h, 4, w + h + sr)
    gc, oc = _configs(w, h, sr, depth)
    wr = E.VecWriter()
    enc = E.Encoder.new(gc, wr)
    for t, f in enumerate(frames):
        enc.encode_frame(E.Frame(f, w, h, 20 * t))
    enc.finish()
    enc.close()
    assert wr.into_inner() == _oracle(oc, frames)


@pytest.mark.parametrize("sr", [1, 7, 15, 16, 40])
def test_batch_without_table(sr):
    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    sizes = [(16, 16), (100, 70), (352, 288), (640, 360)]
    clips = [_frames(w, h, 4, w + sr) for w, h in sizes]
    cfgs = [_configs(w, h, sr, 2) for w, h in sizes]
    writers = [E.VecWriter() for _ in sizes]
    b = Batch.new([g for g, _ in cfgs], writers)
    b.set_tune(75, 4, 128, 0)
    for t in range(4):
        b.encode_step([c[t] for c in clips], [20 * t] * len(sizes))
    b.finish()
    b.close()
    for (_, oc), c, wr in zip(cfgs, clips, writers):
        assert wr.into_inner() == _oracle(oc, c)
