"""Which search kind an encoder or a batch gets, at the limits of a CTA's shared memory and beside
others, and every kind against the oracle: streams byte for byte."""
import pytest

from test_gpu_search_direct import _configs, _frames, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b", [((1920, 64, 12), (352, 64, 12)), ((1920, 64, 31), (352, 64, 16)),
                                 ((64, 64, 16), (1920, 64, 31))])
def test_encoders_of_two_sizes(a, b):
    """Two encoders alive at once, frame by frame in turn: the second one's sizes are not the first's."""
    from riv2_b200 import encoder as E
    runs = []
    for w, h, sr in (a, b):
        gc, oc = _configs(w, h, sr, 4)
        wr = E.VecWriter()
        runs.append((E.Encoder.new(gc, wr), wr, oc, _frames(w, h, 3, w + sr)))
    for t in range(3):
        for enc, _, oc, f in runs:
            enc.encode_frame(E.Frame(f[t], oc.display_width, oc.display_height, 20 * t))
    for enc, wr, oc, f in runs:
        enc.finish()
        enc.close()
        assert wr.into_inner() == _oracle(oc, f)


def test_batches_of_two_ranges():
    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    runs = []
    for sr in (60, 16):
        gc, oc = _configs(352, 64, sr, 2)
        wr = E.VecWriter()
        runs.append((Batch.new([gc], [wr]), wr, oc, _frames(352, 64, 3, sr)))
    for t in range(3):
        for b, _, _, f in runs:
            b.encode_step([f[t]], [20 * t])
    for b, wr, oc, f in runs:
        b.finish()
        b.close()
        assert wr.into_inner() == _oracle(oc, f)


def _encode(gc, frames):
    from riv2_b200 import encoder as E
    wr = E.VecWriter()
    enc = E.Encoder.new(gc, wr)
    for t, f in enumerate(frames):
        enc.encode_frame(E.Frame(f, gc.display_width, gc.display_height, 20 * t))
    enc.finish()
    enc.close()
    return wr.into_inner()


@pytest.mark.parametrize("depth", [0, 4])
@pytest.mark.parametrize("w,h,sr", [(640, 48, 96), (640, 48, 101), (640, 48, 102), (640, 64, 127), (1920, 32, 127)])
def test_widest_ranges(w, h, sr, depth):
    """Both sides of the range above which four windows no longer fit (101), where the band does not
    either."""
    frames = _frames(w, h, 3, w + sr)
    gc, oc = _configs(w, h, sr, depth)
    assert _encode(gc, frames) == _oracle(oc, frames)


@pytest.mark.parametrize("w,h,sr", [(640, 368, 98), (960, 544, 73), (1920, 1088, 36)])
def test_band_kept(w, h, sr):
    """The widest ranges at which a row's band fits 200 KB without a loader: it is kept with the
    loader's slots on top."""
    from riv2_b200 import encoder as E
    p = E.search_plan(w, h, sr)
    assert p["band"] and p["loader"] and not p["table"]


@pytest.mark.parametrize("table", [0, 1])
@pytest.mark.parametrize("clips", [[(352, 64, 101), (64, 64, 12)], [(352, 64, 102), (64, 64, 12), (48, 32, 31)], [(64, 64, 127)],
                                   [(16, 16, 64)] * 149, [(16, 16, 64)] * 147 + [(32, 32, 16)] * 10])
def test_batch_of_wide_ranges(clips, table):
    """Ranges beyond a ring of four windows (101), and more clips than such rings fit the GPU at once
    (148 from a range of 64 on)."""
    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    cfgs = {c: _configs(*c, 2) for c in set(clips)}
    frames = {c: _frames(c[0], c[1], 3, sum(c)) for c in cfgs}
    writers = [E.VecWriter() for _ in clips]
    b = Batch.new([cfgs[c][0] for c in clips], writers)
    b.set_tune(100, 4, 128, table)
    for t in range(3):
        b.encode_step([frames[c][t] for c in clips], [20 * t] * len(clips))
    b.finish()
    b.close()
    want = {c: _oracle(cfgs[c][1], frames[c]) for c in cfgs}
    assert all(w.into_inner() == want[c] for w, c in zip(writers, clips))


@pytest.mark.parametrize("w,h", [(16, 16), (640, 368), (1920, 1088), (3840, 2160)])
@pytest.mark.parametrize("sr", [16, 31, 63])
def test_direct_launch_leaves_the_gpu_to_others(w, h, sr):
    """Without a table a launch has the CTAs of its macroblock rows and no others."""
    from riv2_b200 import encoder as E
    p = E.search_plan(w, h, sr)
    assert not p["fused"] and p["ctas"] == p["row_ctas"] <= h // 16


@pytest.mark.parametrize("sr", [12, 16, 31])
def test_encoders_side_by_side(sr):
    """Four encoders of different sizes, each on a thread of its own, depth 0 and frames in flight."""
    import threading

    from riv2_b200 import encoder as E
    runs = []
    for k, (w, h) in enumerate([(352, 288), (96, 64), (640, 368), (208, 112)]):
        gc, oc = _configs(w, h, sr, 4 * (k % 2))
        wr = E.VecWriter()
        runs.append((E.Encoder.new(gc, wr), wr, oc, _frames(w, h, 5, w + sr)))

    def work(enc, oc, frames):
        for t, f in enumerate(frames):
            enc.encode_frame(E.Frame(f, oc.display_width, oc.display_height, 20 * t))
        enc.finish()

    threads = [threading.Thread(target=work, args=(enc, oc, f)) for enc, _, oc, f in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for enc, wr, oc, f in runs:
        enc.close()
        assert wr.into_inner() == _oracle(oc, f)


def test_learned_encoders_side_by_side():
    """Four encoders of the learned form on threads of their own write what one alone writes (their
    products are of different widths, launched by the threads at the same time)."""
    import os
    import threading

    import numpy as np
    import torch

    import riv2_b200
    from riv2_b200 import encoder as E
    from riv2_b200 import proposal as P
    params = P.load_params(os.path.join(os.path.dirname(riv2_b200.__file__), "weights", "proposal.bin"))
    frames = torch.from_numpy(np.stack(_frames(352, 288, 8, 7))).cuda()
    torch.cuda.synchronize()

    def start():
        gc = _configs(352, 288, 12, 4)[0].with_encode_form(1)
        wr = E.VecWriter()
        enc = E.Encoder.new(gc, wr)
        enc.set_proposal(params)
        return enc, wr

    def work(enc):
        for t in range(160):
            enc.encode_frame_device(frames[t % 8].data_ptr(), 20 * t)
        enc.finish()

    alone, alone_wr = start()
    work(alone)
    alone.close()
    runs = [start() for _ in range(4)]
    threads = [threading.Thread(target=work, args=(enc,)) for enc, _ in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    want = alone_wr.into_inner()
    for enc, wr in runs:
        enc.close()
        assert wr.into_inner() == want


# 64-bit costs, with a table (ranges up to 15) and without, each with a band and (3856 columns) a window:
# the usual weight with the 32-bit kinds switched off, weights whose costs pass 2^27 and 2^58 (no table),
# and a negative one (no table either)
WEIGHTS = [("0", 0.49), ("1", 1e7), ("1", 1e17), ("1", -0.49)]


def _weighted(w, h, sr, depth, weight):
    gc, oc = _configs(w, h, sr, depth)
    oc.rdo_lambda_mult = weight
    return gc.with_rdo_lambda_mult(weight), oc


@pytest.mark.parametrize("small,weight", WEIGHTS)
@pytest.mark.parametrize("w,h,sr", [(352, 288, 12), (3856, 32, 15), (352, 288, 31), (3856, 32, 31)])
@pytest.mark.parametrize("depth", [0, 4])
def test_wide_costs(w, h, sr, depth, small, weight, monkeypatch):
    monkeypatch.setenv("RIV_SEARCH_SMALL", small)
    frames = _frames(w, h, 4, w + sr)
    gc, oc = _weighted(w, h, sr, depth, weight)
    assert _encode(gc, frames) == _oracle(oc, frames)


@pytest.mark.parametrize("table", [0, 1])
def test_batch_of_wide_costs(table):
    """Every kind of search in one step."""
    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    clips = [(352, 288, 12, 1e7), (352, 288, 12, 0.49), (100, 70, 31, 1e7), (208, 112, 31, 0.49), (64, 48, 7, 1e17),
             (64, 48, 12, -0.49)]
    cfgs = [_weighted(w, h, sr, 2, k) for w, h, sr, k in clips]
    frames = [_frames(w, h, 4, w + sr) for w, h, sr, _ in clips]
    writers = [E.VecWriter() for _ in clips]
    b = Batch.new([g for g, _ in cfgs], writers)
    b.set_tune(100, 4, 128, table)
    for t in range(4):
        b.encode_step([f[t] for f in frames], [20 * t] * len(clips))
    b.finish()
    b.close()
    for (_, oc), f, wr in zip(cfgs, frames, writers):
        assert wr.into_inner() == _oracle(oc, f)


@pytest.mark.parametrize("w,h,sr", [(1136, 2400, 31), (1360, 2400, 64)])
def test_more_rows_than_ctas(w, h, sr):
    """150 macroblock rows on one CTA an SM: the last rows are a CTA's second, with a band and with a ring."""
    from riv2_b200 import encoder as E
    p = E.search_plan(w, h, sr)
    assert p["row_ctas"] < h // 16 and p["band"] == (sr == 31) and not p["table"]
    frames = _frames(w, h, 3, w + sr)
    gc, oc = _configs(w, h, sr, 4)
    assert _encode(gc, frames) == _oracle(oc, frames)


# zero-MV threshold, predictor threshold, weight of the MV costs
STOPS = [(800, 0, 0.49), (0, 1500, 0.49), (3000, 6000, 0.49), (0, 0, 0.0), (500, 900, 0.0)]


def _stops(w, h, sr, depth, zero, predictor, weight):
    gc, oc = _weighted(w, h, sr, depth, weight)
    oc.me_zero_mv_threshold, oc.me_predictor_threshold = zero, predictor
    return gc._with(me_zero_mv_threshold=zero, me_predictor_threshold=predictor), oc


@pytest.mark.parametrize("zero,predictor,weight", STOPS)
@pytest.mark.parametrize("w,h,sr", [(352, 288, 12), (357, 131, 16), (352, 288, 31), (3856, 32, 31), (640, 48, 102)])
def test_early_stops_and_free_vectors(w, h, sr, zero, predictor, weight):
    """Searches that end at the zero MV or at a predictor, and MV costs of 0."""
    frames = _frames(w, h, 4, w + sr)
    gc, oc = _stops(w, h, sr, 4, zero, predictor, weight)
    assert _encode(gc, frames) == _oracle(oc, frames)


@pytest.mark.parametrize("table", [0, 1])
def test_batch_early_stops_and_free_vectors(table):
    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    clips = [(352, 288, 12) + s for s in STOPS] + [(100, 70, 31) + s for s in STOPS]
    cfgs = [_stops(w, h, sr, 2, *s) for w, h, sr, *s in clips]
    frames = [_frames(w, h, 4, w + sr) for w, h, sr, *_ in clips]
    writers = [E.VecWriter() for _ in clips]
    b = Batch.new([g for g, _ in cfgs], writers)
    b.set_tune(75, 8, 64, table)
    for t in range(4):
        b.encode_step([f[t] for f in frames], [20 * t] * len(clips))
    b.finish()
    b.close()
    for (_, oc), f, wr in zip(cfgs, frames, writers):
        assert wr.into_inner() == _oracle(oc, f)
