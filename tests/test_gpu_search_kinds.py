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
