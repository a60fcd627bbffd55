"""A writer that refuses a record of one clip of a batch: that record is lost and reported, every other
record of it and of the other clips is written."""
import pytest

from oracle import oracle as O
from test_gpu_failure import _refusing_writer
from test_gpu_search_direct import _configs, _frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dropped", [0, 3, 7])
@pytest.mark.parametrize("depth", [2, 4])
def test_refused_record(depth, dropped):
    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    n, sizes = 8, [(352, 288), (208, 112), (96, 64)]
    clips, records, headers, cfgs = [], [], [], []
    for w, h in sizes:
        gc, oc = _configs(w, h, 12, depth)
        o = O.OracleEncoder(oc)
        clips.append(_frames(w, h, n, w))
        rec = []
        for t, f in enumerate(clips[-1]):
            assert o.encode_rgb(f, 20 * t) == 0
            rec.append(o.last_record())
        records.append(rec)
        headers.append(bytearray(o.finish()[:36]))
        cfgs.append(gc)
    writers = [_refusing_writer(0), _refusing_writer(dropped + 2), _refusing_writer(0)]
    b = Batch.new(cfgs, writers)
    errors = 0
    for t in range(n):
        try:
            b.encode_step([c[t] for c in clips], [20 * t] * 3)
        except E.IoError:
            errors += 1
    try:
        b.finish()
    except E.IoError:
        errors += 1
    b.close()
    assert errors == 1
    headers[1][28:36] = (n - 1).to_bytes(8, "little")
    for i, wr in enumerate(writers):
        want = bytes(headers[i]) + b"".join(r for t, r in enumerate(records[i]) if i != 1 or t != dropped)
        assert bytes(wr.buf) == want
