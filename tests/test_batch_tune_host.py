"""What the multi-clip autotuner compares its candidates by (host only)."""
import ctypes as C

import pytest

from riv2_b200 import encoder as E
from riv2_b200.batch import STAGES


def _score(dim, **us):
    v = (C.c_float * 9)(*[us.get(k, 0.0) for k in STAGES[:9]])
    s = C.c_float()
    assert E.lib().riv_test_batch_tune_score(dim, v, C.byref(s)) == 0
    return s.value


def test_search_candidates_are_compared_by_the_whole_of_their_work():
    """A search from tables leaves the prediction to its own stage; the direct one makes it on the way."""
    table = _score(0, sad_table=300, search=900, predict=220, residual=7, deblock=8)
    direct = _score(0, search=1270, residual=9, deblock=5)
    assert direct < table and table == 1420


@pytest.mark.parametrize("dim,stage", [(1, "residual"), (2, "deblock")])
def test_other_dimensions_are_one_stage(dim, stage):
    assert _score(dim, **{k: 1.0 for k in STAGES[:9] if k != stage}, **{stage: 5.0}) == 5.0
