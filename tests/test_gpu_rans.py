"""rANS batches coded on the GPU against the host's coder (which the oracle pins): the same bytes at
the edges of its 64-symbol steps and 16386-symbol batches, over all frequencies and at the extremes
of a state's growth (the rarest symbols) and of its renormalisation (the most frequent ones)."""
import numpy as np
import pytest

from riv2_b200 import encoder as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["any", "likely", "rarest", "bypass"])
@pytest.mark.parametrize("n", [0, 1, 2, 63, 64, 65, 127, 129, 16385, 16386, 16387, 32773, 70001])
def test_matches_host(n, kind):
    r = np.random.default_rng(n)
    p = r.integers(0, 256, n)
    if kind == "any":
        bit = r.integers(0, 2, n)
    elif kind == "likely":
        bit = (r.random(n) * 256 >= p).astype(np.int64)
    elif kind == "rarest":
        bit = r.integers(0, 2, n)
        p = np.where(bit == 1, 255, r.integers(0, 2, n))
    else:
        p, bit = np.full(n, 128), r.integers(0, 2, n)
    s = (p | bit << 8).astype(np.uint16)
    assert E.rans_stream(s, True) == E.rans_stream(s, False)
