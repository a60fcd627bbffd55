"""The symbol kernels' limits at frames beyond 32 bits of symbols (host only: such a frame's total must
never pass for one that fits the stacks)."""
import ctypes as C

import numpy as np
import pytest

from riv2_b200 import encoder as E

BATCH = 16386   # symbols of a rANS batch
MOST = 384 * 27  # symbols of a macroblock at most


def _room(nmb, counts=()):
    c = np.asarray(counts, dtype=np.uint32)
    room, total = C.c_uint32(), C.c_uint32()
    assert E.lib().riv_test_symbol_room(C.c_uint64(nmb), c.ctypes.data_as(C.POINTER(C.c_uint32)), c.size, C.byref(room), C.byref(total)) == 0
    return room.value, total.value


@pytest.mark.parametrize("nmb", [1, 396, 8160, 32400, 1 << 20, 1 << 22, 1 << 23, 1 << 24])
def test_room(nmb):
    """Whole batches, positions of 31 bits."""
    room = _room(nmb)[0]
    assert room % BATCH == 0 and 0 < room < 1 << 31
    assert room == min(-(-nmb * 512 // BATCH) * BATCH, (1 << 31) // BATCH * BATCH)


@pytest.mark.parametrize("nmb", [414251, 414253, 1 << 20, 1 << 24])
def test_totals_do_not_wrap(nmb):
    """Counts of CTAs of 16 macroblocks, every macroblock with the most symbols there are."""
    room, total = _room(nmb, np.full(nmb // 16, 16 * MOST))
    assert total == min(nmb // 16 * 16 * MOST, 2 ** 32 - 1)
    assert total > room
