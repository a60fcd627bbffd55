"""Stage times of multi-clip steps."""
import pytest

from test_gpu_search_direct import _configs

pytestmark = pytest.mark.gpu


def test_conversion_is_timed():
    """16 clips of 1080p read 99.5 MB of RGB and write 50.1 MB of planes: 18 us at 8 TB/s, more than
    the GPU's memory has.  Steps 0 and 8 are timed (fixed shapes); before step 8 the GPU is busy with the
    steps ahead, so that the stages hardly wait for its conversion, which is over by then."""
    import torch

    from riv2_b200 import encoder as E
    from riv2_b200.batch import Batch
    w, h, n = 1920, 1080, 16
    g = torch.Generator(device="cuda").manual_seed(1)
    frames = torch.randint(0, 256, (n, h, w, 3), dtype=torch.uint8, device="cuda", generator=g)
    ptrs = [f.data_ptr() for f in frames]
    torch.cuda.synchronize()
    b = Batch.new([_configs(w, h, 12, 10, 50, 20)[0]] * n, [E.VecWriter() for _ in range(n)])
    b.set_tune(100, 4, 128, 0)
    b.encode_step_device(ptrs, [0] * n)
    b.finish()
    first = b.counters()
    for t in range(1, 9):
        b.encode_step_device(ptrs, [20 * t] * n)
    b.finish()
    both = b.counters()
    b.close()
    assert (first["timed_steps"], both["timed_steps"]) == (1, 2)
    us = {k: 2 * v - first["stage_us"][k] for k, v in both["stage_us"].items()}
    assert us["convert"] >= 18.0
    assert sum(v for k, v in us.items() if k not in ("convert", "step")) <= us["step"] * 1.01
