"""The training kernels' data movement at the sizes where their vector forms end: row lengths that
are and are not a multiple of the 8 elements of a 16-byte store, tiles that are cut short, buffers
off a 16-byte boundary.  Reference: plain PyTorch on the same values."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

HIN = {1: 24, 2: 12, 3: 6, 4: 6}
HOUT = {1: 12, 2: 6, 3: 6, 4: 3}
STRIDE = {1: 2, 2: 2, 3: 1, 4: 2}


def _env():
    import torch

    from riv2_b200 import proposal as P
    return torch, P.lib(), torch.device("cuda")


def _off(torch, shape, dtype, dev, off):
    """A contiguous tensor that starts `off` elements into its allocation."""
    n = 1
    for k in shape:
        n *= k
    return torch.empty(n + off, dtype=dtype, device=dev)[off:].view(shape)


def _cols(torch, x, layer):
    """(n, hin, hin, c) -> (9, c, n * hout^2): taps of the zero-padded input."""
    n, _, _, c = x.shape
    ho, s = HOUT[layer], STRIDE[layer]
    pad = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    t = [pad[:, ky:ky + s * ho:s, kx:kx + s * ho:s][:, :ho, :ho] for ky in range(3) for kx in range(3)]
    return torch.stack(t).permute(0, 4, 1, 2, 3).reshape(9, c, n * ho * ho)


@pytest.mark.parametrize("off", [0, 2])
@pytest.mark.parametrize("n", [1, 3, 7, 8, 65])
@pytest.mark.parametrize("layer", [1, 2, 3, 4])
def test_im2col_t(layer, n, off):
    torch, L, dev = _env()
    h, c = HIN[layer], 2 if layer == 1 else 32
    kp, m = (32 if layer == 1 else 320), n * HOUT[layer] ** 2
    g = torch.Generator(device="cpu").manual_seed(layer * 100 + n)
    x = _off(torch, (n, h, h, c), torch.bfloat16, dev, off)
    x.copy_(torch.randn((n, h, h, c), generator=g))
    out = _off(torch, (kp, m), torch.bfloat16, dev, off)
    out.fill_(7.0)
    assert L.riv_nn_im2col_t(layer, x.data_ptr(), h * h * c, n, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    want = torch.zeros((kp, m), dtype=torch.bfloat16, device=dev)
    want[:9 * c] = _cols(torch, x, layer).reshape(9 * c, m)
    assert torch.equal(out, want)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 8, 65])
@pytest.mark.parametrize("layer", [2, 3, 4])
def test_col2im(layer, n, off):
    torch, L, dev = _env()
    h, ho, s = HIN[layer], HOUT[layer], STRIDE[layer]
    m, mi = n * ho * ho, n * h * h
    g = torch.Generator(device="cpu").manual_seed(layer * 100 + n)
    dcol = _off(torch, (m, 320), torch.float32, dev, off)
    dcol.copy_(torch.randn((m, 320), generator=g))
    act = _off(torch, (n, h, h, 32), torch.bfloat16, dev, off)
    act.copy_(torch.relu(torch.randn((n, h, h, 32), generator=g)))
    dz = _off(torch, (mi, 32), torch.bfloat16, dev, off)
    dzt = _off(torch, (32, mi), torch.bfloat16, dev, off)
    assert L.riv_nn_col2im(layer, dcol.data_ptr(), n, act.data_ptr(), h * h * 32, dz.data_ptr(), dzt.data_ptr(), None) == 0
    torch.cuda.synchronize()
    d = dcol[:, :288].double().reshape(n, ho, ho, 9, 32)
    acc = torch.zeros((2, n, h + 2, h + 2, 32), dtype=torch.float64, device=dev)
    for t in range(9):
        for k, v in enumerate((d[:, :, :, t], d[:, :, :, t].abs())):
            acc[k, :, t // 3:t // 3 + s * ho:s, t % 3:t % 3 + s * ho:s][:, :ho, :ho] += v
    keep = (act > 0).double()
    want, mag = (acc[k, :, 1:-1, 1:-1] * keep for k in (0, 1))
    # nine f32 additions, then one rounding to bf16 (half a unit in the last place: 2^-9)
    err = (dz.double().reshape(n, h, h, 32) - want).abs()
    assert bool((err <= want.abs() * 2.0 ** -8 + mag * 9 * 2.0 ** -24).all())
    assert torch.equal(dzt, dz.T)


@pytest.mark.parametrize("rows,n,grp", [(1, 32, 1), (63, 128, 1), (64, 40, 1), (72, 32, 9), (585, 32, 9)])
def test_relu_bwd(rows, n, grp):
    torch, L, dev = _env()
    g = torch.Generator(device="cpu").manual_seed(rows)
    ldd = lda = 320 if grp > 1 else n
    groups = (rows + grp - 1) // grp
    d = torch.randn((groups, ldd), generator=g).to(dev)
    act = torch.relu(torch.randn((groups, lda), generator=g)).to(torch.bfloat16).to(dev)
    dz = torch.empty((rows, n), dtype=torch.bfloat16, device=dev)
    dzt = torch.empty((n, rows), dtype=torch.bfloat16, device=dev)
    assert L.riv_nn_relu_bwd(d.data_ptr(), ldd, act.data_ptr(), lda, rows, n, grp, dz.data_ptr(), dzt.data_ptr(), None) == 0
    torch.cuda.synchronize()
    pick = lambda t: t[:, :grp * n].reshape(groups * grp, n)[:rows]  # noqa: E731
    want = torch.where(pick(act) > 0, pick(d), torch.zeros((), device=dev)).to(torch.bfloat16)
    assert torch.equal(dz, want) and torch.equal(dzt, want.T)


@pytest.mark.parametrize("rows,n,ld", [(1, 32, 32), (5, 16, 32), (1000, 100, 128), (4096, 128, 128), (70001, 32, 32)])
def test_colsum(rows, n, ld):
    torch, L, dev = _env()
    g = torch.Generator(device="cpu").manual_seed(rows)
    z = torch.randn((rows, ld), generator=g).to(torch.bfloat16).to(dev)
    out = torch.ones(n, device=dev)
    assert L.riv_nn_colsum(z.data_ptr(), ld, C.c_longlong(rows), n, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    want = 1.0 + z[:, :n].double().sum(0)
    # f32 sums: at most `rows` roundings of 2^-24 of the sum of magnitudes
    assert bool(((out.double() - want).abs() <= (1.0 + z[:, :n].double().abs().sum(0)) * rows * 2.0 ** -24 + 2.0 ** -23).all())


@pytest.mark.parametrize("rows,n,ld", [(1, 32, 32), (513, 32, 32), (1000, 100, 128), (5003, 100, 128), (70001, 32, 32),
                                       (296 * 512, 32, 32), (296 * 512 + 37, 32, 32), (589824, 32, 32)])
def test_colsum_is_exact_for_small_integers(rows, n, ld):
    """Values in -3 .. 3 sum exactly in f32 in any order: a lost or doubled row shows.  296 * 512 rows is
    where the CTAs reach their largest number (16 bytes a load), 296 * 16 with single elements."""
    torch, L, dev = _env()
    g = torch.Generator(device="cpu").manual_seed(rows)
    z = torch.randint(-3, 4, (rows, ld), generator=g).to(torch.bfloat16).to(dev)
    z[-1] = 3.0
    out = torch.ones(n, device=dev)
    assert L.riv_nn_colsum(z.data_ptr(), ld, C.c_longlong(rows), n, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out.double(), 1.0 + z[:, :n].double().sum(0))
