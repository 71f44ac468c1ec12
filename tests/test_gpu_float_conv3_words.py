"""xnor_b200_float_conv3_words (signs of the first convolution on the position grid) and the sign masks against the fp32 output,
with sums and biases that are exactly zero: zero is not positive, whatever its sign."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import torch.nn.functional as F  # noqa: E402

from darknet_b200 import capi, layer as L  # noqa: E402


@pytest.mark.parametrize("pool", [0, 2])
@pytest.mark.parametrize("batch,h,w,n,pitch", [(1, 32, 32, 32, 0), (2, 34, 30, 16, 0), (1, 2, 2, 8, 0), (3, 64, 96, 20, 56), (40, 96, 98, 32, 104)])
def test_signs_of_zero_sums_and_zero_biases(batch, h, w, n, pitch, pool):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + h)
    x = torch.randint(0, 3, (batch, 3, h, w), generator=g, device="cuda").float() / 4
    wt = torch.randint(-1, 2, (n, 27), generator=g, device="cuda").float() / 4
    b = torch.randint(-1, 2, (n,), generator=g, device="cuda").float() / 8
    b[::3] = -0.0
    desc = capi.ConvDesc(batch, 3, h, w, n, 3, 1, 1, capi.LEAKY)
    oh, ow = (h // 2, w // 2) if pool else (h, w)
    if not pool and pitch:
        pitch = ow + 8
    grid = L.GridWords(batch, n, oh, ow, pitch)
    capi.check(capi.lib().xnor_b200_float_conv3_words(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), grid.words.data_ptr(),
                                                     grid.pitch, None), "conv3_words")
    masks = torch.zeros(batch, oh, ow, (n + 7) // 8, dtype=torch.uint8, device="cuda")
    capi.check(capi.lib().xnor_b200_float_conv3_io(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), None, None,
                                                  masks.data_ptr(), None), "conv3_io")
    y = F.conv2d(x.double(), wt.double().view(n, 3, 3, 3), b.double(), 1, 1)
    y = F.max_pool2d(y, 2, 2) if pool else y
    assert int((y == 0).sum()) > 0 or y.numel() < 64
    bits = F.pad(y > 0, (0, 0, 0, 0, 0, 32 - n)).to(torch.int64)
    want = (bits << torch.arange(32, device="cuda").view(1, 32, 1, 1)).sum(1)
    front = capi.lib().xnor_b200_grid_front(grid.pitch)
    body = grid.words[0, front:front + batch * (oh + 1) * grid.pitch].view(batch, oh + 1, grid.pitch).to(torch.int64) & 0xFFFFFFFF
    assert torch.equal(body[:, :oh, :ow], want)
    assert int(body[:, oh].sum()) == 0 and int(body[:, :, ow:].sum()) == 0
    got = sum(masks[..., i].to(torch.int64) << (8 * i) for i in range(masks.shape[-1]))
    assert torch.equal(got, want)


@pytest.mark.parametrize("pool,n", [(2, 16), (0, 32)])
@pytest.mark.parametrize("x_scale,w_scale", [(1.0, 1.0), (1e6, 1.0), (1e-7, 1.0), (1.0, 1e-9), (255.0, 1e5), (1.0, 1e33)])
def test_signs_at_every_scale(x_scale, w_scale, pool, n):
    """Values that fp16 cannot hold, or holds with few bits, still get the sign of the fp32 sum (the masks, formed in fp32)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    x = torch.randn(2, 3, 70, 90, generator=g, device="cuda") * x_scale
    wt = torch.randn(n, 27, generator=g, device="cuda") * w_scale
    wt[1] = 0.0
    b = torch.randn(n, generator=g, device="cuda") * (0.3 * x_scale * w_scale)
    b[2] = 1e30
    desc = capi.ConvDesc(2, 3, 70, 90, n, 3, 1, 1, capi.LINEAR)
    oh, ow = (35, 45) if pool else (70, 90)
    grid = L.GridWords(2, n, oh, ow)
    masks = torch.zeros(2, oh, ow, n // 8, dtype=torch.uint8, device="cuda")
    capi.check(capi.lib().xnor_b200_float_conv3_words(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), grid.words.data_ptr(), 0, None), "words")
    capi.check(capi.lib().xnor_b200_float_conv3_io(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), None, None, masks.data_ptr(), None), "io")
    front = capi.lib().xnor_b200_grid_front(ow + 1)
    body = grid.words[0, front:front + 2 * (oh + 1) * (ow + 1)].view(2, oh + 1, ow + 1)[:, :oh, :ow].to(torch.int64) & 0xFFFFFFFF
    assert torch.equal(body, sum(masks[..., i].to(torch.int64) << (8 * i) for i in range(n // 8)))


@pytest.mark.parametrize("batch,h,w,n,pool", [
    (1, 2048, 2048, 32, 0), (1, 2048, 2112, 17, 0), (1, 2048, 2048, 32, 2), (1, 2048, 2200, 24, 2), (1, 512, 3000, 32, 0),     # the widest windows
    (1, 33, 35, 32, 0), (2, 17, 64, 16, 0), (3, 40, 41, 20, 0), (1, 1, 7, 8, 0), (1, 5, 3, 32, 0), (2, 101, 1999, 32, 0),      # odd rows and columns
])
def test_signs_at_the_widest_and_at_odd_sizes(batch, h, w, n, pool):
    g = torch.Generator(device="cuda")
    g.manual_seed(h + w)
    x = torch.randn(batch, 3, h, w, generator=g, device="cuda")
    wt, b = torch.randn(n, 27, generator=g, device="cuda"), torch.randn(n, generator=g, device="cuda")
    desc = capi.ConvDesc(batch, 3, h, w, n, 3, 1, 1, capi.LINEAR)
    oh, ow = (h // 2, w // 2) if pool else (h, w)
    grid = L.GridWords(batch, n, oh, ow)
    masks = torch.zeros(batch, oh, ow, (n + 7) // 8, dtype=torch.uint8, device="cuda")
    capi.check(capi.lib().xnor_b200_float_conv3_words(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), grid.words.data_ptr(), 0, None), "words")
    capi.check(capi.lib().xnor_b200_float_conv3_io(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), None, None, masks.data_ptr(), None), "io")
    front = capi.lib().xnor_b200_grid_front(ow + 1)
    body = grid.words[0, front:front + batch * (oh + 1) * (ow + 1)].view(batch, oh + 1, ow + 1).to(torch.int64) & 0xFFFFFFFF
    assert torch.equal(body[:, :oh, :ow], sum(masks[..., i].to(torch.int64) << (8 * i) for i in range(masks.shape[-1])))
    assert int(body[:, oh].sum()) == 0 and int(body[:, :, ow:].sum()) == 0
    y = F.conv2d(x.double(), wt.double().view(n, 3, 3, 3), b.double(), 1, 1)
    y = F.max_pool2d(y, 2, 2) if pool else y
    sure = y.abs() > 1e-4                                      # 27 fp32 products of magnitude a few
    bits = (body[:, None, :oh, :ow] >> torch.arange(n, device="cuda").view(1, n, 1, 1)) & 1
    assert torch.equal(bits.bool()[sure], (y > 0)[sure])


@pytest.mark.parametrize("pool,n", [(2, 16), (0, 32)])
@pytest.mark.parametrize("value,top", [(0.5 + 2 ** -12, 0.9), (0.5 + 2 ** -12, 1.0), (0.75 + 2 ** -12 - 2 ** -24, 0.75 + 2 ** -12 - 2 ** -24), (1.0 + 2 ** -11, 1.5), (1.0 + 2 ** -11, 1.0 + 2 ** -11),
                                       (1.0 + 2 ** -11 - 2 ** -23, 1.0), (1.998, 2.0), (2.0 + 2 ** -10, 2.0), (0.3, 3.0e4)])
def test_signs_where_rounding_takes_as_much_as_it_can(value, top, pool, n):
    """Every input off by about half an fp16 unit the same way, and biases that leave next to nothing of the sum, on either side of zero."""
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    h, w = 40, 44
    x = torch.full((1, 3, h, w), value, device="cuda")
    x[0, 1, 7, 9] = top
    wt = (torch.rand(n, 27, generator=g, device="cuda") + 0.5) * torch.tensor([1.0, -1.0], device="cuda").repeat(n // 2)[:, None]
    desc = capi.ConvDesc(1, 3, h, w, n, 3, 1, 1, capi.LINEAR)
    lib, stream = capi.lib(), torch.cuda.current_stream().cuda_stream
    y = torch.empty(1, n, h, w, device="cuda")
    zero = torch.zeros(n, device="cuda")
    capi.check(lib.xnor_b200_float_conv3_io(C.byref(desc), 0, x.data_ptr(), wt.data_ptr(), zero.data_ptr(), y.data_ptr(), None, None, stream), "io")
    oh, ow = (h // 2, w // 2) if pool else (h, w)
    for off in (1e-6, -1e-6, 3e-5, -3e-5, 2e-4, -2e-4, 4e-4, -4e-4):
        b = -y[0, :, 20, 20] * (1.0 + off)
        grid = L.GridWords(1, n, oh, ow)
        masks = torch.zeros(1, oh, ow, n // 8, dtype=torch.uint8, device="cuda")
        capi.check(lib.xnor_b200_float_conv3_words(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), grid.words.data_ptr(), 0, stream), "words")
        capi.check(lib.xnor_b200_float_conv3_io(C.byref(desc), pool, x.data_ptr(), wt.data_ptr(), b.data_ptr(), None, None, masks.data_ptr(), stream), "io")
        front = lib.xnor_b200_grid_front(ow + 1)
        body = grid.words[0, front:front + (oh + 1) * (ow + 1)].view(1, oh + 1, ow + 1)[:, :oh, :ow].to(torch.int64) & 0xFFFFFFFF
        assert torch.equal(body, sum(masks[..., i].to(torch.int64) << (8 * i) for i in range(n // 8))), off
