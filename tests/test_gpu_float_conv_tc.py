"""xnor_b200_float_conv_tc (filters prepared once, K split over clusters, yolo activation) against an fp64 convolution."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import torch.nn.functional as F  # noqa: E402

import synth  # noqa: E402
from darknet_b200 import capi  # noqa: E402


@pytest.mark.parametrize("batch,c,h,w,n,size,leaky,entries", [
    (1, 32, 1, 1, 1, 1, 0, 0),          # one value
    (1, 5, 3, 5, 7, 1, 1, 0),           # less than one K block
    (1, 256, 5, 5, 18, 1, 0, 6),        # 8 K blocks: split 2
    (2, 416, 13, 10, 130, 1, 0, 65),    # 13 K blocks: split 3; tiles across images
    (1, 32, 11, 19, 40, 3, 1, 0),       # 9 K blocks: split 2
    (3, 64, 7, 9, 129, 3, 1, 0),        # 18 K blocks: split 4, halo rows of neighbouring images
    (40, 64, 16, 33, 16, 3, 0, 8),      # one wave full: no split
    (64, 512, 13, 13, 64, 3, 1, 0),     # 144 K blocks a tile, fewer tiles than SMs
    (113, 512, 13, 13, 40, 3, 1, 0),    # 150 tiles: a round of the SMs, and two whose K blocks go to clusters of four
    (150, 416, 13, 13, 130, 1, 0, 65), (64, 96, 31, 33, 33, 1, 1, 11), (9, 128, 40, 41, 129, 1, 1, 0), (9, 129, 40, 41, 129, 1, 0, 0),
                                        # several tiles an SM; 3 and 4 K blocks (each taken out by itself) and 5
    (1, 32, 32, 32, 130, 3, 0, 0), (1, 32, 25, 41, 130, 3, 0, 0),      # 1024 pixels and one more
    (9, 96, 13, 13, 425, 1, 0, 0), (150, 64, 13, 13, 240, 1, 1, 8), (150, 64, 13, 13, 241, 1, 1, 0), (150, 64, 13, 13, 257, 3, 1, 0),
    (113, 512, 13, 13, 144, 3, 1, 0),   # a last filter tile of 41, 112, 113, 1 and 16, the last with its K blocks dealt to clusters
    (2, 300, 23, 22, 33, 1, 1, 11), (3, 300, 19, 18, 33, 1, 1, 11),    # 1012 and 1026, K blocks that are not whole
])
def test_prepared_filters_match_fp64(batch, c, h, w, n, size, leaky, entries):
    seed = batch + c + h + n
    x = torch.from_numpy(synth.bell(seed, (batch, c, h, w))).cuda()
    wt = torch.from_numpy(synth.bell(seed + 1, (n, c, size, size), 0.05)).cuda()
    b = torch.from_numpy(synth.bell(seed + 2, (n,), 0.01)).cuda()
    want = F.conv2d(x.double(), wt.double(), b.double(), 1, size // 2)
    want = torch.where(want > 0, want, want * 0.1) if leaky else want
    if entries:
        logistic = torch.tensor([i not in (2, 3) for i in range(entries)] * (n // entries), device="cuda").view(1, n, 1, 1)
        want = torch.where(logistic, torch.sigmoid(want), want)
    desc = capi.ConvDesc(batch, c, h, w, n, size, 1, size // 2, capi.LEAKY if leaky else capi.LINEAR)
    lib, stream = capi.lib(), torch.cuda.current_stream().cuda_stream
    prepared = torch.empty(lib.xnor_b200_float_conv_tc_weights_bytes(C.byref(desc)) // 4, device="cuda")
    capi.check(lib.xnor_b200_float_conv_tc_prepare(C.byref(desc), wt.data_ptr(), prepared.data_ptr(), stream), "prepare")
    out = torch.full(want.shape, float("nan"), device="cuda")
    capi.check(lib.xnor_b200_float_conv_tc(C.byref(desc), x.data_ptr(), prepared.data_ptr(), b.data_ptr(), out.data_ptr(), entries, stream), "conv")
    err = (out.double() - want).abs().max().item()
    assert err <= 1e-5 + 4e-8 * c * size * size, err
    st = C.c_int(-1)
    capi.check(lib.xnor_b200_take_device_status(C.byref(st)), "xnor_b200_take_device_status")
    assert st.value == 0


def prepared_conv(kind, desc, x, wt, b, entries=0):
    lib, stream = capi.lib(), torch.cuda.current_stream().cuda_stream
    call = {"tc": lambda *a: lib.xnor_b200_float_conv_tc(*a[:-1], entries, a[-1]), "map": lib.xnor_b200_float_conv_map}[kind]
    nbytes = getattr(lib, f"xnor_b200_float_conv_{kind}_weights_bytes")(C.byref(desc))
    assert nbytes
    prepared = torch.empty(nbytes // 4, device="cuda")
    capi.check(getattr(lib, f"xnor_b200_float_conv_{kind}_prepare")(C.byref(desc), wt.data_ptr(), prepared.data_ptr(), stream), "prepare")
    out = torch.full((desc.batch, desc.n, desc.h, desc.w), float("nan"), device="cuda")
    capi.check(call(C.byref(desc), x.data_ptr(), prepared.data_ptr(), b.data_ptr(), out.data_ptr(), stream), "conv")
    return out


def fp64(x, wt, b):
    """The convolution as one matrix product an image, in 64 bits."""
    n, c, size, _ = wt.shape
    cols = F.unfold(x, size, padding=size // 2).double()
    return (wt.double().view(n, -1) @ cols + b.double().view(1, n, 1)).view(x.shape[0], n, *x.shape[2:])


@pytest.mark.parametrize("batch,c,h,w,n,size", [
    (2, 256, 13, 13, 512, 3), (3, 256, 11, 19, 512, 3), (16, 256, 7, 7, 512, 3), (1, 256, 19, 19, 512, 3), (4, 512, 13, 13, 255, 1), (1, 512, 28, 28, 255, 1),
    (1, 1024, 13, 13, 425, 1), (6, 1024, 13, 13, 425, 1), (1, 1024, 14, 14, 1000, 1), (8, 1024, 1, 1, 1000, 1),
    (8, 256, 13, 13, 512, 3), (64, 256, 13, 13, 512, 3), (9, 256, 11, 19, 512, 3), (32, 256, 7, 7, 512, 3), (16, 512, 13, 13, 128, 3),
])
def test_no_less_accurate_than_the_fp32_kernels(batch, c, h, w, n, size):
    """Against the small-map kernel where that one would run (up to 1024 pixels), against cuDNN's fp32 convolution beyond.  A tenth of
    the rounding of a single fp32 result (2^-24, 6e-8) is left for the draw of the values."""
    torch.backends.cudnn.allow_tf32 = False
    g = torch.Generator(device="cuda").manual_seed(batch + c + n)
    x = F.leaky_relu(torch.randn(batch, c, h, w, generator=g, device="cuda") * 3, 0.1)
    wt = torch.randn(n, c, size, size, generator=g, device="cuda") * (c * size * size) ** -0.5
    b = torch.randn(n, generator=g, device="cuda") * 0.01
    want = fp64(x, wt, b)

    def error(y):
        return float((y.double() - want).norm() / want.norm())
    desc = capi.ConvDesc(batch, c, h, w, n, size, 1, size // 2, capi.LINEAR)
    other = prepared_conv("map", desc, x, wt, b) if batch * h * w <= 1024 else F.conv2d(x, wt, b, 1, size // 2)
    assert error(prepared_conv("tc", desc, x, wt, b)) <= error(other) + 6e-9


@pytest.mark.parametrize("batch,c,h,w,n,size,bound", [
    # K blocks of a CTA, each sum taken out by itself: up to 4 of a 1x1 layer, up to 12 of a 3x3 one (9, 5, 12 of 36, 12 of 45)
    (9, 8, 13, 13, 128, 1, 2e-7), (9, 128, 40, 41, 129, 1, 2e-7), (24, 256, 13, 13, 128, 1, 2e-7),
    (64, 32, 13, 13, 512, 3, 2e-7), (9, 64, 13, 13, 128, 3, 2e-7), (24, 128, 13, 13, 128, 3, 2e-7), (9, 160, 13, 13, 128, 3, 2e-7),
    # by pairs: 5, 8 and 32, the last with its left-over tiles dealt to clusters of three; 18, 72 and 144
    (24, 160, 26, 26, 128, 1, 4.5e-7), (24, 256, 26, 26, 128, 1, 4.5e-7), (64, 1024, 13, 13, 425, 1, 4.5e-7),
    (64, 64, 13, 13, 512, 3, 4.5e-7), (64, 256, 13, 13, 512, 3, 4.5e-7), (113, 512, 13, 13, 40, 3, 4.5e-7),
])
def test_error_of_batches(batch, c, h, w, n, size, bound):
    """More than 1024 pixels.  One K block is twelve instructions into one accumulator: about 1.4e-7; two leave 3.3e-7 to 4.0e-7; sums that
    stay there whole 4.3e-7 at 5 (1x1), 5.5e-7 at 8 and 1.9e-6 at 32.  The bounds lie between."""
    g = torch.Generator(device="cuda").manual_seed(batch + c + n)
    x = F.leaky_relu(torch.randn(batch, c, h, w, generator=g, device="cuda") * 3, 0.1)
    wt = torch.randn(n, c, size, size, generator=g, device="cuda") * (c * size * size) ** -0.5
    b = torch.randn(n, generator=g, device="cuda") * 0.01
    want = torch.cat([fp64(x[i:i + 1], wt, b) for i in range(batch)])
    got = prepared_conv("tc", capi.ConvDesc(batch, c, h, w, n, size, 1, size // 2, capi.LINEAR), x, wt, b)
    assert float((got.double() - want).norm() / want.norm()) <= bound


@pytest.mark.parametrize("batch,c,h,w,n,size", [(2, 64, 9, 7, 140, 3), (9, 64, 13, 13, 33, 3), (2, 96, 9, 7, 140, 1), (64, 512, 13, 13, 32, 3),
                                                (9, 96, 13, 13, 140, 1), (9, 300, 13, 13, 33, 1)])
@pytest.mark.parametrize("leaky", [0, 1])
def test_infinite_and_huge_values(batch, c, h, w, n, size, leaky):
    """Infinities and NaN come out where plain arithmetic puts them, and values next to the largest lose nothing."""
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(batch, c, h, w, generator=g, device="cuda")
    wt = torch.randn(n, c, size, size, generator=g, device="cuda") * 0.05
    b = torch.randn(n, generator=g, device="cuda")
    x[:, 0].clamp_(-0.9, 0.9)                                  # no overflow of fp32 that 64 bits would not have
    x[0, 3, 1, 2], x[0, 5, 6, 6], x[1, 0, 0, 0], x[1, 7, 4, 3] = float("inf"), float("-inf"), float("nan"), 3.4e38
    wt[1, 2, 0, 0], wt[2, 1, size - 1, 0], wt[4, 0, 0, size - 1] = float("inf"), float("nan"), -3.4e38
    want = fp64(x, wt, b)
    want = torch.where(want > 0, want, want * 0.1) if leaky else want
    want32 = want.float()
    got = prepared_conv("tc", capi.ConvDesc(batch, c, h, w, n, size, 1, size // 2, capi.LEAKY if leaky else capi.LINEAR), x, wt, b)
    assert torch.equal(got.isnan(), want32.isnan()) and torch.equal(got.isinf(), want32.isinf())
    assert torch.equal(got[got.isinf()], want32[want32.isinf()])
    fine = want32.isfinite()
    assert bool(((got[fine] - want32[fine]).abs() <= 2e-5 + 2e-5 * want32[fine].abs()).all())


@pytest.mark.parametrize("batch,c,h,w,n,entries", [(2, 96, 9, 7, 34, 17), (9, 96, 13, 13, 34, 17), (9, 300, 13, 13, 255, 85)])
def test_infinite_and_huge_values_behind_the_logistic(batch, c, h, w, n, entries):
    """The [yolo] layer's step on values that are formed again: infinities become 0 and 1, but for width and height, and NaN stays."""
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(batch, c, h, w, generator=g, device="cuda")
    wt = torch.randn(n, c, 1, 1, generator=g, device="cuda") * 0.05
    b = torch.randn(n, generator=g, device="cuda")
    x[0, 3, 1, 2], x[0, 5, 6, 6], x[1, 0, 0, 0], x[1, 7, 4, 3] = float("inf"), float("-inf"), float("nan"), 3.4e38
    wt[2, 4], wt[3, 4], wt[5, 1] = float("inf"), float("-inf"), float("nan")
    want = fp64(x, wt, b).float().double()                     # the sum leaves fp32 where 64 bits would hold it
    logistic = torch.tensor([i not in (2, 3) for i in range(entries)] * (n // entries), device="cuda").view(1, n, 1, 1)
    want = torch.where(logistic, torch.sigmoid(want), want).float()
    got = prepared_conv("tc", capi.ConvDesc(batch, c, h, w, n, 1, 1, 0, capi.LINEAR), x, wt, b, entries)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and bool(want.isinf().any())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    fine = want.isfinite()
    assert bool(((got[fine] - want[fine]).abs() <= 2e-5 + 2e-5 * want[fine].abs()).all())
