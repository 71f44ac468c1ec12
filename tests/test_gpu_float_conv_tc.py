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
