"""xnor_b200_conv_words (convolution straight from sign words) against the packed-operand route, which the oracle pins: sizes at
the edges of its tiles (128 positions, 32 / 64 / 128 filters, stages of channel blocks), every kind of source and of output."""
import pytest

import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import torch.nn.functional as F  # noqa: E402

from darknet_b200 import capi, layer as L  # noqa: E402


def build(batch, c, h, w, n, ks, stride, leaky, seed):
    x, wt, b = synth.conv_case(seed, batch, c, h, w, n, ks)
    l = L.make_convolutional_layer(batch, h, w, c, n, ks, stride, ks // 2, capi.LEAKY if leaky else capi.LINEAR)
    l.load_weights(torch.from_numpy(wt).cuda(), torch.from_numpy(b).cuda())
    L.binary_align_weights(l)
    return l, torch.from_numpy(x).cuda()


def reference(l, x):
    capi.set_tuning(gemm_route=capi.ROUTE_TILED)                    # the packed-operand route, pinned
    try:
        return L.forward_convolutional_layer_gpu(l, x).clone()
    finally:
        capi.set_tuning()


def signs_of(y, pitch=0):
    """Grid words of y, made by torch."""
    b, n, h, w = y.shape
    nb = (n + 31) // 32
    bits = F.pad(y > 0, (0, 0, 0, 0, 0, 32 * nb - n)).reshape(b, nb, 32, h, w).to(torch.int64)
    words = (bits << torch.arange(32, device=y.device).view(1, 1, 32, 1, 1)).sum(2)
    pitch = pitch or w + 1
    grid = F.pad(words, (0, pitch - w, 0, 1)).permute(1, 0, 2, 3).reshape(nb, -1)
    front, total = capi.lib().xnor_b200_grid_front(pitch), capi.lib().xnor_b200_grid_block_words(b, h, pitch)
    return F.pad(grid, (front, total - front - grid.shape[1]))


def unsigned(grid):
    return grid.words.to(torch.int64) & 0xFFFFFFFF


CASES = [
    # batch, c, h, w, n, ks, stride
    (1, 32, 1, 1, 32, 3, 1), (1, 32, 7, 9, 32, 3, 1), (2, 64, 13, 13, 96, 3, 1), (3, 256, 26, 26, 160, 3, 1), (1, 512, 13, 13, 1024, 3, 1),
    (2, 16, 40, 31, 32, 3, 1), (2, 75, 52, 52, 64, 3, 1), (1, 3, 33, 5, 8, 3, 1), (5, 97, 10, 6, 33, 3, 1), (40, 96, 13, 13, 128, 3, 1),
    (16, 1024, 14, 14, 1024, 3, 1), (32, 768, 13, 13, 512, 3, 1), (4, 32, 150, 208, 64, 3, 1), (2, 32, 5, 300, 32, 3, 1), (64, 32, 26, 26, 64, 3, 1),
    (1, 32, 16, 16, 64, 3, 2), (2, 64, 15, 13, 128, 3, 2), (3, 128, 28, 28, 256, 3, 2), (1, 512, 28, 28, 512, 3, 2), (2, 40, 9, 8, 17, 3, 2),
    (1, 32, 8, 16, 32, 1, 1), (1, 1024, 13, 13, 256, 1, 1), (7, 64, 11, 9, 33, 1, 1), (2, 50, 20, 20, 70, 1, 1), (64, 256, 14, 14, 128, 1, 1),
    (2, 64, 9, 7, 32, 1, 2), (1, 288, 28, 28, 64, 1, 2),
    # one or two tiles a CTA, whose filters the epilogue warps share; 16 channels and fewer
    (1, 64, 26, 26, 96, 3, 1), (1, 128, 14, 14, 40, 3, 1), (1, 64, 30, 31, 72, 1, 1), (1, 32, 56, 56, 200, 3, 1), (1, 96, 120, 120, 64, 3, 1),
    (1, 16, 7, 9, 32, 3, 1), (3, 16, 208, 33, 32, 3, 1), (2, 9, 30, 62, 64, 3, 1), (1, 16, 1, 1, 160, 3, 1), (64, 15, 26, 26, 33, 3, 1), (2, 17, 20, 20, 32, 3, 1),
    # the last unit begins in the padding row, whose rows of the source lie behind its end
    (1, 40, 7, 51, 32, 1, 2), (1, 40, 15, 27, 32, 1, 2), (1, 16, 1, 207, 32, 1, 2), (1, 64, 31, 127, 32, 3, 2),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d_c%d_%dx%d_n%d_k%d_s%d" % c)
def test_conv_words_equals_the_packed_route(case):
    batch, c, h, w, n, ks, stride = case
    l, x = build(*case, leaky=True, seed=11 + c + n)
    want = reference(l, x)
    wts = L.conv_words_weights(l)
    words = L.sign_words(x)
    assert torch.equal(unsigned(words), signs_of(x))
    src = [words.source()]
    out = torch.full_like(want, float("nan"))
    L.conv_words(l, wts, src, output=out)
    assert torch.equal(out, want)
    sc = torch.randn_like(want)
    out2, total = torch.full_like(want, float("nan")), torch.full_like(want, float("nan"))
    L.conv_words(l, wts, src, output=out2, shortcut_in=sc, shortcut_out=total)
    assert torch.equal(out2, want) and torch.equal(total, sc + want)
    for pitch in (0, l.out_w // 8 * 8 + 8, l.out_w + 3) if n % 32 == 0 else ():
        signs = L.GridWords(batch, n, l.out_h, l.out_w, pitch)
        L.conv_words(l, wts, src, signs=signs)
        assert torch.equal(unsigned(signs), signs_of(want, signs.pitch))
        signs.words.zero_()
        L.conv_words(l, wts, src, output=out.zero_(), signs=signs)
        assert torch.equal(out, want) and torch.equal(unsigned(signs), signs_of(want, signs.pitch))
        signs.words.zero_()
        L.conv_words(l, wts, src, shortcut_in=sc, shortcut_out=total.zero_(), signs=signs)
        assert torch.equal(total, sc + want) and torch.equal(unsigned(signs), signs_of(sc + want, signs.pitch))
    for pitch in (w // 8 * 8 + 8, w + 2):
        if pitch <= 2 * w + 8:
            words = L.sign_words(x, pitch)
            assert torch.equal(unsigned(words), signs_of(x, pitch))
            L.conv_words(l, wts, [words.source()], output=out.zero_(), pitch=pitch if stride == 1 else 0)
            assert torch.equal(out, want)
    status = capi.C.c_int(-1)
    capi.check(capi.lib().xnor_b200_take_device_status(capi.C.byref(status)), "status")
    assert status.value == 0


@pytest.mark.parametrize("ks", [3, 1])
@pytest.mark.parametrize("c,h,w,pool", [(64, 26, 26, (2, 1)), (64, 14, 18, (2, 0)), (96, 13, 13, (1, 1)), (16, 32, 34, (2, 1)), (8, 17, 16, (1, 1))])
def test_pooled_sources(ks, c, h, w, pool):
    stride, pad = pool
    oh, ow = (h + pad - 2) // stride + 1, (w + pad - 2) // stride + 1
    l, _ = build(2, c, oh, ow, 64, ks, 1, False, 5)
    x = torch.from_numpy(synth.bell(3, (2, c, h, w))).cuda()
    padded = F.pad(x, (0, max((ow - 1) * stride + 2 - w, 0), 0, max((oh - 1) * stride + 2 - h, 0)), value=float("-inf"))
    want = reference(l, F.max_pool2d(padded, 2, stride)[:, :, :oh, :ow].contiguous())
    wts = L.conv_words_weights(l)
    out = torch.full_like(want, float("nan"))
    words = L.sign_words(x)
    L.conv_words(l, wts, [words.source(pool_stride=stride, pool_pad=pad)], output=out)
    assert torch.equal(out, want)


@pytest.mark.parametrize("ks,n", [(3, 256), (1, 32)])
@pytest.mark.parametrize("c1,c2", [(128, 256), (32, 32), (96, 64)])
def test_concatenated_sources(ks, n, c1, c2):
    """The [route] of yolov3-tiny: an upsampled tensor and a full-resolution one side by side."""
    l, _ = build(2, c1 + c2, 26, 26, n, ks, 1, True, 9)
    a = torch.from_numpy(synth.bell(4, (2, c1, 13, 13))).cuda()
    b = torch.from_numpy(synth.bell(5, (2, c2, 26, 26))).cuda()
    want = reference(l, torch.cat([F.interpolate(a, scale_factor=2, mode="nearest"), b], 1).contiguous())
    out = torch.full_like(want, float("nan"))
    wa, wb = L.sign_words(a), L.sign_words(b)
    L.conv_words(l, L.conv_words_weights(l), [wa.source(upsample=2), wb.source()], output=out)
    assert torch.equal(out, want)


def test_argument_checks():
    l, x = build(1, 64, 8, 8, 40, 3, 1, True, 2)
    wts, words = L.conv_words_weights(l), L.sign_words(x)
    out = torch.empty(1, 40, 8, 8, device="cuda")
    signs = L.GridWords(1, 64, 8, 8)
    for kw, match in ((dict(signs=signs), "invalid"), (dict(), "NULL"), (dict(output=out, shortcut_out=out), "NULL")):
        with pytest.raises(capi.XnorError, match=match):
            L.conv_words(l, wts, [words.source()], **kw)
    with pytest.raises(capi.XnorError, match="invalid"):
        L.conv_words(l, wts, [L.GridWords(1, 64, 8, 4).source()], output=out)
    five, _ = build(1, 32, 8, 8, 32, 5, 1, True, 2)
    assert L.conv_words_weights(five) is None


def test_a_wait_that_runs_out_is_reported():
    l, x = build(1, 64, 13, 13, 64, 3, 1, True, 2)
    wts, words = L.conv_words_weights(l), L.sign_words(x)
    want, out = reference(l, x), torch.empty(1, 64, 13, 13, device="cuda")
    status = capi.C.c_int(-1)
    capi.set_tuning(tc_wait_polls=4000, tc_withhold_arrival=1)
    try:
        L.conv_words(l, wts, [words.source()], output=out)
        capi.check(capi.lib().xnor_b200_take_device_status(capi.C.byref(status)), "status")
        assert status.value == 1
    finally:
        capi.set_tuning()
    L.conv_words(l, wts, [words.source()], output=out)
    capi.check(capi.lib().xnor_b200_take_device_status(capi.C.byref(status)), "status")
    assert status.value == 0 and torch.equal(out, want)


@pytest.mark.parametrize("case", [
    (2, 32, 5, 702, 32, 3, 1), (2, 32, 5, 703, 32, 3, 1), (1, 64, 3, 1408, 64, 3, 1), (1, 512, 2, 700, 64, 3, 1),
    (1, 64, 5, 850, 64, 3, 2), (1, 64, 5, 851, 64, 3, 2), (1, 64, 4, 1500, 32, 3, 2), (1, 1024, 3, 321, 32, 3, 2), (1, 1024, 3, 322, 32, 3, 2),
    (1, 64, 3, 2246, 32, 1, 2), (1, 64, 3, 2247, 32, 1, 2), (1, 64, 2, 3000, 32, 1, 1), (1, 32, 5, 5, 148 * 128 + 32, 3, 1),
], ids=lambda c: "b%d_c%d_%dx%d_n%d_k%d_s%d" % c)
def test_layers_at_the_widest_maps_and_beyond(case):
    """Where the kernel has no plan the layer keeps the packed route."""
    l, x = build(*case, leaky=True, seed=4)
    want = reference(l, x)
    l.output_gpu.fill_(float("nan"))
    assert torch.equal(L.forward_convolutional_layer_gpu(l, x), want)
    wts = L.conv_words_weights(l)
    assert (wts is None) == (case[3] in (703, 1408, 851, 1500, 322, 2247) or case[4] > 148 * 128)
    if wts is not None:
        out = torch.full_like(want, float("nan"))
        words = L.sign_words(x)
        L.conv_words(l, wts, [words.source()], output=out)
        assert torch.equal(out, want)


def test_layers_of_a_network_walk_a_large_batch_in_turn():
    """Inside one xnor_b200_run_ops call every second layer that writes large fp32 tensors begins at the batch's end: the same values,
    with a plain window, through the window table (stride 2, a pool) and with a shortcut, over a batch that ends within a unit."""
    batch, n, h, w = 5, 128, 100, 151
    ops, checks = [], []
    sc = torch.randn(batch, n, h, w, device="cuda")
    for i, (c, ks, stride, pool, shortcut) in enumerate([(32, 3, 1, 0, False), (32, 3, 1, 0, True), (64, 3, 2, 0, False), (32, 3, 1, 2, True), (40, 1, 1, 0, False), (32, 3, 2, 0, True)]):
        l, _ = build(batch, c, h * stride, w * stride, n, ks, stride, True, 20 + i)
        src = L.sign_words(torch.randn(batch, c, h * stride * max(pool, 1), w * stride * max(pool, 1), device="cuda"))
        wts = L.conv_words_weights(l)
        got, want = (torch.full((batch, n, h, w), float("nan"), device="cuda") for _ in range(2))
        signs, want_signs = L.GridWords(batch, n, h, w), L.GridWords(batch, n, h, w)
        assert got.numel() * 4 > 32 << 20
        kw = dict(shortcut_in=sc, shortcut_out=want) if shortcut else dict(output=want)
        L.conv_words(l, wts, [src.source(pool, 1 if pool else 0)], signs=want_signs, **kw)
        op = capi.Op(kind=capi.OP_CONV_WORDS, desc=l.desc, weights=wts.data_ptr(), mean_arr=l.mean_arr_gpu.data_ptr(), biases=l.biases_gpu.data_ptr())
        op.io.n_sources, op.io.sources[0], op.io.pitch = 1, src.source(pool, 1 if pool else 0), signs.pitch
        if shortcut:
            op.io.shortcut_in, op.io.shortcut_out, op.io.shortcut_signs = sc.data_ptr(), got.data_ptr(), signs.words.data_ptr()
        else:
            op.io.output, op.io.output_signs = got.data_ptr(), signs.words.data_ptr()
        ops.append(op)
        checks.append((l, src, wts, got, want, signs, want_signs))
    array = (capi.Op * len(ops))(*ops)
    capi.check(capi.lib().xnor_b200_run_ops(array, len(ops), sc.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream, None, None, None), "run_ops")
    for l, src, wts, got, want, signs, want_signs in checks:
        assert torch.equal(got, want) and torch.equal(signs.words, want_signs.words)
    status = capi.C.c_int(-1)
    capi.check(capi.lib().xnor_b200_take_device_status(capi.C.byref(status)), "status")
    assert status.value == 0
