"""Which layers xnor_b200_conv_words takes, and how it would run them (host arithmetic only)."""
import ctypes as C

import pytest

pytest.importorskip("torch")

from darknet_b200 import capi, layer as L  # noqa: E402

WORDS = (C.c_uint32 * 8)()
ADDRESS = (C.addressof(WORDS) + 15) // 16 * 16


def plan(batch, c, h, w, n, ks, stride, sources=None, pitch=0):
    """(return value, plan) of a layer that writes fp32; sources: (channels, h, w, pool stride, pool pad, upsample, pitch) each."""
    d = capi.ConvDesc(batch, c, h, w, n, ks, stride, ks // 2, capi.LINEAR)
    io, out = capi.WordsIO(output=ADDRESS, pitch=pitch), capi.WordsPlan()
    sources = sources or [(c, h, w, 0, 0, 0, 0)]
    io.n_sources = len(sources)
    for i, (sc, sh, sw, ps, pp, up, sp) in enumerate(sources):
        io.sources[i] = capi.WordsSource(ADDRESS, (sc + 31) // 32, sh, sw, ps, pp, up, sp)
    return capi.lib().xnor_b200_conv_words_plan(C.byref(d), C.byref(io), C.byref(out)), out


def takes(*shape):
    batch, c, h, w, n, ks, stride = shape
    return capi.lib().xnor_b200_conv_words_weights_bytes(C.byref(capi.ConvDesc(batch, c, h, w, n, ks, stride, ks // 2, capi.LINEAR))) > 0


TOO_LARGE = 6


@pytest.mark.parametrize("shape", [
    (1, 32, 64, 703, 64, 3, 1), (1, 1024, 13, 1408, 64, 3, 1), (1, 64, 64, 1000, 64, 3, 2), (1, 1024, 14, 400, 64, 3, 2), (1, 64, 8, 2300, 64, 1, 2),
    (1, 32, 8, 8, 148 * 128 + 1, 1, 1), (1, 250_000, 4, 4, 32, 3, 1),
], ids=lambda s: "b%d_c%d_%dx%d_n%d_k%d_s%d" % s)
def test_what_has_no_plan_has_no_filters_copy(shape):
    """The size of the filters' copy is the question that callers ask: it must not promise a launch that is then refused."""
    assert not takes(*shape)
    assert plan(*shape)[0] in (TOO_LARGE, 1)


@pytest.mark.parametrize("c,n,ks,stride", [(32, 64, 3, 1), (16, 8, 3, 1), (1024, 1024, 3, 1), (64, 64, 3, 2), (512, 96, 3, 2), (1024, 64, 1, 2), (48, 48, 1, 1)])
def test_the_two_questions_agree_at_every_width(c, n, ks, stride):
    limits = []
    for w in list(range(1, 40)) + list(range(40, 2500, 37)) + [702, 703]:
        ok = plan(2, c, 20, w, n, ks, stride)[0] == capi.OK
        assert takes(2, c, 20, w, n, ks, stride) == ok
        limits += [w] if ok else []
    assert limits and (max(limits) >= 321)


def test_a_pool_in_front_narrows_what_fits():
    assert plan(1, 256, 64, 640, 64, 3, 1)[0] == capi.OK
    assert plan(1, 256, 64, 640, 64, 3, 1, [(256, 128, 1280, 2, 1, 0, 0)])[0] == TOO_LARGE


@pytest.mark.parametrize("shape,words", [
    ((1, 512, 208, 416, 512, 3, 2), False), ((8, 512, 104, 208, 1024, 3, 2), False), ((8, 1024, 80, 160, 1024, 3, 2), False),
    ((8, 512, 104, 208, 256, 3, 2), True), ((1, 512, 13, 208, 512, 3, 2), True), ((8, 512, 52, 104, 512, 3, 2), True), ((64, 256, 56, 56, 512, 3, 2), True),
    ((1, 512, 120, 480, 1024, 3, 1), False), ((1, 1024, 75, 300, 256, 3, 1), False), ((1, 512, 208, 416, 512, 3, 1), True), ((1, 512, 13, 500, 512, 3, 1), True),
    ((8, 1024, 104, 208, 1024, 3, 1), True), ((1, 75, 120, 700, 64, 3, 1), True), ((1, 1000, 75, 300, 256, 3, 1), True),
    ((1, 1024, 13, 13, 256, 1, 1), False), ((64, 256, 56, 56, 64, 1, 1), True), ((8, 1024, 52, 104, 1024, 1, 2), False), ((8, 512, 52, 104, 512, 1, 2), True),
], ids=str)
def test_the_faster_route_is_taken(shape, words):
    """Both sides of the lines, with the shapes they were measured at."""
    batch, c, h, w, n, ks, stride = shape
    l = L.ConvolutionalLayer.__new__(L.ConvolutionalLayer)
    l.batch, l.c, l.h, l.w, l.n, l.size, l.stride = batch, c, h, w, n, ks, stride
    l.outputs = n * ((h + 2 * (ks // 2) - ks) // stride + 1) * ((w + 2 * (ks // 2) - ks) // stride + 1)
    assert L.takes_words(l) == words


def test_every_unit_copies_a_run_that_exists_and_fits():
    """A unit may begin in the padding behind the last image: its run must not begin past the source's end (an empty copy), and no run may
    be longer than its place in shared memory."""
    seen = 0
    for ks, stride in ((1, 1), (1, 2), (3, 1), (3, 2)):
        for c in (16, 40, 96):
            for h in list(range(1, 34)) + [52, 53, 101]:
                for w in list(range(1, 70, 3)) + [51, 104, 207, 301]:
                    for batch in (1, 2, 5):
                        rc, p = plan(batch, c, h, w, 32, ks, stride)
                        assert rc == capi.OK
                        assert 0 < p.run_words_min <= p.run_words_max <= p.run_room, (ks, stride, c, h, w, batch)
                        seen += 1
    for ks in (1, 3):
        for h in range(2, 40):
            for w in (2, 5, 13, 26, 51, 104, 208):
                for ps, pp in ((1, 0), (1, 1), (2, 0), (2, 1)):
                    oh, ow = (h + pp - 2) // ps + 1, (w + pp - 2) // ps + 1
                    for batch in (1, 3):
                        rc, p = plan(batch, 64, oh, ow, 32, ks, 1, [(64, h, w, ps, pp, 0, 0)])
                        assert rc == capi.OK and 0 < p.run_words_min <= p.run_words_max <= p.run_room, (ks, h, w, ps, pp, batch)
                        rc, p = plan(batch, 64, 2 * h, 2 * w, 32, ks, 1, [(32, h, w, 0, 0, 2, 0), (32, 2 * h, 2 * w, 0, 0, 0, 0)])
                        assert rc == capi.OK and 0 < p.run_words_min <= p.run_words_max <= p.run_room, (ks, h, w, "up", batch)
                        seen += 2
    assert seen > 20_000
