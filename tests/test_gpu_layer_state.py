"""What a single layer keeps between calls (its filters in the order of xnor_b200_conv_words, its launches) follows what the program
does to the layer in between.  Every result is compared with the packed-operand route, which reads everything on each call."""
import pytest

import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from darknet_b200 import capi, layer as L  # noqa: E402

WORDS = (2, 64, 13, 11, 64, 3)                 # takes the sign-word route
PACKED = (1, 64, 9, 7, 32, 1)                  # a small 1x1 layer: packed operand + GEMM


def build(shape, seed=7):
    batch, c, h, w, n, ks = shape
    x, wt, b = synth.conv_case(seed, batch, c, h, w, n, ks)
    l = L.make_convolutional_layer(batch, h, w, c, n, ks, 1, ks // 2, capi.LEAKY)
    l.load_weights(torch.from_numpy(wt).cuda(), torch.from_numpy(b).cuda())
    L.binary_align_weights(l)
    assert (l.conv_words_gpu is not None) == (shape is WORDS)
    return l, torch.from_numpy(x).cuda()


def refill(l, seed):
    """Other packed weights, written into the layer's own tensor."""
    shape = (l.batch, l.c, l.h, l.w, l.n, l.size)
    l.align_bit_weights_gpu.copy_(build(WORDS if shape == WORDS else PACKED, seed)[0].align_bit_weights_gpu)


def reference(l, x):
    capi.set_tuning(gemm_route=capi.ROUTE_TILED)
    try:
        return L.forward_convolutional_layer_gpu(l, x).clone()
    finally:
        capi.set_tuning()


def assert_follows(l, x, before=None):
    want = reference(l, x)
    l.output_gpu.fill_(float("nan"))
    assert torch.equal(L.forward_convolutional_layer_gpu(l, x), want)
    assert before is None or not torch.equal(want, before)
    return want


@pytest.mark.parametrize("called_before", [False, True])
@pytest.mark.parametrize("how", ["replaced", "written", "packed again"])
@pytest.mark.parametrize("shape", [WORDS, PACKED], ids=["words", "packed"])
def test_packed_weights_that_change(shape, how, called_before):
    l, x = build(shape)
    other, _ = build(shape, seed=8)
    before = assert_follows(l, x) if called_before else None
    if how == "replaced":
        l.align_bit_weights_gpu = other.align_bit_weights_gpu.clone()
    elif how == "written":
        l.align_bit_weights_gpu.copy_(other.align_bit_weights_gpu)
    else:
        l.load_weights(other.weights_gpu, other.biases_gpu)
        L.binary_align_weights(l)
    before = assert_follows(l, x, before)
    refill(l, 9)
    assert_follows(l, x, before)


def test_packed_weights_that_change_under_inference_mode():
    with torch.inference_mode():
        l, x = build(WORDS)
        before = assert_follows(l, x)
        refill(l, 8)
        assert_follows(l, x, before)


def test_a_captured_call_follows_the_packed_weights():
    l, x = build(WORDS)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        L.forward_convolutional_layer_gpu(l, x)
    stream.synchronize()
    refill(l, 8)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = L.forward_convolutional_layer_gpu(l, x)
    before = assert_follows(l, x)                       # nothing of the capture has run yet
    refill(l, 9)
    want = reference(l, x)
    assert not torch.equal(want, before)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert_follows(l, x)


@pytest.mark.parametrize("called_before", [False, True])
@pytest.mark.parametrize("shape", [WORDS, PACKED], ids=["words", "packed"])
def test_tensors_that_are_replaced(shape, called_before):
    """Each tensor's old memory is filled with NaN (or ones) once the layer has another: a launch that still named it would show."""
    l, x = build(shape)
    before = assert_follows(l, x) if called_before else None
    for name in ("mean_arr_gpu", "biases_gpu"):
        old = getattr(l, name)
        setattr(l, name, old * 1.5)
        old.fill_(float("nan"))
        before = assert_follows(l, x, before)
        getattr(l, name).mul_(2)
        before = assert_follows(l, x, before)
        getattr(l, name).data = getattr(l, name) * 3
        before = assert_follows(l, x, before)
    old, l.scratch = l.scratch, torch.zeros_like(l.scratch)
    old.fill_(255)
    assert_follows(l, x)
    assert bool((old == 255).all())
    old, l.output_gpu = l.output_gpu, torch.empty_like(l.output_gpu)
    old.fill_(7.0)
    assert_follows(l, x)
    assert bool((old == 7.0).all())
    if shape is WORDS:
        l.conv_words_gpu = None                        # without the copy: the packed route
        assert_follows(l, x)


@pytest.mark.parametrize("shape", [WORDS, PACKED], ids=["words", "packed"])
def test_shortcuts_and_activations_that_change(shape):
    l, x = build(shape)
    plain = assert_follows(l, x)
    for seed in (1, 2):
        add = torch.from_numpy(synth.bell(seed, tuple(plain.shape))).cuda()
        l.bin_conv_shortcut_in_gpu, l.bin_conv_shortcut_out_gpu = add, torch.empty_like(add)
        assert torch.equal(L.forward_convolutional_layer_gpu(l, x), plain)
        assert torch.equal(l.bin_conv_shortcut_out_gpu, add + plain)
    total = l.bin_conv_shortcut_out_gpu
    l.bin_conv_shortcut_out_gpu = None
    total.zero_()
    assert_follows(l, x)
    assert not bool(total.any())
    l.desc.activation = capi.LINEAR
    assert_follows(l, x, plain)


def allocations():
    torch.cuda.synchronize()
    return torch.cuda.memory_stats()["allocation.all.allocated"]


@pytest.mark.parametrize("shape", [WORDS, PACKED], ids=["words", "packed"])
def test_a_first_call_has_nothing_left_to_make(shape):
    l, x = build(shape)
    made = allocations()
    l.output_gpu, l.scratch
    L.forward_convolutional_layer_gpu(l, x)
    assert allocations() == made


def test_a_network_of_the_layer_loop_has_its_buffers_when_loaded(tmp_path):
    from darknet_b200 import cfgs, network
    cfg, weights = str(tmp_path / "net.cfg"), str(tmp_path / "net.weights")
    with open(cfg, "w") as fh:
        fh.write(cfgs.CFGS["yolov3-tiny_xnor"](96, 96))
    network.write_synthetic_weights(network.parse_network_cfg(cfg, 1, "cpu"), weights)
    net = network.load_network_custom(cfg, weights, 1, sign_chains=False)
    assert net.plan is None
    made = allocations()
    assert len([(l.xnor_layer.scratch, l.xnor_layer.output_gpu) for l in net.layers if l.xnor_layer is not None]) == 9
    assert allocations() == made
