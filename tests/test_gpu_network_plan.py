"""Networks lowered to native operations against the plain layer loop (no hand-over of signs, every tensor in fp32): cfgs beyond the
three shipped ones."""
import ctypes as C

import pytest

import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from darknet_b200 import capi, cfgs, network  # noqa: E402
from recorded import graph_kernels  # noqa: E402

YOLO = "[yolo]\nmask = 0,1,2\nanchors = 10,14, 23,27, 37,58\nclasses=3\nnum=3\n"
HEAD = cfgs._conv(24, 1, bn=0, activation="linear")


def write(tmp_path, sections, width, height, seed=3):
    cfg, weights = tmp_path / "net.cfg", tmp_path / "net.weights"
    cfg.write_text("\n".join([f"[net]\nbatch=1\nwidth={width}\nheight={height}\nchannels=3\n", *sections]))
    # sums of the first convolution are exact in any order: both routes binarise the same values
    network.write_synthetic_weights(network.parse_network_cfg(str(cfg), 1, "cpu"), str(weights), seed, exact_first_conv=True)
    return str(cfg), str(weights)


def image(batch, width, height, seed=1):
    x = torch.from_numpy(synth.uniform01(seed, (batch, 3, height, width))).cuda()
    return (x * 256).floor() / 256


def both(tmp_path, sections, batch, width, height):
    """(lowered network, its heads, heads of the plain network)"""
    cfg, weights = write(tmp_path, sections, width, height)
    net = network.load_network_custom(cfg, weights, batch)
    plain = network.load_network_custom(cfg, weights, batch, sign_chains=False, fuse_first_conv=False, side_branches=False)
    assert plain.plan is None
    x = image(batch, width, height)
    return net, network.forward_network_gpu(net, x), network.forward_network_gpu(plain, x)


def assert_heads_close(got, want):
    """Everything in front of the float layers is bit-equal; those sum up to 2304 products in another order (2e-5 for sums of
    magnitude one, and a logistic function behind them shrinks that)."""
    assert len(got) == len(want)
    for g, w in zip(got, want):
        assert torch.isfinite(w).all() and float((g - w).abs().max()) <= 1e-4 * max(1.0, float(w.abs().max()))
    status = C.c_int(-1)
    capi.check(capi.lib().xnor_b200_take_device_status(C.byref(status)), "status")
    assert status.value == 0


@pytest.mark.parametrize("between", [[], [cfgs._maxpool(2, 2)]], ids=["direct", "pooled"])
def test_a_float_convolution_between_xnor_layers(between, tmp_path):
    """The two routes add the float layer's 160 products in different orders, about 2e-6 of the largest value apart at most; the
    values that close to zero may change their sign, and a pixel of the head sees 576 of them."""
    sections = [cfgs._conv(32, 3), cfgs._conv(160, 3, xnor=1), cfgs._conv(64, 1, bn=0), *between, cfgs._conv(160, 3, xnor=1), HEAD, YOLO]
    cfg, weights = write(tmp_path, sections, 64, 48)
    nets = [network.load_network_custom(cfg, weights, 2, **kw) for kw in ({}, dict(sign_chains=False, fuse_first_conv=False))]
    assert nets[0].plan is not None and nets[1].plan is None
    x = image(2, 64, 48)
    got, want = (network.forward_network_gpu(net, x) for net in nets)
    values = nets[1].layers[2].output_gpu
    close = float((values.abs() <= 2e-6 * values.abs().max()).float().mean())
    differ = float(((got[0] - want[0]).abs() > 1e-4).float().mean())
    assert differ <= 1e-3 + 576 * close < 0.1 and float(want[0].std()) > 0


@pytest.mark.parametrize("batch,width,height", [(2, 64, 48), (1, 16, 16)], ids=["gemm", "small map"])
def test_a_route_may_read_the_convolution_in_front_of_a_yolo_layer(batch, width, height, tmp_path):
    net, got, want = both(tmp_path, [cfgs._conv(32, 3), cfgs._conv(160, 3, xnor=1), HEAD, YOLO, "[route]\nlayers=-2\n", YOLO], batch, width, height)
    assert net.plan is not None and torch.equal(got[0], got[1])
    assert_heads_close(got, want)


def pour(net, other, how):
    """other's weights into net's layers."""
    for l, o in zip(net.layers, other.layers):
        if l.type != "convolutional":
            continue
        pairs = [(l, o, "biases_gpu")]
        pairs += [(l.xnor_layer, o.xnor_layer, n) for n in ("align_bit_weights_gpu", "mean_arr_gpu", "biases_gpu")] if l.xnor else [(l, o, "weights_gpu")]
        for to, of, name in pairs:
            if how == "written":
                getattr(to, name).copy_(getattr(of, name))
            else:
                setattr(to, name, getattr(of, name).clone())


@pytest.mark.parametrize("how", ["written", "replaced"])
@pytest.mark.parametrize("name,batch", [("yolov3-tiny_xnor", 1), ("yolov3-tiny_xnor", 8), ("darknet53_448_xnor", 2)])
def test_weights_that_change_behind_the_plan(name, batch, how, tmp_path):
    size = 160
    cfg = tmp_path / "net.cfg"
    cfg.write_text(cfgs.CFGS[name](size, size))
    nets = []
    for seed in (1, 2):
        network.write_synthetic_weights(network.parse_network_cfg(str(cfg), 1, "cpu"), str(tmp_path / "w"), seed)
        nets.append(network.load_network_custom(str(cfg), str(tmp_path / "w"), batch))
    net, other = nets
    x = image(batch, size, size)
    first, want = ([h.clone() for h in network.forward_network_gpu(n, x)] for n in nets)
    assert not any(torch.equal(a, b) for a, b in zip(first, want))
    pour(net, other, how)
    plan = net.plan
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(network.forward_network_gpu(net, x), want))
    assert net.plan is not None and net.plan is not plan
    plan = net.plan
    network.forward_network_gpu(net, x)
    assert net.plan is plan
    # changed again, and the first forward behind it only captured
    stream = torch.cuda.Stream()
    pour(net, network.load_network_custom(str(cfg), str(tmp_path / "w"), batch), how)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        heads = network.forward_network_gpu(net, x)
    assert all(torch.equal(a, b) for a, b in zip(network.forward_network_gpu(net, x), want))
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(heads, want))


def test_weights_made_under_inference_mode(tmp_path):
    cfg, weights = write(tmp_path, [cfgs._conv(32, 3), cfgs._conv(160, 3, xnor=1), HEAD, YOLO], 64, 48)
    (tmp_path / "2").mkdir()
    _, weights2 = write(tmp_path / "2", [cfgs._conv(32, 3), cfgs._conv(160, 3, xnor=1), HEAD, YOLO], 64, 48, seed=9)
    x = image(1, 64, 48)
    with torch.inference_mode():
        net, other = network.load_network_custom(cfg, weights), network.load_network_custom(cfg, weights2)
        want = network.forward_network_gpu(other, x)[0].clone()
        xl, ol = net.layers[1].xnor_layer, other.layers[1].xnor_layer
        pour(net, other, "written")
        assert torch.equal(network.forward_network_gpu(net, x)[0], want)
        xl.align_bit_weights_gpu = torch.zeros_like(ol.align_bit_weights_gpu)       # counts no writes
        assert not torch.equal(network.forward_network_gpu(net, x)[0], want)
        xl.align_bit_weights_gpu.copy_(ol.align_bit_weights_gpu)
        assert torch.equal(network.forward_network_gpu(net, x)[0], want)


@pytest.mark.parametrize("name", sorted(cfgs.CFGS))
@pytest.mark.parametrize("width", [704, 1376, 1408, 1920])
def test_wide_networks(name, width, tmp_path):
    """Past some width the sign-word kernel has no plan for a layer and the network runs in the layer loop."""
    sections = cfgs.CFGS[name](width, 64).split("\n[", 1)[1]
    net, got, want = both(tmp_path, ["[" + sections], 1, width, 64)
    assert width < 1408 or net.plan is None
    assert_heads_close(got, want)


def test_a_call_that_fails_behind_a_fork_leaves_nothing_running_beside_the_caller():
    """An operation of an unknown kind behind a long one on the side stream: the call reports it, and what the caller queues next still
    comes behind the long one."""
    from darknet_b200 import layer as L
    x = torch.randn(8, 256, 416, 416, device="cuda")
    words = L.GridWords(8, 256, 416, 416)
    want = L.sign_words(x).words
    signs = capi.Op(kind=capi.OP_SIGN_WORDS, desc=capi.ConvDesc(8, 256, 416, 416), input=capi.OP_INPUT, output=words.words.data_ptr(), pitch=417)
    ops = (capi.Op * 3)(capi.Op(kind=capi.OP_FORK), signs, capi.Op(kind=99))
    side, events = torch.cuda.Stream(), [torch.cuda.Event() for _ in range(2)]
    for e in events:
        e.record(side)
    for _ in range(3):
        words.words.zero_()
        torch.cuda.synchronize()
        rc = capi.lib().xnor_b200_run_ops(ops, 3, x.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream, side.cuda_stream,
                                          *(e.cuda_event for e in events))
        got = words.words.clone()
        assert rc == 1 and torch.equal(got, want)


@pytest.mark.parametrize("name,batch", [("yolov3-tiny_xnor", 1), ("yolov3-tiny_xnor", 8), ("tiny-yolo_xnor", 8), ("darknet53_448_xnor", 2)])
def test_heads_that_cross_to_the_host(name, batch, tmp_path):
    """Page-locked tensors, and others that a plain copy takes; as ordinary calls and captured."""
    size = 160
    cfg = tmp_path / "net.cfg"
    cfg.write_text(cfgs.CFGS[name](size, size))
    network.write_synthetic_weights(network.parse_network_cfg(str(cfg), 1, "cpu"), str(tmp_path / "w"))
    net = network.load_network_custom(str(cfg), str(tmp_path / "w"), batch)
    want = [h.cpu() for h in network.forward_network_gpu(net, image(batch, size, size))]
    pinned = [torch.empty_like(h).pin_memory() for h in want]
    doubles = [torch.empty(h.shape, dtype=torch.float64) for h in want]
    strided = [torch.empty(*h.shape[:-1], 2 * h.shape[-1]).pin_memory()[..., ::2] for h in want]
    for hosts in (pinned, strided, doubles):
        direct = net.heads_direct_to_host
        net.heads_direct_to_host = hosts is pinned
        for seed in (2, 1):
            network.forward_network_gpu(net, image(batch, size, size, seed), heads_host=hosts)
        torch.cuda.synchronize()
        assert all(torch.equal(a.float(), b) for a, b in zip(hosts, want))
        net.heads_direct_to_host = direct
    x, stream, graph = image(batch, size, size), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        network.forward_network_gpu(net, x, heads_host=pinned)
    for h in pinned:
        h.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(pinned, want))


@pytest.mark.parametrize("name,batch", [("yolov3-tiny_xnor", 1), ("yolov3-tiny_xnor", 4), ("tiny-yolo_xnor", 4), ("darknet53_448_xnor", 1), ("darknet53_448_xnor", 4)])
def test_the_layer_loop_still_hands_signs_on(name, batch, tmp_path):
    """The linked layers (sign sinks, sign words, shortcut sums, folded pools) that run a network without a plan, against the plan."""
    size = 160
    cfg = tmp_path / "net.cfg"
    cfg.write_text(cfgs.CFGS[name](size, size))
    network.write_synthetic_weights(network.parse_network_cfg(str(cfg), 1, "cpu"), str(tmp_path / "w"), exact_first_conv=True)
    net = network.load_network_custom(str(cfg), str(tmp_path / "w"), batch)
    assert net.plan is not None and net.sink_links > 0 and any(l.emit_masks or l.emit_planes for l in net.layers)
    assert (net.sum_sign_links > 0) == (name == "darknet53_448_xnor" and batch >= net.sum_signs_min_batch)
    x = image(batch, size, size)
    want = [h.clone() for h in network.forward_network_gpu(net, x)]
    net.plan = None
    for _ in range(2):
        assert_heads_close(network.forward_network_gpu(net, x), want)


@pytest.mark.parametrize("name,batch", [("yolov3-tiny_xnor", 1), ("yolov3-tiny_xnor", 64), ("tiny-yolo_xnor", 64), ("darknet53_448_xnor", 2)])
def test_launches_of_a_forward_are_counted(name, batch, tmp_path):
    """Against the kernels of a captured forward; 3x3 256 -> 512 and 1x1 1024 -> 425 on 64 maps of 13x13 leave tiles for a launch of their own."""
    cfg = tmp_path / "net.cfg"
    size = 448 if name.startswith("darknet") else 416
    cfg.write_text(cfgs.CFGS[name](size, size))
    network.write_synthetic_weights(network.parse_network_cfg(str(cfg), 1, "cpu"), str(tmp_path / "w"), 1)
    net = network.load_network_custom(str(cfg), str(tmp_path / "w"), batch)
    x = image(batch, size, size)
    network.forward_network_gpu(net, x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        network.forward_network_gpu(net, x)
    assert len(graph_kernels(C.c_void_p(graph.raw_cuda_graph()))) == network.own_launches_per_forward(net)
