"""Lowering a network to native operations, on the CPU: which buffers the operations read and write, and what keeps to the layer
loop.  The native kernels do not run; the filters' copies are stand-ins of the right size."""
import pytest

torch = pytest.importorskip("torch")

from darknet_b200 import capi, cfgs, layer as L, network, network_plan  # noqa: E402

YOLO = "[yolo]\nmask = 0,1,2\nanchors = 10,14, 23,27, 37,58\nclasses=3\nnum=3\n"


def conv(n, size, **kw):
    return cfgs._conv(n, size, **kw)


def head_conv():
    return cfgs._conv(24, 1, bn=0, activation="linear")


def lowered(sections, tmp_path, monkeypatch, batch=2, width=64, height=64):
    cfg = tmp_path / "net.cfg"
    cfg.write_text("\n".join([f"[net]\nbatch=1\nwidth={width}\nheight={height}\nchannels=3\n", *sections]))
    net = network.parse_network_cfg(str(cfg), batch, "cpu")
    monkeypatch.setattr(L, "conv_words_weights", lambda l: torch.zeros(L.conv_words_weights_bytes(l) // 4, dtype=torch.int32))
    for l in net.layers:
        if l.type != "convolutional":
            continue
        l.weights_gpu, l.biases_gpu = torch.zeros(l.n, l.c, l.size, l.size), torch.zeros(l.n)
        if l.xnor:
            l.xnor_layer = L.ConvolutionalLayer(batch, l.h, l.w, l.c, l.n, l.size, l.stride, l.pad, capi.LEAKY, "cpu")
            l.xnor_layer.align_bit_weights_gpu = torch.zeros(l.xnor_layer.geom.weights_bytes, dtype=torch.uint8)
            nxt = net.layers[l.index + 1] if l.index + 1 < len(net.layers) else None
            if nxt is not None and nxt.type == "shortcut" and nxt.activation == "linear":
                nxt.blank, nxt.output_gpu = True, torch.zeros(batch, nxt.out_c, nxt.out_h, nxt.out_w)
        elif l.c * l.size * l.size > 128:
            l.weights_tc_gpu = torch.zeros(1)
    net.plan = network_plan.build(net)
    return net


def sign_buffers(plan):
    """(addresses of sign words that operations read, that they write), checked to be written before they are read."""
    read, written = set(), set()
    for op in plan.ops:
        if op.kind == capi.OP_CONV_WORDS:
            for s in list(op.io.sources)[:op.io.n_sources]:
                assert s.words in written, "sign words read before any operation writes them"
                read.add(s.words)
            written |= {op.io.output_signs, op.io.shortcut_signs} - {None}
        elif op.kind in (capi.OP_CONV3, capi.OP_SIGN_WORDS):
            written.add(op.output)
    return read, written


@pytest.mark.parametrize("name", sorted(cfgs.CFGS))
def test_shipped_networks_write_every_sign_tensor_they_read(name, tmp_path, monkeypatch):
    sections = cfgs.CFGS[name](64, 64).split("\n[", 1)[1]
    net = lowered(["[" + sections], tmp_path, monkeypatch)
    read, written = sign_buffers(net.plan)
    assert read == written


@pytest.mark.parametrize("between", [[], [cfgs._maxpool(2, 2)]], ids=["direct", "pooled"])
def test_a_float_convolution_read_by_an_xnor_layer_gets_its_signs_made(between, tmp_path, monkeypatch):
    net = lowered([conv(32, 3), conv(160, 3, xnor=1), conv(64, 1), *between, conv(160, 3, xnor=1), head_conv(), YOLO], tmp_path, monkeypatch)
    kinds = [op.kind for op in net.plan.ops]
    assert kinds[:5] == [capi.OP_CONV3, capi.OP_CONV_WORDS, capi.OP_FLOAT_TC, capi.OP_SIGN_WORDS, capi.OP_CONV_WORDS]
    signs, float_conv = net.plan.ops[3], net.plan.ops[2]
    assert signs.input == float_conv.output and (signs.desc.c, signs.desc.h, signs.desc.w) == (64, 64, 64)
    read, written = sign_buffers(net.plan)
    assert read == written


def test_a_route_may_read_the_convolution_in_front_of_a_yolo_layer(tmp_path, monkeypatch):
    """Its raw values are kept for the [route]; the [yolo] layer's activation is then a pass of its own."""
    net = lowered([conv(32, 3), conv(160, 3, xnor=1), head_conv(), YOLO, "[route]\nlayers=-2\n", YOLO], tmp_path, monkeypatch)
    convs, heads = [[op for op in net.plan.ops if op.kind == k] for k in (capi.OP_FLOAT_TC, capi.OP_YOLO)]
    assert len(convs) == 1 and convs[0].arg == 0 and convs[0].output not in (capi.OP_HEAD, capi.OP_HEAD + 1)
    assert [op.output for op in heads] == [capi.OP_HEAD, capi.OP_HEAD + 1] and all(op.input == convs[0].output for op in heads)


def test_a_plan_notices_weights_that_change(tmp_path, monkeypatch):
    net = lowered([conv(32, 3), conv(160, 3, xnor=1), head_conv(), YOLO], tmp_path, monkeypatch)
    other = lowered([conv(32, 3), conv(160, 3, xnor=1), head_conv(), YOLO], tmp_path, monkeypatch)
    first, xnor, last = net.layers[:3]
    xl = xnor.xnor_layer
    changes = [lambda: xl.align_bit_weights_gpu.fill_(3), lambda: last.weights_gpu.mul_(2)]
    for owner, name in ((first, "weights_gpu"), (first, "biases_gpu"), (xl, "mean_arr_gpu"), (xl, "biases_gpu"), (xl, "align_bit_weights_gpu"),
                        (last, "biases_gpu"), (last, "weights_gpu"), (last, "weights_tc_gpu")):
        changes.append(lambda owner=owner, name=name: setattr(owner, name, getattr(owner, name).clone()))
    changes.append(lambda: setattr(xnor, "xnor_layer", other.layers[1].xnor_layer))
    for change in changes:
        assert net.plan.current()
        change()
        assert not net.plan.current()
        net.plan = network_plan.build(net)
    # what the operations read in place, and other networks, change nothing
    xl = xnor.xnor_layer
    for t in (first.weights_gpu, first.biases_gpu, xl.mean_arr_gpu, xl.biases_gpu, last.biases_gpu):
        t.add_(1)
    other.layers[0].weights_gpu = torch.zeros(1)
    assert net.plan.current() and not other.plan.current()


def test_a_plan_keeps_the_memory_it_names(tmp_path, monkeypatch):
    net = lowered([conv(32, 3), conv(160, 3, xnor=1), head_conv(), YOLO], tmp_path, monkeypatch)
    named = {op.weights for op in net.plan.ops} | {op.biases for op in net.plan.ops} | {op.mean_arr for op in net.plan.ops}
    named |= {op.input for op in net.plan.ops} | {op.io.output for op in net.plan.ops}
    held = {t.data_ptr() for t in net.plan.keep}
    assert named - {None, capi.OP_INPUT} <= held


@pytest.mark.parametrize("name", sorted(cfgs.CFGS))
def test_networks_too_wide_for_the_kernel_keep_to_the_layer_loop(name, tmp_path, monkeypatch):
    for width, fits in ((608, True), (1408, False), (1920, False)):
        sections = cfgs.CFGS[name](width, 64).split("\n[", 1)[1]
        net = lowered(["[" + sections], tmp_path, monkeypatch, batch=1, width=width)
        assert (net.plan is not None) == fits, width


def test_heads_are_marked_where_they_are_finished(tmp_path, monkeypatch):
    net = lowered([conv(32, 3), conv(160, 3, xnor=1), head_conv(), YOLO, "[route]\nlayers=-3\n", conv(160, 3, xnor=1), head_conv(), YOLO], tmp_path, monkeypatch)
    marks = [i for i, op in enumerate(net.plan.ops) if op.kind == capi.OP_MARK]
    assert net.plan.marked == [True, False] and len(marks) == 1
    assert net.plan.ops[marks[0] - 1].output == capi.OP_HEAD and net.plan.ops[marks[0]].output == capi.OP_HEAD + 2
    assert network.own_launches_per_forward(net) == len(net.plan.ops) - 1
