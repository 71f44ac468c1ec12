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
