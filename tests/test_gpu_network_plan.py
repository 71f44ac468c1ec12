"""Networks lowered to native operations against the plain layer loop (no hand-over of signs, every tensor in fp32): cfgs beyond the
three shipped ones."""
import ctypes as C

import pytest

import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from darknet_b200 import capi, cfgs, network  # noqa: E402

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
