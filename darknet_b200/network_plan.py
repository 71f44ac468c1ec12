"""A loaded network lowered to one array of native operations (xnor_b200_run_ops).

Between xnor convolutions only signs travel: every tensor that an xnor convolution reads is kept as grid words (one 32-channel
sign word per pixel), written by the layer that makes it and read through whatever [maxpool], [upsample] or [route] lies in
between (xnor_b200_conv_words).  fp32 tensors exist where a float layer or a fused [shortcut] reads them.

    plan = build(net)                 # once, at the end of calculate_binary_weights; None: a layer that has no native operation
    heads = plan.run(net, x, heads_host)   # forward_network_gpu
"""
from __future__ import annotations

import ctypes as C
import operator
from typing import Dict, List, Optional, Tuple

import torch

from . import capi
from . import layer as L


_VERSION = operator.attrgetter("_version")


class Unsupported(Exception):
    """The network keeps to the layer-by-layer forward."""


class Plan:
    def __init__(self, net) -> None:
        self.net = net                             # while it is built: a plan that kept it would be a cycle, and its memory wait for the collector
        self.shape = (net.batch, net.c, net.h, net.w)
        self.ops: List[capi.Op] = []
        self.keep: List[torch.Tensor] = []         # tensors the operations point at: their memory stays while the plan does
        self.params: List[Tuple[object, str]] = []    # attributes the operations were made from
        self.laid_out: List[torch.Tensor] = []     # those of which the operations read a copy in another order
        self.head_layers: List = []
        self.finished: List[int] = []              # per head: operations up to and with the one that makes it
        self.head_direct: List[bool] = []          # a head whose last operation may store into page-locked host memory
        self.signs: Dict[int, L.GridWords] = {}    # layer index -> its (or for a blank [shortcut] the sum's) signs
        self.floats: Dict[int, torch.Tensor] = {}  # layer index -> fp32 tensor of a float layer
        self.marks: List[Optional[torch.cuda.Event]] = []    # per head: recorded where it is finished, None for the last thing a forward makes
        self.events: List[torch.cuda.Event] = []

    def address(self, t: Optional[torch.Tensor]) -> Optional[int]:
        if t is not None:
            self.keep.append(t.detach())           # an alias: `t.data = ...` takes no memory away from it
        return None if t is None else t.data_ptr()

    def param(self, owner, name: str) -> int:
        """The address of a weight tensor that a program may replace."""
        self.params.append((owner, name))
        return self.address(getattr(owner, name))

    def reads_copy_of(self, owner, name: str) -> None:
        self.params.append((owner, name))
        if not getattr(owner, name).is_inference():        # made under inference_mode: counts no writes
            self.laid_out.append(getattr(owner, name))

    def _state(self) -> Tuple[List, List]:
        return [getattr(o, n) for o, n in self.params], [t._version for t in self.laid_out]

    def current(self) -> bool:
        """Whether the operations still say what the layers say: no weight tensor was replaced, and none whose copy they read was
        written to.  Replacing is noticed where it happens (layer.replaced), so a forward only counts the writes."""
        if self.seen != L.replaced.count:
            if any(now is not then for now, then in zip(self._state()[0], self.tensors)):
                return False
            self.seen = L.replaced.count
        return list(map(_VERSION, self.laid_out)) == self.versions

    def finish(self) -> None:
        self.seen = L.replaced.count
        self.tensors, self.versions = self._state()
        # a head is marked unless nothing of the forward comes behind it
        self.marked = [self.finished[i] < len(self.ops) for i in range(len(self.head_layers))]
        for i in reversed(range(len(self.head_layers))):
            if self.marked[i]:
                self.ops.insert(self.finished[i], capi.Op(kind=capi.OP_MARK, output=capi.OP_HEAD + len(self.head_layers) + i))
        self.array = (capi.Op * len(self.ops))(*self.ops)
        self.n_ops = len(self.ops)
        # the tensors of the heads, then the events behind them
        self.heads_type = C.c_void_p * (2 * max(1, len(self.head_layers)))
        self.head_shapes = [(self.net.batch, l.out_c, l.out_h, l.out_w) for l in self.head_layers]
        if any(self.marked) and self.net.device.type == "cuda":
            if self.net.copy_stream is None:
                self.net.copy_stream = torch.cuda.Stream(self.net.device)
            self.marks = [torch.cuda.Event() if marked else None for marked in self.marked]
            for e in self.marks:
                if e is not None:
                    e.record(self.net.copy_stream)     # a torch event exists from its first record on
        self.side = self.fork = self.join = None
        if any(op.kind == capi.OP_FORK for op in self.ops):
            if self.net.side_stream is None:
                self.net.side_stream = torch.cuda.Stream(self.net.device)
            self.events = [torch.cuda.Event(), torch.cuda.Event()]
            for e in self.events:
                e.record(self.net.side_stream)     # a torch event exists from its first record on
            self.side = self.net.side_stream.cuda_stream
            self.fork, self.join = (e.cuda_event for e in self.events)
        self.net = None

    def takes(self, x: torch.Tensor) -> bool:
        return (x.is_cuda and x.dtype == torch.float32 and x.shape == self.shape and x.is_contiguous() and not capi.packed_route_pinned)

    def run(self, net, x: torch.Tensor, heads_host: Optional[List[torch.Tensor]]) -> List[torch.Tensor]:
        direct = heads_host is not None and net.heads_direct_to_host
        heads = [heads_host[i] if direct and self.head_direct[i] else torch.empty(s, dtype=torch.float32, device=x.device)
                 for i, s in enumerate(self.head_shapes)]
        pointers = self.heads_type(*[h.data_ptr() for h in heads])
        copied = [i for i, h in enumerate(heads) if heads_host is not None and h is not heads_host[i]]
        early = [i for i in copied if self.marked[i]]
        if early:
            for i in early:
                pointers[len(heads) + i] = self.marks[i].cuda_event
        capi.check(capi.lib().xnor_b200_run_ops(self.array, self.n_ops, x.data_ptr(), pointers, 2 * len(heads),
                                               torch._C._cuda_getCurrentRawStream(x.device.index), self.side, self.fork, self.join),
                   "xnor_b200_run_ops")
        for l, h in zip(self.head_layers, heads):
            l.output_gpu = h
        if early:
            # each head crosses as soon as it exists, beside the rest of the network
            with torch.cuda.stream(net.copy_stream):
                for i in early:
                    net.copy_stream.wait_event(self.marks[i])
                    heads_host[i].copy_(heads[i], non_blocking=True)
        for i in copied:
            if i not in early:
                heads_host[i].copy_(heads[i], non_blocking=True)
        if early:
            torch.cuda.current_stream(x.device).wait_stream(net.copy_stream)
        return heads


# One input of an xnor convolution: (layer whose signs are read, pool stride, pool padding, upsample)
Source = Tuple[int, int, int, int]


def _sources(net, k: int, pool: Tuple[int, int] = (0, 0), up: int = 0) -> List[Source]:
    """What the sign words of layer k's output are made of, walked backwards."""
    l = net.layers[k]
    if l.type == "convolutional" or (l.type == "shortcut" and l.blank):
        if l.out_c % 32 != 0 and not (l.type == "convolutional" and not l.xnor):
            raise Unsupported("filters that fill no whole sign words")
        return [(k, pool[0], pool[1], up)]
    if l.type == "maxpool" and pool == (0, 0) and up == 0 and l.size == 2 and l.stride in (1, 2) and l.pad in (0, 1) and k > 0:
        return _sources(net, k - 1, (l.stride, l.pad), 0)
    if l.type == "upsample" and pool == (0, 0) and up == 0 and l.stride == 2 and k > 0:
        return _sources(net, k - 1, (0, 0), 2)
    if l.type == "route":
        return [s for i in l.input_layers for s in _sources(net, i, pool, up)]
    raise Unsupported(f"[{l.type}] in front of an xnor layer")


def _float_layer(net, k: int) -> int:
    """The layer whose fp32 tensor is layer k's output (a [route] of one layer hands it on)."""
    l = net.layers[k]
    if l.type == "route" and len(l.input_layers) == 1:
        return _float_layer(net, l.input_layers[0])
    if l.type in ("convolutional", "avgpool") or (l.type == "shortcut" and l.blank):
        return k
    raise Unsupported(f"[{l.type}] in front of a float layer")


def _first_conv(l) -> bool:
    return (not l.xnor and l.index == 0 and l.c == 3 and l.size == 3 and l.stride == 1 and l.pad == 1 and l.n <= 32
            and l.activation in ("leaky", "linear"))


def build(net) -> Optional[Plan]:
    try:
        return _build(net)
    except Unsupported:
        return None


def _build(net) -> Plan:
    layers = net.layers
    plan = Plan(net)
    # ---- who reads what: signs per layer, fp32 per layer --------------------------------------------------------------
    sources: Dict[int, List[Source]] = {}
    float_in: Dict[int, int] = {}
    pooled_first = False                           # the [maxpool] behind the first convolution is applied by its kernel
    for k, l in enumerate(layers):
        if l.type == "convolutional" and l.xnor:
            if l.xnor_layer is None or L.conv_words_weights_bytes(l.xnor_layer) == 0 or k == 0:
                raise Unsupported("xnor layer of another shape")
            sources[k] = _sources(net, k - 1)
            if len(sources[k]) > 2 or (len(sources[k]) == 2 and any(layers[s[0]].out_c % 32 != 0 for s in sources[k])):
                raise Unsupported("more than two sources")
            if l.stride == 2 and any(s[1] or s[3] for s in sources[k]):
                raise Unsupported("a pool in front of a stride-2 layer")
        elif l.type == "convolutional" and not _first_conv(l):
            float_in[k] = _float_layer(net, k - 1)
        elif l.type in ("avgpool", "yolo", "region", "softmax"):
            float_in[k] = _float_layer(net, k - 1)
        elif l.type == "shortcut":
            if not l.blank:
                raise Unsupported("[shortcut] that is not fused")
            float_in[k] = _float_layer(net, l.input_layers[0])
    sign_read = {s[0] for ss in sources.values() for s in ss}
    fp32_read = set(float_in.values())
    readers: Dict[int, List[int]] = {}
    for k, l in enumerate(layers):
        for i in (l.input_layers if l.type == "route" else [k - 1] + (l.input_layers if l.type == "shortcut" else [])):
            readers.setdefault(i, []).append(k)
    first = layers[0]
    if not _first_conv(first) or 0 in fp32_read:
        raise Unsupported("a first convolution of another shape")
    firsts = [s for ss in sources.values() for s in ss if s[0] == 0]
    pools = {s[1:3] for s in firsts}
    if pools == {(2, 1)} and readers[0] == [1] and first.out_h % 2 == 0 and first.out_w % 2 == 0 and all(s[3] == 0 for s in firsts):
        pooled_first = True
    # ---- grids: rows of a multiple of 8 pixels keep whole memory sectors where a layer of that map writes fp32 -----------
    wide = {(l.out_h, l.out_w) for k, l in enumerate(layers) if k in fp32_read and k in _xnor_outputs(net) and l.out_w % 8 == 0}

    def pitch(h: int, w: int) -> int:
        return w + 8 if (h, w) in wide else w + 1

    def grid(k: int) -> L.GridWords:
        if k not in plan.signs:
            l = layers[k]
            h, w = (l.out_h // 2, l.out_w // 2) if k == 0 and pooled_first else (l.out_h, l.out_w)
            plan.signs[k] = L.GridWords(net.batch, l.out_c, h, w, pitch(h, w), net.device)
        return plan.signs[k]

    # ---- operations in layer order ---------------------------------------------------------------------------------------
    for k, l in enumerate(layers):
        if l.branch_start:
            plan.ops.append(capi.Op(kind=capi.OP_FORK))
        if l.type == "convolutional" and l.xnor:
            _xnor_conv(plan, k, sources[k], grid, sign_read, fp32_read)
        elif l.type == "convolutional" and _first_conv(l):
            g = grid(k)
            plan.ops.append(capi.Op(kind=capi.OP_CONV3, arg=2 if pooled_first else 0, pitch=g.pitch, desc=_desc(net, l), input=capi.OP_INPUT,
                                    output=g.words.data_ptr(), weights=plan.param(l, "weights_gpu"), biases=plan.param(l, "biases_gpu")))
        elif l.type == "convolutional":
            _float_conv(plan, k, float_in[k], readers.get(k) == [k + 1])
            if k in sign_read:
                # an xnor layer reads it: the kernel leaves fp32, its signs are taken in a pass of their own
                g = grid(k)
                plan.ops.append(capi.Op(kind=capi.OP_SIGN_WORDS, desc=capi.ConvDesc(net.batch, l.n, l.out_h, l.out_w), pitch=g.pitch,
                                        input=plan.floats[k].data_ptr(), output=g.words.data_ptr()))
        elif l.type == "avgpool":
            src = layers[float_in[k]]
            plan.floats[k] = torch.empty(net.batch, l.out_c, 1, 1, device=net.device)
            plan.ops.append(capi.Op(kind=capi.OP_AVGPOOL, desc=capi.ConvDesc(net.batch, src.out_c, src.out_h, src.out_w),
                                    input=plan.address(_tensor(plan, float_in[k])), output=plan.floats[k].data_ptr()))
        elif l.type in ("yolo", "region", "softmax"):
            _head(plan, k, float_in[k])
            plan.finished.append(len(plan.ops))
        if l.branch_end:
            plan.ops.append(capi.Op(kind=capi.OP_BACK))
    if not plan.head_layers:
        raise Unsupported("no head")
    _check_signs_are_written(plan)
    for k, l in enumerate(layers):
        l.output_gpu = plan.floats.get(k, l.output_gpu)
    plan.finish()
    return plan


def _check_signs_are_written(plan: Plan) -> None:
    """Grid words start as zeros: an operation in front of the one that writes them would quietly read "nothing is > 0"."""
    written = set()
    for op in plan.ops:
        if op.kind == capi.OP_CONV_WORDS:
            if any(s.words not in written for s in op.io.sources[:op.io.n_sources]):
                raise Unsupported("a sign tensor that no operation writes")
            written |= {op.io.output_signs, op.io.shortcut_signs}
        elif op.kind in (capi.OP_CONV3, capi.OP_SIGN_WORDS):
            written.add(op.output)


def _xnor_outputs(net) -> set:
    return {k for k, l in enumerate(net.layers) if (l.type == "convolutional" and l.xnor) or (l.type == "shortcut" and l.blank)}


def _desc(net, l) -> capi.ConvDesc:
    return capi.ConvDesc(net.batch, l.c, l.h, l.w, l.n, l.size, l.stride, l.pad, capi.LEAKY if l.activation == "leaky" else capi.LINEAR)


def _tensor(plan: Plan, k: int) -> torch.Tensor:
    """The fp32 tensor of layer k."""
    l = plan.net.layers[k]
    if k in plan.floats:
        return plan.floats[k]
    if l.type == "shortcut":
        return l.output_gpu
    return l.xnor_layer.output_gpu


def _xnor_conv(plan: Plan, k: int, sources: List[Source], grid, sign_read: set, fp32_read: set) -> None:
    layers = plan.net.layers
    l = layers[k]
    xl = l.xnor_layer
    weights = L.conv_words_weights(xl)
    plan.params.append((l, "xnor_layer"))
    plan.reads_copy_of(xl, "align_bit_weights_gpu")
    if xl.align_bit_weights_gpu.is_inference():
        plan.ops.append(capi.Op(kind=capi.OP_FILTERS, arg=1, desc=xl.desc, weights=plan.address(xl.align_bit_weights_gpu), output=weights.data_ptr()))
    io = capi.WordsIO()
    io.n_sources = len(sources)
    for i, (s, pool_stride, pool_pad, up) in enumerate(sources):
        g = grid(s)
        if s == 0 and g.h != layers[0].out_h:
            pool_stride = pool_pad = 0                             # pooled by the first convolution's kernel
        io.sources[i] = g.source(pool_stride, pool_pad, up)
    fused = k + 1 < len(layers) and layers[k + 1].blank
    if k in fp32_read:
        io.output = plan.address(xl.output_gpu)
    out = k
    if fused:
        out = k + 1
        if k in sign_read:
            raise Unsupported("signs of a layer and of its fused shortcut")
        io.shortcut_in = plan.address(_tensor(plan, _float_layer(plan.net, layers[out].input_layers[0])))
        if out in fp32_read:
            io.shortcut_out = plan.address(layers[out].output_gpu)
        if out in sign_read:
            io.shortcut_signs = grid(out).words.data_ptr()
    elif k in sign_read:
        io.output_signs = grid(k).words.data_ptr()
    g = plan.signs.get(out)
    io.pitch = g.pitch if g is not None else 0
    if capi.lib().xnor_b200_conv_words_plan(C.byref(xl.desc), C.byref(io), None) != capi.OK:
        raise Unsupported("a map too wide for the sign-word convolution")
    plan.ops.append(capi.Op(kind=capi.OP_CONV_WORDS, desc=xl.desc, io=io, weights=plan.address(weights), mean_arr=plan.param(xl, "mean_arr_gpu"),
                            biases=plan.param(xl, "biases_gpu")))


def _float_conv(plan: Plan, k: int, src: int, one_reader: bool) -> None:
    """A float convolution behind the path; in front of a [yolo] layer that alone reads it with that layer's activation, into the head."""
    net, l = plan.net, plan.net.layers[k]
    nxt = net.layers[k + 1] if k + 1 < len(net.layers) else None
    op = capi.Op(desc=_desc(net, l), input=plan.address(_tensor(plan, src)), biases=plan.param(l, "biases_gpu"))
    head = one_reader and nxt is not None and nxt.type == "yolo" and l.activation == "linear" and float(nxt.opts.get("scale_x_y", 1)) == 1.0
    entries = 5 + int(nxt.opts.get("classes", 20)) if head else 0
    head = head and l.n % entries == 0
    if l.weights_blocked_gpu is not None:
        op.kind, op.weights = capi.OP_FLOAT_MAP, plan.param(l, "weights_blocked_gpu")
        if not l.yolo_entries:
            head = False
    elif l.weights_tc_gpu is not None:
        op.kind, op.weights = capi.OP_FLOAT_TC, plan.param(l, "weights_tc_gpu")
    else:
        raise Unsupported("a float convolution of another shape")
    plan.reads_copy_of(l, "weights_gpu")
    if head:
        op.arg = entries
        op.output = capi.OP_HEAD + len(plan.head_layers)           # the [yolo] layer behind it adds itself
    else:
        plan.floats[k] = torch.empty(net.batch, l.n, l.out_h, l.out_w, device=net.device)
        op.output = plan.floats[k].data_ptr()
    plan.ops.append(op)


def _head(plan: Plan, k: int, src: int) -> None:
    net, l = plan.net, plan.net.layers[k]
    slot = capi.OP_HEAD + len(plan.head_layers)
    conv = plan.ops[-1]
    plan.head_layers.append(l)
    if l.type == "yolo" and conv.output == slot:
        plan.head_direct.append(conv.kind == capi.OP_FLOAT_MAP)
        return
    plan.head_direct.append(False)
    op = capi.Op(desc=capi.ConvDesc(net.batch, l.c, l.h, l.w), input=plan.address(_tensor(plan, src)), output=slot)
    if l.type == "softmax":
        op.kind = capi.OP_SOFTMAX
    elif l.type == "yolo" and float(l.opts.get("scale_x_y", 1)) == 1.0:
        op.kind, op.arg = capi.OP_YOLO, int(l.opts.get("classes", 20))
        op.desc.n = len(l.opts["mask"].split(","))
    elif l.type == "region" and int(l.opts.get("coords", 4)) >= 2:
        op.kind, op.arg, op.pitch = capi.OP_REGION, int(l.opts.get("classes", 20)), int(l.opts.get("coords", 4))
        op.desc.n, op.desc.activation = int(l.opts.get("num", 1)), int(l.opts.get("softmax", 0))
    else:
        raise Unsupported("a head of another kind")
    plan.ops.append(op)
