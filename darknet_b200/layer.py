"""Host-side mirror of Darknet's xnor convolutional layer life cycle, over the C ABI.

The names follow the reference so that tests read like its call sequence:

    l = make_convolutional_layer(batch, h, w, c, n, size, stride, pad, activation, xnor=1)
    l.load_weights(weights, biases)          # what load_convolutional_weights + fuse_conv_batchnorm leave
    binary_align_weights(l)                  # src-lib/convolutional_layer.cpp:1339
    forward_convolutional_layer_gpu(l, x)    # src-lib/convolutional_kernels.cu:181 (xnor branch)

torch is used for device memory and the current stream only; every computation is a call into
libxnor_b200.so.  Nothing here has a CPU path.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from . import capi


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


class _Replaced:
    """Counts how often a weight tensor of any layer was replaced by another: what a lowered network (network_plan) looks at before it
    looks at all of its layers."""

    NAMES = frozenset(("weights_gpu", "biases_gpu", "mean_arr_gpu", "align_bit_weights_gpu", "weights_tc_gpu", "weights_blocked_gpu", "xnor_layer"))

    def __init__(self) -> None:
        self.count = 0

    def watch(self, cls):
        """Class decorator: assignments to these attributes of an instance are counted."""
        def set_attribute(obj, name, value):
            object.__setattr__(obj, name, value)
            if name in self.NAMES:
                self.count += 1
        cls.__setattr__ = set_attribute
        return cls


replaced = _Replaced()


@replaced.watch
class ConvolutionalLayer:
    """The Darknet::Layer fields the xnor path touches (src-lib/darknet_layers.hpp:39-83, :250-261)."""

    def __init__(self, batch, h, w, c, n, size, stride, pad, activation, device="cuda:0") -> None:
        self.desc = capi.ConvDesc(batch, c, h, w, n, size, stride, pad, activation)
        g = capi.geometry(self.desc)
        self.batch, self.h, self.w, self.c, self.n = batch, h, w, c, n
        self.size, self.stride, self.pad, self.activation = size, stride, pad, activation
        self.xnor = 1
        self.out_h, self.out_w, self.out_c = g.out_h, g.out_w, n
        self.outputs = n * g.n_out
        self.lda_align = 256
        self.new_lda = g.new_lda
        self.bit_align = g.bit_align
        self.geom = g
        self.device = torch.device(device)
        self.weights_gpu = torch.zeros(n, c * size * size, dtype=torch.float32, device=self.device)
        self.biases_gpu = torch.zeros(n, dtype=torch.float32, device=self.device)
        self.mean_arr_gpu = torch.zeros(n, dtype=torch.float32, device=self.device)
        self.align_bit_weights_gpu: Optional[torch.Tensor] = None
        self.tap_major_weights_gpu: Optional[torch.Tensor] = None    # xnor_b200_tap_major_weights copy, for channel-mask input
        self._output: Optional[torch.Tensor] = None
        self._scratch: Optional[torch.Tensor] = None
        self.window_major = False      # operand rows in 2x2-window-major pixel order (set when a sink of this layer pools)
        self.bin_conv_shortcut_in_gpu: Optional[torch.Tensor] = None
        self.bin_conv_shortcut_out_gpu: Optional[torch.Tensor] = None
        self.shortcut_signs_gpu: Optional[torch.Tensor] = None       # sign words of the fused shortcut sum, when a layer reads them
        # align_bit_weights_gpu as xnor_b200_conv_words reads it, where that route is taken; made again before a call when it was
        # replaced or written to through torch since
        self.conv_words_gpu: Optional[torch.Tensor] = None
        self._words_of = (None, None)                                # the tensor it was made from and that tensor's version (None: keeps none)
        self.input_words: Optional[GridWords] = None                 # the input's sign words
        self._ops = self._conv_op = self._ops_of = None              # forward_convolutional_layer_gpu: its launches, the last of them, what they name
        self._input_floats = batch * c * h * w

    # The two large buffers are made by binary_align_weights, or when something first asks for them: a layer inside a network that hands
    # signs on needs neither (at batch 256 the packed operands of tiny-yolo are 1.5 GB, their allocation and zero fill most of the load time).
    @property
    def output_gpu(self) -> torch.Tensor:
        if self._output is None:
            self._output = torch.empty(self.batch, self.n, self.out_h, self.out_w, dtype=torch.float32, device=self.device)
        return self._output

    @output_gpu.setter
    def output_gpu(self, t: torch.Tensor) -> None:
        self._output = t

    @property
    def scratch(self) -> torch.Tensor:
        if self._scratch is None:
            # zero-filled: when producers write this operand through sinks, padding taps and row tails are never written
            self._scratch = torch.zeros(capi.lib().xnor_b200_scratch_bytes(C.byref(self.desc)), dtype=torch.uint8, device=self.device)
        return self._scratch

    @scratch.setter
    def scratch(self, t: torch.Tensor) -> None:
        self._scratch = t

    def allocate(self) -> None:
        """Makes both, so that no call has to (the scratch is zero-filled: under stream capture that fill would only be recorded)."""
        self.output_gpu, self.scratch

    def load_weights(self, weights: torch.Tensor, biases: torch.Tensor) -> None:
        self.weights_gpu.copy_(weights.reshape(self.n, -1))
        self.biases_gpu.copy_(biases)


def make_convolutional_layer(batch, h, w, c, n, size, stride, pad, activation, xnor=1, device="cuda:0") -> ConvolutionalLayer:
    """make_convolutional_layer (src-lib/convolutional_layer.cpp:715), xnor layers only."""
    if not xnor:
        raise ValueError("this package implements the xnor=1 path only")
    return ConvolutionalLayer(batch, h, w, c, n, size, stride, pad, activation, device)


def binarize_weights(weights: torch.Tensor, n: int, size: int):
    """binarize_weights (src-lib/convolutional_layer.cpp:196): returns (binary [n][size], mean [n])."""
    binary = torch.empty(n, size, dtype=torch.float32, device=weights.device)
    mean = torch.empty(n, dtype=torch.float32, device=weights.device)
    capi.check(capi.lib().xnor_b200_binarize_weights(weights.data_ptr(), n, size, binary.data_ptr(), mean.data_ptr(), _stream()),
               "xnor_b200_binarize_weights")
    return binary, mean


def binary_align_weights(l: ConvolutionalLayer, invert: bool = False, single_calls: bool = True) -> None:
    """binary_align_weights (src-lib/convolutional_layer.cpp:1339): fills align_bit_weights_gpu and mean_arr_gpu.
    single_calls: also all that forward_convolutional_layer_gpu needs (a network that runs the layer its own way does without)."""
    l.align_bit_weights_gpu = torch.empty(l.geom.weights_bytes, dtype=torch.uint8, device=l.device)
    capi.check(capi.lib().xnor_b200_binary_align_weights(C.byref(l.desc), l.weights_gpu.data_ptr(),
                                                        l.align_bit_weights_gpu.data_ptr(), l.mean_arr_gpu.data_ptr(),
                                                        int(invert), _stream()), "xnor_b200_binary_align_weights")
    if single_calls and not invert and takes_words(l):
        l.conv_words_gpu = conv_words_weights(l)
        l._words_of = (l.align_bit_weights_gpu, _version(l.align_bit_weights_gpu))
        if l.input_words is None and l.conv_words_gpu is not None:
            l.input_words = GridWords(l.batch, l.c, l.h, l.w, device=l.device)
    else:
        l.conv_words_gpu = None
    if single_calls:
        l.allocate()
        _layer_ops(l)


def _version(t: torch.Tensor) -> Optional[int]:
    """Counts the writes to a tensor through torch; None for one made under inference_mode, which does not count them."""
    return None if t.is_inference() else t._version


def takes_words(l: ConvolutionalLayer) -> bool:
    """Whether a single layer call runs as sign words + xnor_b200_conv_words or as packed operand + GEMM.  Measured on B200 over some 700
    shapes (7..640 pixels a side, 8..1024 channels and filters, batch 1..64): 3x3 layers 0.07 to 1.05 of the packed route's time,
    1x1 layers whose channels fill no whole words 0.07 to 1.08.  1x1 layers over whole words gain from a few million fp32 values
    or some hundred million binary operations on (0.6 to 1.06) and lose below (1.0 to 1.4: two kernels of 3 us each do all of it),
    or where a stride drops most of what 1024 channels had their signs taken for (1.06 to 1.49).
    Wide maps of deep layers: a tile's window is mostly halo, and each group of filters widens it again.  3x3 at stride 2, 512 channels to
    512 filters: 208x416 194 us against 98, 152x304 64 / 64; to 1024 filters: 80x160 b8 206 / 160, 104x208 b8 323 / 261.  At stride 1
    512 -> 1024 120x480 382 / 277, 1024 -> 256 75x300 127 / 95; 512 -> 512 208x416 196 / 234 on the other side of the line.  Layers of
    few operations gain at every width (512 -> 512 13x208 at stride 2 18 / 31, at stride 1 13x500 38 / 43)."""
    if l.c % 32 != 0:
        return True
    binops = 2 * l.batch * l.outputs * l.c * l.size * l.size
    if l.size == 1:
        floats = l.batch * (l.c * l.h * l.w // (l.stride * l.stride) + l.outputs)
        return (floats > 4_000_000 or binops > 250_000_000) and not (l.stride == 2 and l.c >= 1024)
    if l.stride == 2:
        return not (l.c >= 512 and l.n >= 512 and l.w >= 160 and binops > 20_000_000_000)
    return not (l.c >= 512 and l.n >= 256 and l.c * l.w > 230_000 and l.w >= 256 and binops > 40_000_000_000)


def pack_input(l: ConvolutionalLayer, x: torch.Tensor) -> torch.Tensor:
    """The packed, transposed activation operand (t_bit_input) of every image: uint8 [batch*N][new_ldb/8]."""
    out = torch.empty(l.batch * l.geom.n_out, l.new_lda // 8, dtype=torch.uint8, device=l.device)
    capi.check(capi.lib().xnor_b200_pack_input(C.byref(l.desc), x.data_ptr(), out.data_ptr(), _stream()), "xnor_b200_pack_input")
    return out


def pack_input_staged(l: ConvolutionalLayer, x: torch.Tensor) -> torch.Tensor:
    """pack_input through the two-pass route (sign words first, rows from the words); c % 32 == 0 only."""
    out = torch.empty(l.batch * l.geom.n_out, l.new_lda // 8, dtype=torch.uint8, device=l.device)
    words = torch.empty(capi.lib().xnor_b200_pack_words_bytes(C.byref(l.desc)), dtype=torch.uint8, device=l.device)
    capi.check(capi.lib().xnor_b200_pack_input_staged(C.byref(l.desc), x.data_ptr(), words.data_ptr(), out.data_ptr(), _stream()),
               "xnor_b200_pack_input_staged")
    return out


def gemm_nn_custom_bin_mean_transposed_gpu(M, N, K, A, lda, B, ldb, C_out, ldc, mean_arr, bias, leaky,
                                           shortcut_in=None, shortcut_out=None) -> None:
    """gemm_nn_custom_bin_mean_transposed_gpu (src-lib/im2col_kernels.cu:1156), non-inverted A."""
    capi.check(capi.lib().xnor_b200_gemm_bin_mean_transposed(M, N, K, A.data_ptr(), lda, B.data_ptr(), ldb, C_out.data_ptr(), ldc,
                                                            mean_arr.data_ptr(), _ptr(bias), int(leaky), _ptr(shortcut_in),
                                                            _ptr(shortcut_out), _stream()), "xnor_b200_gemm_bin_mean_transposed")


def gemm_counts(M, N, K, A, lda, B, ldb) -> torch.Tensor:
    counts = torch.empty(M, N, dtype=torch.int32, device=A.device)
    capi.check(capi.lib().xnor_b200_gemm_counts(M, N, K, A.data_ptr(), lda, B.data_ptr(), ldb, counts.data_ptr(), _stream()),
               "xnor_b200_gemm_counts")
    return counts


def pack_input_pooled(l: ConvolutionalLayer, pool: capi.PoolDesc, x: torch.Tensor) -> torch.Tensor:
    """pack_input of maxpool(x) without materialising the pooled tensor; x is the maxpool's input."""
    out = torch.empty(l.batch * l.geom.n_out, l.new_lda // 8, dtype=torch.uint8, device=l.device)
    capi.check(capi.lib().xnor_b200_pack_input_pooled(C.byref(l.desc), C.byref(pool), x.data_ptr(), out.data_ptr(), _stream()),
               "xnor_b200_pack_input_pooled")
    return out


def forward_convolutional_layer_gpu(l: ConvolutionalLayer, x: torch.Tensor, pool: Optional[capi.PoolDesc] = None) -> torch.Tensor:
    """The xnor branch of forward_convolutional_layer_gpu (src-lib/convolutional_kernels.cu:204-262), whole batch.
    With `pool`, x is the input of a [maxpool] layer that sits directly in front of this convolution."""
    if pool is None and x.is_cuda and not capi.packed_route_pinned:
        if l._ops_of != _named(l):
            _layer_ops(l)
        if l.bin_conv_shortcut_out_gpu is not None or l._conv_op.io.shortcut_out:
            # a caller may name other tensors on every call
            l._conv_op.io.shortcut_in = _ptr(l.bin_conv_shortcut_in_gpu) if l.bin_conv_shortcut_out_gpu is not None else None
            l._conv_op.io.shortcut_out = _ptr(l.bin_conv_shortcut_out_gpu)
        if x.dtype != torch.float32 or x.numel() != l._input_floats or not x.is_contiguous():
            raise ValueError("input must be a contiguous fp32 tensor of batch*c*h*w elements")
        of, version = l._words_of
        changed = l.conv_words_gpu is not None and (of is not l.align_bit_weights_gpu or version is None or of._version != version)
        if changed:
            l._ops[0].arg = 1                                       # makes the filters again
        rc = capi.lib().xnor_b200_run_ops(l._ops, len(l._ops), x.data_ptr(), None, 0, torch._C._cuda_getCurrentRawStream(x.device.index),
                                          None, None, None)
        if rc:
            capi.check(rc, "xnor_b200_run_ops")
        if changed:
            l._ops[0].arg = 0
            if not torch.cuda.is_current_stream_capturing():        # captured work has not run
                l._words_of = (l.align_bit_weights_gpu, _version(l.align_bit_weights_gpu))
        return l.output_gpu
    if l.align_bit_weights_gpu is None:
        raise RuntimeError("binary_align_weights() has not been called for this layer")
    expect = l.batch * l.c * (l.h * l.w if pool is None else pool.in_h * pool.in_w)
    if x.dtype != torch.float32 or not x.is_contiguous() or x.numel() != expect:
        raise ValueError("input must be a contiguous fp32 tensor of batch*c*h*w elements")
    if pool is not None:
        capi.check(capi.lib().xnor_b200_conv_forward_pooled(C.byref(l.desc), C.byref(pool), x.data_ptr(), l.align_bit_weights_gpu.data_ptr(),
                                                           l.mean_arr_gpu.data_ptr(), l.biases_gpu.data_ptr(), l.output_gpu.data_ptr(),
                                                           _ptr(l.bin_conv_shortcut_in_gpu), _ptr(l.bin_conv_shortcut_out_gpu),
                                                           l.scratch.data_ptr(), l.scratch.numel(), _stream()), "xnor_b200_conv_forward_pooled")
        return l.output_gpu
    capi.check(capi.lib().xnor_b200_conv_forward(C.byref(l.desc), x.data_ptr(), l.align_bit_weights_gpu.data_ptr(),
                                                l.mean_arr_gpu.data_ptr(), l.biases_gpu.data_ptr(), l.output_gpu.data_ptr(),
                                                _ptr(l.bin_conv_shortcut_in_gpu), _ptr(l.bin_conv_shortcut_out_gpu),
                                                l.scratch.data_ptr(), l.scratch.numel(), _stream()), "xnor_b200_conv_forward")
    return l.output_gpu


def _named(l: ConvolutionalLayer) -> tuple:
    """What the launches of forward_convolutional_layer_gpu name: the sizes, and where the layer's tensors lie.  Looked up on every call,
    so that they never name memory of a tensor that was replaced."""
    if l.align_bit_weights_gpu is None:
        raise RuntimeError("binary_align_weights() has not been called for this layer")
    return (bytes(l.desc), l.align_bit_weights_gpu.data_ptr(), l.mean_arr_gpu.data_ptr(), l.biases_gpu.data_ptr(), l.output_gpu.data_ptr(),
            (l.scratch if l.conv_words_gpu is None else l.conv_words_gpu).data_ptr(), l.input_words)


def _layer_ops(l: ConvolutionalLayer) -> None:
    """The launches of forward_convolutional_layer_gpu."""
    op = capi.Op(desc=l.desc, mean_arr=l.mean_arr_gpu.data_ptr(), biases=l.biases_gpu.data_ptr())
    if l.conv_words_gpu is not None:
        filters = capi.Op(kind=capi.OP_FILTERS, desc=l.desc, weights=l.align_bit_weights_gpu.data_ptr(), output=l.conv_words_gpu.data_ptr())
        signs = capi.Op(kind=capi.OP_SIGN_WORDS, desc=l.desc, input=capi.OP_INPUT, output=l.input_words.words.data_ptr(), pitch=l.input_words.pitch)
        op.kind, op.weights = capi.OP_CONV_WORDS, l.conv_words_gpu.data_ptr()
        op.io.n_sources = 1
        op.io.sources[0] = l.input_words.source()
        op.io.output = l.output_gpu.data_ptr()
        ops = (capi.Op * 3)(filters, signs, op)
    else:
        op.kind, op.weights = capi.OP_CONV, l.align_bit_weights_gpu.data_ptr()
        op.input, op.output = capi.OP_INPUT, l.output_gpu.data_ptr()
        op.scratch, op.scratch_bytes = l.scratch.data_ptr(), l.scratch.numel()
        ops = (capi.Op * 1)(op)
    l._ops, l._conv_op, l._ops_of = ops, ops[len(ops) - 1], _named(l)


class Sink:
    """One direct consumer of a layer's sign bits (struct xnor_b200_sign_sink): `consumer` is the ConvolutionalLayer
    whose scratch the bits are written into, already in its packed-operand layout."""

    def __init__(self, consumer: "ConvolutionalLayer", channel_offset: int = 0, pool: int = 0, upsample: int = 0) -> None:
        self.consumer, self.channel_offset, self.pool, self.upsample = consumer, channel_offset, pool, upsample


def forward_convolutional_layer_io(l: ConvolutionalLayer, x: Optional[torch.Tensor] = None, x_signs: Optional[torch.Tensor] = None,
                                   pool: Optional[capi.PoolDesc] = None, want_signs: bool = False, packed: bool = False,
                                   sinks=(), want_output: Optional[bool] = None, x_masks: Optional[torch.Tensor] = None,
                                   shortcut_only: bool = False, shortcut_signs: bool = False,
                                   shortcut_sink: Optional["ConvolutionalLayer"] = None) -> Optional[torch.Tensor]:
    """xnor_b200_conv_forward_io.  Input: fp32 `x`, sign words / planes `x_signs`, or `packed` (the producers' sinks have
    filled l.scratch).  Output: the fp32 tensor (default when there are no sinks, or with want_output), the sign words
    int32 [batch][n/32][out_h*out_w] (want_signs), and/or the consumers' operands (sinks).  shortcut_only: only the fused
    shortcut sum (l.bin_conv_shortcut_out_gpu) is written and returned; the layer's own tensor is left untouched.
    shortcut_signs: the sign words of the sum are written to l.shortcut_signs_gpu as well.  shortcut_sink: the 1x1 layer
    that reads the sum; the signs go straight into its packed operand (its scratch)."""
    if l.align_bit_weights_gpu is None:
        raise RuntimeError("binary_align_weights() has not been called for this layer")
    io = capi.ConvIO()
    io.input = _ptr(x)
    io.input_signs = _ptr(x_signs)
    io.pool = C.pointer(pool) if pool is not None else None
    io.input_packed = int(packed)
    io.window_major = int(l.window_major)
    weights = l.align_bit_weights_gpu
    if x_masks is not None:
        if l.tap_major_weights_gpu is None:
            tap_major_weights(l)
        io.input_masks = x_masks.data_ptr()
        io.tap_major_weights = 1
        weights = l.tap_major_weights_gpu
    if want_output is None:
        want_output = not want_signs and not sinks
    out = None
    if want_signs:
        out = torch.empty(l.batch, l.n // 32, l.geom.n_out, dtype=torch.int32, device=l.device)
        io.output_signs = out.data_ptr()
    elif shortcut_only:
        out = l.bin_conv_shortcut_out_gpu
        io.shortcut_in = _ptr(l.bin_conv_shortcut_in_gpu)
        io.shortcut_out = out.data_ptr()
    elif want_output:
        out = l.output_gpu
        io.output = out.data_ptr()
        io.shortcut_in = _ptr(l.bin_conv_shortcut_in_gpu)
        io.shortcut_out = _ptr(l.bin_conv_shortcut_out_gpu)
    if shortcut_signs:
        if l.shortcut_signs_gpu is None:
            l.shortcut_signs_gpu = torch.empty(l.batch, l.n // 32, l.geom.n_out, dtype=torch.int32, device=l.device)
        io.shortcut_signs = l.shortcut_signs_gpu.data_ptr()
    if shortcut_sink is not None:
        sk = capi.SignSink()
        sk.consumer = C.pointer(shortcut_sink.desc)
        sk.consumer_scratch = shortcut_sink.scratch.data_ptr()
        sk.consumer_window_major = int(shortcut_sink.window_major)      # refused by the library: the epilogue writes row-major rows
        io.shortcut_sink = C.pointer(sk)
    if sinks:
        arr = (capi.SignSink * len(sinks))()
        for i, s in enumerate(sinks):
            arr[i].consumer = C.pointer(s.consumer.desc)
            arr[i].consumer_scratch = s.consumer.scratch.data_ptr()
            arr[i].channel_offset = s.channel_offset
            arr[i].pool = s.pool
            arr[i].upsample = s.upsample
            arr[i].consumer_window_major = int(s.consumer.window_major)
        io.sinks = arr
        io.n_sinks = len(sinks)
    capi.check(capi.lib().xnor_b200_conv_forward_io(C.byref(l.desc), C.byref(io), weights.data_ptr(),
                                                   l.mean_arr_gpu.data_ptr(), l.biases_gpu.data_ptr(), l.scratch.data_ptr(),
                                                   l.scratch.numel(), _stream()), "xnor_b200_conv_forward_io")
    return out


def tap_major_weights(l: ConvolutionalLayer) -> None:
    """Fills l.tap_major_weights_gpu (xnor_b200_tap_major_weights): the packed weights in tap-major K order."""
    l.tap_major_weights_gpu = torch.empty_like(l.align_bit_weights_gpu)
    capi.check(capi.lib().xnor_b200_tap_major_weights(C.byref(l.desc), l.align_bit_weights_gpu.data_ptr(),
                                                     l.tap_major_weights_gpu.data_ptr(), _stream()), "xnor_b200_tap_major_weights")


def conv_takes_masks(l: ConvolutionalLayer) -> bool:
    return bool(capi.lib().xnor_b200_conv_takes_masks(C.byref(l.desc)))


def conv_words_weights_bytes(l: ConvolutionalLayer) -> int:
    """Size of the filters' copy that xnor_b200_conv_words reads; 0 for a shape it does not take."""
    return capi.lib().xnor_b200_conv_words_weights_bytes(C.byref(l.desc))


def conv_words_weights(l: ConvolutionalLayer) -> Optional[torch.Tensor]:
    """The layer's filters in the order of xnor_b200_conv_words, made from align_bit_weights_gpu; None for a shape it does not take."""
    nbytes = conv_words_weights_bytes(l)
    if nbytes == 0:
        return None
    out = torch.empty(nbytes // 4, dtype=torch.int32, device=l.device)
    capi.check(capi.lib().xnor_b200_conv_words_weights(C.byref(l.desc), l.align_bit_weights_gpu.data_ptr(), out.data_ptr(), _stream()),
               "xnor_b200_conv_words_weights")
    return out


class GridWords:
    """A sign tensor on the position grid (include/xnor_b200.h): int32 [ceil(c/32)][block words], zero-filled."""

    def __init__(self, batch: int, c: int, h: int, w: int, pitch: int = 0, device="cuda:0") -> None:
        self.batch, self.c, self.h, self.w, self.pitch = batch, c, h, w, pitch or w + 1
        self.blocks = (c + 31) // 32
        self.words = torch.zeros(self.blocks, capi.lib().xnor_b200_grid_block_words(batch, h, self.pitch), dtype=torch.int32, device=device)

    def source(self, pool_stride: int = 0, pool_pad: int = 0, upsample: int = 0) -> capi.WordsSource:
        """This tensor as an input of conv_words, with what lies between it and the layer."""
        return capi.WordsSource(self.words.data_ptr(), self.blocks, self.h, self.w, pool_stride, pool_pad, upsample, self.pitch)


def sign_words(x: torch.Tensor, pitch: int = 0) -> GridWords:
    """The signs of an fp32 tensor [batch][c][h][w]."""
    b, c, h, w = x.shape
    out = GridWords(b, c, h, w, pitch, x.device)
    capi.check(capi.lib().xnor_b200_sign_words(x.data_ptr(), b, c, h, w, out.pitch, out.words.data_ptr(), _stream()), "xnor_b200_sign_words")
    return out


def conv_words(l: ConvolutionalLayer, weights: torch.Tensor, sources, output=None, signs: Optional[GridWords] = None, shortcut_in=None,
               shortcut_out=None, pitch: int = 0) -> None:
    """xnor_b200_conv_words: the layer from its inputs' sign words in one launch.  signs receives the signs of what is written
    last: the output, or with a shortcut the sum."""
    io = capi.WordsIO()
    for i, s in enumerate(sources):
        io.sources[i] = s
    io.n_sources = len(sources)
    io.output = _ptr(output)
    io.shortcut_in, io.shortcut_out = _ptr(shortcut_in), _ptr(shortcut_out)
    if signs is not None and shortcut_out is not None:
        io.shortcut_signs = signs.words.data_ptr()
    elif signs is not None:
        io.output_signs = signs.words.data_ptr()
    io.pitch = signs.pitch if signs is not None else pitch
    capi.check(capi.lib().xnor_b200_conv_words(C.byref(l.desc), C.byref(io), weights.data_ptr(), l.mean_arr_gpu.data_ptr(),
                                              l.biases_gpu.data_ptr(), _stream()), "xnor_b200_conv_words")
