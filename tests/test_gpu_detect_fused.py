"""xnor_b200_detect (decode, suppress and compact in one launch) against a plain CPU restatement, at list lengths around the
kernel's own limits: none, one scan step, a class crowded past what one warp ranks, more detections than slots."""
import ctypes as C
import mmap

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from darknet_b200 import capi, cfgs, network  # noqa: E402
from recorded import graph_kernels  # noqa: E402


def iou(a, b):
    f = np.float32

    def overlap(x1, w1, x2, w2):
        return f(min(f(x1 + f(w1 / f(2))), f(x2 + f(w2 / f(2)))) - max(f(x1 - f(w1 / f(2))), f(x2 - f(w2 / f(2)))))
    w, h = overlap(a[0], a[2], b[0], b[2]), overlap(a[1], a[3], b[1], b[3])
    if w <= 0 or h <= 0:
        return f(0)
    inter = f(w * h)
    return f(inter / f(f(f(a[2] * a[3]) + f(b[2] * b[3])) - inter))


def expected_rows(boxes, obj, probs, thresh):
    probs = probs.copy()
    for k in range(probs.shape[1]):
        order = [d for d in np.argsort(-probs[:, k], kind="stable") if probs[d, k] > 0]
        for r, i in enumerate(order):
            if probs[i, k] == 0:
                continue
            for j in order[r + 1:]:
                if probs[j, k] > 0 and iou(boxes[i], boxes[j]) > thresh:
                    probs[j, k] = 0
    return np.array([[*boxes[d], obj[d], k, probs[d, k]] for d in range(len(obj)) for k in range(probs.shape[1]) if probs[d, k] > 0],
                    np.float32).reshape(-1, 7), probs


@pytest.mark.parametrize("share,size,max_dets,favourite", [(0.0, 32, 64, 0), (0.1, 96, 700, 5), (0.02, 64, 256, 0), (0.2, 96, 700, 0), (0.6, 96, 2048, 3), (0.9, 96, 128, 1),
                                                           (1.0, 128, 4096, 2)])
def test_detect_equals_the_restatement(tmp_path, share, size, max_dets, favourite):
    cfg = tmp_path / "net.cfg"
    cfg.write_text(cfgs.yolov3_tiny_xnor_cfg(size, size))
    batch = 2
    net = network.parse_network_cfg(str(cfg), batch, "cuda:0")
    g = torch.Generator().manual_seed(int(share * 100) + size)
    heads = []
    for l in (l for l in net.layers if l.type == "yolo"):
        h = torch.rand(batch, 3, 85, l.h * l.w, generator=g) * 0.3
        h[:, :, 2:4] -= 0.15
        h[:, :, 4] = torch.where(torch.rand(batch, 3, l.h * l.w, generator=g) < share, 0.9 + 0.1 * h[:, :, 4], 0.1 * h[:, :, 4])
        h[:, :, 5:] = torch.where(torch.rand(batch, 3, 80, l.h * l.w, generator=g) < 0.02, h[:, :, 5:] + 0.6, h[:, :, 5:])
        if favourite:
            h[:, :, 5 + favourite] += 0.65                          # one class that nearly every detection belongs to
        heads.append(h.reshape(batch, 255, l.h, l.w).cuda().contiguous())
    apart = network.DetectionBuffers(batch, 80, max_dets=max_dets, max_rows=20000)
    network.get_network_boxes(net, heads, size, size, 0.5, apart)
    torch.cuda.synchronize()
    count = apart.count.cpu().numpy()
    boxes, obj, probs = (t.cpu().numpy() for t in (apart.boxes, apart.objectness, apart.probs))
    fused = network.DetectionBuffers(batch, 80, max_dets=max_dets, max_rows=20000)
    network.detect(net, heads, size, size, 0.5, 0.45, fused)
    network.do_nms_sort(apart, 0.45)
    network.detection_rows(apart)
    got, same = fused.rows_host(), apart.rows_host()
    assert np.array_equal(fused.count.cpu().numpy(), count)
    for b in range(batch):
        n = min(int(count[b]), max_dets)
        assert int(count[b]) == sum(int((h.view(batch, 3, 85, -1)[b, :, 4] > 0.5).sum()) for h in heads)
        want, kept = expected_rows(boxes[b, :n], obj[b, :n], probs[b, :n], np.float32(0.45))
        assert np.array_equal(got[b], want) and np.array_equal(same[b], want)
        assert np.array_equal(fused.probs[b, :n].cpu().numpy(), kept)


def overlaps(b, thresh):
    """iou() of every pair at once, fp32 operation for operation."""
    f = np.float32
    lo, hi = b[:, :2] - b[:, 2:] * f(0.5), b[:, :2] + b[:, 2:] * f(0.5)
    side = np.minimum(hi[:, None], hi[None]) - np.maximum(lo[:, None], lo[None])
    inter = side[..., 0] * side[..., 1]
    area = b[:, 2] * b[:, 3]
    return (side > 0).all(2) & (inter / ((area[:, None] + area[None]) - inter) > f(thresh))


@pytest.mark.parametrize("found", [1, 32, 33, 128, 129, 767, 768, 769])
def test_detect_at_the_lines_of_the_overlap_matrix(tmp_path, found):
    """Up to 768 detections the overlaps are kept as bits, beyond they are formed on the way; up to 128 of a class a warp ranks them."""
    size, max_dets = 256, 1024
    cfg = tmp_path / "net.cfg"
    cfg.write_text(cfgs.yolov3_tiny_xnor_cfg(size, size))
    net = network.parse_network_cfg(str(cfg), 1, "cuda:0")
    g = torch.Generator().manual_seed(found)
    yolo = [l for l in net.layers if l.type == "yolo"]
    heads = [torch.rand(1, 3, 85, l.h * l.w, generator=g) * 0.3 for l in yolo]
    cells = sum(3 * l.h * l.w for l in yolo)
    chosen = torch.zeros(cells, dtype=torch.bool)
    chosen[torch.randperm(cells, generator=g)[:found]] = True
    parts = chosen.split([3 * l.h * l.w for l in yolo])
    for h, c, l in zip(heads, parts, yolo):
        h[:, :, 4] = torch.where(c.view(1, 3, -1), 0.9 + 0.1 * h[:, :, 4], 0.1 * h[:, :, 4])
        h[:, :, 5:] = torch.where(torch.rand(1, 3, 80, l.h * l.w, generator=g) < 0.02, h[:, :, 5:] + 0.6, h[:, :, 5:])
        h[:, :, 5 + 17] += 0.65                                     # a class that every detection belongs to
    heads = [h.reshape(1, 255, l.h, l.w).cuda().contiguous() for h, l in zip(heads, yolo)]
    apart = network.DetectionBuffers(1, 80, max_dets=max_dets, max_rows=20000)
    network.get_network_boxes(net, heads, size, size, 0.5, apart)
    torch.cuda.synchronize()
    assert int(apart.count.cpu()[0]) == found
    boxes, obj, probs = (t.cpu().numpy()[0, :found].copy() for t in (apart.boxes, apart.objectness, apart.probs))
    over = overlaps(boxes, 0.45)
    for k in range(80):
        order = [d for d in np.argsort(-probs[:, k], kind="stable") if probs[d, k] > 0]
        for r, i in enumerate(order):
            if probs[i, k] > 0:
                later = np.array(order[r + 1:], int)
                probs[later[over[i, later]], k] = 0
    d, k = np.nonzero(probs > 0)
    want = np.concatenate([boxes[d], obj[d, None], k[:, None].astype(np.float32), probs[d, k][:, None]], 1)
    fused = network.DetectionBuffers(1, 80, max_dets=max_dets, max_rows=20000)
    network.detect(net, heads, size, size, 0.5, 0.45, fused)
    network.do_nms_sort(apart, 0.45)
    network.detection_rows(apart)
    for dets in (fused, apart):
        assert np.array_equal(dets.rows_host()[0], want)
        assert np.array_equal(dets.probs[0, :found].cpu().numpy(), probs)


@pytest.mark.parametrize("boxes,thresh", [
    ([(1e6, 1e6, 0.07, 0.07)] * 2, -0.5),                                   # far out: the intersection rounds to more than both, their union below 0
    ([(1e6, 1e6, 0.07, 0.07), (5, 5, 1, 1), (5.2, 5, 1, 1)], -3.0),
    ([(0, 0, 1e8, 1e8), (0, 0, 1e-14, 1e-14)], 7 * 2.0 ** -149),            # 7.1 units of the smallest value, which rounds to seven
    ([(5, 5, 1, 1), (5.2, 5, 1, 1), (5.9, 5, 1, 1), (9, 9, 1, 1)], 0.0),
])
def test_suppression_at_odd_thresholds(boxes, thresh):
    n = len(boxes)
    dets = network.DetectionBuffers(1, 1, max_dets=8, max_rows=8)
    dets.boxes[0, :n], dets.objectness[0, :n] = torch.tensor(boxes), 1.0
    dets.probs[0, :n, 0] = torch.linspace(0.9, 0.5, n)
    dets.count.fill_(n)
    want, _ = expected_rows(*(t[0, :n].cpu().numpy() for t in (dets.boxes, dets.objectness, dets.probs)), np.float32(thresh))
    network.do_nms_sort(dets, float(np.float32(thresh)))
    network.detection_rows(dets)
    assert np.array_equal(dets.rows_host()[0], want)


def sparse_heads(found, size, crowd=0, classes=80, at=17):
    """Activated heads of one image with `found` detections of about one class each, and `crowd` of them of class `at` too."""
    g = torch.Generator().manual_seed(found + crowd)
    heads = [torch.rand(1, 3, 5 + classes, hw, hw, generator=g) * 0.3 for hw in (size // 32, size // 16)]
    places = torch.randperm(sum(h[:, :, 4].numel() for h in heads), generator=g)[:found]
    obj, extra = (torch.zeros(sum(h[:, :, 4].numel() for h in heads)) for _ in range(2))
    obj[places], extra[places[:crowd]] = 0.9, 0.6
    parts = [h[:, :, 4].numel() for h in heads]
    for h, o, e in zip(heads, obj.split(parts), extra.split(parts)):
        h[:, :, 4] = o.view_as(h[:, :, 4]) + 0.1 * torch.rand(h[:, :, 4].shape, generator=g)
        h[:, :, 5:] += 0.6 * (torch.rand(h[:, :, 5:].shape, generator=g) < 1 / classes)
        h[:, :, 5 + at] = 0.3 * torch.rand(h[:, :, 4].shape, generator=g) + e.view_as(h[:, :, 4])
    return [h.reshape(1, -1, *h.shape[3:]).cuda().contiguous() for h in heads]


def class_cfg(tmp_path, size, classes):
    cfg = tmp_path / f"net{classes}.cfg"
    cfg.write_text(cfgs.yolov3_tiny_xnor_cfg(size, size).replace("classes=80", f"classes={classes}").replace("filters=255", f"filters={3 * (5 + classes)}"))
    return network.parse_network_cfg(str(cfg), 1, "cuda:0")


@pytest.mark.parametrize("classes", [80, 140])
@pytest.mark.parametrize("found,crowd", [(256, 2), (257, 2), (300, 32), (300, 33), (300, 64), (300, 65), (300, 95), (300, 96), (300, 97), (700, 96), (700, 200), (768, 30)])
def test_detect_of_classes_with_few_candidates(tmp_path, found, crowd, classes):
    """More than 256 detections: up to 96 candidates in every class the overlaps are those of each class, else of all pairs; more than 128
    classes come in rounds, of which the first may be without and the next with the matrix."""
    size, max_dets = 256, 768
    net = class_cfg(tmp_path, size, classes)
    at = 17 if classes == 80 else 135                               # of 140 in the second round
    heads = sparse_heads(found, size, crowd, classes, at)
    apart = network.DetectionBuffers(1, classes, max_dets=max_dets, max_rows=20000)
    network.get_network_boxes(net, heads, size, size, 0.5, apart)
    torch.cuda.synchronize()
    assert int(apart.count.cpu()[0]) == found
    boxes, obj, probs = (t.cpu().numpy()[0, :found].copy() for t in (apart.boxes, apart.objectness, apart.probs))
    members = (probs > 0).sum(0)
    assert members[at] == crowd and np.delete(members, at).max() <= 32
    want, kept = expected_rows(boxes, obj, probs, 0.45)
    fused = network.DetectionBuffers(1, classes, max_dets=max_dets, max_rows=20000)
    network.detect(net, heads, size, size, 0.5, 0.45, fused)
    network.do_nms_sort(apart, 0.45)
    network.detection_rows(apart)
    for dets in (fused, apart):
        assert np.array_equal(dets.rows_host()[0], want)
        assert np.array_equal(dets.probs[0, :found].cpu().numpy(), kept)


def test_few_candidates_a_class_take_no_longer_with_a_list_that_fits_the_matrix(tmp_path):
    """760 detections of one class each: no slower than by the lists that serve 776 of them (with all pairs formed it was 1.6 times)."""
    net = class_cfg(tmp_path, 416, 80)
    times = []
    for found in (760, 776):
        heads, dets = sparse_heads(found, 416), network.DetectionBuffers(1, 80)
        network.detect(net, heads, 416, 416, 0.5, 0.45, dets)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                network.detect(net, heads, 416, 416, 0.5, 0.45, dets)
        best = float("inf")
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[0] <= 1.15 * times[1], times


@pytest.mark.parametrize("pinned", [True, False])
def test_rows_to_host_into_either_kind_of_memory(pinned):
    """A short list in page-locked memory is written by a kernel, any other through the copies."""
    rows, count = torch.randn(3, 40, 7, device="cuda"), torch.tensor([5, 40, 0], dtype=torch.int32, device="cuda")
    host = torch.full((3, 33, 7), -1.0, pin_memory=pinned)
    host_count = torch.full((3,), -1, dtype=torch.int32, pin_memory=pinned)
    capi.check(capi.lib().xnor_b200_rows_to_host(rows.data_ptr(), 40, count.data_ptr(), 3, 33, host.data_ptr(), host_count.data_ptr(),
                                                 torch.cuda.current_stream().cuda_stream), "xnor_b200_rows_to_host")
    torch.cuda.synchronize()
    assert torch.equal(host, rows[:, :33].cpu()) and torch.equal(host_count, count.cpu())


def recorded_kernels(call):
    """Kernels that `call(stream)` records into a graph, which is not run."""
    cu, graph, stream = C.CDLL("libcuda.so.1"), C.c_void_p(), torch.cuda.Stream()
    handle = C.c_void_p(stream.cuda_stream)
    assert cu.cuStreamBeginCapture_v2(handle, 2) == 0
    call(stream.cuda_stream)
    if cu.cuStreamEndCapture(handle, C.byref(graph)) != 0:          # what the call did cannot be recorded: no kernel, then
        return []
    kernels = graph_kernels(graph)
    assert cu.cuGraphDestroy(graph) == 0
    return kernels


@pytest.mark.parametrize("batch,max_dets,ctas", [(19, 300, 2), (19, 440, 2), (19, 608, 2), (64, 768, 2), (64, 1024, 2), (64, 2048, 1), (18, 768, 1)])
def test_many_images_share_the_sms(tmp_path, batch, max_dets, ctas):
    """More CTAs than SMs: two on each wherever the candidate lists leave room for a second one."""
    cfg = tmp_path / "net.cfg"
    cfg.write_text(cfgs.yolov3_tiny_xnor_cfg(96, 96))
    net = network.parse_network_cfg(str(cfg), batch, "cuda:0")
    heads = [torch.zeros(batch, 255, l.h, l.w, device="cuda") for l in net.layers if l.type == "yolo"]
    dets = network.DetectionBuffers(batch, 80, max_dets=max_dets)

    def call(stream):
        with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
            network.detect(net, heads, 96, 96, 0.5, 0.45, dets)
    kernel, = recorded_kernels(call)
    static, reserved = 5400, 1024
    assert ctas * (kernel.shared + static + reserved) <= 228 * 1024


@pytest.mark.parametrize("found", [256, 351, 352, 353, 384, 700])
def test_detect_at_the_lines_of_many_images(tmp_path, found):
    """Where the matrix is smaller, since two CTAs share an SM: the list of each image is what it is alone."""
    size, batch, max_dets = 256, 19, 700
    cfg = tmp_path / "net.cfg"
    cfg.write_text(cfgs.yolov3_tiny_xnor_cfg(size, size))
    g = torch.Generator().manual_seed(found)
    heads = [torch.rand(1, 3, 85, hw, hw, generator=g) * 0.3 for hw in (size // 32, size // 16)]
    objs = torch.cat([h[:, :, 4].flatten() for h in heads])
    objs.mul_(0.1)[torch.randperm(len(objs), generator=g)[:found]] += 0.9
    for h, o in zip(heads, objs.split([h[:, :, 4].numel() for h in heads])):
        h[:, :, 4] = o.view_as(h[:, :, 4])
        h[:, :, 5:] += 0.6 * (torch.rand(h[:, :, 5:].shape, generator=g) < 0.1)
        h[:, :, 5 + 17] += 0.5
    alone = None
    for n in (1, batch):
        net = network.parse_network_cfg(str(cfg), n, "cuda:0")
        dets = network.DetectionBuffers(n, 80, max_dets=max_dets, max_rows=20000)
        network.detect(net, [h.reshape(1, 255, *h.shape[3:]).repeat(n, 1, 1, 1).cuda() for h in heads], size, size, 0.5, 0.45, dets)
        rows = dets.rows_host()
        assert set(dets.count.tolist()) == {found}
        alone = rows[0] if alone is None else alone
        assert all(np.array_equal(r, alone) for r in rows)


def test_rows_go_by_a_kernel_into_one_page_locked_range_only():
    """Two registrations with a gap between them, one behind the other, one that ends too early, one the device may only read: copies, which
    leave the range to the runtime.  Recorded only: a kernel that stored there would write to addresses that the device does not have."""
    rt, page = torch.cuda.cudart(), mmap.PAGESIZE
    rows, count = torch.zeros(2, 512, 7, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")
    memory = mmap.mmap(-1, 24 * page)
    base = C.addressof(C.c_char.from_buffer(memory))
    pinned_rows, pinned_count = torch.empty(2, 512, 7, pin_memory=True), torch.empty(2, dtype=torch.int32, pin_memory=True)

    def kernels(host_rows, host_count, take):
        return len(recorded_kernels(lambda stream: capi.lib().xnor_b200_rows_to_host(rows.data_ptr(), 512, count.data_ptr(), 2, take, host_rows, host_count, stream)))
    ranges = [(0, 2, 0), (4, 2, 0), (8, 2, 0), (10, 2, 0), (14, 4, 0), (20, 4, 8)]       # first page, pages, flags (8: read-only)
    for first, pages, flags in ranges:
        assert int(rt.cudaHostRegister(base + first * page, pages * page, flags)) == 0
    try:
        take = 6 * page // 56                                       # rows of two images that fill six pages, all but a few bytes
        assert kernels(base, pinned_count.data_ptr(), take) == 0    # pages 0..5, 2 and 3 not registered
        assert kernels(base + 8 * page, pinned_count.data_ptr(), 4 * page // 56) == 0
        assert kernels(base + 15 * page, pinned_count.data_ptr(), 4 * page // 56) == 0
        assert kernels(base + 20 * page, pinned_count.data_ptr(), page // 56) == 0
        assert kernels(pinned_rows.data_ptr(), base + 16 * page - 4, take) == 1      # counts across two pages of one registration
        assert kernels(pinned_rows.data_ptr(), base + 18 * page - 4, take) == 0      # ... and over the end of it
        assert kernels(base + 15 * page + 8, pinned_count.data_ptr(), 2 * page // 56) == 1
        assert kernels(pinned_rows.data_ptr(), pinned_count.data_ptr(), 512) == 1
    finally:
        for first, _, _ in ranges:
            assert int(rt.cudaHostUnregister(base + first * page)) == 0


@pytest.mark.parametrize("side", [False, True])
def test_rows_that_are_not_the_current_devices_go_by_copies(side):
    """Copies take rows from anywhere the runtime knows, here page-locked memory of the host; a kernel is for device memory and streams of the
    current device alone."""
    stream = torch.cuda.Stream() if side else torch.cuda.default_stream()
    rows, count = torch.randn(3, 40, 7), torch.tensor([5, 40, 0], dtype=torch.int32)
    host, host_count = torch.zeros(3, 40, 7, pin_memory=True), torch.zeros(3, dtype=torch.int32, pin_memory=True)
    for r, c, kernels in ((rows.cuda(), count.cuda(), 1), (rows.pin_memory(), count.cuda(), 0), (rows.cuda(), count.pin_memory(), 0)):
        def call(handle):
            return capi.lib().xnor_b200_rows_to_host(r.data_ptr(), 40, c.data_ptr(), 3, 40, host.data_ptr(), host_count.data_ptr(), handle)
        torch.cuda.synchronize()
        assert len(recorded_kernels(call)) == kernels
        if kernels:
            capi.check(call(stream.cuda_stream), "xnor_b200_rows_to_host")
            torch.cuda.synchronize()
            assert torch.equal(host, rows) and torch.equal(host_count, count)


@pytest.mark.parametrize("batch,take,kernels", [(1, 4096, 1), (16, 585, 1), (16, 586, 0), (64, 512, 0)])
def test_long_lists_go_by_copies(batch, take, kernels):
    """Up to 256 KB (16 images of 585 rows: 262080 bytes) by a kernel; beyond, by the copy engine, beside which the SMs are free."""
    rows, count = torch.randn(batch, 4096, 7, device="cuda"), torch.arange(batch, dtype=torch.int32, device="cuda")
    host, host_count = torch.zeros(batch, take, 7, pin_memory=True), torch.zeros(batch, dtype=torch.int32, pin_memory=True)

    def call(stream):
        return capi.lib().xnor_b200_rows_to_host(rows.data_ptr(), 4096, count.data_ptr(), batch, take, host.data_ptr(), host_count.data_ptr(), stream)
    assert len(recorded_kernels(call)) == kernels
    capi.check(call(torch.cuda.current_stream().cuda_stream), "xnor_b200_rows_to_host")
    torch.cuda.synchronize()
    assert torch.equal(host, rows[:, :take].cpu()) and torch.equal(host_count, count.cpu())


def test_a_failed_call_is_reported_once():
    """What a call reported is not the next one's: here counts that would go over the end of a registration, refused when they are recorded."""
    rt, page = torch.cuda.cudart(), mmap.PAGESIZE
    rows, count = torch.randn(2, 40, 7, device="cuda"), torch.tensor([3, 40], dtype=torch.int32, device="cuda")
    host, host_count = torch.zeros(2, 40, 7, pin_memory=True), torch.zeros(2, dtype=torch.int32, pin_memory=True)
    memory = mmap.mmap(-1, 2 * page)
    base = C.addressof(C.c_char.from_buffer(memory))
    codes = []

    def call(at, stream):
        codes.append(capi.lib().xnor_b200_rows_to_host(rows.data_ptr(), 40, count.data_ptr(), 2, 40, host.data_ptr(), at, stream))
    assert int(rt.cudaHostRegister(base, page, 0)) == 0
    try:
        recorded_kernels(lambda stream: call(base + page - 4, stream))
    finally:
        assert int(rt.cudaHostUnregister(base)) == 0
    call(host_count.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert codes[0] != capi.OK and codes[1] == capi.OK
    assert torch.equal(host, rows.cpu()) and torch.equal(host_count, count.cpu())


@pytest.mark.parametrize("counts,max_rows", [([0, 512], 4096), ([513, 3], 4096), ([2049, 700], 4096), ([900, 901], 900)])
def test_rows_host_of_long_lists(counts, max_rows):
    """Lists longer than the first copy: whole the first time, and from then on in one copy."""
    dets = network.DetectionBuffers(2, 4, max_rows=max_rows)
    for _ in range(2):
        dets.rows.normal_()
        dets.row_count.copy_(torch.tensor(counts, dtype=torch.int32))
        got = dets.rows_host()
        for b, n in enumerate(counts):
            assert got[b].shape == (min(n, max_rows), 7) and (got[b] == dets.rows[b, :min(n, max_rows)].cpu().numpy()).all()
        assert min(max(counts), max_rows) <= dets.take <= max_rows


@pytest.mark.parametrize("n_heads,nms", [(4, 0.45), (5, 0.45), (7, 0.45), (5, 0.0)])
def test_networks_of_many_heads(tmp_path, n_heads, nms):
    """One launch takes four heads; more go through the separate calls, in the same order."""
    yolo = "[yolo]\nmask = 0\nanchors = 10,14\nclasses=3\nnum=1\n"
    cfg = tmp_path / "net.cfg"
    cfg.write_text("\n".join(["[net]\nwidth=64\nheight=64\nchannels=3\n"] + [cfgs._conv(8, 3, stride=2, bn=0, activation="linear") + "\n" + yolo] * n_heads))
    net = network.parse_network_cfg(str(cfg), 2, "cuda:0")
    g = torch.Generator().manual_seed(n_heads)
    heads = [torch.rand(2, 8, l.h, l.w, generator=g).cuda() for l in net.layers if l.type == "yolo"]
    assert len(heads) == n_heads
    apart, joined = (network.DetectionBuffers(2, 3) for _ in range(2))
    network.get_network_boxes(net, heads, 64, 64, 0.5, apart)
    if nms:
        network.do_nms_sort(apart, nms)
    network.detection_rows(apart)
    want = apart.rows_host()
    network.detect(net, heads, 64, 64, 0.5, nms, joined)
    got = joined.rows_host()
    assert all(len(w) > 20 and np.array_equal(a, w) for a, w in zip(got, want))


def head_of(output, w, h, n, classes):
    head = capi.YoloHead(output=output.data_ptr(), w=w, h=h, n=n, classes=classes)
    for a in range(2 * n):
        head.anchors[a] = 10.0
    return head


def test_more_images_than_a_grid_has_rows():
    batch = 70_000
    head = torch.zeros(batch, 1, 6, 1, device="cuda")
    head[::3, 0, 4:] = 0.9
    dets = network.DetectionBuffers(batch, 1, max_dets=1, max_rows=1)
    stream = torch.cuda.current_stream().cuda_stream
    capi.check(capi.lib().xnor_b200_yolo_detections(capi.C.byref(head_of(head, 1, 1, 1, 1)), batch, 32, 32, 32, 32, 0.5, 1, 0, 0,
                                                    capi.C.byref(dets.desc), stream), "xnor_b200_yolo_detections")
    network.detection_rows(dets)
    want = torch.zeros(batch, dtype=torch.int32, device="cuda")
    want[::3] = 1
    assert torch.equal(dets.count, want) and torch.equal(dets.row_count, want)
    assert bool((dets.rows[::3, 0, 4] == head[0, 0, 4, 0]).all())


def test_a_head_of_very_many_cells():
    """Candidate numbers past 2^28 (a head of 6.4 GB): the last cells are found, in order, at their places."""
    w = h = 16384
    head = torch.zeros(1, 6, h, w, device="cuda")
    cells = [0, 12345, w * h - 2, w * h - 1]
    for k, cell in enumerate(cells):
        head.view(6, -1)[4:, cell] = 0.9 + 0.01 * k
    dets = network.DetectionBuffers(1, 1, max_dets=8, max_rows=8)
    two = torch.zeros(1, 6, 2, 2, device="cuda")
    two[0, 4:, 1, 0] = 0.8
    heads = (capi.YoloHead * 2)(head_of(head, w, h, 1, 1), head_of(two, 2, 2, 1, 1))
    capi.check(capi.lib().xnor_b200_detect(heads, 2, 1, w, h, w, h, 0.5, 1, 0, 0.0, capi.C.byref(dets.desc), dets.rows.data_ptr(), 8,
                                           dets.row_count.data_ptr(), torch.cuda.current_stream().cuda_stream), "xnor_b200_detect")
    rows = dets.rows_host()[0]
    assert rows[:, 4].tolist() == [np.float32(v) for v in (0.9, 0.91, 0.92, 0.93, 0.8)]
    want = [((c % w) / w, (c // w) / h) for c in cells] + [(0.0, 0.5)]
    assert np.allclose(rows[:, :2], want, atol=1e-6)
