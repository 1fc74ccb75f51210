"""Kernels at the sizes where their tilings, remainders and fallbacks change, against the oracle.

Bounds: data movement and batchnorm bit-exact; sums of n fp32 products 1e-5 + 1e-5|ref| (tests of the same kernels
at ordinary sizes use the same); selections exact wherever the oracle's scores are not tied within fp32 rounding.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
from test_ops_gpu import _check_per_class, close  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [5, 8, 16, 20, 36, 48, 144, 389])
@pytest.mark.parametrize("kernel,stride,size", [(3, 1, (19, 33)), (3, 2, (38, 21)), (5, 1, (12, 40)), (5, 2, (31, 17)), (3, 1, (4, 8))])
def test_depthwise_any_width(oracle_port, channels, kernel, stride, size):
    """Channel slabs of 32 and 16 with a ragged last one, lanes past the width, 3x3 and 5x5 windows; a clip whose
    lower bound must not lift the padded lanes."""
    from gpu_ops import run_case_cuda
    rng = np.random.default_rng(channels * 10 + kernel)
    x = rng.standard_normal((2,) + size + (channels,), dtype=np.float32)
    w = rng.standard_normal((channels, 1, kernel, kernel), dtype=np.float32) * np.float32(0.3)
    b = rng.standard_normal(channels, dtype=np.float32)
    case = dict(op="conv2d", x=x, w=w, bias=b, stride=stride, pad=kernel // 2, dilation=1, group=channels, act=1, lo=0.5, hi=6.0)
    close(run_case_cuda(case), oracle_port.conv2d(x, w, b, stride, kernel // 2, 1, channels, 1, 0.5, 6.0))


@pytest.mark.parametrize("size", [(75, 75), (31, 66), (17, 99), (9, 151), (150, 12), (4, 127), (33, 8)])
@pytest.mark.parametrize("images,channels,kernel", [(1, 40, 3), (12, 64, 3), (3, 20, 5)])
def test_depthwise_tile_shapes(oracle_port, size, images, channels, kernel):
    """Stride 1: parts of the width from 5 to 32 pixels, every row count, tiles that hang over the right and lower edges."""
    from gpu_ops import run_case_cuda
    rng = np.random.default_rng(size[1] + channels)
    x = rng.standard_normal((images,) + size + (channels,), dtype=np.float32)
    w = rng.standard_normal((channels, 1, kernel, kernel), dtype=np.float32) * np.float32(0.3)
    b = rng.standard_normal(channels, dtype=np.float32)
    case = dict(op="conv2d", x=x, w=w, bias=b, stride=1, pad=kernel // 2, dilation=1, group=channels, act=2, lo=0.0, hi=6.0)
    close(run_case_cuda(case), oracle_port.conv2d(x, w, b, 1, kernel // 2, 1, channels, 2, 0.0, 6.0))


@pytest.mark.parametrize("shape,width", [((12, 9, 45, 832), 15), ((10, 41, 27, 807), 14), ((8, 15, 47, 800), 16)])
def test_depthwise_shapes_estimated_alike(shape, width, monkeypatch):
    """Maps that another width, of a time estimated within 1.5 %, took 12-15 % longer for: not slower than in the named one."""
    import torch
    from ogle_b200 import ops
    N, H, W, ch = shape
    g = torch.Generator(device="cuda").manual_seed(ch)
    x = torch.zeros((N, H, W, ops.up4(ch)), device="cuda")
    x[..., :ch] = torch.randn((N, H, W, ch), generator=g, device="cuda")
    p = ops.conv_params(N, H, W, ch, ch, 3, 1, 1, 1, ch, False, ops.ACT_RELU, 0.0, 0.0, ops.MATH_FP32)
    packed, y = ops.conv2d_prepack(p, torch.randn((ch, 1, 3, 3), generator=g, device="cuda")), torch.empty_like(x)
    took = []
    for forced in (False, True):
        if forced:
            monkeypatch.setenv("OGLE_DW_TW", str(width))
        took.append(_median_us(_in_a_graph(lambda: ops.conv2d(p, x, packed, None, y, workspace=None))))
    assert took[0] <= 1.06 * took[1], took


def test_depthwise_shapes_of_a_network_are_weighed_once():
    """A pass over the thirteen depthwise layers of a network takes the host no longer a layer than one of them over and over;
    layers that it has not seen lately take longer."""
    import ctypes as C
    import time
    from ogle_b200 import _lib, ops
    name = _lib.cuda_lib().ogle_cuda_conv2d_kernel_name
    layers = [(150, 32, 1), (150, 64, 2), (75, 128, 1), (75, 128, 2), (38, 256, 1), (38, 256, 2), (19, 512, 1), (19, 512, 2), (10, 1024, 1),
              (75, 144, 1), (56, 96, 1), (28, 192, 1), (14, 384, 1)]
    of = lambda images: [C.byref(ops.conv_params(images, h, h, c, c, 3, s, 1, 1, c, True, ops.ACT_RELU, 0.0, 0.0, ops.MATH_TF32X3)) for h, c, s in layers]

    def took(calls):
        best = 1e9
        for _ in range(200):
            t = time.perf_counter()
            for p in calls:
                name(p)
            best = min(best, (time.perf_counter() - t) / len(calls))
        return best

    network = of(1)
    one, turns, unseen = took([p for p in network for _ in range(4)]), took(network * 4), took([p for n in range(2, 34) for p in of(n)])
    assert turns - one <= 0.5 * (unseen - one), (one, turns, unseen)


@pytest.mark.parametrize("channels", [1, 6, 12, 20, 129, 1028])
def test_batchnorm_any_width_is_exact(oracle_port, channels):
    from gpu_ops import run_case_cuda
    rng = np.random.default_rng(channels)
    x = rng.standard_normal((3, 7, 11, channels), dtype=np.float32)
    g, b, m = (rng.standard_normal(channels, dtype=np.float32) for _ in range(3))
    v = rng.random(channels, dtype=np.float32) + np.float32(0.1)
    got = run_case_cuda(dict(op="batchnorm", x=x, gamma=g, beta=b, mean=m, var=v, eps=1e-5))
    assert np.array_equal(got, oracle_port.batchnorm(x, g, b, m, v, 1e-5))


@pytest.mark.parametrize("widths", [(3, 5), (1, 1, 1, 1, 1), (8, 4, 2), (6, 8), (130, 7, 33)])
def test_concat_ragged_channels_is_exact(widths):
    from gpu_ops import run_case_cuda
    rng = np.random.default_rng(sum(widths))
    xs = [rng.random((2, 5, 9, w), dtype=np.float32) for w in widths]
    assert np.array_equal(run_case_cuda(dict(op="concat", xs=xs, axis=3)), np.concatenate(xs, axis=3))


def test_average_pool_divides_exactly(oracle_port):
    """3x3 stride 2 averages at both signs, zeros, tiny and huge values: the quotient of the window's sum by 9 is the
    correctly rounded one (a window that holds one value and zeros has no summation order)."""
    from gpu_ops import run_case_cuda
    rng = np.random.default_rng(5)
    x = np.zeros((1, 64, 64, 8), np.float32)
    # odd positions: each window 2i..2i+2 holds exactly one of them (even ones would put four values in a window, whose
    # sum depends on their order)
    x[:, 1::2, 1::2] = (rng.standard_normal((1, 32, 32, 8)) * 10.0 ** rng.uniform(-44, 38, (1, 32, 32, 8))).astype(np.float32)
    got = run_case_cuda(dict(op="pool", x=x, kernel=3, stride=2, pad=0, type_=1))
    assert np.array_equal(got[0, :, :, :], oracle_port.pool(x, 3, 2, 0, 1)[0])


@pytest.mark.parametrize("anchors,classes,top_k,spread", [
    (1917, 21, 200, 2.0),       # the benchmark's decoder
    (1917, 21, 200, 1e-3),      # all scores within a fraction of a bin
    (1917, 21, 200, 0.0),       # all scores equal: index order
    (1920, 3, 256, 5.0),        # scores crowd at 0 and 1
    (31, 2, 100, 1.0),          # fewer anchors than results
    (4001, 30, 37, 1.0),        # scores of a few classes at a time, ragged anchor count
    (1001, 40, 5, 1.0),         # rows of logits that are not kept in registers
])
def test_detect_selection_edges(oracle_port, anchors, classes, top_k, spread):
    rng = np.random.default_rng(anchors + classes)
    logits = (rng.standard_normal((2, anchors, classes)) * spread).astype(np.float32)
    boxes = rng.random((2, anchors, 4), dtype=np.float32)
    for thr in (0.01, 0.0, 0.3):
        _check_per_class(oracle_port, logits, boxes, thr, top_k, (classes + 3) // 4 * 4)


@pytest.mark.parametrize("classes", [2, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 32])
def test_detect_rows_of_every_length(oracle_port, classes):
    """A kernel for each number of 128-bit pieces in a row of logits, the last of them full and with one value: all classes
    in one block of as many warps as classes and of half as many, half of the classes a block, classes in two passes."""
    rng = np.random.default_rng(classes)
    for images, anchors in ((2, 70), (1, 500), (150, 90), (1, 3000)):
        logits = (rng.standard_normal((images, anchors, classes)) * 2).astype(np.float32)
        _check_per_class(oracle_port, logits, rng.random((images, anchors, 4), dtype=np.float32), 0.02, 20, (classes + 3) // 4 * 4)


@pytest.mark.parametrize("anchors,classes,spread,thr", [(1917, 2, 3.0, 0.3), (1917, 21, 1e-3, 0.01), (333, 5, 0.0, 0.1), (40, 33, 2.0, -1.0)])
def test_reference_rule_edges(oracle_port, anchors, classes, spread, thr):
    """The reference detector's rule, decoded by the caller and decoded on the way, over the same edges."""
    import ctypes as C
    import torch
    from ogle_b200 import _lib, ops
    rng = np.random.default_rng(anchors + classes)
    N, K = 3, 100
    logits = torch.zeros((N, anchors, ops.up4(classes)))
    logits[..., :classes] = torch.from_numpy((rng.standard_normal((N, anchors, classes)) * spread).astype(np.float32))
    logits = logits.cuda()
    pred = ops.dense_to_device(rng.standard_normal((N, anchors, 4), dtype=np.float32) * np.float32(0.5))
    priors = ops.dense_to_device(np.concatenate([rng.random((anchors, 2)), rng.random((anchors, 2)) * 0.3 + 0.05], 1))
    boxes = ops.ssd_decode(pred, priors)
    out = ops.ssd_detect(logits, boxes, classes, 0, thr, K, 0.45, 300, 300)
    p = _lib.DetectParams()
    p.N, p.A, p.C, p.logit_stride, p.mode = N, anchors, classes, logits.shape[-1], 0
    p.score_thr, p.top_k, p.nms_thr, p.image_w, p.image_h = thr, K, 0.45, 300, 300
    fused = [torch.empty_like(t) for t in out]
    var = (C.c_float * 4)(0.1, 0.1, 0.2, 0.2)
    assert _lib.cuda_lib().ogle_cuda_ssd_decode_detect(C.byref(p), ops._p(logits), ops._p(pred), ops._p(priors), var,
                                                       *[C.c_void_p(t.data_ptr()) for t in fused], ops._stream()) == 0
    for a, b in zip(out, fused):
        assert torch.equal(a, b)
    score, anchor, cls, box, count = [t.cpu().numpy() for t in out]
    for n in range(N):
        ref = oracle_port.detect(boxes[n].cpu().numpy(), logits[n, :, :classes].cpu().numpy(), 300, 300, thr, K, 0.45)
        k = len(ref["anchor"])
        assert count[n] == k
        assert np.abs(score[n, :k] - ref["score"]).max(initial=0) <= 2e-6
        if spread != 1e-3:         # (scores that differ by less than their rounding may change places)
            assert np.array_equal(anchor[n, :k], ref["anchor"]) and np.array_equal(box[n, :k].astype(np.int32), ref["rect"])
        assert (anchor[n, k:] == -1).all()


def _in_a_graph(fn, launches=20):
    """Replays of that many launches, for what takes the device less than the host takes to ask for it."""
    import torch
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        fn()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(launches):
                fn()
    return graph.replay


def _median_us(fn):
    import torch
    times = []
    for _ in range(9):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        fn()
        e0.record()
        for _ in range(10):
            fn()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1) * 100)
    return sorted(times)[4]


def test_few_anchors_leave_room_for_blocks():
    """Blocks of few anchors share an SM, which the registers have to allow: 300 anchors took 0.30 of the time of 1917 (50 of
    165 us) with as many blocks as their scores let on, and 0.42 with a block an SM."""
    import torch
    from ogle_b200 import ops

    def took(anchors):
        g = torch.Generator(device="cuda").manual_seed(anchors)
        logits = torch.randn((1024, anchors, 24), generator=g, device="cuda") * 2
        boxes = torch.rand((1024, anchors, 4), generator=g, device="cuda")
        return _median_us(lambda: ops.ssd_detect(logits, boxes, 21, 1, 0.01, 100, 0.45, 300, 300))

    assert took(300) <= 0.36 * took(1917)


@pytest.mark.parametrize("anchors,classes", [(200, 5), (200, 40)])
@pytest.mark.parametrize("mode", [0, 1])
def test_detect_drops_rows_without_scores(mode, anchors, classes):
    """NaN logits, and logits whose exponentials overflow (their quotients are inf / inf): no class of such an anchor is a
    candidate, in rows held in registers and in longer ones."""
    import torch
    from ogle_b200 import ops
    g = torch.Generator().manual_seed(classes)
    z = torch.randn((1, anchors, classes), generator=g)
    z[0, 7, 2] = float("nan")
    z[0, 31, 0] = float("nan")
    z[0, 50, 1] = 95.0
    z[0, 51, :] = 89.0
    z[0, 77, 3] = float("inf")
    z[0, 78, 1] = float("-inf")           # a class that cannot be, the others have scores
    e = torch.exp(z[0])
    s = e / e.sum(1, keepdim=True)
    bad = {7, 31, 50, 51, 77}
    logits = torch.nn.functional.pad(z, (0, ops.up4(classes) - classes)).cuda()
    boxes = torch.zeros((1, anchors, 4), device="cuda")
    thr = 1e-4
    score, anchor, cls, box, count = [t.cpu() for t in ops.ssd_detect(logits, boxes, classes, mode, thr, 256, 0.0, 300, 300)]
    for c in range(1, classes) if mode else (0,):
        rows = slice((c - 1) * 256, c * 256) if mode else slice(0, 256)
        n = int(count.flatten()[c - 1 if mode else 0])
        got = anchor.flatten()[rows][:n].tolist()
        v = s[:, c] if mode else s[:, 1:].max(1).values
        want = {i for i in range(anchors) if i not in bad and v[i] > thr}
        edge = {i for i in range(anchors) if i not in bad and abs(v[i] - thr) < 1e-6}
        assert set(got) ^ want <= edge and not set(got) & bad


@pytest.mark.parametrize("batch,anchors,classes,mode", [
    (1, 56444, 2, 1), (149, 56444, 2, 1), (1, 55548, 3, 1), (148, 53756, 5, 1), (1, 39420, 21, 1), (1, 27774, 2, 0), (200, 27774, 3, 0)])
def test_detect_takes_the_largest_anchor_counts(oracle_port, batch, anchors, classes, mode):
    """Scores of one class (mode 1) or one image (mode 0) have to fit a block's shared memory; how many do does not
    depend on the batch."""
    import torch
    from ogle_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(anchors)
    logits = torch.zeros((batch, anchors, ops.up4(classes)), device="cuda")
    logits[..., :classes] = torch.randn((batch, anchors, classes), generator=g, device="cuda") * 3.0
    xy = torch.rand((batch, anchors, 2), generator=g, device="cuda")
    boxes = torch.cat([xy, xy + 0.05], 2)
    score, anchor, cls, box, count = ops.ssd_detect(logits, boxes, classes, mode, 0.5, 50, 0.0, 300, 300)
    e = torch.softmax(logits[..., :classes].double(), 2)
    for c in range(1, classes) if mode else (0,):
        # (distinct scores: the best fifty of each image, whatever the class in mode 0)
        want = (e[..., c] if mode else e[..., 1:].max(2).values).topk(50, 1)
        rows = slice((c - 1) * 50, c * 50) if mode else slice(0, 50)
        assert (count[:, c - 1] if mode else count).flatten().eq(50).all()
        assert (score.reshape(batch, -1)[:, rows].double() - want.values).abs().max() <= 2e-6
        got = anchor.reshape(batch, -1)[:, rows].long()
        mine = (e[..., c] if mode else e[..., 1:].max(2).values).gather(1, got)
        assert (mine - want.values).abs().max() <= 2e-6


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, kernel, stride, pad, dilation: rows, columns and reductions that end inside a tile; launches of
    # one tile split over a cluster of 8, of a few tiles, and of enough for the large tiles (128 x 32, x 64, x 128)
    (1, 7, 7, 512, 33, 3, 1, 1, 1), (2, 5, 3, 4, 8, 1, 1, 0, 1), (1, 9, 11, 20, 70, 3, 2, 1, 1), (3, 20, 17, 12, 129, 5, 1, 2, 1),
    (2, 33, 31, 6, 9, 3, 2, 2, 2), (3, 160, 161, 5, 24, 1, 1, 0, 1), (2, 200, 197, 8, 50, 1, 1, 0, 1), (2, 150, 149, 16, 100, 1, 1, 0, 1)])
def test_fp32_convolution_edges(oracle_port, shape):
    from gpu_ops import run_case_cuda
    N, H, W, C, K, k, s, p, d = shape
    rng = np.random.default_rng(C + K)
    x = rng.standard_normal((N, H, W, C), dtype=np.float32)
    w = (rng.standard_normal((K, C, k, k)) / np.sqrt(C * k * k)).astype(np.float32)
    b = rng.standard_normal(K, dtype=np.float32)
    case = dict(op="conv2d", x=x, w=w, bias=b, stride=s, pad=p, dilation=d, group=1, act=1, lo=0.5, hi=2.0)
    close(run_case_cuda(case), oracle_port.conv2d(x, w, b, s, p, d, 1, 1, 0.5, 2.0))


@pytest.mark.parametrize("m,k,n,trans_b", [(1, 5, 3, 0), (1, 5, 3, 1), (65, 129, 63, 0), (63, 131, 66, 1), (8, 512, 1000, 1), (700, 33, 300, 0)])
def test_fp32_gemm_edges(oracle_port, m, k, n, trans_b):
    """Rows that end between 16-byte pieces (k and n not multiples of 4), both layouts of B, matrix bias."""
    from gpu_ops import run_case_cuda
    rng = np.random.default_rng(m + k + n)
    A = rng.standard_normal((m, k), dtype=np.float32)
    B = (rng.standard_normal((n, k) if trans_b else (k, n)) / np.sqrt(k)).astype(np.float32)
    Cm = rng.standard_normal((m, n), dtype=np.float32)
    got = run_case_cuda(dict(op="gemm", A=A, B=B, Cm=Cm, transB=trans_b, alpha=0.5, beta=2.0))
    close(got, oracle_port.gemm(A, B, Cm, trans_b, 0.5, 2.0))


@pytest.mark.parametrize("m,k,n,trans_b", [
    # two rows a thread: tiles of 64 x 64 and 64 x 32, up to 64 elements and, with one to three tiles an SM, up to 128
    (300, 64, 77, 0), (300, 63, 31, 0), (5000, 117, 100, 0), (77, 62, 90, 1), (5000, 101, 90, 1),
    # narrow outputs, alone and split over clusters
    (2000, 300, 31, 0), (130, 1030, 30, 0),
    # a transposed B: 64 x 64 alone and split, 128 x 128, 128 x 64, a reduction shorter than the ring
    (700, 90, 700, 1), (60, 2050, 130, 1), (4700, 70, 1000, 1), (9600, 70, 520, 1), (9600, 65, 520, 1),
    # 128 x 64 where 128 x 128 would leave one tile too many on some SMs
    (1419, 131, 3435, 0)])
def test_fp32_contraction_forms(m, k, n, trans_b):
    import torch
    from ogle_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m + n)
    pad = lambda t: torch.nn.functional.pad(t, (0, ops.up4(t.shape[-1]) - t.shape[-1]), value=float("nan"))     # never to be read
    a, b = torch.randn((m, k), generator=g, device="cuda"), torch.randn((n, k) if trans_b else (k, n), generator=g, device="cuda")
    c = torch.randn(n, generator=g, device="cuda")
    got = ops.gemm(pad(a), pad(b), torch.nn.functional.pad(c, (0, ops.up4(n) - n)), m, k, n, trans_b, 0.5, 2.0, 2, ops.MATH_FP32)
    b64 = b.double().t() if trans_b else b.double()
    want = 0.5 * (a.double() @ b64) + 2.0 * c.double()
    # every partial sum rounded once: at most k * 2^-24 of the sum of the terms' magnitudes
    bound = (k + 4) * 2.0 ** -24 * (0.5 * (a.abs().double() @ b64.abs()) + 2.0 * c.abs().double())
    assert ((got[:, :n].double() - want).abs() <= bound).all()
    assert (got[:, n:] == 0).all()


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, kernel, stride, pad, dilation: tiles of 128 and of 64 pixels, alone and over clusters of 2, 4, 5, 6 and 8;
    # channels that end inside a step, columns and pixels inside a tile, strides, dilations, padding wider than the window
    (5, 60, 45, 54, 374, 3, 1, 0, 2), (4, 43, 38, 115, 286, 1, 1, 1, 1), (2, 43, 41, 262, 214, 3, 1, 3, 1), (3, 48, 27, 296, 367, 1, 1, 0, 1),
    (4, 44, 14, 157, 237, 3, 1, 0, 1), (4, 43, 26, 25, 183, 5, 1, 1, 1), (6, 45, 30, 57, 33, 3, 1, 0, 1), (1, 6, 27, 355, 62, 5, 2, 4, 2),
    (4, 10, 22, 309, 87, 5, 3, 4, 2), (4, 41, 43, 106, 389, 5, 2, 2, 1), (2, 56, 55, 154, 86, 5, 1, 5, 2), (3, 45, 30, 25, 219, 5, 1, 2, 2),
    (5, 59, 21, 315, 92, 3, 1, 3, 2), (2, 30, 42, 121, 113, 3, 1, 3, 1), (3, 13, 18, 286, 362, 5, 1, 2, 1),
    (7, 43, 26, 25, 183, 5, 1, 1, 1), (1, 6, 27, 703, 62, 5, 2, 4, 2), (4, 10, 22, 701, 87, 5, 3, 4, 2), (3, 41, 43, 106, 389, 5, 2, 2, 1),
    (7, 45, 30, 25, 219, 5, 1, 2, 2)])
def test_fp32_contraction_by_the_copy_engine(shape):
    import ctypes as C
    import torch
    from ogle_b200 import _lib, ops
    N, H, W, ci, K, k, s, pd, d = shape
    g = torch.Generator(device="cuda").manual_seed(ci + K)
    x = torch.zeros((N, H, W, ops.up4(ci)), device="cuda")
    x[..., :ci] = torch.randn((N, H, W, ci), generator=g, device="cuda")
    w, b = torch.randn((K, ci, k, k), generator=g, device="cuda"), torch.randn(K, generator=g, device="cuda")
    p = ops.conv_params(N, H, W, ci, K, k, s, pd, d, 1, True, ops.ACT_CLIP, -3.0, 40.0, ops.MATH_FP32)
    if k == 1 and pd == 0:
        p.min_value = 0.0           # (a pointwise clip is to [0, max])
    # (five layers that the other form serves at least as fast: 35.8 us against 38.1, 67.9 and 70.3, 60.5 and 60.6, 116.1 and 117.2, 36.4 and 40.0)
    other = shape in ((4, 43, 26, 25, 183, 5, 1, 1, 1), (1, 6, 27, 355, 62, 5, 2, 4, 2), (4, 10, 22, 309, 87, 5, 3, 4, 2),
                      (4, 41, 43, 106, 389, 5, 2, 2, 1), (3, 45, 30, 25, 219, 5, 1, 2, 2))
    assert _lib.cuda_lib().ogle_cuda_conv2d_kernel_name(C.byref(p)) == (b"conv_igemm_kernel" if other else b"conv_igemm_tma_kernel")
    got = ops.conv2d(p, x, ops.conv2d_prepack(p, w), b)
    x64 = x[..., :ci].permute(0, 3, 1, 2).double()
    conv = lambda u, v, c: torch.nn.functional.conv2d(u, v, c, s, pd, d).permute(0, 2, 3, 1)
    want = conv(x64, w.double(), b.double()).clamp(p.min_value, 40.0)
    # every partial sum rounded once: at most (terms) * 2^-24 of the sum of the terms' magnitudes
    bound = (k * k * ci + 4) * 2.0 ** -24 * conv(x64.abs(), w.double().abs(), b.double().abs())
    assert ((got[..., :K].double() - want).abs() <= bound).all()
    assert (got[..., K:] == 0).all()


@pytest.mark.parametrize("shape", [
    # N, H, C, K, kernel, stride: the fp32 contraction by the copy engine in one piece, over clusters, of a matrix;
    # the direct stem with more tiles than stages, and fewer
    (16, 40, 96, 160, 3, 1), (8, 14, 256, 256, 3, 1), (32, 56, 96, 200, 1, 1), (64, 150, 3, 32, 3, 2), (2, 20, 3, 64, 3, 1)])
def test_fp32_waits_that_run_out(shape):
    """Limits at which some threads or blocks give up and others do not: the launch returns, with the status set or with the
    result, and the next one is right again."""
    import ctypes as C
    import torch
    from ogle_b200 import _lib, ops
    lib = _lib.cuda_lib()
    N, H, ci, K, k, s = shape
    g = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda *d: torch.randn(d, generator=g, device="cuda")
    x, w, b = torch.zeros((N, H, H, ops.up4(ci)), device="cuda"), rand(K, ci, k, k) / (ci * k * k) ** 0.5, rand(K)
    x[..., :ci] = rand(N, H, H, ci)
    p = ops.conv_params(N, H, H, ci, K, k, s, k // 2, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, ops.MATH_FP32)
    assert lib.ogle_cuda_conv2d_kernel_name(C.byref(p)) == (b"conv3x3_smallc_kernel" if ci == 3 else b"conv_igemm_tma_kernel")
    packed = ops.conv2d_prepack(p, w)
    want = ops.conv2d(p, x, packed, b)
    seen = set()
    try:
        for limit in [0, 1, 2, 3, 4, 6, 8, 11, 16, 23, 32, 64, 128, 256, 1024, 4096] * 2:
            lib.ogle_cuda_set_wait_limit(limit)
            got = ops.conv2d(p, x, packed, b)
            status = lib.ogle_cuda_device_status()
            assert status == -6 or (status == 0 and torch.equal(got, want)), (limit, status)
            seen.add(status)
            lib.ogle_cuda_clear_device_status()
    finally:
        lib.ogle_cuda_set_wait_limit(-1)
        lib.ogle_cuda_clear_device_status()
    assert -6 in seen
    assert torch.equal(ops.conv2d(p, x, packed, b), want) and lib.ogle_cuda_device_status() == 0


def test_fp32_gemm_of_many_columns():
    """Up to 65535 column tiles of 64."""
    import torch
    from ogle_b200 import ops
    k, n = 4, 65535 * 64
    a, b = torch.randn((1, k), device="cuda"), torch.randn((k, n), device="cuda")
    got = ops.gemm(a, b, None, 1, k, n, 0, 1.0, 0.0, 0, ops.MATH_FP32)
    want = a.double() @ b.double()
    # four products, each sum rounded: 2^-23 of the terms' magnitudes at most
    assert ((got.double() - want).abs() <= 2.0 ** -22 * (a.abs().double() @ b.abs().double())).all()


def test_fp32_convolution_of_an_image_of_2_to_the_31_pixels():
    """One image that 32-bit pixel numbers do not reach (34 GB of them), every 64th pixel of it taken."""
    import torch
    from ogle_b200 import ops
    if torch.cuda.mem_get_info()[0] < 45 << 30:
        pytest.skip("needs 45 GB of device memory")
    h, w, s = 65536, 32768, 64
    x = torch.zeros((1, h, w, 4), device="cuda")
    picked = torch.randn((h // s, w // s), device="cuda")
    x[0, ::s, ::s, 0] = picked
    p = ops.conv_params(1, h, w, 1, 8, 1, s, 0, 1, 1, True, 0, 0.0, 0.0, ops.MATH_FP32)
    f, b = torch.randn((8, 1, 1, 1), device="cuda"), torch.randn(8, device="cuda")
    y = ops.conv2d(p, x, ops.conv2d_prepack(p, f), b)
    assert torch.equal(y[0], picked[..., None] * f.flatten() + b)       # one product, rounded, and one sum
    del x
    torch.cuda.empty_cache()


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, kernel, stride, pad, act, split: one tile over 2-8 blocks, ranges of unequal length, rows and columns
    # that end inside a tile, several tiles, three tile widths
    (1, 7, 7, 512, 30, 3, 1, 1, 0, 8), (1, 9, 11, 100, 129, 3, 2, 1, 2, 3), (2, 19, 19, 256, 75, 3, 1, 1, 1, 5), (1, 1, 1, 96, 4, 1, 1, 0, 2, 3),
    (3, 20, 17, 64, 510, 1, 1, 0, 2, 2), (1, 40, 150, 48, 33, 5, 1, 2, 0, 7), (5, 3, 3, 160, 257, 1, 1, 0, 0, 4),
    # ranges of two, two and one chunk; a map cut along the width
    (5, 3, 3, 160, 257, 1, 1, 0, 0, 3), (1, 12, 75, 48, 33, 5, 1, 2, 0, 4)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_reduction_split_inside_a_cluster(oracle_port, shape, math):
    """Into a channel slice of a wider tensor, alone and with a residual operand; the same sums on every call."""
    import torch
    from ogle_b200 import ops
    N, H, W, C, K, k, s, pd, act, split = shape
    rng = np.random.default_rng(C + K)
    x = rng.standard_normal((N, H, W, C), dtype=np.float32)
    w = (rng.standard_normal((K, C, k, k)) / np.sqrt(C * k * k)).astype(np.float32)
    b = rng.standard_normal(K, dtype=np.float32)
    p = ops.conv_params(N, H, W, C, K, k, s, pd, 1, 1, True, act, -0.5, 1.5, getattr(ops, math))
    p.split = split
    # (60 tiles of the map that is 150 wide are more clusters of seven blocks than fit, and no scratch is lent; five
    # chunks do not make four ranges)
    form = (1, 1) if W == 150 or (C == 160 and split == 4) else (3, split)
    packed = ops.conv2d_prepack(p, ops.dense_to_device(w))
    x4, b4 = ops.upload(x), ops.dense_to_device(b)
    if act != 1:
        res = rng.standard_normal((N,) + tuple(p.out_hwc), dtype=np.float32)
        fused = ops.conv2d_residual(p, x4, packed, b4, ops.upload(res))
        assert (ops.last_contraction().form, ops.last_contraction().ranges) == form
    p.out_channel_stride, p.out_channel_offset = ops.up4(K) + 8, 4
    outs = [torch.full((N, p.out_hwc[0], p.out_hwc[1], ops.up4(K) + 8), -7.0, device="cuda") for _ in range(2)]
    for out in outs:
        ops.conv2d(p, x4, packed, b4, out, workspace=None)
        assert (ops.last_contraction().form, ops.last_contraction().ranges) == form
    assert torch.equal(outs[0], outs[1])
    got = outs[0].cpu().numpy()
    assert (got[..., :4] == -7).all() and (got[..., 4 + ops.up4(K):] == -7).all() and (got[..., 4 + K:4 + ops.up4(K)] == 0).all()
    # fp32-grade products and sums, or operands of ten mantissa bits (2^-11 relative each) over the reduction
    tol = 3e-5 if math == "MATH_TF32X3" else 6e-3
    ref = oracle_port.conv2d(x, w, b, s, pd, 1, 1, act, -0.5, 1.5)
    assert np.abs(got[..., 4:4 + K] - ref).max() <= tol * max(1.0, np.abs(ref).max())
    if act != 1:
        plain = oracle_port.conv2d(x, w, b, s, pd, 1, 1, 0, 0.0, 0.0) + res
        want = np.maximum(plain, 0) if act == 2 else plain
        assert np.abs(ops.download(fused, K) - want).max() <= tol * np.abs(plain).max()


@pytest.mark.parametrize("m,k,n,bias_mode", [(1, 512, 1000, 2), (1, 130, 10, 0), (129, 1500, 700, 1), (300, 4096, 33, 2), (1000, 1500, 700, 2)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_gemm_over_clusters(m, k, n, bias_mode, math):
    """Launches of few tiles, whose reductions split over clusters: vector and matrix bias, odd sizes, against 64 bits."""
    import torch
    from ogle_b200 import ops
    g = torch.Generator().manual_seed(m + k)
    a, b = torch.randn((m, k), generator=g), torch.randn((n, k), generator=g)
    c = torch.randn((n,) if bias_mode == 2 else (m, n), generator=g)
    c4 = None if bias_mode == 0 else torch.nn.functional.pad(c, (0, ops.up4(n) - n)).cuda()
    pad = lambda t: torch.nn.functional.pad(t, (0, ops.up4(k) - k)).cuda()
    mode = getattr(ops, math)
    got = ops.gemm_ws(pad(a), pad(b), c4, m, k, n, 1, 0.5, 2.0 if bias_mode else 0.0, bias_mode, mode)
    # (five chunks gain nothing, and a split-mode result may not move as far as it would with a cut of 4096 elements)
    assert ops.last_contraction().form == (1 if k == 130 or (k == 4096 and mode == ops.MATH_TF32X3) else 3)
    want = 0.5 * (a.double() @ b.double().t()) + (2.0 * c.double() if bias_mode else 0.0)
    err = (got[:, :n].cpu().double() - want).norm() / want.norm()
    # k/8 + k/16 truncated additions to a sum, each off by at most 2^-23 of it, 2^-24 on average: k * 1.1e-8 in an
    # unsplit reduction, less in a split one; in one-pass mode 2^-11 per operand
    assert err <= (1.2e-8 * k + 2e-6 if mode == ops.MATH_TF32X3 else 2e-3)
    assert (got[:, n:] == 0).all()


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, kernel, stride, pad: maps cut along the width (75, 70, 150, 129 pixels), reductions of eight chunks
    # and more whose tile width and form the launch chooses (pairs of SMs among them)
    (2, 75, 75, 20, 40, 3, 1, 1), (3, 141, 139, 17, 30, 3, 2, 1), (1, 150, 150, 32, 96, 3, 1, 1), (2, 9, 129, 16, 8, 3, 1, 1),
    (3, 66, 90, 32, 160, 5, 1, 2), (6, 60, 64, 40, 256, 3, 1, 1), (1, 120, 120, 288, 250, 1, 1, 0)])
def test_tile_choice_keeps_the_sums(oracle_port, shape):
    """Whatever tiles an unsplit launch chooses, an output value sums its reduction in the same order: the bits of the
    launch with a fixed width on single SMs, with and without a residual operand."""
    import torch
    from ogle_b200 import ops
    N, H, W, C, K, k, s, pd = shape
    rng = np.random.default_rng(W + K)
    x = rng.standard_normal((N, H, W, C), dtype=np.float32)
    w = (rng.standard_normal((K, C, k, k)) / np.sqrt(C * k * k)).astype(np.float32)
    b = rng.standard_normal(K, dtype=np.float32)
    x4, b4, w4 = ops.upload(x), ops.dense_to_device(b), ops.dense_to_device(w)
    ref = oracle_port.conv2d(x[:1], w, b, s, pd, 1, 1, 2, 0.0, 0.0)
    for math, tol in ((ops.MATH_TF32X3, 3e-5), (ops.MATH_TF32, 6e-3)):
        outs, fused = [], []
        for n_tile, pair in ((0, 0), (32, 1)):
            p = ops.conv_params(N, H, W, C, K, k, s, pd, 1, 1, True, 2, 0.0, 0.0, math)
            p.split, p.n_tile, p.sm_pair = 1, n_tile, pair
            packed = ops.conv2d_prepack(p, w4)
            res = ops.upload(np.random.default_rng(1).standard_normal((N,) + tuple(p.out_hwc), dtype=np.float32))
            outs.append(ops.conv2d(p, x4, packed, b4, workspace=None))
            fused.append(ops.conv2d_residual(p, x4, packed, b4, res))
        assert torch.equal(outs[0], outs[1]) and torch.equal(fused[0], fused[1])
        assert np.abs(ops.download(outs[0], K)[:1] - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("m,k,n", [(256, 1024, 300), (2560, 512, 1024), (64, 4096, 512), (3000, 96, 200)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_products_queued_on_one_workspace(m, k, n, math):
    """Each call's packing pass overwrites what the product before it reads, and each product starts its set-up while the
    packing pass before it still runs: six of them queued without a wait between, each against its own packed B."""
    import torch
    from ogle_b200 import ops
    mode = getattr(ops, math)
    g = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randn((m, k), generator=g, device="cuda")
    bs = [torch.randn((k, n), generator=g, device="cuda") for _ in range(6)]
    packs = [ops.gemm_pack_b(b, m, k, n, 0, mode) for b in bs]
    wants = [ops.gemm_packed(a, p, None, m, k, n, 0, 1.0, 0.0, 0, mode) for p in packs]
    workspace = torch.empty_like(packs[0])
    torch.cuda.synchronize()
    gots = [ops.gemm_ws(a, b, None, m, k, n, 0, 1.0, 0.0, 0, mode, workspace=workspace) for b in bs]
    for got, want in zip(gots, wants):
        assert torch.equal(got, want)


@pytest.mark.parametrize("width", [75, 90, 150])
def test_cut_tiles_with_channels_on_m(oracle_port, width):
    """Maps cut along the width in the channels-on-M form, whose residual operand is then found pixel by pixel, and with
    two outputs: the bits of the plain form."""
    import torch
    from ogle_b200 import ops
    N, H, C, K = 3, 41, 64, 70
    g = torch.Generator(device="cuda").manual_seed(width)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, w, b, res = rand(N, H, width, C), rand(K, C, 3, 3) / 24.0, rand(K), rand(N, H, width, ops.up4(K))
    for math in (ops.MATH_TF32X3, ops.MATH_TF32):
        outs = []
        for on_m in (1, 2):
            p = ops.conv_params(N, H, width, C, K, 3, 1, 1, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, math)
            p.split, p.channels_on_m, p.sm_pair = 1, on_m, 1
            packed = ops.conv2d_prepack(p, w)
            outs += [ops.conv2d(p, x, packed, b, workspace=None), ops.conv2d_residual(p, x, packed, b, res)]
            assert ops.last_contraction().form == (5 if on_m == 2 else 1)
        assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[3])
        one, two = ops.conv2d_pair(x, w[:24], b[:24], w[24:64], b[24:64], N, H, width, C, 3, 1, 1, 1, ops.ACT_RELU, 0.0, 0.0, math,
                                   use_workspace=False)
        assert torch.equal(one, outs[0][..., :24]) and torch.equal(two, outs[0][..., 24:64])


TAPS_CODE = """
import sys, torch
from ogle_b200 import ops
g = torch.Generator(device="cuda").manual_seed(3)
rand = lambda *s: torch.randn(s, generator=g, device="cuda")
# N, H, W, C, K: one pixel a row and one row an image, tiles that end at, before and behind a row, an image and the tensor
# (126 pixels each), channels and filters that fill no chunk, slab or tile
for N, H, W, C, K in [(126, 1, 1, 32, 32), (127, 1, 1, 16, 4), (1, 1, 125, 32, 64), (1, 1, 127, 32, 64), (64, 2, 1, 40, 64), (3, 6, 7, 64, 65), (2, 7, 9, 70, 33),
                      (1, 126, 2, 32, 96), (2, 3, 126, 64, 64), (5, 16, 128, 36, 100), (4, 56, 56, 64, 64), (150, 28, 28, 32, 130), (3, 90, 129, 100, 62)]:
    for math in (ops.MATH_TF32X3, ops.MATH_TF32):
        for act in (ops.ACT_NONE, ops.ACT_RELU, ops.ACT_CLIP):
            p = ops.conv_params(N, H, W, C, K, 3, 1, 1, 1, 1, True, act, -0.5, 1.5, math)
            p.split = 1
            x = torch.zeros((N, H, W, ops.up4(C)), device="cuda")
            x[..., :C] = rand(N, H, W, C)
            w, b, res = rand(K, C, 3, 3) / (9 * C) ** 0.5, rand(K), rand(N, H, W, ops.up4(K))
            packed = ops.conv2d_prepack(p, w)
            sums = torch.nn.functional.conv2d(x[..., :C].permute(0, 3, 1, 2).double(), w.double(), b.double(), padding=1).permute(0, 2, 3, 1)
            finish = lambda v: v if act == ops.ACT_NONE else (v.clamp(min=0) if act == ops.ACT_RELU else v.clamp(-0.5, 1.5))
            # split mode: sums in tensor memory lose 6e-9 of their norm per element, products and operands 1e-6; one pass:
            # operands of ten mantissa bits, the activation's cut off (2^-10 at most, half of it on average)
            bound = (2e-6 + 6e-9 * 9 * C if math == ops.MATH_TF32X3 else 1e-3) * float(sums.norm())
            def check(got, want, form=6):
                assert ops.last_contraction().form == form, (N, H, W, C, K, ops.last_contraction().form)
                assert float((got.double() - want).norm()) <= bound, (N, H, W, C, K, math, act, float((got.double() - want).norm()) / bound)
            wide = torch.full((N, H, W, ops.up4(K) + 8), -7.0, device="cuda")
            p.out_channel_stride, p.out_channel_offset = ops.up4(K) + 8, 4
            ops.conv2d(p, x, packed, b, wide)
            check(wide[..., 4:4 + K], finish(sums))
            assert (wide[..., :4] == -7).all() and (wide[..., 4 + ops.up4(K):] == -7).all() and (wide[..., 4 + K:4 + ops.up4(K)] == 0).all()
            p.out_channel_stride = p.out_channel_offset = 0
            plain = ops.conv2d(p, x, packed, b)
            assert torch.equal(plain[..., :K], wide[..., 4:4 + K])
            if act != ops.ACT_CLIP:
                check(ops.conv2d_residual(p, x, packed, b, res)[..., :K], finish(sums + res[..., :K]))
            for tile, pair in ((32, 0), (0, 2)):                      # neither touches the bits
                p.n_tile, p.sm_pair = tile, pair
                assert torch.equal(ops.conv2d(p, x, packed, b), plain)
"""


def test_taps_side_by_side_at_the_edges_of_their_tiles():
    """Forced (the switch is read once per process), so that the smallest launches take the form too."""
    import subprocess
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", TAPS_CODE], cwd=root, env=dict(os.environ, OGLE_TC_TAPS="1"), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


def test_taps_side_by_side_two_outputs_and_bounded_waits():
    """By the library's own choice: the two outputs of sibling layers, and roles that give up at once."""
    import torch
    from ogle_b200 import _lib, ops
    lib = _lib.cuda_lib()
    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    N, H, C, K = 64, 38, 64, 52
    x, w, b = rand(N, H, H, C), rand(K, C, 3, 3) / 24.0, rand(K)
    for math in (ops.MATH_TF32X3, ops.MATH_TF32):
        p = ops.conv_params(N, H, H, C, K, 3, 1, 1, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, math)
        packed = ops.conv2d_prepack(p, w)
        want = ops.conv2d(p, x, packed, b, workspace=None)
        assert ops.last_contraction().form == 6
        one, two = ops.conv2d_pair(x, w[:20], b[:20], w[20:], b[20:], N, H, H, C, 3, 1, 1, 1, ops.ACT_RELU, 0.0, 0.0, math, use_workspace=False)
        assert ops.last_contraction().form == 6
        assert torch.equal(one, want[..., :20]) and torch.equal(two, want[..., 20:])
        try:
            assert lib.ogle_cuda_device_status() == 0
            lib.ogle_cuda_set_wait_limit(0)
            ops.conv2d(p, x, packed, b, workspace=None)
            assert lib.ogle_cuda_device_status() == -6 and 1 <= lib.ogle_cuda_device_status_detail() <= 7
        finally:
            lib.ogle_cuda_set_wait_limit(-1)
            lib.ogle_cuda_clear_device_status()
        assert torch.equal(ops.conv2d(p, x, packed, b, workspace=None), want)
        assert lib.ogle_cuda_device_status() == 0


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, math: near the line between whole tiles and taps side by side, where tiles laid out for a split reduction
    # (no activation), or widths chosen with scratch at hand, would have it fall to either side
    (1, 34, 34, 192, 512, "MATH_TF32"), (1, 67, 56, 160, 150, "MATH_TF32"), (21, 10, 36, 191, 294, "MATH_TF32"),
    (4, 77, 11, 176, 316, "MATH_TF32"), (2, 37, 108, 218, 122, "MATH_TF32"), (128, 47, 61, 512, 512, "MATH_TF32X3")])
def test_taps_by_shape_alone(shape):
    """Unsplit, a layer's bits depend neither on scratch nor on where the residual operand and the activation are applied."""
    import torch
    from ogle_b200 import ops
    N, H, W, C, K, math = shape
    g = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda *d: torch.randn(d, generator=g, device="cuda")
    x, w, b = torch.zeros((N, H, W, ops.up4(C)), device="cuda"), rand(K, C, 3, 3) / (9 * C) ** 0.5, rand(K)
    x[..., :C] = rand(N, H, W, C)
    res = rand(N, H, W, ops.up4(K))
    res[..., K:] = 0.0
    lent = torch.empty(48 << 18, device="cuda")
    p = ops.conv_params(N, H, W, C, K, 3, 1, 1, 1, 1, True, ops.ACT_NONE, 0.0, 0.0, getattr(ops, math))
    p.split = 1
    packed = ops.conv2d_prepack(p, w)
    plain = ops.conv2d(p, x, packed, b, workspace=None)
    form = ops.last_contraction().form
    assert torch.equal(ops.conv2d(p, x, packed, b, workspace=lent), plain)
    p.act = ops.ACT_RELU
    for scratch in (None, lent):
        assert torch.equal(ops.conv2d(p, x, packed, b, workspace=scratch), plain.clamp(min=0))
    assert torch.equal(ops.conv2d_residual(p, x, packed, b, res), (plain + res).clamp(min=0))
    assert (ops.last_contraction().form == 6) == (form == 6)


WHOLE_CODE = """
import torch
from ogle_b200 import _lib, ops
g = torch.Generator(device="cuda").manual_seed(11)
rand = lambda *s: torch.randn(s, generator=g, device="cuda")
# 3x3 layers of stride 1 which by themselves would lie with their taps side by side: in whole tiles of every width and on
# pairs of SMs, rows of an image, several images and pieces of a row to a tile
for N, H, W, C, K in [(2, 38, 38, 64, 256), (6, 60, 64, 40, 256), (2, 75, 75, 20, 64), (1, 150, 150, 32, 96), (40, 28, 28, 64, 130), (200, 7, 9, 70, 128)]:
    x = torch.zeros((N, H, W, ops.up4(C)), device="cuda")
    x[..., :C] = rand(N, H, W, C)
    w, b = rand(K, C, 3, 3) / (9 * C) ** 0.5, rand(K)
    want = torch.nn.functional.conv2d(x[..., :C].permute(0, 3, 1, 2).double(), w.double(), b.double(), padding=1).permute(0, 2, 3, 1)
    for math in (ops.MATH_TF32X3, ops.MATH_TF32):
        p = ops.conv_params(N, H, W, C, K, 3, 1, 1, 1, 1, True, ops.ACT_NONE, 0.0, 0.0, math)
        p.split, p.channels_on_m = 1, 1
        packed = ops.conv2d_prepack(p, w)
        outs = []
        for n_tile, pair in [(bn, 1) for bn in range(32, 257, 32) if bn <= (K + 31) // 32 * 32] + [(bn, 2) for bn in (64, 128, 192, 256) if bn <= (K + 31) // 32 * 32]:
            p.n_tile, p.sm_pair = n_tile, pair
            outs.append(ops.conv2d(p, x, packed, b, workspace=None))
            assert (ops.last_contraction().form, ops.last_contraction().n_tile) == (1 if pair == 1 else 4, n_tile), (N, K, n_tile, pair, ops.last_contraction().form)
            assert torch.equal(outs[0], outs[-1]), (N, H, C, K, math, n_tile, pair)
        # (the bound of the taps' test)
        assert float((outs[0][..., :K].double() - want).norm()) <= (2e-6 + 6e-9 * 9 * C if math == ops.MATH_TF32X3 else 1e-3) * float(want.norm())
assert _lib.cuda_lib().ogle_cuda_device_status() == 0
"""


def test_whole_tiles_and_pairs_of_layers_that_take_taps():
    """The form switched off (the switch is read once per process), so that the others are compared on such layers too."""
    import subprocess
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", WHOLE_CODE], cwd=root, env=dict(os.environ, OGLE_TC_TAPS="0"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("shape", [(64, 28, 28, 64, 64), (16, 40, 30, 200, 96), (128, 14, 14, 256, 128)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_taps_are_as_near_to_64_bits_as_whole_tiles(shape, math):
    """A third of the length of a sum in tensor memory: split-mode results are nearer (1.8e-6 of the norm and 3.4e-6 at 576
    elements); in one pass the operands' ten bits are all there is to see."""
    import torch
    from ogle_b200 import ops
    N, H, W, C, K = shape
    g = torch.Generator(device="cuda").manual_seed(C)
    x = torch.rand((N, H, W, C), generator=g, device="cuda")
    w = torch.randn((K, C, 3, 3), generator=g, device="cuda") / (9 * C) ** 0.5 + 0.02
    want = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), w.double(), padding=1).permute(0, 2, 3, 1)
    p = ops.conv_params(N, H, W, C, K, 3, 1, 1, 1, 1, False, ops.ACT_NONE, 0.0, 0.0, getattr(ops, math))
    p.split = 1
    packed = ops.conv2d_prepack(p, w)
    errors, forms = [], []
    for p.channels_on_m in (0, 1):                                    # (1: whole tiles)
        errors.append(float((ops.conv2d(p, x, packed, workspace=None)[..., :K].double() - want).norm() / want.norm()))
        forms.append(ops.last_contraction().form)
    assert forms[1] in (1, 4) and (forms[0] == 6 or math == "MATH_TF32")
    assert errors[0] <= (0.8 if math == "MATH_TF32X3" else 1.001) * errors[1], errors


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_taps_keep_non_finite_values_in_their_windows(bad, math):
    """At the ends of rows and images, at the ends of tiles of 126 pixels and of warps: the values whose window holds one are
    not finite, all others are what they were."""
    import torch
    from ogle_b200 import ops
    N, H, W, C, K = 40, 31, 33, 64, 64
    g = torch.Generator(device="cuda").manual_seed(2)
    x, w = torch.randn((N, H, W, C), generator=g, device="cuda"), torch.randn((K, C, 3, 3), generator=g, device="cuda") / 24.0
    p = ops.conv_params(N, H, W, C, K, 3, 1, 1, 1, 1, False, ops.ACT_NONE, 0.0, 0.0, getattr(ops, math))
    p.split = 1
    packed = ops.conv2d_prepack(p, w)
    clean = ops.conv2d(p, x, packed, workspace=None)
    assert ops.last_contraction().form == 6
    flat = x.view(-1, C)
    M = N * H * W
    places = [W - 1, 2 * W, H * W - 1, H * W, M - 1, 0, 5 * H * W + 10 * W - 1, 125 + 126 * 40, 126 * 60, 126 * 80 + 31, 126 * 100 + 32, 126 * 120 + 95]
    hit = torch.zeros(M, device="cuda")
    for i in places:
        flat[i, 7] = bad
        hit[i] = 1.0
    hit = torch.nn.functional.max_pool2d(hit.view(N, 1, H, W), 3, 1, 1).view(N, H, W) > 0
    got = ops.conv2d(p, x, packed, workspace=None)
    assert not torch.isfinite(got[hit]).any()
    assert torch.equal(got[~hit], clean[~hit])


ON_M_CODE = """
import torch
from ogle_b200 import _lib, ops
g = torch.Generator(device="cuda").manual_seed(7)
rand = lambda *s: torch.randn(s, generator=g, device="cuda")
# many-tile 3x3 layers, which would lie with their taps side by side; the last has too many channels to lie on M
for N, H, W, C, K in [(128, 28, 28, 64, 64), (6, 75, 75, 40, 96), (9, 50, 61, 32, 128), (16, 28, 28, 128, 160)]:
    for math in (ops.MATH_TF32X3, ops.MATH_TF32):
        x, w, b = rand(N, H, W, C), rand(K, C, 3, 3) / (9 * C) ** 0.5, rand(K)
        res = rand(N, H, W, ops.up4(K))
        p = ops.conv_params(N, H, W, C, K, 3, 1, 1, 1, 1, True, ops.ACT_NONE, 0.0, 0.0, math)
        p.split = 1
        packed = ops.conv2d_prepack(p, w)
        want = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), w.double(), b.double(), padding=1).permute(0, 2, 3, 1)
        # (as for the taps: sums in tensor memory lose 6e-9 of their norm per element, products and operands 1e-6; one pass: 2^-10)
        bound = (2e-6 + 6e-9 * 9 * C if math == ops.MATH_TF32X3 else 1e-3) * float(want.norm())
        form = 5 if K <= 128 else 6
        for got, ref in ((ops.conv2d(p, x, packed, b, workspace=None), want), (ops.conv2d_residual(p, x, packed, b, res), want + res[..., :K])):
            assert ops.last_contraction().form == form, (N, H, W, C, K, math, ops.last_contraction().form)
            assert float((got[..., :K].double() - ref).norm()) <= bound, (N, H, W, C, K, math)
        if K == 64:
            one, two = ops.conv2d_pair(x, w[:20], b[:20], w[20:], b[20:], N, H, W, C, 3, 1, 1, 1, ops.ACT_NONE, 0.0, 0.0, math, use_workspace=False)
            assert ops.last_contraction().form == 5
            assert float((torch.cat([one[..., :20], two[..., :44]], -1).double() - want).norm()) <= bound
assert _lib.cuda_lib().ogle_cuda_device_status() == 0
"""


def test_channels_on_m_forced_on_layers_of_taps_side_by_side():
    """The switch that puts channels on M wherever they fit (switches are read once per process) comes before the taps' own."""
    import subprocess
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", ON_M_CODE], cwd=root, env=dict(os.environ, OGLE_TC_T="1", OGLE_TC_TAPS="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("K", [64, 128, 160])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_channels_on_m_only_where_it_runs(K, math):
    """Where channels on M cannot run, channels_on_m = 1 and 2 leave a layer as it is; where it can, the two give the same
    bits."""
    import torch
    from ogle_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    N, H = (64, 28) if K <= 128 else (8, 56)
    x, w, b = rand(N, H, H, 64), rand(K, 64, 3, 3) / 24.0, rand(K)
    p = ops.conv_params(N, H, H, 64, K, 3, 1, 1, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, getattr(ops, math))
    p.split = 1
    packed = ops.conv2d_prepack(p, w)
    outs, forms = [], []
    for p.channels_on_m in (0, 1, 2):
        outs.append(ops.conv2d(p, x, packed, b, workspace=None))
        forms.append(ops.last_contraction().form)
    assert forms[0] == 6 or math == "MATH_TF32"                        # (one pass, many channels: whole tiles)
    assert forms[1] in (1, 4) and forms[2] == 5 if K <= 128 else forms == forms[:1] * 3
    assert torch.equal(outs[1], outs[2]) and (K <= 128 or torch.equal(outs[0], outs[1]))


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, kernel, stride: one tile and many, rows and columns that end inside a tile or slab, several slabs a
    # group, pieces of images, the gather form
    (1, 3, 5, 64, 4, 1, 1), (3, 41, 67, 32, 70, 1, 1), (2, 61, 50, 48, 256, 1, 1), (7, 15, 13, 96, 130, 1, 2), (4, 27, 40, 40, 100, 3, 2),
    (3, 33, 150, 16, 33, 5, 1), (2, 64, 50, 3, 64, 7, 2), (2, 64, 50, 3, 130, 7, 2), (150, 56, 56, 32, 64, 1, 1)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_residual_operand_by_the_copy_engine(shape, math):
    """The values of the convolution, the residual added and the activation, in those single-precision steps; roles that
    give up with a copy of the operand in flight."""
    import torch
    from ogle_b200 import _lib, ops
    lib = _lib.cuda_lib()
    N, H, W, C, K, k, s = shape
    g = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda *d: torch.randn(d, generator=g, device="cuda")
    x, w, b = torch.zeros((N, H, W, ops.up4(C)), device="cuda"), rand(K, C, k, k) / (C * k * k) ** 0.5, rand(K)
    x[..., :C] = rand(N, H, W, C)
    p = ops.conv_params(N, H, W, C, K, k, s, k // 2, 1, 1, True, ops.ACT_NONE, 0.0, 0.0, getattr(ops, math))
    p.split = 1
    packed = ops.conv2d_prepack(p, w)
    plain = ops.conv2d(p, x, packed, b, workspace=None)
    res = rand(*plain.shape)
    res[..., K:] = 0.0
    for act in (ops.ACT_NONE, ops.ACT_RELU):
        p.act = act
        got = ops.conv2d_residual(p, x, packed, b, res)
        # (64 channels of a stem are gathered in split mode only: in one pass the window is the operand)
        assert ops.last_contraction().form in ((9,) if C == 3 and K == 64 and math == "MATH_TF32" else (1, 6))
        assert torch.equal(got, plain + res if act == ops.ACT_NONE else (plain + res).clamp(min=0))
    try:
        lib.ogle_cuda_set_wait_limit(0)
        ops.conv2d_residual(p, x, packed, b, res)
        assert lib.ogle_cuda_device_status() == -6
    finally:
        lib.ogle_cuda_set_wait_limit(-1)
        lib.ogle_cuda_clear_device_status()
    assert torch.equal(ops.conv2d_residual(p, x, packed, b, res), got)


@pytest.mark.parametrize("shape", [
    # N, H, W, K, kernel, stride: maps of few rows, whose windows are up to 134 pixels wide (of as many rows as fit), and the
    # widths, strides and channel counts at which they are not
    (3, 1, 300, 64, 5, 1), (2, 1, 128, 40, 7, 1), (2, 3, 257, 130, 5, 1), (9, 5, 128, 64, 5, 1), (2, 2, 200, 64, 5, 2), (3, 1, 1000, 224, 5, 1),
    (3, 1, 300, 250, 5, 1), (2, 1, 127, 256, 5, 1), (2, 4, 16, 64, 7, 1)])
@pytest.mark.parametrize("channels", [3, 2])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_stems_of_flat_maps(shape, channels, math):
    import torch
    from ogle_b200 import ops
    N, H, W, K, k, s = shape
    g = torch.Generator(device="cuda").manual_seed(W + K)
    x = torch.zeros((N, H, W, 4), device="cuda")
    x[..., :channels] = torch.randn((N, H, W, channels), generator=g, device="cuda")
    w, b = torch.randn((K, channels, k, k), generator=g, device="cuda") / (3 * k * k) ** 0.5, torch.randn(K, generator=g, device="cuda")
    p = ops.conv_params(N, H, W, channels, K, k, s, k // 2, 1, 1, True, ops.ACT_NONE, 0.0, 0.0, getattr(ops, math))
    packed = ops.conv2d_prepack(p, w)
    want = torch.nn.functional.conv2d(x[..., :channels].permute(0, 3, 1, 2).double(), w.double(), b.double(), s, k // 2).permute(0, 2, 3, 1)
    # 147 products and sums of fp32 grade, or of operands with ten mantissa bits
    bound = (3e-6 if math == "MATH_TF32X3" else 1e-3) * float(want.norm())
    got = ops.conv2d(p, x, packed, b, workspace=None)
    # (up to 64 channels the window is the operand, but on maps of which its tiles would be half empty)
    window = K <= 64 and (H, W) not in ((4, 16), (2, 200))
    assert (ops.last_contraction().form == 9) == window
    assert float((got[..., :K].double() - want).norm()) <= bound
    res = torch.randn(got.shape, generator=g, device="cuda")
    p.split = 1
    got = ops.conv2d_residual(p, x, packed, b, res)
    assert (ops.last_contraction().form == 9) == window
    assert float((got[..., :K].double() - want - res[..., :K].double()).norm()) <= bound


def test_flat_maps_fill_their_tiles():
    """A map one row high takes about what a square one of as many pixels does: 1.05 of it with tiles of a row, 1.9 in tiles
    of two."""
    import torch
    from ogle_b200 import ops

    def took(N, H, W):
        g = torch.Generator(device="cuda").manual_seed(W)
        p = ops.conv_params(N, H, W, 3, 64, 5, 1, 2, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, ops.MATH_TF32)
        packed = ops.conv2d_prepack(p, torch.randn((64, 3, 5, 5), generator=g, device="cuda") / 8.0)
        x, b = torch.randn((N, H, W, 4), generator=g, device="cuda"), torch.randn(64, generator=g, device="cuda")
        return _median_us(lambda: ops.conv2d(p, x, packed, b, workspace=None))

    assert took(512, 1, 1024) <= 1.4 * took(32, 128, 128)


@pytest.mark.parametrize("shape", [
    # N, H, W, K, kernel, stride: one tile, several a block, tiles that hang over every edge; filters that fit beside the windows and
    # not (of up to 48 channels the window is the operand, unless its tiles cover the map badly)
    (1, 32, 32, 16, 7, 2), (9, 113, 75, 64, 7, 2), (40, 70, 70, 40, 5, 1), (3, 130, 130, 128, 7, 1), (5, 64, 64, 200, 5, 2), (30, 64, 64, 8, 3, 2),
    (1, 8, 16, 16, 7, 1), (100, 7, 75, 40, 5, 1)])
def test_kept_filters_and_windows_of_rgb_stems(shape):
    """Filters copied once a block and a window once a tile, against copies per chunk - the form with a residual operand, here
    zeros - bit for bit, and with roles that give up."""
    import torch
    from ogle_b200 import _lib, ops
    lib = _lib.cuda_lib()
    N, H, W, K, k, s = shape
    g = torch.Generator(device="cuda").manual_seed(K)
    x = torch.zeros((N, H, W, 4), device="cuda")
    x[..., :3] = torch.randn((N, H, W, 3), generator=g, device="cuda")
    w, b = torch.randn((K, 3, k, k), generator=g, device="cuda") / (3 * k * k) ** 0.5, torch.randn(K, generator=g, device="cuda")
    p = ops.conv_params(N, H, W, 3, K, k, s, k // 2, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, ops.MATH_TF32X3)
    packed = ops.conv2d_prepack(p, w)
    want = torch.nn.functional.conv2d(x[..., :3].permute(0, 3, 1, 2).double(), w.double(), b.double(), s, k // 2).permute(0, 2, 3, 1).clamp(min=0)
    got = ops.conv2d(p, x, packed, b, workspace=None)
    # 147 products and sums of fp32 grade
    assert float((got[..., :K].double() - want).norm()) <= 3e-6 * float(want.norm())
    if k == 3:
        return                                                        # (the direct kernel's)
    # all filters, two windows and the staging slabs in 224 KB, and one filter tile
    window = shape in ((1, 32, 32, 16, 7, 2), (40, 70, 70, 40, 5, 1))
    assert ops.last_contraction().form == (9 if window else 7 if K <= 64 else 1)
    assert torch.equal(ops.conv2d_residual(p, x, packed, b, torch.zeros_like(got)), got)
    assert ops.last_contraction().form == (9 if window else 1)
    try:
        lib.ogle_cuda_set_wait_limit(0)
        ops.conv2d(p, x, packed, b, workspace=None)
        assert lib.ogle_cuda_device_status() == -6
    finally:
        lib.ogle_cuda_set_wait_limit(-1)
        lib.ogle_cuda_clear_device_status()
    assert torch.equal(ops.conv2d(p, x, packed, b, workspace=None), got)


@pytest.mark.parametrize("form", ["whole", "whole, alternate tiles", "whole, residual", "taps", "taps, residual", "kept", "gather", "window", "scratch", "cluster", "pairs",
                                  "channels on M", "channels on M, turns"])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_waits_that_run_out_for_some(form, math):
    """Limits at which some roles, warps or blocks give up and others do not: the launch returns, with the status set or with
    the result, and the next one is right again."""
    import torch
    from ogle_b200 import _lib, ops
    lib = _lib.cuda_lib()
    # N, H, C, K, kernel, stride
    N, H, C, K, k, s = {"whole": (16, 40, 96, 160, 1, 1), "whole, alternate tiles": (64, 40, 32, 64, 1, 1), "whole, residual": (16, 40, 96, 160, 3, 2),
                        "taps": (64, 28, 64, 64, 3, 1), "taps, residual": (64, 28, 64, 32, 3, 1), "kept": (20, 112, 3, 64, 7, 2),
                        "gather": (20, 112, 3, 130, 7, 2), "window": (20, 112, 2, 64, 7, 2),
                        "scratch": (8, 10, 512, 100, 3, 1), "cluster": (1, 19, 256, 256, 1, 1), "pairs": (16, 40, 96, 256, 1, 1),
                        "channels on M": (32, 28, 64, 64, 3, 1), "channels on M, turns": (32, 28, 64, 128, 3, 1)}[form]
    g = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda *d: torch.randn(d, generator=g, device="cuda")
    x, w, b = torch.zeros((N, H, H, ops.up4(C)), device="cuda"), rand(K, C, k, k) / (C * k * k) ** 0.5, rand(K)
    x[..., :C] = rand(N, H, H, C)
    p = ops.conv_params(N, H, H, C, K, k, s, k // 2, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, getattr(ops, math))
    p.split = {"scratch": 12, "cluster": 4}.get(form, 1)
    p.sm_pair, p.channels_on_m = 2 if form == "pairs" else 0, 2 if "M" in form else 0
    p.n_tile = 128 if form == "pairs" else 0
    packed = ops.conv2d_prepack(p, w)
    res = rand(N, p.out_hwc[0], p.out_hwc[1], ops.up4(K))
    run = (lambda: ops.conv2d_residual(p, x, packed, b, res)) if "residual" in form else (lambda: ops.conv2d(p, x, packed, b))
    want = run()
    # (one pass keeps no filters: such a stem has its window for an operand)
    forms = {"taps": 6, "taps, residual": 6, "kept": 7 if math == "MATH_TF32X3" else 9, "window": 9, "scratch": 2, "cluster": 3, "pairs": 4}
    assert lib.ogle_cuda_device_status() == 0 and ops.last_contraction().form == forms.get(form, 5 if "M" in form else 1)
    seen = set()
    try:
        for limit in [0, 1, 2, 3, 4, 6, 8, 11, 16, 23, 32, 45, 64, 90, 128, 181, 256, 362, 512, 1024, 2048, 4096] * 2:
            lib.ogle_cuda_set_wait_limit(limit)
            got = run()
            status = lib.ogle_cuda_device_status()
            assert status == -6 or (status == 0 and torch.equal(got, want)), (limit, status)
            seen.add(status)
            lib.ogle_cuda_clear_device_status()
    finally:
        lib.ogle_cuda_set_wait_limit(-1)
        lib.ogle_cuda_clear_device_status()
    assert -6 in seen
    assert torch.equal(run(), want) and lib.ogle_cuda_device_status() == 0


def test_bounded_waits_of_the_cluster_form(oracle_port):
    """Zero polls allowed: every block of a cluster gives up, all meet at the cluster's barriers, the launch returns with
    the status word set, and with the limit restored the same call gives what it gave before."""
    import torch
    from ogle_b200 import _lib, ops
    lib = _lib.cuda_lib()
    g = torch.Generator(device="cuda").manual_seed(7)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, w, b = rand(1, 9, 9, 256), rand(80, 256, 3, 3) / 48.0, rand(80)
    assert lib.ogle_cuda_device_status() == 0
    try:
        for math in (ops.MATH_TF32, ops.MATH_TF32X3):
            p = ops.conv_params(1, 9, 9, 256, 80, 3, 1, 1, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, math)
            p.split = 6
            packed = ops.conv2d_prepack(p, w)
            want = ops.conv2d(p, x, packed, b, workspace=None)
            lib.ogle_cuda_set_wait_limit(0)
            ops.conv2d(p, x, packed, b, workspace=None)
            assert ops.last_contraction().form == 3
            assert lib.ogle_cuda_device_status() == -6 and 1 <= lib.ogle_cuda_device_status_detail() <= 7
            assert lib.ogle_cuda_clear_device_status() == 0
            lib.ogle_cuda_set_wait_limit(-1)
            assert torch.equal(ops.conv2d(p, x, packed, b, workspace=None), want)
            assert lib.ogle_cuda_device_status() == 0
    finally:
        lib.ogle_cuda_set_wait_limit(-1)
        lib.ogle_cuda_clear_device_status()


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, kernel: few tiles, whose reductions the library splits by itself inside clusters or through scratch
    (1, 19, 19, 512, 512, 1), (1, 10, 10, 1024, 150, 3), (2, 7, 7, 512, 512, 3), (1, 19, 19, 128, 300, 3), (4, 14, 14, 256, 256, 3),
    (1, 38, 38, 256, 90, 1)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_width_and_form_do_not_touch_the_sums(shape, math):
    """n_tile and sm_pair change how a launch is laid out, not its results, also where the library chooses the number of
    ranges of the reduction: with an activation and no scratch, with scratch, with a residual operand, two outputs."""
    import torch
    from ogle_b200 import ops
    N, H, W, C, K, k = shape
    g = torch.Generator(device="cuda").manual_seed(C + K)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, w, b, res = rand(N, H, W, C), rand(K, C, k, k) / (C * k * k) ** 0.5, rand(K), rand(N, H, W, ops.up4(K))
    lent = torch.empty(48 << 18, device="cuda")
    first = None
    for n_tile, pair in ((0, 0), (32, 0), (64, 0), (96, 1), (128, 0), (256, 0), (64, 2), (256, 2), (0, 2)):
        p = ops.conv_params(N, H, W, C, K, k, 1, k // 2, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, getattr(ops, math))
        p.n_tile, p.sm_pair = n_tile, pair
        packed = ops.conv2d_prepack(p, w)
        outs = [ops.conv2d(p, x, packed, b, workspace=None), ops.conv2d(p, x, packed, b, workspace=lent),
                ops.conv2d_residual(p, x, packed, b, res)]
        first = first or outs
        for a, c in zip(first, outs):
            assert torch.equal(a, c), (n_tile, pair)


@pytest.mark.parametrize("shape", [
    # N, H, C, K, kernel: heads and late layers whose reductions go through scratch in 2 to 16 ranges
    (1, 10, 1024, 150, 3), (8, 10, 1024, 150, 3), (1, 19, 512, 75, 3), (4, 5, 512, 150, 3), (4, 7, 512, 512, 3), (8, 10, 512, 1024, 1),
    (1, 5, 820, 100, 5), (2, 3, 256, 126, 3), (8, 10, 1024, 256, 1)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_clusters_do_not_take_longer_ranges(shape, math):
    """With scratch lent, a reduction that is added up inside clusters instead has at least as many ranges as the scratch
    was planned for (sums in tensor memory lose with their length), and is no further from 64 bits."""
    import ctypes as C
    import torch
    from ogle_b200 import _lib, ops
    N, H, ch, K, k = shape
    g = torch.Generator(device="cuda").manual_seed(ch + K)
    x = torch.rand((N, H, H, ch), generator=g, device="cuda")
    w = torch.randn((K, ch, k, k), generator=g, device="cuda") / (ch * k * k) ** 0.5 + 0.02
    want = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), w.double(), padding=k // 2).permute(0, 2, 3, 1)
    need = _lib.cuda_lib().ogle_cuda_conv2d_workspace_bytes

    def run(split):
        p = ops.conv_params(N, H, H, ch, K, k, 1, k // 2, 1, 1, False, ops.ACT_RELU, 0.0, 0.0, getattr(ops, math))
        p.split = split
        y = ops.conv2d(p, x, ops.conv2d_prepack(p, w))
        want_act = want.clamp(min=0)
        return ops.last_contraction().ranges, float((y[..., :K].double() - want_act).norm() / want_act.norm()), need(C.byref(p))

    ranges, err, planned = run(0)
    planned = round(planned * 4 / max(run(4)[2], 1)) if planned else 1
    assert ranges >= planned, (ranges, planned)
    # (two numbers of ranges that round alike differ by their remainders only)
    assert err <= 1.05 * run(planned)[1] + 1e-8


@pytest.mark.parametrize("m,k,n,form", [
    # reductions that clusters can still cut, and longer ones; columns for a warp each, for several and for four a warp
    (4, 2500, 1500, 3), (4, 2500, 3000, 8), (4, 2500, 1000, 8), (4, 2700, 1500, 8), (3, 2500, 1500, 8), (2, 2500, 5000, 3), (2, 2700, 5000, 8), (1, 2500, 5000, 8)])
def test_long_products_of_few_rows(m, k, n, form):
    """Which kernel serves them, and as exactly as either does."""
    import torch
    from ogle_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m * k + n)
    a, b = torch.randn((m, k), generator=g, device="cuda"), torch.randn((k, n), generator=g, device="cuda")
    got = ops.gemm_packed(a, ops.gemm_pack_b(b, m, k, n, 0, ops.MATH_TF32X3), None, m, k, n, 0, 1.0, 1.0, 0, ops.MATH_TF32X3)
    assert ops.last_contraction().form == form
    want = a.double() @ b.double()
    # products of fp32 grade; sums in tensor memory lose 6e-9 of the norm per element
    assert float((got.double() - want).norm()) <= (2e-5 if form == 3 else 5e-6) * float(want.norm())


@pytest.mark.parametrize("m,k,n,bias_mode", [
    # a row, two, up to four and up to eight; one to eight warps to a column, four columns to a warp; reductions and columns
    # that end inside a step, a piece, the pack's padding
    (1, 512, 1000, 2), (1, 5, 3, 1), (1, 131, 9473, 2), (1, 4099, 10, 0), (2, 1030, 77, 2), (2, 33, 4801, 0), (3, 129, 130, 1),
    (4, 2049, 300, 2), (4, 448, 1500, 2), (8, 864, 700, 0), (3, 3001, 2200, 0), (5, 64, 9, 1), (8, 700, 1001, 2), (7, 97, 6000, 2)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_products_of_few_rows(m, k, n, bias_mode, math):
    """Against 64 bits with B as the pack holds it, whose every product is rounded only as the sum is."""
    import torch
    from ogle_b200 import ops
    mode = getattr(ops, math)
    if mode == ops.MATH_TF32 and (m, k) == (3, 3001):
        pytest.skip("so many products of one pass are the tensor cores'")
    g = torch.Generator(device="cuda").manual_seed(m * k + n)
    pad = lambda t, v: torch.nn.functional.pad(t, (0, ops.up4(t.shape[-1]) - t.shape[-1]), value=v)
    a, b = torch.randn((m, k), generator=g, device="cuda"), torch.randn((n, k), generator=g, device="cuda")
    c = torch.randn((n,) if bias_mode == 2 else (m, n), generator=g, device="cuda")
    got = ops.gemm_packed(pad(a, float("nan")), ops.gemm_pack_b(pad(b, float("nan")), m, k, n, 1, mode),      # (NaN: never to be read)
                          None if bias_mode == 0 else pad(c, 0.0), m, k, n, 1, 0.5, 2.0 if bias_mode else 0.0, bias_mode, mode)
    assert ops.last_contraction().form == 8
    hi = (b.view(torch.int32) & ~0x1fff).view(torch.float32)
    held = (hi.double() + ((b - hi).bfloat16().double() if mode == ops.MATH_TF32X3 else 0.0)).t()
    bias = 2.0 * c.double() if bias_mode else torch.zeros((), dtype=torch.float64, device="cuda")
    want = 0.5 * (a.double() @ held) + bias
    # every partial sum rounded once: at most k * 2^-24 of the sum of the terms' magnitudes
    bound = (k + 8) * 2.0 ** -24 * (0.5 * (a.abs().double() @ held.abs()) + bias.abs())
    assert ((got[:, :n].double() - want).abs() <= bound).all()
    assert (got[:, n:] == 0).all()


def test_few_rows_whose_reduction_ends_inside_a_step():
    """A reduction of three and a half steps takes no longer than one of four (1.4 of it when lanes took turns)."""
    import torch
    from ogle_b200 import ops

    def took(k):
        g = torch.Generator(device="cuda").manual_seed(k)
        a, b = torch.randn((4, k), generator=g, device="cuda"), torch.randn((k, 1500), generator=g, device="cuda")
        packed = ops.gemm_pack_b(b, 4, k, 1500, 0, ops.MATH_TF32X3)
        call = lambda: ops.gemm_packed(a, packed, None, 4, k, 1500, 0, 1.0, 1.0, 0, ops.MATH_TF32X3)
        call()
        assert ops.last_contraction().form == 8
        return _median_us(_in_a_graph(call))

    assert took(448) <= 1.15 * took(512)


@pytest.mark.parametrize("shape", [
    # N, H, W, C, K, kernel, stride, pad, dilation: a pixel, two, some, several images; channels that end inside a piece;
    # padding, strides and dilations that leave taps outside the image
    (1, 1, 1, 256, 150, 3, 1, 1, 1), (1, 2, 1, 45, 33, 1, 1, 0, 1), (2, 1, 1, 130, 7, 5, 1, 2, 1), (1, 3, 3, 128, 220, 3, 2, 1, 1),
    (5, 2, 3, 50, 61, 3, 1, 1, 1), (1, 1, 4, 448, 200, 1, 1, 0, 1), (1, 5, 4, 97, 65, 3, 2, 3, 2), (32, 1, 1, 64, 36, 1, 1, 0, 1), (8, 2, 2, 128, 222, 3, 2, 1, 1)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
@pytest.mark.parametrize("output", ["alone", "slice", "residual", "pair"])
def test_convolutions_of_few_pixels(shape, math, output):
    """Against 64 bits with the filters as the pack holds them, whose every product is rounded only as the sum is: by
    itself, into a slice of a wider tensor, with a residual operand, as two convolutions in one."""
    import ctypes as C
    import torch
    from ogle_b200 import _lib, ops
    N, H, W, ci, K, k, s, pd, d = shape
    mode = getattr(ops, math)
    g = torch.Generator(device="cuda").manual_seed(ci + K)
    x = torch.zeros((N, H, W, ops.up4(ci)), device="cuda")
    x[..., :ci] = torch.randn((N, H, W, ci), generator=g, device="cuda")
    filters = [torch.randn((n, ci, k, k), generator=g, device="cuda") for n in ((K, 5) if output == "pair" else (K,))]
    biases = [torch.randn(w.shape[0], generator=g, device="cuda") for w in filters]
    p = ops.conv_params(N, H, W, ci, K, k, s, pd, d, 1, True, ops.ACT_RELU, 0.0, 0.0, mode)
    pixels = (N, p.out_hwc[0], p.out_hwc[1])
    res = torch.randn(pixels + (ops.up4(K),), generator=g, device="cuda")
    if output == "pair":
        gots = ops.conv2d_pair(x, filters[0], biases[0], filters[1], biases[1], N, H, W, ci, k, s, pd, d, ops.ACT_RELU, math_mode=mode)
    elif output == "residual":
        gots = [ops.conv2d_residual(p, x, ops.conv2d_prepack(p, filters[0]), biases[0], res)]
    elif output == "slice":
        p.out_channel_offset, p.out_channel_stride = 8, ops.up4(K) + 12
        wide = torch.full(pixels + (ops.up4(K) + 12,), 7.0, device="cuda")
        packed = ops.conv2d_prepack(p, filters[0])
        _lib.check(_lib.cuda_lib().ogle_cuda_conv2d(C.byref(p), ops._p(x), ops._p(packed), ops._p(biases[0]), ops._p(wide), ops._stream()), "conv2d")
        assert (wide[..., :8] == 7).all() and (wide[..., 8 + ops.up4(K):] == 7).all()
        gots = [wide[..., 8:8 + ops.up4(K)]]
    else:
        gots = [ops.conv2d(p, x, ops.conv2d_prepack(p, filters[0]), biases[0])]
        # (no tiles: how they are to be laid out does not matter)
        for name, value in (("n_tile", 32), ("sm_pair", 1), ("channels_on_m", 1)):
            setattr(p, name, value)
            assert torch.equal(ops.conv2d(p, x, ops.conv2d_prepack(p, filters[0]), biases[0]), gots[0])
            setattr(p, name, 0)
    assert ops.last_contraction().form == 8
    x64 = x[..., :ci].permute(0, 3, 1, 2).double()
    conv = lambda u, v: torch.nn.functional.conv2d(u, v, None, s, pd, d).permute(0, 2, 3, 1)
    for got, w, b in zip(gots, filters, biases):
        hi = (w.view(torch.int32) & ~0x1fff).view(torch.float32)
        held = hi.double() + ((w - hi).bfloat16().double() if mode == ops.MATH_TF32X3 else 0.0)
        other = b.double() + (res[..., :K].double() if output == "residual" else 0.0)
        want = (conv(x64, held) + other).clamp(min=0)
        # every partial sum rounded once: at most (terms) * 2^-24 of the sum of the terms' magnitudes
        bound = (k * k * ci + 8) * 2.0 ** -24 * (conv(x64.abs(), held.abs()) + b.abs().double() + (res[..., :K].abs().double() if output == "residual" else 0.0))
        n = w.shape[0]
        assert ((got[..., :n].double() - want).abs() <= bound).all()
        assert (got[..., n:ops.up4(n)] == 0).all()


@pytest.mark.parametrize("name,value", [("OGLE_TC_PAIR", "1"), ("OGLE_TC_PAIR", "0"), ("OGLE_TC_BN", "64"), ("OGLE_TC_BN", "192")])
def test_forced_forms_are_the_ones_that_run(name, value):
    """The switches for measurements are read once per process: convolutions, with and without a residual operand, and
    gemms of launches that would otherwise take clusters, pairs or another width."""
    import subprocess
    code = """
import os, torch
from ogle_b200 import ops
name, value = %r, %r
for N, H, C, K, k in ((1, 19, 512, 512, 1), (16, 38, 256, 512, 1), (4, 20, 64, 256, 3), (2, 30, 40, 192, 3)):
    for math in (ops.MATH_TF32X3, ops.MATH_TF32):
        p = ops.conv_params(N, H, H, C, K, k, 1, k // 2, 1, 1, True, 2, 0.0, 0.0, math)
        p.n_tile = 64 if name == "OGLE_TC_PAIR" else 0        # (pairs need a width that halves)
        packed = ops.conv2d_prepack(p, torch.randn((K, C, k, k), device="cuda"))
        x, b = torch.randn((N, H, H, C), device="cuda"), torch.randn(K, device="cuda")
        ops.conv2d(p, x, packed, b, workspace=None)
        seen = [ops.last_contraction()]
        if name == "OGLE_TC_BN":
            ops.conv2d_residual(p, x, packed, b, torch.randn((N, H, H, K), device="cuda"))
            seen.append(ops.last_contraction())
        if k == 1 and value != "1":
            a, w = x.reshape(-1, C), torch.randn((K, C), device="cuda")
            ops.gemm_packed(a, ops.gemm_pack_b(w, a.shape[0], C, K, 1, math), None, a.shape[0], C, K, 1, 1.0, 0.0, 0, math)
            seen.append(ops.last_contraction())
        for s in seen:
            if name == "OGLE_TC_BN":
                assert s.n_tile == int(value), (N, H, K, s.form, s.n_tile)
            elif value == "0":
                assert s.form != 4
            else:
                assert s.form == 4, (N, H, K, s.form, s.n_tile)
""" % (name, value)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, **{name: value}), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("shape", [
    # N, H, W, channels, K, stride: fewer tiles than stages, stages filled over and over, warps without a row, widths at which a
    # thread has five pixels and four, both ends of the channel counts that are known at compile time and are not
    (1, 9, 11, 3, 32, 2), (3, 3, 300, 3, 32, 1), (70, 90, 150, 3, 32, 2), (40, 64, 64, 4, 29, 1), (30, 64, 64, 3, 32, 2), (25, 112, 112, 3, 64, 2),
    (9, 75, 61, 4, 62, 1), (6, 40, 64, 1, 64, 1), (12, 90, 250, 3, 16, 1), (5, 60, 200, 2, 7, 1), (2, 1, 500, 3, 64, 1)])
def test_direct_stems_whose_warps_run_free(shape):
    import ctypes as C
    import torch
    from ogle_b200 import _lib, ops
    N, H, W, ch, K, s = shape
    g = torch.Generator(device="cuda").manual_seed(W + K)
    x = torch.zeros((N, H, W, 4), device="cuda")
    x[..., :ch] = torch.randn((N, H, W, ch), generator=g, device="cuda")
    w, b = torch.randn((K, ch, 3, 3), generator=g, device="cuda"), torch.randn(K, generator=g, device="cuda")

    def conv64(x, w, b):
        return torch.nn.functional.conv2d(x[..., :ch].permute(0, 3, 1, 2).double(), w.double(), b.double(), s, 1).permute(0, 2, 3, 1)

    want, size = conv64(x, w, b), conv64(x.abs(), w.abs(), b.abs())
    for act, clamp in ((ops.ACT_NONE, (None, None)), (ops.ACT_RELU, (0.0, None)), (ops.ACT_CLIP, (-1.0, 2.5))):
        p = ops.conv_params(N, H, W, ch, K, 3, s, 1, 1, 1, True, act, -1.0, 2.5, ops.MATH_FP32, 0, ops.up4(K) + 8, 4)
        assert _lib.cuda_lib().ogle_cuda_conv2d_kernel_name(C.byref(p)) == b"conv3x3_smallc_kernel"
        out = torch.full((N, want.shape[1], want.shape[2], ops.up4(K) + 8), -7.0, device="cuda")
        ops.conv2d(p, x, ops.conv2d_prepack(p, w), b, out, workspace=None)
        ref = want if act == ops.ACT_NONE else want.clamp(*clamp)
        # 9 * ch + 1 roundings of partial sums no larger than the sum of sizes
        assert bool(((out[..., 4:4 + K].double() - ref).abs() <= (9 * ch + 1) * 2.0 ** -24 * size).all())
        assert bool((out[..., :4] == -7.0).all()) and bool((out[..., 4 + ops.up4(K):] == -7.0).all())
        assert bool((out[..., 4 + K:4 + ops.up4(K)] == 0.0).all())
    assert _lib.cuda_lib().ogle_cuda_device_status() == 0


@pytest.mark.parametrize("shape", [
    # N, H, W, channels, K, kernel, stride, padding: tiles that hang over both edges, fewer and more than a round of blocks, channel
    # counts around a multiply's and a slab's width, paddings of either parity, tiles of a row
    (1, 32, 32, 3, 16, 7, 2, 3), (9, 113, 75, 3, 17, 7, 2, 2), (2, 64, 60, 4, 48, 7, 1, 3), (40, 70, 70, 3, 40, 5, 1, 2), (3, 64, 80, 1, 64, 5, 2, 0),
    (4, 61, 47, 2, 33, 5, 1, 1), (40, 120, 120, 3, 64, 7, 2, 3), (5, 47, 63, 1, 1, 7, 1, 0), (6, 90, 40, 4, 32, 5, 2, 1), (2, 77, 200, 2, 64, 7, 2, 3),
    (9, 1, 300, 3, 50, 5, 1, 2), (4, 3, 1024, 4, 64, 7, 1, 3)])
@pytest.mark.parametrize("math", ["MATH_TF32X3", "MATH_TF32"])
def test_stems_whose_window_is_the_operand(shape, math):
    """Against 64 bits, in a slice of a wider tensor, with a residual operand, beside an infinite pixel and with lanes behind
    the channels that are not numbers."""
    import torch
    from ogle_b200 import _lib, ops
    N, H, W, ch, K, k, s, pad = shape
    g = torch.Generator(device="cuda").manual_seed(W + K)
    x = torch.full((N, H, W, 4), float("nan"), device="cuda")
    x[..., :ch] = torch.randn((N, H, W, ch), generator=g, device="cuda")
    w, b = torch.randn((K, ch, k, k), generator=g, device="cuda") / (ch * k * k) ** 0.5, torch.randn(K, generator=g, device="cuda")
    p = ops.conv_params(N, H, W, ch, K, k, s, pad, 1, 1, True, ops.ACT_CLIP, -0.5, 1.5, getattr(ops, math), 0, ops.up4(K) + 8, 4)
    packed = ops.conv2d_prepack(p, w)
    want = torch.nn.functional.conv2d(x[..., :ch].permute(0, 3, 1, 2).double(), w.double(), b.double(), s, pad).permute(0, 2, 3, 1)
    # at most 196 products and sums of fp32 grade, or of operands with ten mantissa bits
    bound = (3e-6 if math == "MATH_TF32X3" else 1e-3) * float(want.norm())
    out = torch.full(want.shape[:3] + (ops.up4(K) + 8,), -7.0, device="cuda")
    ops.conv2d(p, x, packed, b, out, workspace=None)
    assert ops.last_contraction().form == 9
    assert float((out[..., 4:4 + K].double() - want.clamp(-0.5, 1.5)).norm()) <= bound
    assert bool((out[..., :4] == -7.0).all()) and bool((out[..., 4 + ops.up4(K):] == -7.0).all())
    assert bool((out[..., 4 + K:4 + ops.up4(K)] == 0.0).all())
    p = ops.conv_params(N, H, W, ch, K, k, s, pad, 1, 1, True, ops.ACT_NONE, 0.0, 0.0, getattr(ops, math))
    res = torch.randn(want.shape[:3] + (ops.up4(K),), generator=g, device="cuda")
    plain, got = ops.conv2d(p, x, packed, b, workspace=None), ops.conv2d_residual(p, x, packed, b, res)
    assert ops.last_contraction().form == 9
    assert torch.equal(got[..., :K], plain[..., :K] + res[..., :K]) and bool((got[..., K:] == 0.0).all())
    p.n_tile = 32
    assert torch.equal(ops.conv2d(p, x, packed, b, workspace=None), plain)
    p.n_tile = 0
    # an infinite pixel reaches the outputs whose windows hold it and no others
    y0, x0 = H // 2, W // 2
    x[0, y0, x0, 0] = float("inf")
    hit = torch.nn.functional.conv2d((x[:, :, :, 0] == float("inf")).double()[:, None], torch.ones((1, 1, k, k), device="cuda").double(), None, s, pad)[:, 0] > 0
    again = ops.conv2d(p, x, packed, b, workspace=None)
    assert torch.equal(again[~hit], plain[~hit])
    assert not bool(torch.isfinite(again[hit][:, :K]).any())
    assert _lib.cuda_lib().ogle_cuda_device_status() == 0


@pytest.mark.parametrize("case", [
    # C, K, kernel, stride, group, math, size
    (64, 64, 3, 1, 64, 2, 40), (50, 50, 5, 2, 50, 2, 40), (64, 64, 3, 1, 64, 2, 3), (64, 64, 7, 1, 64, 2, 40), (64, 32, 3, 1, 4, 2, 40),
    (3, 32, 3, 2, 1, 2, 40), (64, 64, 1, 1, 1, 0, 40), (64, 64, 1, 1, 1, 2, 40), (256, 256, 3, 1, 1, 0, 40)])
def test_kernel_names_are_those_of_the_sources(case):
    """What a profile is filtered by is the name of a kernel that exists."""
    import ctypes as C
    import glob
    import re
    from ogle_b200 import _lib, ops
    ci, k, f, s, g, math, size = case
    p = ops.conv_params(1, size, size, ci, k, f, s, f // 2, 1, g, True, 0, 0.0, 0.0, math)
    name = _lib.cuda_lib().ogle_cuda_conv2d_kernel_name(C.byref(p)).decode()
    root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ogle_b200", "csrc", "kernels")
    kernels = set()
    for path in glob.glob(os.path.join(root, "*.cu")):
        kernels |= set(re.findall(r"__global__[^;{]*?\b(\w+)\s*\(\s*(?:const|CUtensorMap|float)", open(path).read()))
    assert name in kernels


@pytest.mark.parametrize("case", [
    # images, size, C, K, kernel, stride, split asked for, name: both sides of what decides between the tensor-core path's kernels
    (1, 3, 256, 128, 1, 1, 0, "few_rows_kernel"), (1, 3, 256, 128, 1, 1, 2, "conv_tc2_kernel"), (32, 1, 64, 400, 1, 1, 0, "few_rows_kernel"),
    (33, 1, 64, 400, 1, 1, 0, "conv_tc2_kernel"), (32, 1, 64, 512, 1, 1, 0, "conv_tc2_kernel"), (24, 1, 64, 700, 1, 1, 0, "few_rows_kernel"),
    (32, 1, 33, 1366, 1, 1, 0, "conv_tc2_kernel"), (8, 1, 128, 2900, 1, 1, 0, "few_rows_kernel"), (6, 1, 164, 2342, 1, 1, 0, "conv_tc2_kernel"),
    (2, 1, 64, 3000, 1, 1, 0, "few_rows_kernel"), (2, 2, 128, 300, 3, 1, 0, "few_rows_kernel"), (2, 2, 128, 330, 3, 1, 0, "conv_tc2_kernel"),
    (2, 64, 3, 48, 7, 2, 0, "conv_window_kernel"), (2, 64, 3, 49, 7, 2, 0, "conv_tc2_kernel"), (2, 64, 2, 64, 7, 2, 0, "conv_window_kernel"),
    (2, 64, 3, 65, 5, 1, 0, "conv_tc2_kernel"), (80, 120, 3, 64, 7, 2, 0, "conv_window_kernel"),
    (3, 90, 1, 64, 7, 2, 0, "conv_tc2_kernel"), (3, 90, 1, 60, 7, 2, 0, "conv_window_kernel"), (3, 90, 1, 32, 5, 2, 0, "conv_window_kernel")])
@pytest.mark.parametrize("residual", [False, True])
def test_kernel_names_say_what_runs(case, residual):
    import ctypes as C
    import torch
    from ogle_b200 import _lib, ops
    N, size, ci, k, f, s, split, name = case
    p = ops.conv_params(N, size, size, ci, k, f, s, f // 2, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, ops.MATH_TF32X3)
    p.split = split
    assert _lib.cuda_lib().ogle_cuda_conv2d_kernel_name(C.byref(p)).decode() == name
    x, b = torch.zeros((N, size, size, ops.up4(ci)), device="cuda"), torch.ones(k, device="cuda")
    packed = ops.conv2d_prepack(p, torch.zeros((k, ci, f, f), device="cuda"))
    y = ops.conv2d(p, x, packed, b)
    if residual:
        ops.conv2d_residual(p, x, packed, b, torch.zeros_like(y))
    form = ops.last_contraction().form
    assert {8: "few_rows_kernel", 9: "conv_window_kernel"}.get(form, "conv_tc2_kernel") == name


@pytest.mark.parametrize("shape,name", [
    # N, H, W, C, K, kernel, stride: two blocks an SM and fewer, six, and others, on either side of the two forms' times
    ((3, 40, 28, 87, 220, 3, 1), "conv_igemm_kernel"), ((55, 24, 5, 49, 139, 5, 2), "conv_igemm_kernel"), ((1, 7, 14, 578, 55, 3, 1), "conv_igemm_kernel"),
    ((8, 38, 6, 53, 423, 3, 1), "conv_igemm_kernel"), ((8, 56, 56, 64, 64, 3, 1), "conv_igemm_tma_kernel"), ((8, 28, 28, 128, 256, 3, 2), "conv_igemm_tma_kernel"),
    ((5, 63, 25, 315, 92, 3, 1), "conv_igemm_tma_kernel"), ((1, 7, 10, 698, 304, 3, 2), "conv_igemm_tma_kernel"), ((8, 7, 7, 512, 512, 3, 1), "conv_igemm_tma_kernel"), ((32, 38, 38, 256, 256, 3, 1), "conv_igemm_tma_kernel")])
def test_fp32_contraction_takes_the_faster_form(shape, name):
    import ctypes as C
    from ogle_b200 import _lib, ops
    N, H, W, ci, K, k, s = shape
    p = ops.conv_params(N, H, W, ci, K, k, s, k // 2, 1, 1, True, ops.ACT_RELU, 0.0, 0.0, ops.MATH_FP32)
    assert _lib.cuda_lib().ogle_cuda_conv2d_kernel_name(C.byref(p)).decode() == name


@pytest.mark.parametrize("env,overlapped", [(None, 1), ("0", 0), ("1", 1)])
def test_products_overlap_their_packing_pass_unless_told_otherwise(env, overlapped):
    """gemm_ws in all its forms - clusters, pairs of SMs, whole tiles - asks for it; OGLE_PDL, read once per process, wins."""
    import subprocess
    code = """
import torch
from ogle_b200 import ops
forms = set()
for m, k, n in ((64, 512, 300), (25600, 512, 1024), (20000, 64, 100)):
    a, b = torch.randn((m, k), device="cuda"), torch.randn((k, n), device="cuda")
    ops.gemm_ws(a, b, None, m, k, n, 0, 1.0, 0.0, 0, ops.MATH_TF32X3)
    last = ops.last_contraction()
    forms.add(last.form)
    assert last.overlapped == %d, (m, last.form, last.overlapped)
assert forms == {1, 3, 4}, forms
""" % overlapped
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    clean = {k: v for k, v in os.environ.items() if k != "OGLE_PDL"}
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(clean, **({"OGLE_PDL": env} if env else {})), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
