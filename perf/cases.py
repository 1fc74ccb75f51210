"""Performance cases of the framework: what its users have it compute, through its public entry points.

A case is a dict of plain values. `listed()` gives the named ones, `draw(rng)` one more of the same ranges,
`prepare(case, seed)` what a program holds before the call (model loaded, session sized and warm, filters packed,
inputs in place), `run(state)` one pass with its outputs, `work(case)` the bytes and operations a pass cannot do
without and `tolerance(case)` how far two correct implementations may differ.

Kinds, by what they stand for:
  detect       SSD detector on 8-bit BGR frames in host memory (session.Detector): upload, resize and mean subtraction,
               network, box decode, score selection and overlap removal, detections back on the host
  ssd_host     the same network called on fp32 tensors in host memory (FBOSession.Run + GetOutputs)
  ssd, resnet  the two networks on inputs that are already on the GPU (FBOSession.RunDevice), outputs left there
  conv         one convolution layer called as an operator: dense, strided, pointwise or depthwise
  pool_concat  max and average pooling of one feature map, concatenated, batch-normalised and rectified
  gemm         matrix product of two run-time operands (B is packed on every call)
  dense        matrix product against a constant, packed B: a classifier's last layer
  postprocess  box decode and detection selection on a batch of network outputs
"""
import math
import os
import tempfile

import numpy as np
import torch

from ogle_b200 import models, ops, session

MATH = {"fp32": ops.MATH_FP32, "tf32": ops.MATH_TF32, "tf32x3": ops.MATH_TF32X3}
ACT = {"none": ops.ACT_NONE, "relu": ops.ACT_RELU, "clip": ops.ACT_CLIP}
ANCHORS = 1917            # of the 300 x 300 SSD heads
MEAN_RGB = (123.0, 117.0, 104.0)
BACKGROUND_BIAS = 6.0     # of the class heads: a trained detector calls nearly every anchor background


def listed():
    return [
        # one camera frame at a time: the smallest unit of work of a live detector, where latency counts
        dict(name="camera_frame", kind="detect", batch=1, height=480, width=640, classes=2, packed=False),
        # frames of the network's own size collected in one pinned buffer: a small serving batch
        dict(name="frame_batch_8", kind="detect", batch=8, height=300, width=300, classes=21, packed=True),
        # a program that keeps its tensors on the host and wants the raw head outputs back
        dict(name="host_tensors_4", kind="ssd_host", batch=4, classes=21, math="tf32x3"),
        # the benchmark's network at the benchmark's batch: offline throughput
        dict(name="ssd_resident_256", kind="ssd", batch=256, classes=21, math="tf32x3"),
        # the classifier at the benchmark's batch
        dict(name="resnet_resident_128", kind="resnet", batch=128, math="tf32x3"),
        # full fp32 arithmetic: reference results, accuracy checks
        dict(name="resnet_fp32_8", kind="resnet", batch=8, math="fp32"),
        # an operator call on sizes no tile divides, in the one-pass mode
        dict(name="conv3x3_ragged_tf32", kind="conv", batch=5, height=47, width=61, channels=150, filters=250, kernel=3,
             stride=1, depthwise=False, act="relu", math="tf32"),
        # a depthwise layer whose width is no multiple of a 32-channel slab
        dict(name="depthwise_144", kind="conv", batch=16, height=75, width=75, channels=144, filters=144, kernel=3, stride=1,
             depthwise=True, act="relu", math="tf32x3"),
        # the bandwidth-bound operators between convolutions
        dict(name="pool_concat_192", kind="pool_concat", batch=32, height=76, width=76, channels=192),
        # a product of two activations, no size a multiple of a tile
        dict(name="gemm_runtime_b", kind="gemm", m=1000, k=1500, n=700, trans_b=False, bias=True, math="tf32x3"),
        # the classifier head of one image: the smallest call there is, launch and host work only
        dict(name="dense_single", kind="dense", m=1, k=512, n=1000, bias=True, math="tf32x3"),
        # the standalone decoder configuration: 1024 images, 21 classes, top 200 of each
        dict(name="postprocess_1024", kind="postprocess", batch=1024, anchors=ANCHORS, classes=21, per_class=True, top_k=200),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["detect", "ssd_host", "ssd", "resnet", "conv", "depthwise", "pool_concat", "gemm", "dense", "postprocess"])
    if kind == "detect":
        packed = rng.random() < 0.5
        return dict(kind=kind, batch=_log_int(rng, 1, 8), height=300 if packed else rng.randint(120, 1080),
                    width=300 if packed else rng.randint(160, 1920), classes=rng.choice([2, 21]), packed=packed)
    if kind == "ssd_host":
        return dict(kind=kind, batch=_log_int(rng, 1, 16), classes=rng.randint(2, 30), math=rng.choice(["tf32x3", "tf32"]))
    if kind in ("ssd", "resnet"):
        arithmetic = rng.choice(["tf32x3", "tf32x3", "tf32", "fp32"])
        most = 16 if arithmetic == "fp32" else (256 if kind == "ssd" else 128)
        case = dict(kind=kind, batch=_log_int(rng, 1, most), math=arithmetic)
        if kind == "ssd":
            case["classes"] = rng.randint(2, 30)
        return case
    if kind == "conv":
        while True:
            case = dict(kind="conv", batch=_log_int(rng, 1, 64), height=_log_int(rng, 5, 150), width=_log_int(rng, 5, 150),
                        channels=_log_int(rng, 3, 1024), filters=_log_int(rng, 8, 1024), kernel=rng.choice([1, 1, 3, 3, 5]),
                        stride=rng.choice([1, 1, 2]), depthwise=False, act=rng.choice(["none", "relu", "clip"]),
                        math=rng.choice(["tf32x3", "tf32", "fp32"]))
            w = work(case)
            # few input channels are computed without the matrix unit, as fp32 layers are
            if w["bytes"] < 2e9 and w["flops"] < (3e10 if case["math"] == "fp32" or case["channels"] < 16 else 3e11):
                return case
    if kind == "depthwise":
        while True:
            c = _log_int(rng, 8, 1024)
            c = c if rng.random() < 0.5 else max(32, c // 32 * 32)
            case = dict(kind="conv", batch=_log_int(rng, 1, 64), height=_log_int(rng, 7, 150), width=_log_int(rng, 7, 150), channels=c,
                        filters=c, kernel=rng.choice([3, 3, 3, 5]), stride=rng.choice([1, 2]), depthwise=True,
                        act=rng.choice(["none", "relu", "clip"]), math="tf32x3")
            if work(case)["bytes"] < 4e9:
                return case
    if kind == "pool_concat":
        while True:
            case = dict(kind=kind, batch=_log_int(rng, 1, 64), height=_log_int(rng, 8, 150), width=_log_int(rng, 8, 150),
                        channels=_log_int(rng, 8, 512))
            if work(case)["bytes"] < 4e9:
                return case
    if kind in ("gemm", "dense"):
        m = _log_int(rng, 1, 256) if kind == "dense" else _log_int(rng, 64, 4096)
        return dict(kind=kind, m=m, k=_log_int(rng, 64, 4096), n=_log_int(rng, 10, 4096), bias=rng.random() < 0.7,
                    math=rng.choice(["tf32x3", "tf32"]), **({"trans_b": rng.random() < 0.5} if kind == "gemm" else {}))
    while True:
        case = dict(kind=kind, batch=_log_int(rng, 1, 1024), anchors=rng.choice([ANCHORS, rng.randint(300, 4000)]),
                    classes=rng.randint(2, 30), per_class=rng.random() < 0.5, top_k=_log_int(rng, 10, 200))
        if case["batch"] * case["anchors"] * case["classes"] <= 1024 * ANCHORS * 21:
            return case


# ------------------------------------------------------------------------------------------------ models
_files = {}
_folder = None


def _model(kind, batch, classes, frames=False):
    """(path of a saved model, its info): built once per process, as a deployed model is a file on disk."""
    global _folder
    key = (kind, batch, classes, frames)
    if key not in _files:
        if _folder is None:
            _folder = tempfile.TemporaryDirectory(prefix="ogle_perf_")
        if kind == "resnet":
            model, info = models.resnet18(batch=batch, seed=0, weight_std="he")
        else:
            model, info = models.mobilenet_v1_ssd(batch=batch, num_classes=classes, seed=0, weight_std="he")
        consts = [(n.name, n.attr["const_attr"]["value"]) for n in model.nodes if n.type == "Const"]
        if frames:
            # weights as training leaves them: the stem scales 8-bit pixels down, the class heads favour background
            consts[0][1].float_data = np.asarray(consts[0][1].float_data, np.float32) / np.float32(64.0)
            for _, bias in [c for c in consts if c[0].endswith(".bias")][1::2]:
                b = np.array(bias.float_data, np.float32).reshape(-1, classes)
                b[:, 0] += BACKGROUND_BIAS
                bias.float_data = b.reshape(-1)
        info["weight_bytes"] = 4 * sum(int(np.prod(c.dims)) for name, c in consts if name.endswith((".weight", ".bias", ":2")))
        path = os.path.join(_folder.name, "%s_%d_%d_%d.dlx" % key)
        model.save(path)
        _files[key] = (path, info)
    return _files[key]


class _DeviceTensor:
    """A session's tensor, by its device address, for torch.as_tensor; keeps the session, which owns the memory."""

    def __init__(self, sess, shape, pointer):
        self.session = sess
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f4", data=(pointer, False), version=2)


def _device_output(sess, name):
    shape, _, pointer = sess.tensor_info(name)
    return torch.as_tensor(_DeviceTensor(sess, shape[:-1] + [ops.up4(shape[-1])], pointer), device="cuda")


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, std=1.0):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std


def _padded_randn(g, *shape):
    """N(0,1) in the padded device layout: lanes past the last dimension are zero."""
    x = torch.zeros(shape[:-1] + (ops.up4(shape[-1]),), device="cuda", dtype=torch.float32)
    x[..., :shape[-1]] = _randn(g, *shape)
    return x


def _frames(seed, n, h, w):
    """n 8-bit BGR pictures: smooth structure at the scale of objects plus sensor noise."""
    g = _generator(seed)
    low = torch.rand((n, 3, h // 40 + 2, w // 40 + 2), generator=g, device="cuda") * 255.0
    x = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear", align_corners=False)
    x = x + torch.randn(x.shape, generator=g, device="cuda") * 4.0
    return x.clamp(0, 255).to(torch.uint8).permute(0, 2, 3, 1).contiguous().cpu().numpy()


# --------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_detect(case, seed):
    n, h, w = case["batch"], case["height"], case["width"]
    path, _ = _model("ssd", n, case["classes"], frames=True)
    det = session.Detector(path, mode=0, score_thr=0.3, top_k=100, nms_thr=0.45)
    pixels = _frames(seed, n, h, w)
    if case["packed"]:
        buffer = session.PinnedArray((n, h, w, 3), np.uint8)
        buffer.array[...] = pixels
        state = dict(run=_run_detect_packed, det=det, buffer=buffer, n=n, h=h, w=w)
    else:
        state = dict(run=_run_detect_frames, det=det, frames=[np.ascontiguousarray(f) for f in pixels])
    for _ in range(3):            # sized, captured and replayed once: as a detector that has been running
        run(state)
    return state


def _run_detect_packed(s):
    s["det"].detect_bgr8_frames_async(s["buffer"].ptr, s["n"], s["h"], s["w"], 300, 300, MEAN_RGB)
    return s["det"].wait()


def _run_detect_frames(s):
    s["det"].detect_bgr8_async(s["frames"], 300, 300, MEAN_RGB)
    return s["det"].wait()


_stream = None


def _session(path, case):
    """A session on the program's one compute stream: passes run one after the other."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    sess = session.FBOSession(stream=_stream.cuda_stream)
    sess.set_option("math_mode", MATH[case["math"]])
    sess.LoadGraph(path)
    return sess


def _images(seed, n, size):
    """[n, size, size, 3] in [-1, 1]: uniform pixels, normalised"""
    return torch.rand((n, size, size, 3), generator=_generator(seed), device="cuda") * 2.0 - 1.0


def _prepare_ssd_host(case, seed):
    path, _ = _model("ssd", case["batch"], case["classes"])
    state = dict(run=_run_ssd_host, sess=_session(path, case), x=_images(seed, case["batch"], 300).cpu().numpy())
    for _ in range(3):
        run(state)
    return state


def _run_ssd_host(s):
    s["sess"].Run({"input": s["x"]})
    return s["sess"].GetOutputs(["box_preds", "cls_logits"], ["ANY", "ANY"])


def _prepare_resident(case, seed, path, size, outputs):
    n = case["batch"]
    sess = _session(path, case)
    sess.Run({"input": np.zeros((n, size, size, 3), np.float32)})        # sizes the session
    x = torch.zeros((n, size, size, 4), device="cuda")
    x[..., :3] = _images(seed, n, size)
    torch.cuda.synchronize()
    state = dict(run=_run_resident, sess=sess, x=x, inputs={"input": x.data_ptr()}, outputs=[_device_output(sess, o) for o in outputs])
    for _ in range(2):
        run(state)
    sess.synchronize()
    return state


def _prepare_ssd(case, seed):
    return _prepare_resident(case, seed, _model("ssd", case["batch"], case["classes"])[0], 300, ("box_preds", "cls_logits"))


def _prepare_resnet(case, seed):
    return _prepare_resident(case, seed, _model("resnet", case["batch"], 1000)[0], 224, ("logits",))


def _run_resident(s):
    s["sess"].RunDevice(s["inputs"])
    return s["outputs"]


def _prepare_conv(case, seed):
    g = _generator(seed)
    c, k, f = case["channels"], case["filters"], case["kernel"]
    group = c if case["depthwise"] else 1
    p = ops.conv_params(case["batch"], case["height"], case["width"], c, k, f, case["stride"], f // 2, 1, group, True,
                        ACT[case["act"]], 0.0, 6.0, MATH[case["math"]])
    packed = ops.conv2d_prepack(p, _randn(g, k, c // group, f, f, std=math.sqrt(2.0 / (c // group * f * f))))
    return dict(run=_run_conv, p=p, packed=packed, x=_padded_randn(g, case["batch"], case["height"], case["width"], c), bias=_randn(g, k, std=0.1))


def _run_conv(s):
    return ops.conv2d(s["p"], s["x"], s["packed"], s["bias"])


def _prepare_pool_concat(case, seed):
    g = _generator(seed)
    n, h, w, c = case["batch"], case["height"], case["width"], case["channels"]
    largest = ops.pool_params(n, h, w, c, 3, 2, 1, 0)
    average = ops.pool_params(n, h, w, c, 3, 2, 1, 1)
    shape = [n] + list(largest.out_hwc)
    stats = [torch.rand(2 * c, generator=g, device="cuda") + 0.5 for _ in range(4)]      # gamma, beta, mean, var
    return dict(run=_run_pool_concat, x=_padded_randn(g, n, h, w, c), largest=largest, average=average, shapes=[shape, shape],
                stats=stats, channels=2 * c)


def _run_pool_concat(s):
    both, _ = ops.concat([ops.pool(s["largest"], s["x"]), ops.pool(s["average"], s["x"])], s["shapes"], 3)
    return ops.relu(ops.batchnorm(both, *s["stats"], s["channels"], 1e-5))


def _prepare_gemm(case, seed):
    g = _generator(seed)
    m, k, n = case["m"], case["k"], case["n"]
    b = _padded_randn(g, n, k) if case["trans_b"] else _padded_randn(g, k, n)
    mode = MATH[case["math"]]
    # scratch for the packed B, in the size the library asks for
    workspace = torch.empty_like(ops.gemm_pack_b(b, m, k, n, int(case["trans_b"]), mode))
    return dict(run=_run_gemm, a=_padded_randn(g, m, k), b=b, c=_padded_randn(g, n) if case["bias"] else None,
                sizes=(m, k, n, int(case["trans_b"]), 1.0, 1.0, 2 if case["bias"] else 0, mode), workspace=workspace)


def _run_gemm(s):
    return ops.gemm_ws(s["a"], s["b"], s["c"], *s["sizes"], workspace=s["workspace"])


def _prepare_dense(case, seed):
    g = _generator(seed)
    m, k, n = case["m"], case["k"], case["n"]
    mode = MATH[case["math"]]
    packed = ops.gemm_pack_b(_padded_randn(g, n, k), m, k, n, 1, mode)
    return dict(run=_run_dense, a=_padded_randn(g, m, k), packed=packed, c=_padded_randn(g, n) if case["bias"] else None,
                sizes=(m, k, n, 1, 1.0, 1.0, 2 if case["bias"] else 0, mode))


def _run_dense(s):
    return ops.gemm_packed(s["a"], s["packed"], s["c"], *s["sizes"])


def _prepare_postprocess(case, seed):
    g = _generator(seed)
    n, a, c = case["batch"], case["anchors"], case["classes"]
    if a == ANCHORS:
        priors = torch.from_numpy(models.ssd_prior_boxes()).cuda()
    else:
        priors = torch.cat([torch.rand((a, 2), generator=g, device="cuda"), torch.rand((a, 2), generator=g, device="cuda") * 0.4 + 0.05], 1)
    logits = torch.zeros((n, a, ops.up4(c)), device="cuda")
    logits[..., :c] = _randn(g, n, a, c, std=2.0)
    return dict(run=_run_postprocess, deltas=_randn(g, n, a, 4, std=0.5), priors=priors.contiguous(), logits=logits, classes=c,
                mode=int(case["per_class"]), threshold=0.01 if case["per_class"] else 0.3, top_k=case["top_k"])


def _run_postprocess(s):
    boxes = ops.ssd_decode(s["deltas"], s["priors"])
    return ops.ssd_detect(s["logits"], boxes, s["classes"], s["mode"], s["threshold"], s["top_k"], 0.45, 300, 300)


# ------------------------------------------------------------------------------------- work and tolerance
def work(case):
    kind = case["kind"]
    if kind in ("detect", "ssd_host", "ssd", "resnet"):
        n = case["batch"]
        _, info = _model("resnet" if kind == "resnet" else "ssd", n, 1000 if kind == "resnet" else case["classes"], kind == "detect")
        flops = float(info["flops_per_image"]) * n
        if kind == "detect":
            moved = n * (case["height"] * case["width"] * 3 + 100 * 28 + 4)
        elif kind == "resnet":
            moved = n * 4 * (224 * 224 * 3 + 1000)
        else:
            moved = n * 4 * (300 * 300 * 3 + ANCHORS * (4 + case["classes"]))
        return {"bytes": moved + info["weight_bytes"], "flops": flops}
    if kind == "conv":
        n, h, w, c, k, f, s = (case[q] for q in ("batch", "height", "width", "channels", "filters", "kernel", "stride"))
        ho, wo = (h - 1) // s + 1, (w - 1) // s + 1            # padding f // 2
        per = 1 if case["depthwise"] else c
        return {"bytes": 4.0 * (n * h * w * c + n * ho * wo * k + k * per * f * f + k), "flops": 2.0 * n * ho * wo * k * per * f * f}
    if kind == "pool_concat":
        n, h, w, c = case["batch"], case["height"], case["width"], case["channels"]
        out = n * ((h - 1) // 2 + 1) * ((w - 1) // 2 + 1) * c
        return {"bytes": 4.0 * (n * h * w * c + 2 * out + 8 * c), "flops": 2 * 9.0 * out + 2 * 6.0 * out}
    if kind in ("gemm", "dense"):
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4.0 * (m * k + k * n + m * n + (n if case["bias"] else 0)), "flops": 2.0 * m * k * n}
    n, a, c = case["batch"], case["anchors"], case["classes"]
    rows = (c - 1) * case["top_k"] if case["per_class"] else case["top_k"]
    return {"bytes": 4.0 * (n * a * (c + 4) + a * 4 + n * a * 4) + 28.0 * n * rows, "flops": 3.0 * n * a * c + 20.0 * n * a}


def tolerance(case):
    kind = case["kind"]
    if kind == "detect":
        # boxes are whole pixels: an edge that lies on a pixel's border may fall to either side
        return {"rel": 5e-3, "max": 0.1, "differ": 5e-3}
    if kind == "postprocess":
        # scores are fp32 quotients; where two are within an ulp of one another their rows may change places
        return {"rel": 1e-3, "max": 0.99, "differ": 1e-3}
    if kind == "pool_concat":
        return {"rel": 1e-6}
    network = kind in ("ssd_host", "ssd", "resnet")
    if case["math"] == "tf32":
        # operands carry ten mantissa bits
        return {"rel": 1e-2 if network else 2e-3}
    # fp32 products and sums in another order; a network adds up the rounding of some thirty layers
    return {"rel": 1e-4 if network else 1e-5}
