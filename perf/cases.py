"""Performance cases of the detector-inference path, through the entry points a program calls: `GpuExecutableNetwork`
(detect_device / detect / detect_u8 / submit_u8 + collect / forward), the operator methods of `B200Backend`, and
`B200Backend.yolo_decode_nms`.

A case is a dict of plain values with one of five kinds:

  detect  one call on one batch, detections out.  feed = device (the batch is resident in HBM), host (a NumPy f32 batch) or u8
          (a list of camera images, letterboxed on the device)
  stream  a run of batches of camera images through submit_u8 / collect, two batches in flight (a serving or validation loop)
  heads   forward of a host batch and download of the raw head tensors: what the runtime does that decodes on its own side, in
          the two precisions that keep floating activations (f32, f16)
  nms     decode + per-class NMS of head tensors alone
  ops     a detector tail driven operator by operator, as a runtime over the tensor traits drives it: strided convolution,
          3x3 / 1x1 pairs, shortcuts, head convolution, decode + NMS

Every model is a fixed one (weights are drawn once, as a .weights file would be read once); the seed draws the images.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import lightnet_b200 as ln
from lightnet_b200 import synth, zoo

CFG = {"yolov3-tiny": zoo.yolov3_tiny_cfg, "yolov4": zoo.yolov4_cfg, "yolov7": zoo.yolov7_cfg}
# convolution operations (2 per multiply-add) per input pixel, convolution weights, head channels x cells per input pixel
MODEL = {"yolov3-tiny": (32157.0, 8845488, 255 * (1 / 1024 + 1 / 256)), "yolov4": (347314.0, 64296032, 255 * (1 / 1024 + 1 / 256 + 1 / 64)),
         "yolov7": (255154.0, 36881504, 255 * (1 / 1024 + 1 / 256 + 1 / 64))}
PRECISION = {"f32": ln.LN_F32, "f16": ln.LN_F16, "int8": ln.LN_Q8, "fp8": ln.LN_F8}
QMAX = {"int8": 127.0, "fp8": 448.0}
MOST_FLOPS = 64 * 608 * 608 * MODEL["yolov4"][0]  # the largest listed case
CONF, IOU = 0.25, 0.45                            # detector defaults


def listed():
    return [
        # one webcam frame through the small detector: launches and host work are everything
        dict(name="tiny_u8_frame", kind="detect", feed="u8", model="yolov3-tiny", width=416, height=416, batch=1, precision="int8", frames="640x480"),
        # the f32 operator path at the reference's default size
        dict(name="tiny_f32_heads", kind="heads", model="yolov3-tiny", width=416, height=416, batch=1, precision="f32"),
        # the same path on the large detector: what a calibration run and a parity check pay per image
        dict(name="v4_f32_heads", kind="heads", model="yolov4", width=608, height=608, batch=1, precision="f32"),
        # binary16 storage, a few images of a wide stream
        dict(name="v4_f16_heads_b3", kind="heads", model="yolov4", width=480, height=288, batch=3, precision="f16"),
        # one image, latency-bound serving
        dict(name="v4_int8_b1", kind="detect", feed="device", model="yolov4", width=608, height=608, batch=1, precision="int8"),
        # the benchmark's batch: throughput
        dict(name="v4_int8_b64", kind="detect", feed="device", model="yolov4", width=608, height=608, batch=64, precision="int8"),
        # the FP8 benchmark's batch
        dict(name="v7_fp8_b32", kind="detect", feed="device", model="yolov7", width=640, height=640, batch=32, precision="fp8"),
        # a small, uneven batch of camera images of several sizes in a network that is not square
        dict(name="v7_fp8_u8_b5", kind="detect", feed="u8", model="yolov7", width=480, height=352, batch=5, precision="fp8",
             frames="640x480,500x375,333x500,1280x720"),
        # four batches streamed from page-locked pixels
        dict(name="v4_int8_stream", kind="stream", model="yolov4", width=608, height=608, batch=16, batches=4, precision="int8", frames="640x480"),
        # the decode + NMS stress of the benchmark: threshold 0.001, top-k 300
        dict(name="nms_stress_b256", kind="nms", batch=256, grid_w=20, grid_h=20, heads=3, classes=80, new_coords=0, conf=0.001, iou=0.65, top_k=300),
        # two heads of one wide image at the detector's default threshold, few classes
        dict(name="nms_b1", kind="nms", batch=1, grid_w=15, grid_h=9, heads=2, classes=20, new_coords=0, conf=CONF, iou=IOU, top_k=0),
        # the shapes of the single-layer sweep (3x3 s2 C128->K256, 3x3 C256->K512, 1x1 C512->K256) as operator calls
        dict(name="ops_int8_b16", kind="ops", batch=16, channels=128, grid_w=52, grid_h=52, blocks=2, shortcut=0, precision="int8", activation="leaky"),
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], even over its logarithm."""
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def _net_size(rng, model):
    lo = 3 if model == "yolov3-tiny" else 8
    return 32 * _spread(rng, lo, 20), 32 * _spread(rng, lo, 20)


def _frames(rng):
    return ",".join("%dx%d" % (_spread(rng, 160, 1920), _spread(rng, 120, 1080)) for _ in range(rng.randint(1, 4)))


def draw(rng):
    kind = rng.choice(["detect", "detect", "detect", "stream", "heads", "nms", "nms", "ops"])
    if kind == "nms":
        heads, classes = rng.choice([2, 3]), rng.choice([1, 2, 20, 80])
        gw, gh = rng.randint(6, 20), rng.randint(6, 20)
        floats = gw * gh * 3 * (5 + classes) * sum(4 ** k for k in range(heads))
        return dict(kind="nms", batch=_spread(rng, 1, max(1, min(256, 256 * 25200 * 85 // floats))), grid_w=gw, grid_h=gh, heads=heads, classes=classes,
                    new_coords=rng.choice([0, 0, 1]), conf=rng.choice([0.001, 0.05, CONF]), iou=rng.choice([IOU, 0.65]), top_k=rng.choice([0, 100, 300]))
    if kind == "ops":
        return dict(kind="ops", batch=_spread(rng, 1, 32), channels=32 * rng.randint(1, 8), grid_w=rng.randint(13, 60), grid_h=rng.randint(13, 60),
                    blocks=rng.randint(1, 4), shortcut=rng.randint(0, 1), precision=rng.choice(["int8", "fp8"]),
                    activation=rng.choice(["leaky", "mish", "swish"]))
    model = rng.choice(["yolov3-tiny", "yolov4", "yolov7"])
    w, h = _net_size(rng, model)
    flops = w * h * MODEL[model][0]
    if kind == "heads":
        precision = rng.choice(["f32", "f16"])
        most = (608 * 608 if precision == "f32" else 4 * 608 * 608) * MODEL["yolov4"][0]  # one and four images of the large detector
        while flops > most:
            w, h = _net_size(rng, model)
            flops = w * h * MODEL[model][0]
        return dict(kind="heads", model=model, width=w, height=h, batch=_spread(rng, 1, max(1, min(16, int(most // flops)))), precision=precision)
    precision = rng.choice(["int8", "int8", "fp8"])
    most = max(1, int(MOST_FLOPS // flops))
    if kind == "stream":
        batches = rng.randint(2, 4)
        return dict(kind="stream", model=model, width=w, height=h, batch=_spread(rng, 1, min(64 // batches, most // batches)), batches=batches,
                    precision=precision, frames=_frames(rng))
    feed = rng.choice(["device", "host", "u8"])
    case = dict(kind="detect", feed=feed, model=model, width=w, height=h, batch=_spread(rng, 1, min(64, most) if feed == "device" else min(16, most)),
                precision=precision)
    if feed == "u8":
        case["frames"] = _frames(rng)
    return case


# ---- what a program has in hand before the call ------------------------------------------------------------------------------


class _Session:
    """The one backend of the process and the network it currently serves."""

    backend = None
    key = None
    net = None

    @classmethod
    def get(cls):
        if cls.backend is None:
            cls.backend = ln.B200Backend(0)
        return cls.backend

    @classmethod
    def network(cls, case):
        key = tuple(case[k] for k in ("model", "width", "height", "batch", "precision"))
        if cls.key != key:
            cls.net = cls.key = None  # the network before is given back first
            cls.net, cls.key = _build_network(cls.get(), *key), key
        return cls.net


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _gain(activation):
    """Variance of the weights times the fan-in that keeps the variance of the pre-activations from layer to layer (He's 2 but
    for swish, whose second moment is 0.355 of its input's)."""
    return 2.8 if activation == ln.ACTIVATIONS["swish"] else 2.0


def _weights(layers, seed):
    """Darknet payload, as synth.he_weights lays it out (He-normal weights, identity batch norm), drawn on the GPU."""
    g = _generator(seed)
    parts, at, where = [], 0, {}
    for i, l in enumerate(layers):
        if l["kind"] != "conv":
            continue
        f, n = l["filters"], l["filters"] * l["in_c"] * l["size"] ** 2
        zero, one = torch.zeros(f, device="cuda"), torch.ones(f, device="cuda")
        parts += [zero, one, zero, one] if l["bn"] else [zero]
        parts.append(torch.randn(n, generator=g, device="cuda") * math.sqrt(_gain(l["act"]) / (n / f)))
        where[i] = (at, at + (4 if l["bn"] else 1) * f, n)  # biases (no batch norm: directly in front of the weights), weights, count
        at += (4 if l["bn"] else 1) * f + n
    return torch.cat(parts).cpu().numpy(), where


def _images(n, w, h, g):
    """f32 [n, 3, h, w] in [0, 1): smooth shapes with some noise on top, on the GPU."""
    low = torch.rand((n, 3, max(2, h // 24), max(2, w // 24)), generator=g, device="cuda")
    x = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear", align_corners=True)
    return 0.9 * x + 0.0999 * torch.rand(x.shape, generator=g, device="cuda")


def _frames_u8(case, n, g):
    """n camera images [h, w, 3] of 8 bits, the sizes of the case in turn."""
    sizes = [tuple(int(v) for v in s.split("x")) for s in case["frames"].split(",")]
    return [(_images(1, w, h, g)[0].permute(1, 2, 0) * 256).to(torch.uint8).contiguous().cpu().numpy() for w, h in (sizes[i % len(sizes)] for i in range(n))]


def _head_targets(channels, classes, class_logit=-4.0):
    """Mean and deviation of each head channel of a trained-looking detector: those of the decode + NMS stress inputs, with
    another mean of the class logits where the workload has another number of candidates.  (One or two classes: the objectness
    decides.)"""
    mean, std = np.full(channels, class_logit if classes > 2 else 1.0, np.float32), np.full(channels, 2.0, np.float32)
    for a in range(0, channels, 5 + classes):
        mean[a:a + 4], mean[a + 4] = 0.0, -4.0
        std[a:a + 2], std[a + 2:a + 4] = 1.0, 0.5
    return mean, std


def _build_network(be, model, width, height, batch, precision):
    prec = PRECISION[precision]
    if precision in ("f32", "f16"):
        net = ln.GpuExecutableNetwork(be, CFG[model](width, height), batch, prec)
        net.load_weights(_weights(net.layers(), 11)[0])
        return net
    # 8 bits: calibrate the scales on four images, then give the head convolutions the statistics of a trained detector on
    # them (random heads would pass a quarter of all candidates with a score of exactly 1)
    probe = ln.GpuExecutableNetwork(be, CFG[model](width, height).replace("activation=logistic", "activation=linear"), 4, prec)
    layers = probe.layers()
    blob, where = _weights(layers, 11)
    images = _images(4, width, height, _generator(12)).cpu().numpy()
    probe.load_weights(blob)
    probe.calibrate(images)
    probe.forward(images)
    convs = [i for i in range(len(layers) - 1) if layers[i]["kind"] == "conv" and layers[i + 1]["kind"] == "yolo"]
    for k, i in enumerate(convs):
        head = be.download_f32(probe.head(k)).transpose(1, 0, 2, 3).reshape(layers[i]["filters"], -1)
        mean, std = _head_targets(len(head), 80, -5.5)
        gain = std / np.maximum(head.std(1), 1e-3 * np.abs(head).max() + 1e-20)
        b0, w0, n = where[i]
        blob[w0:w0 + n] *= np.repeat(gain, n // len(head))
        blob[b0:b0 + len(head)] = mean - gain * head.mean(1)
    scales = probe.scales()
    del probe
    net = ln.GpuExecutableNetwork(be, CFG[model](width, height), batch, prec)
    net.load_weights(blob)
    net.set_scales(scales)
    return net


def _prepare_detect(case, seed):
    be, net, g = _Session.get(), _Session.network(case), _generator(seed)
    b, w, h = case["batch"], case["width"], case["height"]
    if case["feed"] == "u8":
        return dict(case=case, net=net, images=_frames_u8(case, b, g))
    x = _images(b, w, h, g).cpu().numpy()
    if case["feed"] == "device":
        x = be.upload_f32(x.shape, x)
    return dict(case=case, net=net, x=x, size=(np.full(b, w, np.int32), np.full(b, h, np.int32)))


def _prepare_stream(case, seed):
    net, g = _Session.network(case), _generator(seed)
    packs = []
    for _ in range(case["batches"]):
        flat, offsets, widths, heights = ln.pack_u8_images(_frames_u8(case, case["batch"], g))
        packs.append((torch.from_numpy(flat).pin_memory().numpy(), offsets, widths, heights))
    return dict(case=case, net=net, packs=packs)


def _prepare_heads(case, seed):
    net = _Session.network(case)
    return dict(case=case, net=net, x=_images(case["batch"], case["width"], case["height"], _generator(seed)).cpu().numpy())


def _prepare_nms(case, seed):
    be, g = _Session.get(), _generator(seed)
    b, cls, n = case["batch"], case["classes"], case["heads"]
    mean, std = (torch.from_numpy(v).cuda()[None, :, None, None] for v in _head_targets(3 * (5 + cls), cls))
    heads = []
    for k in range(n):
        gw, gh = case["grid_w"] << (n - 1 - k), case["grid_h"] << (n - 1 - k)
        raw = torch.randn((b, 3 * (5 + cls), gh, gw), generator=g, device="cuda").mul_(std).add_(mean)
        raw = (raw.sigmoid_() if case["new_coords"] else raw).cpu().numpy()
        heads.append(dict(raw=be.upload_f32(raw.shape, raw), classes=cls, anchors=[(float(p), float(q)) for p, q in synth.COCO_ANCHORS[3 * k:3 * k + 3]],
                          scale_x_y=2.0 if case["new_coords"] else 1.0, new_coords=case["new_coords"]))
    w, h = 32 * case["grid_w"], 32 * case["grid_h"]
    return dict(case=case, be=be, heads=heads, size=(w, h))


def _prepare_ops(case, seed):
    be, gw = _Session.get(), _generator(13)
    c, prec, qmax = case["channels"], PRECISION[case["precision"]], QMAX[case["precision"]]
    n, w, h = case["batch"], 2 * case["grid_w"], 2 * case["grid_h"]

    def conv(cin, f, k, target=None):
        wt = torch.randn((f, cin, k, k), generator=gw, device="cuda") * math.sqrt(_gain(ln.ACTIVATIONS[case["activation"]]) / (cin * k * k))
        bias = torch.zeros(f, device="cuda")
        if target is not None:  # head: logits of a trained-looking detector
            bias, std = (torch.from_numpy(v).cuda() for v in target)
            wt *= std[:, None, None, None]
        wt, bias = wt.cpu().numpy(), bias.cpu().numpy().reshape(1, f, 1, 1)
        t = be.upload_f32(wt.shape, wt)
        return be.conv_weights_q(t, f, cin, k, prec), be.upload_f32(bias.shape, bias)

    layers = dict(down=conv(c, 2 * c, 3), head=conv(2 * c, 255, 1, _head_targets(255, 80)))
    layers["blocks"] = [(conv(2 * c, 4 * c, 3), conv(4 * c, 2 * c, 1)) for _ in range(case["blocks"])]
    x = torch.nn.functional.leaky_relu(torch.randn((n, c, h, w), generator=_generator(seed), device="cuda"), 0.1).cpu().numpy()
    return dict(case=case, be=be, layers=layers, x=be.upload_q(x.shape, x, 6.0 / qmax, prec), y_scale=6.0 / qmax,
                anchors=[(float(p), float(q)) for p, q in synth.COCO_ANCHORS[3:6]])


def prepare(case, seed):
    return {"detect": _prepare_detect, "stream": _prepare_stream, "heads": _prepare_heads, "nms": _prepare_nms, "ops": _prepare_ops}[case["kind"]](case, seed)


def _padded(found, slots=1024):
    """Detections of a batch as one [images, slots, 7] array, zeros behind the last record: the form a batched caller hands on."""
    out = np.zeros((len(found), slots, 7), np.float32)
    for i, f in enumerate(found):
        out[i, :len(f)] = f
    return out


# ---- one pass -------------------------------------------------------------------------------------------------------------


def _run_detect(s):
    feed = s["case"]["feed"]
    if feed == "u8":
        return _padded(s["net"].detect_u8(s["images"], CONF, IOU))
    call = s["net"].detect_device if feed == "device" else s["net"].detect
    return _padded(call(s["x"], s["size"][0], s["size"][1], CONF, IOU))


def _run_stream(s):
    net, packs, out = s["net"], s["packs"], []
    net.submit_u8(None, packed=packs[0])
    for i in range(len(packs)):
        if i + 1 < len(packs):
            net.submit_u8(None, packed=packs[i + 1])
        out.append(_padded(net.collect(packs[i][2], packs[i][3], CONF, IOU)))
    return out


def _run_heads(s):
    net = s["net"]
    net.forward(s["x"])
    return [net.backend.download_f32(net.head(k)) for k in range(net.num_heads())]


def _run_nms(s):
    c = s["case"]
    found = s["be"].yolo_decode_nms(s["heads"], s["size"][0], s["size"][1], s["size"][0], s["size"][1], c["conf"], c["iou"], True, c["top_k"])
    return _padded(found, c["top_k"] or 1024)


def _run_ops(s):
    be, case, layers = s["be"], s["case"], s["layers"]
    n, w, h, c, act, ys = case["batch"], case["grid_w"], case["grid_h"], case["channels"], case["activation"], s["y_scale"]

    def conv(x, layer, cin, f, k, stride=1, act=act, out_kind=ln.LN_OUT_Q):
        return be.conv2d_bias_act_q(x, layer[0], layer[1], (n, f, h, w), cin, h * stride, w * stride, f, k, stride, stride, 1, k // 2, 1, act, ys, out_kind)

    x = conv(s["x"], layers["down"], c, 2 * c, 3, 2)
    for wide, narrow in layers["blocks"]:
        y = conv(conv(x, wide, 2 * c, 4 * c, 3), narrow, 4 * c, 2 * c, 1)
        x = be.shortcut_add_act_q(y, x, "linear", ys) if case["shortcut"] else y
    raw = conv(x, layers["head"], 2 * c, 255, 1, 1, "linear", ln.LN_OUT_F32)
    return _padded(be.yolo_decode_nms([dict(raw=raw, classes=80, anchors=s["anchors"])], 16 * w, 16 * h, 16 * w, 16 * h, CONF, IOU))


def run(state):
    return {"detect": _run_detect, "stream": _run_stream, "heads": _run_heads, "nms": _run_nms, "ops": _run_ops}[state["case"]["kind"]](state)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------

RECORDS = 64 * 28  # bytes of detections per image that a caller reads, of the order of


def work(case):
    """Inputs, weights (at their storage width) and results once; operations of the convolutions, two per multiply-add."""
    kind, b = case["kind"], case["batch"]
    if kind == "nms":
        floats = case["grid_w"] * case["grid_h"] * 3 * (5 + case["classes"]) * sum(4 ** k for k in range(case["heads"]))
        return {"bytes": b * (4 * floats + RECORDS), "flops": 0}
    if kind == "ops":
        c, cells = case["channels"], case["grid_w"] * case["grid_h"]
        weights = 18 * c * c + case["blocks"] * (72 + 8) * c * c + 2 * c * 255
        return {"bytes": b * (4 * cells * c + RECORDS) + weights, "flops": 2 * b * cells * weights}
    per_pixel, weights, head = MODEL[case["model"]]
    pixels = case["width"] * case["height"]
    width = {"f32": 4, "f16": 2}.get(case["precision"], 1)
    n = b * case.get("batches", 1)
    if "frames" in case:
        sizes = [tuple(int(v) for v in s.split("x")) for s in case["frames"].split(",")]
        source = case.get("batches", 1) * sum(3 * sizes[i % len(sizes)][0] * sizes[i % len(sizes)][1] for i in range(b))
    else:
        source = n * 12 * pixels
    result = n * (4 * int(pixels * head) if kind == "heads" else RECORDS)
    return {"bytes": source + weights * width + result, "flops": n * pixels * per_pixel}


def tolerance(case):
    """8-bit codes are whole numbers and decode + NMS is defined bit for bit, so detections are compared as they are.  f32 heads:
    32-bit sums of up to 4608 terms in up to 110 layers.  f16 heads: one rounding to 11 bits per layer and stored operator."""
    if case["kind"] == "heads":
        return {"rel": 5e-5} if case["precision"] == "f32" else {"rel": 1e-2}
    return "exact"
