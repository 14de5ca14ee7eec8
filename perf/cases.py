"""Timed cases of the quantized forward path, through the calls a user makes: dl::Model (espdl_b200.model.Model) for whole
networks and the C ABI (espdl_b200.abi) for single operators on device tensors.

A case is a dict of plain values.  `kind` says which call it is:
  net    a network through Model.  mode "run": host arrays in, host arrays out; "device": inputs and outputs stay on the GPU;
         "image": uint8 camera frames -> preprocess -> run_device -> classify / detect
  gemm   A[m][k] x W[n][k]                              espdl_b200_conv2d, 1x1 geometry
  conv   dense or depthwise convolution of NHWC images   espdl_b200_conv2d
  mem    an operator bound by memory traffic             espdl_b200_eltwise / _pool / _softmax / _norm / _copy
Every integer result is defined bit for bit by the reference's arithmetic.
"""
import ctypes as C
import math
import os
import tempfile

import numpy as np
import torch

import __graft_entry__ as entry

entry._package()
from espdl_b200 import abi, espdl_file, model, zoo  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = os.path.join(ROOT, "tests", "golden")
MOST_FLOPS = 6e11  # of one pass: the classifier at batch 1024

# network -> (file under tests/golden/espdl, or None for one that is generated; largest batch drawn)
NETS = {
    "streaming_tcn": ("esp32p4__streaming_tcn.espdl", 64),            # 1-D convolutions over a sensor window, 20 nodes
    "mobilenet_v2": (None, 1024),                                     # the benchmark's classifier, 224x224
    "yolo11n_320": ("esp32p4__zoo_yolo11n_320.espdl", 64),            # the shipped detector, 320x320
    "yolo11n_640": (None, 32),                                        # the detector at the benchmarked resolution
    "ocr_det": ("esp32p4__zoo_ocr_det.espdl", 4),                     # text detection, 736x736
    "person_reid": ("esp32p4__zoo_person_reid.espdl", 128),           # re-identification of 192x96 person crops
}
HEADS_320 = [("box0", "score0"), ("box1", "score1"), ("box2", "score2")]
TOP_BOXES = 10
MEM_OPS = ("add", "requantize", "maxpool", "softmax", "layernorm", "transpose")


def listed():
    return [
        # one window of a sensor stream: the smallest network, all launch latency
        dict(name="tcn_run_1", kind="net", net="streaming_tcn", mode="run", batch=1),
        # a camera application of the classifier: one VGA frame in, five categories out
        dict(name="mobilenet_v2_image_1", kind="net", net="mobilenet_v2", mode="image", batch=1, src_h=480, src_w=640),
        # offline classification of a resident batch: the benchmark's step
        dict(name="mobilenet_v2_device_1024", kind="net", net="mobilenet_v2", mode="device", batch=1024),
        # a camera application of the detector: one VGA frame, letterboxed, boxes out
        dict(name="yolo11n_320_image_1", kind="net", net="yolo11n_320", mode="image", batch=1, src_h=480, src_w=640),
        # video analytics: frames of 16 cameras
        dict(name="yolo11n_640_device_16", kind="net", net="yolo11n_640", mode="device", batch=16),
        # a document page: large maps, squeeze-and-excite blocks, Gelu tables, half-to-even rounding
        dict(name="ocr_det_run_1", kind="net", net="ocr_det", mode="run", batch=1),
        # the person crops of a frame, an odd number of them
        dict(name="person_reid_run_27", kind="net", net="person_reid", mode="run", batch=27),
        # matrix products of the operator benchmark: int8 and int16
        dict(name="gemm_s8_4096x1024x1024", kind="gemm", bits=8, m=4096, k=1024, n=1024),
        dict(name="gemm_s16_4096x1024x1024", kind="gemm", bits=16, m=4096, k=1024, n=1024),
        # the 3x3 layer of the operator benchmark over a large batch
        dict(name="conv3x3_s8_1024x56x56x64", kind="conv", bits=8, batch=1024, h=56, w=56, cin=64, cout=64, k=3, stride=1, depthwise=False),
        # a 3x3 layer that a mixed-precision detector keeps in int16
        dict(name="conv3x3_s16_4x40x40x64", kind="conv", bits=16, batch=4, h=40, w=40, cin=64, cout=64, k=3, stride=1, depthwise=False),
        # token normalisation: rows of 768 at the size of the operator benchmark's tensors (77 MB)
        dict(name="layernorm_s8_100352x768", kind="mem", op="layernorm", bits=8, rows=100352, len=768),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    """One more case of the listed ranges: sizes spread over their logarithm, ragged ones among them."""
    kind = rng.choices(("net", "gemm", "conv", "mem"), (6, 3, 3, 2))[0]
    bits = 16 if rng.random() < 0.3 else 8
    if kind == "net":
        net = rng.choice(sorted(NETS))
        mode = rng.choice(("run", "device", "image") if net in ("mobilenet_v2", "yolo11n_320") else ("run", "device"))
        # host arrays and frames come in the numbers an application has at hand
        case = dict(kind="net", net=net, mode=mode, batch=_log(rng, 1, min(NETS[net][1], {"run": 128, "device": 1024, "image": 8}[mode])))
        if mode == "image":
            case.update(src_h=rng.randint(120, 1080), src_w=rng.randint(160, 1920))
        return case
    if kind == "gemm":
        k = _log(rng, 16, 4096)
        if rng.random() < 0.75:
            k = max(16, k // 16 * 16)
        m, n = _log(rng, 1, 65536), _log(rng, 8, 4096)
        limit = MOST_FLOPS / (4 if bits == 16 else 1) / (1 if k % 16 == 0 else 100)
        while 2.0 * m * k * n > limit:
            m = m // 2 + 1
        return dict(kind="gemm", bits=bits, m=m, k=k, n=n)
    if kind == "conv":
        hw, depthwise = _log(rng, 7, 112), rng.random() < 0.3
        cin = rng.choice((3, 8, 16, 24, 32, 48, 64, 96, 128, 192, 256))
        cout = cin if depthwise else rng.choice((8, 16, 24, 32, 48, 64, 80, 96, 128, 192, 256))
        k = rng.choice((3, 3, 3, 5) if depthwise else (1, 3, 3, 3, 5))
        case = dict(kind="conv", bits=bits, batch=_log(rng, 1, 1024), h=hw, w=max(7, hw + rng.randint(-3, 3)), cin=cin, cout=cout, k=k,
                    stride=rng.choice((1, 1, 2)), depthwise=depthwise)
        while work(case)["flops"] > MOST_FLOPS / (100 if bits == 16 or cin % 16 else 2) or work(case)["bytes"] > 6e8:
            case["batch"] = case["batch"] // 2 + 1
            if case["batch"] <= 2:
                case["batch"], case["h"], case["w"] = 1, min(hw, 40), min(case["w"], 40)
                break
        return case
    op = rng.choice(MEM_OPS)
    length = _log(rng, 16, 1024)
    return dict(kind="mem", op=op, bits=8 if op == "softmax" else bits, rows=max(1, _log(rng, 20000, 80000000) // length), len=length)


# ------------------------------------------------------------------------------------------ networks
_paths = {}


def _net_path(net):
    """The network's file: shipped with the tests, or generated once per process from a fixed seed."""
    if net not in _paths:
        shipped = NETS[net][0]
        if shipped:
            _paths[net] = os.path.join(GOLDEN, "espdl", shipped)
        else:
            g = zoo.mobilenet_v2(seed=5) if net == "mobilenet_v2" else zoo.yolo11n_640(os.path.join(GOLDEN, "yolo11n_640_topology.json"), seed=6)
            fd, _paths[net] = tempfile.mkstemp(suffix=".espdl", prefix=net + "_")
            os.close(fd)
            g.save(_paths[net])
    return _paths[net]


class _Owned:
    """A buffer of a model as an array that keeps the model alive."""

    def __init__(self, owner, io, on_device):
        self.owner = owner
        spec = {"shape": tuple(io.shape), "typestr": np.dtype(model.NP[io.dtype]).str,
                "data": (io.device_ptr if on_device else io.host_ptr, False), "version": 3}
        setattr(self, "__cuda_array_interface__" if on_device else "__array_interface__", spec)


def _prepare_net(case, seed):
    m = model.Model(_net_path(case["net"]), batch=case["batch"])
    rng = np.random.default_rng(seed)
    s = dict(kind="net", case=case, model=m)
    if case["mode"] == "image":
        # frames with the smooth variation and the noise of a camera picture
        h, w = case["src_h"], case["src_w"]
        coarse = rng.integers(0, 256, size=(case["batch"], h // 40 + 2, w // 40 + 2, 3), dtype=np.int16)
        frames = coarse.repeat(40, axis=1).repeat(40, axis=2)[:, :h, :w]
        s["frames"] = np.clip(frames + rng.integers(-20, 21, size=frames.shape, dtype=np.int16), 0, 255).astype(np.uint8)
        s["out"] = {o.name: torch.as_tensor(_Owned(m, o, True), device="cuda") for o in m.outputs}
        return s
    for t in m.inputs:
        info = np.iinfo(t.array.dtype)
        t.array[...] = rng.integers(info.min, info.max + 1, size=t.shape, dtype=t.array.dtype)
    if case["mode"] == "run":
        s["out"] = {o.name: np.asarray(_Owned(m, o, False)) for o in m.outputs}
    else:
        m.run()  # brings the inputs to the device, where they stay
        s["out"] = {o.name: torch.as_tensor(_Owned(m, o, True), device="cuda") for o in m.outputs}
    return s


def _run_net(s):
    case, m = s["case"], s["model"]
    if case["mode"] == "run":
        m.run()
        return s["out"]
    if case["mode"] == "device":
        m.run_device()
        return s["out"]
    if case["net"] == "mobilenet_v2":
        m.preprocess(s["frames"], mean=(123.675, 116.28, 103.53), std=(58.395, 57.12, 57.375), rgb_swap=True)
        m.run_device()
        found = [m.classify(image=i, top_k=5) for i in range(case["batch"])]
        return dict(s["out"], categories=np.array([[c for c, _ in f] for f in found], dtype=np.int32),
                    scores=np.array([[p for _, p in f] for f in found], dtype=np.float32))
    m.preprocess(s["frames"], mean=(0.0, 0.0, 0.0), std=(255.0, 255.0, 255.0), letterbox=114)
    m.run_device()
    found = [m.detect(HEADS_320, (8, 16, 32), 0.25, 0.7, TOP_BOXES, case["src_w"], case["src_h"], image=i) for i in range(case["batch"])]
    boxes = np.full((case["batch"], TOP_BOXES, 5), -1, dtype=np.int32)  # category and corners of each box found, best first
    scores = np.zeros((case["batch"], TOP_BOXES), dtype=np.float32)
    for i, of_image in enumerate(found):
        for j, (category, score, corners) in enumerate(of_image):
            boxes[i, j], scores[i, j] = (category,) + corners, score
    return dict(s["out"], boxes=boxes, scores=scores)


_net_figures = {}


def _net_work(case):
    """Parameters once, graph inputs (or frames) and outputs once per image, two operations per multiply-accumulate."""
    net = case["net"]
    if net not in _net_figures:
        p = espdl_file.read(_net_path(net))
        shapes = {v["name"]: v["shape"] for v in list(p["value_info"].values()) + p["inputs"] + p["outputs"]}
        params = sum(t["data"].nbytes for t in p["initializers"].values())
        macs = 0
        for node in p["nodes"]:
            out = int(np.prod(shapes[node["outputs"][0]]))
            if node["op_type"] in ("Conv", "Gemm"):
                wd = p["initializers"][node["inputs"][1]]["dims"]
                macs += out * int(np.prod(wd)) // (int(wd[-1]) if node["attrs"].get("group", 1) == 1 else int(wd[-2]) * int(wd[-1]))
            elif node["op_type"] == "MatMul":
                macs += out * int(shapes[node["inputs"][0]][-1])
        _net_figures[net] = (params, sum(int(np.prod(i["shape"])) for i in p["inputs"]), sum(int(np.prod(o["shape"])) for o in p["outputs"]), macs)
    params, n_in, n_out, macs = _net_figures[net]
    if case["mode"] == "image":
        n_in = min(n_in, case["src_h"] * case["src_w"] * 3)  # the resize reads one source pixel per destination pixel
    return {"bytes": params + case["batch"] * (n_in + n_out), "flops": 2 * macs * case["batch"]}


# ------------------------------------------------------------------------------------------ single operators
_ready = []


def _lib():
    L = abi.load()
    if not _ready:
        abi.check(L.espdl_b200_init(0), "espdl_b200_init")
        _ready.append(True)
    return L


def _codes(gen, shape, bits, rms):
    """Quantised values as activations have them: bell-shaped, saturated at the ends of the type."""
    top = (1 << (bits - 1)) - 1
    x = torch.randn(shape, generator=gen, device="cuda").mul_(rms).round_().clamp_(-top - 1, top)
    return x.to(torch.int8 if bits == 8 else torch.int16)


def _out_hw(case):
    pad = case["k"] // 2
    return [(case[a] + 2 * pad - case["k"]) // case["stride"] + 1 for a in ("h", "w")]


def _prepare_conv(case, seed):
    """A layer with per-channel filter exponents, a bias and ReLU whose results use the range of the type."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    bits = case["bits"]
    rms = 28.0 if bits == 8 else 3000.0
    if case["kind"] == "gemm":
        n, h, w, cin, cout, k, stride, depthwise, oh, ow = 1, 1, case["m"], case["k"], case["n"], 1, 1, False, 1, case["m"]
    else:
        n, h, w, cin, cout, k, stride, depthwise = (case[a] for a in ("batch", "h", "w", "cin", "cout", "k", "stride", "depthwise"))
        oh, ow = _out_hw(case)
    taps = k * k * (1 if depthwise else cin)
    shift = max(1, int(round(math.log2(rms * math.sqrt(taps)))))
    x = _codes(gen, (n, h, w, cin), bits, rms)
    wt = _codes(gen, (k, k, cin) if depthwise else (cout, k, k, cin), bits, rms)
    bias = (torch.randn(cout, generator=gen, device="cuda") * (0.3 * rms * 2.0 ** shift)).to(torch.int32 if bits == 8 else torch.int64)
    e_out = -5
    exps = torch.randint(-1, 2, (cout,), generator=gen, device="cuda", dtype=torch.int32) + (e_out + 7 - shift)
    out = torch.empty((n, oh, ow, cout), dtype=x.dtype, device="cuda")
    d = abi.ConvDesc()
    d.input, d.filter, d.bias, d.output, d.filter_exponents = (t.data_ptr() for t in (x, wt, bias, out, exps))
    d.dtype = abi.DTYPE_INT8 if bits == 8 else abi.DTYPE_INT16
    d.n, d.in_h, d.in_w, d.in_c, d.out_h, d.out_w, d.out_c = n, h, w, cin, oh, ow, cout
    d.kh = d.kw = k
    d.stride_h = d.stride_w = stride
    d.dilation_h = d.dilation_w = 1
    d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = k // 2
    d.group = cin if depthwise else 1
    d.in_exponent, d.out_exponent, d.per_channel, d.activation = -7, e_out, 1, abi.ACT_RELU
    return dict(kind="op", call=_lib().espdl_b200_conv2d, desc=d, keep=(x, wt, bias, exps), out=out)


def _mem_shape(case):
    """The rows of a pooled or transposed tensor as square images; None where the operator sees rows only."""
    side = max(1, min(64, int(math.sqrt(case["rows"]))))
    return max(1, case["rows"] // (side * side)), side


def _mem_count(case):
    if case["op"] in ("maxpool", "transpose"):
        n, side = _mem_shape(case)
        return n * side * side * case["len"]
    return case["rows"] * case["len"]


def _prepare_mem(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    L, bits, op = _lib(), case["bits"], case["op"]
    count, length = _mem_count(case), case["len"]
    dtype = abi.DTYPE_INT8 if bits == 8 else abi.DTYPE_INT16
    x = _codes(gen, (count // length, length), bits, 28.0 if bits == 8 else 3000.0)
    out = torch.empty_like(x)
    keep = [x]
    if op in ("add", "requantize"):
        call, d = L.espdl_b200_eltwise, abi.EltwiseDesc()
        d.op, d.in_dtype, d.out_dtype, d.ndim = (abi.ELT_ADD if op == "add" else abi.ELT_REQUANTIZE), dtype, dtype, 2
        for i, v in enumerate(x.shape):
            d.out_shape[i] = d.in0_shape[i] = v
            d.in1_shape[i] = v if op == "add" else 1
        d.in0_exponent, d.in1_exponent, d.out_exponent = -5, -5, (-5 if op == "add" else -4)
        if op == "add":
            keep.append(_codes(gen, x.shape, bits, 28.0 if bits == 8 else 3000.0))
            d.input1 = keep[1].data_ptr()
    elif op == "maxpool":  # the 5x5 stride-1 window of a spatial pyramid
        n, side = _mem_shape(case)
        call, d = L.espdl_b200_pool, abi.PoolDesc()
        d.op, d.dtype = abi.POOL_MAX, dtype
        d.n, d.in_h, d.in_w, d.c, d.out_h, d.out_w = n, side, side, length, side, side
        d.kh = d.kw = 5
        d.stride_h = d.stride_w = 1
        d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = 2
        d.in_exponent = d.out_exponent = -5
    elif op == "softmax":  # attention rows, quantised again for the product that follows
        call, d = L.espdl_b200_softmax, abi.SoftmaxDesc()
        keep.append(torch.from_numpy(np.exp(np.float32(2.0 ** -4) * np.arange(-128, 128, dtype=np.float32))).cuda())
        d.exp_table = keep[1].data_ptr()
        d.rows, d.len, d.out_dtype, d.out_exponent, d.in_exponent = count // length, length, abi.DTYPE_INT8, -7, -4
    elif op == "layernorm":
        call, d = L.espdl_b200_norm, abi.NormDesc()
        d.op, d.dtype, d.rows, d.len = abi.NORM_LAYER, dtype, count // length, length
        keep += [_codes(gen, (length,), bits, 40.0 if bits == 8 else 10000.0), _codes(gen, (length,), bits, 10.0 if bits == 8 else 2500.0)]
        d.scale, d.bias = keep[1].data_ptr(), keep[2].data_ptr()
        d.in_exponent, d.out_exponent, d.scale_exponent, d.bias_exponent = (-5, -5, -6, -6) if bits == 8 else (-12, -12, -14, -14)
        d.epsilon = 1e-5
    else:  # NHWC -> NCHW of every image
        n, side = _mem_shape(case)
        call, d = L.espdl_b200_copy, abi.CopyDesc()
        d.elem_size, d.ndim = bits // 8, 3
        hw = side * side
        for i, (sz, ss, ds) in enumerate([(n, hw * length, hw * length), (length, 1, hw), (hw, length, 1)]):
            d.shape[i], d.src_stride[i], d.dst_stride[i] = sz, ss, ds
        d.src, d.dst = x.data_ptr(), out.data_ptr()
    if op != "transpose":
        d.output = out.data_ptr()
        if op in ("add", "requantize"):
            d.input0 = x.data_ptr()
        else:
            d.input = x.data_ptr()
    return dict(kind="op", call=call, desc=d, keep=keep, out=out)


# ------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    if case["kind"] == "net":
        return _prepare_net(case, seed)
    return _prepare_mem(case, seed) if case["kind"] == "mem" else _prepare_conv(case, seed)


def run(state):
    if state["kind"] == "net":
        return _run_net(state)
    abi.check(state["call"](C.byref(state["desc"]), None), "operator")
    return state["out"]


def work(case):
    if case["kind"] == "net":
        return _net_work(case)
    es = case["bits"] // 8
    if case["kind"] == "gemm":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": es * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    if case["kind"] == "conv":
        oh, ow = _out_hw(case)
        macs = case["k"] ** 2 * (1 if case["depthwise"] else case["cin"])
        outs = case["batch"] * oh * ow * case["cout"]
        return {"bytes": es * (case["batch"] * case["h"] * case["w"] * case["cin"] + macs * case["cout"] + outs), "flops": 2 * macs * outs}
    count = _mem_count(case)
    return {"bytes": es * count * (3 if case["op"] == "add" else 2), "flops": 0}


def tolerance(case):
    """Integer outputs are defined to the last bit; the scores that classify() and detect() give are 32-bit floats."""
    return {"rel": 1e-5} if case["kind"] == "net" and case["mode"] == "image" else "exact"
