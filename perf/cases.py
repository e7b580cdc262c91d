"""The performance cases of the quantized operator library: what a user has it do, through its public entry points.

A program that uses the library either prepares single operators and enqueues them on device tensors (conv2d, depthwise,
fully_connected, deconv followed by Op.execute), or builds an operator list once (a whole network) and runs it batch by
batch: with host buffers and a blocking call (OpList.execute_host_ptrs), with host buffers in a pipeline
(OpList.submit_host_ptrs) or on tensors that are on the device already (OpList.execute_device).  The listed cases are the
benchmark configurations of this repository with the network at both ends of its batch range, and ragged layers between
them (channel counts of 48, 72, 120 and 200, odd image sizes, strides, signed activations); `draw` gives others of the
same ranges.  All results are bytes and exact.
"""
import functools
import importlib
import math

import numpy as np
import torch

enn = importlib.import_module("cl-eden-kernel_b200")
mobilenet = importlib.import_module("cl-eden-kernel_b200.mobilenet")

U8, S8 = "u8", "s8"


def _conv(name, op, n, h, w, cin, cout, k, stride, act, weights, relu6):
    """op: conv | depthwise | deconv (deconv: `stride` is the upsampling factor); act: u8 | s8 activations; weights:
    tensor (u8, one scale and zero point) | channel (int8, a scale per output channel)."""
    case = dict(op=op, n=n, h=h, w=w, cin=cin, cout=cout, k=k, stride=stride, act=act, weights=weights, relu6=relu6)
    return dict(case, name=name) if name else case


def _fc(name, m, k, n, act=U8, weights="channel"):
    case = dict(op="fc", m=m, k=k, n=n, act=act, weights=weights)
    return dict(case, name=name) if name else case


def _net(name, batch, resolution, call):
    """call: execute (host buffers, blocking) | submit (host buffers, pipelined) | device (tensors on the device)."""
    case = dict(op="net", batch=batch, resolution=resolution, call=call)
    return dict(case, name=name) if name else case


def listed():
    return [
        # One 3x3 convolution on one image: an interactive call, all launch and pipeline latency.
        _conv("conv3x3_1x56x56x64", "conv", 1, 56, 56, 64, 64, 3, 1, U8, "tensor", True),
        # The same layer on a full batch: the body of a convolutional network, offline throughput.
        _conv("conv3x3_256x56x56x64", "conv", 256, 56, 56, 64, 64, 3, 1, U8, "tensor", True),
        # A downsampling convolution with signed activations, odd image size and a channel count that fills no tile.
        _conv("conv3x3s2_32x57x57x48", "conv", 32, 57, 57, 48, 96, 3, 2, S8, "channel", True),
        # A pointwise layer of a slim mobile network: channel counts that are multiples of 8 and of nothing larger.
        _conv("conv1x1_16x28x28x72", "conv", 16, 28, 28, 72, 200, 1, 1, U8, "channel", False),
        # Depthwise layers: the benchmark's stride-1 layer; a stride-2 layer with odd sizes.
        _conv("dw3x3_64x112x112x32", "depthwise", 64, 112, 112, 32, 32, 3, 1, U8, "channel", True),
        _conv("dw3x3s2_24x75x75x120", "depthwise", 24, 75, 75, 120, 120, 3, 2, U8, "channel", True),
        # FullyConnected at batch 1 (weight streaming), at a small batch, and as a large matrix product.
        _fc("fc_1x4096x4096", 1, 4096, 4096),
        _fc("fc_256x1024x1024", 256, 1024, 1024),
        _fc("fc_4096x4096x4096", 4096, 4096, 4096),
        # The upsampling layer of a decoder.
        _conv("deconv4x4s2_8x64x64x128", "deconv", 8, 64, 64, 128, 64, 4, 2, U8, "tensor", False),
        # The whole network: one image from a host buffer to logits in a host buffer, and the benchmark's batch of 256.
        _net("mobilenetv2_1x224", 1, 224, "execute"),
        _net("mobilenetv2_256x224", 256, 224, "device"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _channels(rng, lo, hi):
    """Channel counts as networks have them: multiples of 8 mostly, now and then a multiple of 4 only."""
    step = 4 if rng.random() < 0.15 else 8
    return max(step, _log(rng, lo, hi) // step * step)


MOST_MACS = 40e9        # about half of the largest listed case's
MOST_BYTES = 400e6


def draw(rng):
    while True:
        kind = rng.choice(["conv", "pointwise", "depthwise", "fc", "deconv", "net"])
        act = S8 if rng.random() < 0.2 else U8
        weights = rng.choice(["channel", "tensor"])
        relu6 = rng.random() < 0.6
        n = _log(rng, 1, 256)
        if kind == "conv":
            h = _log(rng, 7, 112)
            stem = rng.random() < 0.15      # the first layer of a network: three channels, large image
            case = _conv(None, "conv", n, 2 * h if stem else h, 2 * h if stem else h, 3 if stem else _channels(rng, 16, 256), _channels(rng, 16, 256),
                         5 if rng.random() < 0.1 else 3, 2 if stem else rng.choice([1, 1, 2]), act, weights, relu6)
        elif kind == "pointwise":
            h = _log(rng, 7, 112)
            case = _conv(None, "conv", n, h, h, _channels(rng, 16, 960), _channels(rng, 16, 1280), 1, 1, act, weights, relu6)
        elif kind == "depthwise":
            h, c = _log(rng, 7, 112), _channels(rng, 16, 960)
            case = _conv(None, "depthwise", n, h, h, c, c, 5 if rng.random() < 0.15 else 3, rng.choice([1, 1, 2]), act, weights, relu6)
        elif kind == "deconv":
            k, stride = rng.choice([(4, 2), (4, 2), (2, 2), (3, 2)])
            h = _log(rng, 8, 64)
            case = _conv(None, "deconv", _log(rng, 1, 32), h, h, _channels(rng, 16, 256), _channels(rng, 8, 128), k, stride, act, weights, False)
        elif kind == "fc":
            case = _fc(None, _log(rng, 1, 4096), _channels(rng, 64, 4096), _log(rng, 10, 4096), act, weights)
        else:
            call = rng.choice(["execute", "submit", "device"])
            return _net(None, n if call == "device" else _log(rng, 1, 128), rng.choice([96, 128, 160, 192, 224]), call)
        w = work(case)
        if w["flops"] <= 2 * MOST_MACS and w["bytes"] <= MOST_BYTES:
            return case


# ---- geometry and quantisation ----------------------------------------------------------------------------------------

def _pads(c):
    """(top/left, bottom/right) padding and output height / width."""
    if c["op"] == "deconv":
        p = (c["k"] - c["stride"]) // 2
        return p, p, (c["h"] - 1) * c["stride"] + c["k"] - 2 * p, (c["w"] - 1) * c["stride"] + c["k"] - 2 * p
    out = -(-c["h"] // c["stride"])                                    # SAME padding, square images
    total = max(0, (out - 1) * c["stride"] + c["k"] - c["h"])
    return total // 2, total - total // 2, out, out


def work(case):
    """Inputs, weights, bias and scales read once, outputs written once; two operations per multiply-accumulate."""
    if case["op"] == "net":
        layers, _ = _network(case["resolution"])
        macs, _ = mobilenet.graph_work(layers, case["batch"])
        weights = sum(L["w"].size + 12 * L["cout"] for L in layers if "w" in L)
        return {"bytes": case["batch"] * (case["resolution"] ** 2 * 3 + layers[-1]["cout"]) + weights, "flops": 2 * macs}
    if case["op"] == "fc":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": m * k + k * n + m * n + 12 * n, "flops": 2 * m * k * n}
    _, _, oh, ow = _pads(case)
    taps, cin, cout = case["k"] ** 2, case["cin"], case["cout"]
    filt = taps * (1 if case["op"] == "depthwise" else cin)            # weights per output channel
    macs = case["n"] * (case["h"] * case["w"] if case["op"] == "deconv" else oh * ow) * cout * filt
    return {"bytes": case["n"] * (case["h"] * case["w"] * cin + oh * ow * cout) + (filt + 12) * cout, "flops": 2 * macs}


def tolerance(case):
    return "exact"      # integer arithmetic throughout


# ---- states -----------------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _context():
    return enn.Context(0)      # the program's device and in-order stream


@functools.lru_cache(maxsize=None)
def _network(resolution):
    """The program's model: fixed weights and scales, as if read from a file."""
    return mobilenet.build_model(seed=0, calib_images=1, resolution=resolution)


class _State:
    """What the program holds for its calls."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


class _Op:
    """A prepared operator, released with its last user."""

    def __init__(self, op):
        self.op = op

    def __del__(self):
        self.op.release()


class _Net:
    """An operator list, destroyed with its last user."""

    def __init__(self, oplist, info):
        self.oplist, self.tensor_ids = oplist, info["tensor_ids"]

    def __del__(self):
        self.oplist.destroy()

    def tensor(self, name, shape):
        """The list's own tensor `name` as a torch tensor, without a copy; the list lives as long as that tensor."""
        ptr = self.oplist.tensor_ptr(self.tensor_ids[name]).value
        return torch.as_tensor(_DeviceView(self, ptr, shape), device="cuda")


class _DeviceView:
    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "|u1", "data": (ptr, False), "version": 2}


def _bytes(gen, shape, act):
    lo = -128 if act == S8 else 0
    return torch.randint(lo, lo + 256, shape, dtype=torch.int8 if act == S8 else torch.uint8, device="cuda", generator=gen)


def prepare(case, seed):
    ctx = _context()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    if case["op"] == "net":
        layers, _ = _network(case["resolution"])
        shape = (case["batch"], case["resolution"], case["resolution"], 3)
        net = _Net(*mobilenet.make_oplist(enn, ctx, layers, case["batch"], case["resolution"]))
        images = _bytes(gen, shape, U8)
        logits = (case["batch"], layers[-1]["cout"])
        if case["call"] == "device":       # images are decoded on the device straight into the list's input tensor
            x = net.tensor("input", shape)
            x.copy_(images)
            return _State(call="device", net=net, x=x, y=net.tensor("fc", logits))
        return _State(call=case["call"], net=net, x=images.cpu().pin_memory(), y=torch.empty(logits, dtype=torch.uint8).pin_memory())

    per_channel = case["weights"] == "channel"
    zp = 0 if case["act"] == S8 else 128
    if case["op"] == "fc":
        m, k, n = case["m"], case["k"], case["n"]
        x, out_shape, reduction, wshape = _bytes(gen, (m, k), case["act"]), (m, n), k, (n, k)
        relu6 = False
    else:
        n = case["cout"]
        lo, hi, oh, ow = _pads(case)
        x, out_shape = _bytes(gen, (case["n"], case["h"], case["w"], case["cin"]), case["act"]), (case["n"], oh, ow, n)
        k, cin = case["k"], case["cin"]
        if case["op"] == "depthwise":
            reduction, wshape = k * k, (1, k, k, n)
        else:
            reduction, wshape = k * k * cin // (case["stride"] ** 2 if case["op"] == "deconv" else 1), (n, k, k, cin)
        relu6 = case["relu6"]
    # Bytes over their whole range, as calibrated tensors have them; weight scales that give outputs a deviation of about two.
    if per_channel:
        w = rng.integers(-127, 128, wshape, dtype=np.int8)
    else:
        w = rng.integers(0, 256, wshape, dtype=np.uint8)
    bias = rng.integers(-1000, 1001, n, dtype=np.int32)
    in_scale, w_zp = 0.02, 0 if per_channel else 125
    w_scale = 2.0 / (math.sqrt(reduction) * 73.9 * 73.3 * in_scale)
    scales = (w_scale * np.exp(rng.uniform(math.log(0.5), math.log(2.0), n))).astype(np.float32) if per_channel else None
    if relu6:
        out_scale, out_zp = 6.0 / 255.0, zp - 128
    else:
        out_scale, out_zp = 8.0 / 127.0, zp
    quant = dict(activation=enn.ACT_RELU6 if relu6 else enn.ACT_NONE, act_dtype=enn.S8 if case["act"] == S8 else enn.U8,
                 weight_dtype=enn.S8 if per_channel else enn.U8, per_channel=int(per_channel), in_scale=in_scale, in_zp=zp, w_scale=w_scale,
                 w_zp=w_zp, out_scale=out_scale, out_zp=out_zp)
    if case["op"] == "fc":
        d = enn.FcDesc(m=m, k=k, n=n, bias_scale=float(np.float32(in_scale) * np.float32(w_scale)), **quant)
        op = enn.fully_connected(ctx, d, w, bias, scales)
    else:
        d = enn.conv_desc(n=case["n"], h=case["h"], w=case["w"], cin=case["cin"], cout=n, kh=k, kw=k, stride_h=case["stride"],
                          stride_w=case["stride"], pad_t=lo, pad_l=lo, pad_b=hi, pad_r=hi, weight_layout=enn.W_OHWI, **quant)
        make = {"conv": enn.conv2d, "depthwise": enn.depthwise, "deconv": enn.deconv}[case["op"]]
        op = make(ctx, d, w, bias, scales)
    y = torch.empty(out_shape, dtype=x.dtype, device="cuda")
    return _State(call="op", op=_Op(op), x=x, y=y)


def run(state):
    if state.call == "op":
        state.op.op.execute(state.x.data_ptr(), state.y.data_ptr())
    elif state.call == "device":
        state.net.oplist.execute_device()
    elif state.call == "submit":
        state.net.oplist.submit_host_ptrs([state.x.data_ptr()], [state.y.data_ptr()])
    else:
        state.net.oplist.execute_host_ptrs([state.x.data_ptr()], [state.y.data_ptr()])
    return state.y
