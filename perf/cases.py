"""Performance cases: what programs built on this framework ask of it, from one small operator
call to a whole detector over a batch.

A case is a dict of plain values. ``kind`` names the entry points it goes through:

  net        a compiled model through the LITE_* runtime (``lite.Network``): the two int8
             classifiers and the fp32 detector of the model zoo
  conv       one qint8 ConvBias through ``ops``, in the NHWC layout compiled models use inside
             or in the reference's own NCHW / OIHW layouts
  matmul_s8  int8 x int8 -> int32 -> int8 matrix product with a weight matrix packed once
  matmul_f32 fp32 matrix product of two activations
  qelem      a stand-alone quantised elementwise step (a residual add no ConvBias absorbs)

``listed()`` are fixed cases, ``draw()`` gives further ones of the same ranges; ``prepare``
makes what a program holds before the call, ``run`` is one pass, ``work`` the bytes and
operations the pass cannot do without, ``tolerance`` how far two correct implementations may
be apart.
"""
import functools
import math

import numpy as np
import torch

from megcc_b200 import lite, ops, zoo


def listed():
    return [
        # Offline classification, the headline configuration: a large batch that already lies
        # in device memory, logits left there, forwards queued one behind the other.
        dict(name="resnet18_b256", kind="net", model="resnet18", batch=256, hw=224,
             per_channel=False, nchw44=False, host=False),
        # An interactive request: one image from host memory, the logits read by the host.
        dict(name="resnet18_b1_host", kind="net", model="resnet18", batch=1, hw=224,
             per_channel=False, nchw44=False, host=True),
        # A dynamic batcher's ragged batch, host to host, weights quantised per output channel.
        dict(name="resnet18_b37_per_channel", kind="net", model="resnet18", batch=37, hw=224,
             per_channel=True, nchw44=False, host=True),
        # The mobile classifier at its two benchmark batches (per-channel weights).
        dict(name="mobilenetv1_b64", kind="net", model="mobilenetv1", batch=64, hw=224,
             per_channel=True, nchw44=False, host=False),
        dict(name="mobilenetv1_b1_host", kind="net", model="mobilenetv1", batch=1, hw=224,
             per_channel=True, nchw44=False, host=True),
        # The fp32 detector: its benchmark batch, and one smaller frame of a camera stream.
        dict(name="yolox_s_b32", kind="net", model="yolox_s", batch=32, hw=640,
             per_channel=False, nchw44=False, host=False),
        dict(name="yolox_s_b1_416_host", kind="net", model="yolox_s", batch=1, hw=416,
             per_channel=False, nchw44=False, host=True),
        # The single-operator configuration, in the reference's layouts.
        dict(name="conv_64_56_nchw", kind="conv", layout="nchw", n=1, ic=64, oc=64, h=56, w=56,
             k=3, stride=1, depthwise=False, act="RELU", per_channel=False, residual=False),
        # A late layer of a residual network called on its own at a small odd batch, with the
        # residual add in the same call.
        dict(name="conv_256_14_residual", kind="conv", layout="nhwc", n=5, ic=256, oc=256, h=14,
             w=14, k=3, stride=1, depthwise=False, act="IDENTITY", per_channel=False,
             residual=True),
        # The fully connected shape of the int8 matrix-product sweep, and an fp32 product of
        # the companion sweep.
        dict(name="matmul_s8_4096_1000_2048", kind="matmul_s8", m=4096, n=1000, k=2048),
        dict(name="matmul_f32_2048", kind="matmul_f32", m=2048, n=2048, k=2048),
        # ... and one whose extents are no whole number of vectors' worth of tiles.
        dict(name="matmul_f32_1000", kind="matmul_f32", m=1000, n=1000, k=1000),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(("net", "net", "net", "conv", "conv", "matmul_s8", "matmul_f32", "qelem"))
    if kind == "net":
        model = rng.choice(("resnet18", "mobilenetv1", "yolox_s"))
        if model == "yolox_s":  # frames of a multiple of the coarsest stride
            hw = 32 * _log_int(rng, 4, 20)
            batch = _log_int(rng, 1, max(1, min(64, 32 * 640 * 640 // (hw * hw))))
        else:  # any square image a classifier's five stride-2 steps leave something of
            hw = rng.choice((96, 128, 160, 161, 192, 224, 224, 224, 250, 288))
            batch = _log_int(rng, 1, min(256, 256 * 224 * 224 // (hw * hw)))
        int8 = model != "yolox_s"
        # (the NCHW44 form exists for per-tensor and per-channel weights alike)
        return dict(kind=kind, model=model, batch=batch, hw=hw,
                    per_channel=int8 and rng.random() < 0.5, nchw44=int8 and rng.random() < 0.2,
                    host=rng.random() < 0.5)
    if kind == "conv":
        layout = rng.choice(("nhwc", "nhwc", "nchw"))
        depthwise = rng.random() < 0.25
        ic = rng.choice((16, 24, 32, 64, 64, 96, 128, 128, 192, 256, 512))
        oc = ic if depthwise else rng.choice((16, 40, 64, 64, 96, 128, 128, 256, 512, 1000))
        h, w = _log_int(rng, 7, 112), 0
        w = h if rng.random() < 0.6 else _log_int(rng, 7, 112)
        k = 3 if depthwise else rng.choice((1, 3, 3))
        stride = rng.choice((1, 1, 2))
        residual = layout == "nhwc" and not depthwise and rng.random() < 0.3
        act = "IDENTITY" if residual else rng.choice(("RELU", "RELU", "IDENTITY", "H_SWISH"))
        # at most 64 MiB of input and 2^34 operations
        most = min(1 << 26, (1 << 34) // (2 * k * k * (1 if depthwise else oc))) // (ic * h * w)
        return dict(kind=kind, layout=layout, n=_log_int(rng, 1, max(1, min(256, most))), ic=ic,
                    oc=oc, h=h, w=w, k=k, stride=stride, depthwise=depthwise, act=act,
                    per_channel=not residual and rng.random() < 0.3, residual=residual)
    if kind == "qelem":
        c, h, w = rng.choice((15, 32, 64, 100, 128, 256)), _log_int(rng, 7, 112), _log_int(rng, 7, 56)
        return dict(kind=kind, mode=rng.choice(("QADD", "QFUSE_ADD_RELU", "QMUL")),
                    n=_log_int(rng, 1, min(256, (1 << 26) // (c * h * w))), c=c, h=h, w=w)
    # most programs keep their extents to whole vectors; the others are smaller products
    whole = rng.random() < 0.7
    top, most = (8192, 1 << 38) if kind == "matmul_s8" else (4096, 1 << 36)
    m, n, k = (_log_int(rng, 64, top if whole else 2048) for _ in range(3))
    if whole:
        m, n, k = (max(64, v // 32 * 32) for v in (m, n, k))
    while m * n * k > (most if whole else 1 << 31):
        m = max(64, m // 64 * 32) if whole else m // 2
    return dict(kind=kind, m=m, n=n, k=k)


# ---- models: described and compiled once per process, as a program does at start-up ----
@functools.lru_cache(maxsize=None)
def _spec(model, hw, per_channel):
    if model == "yolox_s":
        return zoo.yolox_s(hw=hw)
    make = zoo.resnet18 if model == "resnet18" else zoo.mobilenet_v1
    return make(hw=hw, per_channel=per_channel)


@functools.lru_cache(maxsize=32)
def _compiled(model, hw, per_channel, nchw44, batch):
    spec = _spec(model, hw, per_channel)
    g = spec.to_graph() if model == "yolox_s" else spec.to_graph(nchw44=nchw44)
    return g.compile([batch])


def _outputs(case):
    """[(tensor name, shape)] of a model's outputs, as the runtime hands them back."""
    spec = _spec(case["model"], case["hw"], case["per_channel"])
    if case["model"] != "yolox_s":
        return [(spec.output + ":out", (case["batch"], spec.shapes[spec.output][0]))]
    return [(o + ":out", (case["batch"],) + tuple(spec.shapes[o])) for o in spec.outputs]


class _DeviceArray:
    """An output that stays in the network's device memory, for torch to look at in place. It
    keeps the network: the memory is the network's."""

    def __init__(self, net, ptr, shape, typestr):
        self.net = net
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False),
                                             version=3)


def _uniform_s8(gen, shape, lo=-128):
    return torch.randint(lo, 128, shape, dtype=torch.int8, device="cuda", generator=gen)


def _prepare_net(case, gen):
    f32 = case["model"] == "yolox_s"
    shape = (case["batch"], 3, case["hw"], case["hw"])
    x = torch.rand(shape, device="cuda", generator=gen) if f32 else _uniform_s8(gen, shape)
    if case["host"]:
        x = x.cpu().pin_memory()
    else:
        torch.cuda.current_stream().synchronize()  # the network reads it on its own stream
    outs = _outputs(case)
    model = _compiled(case["model"], case["hw"], case["per_channel"], case["nchw44"],
                      case["batch"])
    net = lite.Network(model, device_io=() if case["host"] else tuple(n for n, _ in outs))
    net.set_input_ptr("data", x.data_ptr(), x.numel() * x.element_size())
    return dict(kind="net", net=net, x=x, outs=outs, host=case["host"], f32=f32, views=None)


def _run_net(s):
    net = s["net"]
    net.forward()
    if s["host"]:
        net.wait()
        dtype = np.float32 if s["f32"] else np.int8
        return [net.output(n, dtype).reshape(shape) for n, shape in s["outs"]]
    if s["views"] is None:  # the addresses are fixed from the first forward on
        s["views"] = [torch.as_tensor(_DeviceArray(net, net.output_ptr(n), shape,
                                                   "<f4" if s["f32"] else "|i1"), device="cuda")
                      for n, shape in s["outs"]]
    return s["views"]


def _conv_out(case):
    pad = case["k"] // 2
    return tuple((case[d] + 2 * pad - case["k"]) // case["stride"] + 1 for d in ("h", "w"))


def _prepare_conv(case, gen):
    n, ic, oc, h, w, k = (case[v] for v in ("n", "ic", "oc", "h", "w", "k"))
    groups = ic if case["depthwise"] else 1
    icpg = ic // groups
    # the output scale keeps results spread over int8: about 40 rms, as in the model zoo
    s_src, s_flt = 0.05, 0.01
    s_dst = s_src * s_flt * 74.0 * 73.3 * math.sqrt(icpg * k * k) / 40.0
    p = ops.conv_param(n, ic, h, w, oc, k, k, case["stride"], k // 2, groups, case["act"], s_src,
                       s_flt, s_dst)
    nhwc = case["layout"] == "nhwc"
    src = _uniform_s8(gen, (n, h, w, ic) if nhwc else (n, ic, h, w))
    flt = _uniform_s8(gen, (groups, oc // groups, icpg, k, k) if groups > 1 else (oc, icpg, k, k),
                      -127)
    bias = torch.randint(-1000, 1001, (oc,), dtype=torch.int32, device="cuda", generator=gen)
    scales = z = None
    if case["per_channel"]:
        scales = 0.005 + 0.015 * torch.rand(oc, device="cuda", generator=gen)
    if case["residual"]:
        z = _uniform_s8(gen, (n,) + _conv_out(case) + (oc,))
    return dict(kind="conv", p=p, src=src, flt=ops.pack_filter(p, flt) if nhwc else flt,
                bias=bias, scales=scales, z=z, nhwc=nhwc, s_dst=s_dst)


def _run_conv(s):
    if not s["nhwc"]:
        return ops.conv_bias_qs8_nchw(s["p"], s["src"], s["flt"], s["bias"], s["scales"])
    if s["z"] is not None:
        return ops.conv_bias_qs8_nhwc_fused(s["p"], s["src"], s["flt"], s["bias"], s["z"],
                                            "QFUSE_ADD_RELU", s["s_dst"], s["s_dst"])
    return ops.conv_bias_qs8_nhwc(s["p"], s["src"], s["flt"], s["bias"], flt_scales=s["scales"])


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "net":
        return _prepare_net(case, gen)
    if kind == "conv":
        return _prepare_conv(case, gen)
    if kind == "qelem":
        shape = (case["n"], case["h"], case["w"], case["c"])
        return dict(kind=kind, mode=case["mode"], a=_uniform_s8(gen, shape),
                    b=_uniform_s8(gen, shape))
    m, n, k = case["m"], case["n"], case["k"]
    if kind == "matmul_s8":
        a, b = _uniform_s8(gen, (m, k), -127), _uniform_s8(gen, (k, n), -127)
        return dict(kind=kind, a=a, b=ops.matmul_pack_b(b), s_dst=0.002 * 73.3 ** 2 * k ** 0.5 / 40)
    return dict(kind=kind, a=torch.randn((m, k), device="cuda", generator=gen),
                b=torch.randn((k, n), device="cuda", generator=gen))


def run(state):
    kind = state["kind"]
    if kind == "net":
        return _run_net(state)
    if kind == "conv":
        return _run_conv(state)
    if kind == "qelem":
        return ops.qelemwise_qs8(state["mode"], state["a"], state["b"], 0.031, 0.047, 0.052)
    if kind == "matmul_s8":
        return ops.matmul_s8_qs8(state["a"], state["b"], 0.002, state["s_dst"])
    return ops.matmul_f32(state["a"], state["b"])


def work(case):
    kind = case["kind"]
    if kind == "net":
        # the image in, the outputs out, the weights once; feature maps in between could stay
        # on chip
        spec = _spec(case["model"], case["hw"], case["per_channel"])
        el = 4 if case["model"] == "yolox_s" else 1
        weights = sum(l["flt"].size * el + l["bias"].size * 4 for l in spec.layers
                      if l["op"] == "conv")
        io = 3 * case["hw"] ** 2 * case["batch"] + sum(math.prod(s) for _, s in _outputs(case))
        return dict(bytes=io * el + weights, flops=2.0 * _macs(case) * case["batch"])
    if kind == "conv":
        oh, ow = _conv_out(case)
        out = case["n"] * oh * ow * case["oc"]
        taps = case["k"] ** 2 * (1 if case["depthwise"] else case["ic"])
        bytes_ = (case["n"] * case["h"] * case["w"] * case["ic"] + case["oc"] * taps +
                  4 * case["oc"] * (2 if case["per_channel"] else 1) +
                  out * (2 if case["residual"] else 1))
        return dict(bytes=bytes_, flops=2.0 * out * taps)
    if kind == "qelem":
        elems = case["n"] * case["c"] * case["h"] * case["w"]
        return dict(bytes=3 * elems, flops=4.0 * elems)
    m, n, k = case["m"], case["n"], case["k"]
    el = 1 if kind == "matmul_s8" else 4
    return dict(bytes=el * (m * k + k * n + m * n), flops=2.0 * m * n * k)


@functools.lru_cache(maxsize=None)
def _macs_of(model, hw, per_channel):
    return _spec(model, hw, per_channel).macs_per_image()


def _macs(case):
    return _macs_of(case["model"], case["hw"], case["per_channel"])


def tolerance(case):
    # int8 results follow the reference's operation order bit for bit
    if case["kind"] == "matmul_f32":
        return dict(rel=1e-5)  # one fp32 sum per value, in whatever order
    if case["kind"] == "net" and case["model"] == "yolox_s":
        return dict(rel=2e-5)  # sixty fp32 layers deep
    return "exact"
