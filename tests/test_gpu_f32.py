"""fp32 operators through the C ABI against the CPU checker: 1e-4 relative / 1e-5 absolute
for the contractions (fp32 sums in another order), exact for the data-movement operators."""
import numpy as np
import pytest

import cases
import golden_util as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-4, 1e-5


@pytest.fixture(scope="module")
def ops():
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    from megcc_b200 import ops as O
    return O


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def close(got, want, rtol=RTOL, atol=ATOL):
    """|got - want| <= atol + rtol * |want| elementwise, and no NaN."""
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    assert got.shape == want.shape
    assert np.isfinite(got).all()
    err = np.abs(got - want) - (atol + rtol * np.abs(want))
    worst = float(err.max())
    assert worst <= 0, f"worst excess {worst:.3e} at {np.unravel_index(err.argmax(), err.shape)}"


def to_nchw(t):
    return t.cpu().numpy().transpose(0, 3, 1, 2)


CONV_CASES = [
    # name, n, ic, oc, h, w, k, stride, pad, act, algo
    ("umma_3x3_32_64", 2, 32, 64, 40, 40, 3, 1, 1, "SILU", "umma"),
    ("umma_3x3_s2_64_128", 2, 64, 128, 40, 40, 3, 2, 1, "SILU", "umma"),
    ("umma_1x1_128_64", 2, 128, 64, 24, 24, 1, 1, 0, "SILU", "umma"),
    ("umma_1x1_1024_512", 8, 1024, 512, 10, 10, 1, 1, 0, "IDENTITY", "umma"),
    ("umma_stem_16_32", 1, 16, 32, 64, 64, 3, 1, 1, "SILU", "umma"),
    ("umma_3x3_256_256", 4, 256, 256, 20, 20, 3, 1, 1, "RELU", "umma"),
    ("umma_ragged_oc80", 2, 128, 80, 20, 20, 1, 1, 0, "SIGMOID", "umma"),
    ("umma_ragged_m", 3, 32, 48, 27, 29, 3, 1, 1, "H_SWISH", "umma"),
    ("direct_head_oc4", 2, 128, 4, 20, 20, 1, 1, 0, "IDENTITY", "direct"),
    ("direct_head_oc1", 2, 128, 1, 20, 20, 1, 1, 0, "SIGMOID", "direct"),
    ("direct_odd", 2, 12, 20, 17, 19, 3, 2, 1, "SILU", "auto"),
    ("direct_grouped", 2, 24, 36, 15, 15, 3, 1, 1, "RELU", "auto"),
]


@pytest.mark.parametrize("case", CONV_CASES, ids=[c[0] for c in CONV_CASES])
def test_conv_bias_f32_matches_oracle(ops, oracle, case):
    name, n, ic, oc, h, w, k, stride, pad, act, algo = case
    groups = 6 if name == "direct_grouped" else 1
    r = cases.rng_for("f32_" + name)
    src = r.standard_normal((n, ic, h, w)).astype(np.float32)
    flt = (r.standard_normal((oc, ic // groups, k, k)) / np.sqrt(ic // groups * k * k)).astype(np.float32)
    bias = r.standard_normal(oc).astype(np.float32)
    p = ops.conv_f32_param(n, ic, h, w, oc, k, k, stride, pad, groups, act)
    packed = ops.pack_filter_f32(p, dev(flt))
    out = ops.conv_bias_f32_nhwc(p, ops.nchw_to_nhwc_f32(dev(src)), packed, dev(bias), algo=algo)
    want = oracle.conv_bias_f32(src, flt, bias, stride, pad, act, groups)
    close(to_nchw(out), want)
    assert ops.device_status() == 0


def test_conv_and_matmul_f32_against_reference_vectors(ops):
    """Outputs of the reference's own fp32 kernels (GI im2col ConvBias, GI 4x12 MatrixMul),
    committed under tests/golden/: 1e-4 relative / 1e-5 absolute."""
    for c in cases.f32_conv_catalogue():
        src, flt, bias = cases.f32_conv_inputs(c)
        p = ops.conv_f32_param(c["n"], c["ic"], c["h"], c["w"], c["oc"], c["k"], c["k"], c["stride"],
                               c["pad"], 1, c["act"])
        out = ops.conv_bias_f32_nhwc(p, ops.nchw_to_nhwc_f32(dev(src)),
                                     ops.pack_filter_f32(p, dev(flt)),
                                     None if bias is None else dev(bias))
        G.check_close("f32_ops", c["name"], to_nchw(out), RTOL, ATOL, src, flt, bias)
    for c in cases.f32_matmul_catalogue():
        a, b = cases.f32_matmul_inputs(c)
        G.check_close("f32_ops", c["name"], ops.matmul_f32(dev(a), dev(b)).cpu().numpy(), RTOL,
                      ATOL * np.sqrt(c["k"]), a, b)
    assert ops.device_status() == 0


def test_conv_f32_residual_and_channel_slice_of_a_wider_buffer(ops, oracle):
    """+ z after the activation (bottleneck shortcut), written into channels 32..95 of a
    128-channel buffer (a Concat without the copy)."""
    r = cases.rng_for("f32_residual_slice")
    n, ic, oc, hw = 2, 64, 64, 24
    src = r.standard_normal((n, ic, hw, hw)).astype(np.float32)
    flt = (r.standard_normal((oc, ic, 3, 3)) / 24).astype(np.float32)
    bias = r.standard_normal(oc).astype(np.float32)
    z = r.standard_normal((n, oc, hw, hw)).astype(np.float32)
    p = ops.conv_f32_param(n, ic, hw, hw, oc, 3, 3, 1, 1, 1, "SILU")
    wide = torch.full((n, hw, hw, 128), 7.0, dtype=torch.float32, device="cuda")
    ops.conv_bias_f32_nhwc(p, ops.nchw_to_nhwc_f32(dev(src)), ops.pack_filter_f32(p, dev(flt)),
                           dev(bias), z=ops.nchw_to_nhwc_f32(dev(z)), dst=wide[:, :, :, 32:],
                           dst_pitch=128, algo="umma")
    got = wide.cpu().numpy()
    want = oracle.conv_bias_f32(src, flt, bias, 1, 1, "SILU", z=z)
    close(got[:, :, :, 32:96].transpose(0, 3, 1, 2), want)
    assert (got[:, :, :, :32] == 7.0).all() and (got[:, :, :, 96:] == 7.0).all()


MATMUL_SHAPES = [(512, 512, 512), (300, 72, 640), (1024, 1000, 2048), (64, 15, 48), (2048, 2048, 2048)]


@pytest.mark.parametrize("shape", MATMUL_SHAPES, ids=["x".join(map(str, s)) for s in MATMUL_SHAPES])
def test_matmul_f32_matches_oracle(ops, oracle, shape):
    m, n, k = shape
    r = cases.rng_for("f32_matmul_%dx%dx%d" % shape)
    a = r.standard_normal((m, k)).astype(np.float32)
    b = r.standard_normal((k, n)).astype(np.float32)
    got = ops.matmul_f32(dev(a), dev(b)).cpu().numpy()
    want = oracle.matmul_f32(a, b)
    # N(0,1) operands: the sum has magnitude ~sqrt(k), and the tolerance is relative to the
    # result with the absolute part scaled likewise
    close(got, want, RTOL, ATOL * np.sqrt(k))
    assert ops.device_status() == 0


# tile widths, K splits over a cluster, the resident filter (more than 148 row tiles in one tile
# column), partial channel rows and channel tails of the tensor-core kernel
TILE_CASES = [
    # n, ic, oc, h, w, k, stride, bn, split
    (1, 64, 128, 23, 17, 3, 1, 128, 8), (1, 64, 128, 23, 17, 3, 2, 64, 4),
    (2, 36, 72, 14, 19, 3, 1, 32, 2), (1, 100, 33, 31, 9, 1, 1, 64, 4),
    (1, 16, 32, 139, 141, 3, 1, 32, 1), (1, 16, 40, 139, 141, 3, 2, 64, 1),
    (1, 32, 20, 139, 141, 3, 1, 32, 1), (3, 68, 128, 81, 80, 1, 1, 128, 1),
    (1, 20, 5, 7, 7, 1, 1, 32, 1), (1, 512, 130, 5, 5, 1, 1, 0, 0), (1, 128, 64, 9, 9, 3, 1, 0, 0),
]


@pytest.mark.parametrize("case", TILE_CASES, ids=["-".join(map(str, c)) for c in TILE_CASES])
def test_conv_f32_tile_forms_match_oracle(ops, oracle, case):
    n, ic, oc, h, w, k, stride, bn, split = case
    r = cases.rng_for("f32_tiles_" + "_".join(map(str, case)))
    src = r.standard_normal((n, ic, h, w)).astype(np.float32)
    flt = (r.standard_normal((oc, ic, k, k)) / np.sqrt(ic * k * k)).astype(np.float32)
    bias, z = (r.standard_normal(s).astype(np.float32) for s in ((oc,), (n, oc, -(-h // stride), -(-w // stride))))
    p = ops.conv_f32_param(n, ic, h, w, oc, k, k, stride, k // 2, 1, "SILU")
    room = torch.zeros(1 << 17, dtype=torch.float32, device="cuda")  # readable behind a small input
    x = room[:src.size].view(n, h, w, ic) if src.size < (1 << 16) else torch.empty(
        (n, h, w, ic), device="cuda")
    x.copy_(dev(src.transpose(0, 2, 3, 1)))
    from megcc_b200._lib import check, lib
    check(lib().mb200_register_readable_range(room.data_ptr(), room.numel() * 4))
    old = [(name, ops.set_option(name, v)) for name, v in (("f32_bn", bn), ("f32_split", split))]
    try:
        got = [ops.conv_bias_f32_nhwc(p, x, ops.pack_filter_f32(p, dev(flt)), dev(bias),
                                      z=dev(z.transpose(0, 2, 3, 1)), algo="umma") for _ in range(3)]
    finally:
        for name, v in old:
            ops.set_option(name, v)
        torch.cuda.synchronize()
        lib().mb200_unregister_readable_range(room.data_ptr())
    assert all(torch.equal(got[0], g) for g in got)  # the sums do not depend on timing
    close(to_nchw(got[0]), oracle.conv_bias_f32(src, flt, bias, stride, k // 2, "SILU", z=z))
    assert ops.device_status() == 0


@pytest.mark.parametrize("ic,oc,stride", [(32, 64, 2), (64, 32, 1)])
def test_conv_f32_of_a_whole_batch_is_the_same_every_time(ops, ic, oc, stride):
    """Layers whose resident filter leaves an odd number of ring stages to two groups of converter
    warps, on an input far beyond the L2, where a load may be overtaken by those behind it: two
    thousand launches give the same bits, and they are the general kernel's within the bar."""
    n, hw = 16, 320
    g = torch.Generator(device="cuda")
    g.manual_seed(17)
    x = torch.randn((n, hw, hw, ic), device="cuda", generator=g)
    flt = torch.randn((oc, ic, 3, 3), device="cuda", generator=g) / (ic * 9) ** 0.5
    bias = torch.randn(oc, device="cuda", generator=g)
    p = ops.conv_f32_param(n, ic, hw, hw, oc, 3, 3, stride, 1, 1, "SILU")
    packed = ops.pack_filter_f32(p, flt)
    want = ops.conv_bias_f32_nhwc(p, x, packed, bias, algo="direct")
    first = ops.conv_bias_f32_nhwc(p, x, packed, bias, algo="umma")
    assert ((first - want).abs() <= ATOL + RTOL * want.abs()).all()
    out = torch.empty_like(first)
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(2000):
        ops.conv_bias_f32_nhwc(p, x, packed, bias, dst=out, algo="umma")
        wrong += (out != first).any()
    assert int(wrong) == 0
    assert ops.device_status() == 0


@pytest.mark.parametrize("shape", [(1000, 1000, 1000), (129, 65, 4100), (77, 31, 999)],
                         ids=["k1000", "k4100_split", "k999_odd"])
def test_matmul_f32_partial_rows_match_oracle(ops, oracle, shape):
    test_matmul_f32_matches_oracle(ops, oracle, shape)


@pytest.mark.parametrize("mode", ["RELU", "SIGMOID", "SILU", "H_SWISH", "EXP", "ADD", "SUB",
                                  "MUL", "MAX", "FUSE_ADD_RELU"])
def test_elemwise_f32_matches_oracle(ops, oracle, mode):
    r = cases.rng_for("f32_elem_" + mode)
    a = (3 * r.standard_normal((3, 5, 7, 11))).astype(np.float32)
    b = (3 * r.standard_normal((3, 5, 7, 11))).astype(np.float32)
    binary = mode in ("ADD", "SUB", "MUL", "MAX", "FUSE_ADD_RELU")
    got = ops.elemwise_f32(mode, dev(a), dev(b) if binary else None).cpu().numpy()
    want = oracle.elemwise_f32(mode, a, b if binary else None)
    close(got, want, 1e-5, 1e-6)


def test_concat_resize_pool_focus_relayout_are_exact(ops, oracle):
    r = cases.rng_for("f32_movement")
    xs = [r.standard_normal((2, c, 9, 11)).astype(np.float32) for c in (16, 32, 8, 12)]
    got = ops.concat_f32_nhwc([ops.nchw_to_nhwc_f32(dev(x)) for x in xs])
    assert (to_nchw(got) == oracle.concat_f32(xs)).all()
    odd = [r.standard_normal((1, c, 5, 5)).astype(np.float32) for c in (3, 5)]
    got = ops.concat_f32_nhwc([ops.nchw_to_nhwc_f32(dev(x)) for x in odd])
    assert (to_nchw(got) == oracle.concat_f32(odd)).all()
    x = r.standard_normal((2, 24, 10, 13)).astype(np.float32)
    got = ops.resize_nearest_f32_nhwc(ops.nchw_to_nhwc_f32(dev(x)), 20, 26)
    assert (to_nchw(got) == oracle.resize_nearest_f32(x, 20, 26)).all()
    got = ops.resize_nearest_f32_nhwc(ops.nchw_to_nhwc_f32(dev(x)), 17, 31)
    assert (to_nchw(got) == oracle.resize_nearest_f32(x, 17, 31)).all()
    for window in (5, 9, 13):
        x = r.standard_normal((2, 32, 20, 20)).astype(np.float32)
        got = ops.pooling_f32_nhwc(ops.nchw_to_nhwc_f32(dev(x)), "MAX", window, 1, window // 2)
        assert (to_nchw(got) == oracle.pooling_f32(x, "MAX", window, 1, window // 2)).all()
    x = r.standard_normal((2, 6, 12, 12)).astype(np.float32)
    for mode in ("AVERAGE", "AVERAGE_COUNT_EXCLUDE_PADDING"):
        got = ops.pooling_f32_nhwc(ops.nchw_to_nhwc_f32(dev(x)), mode, 3, 2, 1)
        close(to_nchw(got), oracle.pooling_f32(x, mode, 3, 2, 1), 1e-6, 1e-7)
    img = r.uniform(0, 1, (2, 3, 32, 48)).astype(np.float32)
    got = ops.focus_f32(dev(img), 16)
    assert (to_nchw(got) == oracle.focus_f32(img, 16)).all()
    y = ops.nchw_to_nhwc_f32(dev(x))
    assert (ops.nhwc_to_nchw_f32(y).cpu().numpy() == x).all()


# ---- whole fp32 models through the compiler and the LITE_* runtime -------------------------
def run_f32_model(spec, x, forwards=3):
    from megcc_b200 import lite
    from oracle import netwalk, oracle as O
    want = netwalk.run_f32(spec, x, O)
    net = lite.Network(spec.to_graph().compile([x.shape[0]]))
    outs = []
    for _ in range(forwards):  # eager, capture, replay
        net.set_input("data", x)
        net.forward()
        net.wait()
        outs.append([net.output(n, dtype=np.float32).reshape(w.shape)
                     for n, w in zip(net.output_names(), want)])
    net.close()
    return outs, want


@pytest.mark.parametrize("hw,batch", [(128, 4), (64, 2), (224, 1)])
def test_yolox_s_matches_oracle(ops, hw, batch):
    """YOLOX-s-style detector (83 ConvBias layers, SPP, PAFPN, three decoupled heads) against
    the CPU checker walking the same layer list. 128 x 128 at batch 4 runs nearly every
    ConvBias on the tensor cores; 64 x 64 at batch 2 leaves the deep, small maps to the
    general kernel."""
    from megcc_b200 import zoo
    spec = zoo.yolox_s(hw=hw)
    x = cases.rng_for(f"yolox_{hw}").uniform(0, 1, (batch, 3, hw, hw)).astype(np.float32)
    outs, want = run_f32_model(spec, x)
    for i, got in enumerate(outs):
        for g, w in zip(got, want):
            close(g, w)
    # the outputs must exercise the arithmetic: regressions and scores spread, nothing
    # collapsed to a constant or saturated
    assert all(w[:, :4].std() > 0.1 and 0.02 < w[:, 5:].std() < 0.45 for w in want)
    assert ops.device_status() == 0


def test_fp32_matmul_model_matches_oracle(ops, oracle):
    """conv -> global average pool -> MatrixMul (fp32) through the compiler and the runtime."""
    from megcc_b200 import lite
    from megcc_b200.compiler import Graph
    r = cases.rng_for("f32_gap_matmul")
    n = 256
    g = Graph("gap_matmul_f32")
    x = g.input_f32("data", 32, 8, 8)
    f = (r.standard_normal((64, 32, 3, 3)) / 17).astype(np.float32)
    y = g.conv_f32("conv", x, f, None, 1, 1, "RELU")
    y = g.pooling("gap", y, "AVERAGE", 8, 8, 0)
    b = r.standard_normal((64, 200)).astype(np.float32)
    y = g.matmul_f32("fc", y, b)
    g.mark_output(y)
    src = r.standard_normal((n, 32, 8, 8)).astype(np.float32)
    conv = oracle.conv_bias_f32(src, f, None, 1, 1, "RELU")
    pooled = oracle.pooling_f32(conv, "AVERAGE", 8, 8, 0).reshape(n, 64)
    want = oracle.matmul_f32(pooled, b)
    net = lite.Network(g.compile([n]))
    for _ in range(3):
        net.set_input("data", src)
        net.forward()
        net.wait()
        got = net.output(net.output_names()[0], dtype=np.float32).reshape(n, 200)
        close(got, want, RTOL, 3 * ATOL)
    net.close()


# channels per CTA of the row-maxima kernel (1, 2 or 8 groups of four), no padding, the largest map
# that fits shared memory and one that does not
@pytest.mark.parametrize("shape,window,pad", [
    ((1, 4, 7, 5), 4, 0), ((3, 12, 6, 31), 5, 2), ((40, 128, 5, 5), 5, 2), ((1, 64, 13, 13), 13, 6),
    ((1, 8, 56, 56), 5, 2), ((1, 4, 80, 80), 4, 1)], ids=lambda v: str(v))
def test_max_pooling_by_rows_is_exact(ops, oracle, shape, window, pad):
    x = cases.rng_for(f"f32_rowmax_{shape}_{window}").standard_normal(shape).astype(np.float32)
    got = ops.pooling_f32_nhwc(ops.nchw_to_nhwc_f32(dev(x)), "MAX", window, 1, pad)
    assert (to_nchw(got) == oracle.pooling_f32(x, "MAX", window, 1, pad)).all()


# concats whose inputs are written in place: all of them, some of them (an elementwise operator
# writes dense pixels), a slice that other operators read, one input taken twice
@pytest.mark.parametrize("batch", [1, 3, 160])
@pytest.mark.parametrize("form", ["all", "some", "twice"])
def test_concat_slices_in_place_match_oracle(ops, oracle, batch, form):
    from megcc_b200 import lite
    from megcc_b200.compiler import Graph
    r = cases.rng_for(f"f32_slices_{form}")
    f = {n: (r.standard_normal(s) / np.sqrt(s[1] * s[2] * s[3])).astype(np.float32) for n, s in (
        ("a", (32, 16, 3, 3)), ("b", (64, 32, 1, 1)), ("c", (32, 64, 3, 3)), ("e", (40, 128, 1, 1)),
        ("d", (32, 32, 3, 3)))}
    g = Graph("slices")
    x = g.input_f32("data", 16, 12, 10)
    a = g.conv_f32("a", x, f["a"], None, 1, 1, "RELU")
    b = g.conv_f32("b", a, f["b"], None, 1, 0, "SILU")
    d = g.conv_f32("d", a, f["d"], None, 1, 1, "IDENTITY", z=a)
    third = {"all": lambda: g.pooling("p", d, "MAX", 5, 1, 2),
             "some": lambda: g.elemwise_f32("p", "RELU", d), "twice": lambda: a}[form]()
    cat = g.concat("cat", [a, third, b])
    y = g.conv_f32("e", cat, f["e"], None, 1, 0, "SIGMOID")
    z = g.conv_f32("c", b, f["c"], None, 1, 1, "RELU", z=d)
    g.mark_output(y)
    g.mark_output(z)
    src = r.standard_normal((batch, 16, 12, 10)).astype(np.float32)
    conv = lambda v, n, pad, act, **k: oracle.conv_bias_f32(v, f[n], None, 1, pad, act, **k)
    wa = conv(src, "a", 1, "RELU")
    wb = conv(wa, "b", 0, "SILU")
    wd = conv(wa, "d", 1, "IDENTITY", z=wa)
    w3 = {"all": lambda: oracle.pooling_f32(wd, "MAX", 5, 1, 2),
          "some": lambda: np.maximum(wd, 0), "twice": lambda: wa}[form]()
    want = [conv(oracle.concat_f32([wa, w3, wb]), "e", 0, "SIGMOID"), conv(wb, "c", 1, "RELU", z=wd)]
    net = lite.Network(g.compile([batch]))
    for _ in range(3):
        net.set_input("data", src)
        net.forward()
        net.wait()
        for n, w in zip(net.output_names(), want):
            close(net.output(n, dtype=np.float32).reshape(w.shape), w)
    net.close()


# the kernel on fp16 planes (128-column tiles): a last segment of half the elements, channels beside 32, one
# and several tile columns, a resident filter, strides, residual step, pitches; and pixels whose magnitudes
# lie far apart, which share a filter but not a scale
@pytest.mark.parametrize("case", [(9, 32, 128, 12, 11, 3, 1), (2, 36, 72, 30, 30, 1, 1), (2, 96, 200, 17, 19, 3, 2),
                                  (9, 64, 129, 9, 7, 3, 1), (160, 128, 128, 13, 13, 1, 1), (1, 256, 256, 14, 13, 3, 1)],
                         ids=lambda c: "x".join(map(str, c)))
@pytest.mark.parametrize("form", ["SILU", "residual", "far apart"])
def test_fp16_planes_match_64_bits(ops, oracle, case, form):
    n, ic, oc, h, w, k, stride = case
    r = cases.rng_for(f"f32_half_{case}_{form}")
    src = r.standard_normal((n, ic, h, w)).astype(np.float32)
    flt = (r.standard_normal((oc, ic, k, k)) / np.sqrt(ic * k * k)).astype(np.float32)
    if form == "far apart":
        src *= np.exp2(r.integers(-60, 60, (n, 1, h, w))).astype(np.float32)
        flt *= np.exp2(r.integers(-40, 40, (oc, 1, 1, 1))).astype(np.float32)
        flt[0] = 0
    act = "SILU" if form == "SILU" else "IDENTITY"
    bias = None if form == "far apart" else r.standard_normal(oc).astype(np.float32)
    p = ops.conv_f32_param(n, ic, h, w, oc, k, k, stride, k // 2, 1, act)
    x64, f64 = torch.from_numpy(src).double(), torch.from_numpy(flt).double()
    want = torch.nn.functional.conv2d(x64, f64, None if bias is None else torch.from_numpy(bias).double(),
                                      stride=stride, padding=k // 2)
    z = None
    if form == "SILU":
        want = want * torch.sigmoid(want)
    elif form == "residual":
        z = r.standard_normal(tuple(want.permute(0, 2, 3, 1).shape)).astype(np.float32)
        want = want + torch.from_numpy(z).double().permute(0, 3, 1, 2)
    # the terms of one output, in magnitude: every rounding is relative to them. 2^-22 for the split, 2^-24 for
    # each of at most 36 segment sums and the truncations of a segment's chain; in all below 2^-19
    terms = torch.nn.functional.conv2d(x64.abs(), f64.abs(), stride=stride, padding=k // 2)
    old = ops.set_option("f32_half", 2)
    try:
        got = ops.conv_bias_f32_nhwc(p, ops.nchw_to_nhwc_f32(dev(src)), ops.pack_filter_f32(p, dev(flt)),
                                     None if bias is None else dev(bias), z=None if z is None else dev(z),
                                     algo="umma")
    finally:
        ops.set_option("f32_half", old)
    err = (got.cpu().double().permute(0, 3, 1, 2) - want).abs()
    slack = 0 if form == "far apart" else 1e-5 * (1 + want.abs())  # bias, activation and residual in fp32
    assert bool((err <= terms * 2.0 ** -19 + slack).all())
    assert ops.device_status() == 0


# products whose rows the TMA cannot address are copied to a pitch that it can; a result off the vector
# boundary, every remainder of k, both planes' choices
@pytest.mark.parametrize("shape", [(130, 65, 63), (1, 7, 5), (128, 64, 1), (257, 300, 1026), (2100, 260, 130)],
                         ids=lambda c: "x".join(map(str, c)))
@pytest.mark.parametrize("half", [0, 1, 2])
@pytest.mark.parametrize("offset", [0, 1])
def test_fp32_products_of_any_depth(ops, shape, half, offset):
    m, n, k = shape
    r = cases.rng_for(f"f32_any_depth_{shape}")
    room = torch.zeros(m * k + offset, device="cuda")
    a = room[offset:].view(m, k)
    a.copy_(dev(r.standard_normal((m, k)).astype(np.float32)))
    b = dev(r.standard_normal((k, n)).astype(np.float32))
    old = ops.set_option("f32_half", half)
    try:
        got = ops.matmul_f32(a, b)
    finally:
        ops.set_option("f32_half", old)
    want, terms = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    assert bool(((got.double() - want).abs() <= terms * 2.0 ** -19).all())
    assert ops.device_status() == 0


# fp32 3x3 layers from halo patches: images below, at and beside one patch (16 x 8), channels that fill a part of
# a 64-channel block, a 16- and a 32-channel step, one and several tile columns and blocks, results off the
# vector boundary; pixels whose magnitudes lie far apart share a filter but not a scale
@pytest.mark.parametrize("case", [(16, 16, 8, 16, 8), (7, 32, 32, 17, 9), (61, 36, 33, 5, 3), (2, 64, 64, 33, 23),
                                  (2, 132, 72, 15, 16), (300, 128, 128, 1, 1), (1, 196, 257, 20, 20),
                                  (40, 32, 30, 32, 40)], ids=lambda c: "x".join(map(str, c)))
@pytest.mark.parametrize("form", ["SILU", "residual", "far apart"])
def test_fp32_halo_patches_match_64_bits(ops, case, form):
    n, ic, oc, h, w = case
    r = cases.rng_for(f"f32_patch_{case}_{form}")
    src = r.standard_normal((n, ic, h, w)).astype(np.float32)
    flt = (r.standard_normal((oc, ic, 3, 3)) / np.sqrt(ic * 9)).astype(np.float32)
    if form == "far apart":
        src *= np.exp2(r.integers(-60, 60, (n, 1, h, w))).astype(np.float32)
        flt *= np.exp2(r.integers(-40, 40, (oc, 1, 1, 1))).astype(np.float32)
        flt[0] = 0
    bias = None if form == "far apart" else r.standard_normal(oc).astype(np.float32)
    p = ops.conv_f32_param(n, ic, h, w, oc, 3, 3, 1, 1, 1, "SILU" if form == "SILU" else "IDENTITY")
    x64, f64 = torch.from_numpy(src).double(), torch.from_numpy(flt).double()
    want = torch.nn.functional.conv2d(x64, f64, None if bias is None else torch.from_numpy(bias).double(), padding=1)
    z = None
    if form == "SILU":
        want = want * torch.sigmoid(want)
    elif form == "residual":
        z = r.standard_normal(tuple(want.permute(0, 2, 3, 1).shape)).astype(np.float32)
        want = want + torch.from_numpy(z).double().permute(0, 3, 1, 2)
    # as above: 2^-22 for the split, 2^-24 for each of at most 36 segment sums, the truncations of a chain
    terms = torch.nn.functional.conv2d(x64.abs(), f64.abs(), padding=1)
    slack = 0 if form == "far apart" else 1e-5 * (1 + want.abs())  # bias, activation and residual in fp32
    x, f = ops.nchw_to_nhwc_f32(dev(src)), ops.pack_filter_f32(p, dev(flt))
    for mode in (0, 1, 2):
        old = ops.set_option("f32_patch", mode)
        try:
            got = ops.conv_bias_f32_nhwc(p, x, f, None if bias is None else dev(bias),
                                         z=None if z is None else dev(z), algo="umma")
        finally:
            ops.set_option("f32_patch", old)
        err = (got.cpu().double().permute(0, 3, 1, 2) - want).abs()
        assert bool((err <= terms * 2.0 ** -19 + slack).all()), (mode, float((err / terms).max()))
    assert ops.device_status() == 0


# a filter packed under one input, stride and padding and used under another, in every kernel it holds planes for
@pytest.mark.parametrize("case", [(256, 256, 1), (64, 128, 1), (20, 72, 1), (64, 64, 3), (32, 128, 3)],
                         ids=lambda c: "x".join(map(str, c)))
@pytest.mark.parametrize("packed_as", ["point", "stride 2", "no padding", "product"])
def test_packed_filters_serve_every_input(ops, case, packed_as):
    import ctypes as C
    from megcc_b200._lib import check, lib
    ic, oc, k = case
    if packed_as == "product" and k != 1:
        pytest.skip("a product's B is a 1x1 filter")
    r = cases.rng_for(f"f32_packed_{case}")
    flt = dev((r.standard_normal((oc, ic, k, k)) / np.sqrt(ic * k * k)).astype(np.float32))
    if packed_as == "product":
        b = flt.view(oc, ic).t().contiguous()
        packed = torch.empty(lib().mb200_matmul_f32_packed_b_bytes(ic, oc) // 4, device="cuda")
        check(lib().mb200_matmul_f32_pack_b(ic, oc, C.c_void_p(b.data_ptr()), C.c_void_p(packed.data_ptr()),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    else:
        e, stride, pad = (1, 1, k // 2) if packed_as == "point" else (9, 2, k // 2) if packed_as == "stride 2" else (9, 1, 0)
        packed = ops.pack_filter_f32(ops.conv_f32_param(1, ic, e, e, oc, k, k, stride, pad), flt)
    for n, h, stride, pad in ((1, 6, 1, k // 2), (32, 20, 1, k // 2), (32, 20, 2, k // 2), (8, 20, 1, 0)):
        x = dev(r.standard_normal((n, ic, h, h)).astype(np.float32))
        p = ops.conv_f32_param(n, ic, h, h, oc, k, k, stride, pad)
        want = torch.nn.functional.conv2d(x.double(), flt.double(), stride=stride, padding=pad)
        terms = torch.nn.functional.conv2d(x.double().abs(), flt.double().abs(), stride=stride, padding=pad)
        for half, patch in ((1, 1), (2, 0), (0, 2), (0, 0)):
            old = ops.set_option("f32_half", half), ops.set_option("f32_patch", patch)
            try:
                got = ops.conv_bias_f32_nhwc(p, ops.nchw_to_nhwc_f32(x), packed)
            finally:
                ops.set_option("f32_half", old[0]), ops.set_option("f32_patch", old[1])
            # (2^-22 for the split, 2^-24 for each of at most 36 segment sums, the truncations of a chain)
            assert bool(((got.double().permute(0, 3, 1, 2) - want).abs() <= terms * 2.0 ** -19).all()), (n, h, stride, pad, half, patch)
    assert ops.device_status() == 0


# Operands that lie far apart along K, the one axis with no scale of its own: a channel 2^p times the others
# under weights 2^-p times the others (every term of a sum then has the same size), and the other way round; a
# huge channel under zero weights, for all results or for all but one; zeros on both sides beside values too
# small for the planes; one weight too small; all of it at the ends of fp32's range. The kernels on fp16 planes,
# tiles of one and several steps and columns
def far_apart(form, src, flt):  # src [n][k]..., flt [oc][k]...
    k = src.shape[1]
    if form.startswith("2^"):
        p = float(form[2:])
        src[:, k // 2] *= np.float32(2.0 ** p)
        flt[:, k // 2] *= np.float32(2.0 ** -p)
    elif form.startswith("sentinel"):
        src[:, k // 3] = -1e30
        flt[:, k // 3] = 0
        if form == "sentinel but one":
            flt[1, k // 3] = 1e-3
    elif form == "zeros":
        np.maximum(src, 0, out=src)
        src[:, ::3] *= np.float32(2.0 ** -35)
        flt[:, 1::3] = 0
        flt[::2, 2::3] = 0
    elif form == "one weight":
        src[:, k // 2] *= np.float32(2.0 ** 40)
        flt[flt.shape[0] // 2, k // 2] *= np.float32(2.0 ** -40)
    elif form == "large":
        src *= np.float32(2.0 ** 112)
        flt *= np.float32(2.0 ** -70)
    elif form == "small":
        src *= np.float32(2.0 ** -100)
        flt *= np.float32(2.0 ** 70)


FAR_APART = [f"2^{p}" for p in (14, 18, 24, 28, 29, 31, 33, 40, -18, -28, -30, -40)] + [
    "sentinel", "sentinel but one", "zeros", "one weight", "large", "small"]


@pytest.mark.parametrize("case", [("f32_patch", 16, 16, 8, 16, 8, 3, 1), ("f32_patch", 2, 64, 64, 33, 23, 3, 1),
                                  ("f32_patch", 1, 196, 257, 20, 20, 3, 1), ("f32_patch", 60, 128, 128, 33, 40, 3, 1),
                                  ("f32_half", 9, 64, 129, 9, 7, 3, 1), ("f32_half", 2, 96, 200, 17, 19, 3, 2),
                                  ("f32_half", 160, 128, 128, 13, 13, 1, 1)], ids=lambda c: "x".join(map(str, c)))
def test_operands_far_apart_along_k(ops, case):
    option, n, ic, oc, h, w, k, stride = case
    for form in FAR_APART:
        r = cases.rng_for(f"f32_along_k_{case}")
        src = r.standard_normal((n, ic, h, w)).astype(np.float32)
        flt = (r.standard_normal((oc, ic, k, k)) / np.sqrt(ic * k * k)).astype(np.float32)
        far_apart(form, src, flt)
        x, f = dev(src), dev(flt)
        want = torch.nn.functional.conv2d(x.double(), f.double(), stride=stride, padding=k // 2)
        terms = torch.nn.functional.conv2d(x.double().abs(), f.double().abs(), stride=stride, padding=k // 2)
        z = dev(r.standard_normal((n, h // stride + h % stride, w // stride + w % stride, oc)).astype(np.float32))
        if form in ("large", "small"):
            z.zero_()
        p = ops.conv_f32_param(n, ic, h, w, oc, k, k, stride, k // 2)
        old = ops.set_option(option, 2), ops.set_option("f32_patch", 2 if option == "f32_patch" else 0)
        try:
            got = ops.conv_bias_f32_nhwc(p, ops.nchw_to_nhwc_f32(x), ops.pack_filter_f32(p, f), z=z, algo="umma")
        finally:
            ops.set_option("f32_patch", old[1]), ops.set_option(option, old[0])
        z = z.double().permute(0, 3, 1, 2)
        err = (got.double().permute(0, 3, 1, 2) - (want + z)).abs()
        # 2^-22 for the split, at most 2^-20 for values too small for the planes, 2^-24 for each of at most 36 segment
        # sums and for the truncations of a chain; and the rounding of the sum with z
        bound = terms * 2.0 ** -19 + (want.abs() + z.abs()) * 2.0 ** -24
        assert bool((err <= bound).all()), (form, float((err / bound).max()))
    assert ops.device_status() == 0


@pytest.mark.parametrize("shape", [(257, 300, 1026), (400, 260, 64), (130, 129, 130)], ids=lambda c: "x".join(map(str, c)))
def test_products_of_operands_far_apart_along_k(ops, shape):
    m, n, k = shape
    for form in FAR_APART:
        r = cases.rng_for(f"f32_product_along_k_{shape}")
        a, bt = r.standard_normal((m, k)).astype(np.float32), r.standard_normal((n, k)).astype(np.float32)
        far_apart(form, a, bt)
        a, b = dev(a), dev(bt.T)
        want, terms = a.double() @ b.double(), a.double().abs() @ b.double().abs()
        for half in (2, 0):
            old = ops.set_option("f32_half", half)
            try:
                got = ops.matmul_f32(a, b)
            finally:
                ops.set_option("f32_half", old)
            err = (got.double() - want).abs()
            assert bool((err <= terms * 2.0 ** -19).all()), (form, half, float((err / terms).max()) * 2 ** 19)
    assert ops.device_status() == 0


# a residual in the result's own place, which a tile that is stored twice must not see twice
@pytest.mark.parametrize("case", [(2, 64, 64, 33, 23, 3), (160, 128, 128, 13, 13, 1)], ids=lambda c: "x".join(map(str, c)))
def test_residual_in_the_results_place(ops, case):
    n, ic, oc, h, w, k = case
    r = cases.rng_for(f"f32_in_place_{case}")
    src = r.standard_normal((n, ic, h, w)).astype(np.float32)
    flt = (r.standard_normal((oc, ic, k, k)) / np.sqrt(ic * k * k)).astype(np.float32)
    far_apart("sentinel but one", src, flt)
    x, f = dev(src), dev(flt)
    out = dev(r.standard_normal((n, h, w, oc)).astype(np.float32))
    z = out.double().permute(0, 3, 1, 2)
    want = torch.nn.functional.conv2d(x.double(), f.double(), padding=k // 2) + z
    terms = torch.nn.functional.conv2d(x.double().abs(), f.double().abs(), padding=k // 2)
    old = ops.set_option("f32_half", 2), ops.set_option("f32_patch", 2)
    try:
        p = ops.conv_f32_param(n, ic, h, w, oc, k, k, 1, k // 2)
        ops.conv_bias_f32_nhwc(p, ops.nchw_to_nhwc_f32(x), ops.pack_filter_f32(p, f), z=out, dst=out, algo="umma")
    finally:
        ops.set_option("f32_half", old[0]), ops.set_option("f32_patch", old[1])
    err = (out.double().permute(0, 3, 1, 2) - want).abs()
    assert bool((err <= terms * 2.0 ** -19 + (want.abs() + z.abs()) * 2.0 ** -24).all())
    assert ops.device_status() == 0


# a network whose filters hold a dead input channel (weights that have decayed to 1e-25 beside ordinary ones),
# with its activations large enough to matter: known as the weights are packed
def test_networks_with_weights_far_apart(ops, oracle):
    from megcc_b200 import lite
    from megcc_b200.compiler import Graph
    r = cases.rng_for("f32_dead_channel")
    shapes = {"a": (128, 64, 1, 1), "b": (64, 128, 3, 3), "c": (32, 64, 3, 3)}
    f = {n: (r.standard_normal(s) / np.sqrt(s[1] * s[2] * s[3])).astype(np.float32) for n, s in shapes.items()}
    f["a"][:, 3] *= np.float32(1e-25)
    f["b"][:, 7] *= np.float32(1e-25)
    src = r.standard_normal((64, 64, 12, 12)).astype(np.float32)
    src[:, 3] *= np.float32(1e24)
    g = Graph("dead")
    x = g.input_f32("data", 64, 12, 12)
    a = g.conv_f32("a", x, f["a"], None, 1, 0, "RELU")
    b = g.conv_f32("b", a, f["b"], None, 1, 1, "SILU")
    g.mark_output(g.conv_f32("c", b, f["c"], None, 1, 1, "IDENTITY"))
    conv = lambda v, n, pad, act: oracle.conv_bias_f32(v, f[n], None, 1, pad, act)
    want = conv(conv(conv(src, "a", 0, "RELU"), "b", 1, "SILU"), "c", 1, "IDENTITY")
    old = ops.set_option("f32_half", 2), ops.set_option("f32_patch", 2)
    try:
        net = lite.Network(g.compile([64]))
        net.set_input("data", src)
        net.forward()
        net.wait()
        close(net.output(net.output_names()[0], dtype=np.float32).reshape(want.shape), want)
        net.close()
    finally:
        ops.set_option("f32_half", old[0]), ops.set_option("f32_patch", old[1])
    assert ops.device_status() == 0


# Halo patches only where they gain more than a kernel of its own costs among others
@pytest.mark.parametrize("n,ic,oc,h,patches", [
    (1, 16, 32, 128, False), (1, 16, 32, 208, False), (1, 32, 32, 120, False), (1, 64, 32, 136, False),
    (1, 64, 64, 52, False), (4, 16, 64, 320, False), (1, 32, 32, 320, True), (32, 64, 64, 80, True),
    (8, 16, 32, 320, True), (1, 128, 128, 112, True)])
def test_layers_that_take_halo_patches(ops, capfd, n, ic, oc, h, patches):
    src, flt = torch.zeros((n, h, h, ic), device="cuda"), torch.zeros((oc, ic, 3, 3), device="cuda")
    p = ops.conv_f32_param(n, ic, h, h, oc, 3, 3, 1, 1)
    packed = ops.pack_filter_f32(p, flt)
    old = ops.set_option("debug", 1)
    try:
        ops.conv_bias_f32_nhwc(p, src, packed)
    finally:
        ops.set_option("debug", old)
    assert ("conv_f32_patch" in capfd.readouterr().err) == patches
