"""GPU parity of the dispatch branches taken by size: im2col-mode convolutions, streamed fully connected layers, the fused
pool and bias backward pass, top-k and softmax at their borders, and uploads and downloads longer than the page-locked ring."""
import os

import numpy as np
import pytest

from conftest import rel_l2
from gpu_util import TOL_3X, TOL_TF32, conv_case, variants_used

pytestmark = pytest.mark.gpu


def check(got, ref, tol):
    for k in ("y", "dw", "db", "dx"):
        if ref[k] is None:
            continue
        err = rel_l2(got[k].ravel(), ref[k].ravel())
        assert np.isfinite(got[k]).all() and err <= tol, "%s: relative L2 error %.3e > %.1e" % (k, err, tol)


# (N, C, H, W, K, size, stride, pad, activation, groups, dilation)
IM2COL = [
    (9, 32, 13, 13, 48, 3, 1, 1, 1, 1, 1),      # tiles across rows and images, a last tile that is partly empty
    (5, 64, 27, 27, 160, 5, 1, 2, 2, 1, 1),     # filters that do not divide the widest tile
    (9, 64, 24, 24, 64, 3, 2, 1, 0, 1, 1),      # stride: four residue classes backwards
    (6, 32, 29, 23, 40, 3, 3, 1, 1, 1, 1),      # stride 3 (more classes than a launch holds), odd map
    (4, 32, 25, 25, 64, 3, 1, 1, 2, 1, 2),      # dilation
    (8, 64, 15, 17, 64, 3, 1, 1, 1, 2, 1),      # channel groups
    (20, 48, 14, 14, 52, 3, 1, 0, 1, 1, 1),     # channels and filters that are no multiple of 32
    (16, 256, 9, 9, 256, 3, 1, 1, 0, 1, 1),     # few tiles, long K: the last round is split along K
    (7, 96, 11, 11, 300, 1, 1, 0, 2, 1, 1),     # 1x1
]

# in TF32 these belong to other kernels: long K loops of few tiles to clusters, a tensor of less than 128 KB to ragged tiles
TILED = {(0, "dgrad"): "conv_dgrad_tma.cl", (7, "dgrad"): "conv_dgrad_tma.cl", (8, "fprop"): "conv_fprop_tma.ragged"}


@pytest.mark.parametrize("math", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", IM2COL)
def test_conv_im2col(aet, ctx, oracle, oracle64, shape, math):
    N, C, H, W, K, size, stride, pad, act, groups, dilation = shape
    x3 = math == "3xtf32"
    ctx.set_math(aet.MATH_3XTF32 if x3 else aet.MATH_TF32)
    try:
        ctx.profile(1)
        got, ref = conv_case(aet, ctx, oracle64 if x3 else oracle, N, C, H, W, K, size, stride, pad, act, seed=900 + K, groups=groups,
                             dilation=dilation)
        names = variants_used(ctx)
    finally:
        ctx.profile(0)
        ctx.set_math(aet.MATH_TF32)
    check(got, ref, TOL_3X if x3 else TOL_TF32)
    for kind in ("fprop", "dgrad", "wgrad"):
        want = "conv_%s_tma.i2c_" % kind
        if kind == "dgrad" and stride > 2:
            want = "conv_dgrad_gather"
        elif not x3:
            want = TILED.get((IM2COL.index(shape), kind), want)
        assert any(n.startswith(want) and (not n.startswith("conv_%s_tma.i2c_" % kind) or ("_x3" in n) == x3) for n in names), (want, names)


@pytest.mark.parametrize("shape", [
    (17, 36, 28, 19, 40, 5, 1, 2),      # 289 slabs of pixels: the gather kernel sums five in an accumulator
    (33, 72, 29, 30, 64, 1, 1, 0),
    (33, 48, 17, 10, 4, 5, 1, 2),       # four filters
    (64, 64, 16, 16, 128, 3, 1, 1),     # filters by two, a pair of CTAs
])
def test_weight_gradient_in_3xtf32_sums_no_more_at_a_time_than_the_gather_kernel(aet, ctx, shape):
    """Both kernels against float64.  The error is that of the tensor core's running sums, so it grows with what one
    accumulator takes; over the 500 and more weights here its norm varies by a few per cent."""
    import torch
    n, c, h, w, k, size, stride, pad = shape
    rng = np.random.default_rng(h * w)
    x = rng.standard_normal((n, c, h, w)).astype(np.float32)
    dy = rng.standard_normal((n, k, (h + 2 * pad - size) // stride + 1, (w + 2 * pad - size) // stride + 1)).astype(np.float32)
    ref = torch.nn.grad.conv2d_weight(torch.from_numpy(x).double(), (k, c, size, size), torch.from_numpy(dy).double(), stride, pad).numpy()
    err = {}
    ctx.set_math(aet.MATH_3XTF32)
    try:
        for gather in (0, 1):
            ctx.set_option("gather_only", gather)
            layer = aet.ConvolutionalLayer(ctx, n, h, w, c, k, size, stride, stride, pad, aet.LINEAR, 0, 1)
            xin = aet.Tensor(ctx, n, c, h, w)
            xin.write(x)
            layer.write(aet.P_DELTA, dy)
            ctx.profile(1)
            layer.backward(aet.make_state(input=xin, train=1))
            assert any(v.startswith("conv_wgrad_gather" if gather else "conv_wgrad_tma.i2c_") for v in variants_used(ctx))
            ctx.profile(0)
            err[gather] = rel_l2(layer.read(aet.P_WEIGHT_UPDATES), ref)
            layer.close()
            xin.close()
    finally:
        ctx.profile(0)
        ctx.set_option("gather_only", 0)
        ctx.set_math(aet.MATH_TF32)
    assert err[0] <= 1.1 * err[1] <= TOL_3X, err


@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("inputs,filters", [(64, 10), (4100, 37), (9216, 512)])
def test_fully_connected_of_few_images(aet, ctx, oracle, batch, inputs, filters):
    got, ref = conv_case(aet, ctx, oracle, batch, inputs, 1, 1, filters, 1, 1, 0, 1, seed=40 + batch)
    check(got, ref, TOL_TF32)


POOL_CFG = """[net]
batch=%d
width=%d
height=%d
channels=3
learning_rate=0.01
[convolutional]
filters=%d
size=3
pad=1
activation=%s
[maxpool]
size=%d
stride=2
padding=%d
[convolutional]
filters=10
size=1
activation=linear
[avgpool]
[softmax]
"""


@pytest.mark.parametrize("case", [(3, 11, 13, 8, "relu", 3, 0), (4, 12, 10, 20, "leaky", 2, 0), (2, 13, 13, 12, "leaky", 2, 1),
                                  (2, 9, 9, 8, "linear", 3, 1), (1, 8, 8, 1100, "relu", 3, 0), (2, 55, 55, 96, "logistic", 3, 0),
                                  (2, 9, 9, 8, "leaky", 3, 2)])
def test_pool_backward_with_bias_backward(aet, ctx, case):
    """The joined pass against the two passes it replaces: same windows in the same order, so the delta is the same bit for
    bit; the bias and weight sums are grouped differently (FP32, up to 2 * 55 * 55 terms a channel)."""
    batch, classes = case[0], 10
    joined = case[6] // 2 == 0   # a pool with an offset keeps the two passes
    out, launched = [], []
    for fuse in (1, 0):
        ctx.set_option("fuse", fuse)
        ctx.set_option("linear_head", 0)   # the heads differ in rounding
        try:
            net = aet.NNetwork(ctx, cfg_text=POOL_CFG % case, train=1)
        finally:
            ctx.set_option("fuse", 1)
            ctx.set_option("linear_head", 1)
        rng = np.random.default_rng(7)
        net.use_graph(False)
        net.input.write(rng.random(net.input_shape, dtype=np.float32))
        net.truth.write(np.eye(classes, dtype=np.float32)[rng.integers(0, classes, batch)])
        st = aet.make_state(input=net.input, truth=net.truth, train=1)
        net.forward(st)
        ctx.profile(1)
        net.backward(st)
        launched.append({n.split("#")[0] for n in variants_used(ctx)})
        ctx.profile(0)
        ctx.check()
        out.append([net.layer(0).read(p) for p in (aet.P_DELTA, aet.P_BIAS_UPDATES, aet.P_WEIGHT_UPDATES)])
        net.close()
    assert ("pool_bias_act_bwd" in launched[0]) == joined and "pool_bias_act_bwd" not in launched[1], launched
    assert out[1][0].any() and np.array_equal(out[0][0], out[1][0])
    for fused, plain in zip(out[0][1:], out[1][1:]):
        assert rel_l2(fused, plain) <= 1e-5


TOPK_CFG = """[net]
batch=4
width=1
height=1
channels=%d
learning_rate=0.01
[convolutional]
filters=%d
size=1
activation=linear
[softmax]
"""


@pytest.mark.parametrize("classes", [5, 1000, 1024, 1025])
@pytest.mark.parametrize("ties", [False, True])
def test_top_k_at_the_register_limit(aet, ctx, oracle, classes, ties):
    """Distinct scores take the register path, repeated ones and more than 1024 the loop; both follow the oracle's order."""
    net = aet.NNetwork(ctx, cfg_text=TOPK_CFG % (8, classes), train=0)
    rng = np.random.default_rng(classes)
    w = rng.standard_normal((classes, 8, 1, 1)).astype(np.float32)
    if ties:
        w[classes // 2:] = w[:classes - classes // 2]
    net.layer(0).write(aet.P_WEIGHTS, w)
    x = rng.random((4, 8, 1, 1), dtype=np.float32)
    k = min(5, classes)
    idx = net.predict_topk(x, k)
    score = net.predict(x).reshape(4, classes)
    for i in range(4):
        assert np.array_equal(idx[i], oracle.top_k(score[i], k)), i
    net.close()


@pytest.mark.parametrize("shape", [(1, 3, 5, 7), (3, 3, 227, 227), (50, 3, 181, 167), (40, 64, 33, 31), (9, 100, 64, 64), (300, 1, 61, 61)])
def test_transfers_through_the_ring(aet, ctx, shape):
    """Exact round trips at sizes below, at and above the pieces that an upload or download goes in."""
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal(shape).astype(np.float32)
    t = aet.Tensor(ctx, *shape)
    for _ in range(2):
        t.write(x)
        assert np.array_equal(t.read(), x)
        x = x[::-1].copy()
    t.close()


def test_predictions_captured_and_plain_agree(aet, ctx, oracle):
    """Captured passes give what plain ones give, call after call and after weights were written; the classifier convolution's
    output, which the linear head leaves out, is there when its tensor is read."""
    batch = 16
    net = aet.NNetwork(ctx, cfg_path=os.path.join(aet.CFG_DIR, "cifar_small.cfg"), train=0, batch=batch)
    rng = np.random.default_rng(3)
    x = rng.random((5, batch, 3, 32, 32), dtype=np.float32)
    net.use_graph(False)
    want = [net.predict(b).copy() for b in x]
    net.use_graph(True)
    for _ in range(3):
        for b, y in zip(x, want):
            assert np.array_equal(net.predict(b), y)
    head = net.layer(net.layer_count - 3)
    logits = head.output.read().reshape(batch, 10, -1).mean(2)
    p = np.exp(logits - logits.max(1, keepdims=True))
    assert rel_l2(p / p.sum(1, keepdims=True), want[-1].reshape(batch, 10)) <= TOL_TF32
    net.layer(0).write(aet.P_WEIGHTS, net.layer(0).read(aet.P_WEIGHTS) * 1.5)
    changed = net.predict(x[0]).copy()
    net.use_graph(False)
    assert np.array_equal(net.predict(x[0]), changed)
    net.close()


@pytest.mark.parametrize("shape", [
    (1, 64, 16, 16, 128, 3, 1, 1, 2),      # eight parts of 18 slabs: the last one is shorter
    (1, 128, 8, 8, 250, 3, 1, 1, 1),       # half of the pixel tile and part of the last filter tile do not exist
    (1, 384, 13, 13, 256, 3, 1, 1, 1),     # ragged map, long K
    (2, 96, 27, 27, 64, 5, 1, 2, 0),       # seven ragged tiles per image
    (5, 128, 8, 8, 128, 3, 1, 1, 2),       # an odd number of images
    (13, 128, 8, 8, 128, 3, 1, 1, 0),      # four parts
])
def test_conv_of_few_images_shares_k_in_clusters(aet, ctx, oracle, shape):
    ctx.profile(1)
    try:
        got, ref = conv_case(aet, ctx, oracle, *shape, seed=970 + shape[1])
        names = {n.split("#")[0] for n in variants_used(ctx)}
    finally:
        ctx.profile(0)
    assert {"conv_fprop_tma.cl", "conv_dgrad_tma.cl"} <= names, names
    check(got, ref, TOL_TF32)


@pytest.mark.parametrize("shape,names_of", [
    ((43, 96, 27, 27, 64, 5, 1, 2, 2), ("fprop_tma.i2c_n64x2", "dgrad_tma.i2c_n96x2")),     # the last tile's second half is empty
    ((63, 32, 40, 40, 128, 3, 2, 1, 0), ("dgrad_tma.i2c_n32x2",)),                          # four residue classes, each with such a tile
    ((18, 96, 23, 23, 48, 7, 1, 3, 1), ("fprop_tma.i2c_n64x2",)),                           # split along K, ragged filters
    ((18, 96, 23, 23, 72, 7, 1, 3, 0), ("dgrad_tma.i2c_n96x2",)),                           # split along K
])
def test_two_pixel_tiles_per_cta(aet, ctx, oracle, shape, names_of):
    ctx.set_math(aet.MATH_TF32)
    ctx.profile(1)
    try:
        got, ref = conv_case(aet, ctx, oracle, *shape, seed=960 + shape[1], threads=True)
        names = variants_used(ctx)
    finally:
        ctx.profile(0)
    check(got, ref, TOL_TF32)
    for want in names_of:
        assert any(n.startswith("conv_" + want) for n in names), (want, names)


@pytest.mark.parametrize("shape", [(17, 64, 28, 26, 24, 3, 1, 0, 2), (33, 96, 19, 19, 100, 3, 1, 2, 0), (33, 96, 47, 25, 128, 4, 2, 2, 1)])
def test_layers_of_one_round_keep_one_pixel_tile_per_cta(aet, ctx, oracle, shape):
    """Where the chip is not full, two tiles per CTA and their split sums took up to 1.6 times as long."""
    ctx.set_math(aet.MATH_TF32)
    ctx.profile(1)
    try:
        got, ref = conv_case(aet, ctx, oracle, *shape, seed=970 + shape[1], threads=True)
        names = variants_used(ctx)
    finally:
        ctx.profile(0)
    check(got, ref, TOL_TF32)
    assert any("_tma.i2c_" in n for n in names) and not any(n.endswith("x2") for n in names), names


def test_batch_statistics_of_two_pixel_tiles_per_cta(aet, ctx):
    """The statistics that come out of such tiles' epilogue, by way of the output they normalise: against the gather kernel."""
    n, c, h, k = 43, 96, 27, 60
    rng = np.random.default_rng(5)
    x = rng.standard_normal((n, c, h, h)).astype(np.float32)
    w = rng.standard_normal((k, c, 5, 5)).astype(np.float32) * 0.03
    out = {}
    for gather in (0, 1):
        ctx.set_option("gather_only", gather)
        try:
            layer = aet.ConvolutionalLayer(ctx, n, h, h, c, k, 5, 1, 1, 2, aet.LINEAR, 1, 1)
            xin = aet.Tensor(ctx, n, c, h, h)
            xin.write(x)
            layer.write(aet.P_WEIGHTS, w)
            ctx.profile(1)
            layer.forward(aet.make_state(input=xin, train=1))
            assert gather or any(v.startswith("conv_fprop_tma.i2c_n64x2") for v in variants_used(ctx))
            out[gather] = layer.read(aet.P_OUTPUT), layer.read(aet.P_ROLLING_MEAN), layer.read(aet.P_ROLLING_VARIANCE)
            layer.close()
            xin.close()
        finally:
            ctx.profile(0)
            ctx.set_option("gather_only", 0)
    for a, b in zip(out[0], out[1]):
        assert np.isfinite(a).all() and rel_l2(a, b) <= TOL_TF32
