"""Training steps whose weight gradients apply the update in their epilogue, against the same step made call by call."""
import numpy as np
import pytest

from conftest import rel_l2
from gpu_util import device_memory_taken, variants_used

pytestmark = pytest.mark.gpu

HEAD = "[net]\nbatch=%d\nwidth=%d\nheight=%d\nchannels=%d\nlearning_rate=0.05\nmomentum=0.9\ndecay=0.0005\npolicy=constant\n\n"
CONV = "[convolutional]\nfilters=%d\nsize=%d\nstride=1\npad=%d\nactivation=%s\n%s\n"


def two_nets(aet, ctx, text, batch):
    rng = np.random.default_rng(batch)
    nets = [aet.NNetwork(ctx, cfg_text=text, train=1, batch=batch) for _ in range(2)]
    x = rng.random(nets[0].input_shape, np.float32)
    t = np.eye(nets[0].outputs, dtype=np.float32)[rng.integers(0, nets[0].outputs, nets[0].batch)]
    for n in nets:
        n.use_graph(False)
        n.input.write(x)
        n.truth.write(t)
    return nets


def step_by_calls(aet, net):
    st = aet.make_state(input=net.input, truth=net.truth, train=1)
    net.forward(st)
    net.backward(aet.make_state(input=net.input, truth=net.truth, train=1))
    net.update()


def compare(aet, fused, plain, tol):
    for i in range(fused.layer_count):
        a, b = fused.layer(i), plain.layer(i)
        for which in (aet.P_WEIGHTS, aet.P_WEIGHT_UPDATES, aet.P_BIASES, aet.P_BIAS_UPDATES):
            if a.param_count(which):
                u, v = a.read(which), b.read(which)
                assert np.isfinite(u).all() and rel_l2(u, v) <= tol, (i, which, rel_l2(u, v))


def copy_parameters(aet, src, dst):
    for i in range(src.layer_count):
        for which in (aet.P_WEIGHTS, aet.P_WEIGHT_UPDATES, aet.P_BIASES, aet.P_BIAS_UPDATES):
            if src.layer(i).param_count(which):
                dst.layer(i).write(which, src.layer(i).read(which))


# (batch, map, channels, filters): one slab and eight of them, filters beside the tiles' widths, channels that end inside a block, and
# (last) five tiles of 192 filters for each CTA, the last one of which has 68
@pytest.mark.parametrize("shape", [(8, 8, 256, 385), (40, 7, 132, 1100), (128, 8, 64, 1540), (256, 6, 128, 1400), (16, 8, 64, 4100)])
@pytest.mark.parametrize("graph", [False, True])
def test_fully_connected_layers_update_themselves(aet, ctx, shape, graph):
    """Same products in the same precision; the sums of a split gradient and of one that is not differ by rounding, a few
    times 1e-7 of a gradient.  Every step starts from the same state on both sides: a value at an activation's kink, or one at
    the edge between two TF32 values, would carry such a difference on as 1e-3."""
    batch, side, channels, filters = shape
    text = (HEAD % (batch, side, side, 32) + CONV % (channels, 3, 1, "leaky", "") + CONV % (filters, side, 0, "relu", "learning_rate=0.5\n") +
            CONV % (10, 1, 0, "linear", "") + "[softmax]\n")
    fused, plain = two_nets(aet, ctx, text, batch)
    try:
        ctx.profile(0 if graph else 1)
        fused.use_graph(graph)
        for _ in range(3):
            fused.train_device()
            step_by_calls(aet, plain)
            compare(aet, fused, plain, 2e-5)
            copy_parameters(aet, fused, plain)
        if not graph:
            assert any("_sgd" in n for n in variants_used(ctx)), variants_used(ctx)
    finally:
        ctx.profile(0)
        fused.close()
        plain.close()


def self_updates(ctx):
    return sum(r["launches"] for r in ctx.profile_read() if "_sgd" in r["name"])


WIDE = HEAD % (32, 1, 1, 2512) + CONV % (2512, 1, 0, "relu", "") + CONV % (10, 1, 0, "linear", "") + "[softmax]\n"   # 6.3 million weights


def test_a_captured_step_lets_its_layers_update_themselves(aet, ctx):
    """Such a layer's gradient is never in the arena: a mark there is still there after the step.  The separate kernels write the
    gradient over it and the update clears it."""
    import ctypes
    import torch
    torch.cuda.init()
    cudart = ctypes.CDLL("libcudart.so.12")
    net, spare = two_nets(aet, ctx, WIDE, 32)
    try:
        arena, count = net.grad_arena()
        mark, seen = ctypes.c_float(7.0), ctypes.c_float(0.0)
        middle = ctypes.c_void_p(arena + 4 * (count // 2))   # the wide layer takes nearly all of the arena

        def copy(dst, src, kind):
            ctx.synchronize()
            assert cudart.cudaMemcpy(dst, src, ctypes.c_size_t(4), ctypes.c_int(kind)) == 0

        net.use_graph(True)
        for expected in (7.0, 7.0, 0.0):
            for _ in range(3):
                net.train_device()
            copy(middle, ctypes.byref(mark), 1)
            if expected == 0.0:   # a backward pass by hand: the arena no longer counts as empty
                net.backward(aet.make_state(input=net.input, truth=net.truth, train=1))
            net.train_device()
            copy(ctypes.byref(seen), middle, 2)
            assert seen.value == expected
            copy(middle, ctypes.byref(ctypes.c_float(0.0)), 1)
    finally:
        net.close()
        spare.close()


@pytest.mark.parametrize("guard", ["adam", "subdivisions", "3xtf32", "batch", "small", "communicator", "left over"])
def test_layers_that_must_not_update_themselves(aet, ctx, guard):
    """Where somebody else has a part in the gradient or the update, or the rule's range ends, the separate kernels run."""
    batch, text = 32, WIDE
    if guard == "adam":
        text = WIDE.replace("policy=constant", "policy=constant\nadam=1")
    if guard == "batch":
        batch = 257
    if guard == "small":
        text = WIDE.replace("filters=2512", "filters=2400")
    if guard == "subdivisions":
        batch, text = 0, WIDE.replace("batch=32", "batch=64\nsubdivisions=2")
    if guard == "3xtf32":
        ctx.set_math(aet.MATH_3XTF32)
    net, plain = two_nets(aet, ctx, text, batch)
    try:
        if guard == "communicator":
            net.comm_init(aet.comm_unique_id(), 0, 1)
        if guard == "left over":
            state = aet.make_state(input=net.input, truth=net.truth, train=1)
            for n in (net, plain):
                n.forward(state)
                n.backward(state)
        ctx.profile(1)
        for _ in range(2 if guard == "subdivisions" else 1):
            net.train_device()
        assert self_updates(ctx) == 0, variants_used(ctx)
        ctx.profile(0)
        if guard == "adam":   # divides by the gradient's size: the rounding of one that is nearly zero becomes a whole step
            return
        if guard == "subdivisions":
            state = aet.make_state(input=plain.input, truth=plain.truth, train=1)
            plain.forward(state)
            plain.backward(state)
        step_by_calls(aet, plain)
        compare(aet, net, plain, 2e-5)
    finally:
        ctx.profile(0)
        ctx.set_math(aet.MATH_TF32)
        net.close()
        plain.close()


def test_a_ninth_wide_layer_is_updated_with_the_others(aet, ctx):
    text = HEAD % (16, 1, 1, 2512) + 9 * (CONV % (2512, 1, 0, "leaky", "")) + CONV % (10, 1, 0, "linear", "") + "[softmax]\n"
    fused, plain = two_nets(aet, ctx, text, 16)
    try:
        ctx.profile(1)
        fused.train_device()
        assert self_updates(ctx) == 8, variants_used(ctx)
        ctx.profile(0)
        step_by_calls(aet, plain)
        compare(aet, fused, plain, 2e-5)
    finally:
        ctx.profile(0)
        fused.close()
        plain.close()


# 4096 x 1540: the last eight filters of the last tile are four
@pytest.mark.parametrize("held", [False, True])
def test_self_updating_layers_scrub_and_hold_still(aet, ctx, held):
    """Non-finite weights and pending updates are replaced as by the update kernel, and a layer that is not updated yet collects
    its gradient, unscaled.  (The other side has a communicator of one rank: the same training step with the separate kernels.)"""
    text = (HEAD % (16, 8, 8, 32) + CONV % (64, 3, 1, "leaky", "") + CONV % (1540, 8, 0, "relu", "dont_update=1\n" if held else "") + CONV % (10, 1, 0, "linear", "") +
            "[softmax]\n")
    fused, plain = two_nets(aet, ctx, text, 16)
    try:
        plain.comm_init(aet.comm_unique_id(), 0, 1)
        spots = [(0, 0, 0), (700, 5, 63), (1539, 63, 17)]   # filter, tap, channel: the first, a later tile's, one of the last four filters'
        host = [k * 4096 + c * 64 + tap for k, tap, c in spots]
        device = [k * 4096 + tap * 64 + c for k, tap, c in spots]
        if not held:
            for n in (fused, plain):
                w, u = n.layer(1).read(aet.P_WEIGHTS), n.layer(1).read(aet.P_WEIGHT_UPDATES)
                w[host] = np.nan, np.inf, -np.inf
                u[[3, 1017, len(u) - 1]] = np.nan, np.inf, -np.inf
                n.layer(1).write(aet.P_WEIGHTS, w)
                n.layer(1).write(aet.P_WEIGHT_UPDATES, u)
        start = fused.layer(1).read(aet.P_WEIGHTS)
        ctx.profile(1)
        for step in range(2):
            for n in (fused, plain):
                n.train_device()
                assert self_updates(ctx) == step + 1
                if not held:   # the biases stay what the first step has made of them
                    with pytest.raises(aet.AetError, match="non-finite"):
                        ctx.check()
            ctx.check()
            w, u = [[n.layer(1).read(which) for n in (fused, plain)] for which in (aet.P_WEIGHTS, aet.P_WEIGHT_UPDATES)]
            assert np.isfinite(w[0]).all() and np.isfinite(u[0]).all()
            assert rel_l2(*w) <= 2e-5 and rel_l2(*u) <= 2e-5
            if held:   # iteration 1: held, and the gradient is there
                assert np.array_equal(w[0], start) == (step == 0) and np.abs(u[0]).max() > 0
            elif step == 0:   # 1 / (index + 1), and then the step: the rate times the decay of it
                assert np.allclose(w[0][host], 1.0 / (np.array(device) + 1.0), rtol=2 * 0.05 * 0.0005)
            copy_parameters(aet, fused, plain)
    finally:
        ctx.profile(0)
        fused.close()
        plain.close()


def parameters(aet, net):
    return [net.layer(i).read(which) for i in range(net.layer_count) for which in (aet.P_WEIGHTS, aet.P_WEIGHT_UPDATES, aet.P_BIASES, aet.P_BIAS_UPDATES)
            if net.layer(i).param_count(which)]


def test_a_step_that_fails_leaves_everything_as_it_was(aet):
    """No memory for a convolution's weight gradient, after the fully connected layers behind it had theirs: no parameter has
    moved, no gradient is left over, and the step that is made again is the step."""
    text = (HEAD % (32, 8, 8, 16) + CONV % (512, 3, 1, "leaky", "") + CONV % (512, 3, 1, "leaky", "") + CONV % (256, 8, 0, "relu", "") +
            CONV % (10, 1, 0, "linear", "") + "[softmax]\n")
    own = aet.Context(0)
    failing, other = two_nets(aet, own, text, 32)
    warm, spare = two_nets(aet, own, text, 32)
    try:
        # the kernels are loaded and the main stream has its scratch; the second stream's is still to come
        own.set_option("overlap_wgrad", 0)
        own.profile(1)
        warm.train_device()
        assert any("_sgd" in n for n in variants_used(own)), variants_used(own)
        own.profile(0)
        own.set_option("overlap_wgrad", 1)
        before = parameters(aet, failing)
        with device_memory_taken(10 << 20):
            with pytest.raises(aet.AetError, match="out of memory"):
                failing.train_device()
        for a, b in zip(before, parameters(aet, failing)):
            assert np.array_equal(a, b)
        for _ in range(2):
            failing.train_device()
            other.train_device()
            for a, b in zip(parameters(aet, failing), parameters(aet, other)):
                assert np.array_equal(a, b)
    finally:
        for thing in (failing, other, warm, spare, own):
            thing.close()


IMAGE_NET = ("[net]\nbatch=%d\nwidth=%d\nheight=%d\nchannels=%d\nparity=%s\nlearning_rate=0.01\nmomentum=0.9\ndecay=0.0005\npolicy=constant\n\n"
             "[convolutional]\nfilters=%d\nsize=3\nstride=1\npad=1\nbatch_normalize=1\nactivation=leaky\n\n[maxpool]\nsize=2\nstride=2\n\n"
             "[convolutional]\nfilters=%d\nsize=3\nstride=1\npad=1\nbatch_normalize=1\nactivation=leaky\n\n[maxpool]\nsize=2\nstride=2\n\n"
             "[convolutional]\nfilters=%d\nsize=1\nstride=1\npad=0\nactivation=linear\n\n[avgpool]\n\n[softmax]\ngroups=1\n")


def compare_all(aet, fused, plain, tol):
    for i in range(fused.layer_count):
        a, b = fused.layer(i), plain.layer(i)
        for which in (aet.P_WEIGHTS, aet.P_WEIGHT_UPDATES, aet.P_BIASES, aet.P_BIAS_UPDATES, aet.P_SCALES, aet.P_SCALE_UPDATES, aet.P_ROLLING_MEAN,
                      aet.P_DELTA, aet.P_OUTPUT):
            if a.param_count(which):
                u, v = a.read(which), b.read(which)
                assert np.isfinite(u).all() and rel_l2(u, v) <= tol, (i, which, rel_l2(u, v))


# (batch, map, image channels, filters of the first and second layer, classes, parity)
@pytest.mark.parametrize("case", [(37, 32, 3, 64, 128, 10, "mtcs"), (5, 24, 1, 128, 96, 3, "cpu"), (9, 36, 2, 61, 260, 32, "mtcs")])
@pytest.mark.parametrize("graph", [False, True])
def test_head_delta_with_the_forward_pass(aet, ctx, case, graph):
    """In a training step the classifier head forms its input's delta with the forward pass.  Every sum of the head has the order that
    it has call by call: outputs, deltas and the head's parameters are the same bit for bit.  (The other layers' weight gradients
    may be split otherwise in a step, where they overwrite the gradient instead of adding to it.)"""
    batch, side, channels, n0, n1, classes, parity = case
    text = IMAGE_NET % (batch, side, side, channels, parity, n0, n1, classes)
    fused, plain = two_nets(aet, ctx, text, batch)
    try:
        fused.use_graph(graph)
        ctx.profile(0 if graph else 1)
        for step in range(2):
            fused.train_device()
            step_by_calls(aet, plain)
            if step == 0:
                for i in range(fused.layer_count):
                    a, b = fused.layer(i), plain.layer(i)
                    for which in (aet.P_OUTPUT, aet.P_DELTA) + ((aet.P_WEIGHTS, aet.P_WEIGHT_UPDATES, aet.P_BIASES, aet.P_BIAS_UPDATES) if i == 4 else ()):
                        assert not a.param_count(which) or np.array_equal(a.read(which), b.read(which)), (i, which)
        if not graph:
            names = variants_used(ctx)
            assert any(n.startswith("linear_head_forward.dx") for n in names), names
        # of values that differ in the last of 24 bits one in 2^13 falls on the other side of a TF32 step of 2^-10 of its size:
        # sqrt(2^-13) 2^-10 = 1.1e-5 for each of the three convolutions that such a value passes
        compare_all(aet, fused, plain, 3.3e-5)
    finally:
        ctx.profile(0)
        ctx.set_parity(aet.PARITY_MTCS)
        fused.close()
        plain.close()


@pytest.mark.parametrize("behind", ["[softmax]\n", "[dropout]\nprobability=0.5\n\n[softmax]\n", "[shortcut]\nfrom=-2\nactivation=linear\n\n[softmax]\n",
                                    "[shortcut]\nfrom=-4\nactivation=linear\n\n[softmax]\n"])
def test_layers_behind_the_classifier_head(aet, ctx, behind):
    """What the layers behind a head's softmax add to its delta, or to that of the layer in front of the head, counts in a
    training step as it does call by call."""
    text = (HEAD % (9, 16, 16, 3) + CONV % (32, 3, 1, "leaky", "") + "[maxpool]\nsize=16\nstride=16\npadding=0\n\n" + CONV % (10, 1, 0, "leaky", "") +
            CONV % (10, 1, 0, "linear", "") + "[avgpool]\n\n[softmax]\n\n" + behind)
    fused, plain = two_nets(aet, ctx, text, 9)
    try:
        if "dropout" in behind:
            r = np.random.default_rng(7).random(fused.layer(6).param_count(aet.P_RAND), np.float32)
            for n in (fused, plain):
                n.layer(6).write(aet.P_RAND, r)
        for _ in range(2):
            fused.train_device()
            step_by_calls(aet, plain)
        compare_all(aet, fused, plain, 3.3e-5)   # as above
    finally:
        fused.close()
        plain.close()


@pytest.mark.parametrize("case", [(3, 3, 2, "leaky", 0, 27, 96), (2, 2, 2, "relu", 0, 16, 20), (3, 3, 2, "linear", 0, 14, 33), (2, 2, 2, "leaky", 1, 15, 32),
                                  (3, 3, 2, "tanh", 0, 13, 32)])
@pytest.mark.parametrize("dropout", [False, True])
def test_pool_backward_from_the_pooled_values(aet, ctx, case, dropout):
    """The convolution in front of a max-pool (no batch norm) takes its activation's gradient from the pooled output in a training
    step; not behind a dropout layer, which changes that output, and not for activations other than the simple ones."""
    batch, size, stride, act, padding, side, filters = case
    text = (HEAD % (batch + 2, side, side, 3) + CONV % (filters, 3, 1, act, "") + "[maxpool]\nsize=%d\nstride=%d\npadding=%d\n\n" % (size, stride, padding) +
            ("[dropout]\nprobability=0.5\n\n" if dropout else "") + CONV % (10, 1, 0, "linear", "") + "[avgpool]\n\n[softmax]\n")
    fused, plain = two_nets(aet, ctx, text, batch + 2)
    try:
        if dropout:
            r = np.random.default_rng(7).random(fused.layer(2).param_count(aet.P_RAND), np.float32)
            for n in (fused, plain):
                n.layer(2).write(aet.P_RAND, r)
        ctx.profile(1)
        fused.train_device()
        names = variants_used(ctx)
        ctx.profile(0)
        pooled = act != "tanh" and not dropout and padding // 2 == 0
        assert any(n.startswith("pool_bias_act_bwd.pooled") for n in names) == pooled, names
        step_by_calls(aet, plain)
        compare(aet, fused, plain, 1e-6)
        # up to four windows' deltas meet in a value, call by call in another order
        assert rel_l2(fused.layer(0).read(aet.P_DELTA), plain.layer(0).read(aet.P_DELTA)) <= 4 * 2.0 ** -24
    finally:
        ctx.profile(0)
        fused.close()
        plain.close()
