"""Training steps whose weight gradients apply the update in their epilogue, against the same step made call by call."""
import os

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
    t = np.eye(nets[0].outputs, dtype=np.float32)[rng.integers(0, nets[0].outputs, batch)]
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


def test_self_updating_layers_scrub_and_hold_still(aet, ctx):
    """Non-finite pending updates are cleared as by the update kernel, and a layer that is not updated yet only collects."""
    for extra in ("", "dont_update=1\n"):
        text = HEAD % (16, 8, 8, 32) + CONV % (64, 3, 1, "leaky", "") + CONV % (1540, 8, 0, "relu", extra) + CONV % (10, 1, 0, "linear", "") + "[softmax]\n"
        fused, plain = two_nets(aet, ctx, text, 16)
        try:
            for n in (fused, plain):
                u = n.layer(1).read(aet.P_WEIGHT_UPDATES)
                u[[3, 1017, len(u) - 1]] = np.nan, np.inf, -np.inf
                if not extra:
                    n.layer(1).write(aet.P_WEIGHT_UPDATES, u)
            start = fused.layer(1).read(aet.P_WEIGHTS)
            for step in range(2):
                fused.train_device()
                if not extra and step == 0:
                    with pytest.raises(aet.AetError):
                        ctx.check()
                if extra:   # iteration 1: held
                    assert np.array_equal(fused.layer(1).read(aet.P_WEIGHTS), start) == (step == 0)
                    continue
                step_by_calls(aet, plain)
                if step == 0:
                    with pytest.raises(aet.AetError):
                        ctx.check()
            if not extra:
                compare(aet, fused, plain, 2e-5)
        finally:
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
