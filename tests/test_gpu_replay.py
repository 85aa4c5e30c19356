"""What calls leave behind and find: replayed passes, outputs that a fused pass left out, streams that cannot be captured."""
import ctypes
import os
import threading
import time

import numpy as np
import pytest

from conftest import rel_l2
from gpu_util import TOL_TF32

pytestmark = pytest.mark.gpu


def cifar(aet, ctx, batch=8, train=1):
    return aet.NNetwork(ctx, cfg_path=os.path.join(aet.CFG_DIR, "cifar_small.cfg"), train=train, batch=batch)


def batches(net, count, seed=11):
    rng = np.random.default_rng(seed)
    for _ in range(count):
        x = rng.random(net.input_shape, dtype=np.float32)
        t = np.eye(net.outputs, dtype=np.float32)[rng.integers(0, net.outputs, net.batch)]
        yield x, t


@pytest.mark.parametrize("replayed", [False, True])
def test_written_output_is_kept(aet, ctx, replayed):
    """What a program writes into an output tensor replaces what a fused pass left to be formed there."""
    net = cifar(aet, ctx)
    net.use_graph(replayed)
    head = net.layer_count - 3
    for x, t in batches(net, 3):
        net.train(x, t)
    for i in (0, head):
        out = net.layer(i).output
        v = np.random.default_rng(i).standard_normal(out.shape).astype(np.float32)
        for k in range(3):
            net.predict(x) if k else net.train(x, t)
            out.write(v)
            assert np.array_equal(out.read(), v), (i, k)
            assert np.array_equal(net.layer(i).read(aet.P_OUTPUT), v.ravel()), (i, k)
            net.predict(x) if k else net.train(x, t)
            out.zero()
            assert not out.read().any(), (i, k)
    net.close()


def test_replayed_prediction_leaves_the_deltas(aet, ctx):
    """A prediction captured while the deltas counted as cleared does not clear them when it is replayed later."""
    out = []
    for graph in (True, False):
        net = cifar(aet, ctx)
        net.use_graph(graph)
        (x, t), = batches(net, 1)
        net.input.write(x)
        net.truth.write(t)
        st = aet.make_state(input=net.input, truth=net.truth, train=1)
        net.forward(st)
        for _ in range(3):
            net.predict(x)
        net.forward(st)
        net.backward(st)
        net.predict(x)
        out.append([net.layer(i).read(aet.P_DELTA) for i in range(1, net.layer_count - 3)])
        net.close()
    for a, b in zip(*out):
        assert b.any() and np.array_equal(a, b)


SOFTMAXES_CFG = """[net]
batch=4
width=1
height=1
channels=10
learning_rate=0.5
[convolutional]
filters=10
size=1
activation=linear
[softmax]
[convolutional]
filters=10
size=1
activation=linear
[softmax]
"""


def test_cost_of_every_softmax_after_replayed_steps(aet, ctx):
    out = []
    for graph in (True, False):
        net = aet.NNetwork(ctx, cfg_text=SOFTMAXES_CFG, train=1)
        net.use_graph(graph)
        got = []
        for x, t in batches(net, 6):
            net.train(x, t)
            got.append(net.cost())
        out.append(got)
        net.close()
    assert out[0] == out[1]


def test_left_out_head_output_is_the_one_of_its_pass(aet, ctx, tmp_path):
    """The classifier convolution's output, which a prediction leaves out, is that of the prediction's weights and input,
    whatever is written before it is read."""
    net = cifar(aet, ctx)
    ctx.set_option("linear_head", 0)
    try:
        plain = cifar(aet, ctx)
    finally:
        ctx.set_option("linear_head", 1)
    (x, t), = batches(net, 1)
    net.save_weights(str(tmp_path / "w"))
    plain.load_weights(str(tmp_path / "w"))
    plain.predict(x)
    at = net.layer_count - 3
    want = plain.layer(at).read(aet.P_OUTPUT)
    head, before = net.layer(at), net.layer(at - 1)
    w, b = head.read(aet.P_WEIGHTS), head.read(aet.P_BIASES)

    def by_hand():
        st = aet.make_state(input=net.layer(at - 2).output, train=0)
        net.layer(at - 2).output.write(np.zeros(net.layer(at - 2).output.shape, np.float32))
        before.forward(st)

    changes = [lambda: head.write(aet.P_WEIGHTS, 2 * w), lambda: head.write(aet.P_BIASES, b + 1),
               lambda: before.output.write(np.ones(before.output.shape, np.float32)), lambda: before.output.zero(), by_hand, net.update,
               lambda: head.update(net.batch, 0.1, 0.9, 0.1)]
    for replayed in (False, True):
        net.use_graph(replayed)
        for n, change in enumerate(changes):
            net.load_weights(str(tmp_path / "w"))
            for _ in range(3):
                net.predict(x)
            change()
            assert rel_l2(head.read(aet.P_OUTPUT), want) <= TOL_TF32, (replayed, n)
    net.close()
    plain.close()


TOPK_CFG = """[net]
batch=4
width=1
height=1
channels=8
learning_rate=0.01
[convolutional]
filters=%d
size=1
activation=linear
[softmax]
"""


def test_top_k_list_grows_between_calls(aet, oracle):
    """A context of its own, so that nothing else has sized its scratch memory."""
    ctx = aet.Context(0)
    classes = 60
    net = aet.NNetwork(ctx, cfg_text=TOPK_CFG % classes, train=0)
    rng = np.random.default_rng(5)
    net.layer(0).write(aet.P_WEIGHTS, rng.standard_normal((classes, 8, 1, 1)).astype(np.float32))
    x = rng.random((4, 8, 1, 1), dtype=np.float32)
    ids = np.arange(4, dtype=np.int32)
    for k in (5, 40, 40, 40, 5, 60, 60, 5, 40):
        idx = net.predict_topk(x, k)
        net.validate(x, ids, k)
        score = net.predict(x).reshape(4, classes)
        for i in range(4):
            assert np.array_equal(idx[i], oracle.top_k(score[i], k)), (k, i)
    net.close()
    ctx.close()


def test_legacy_default_stream(aet):
    """The legacy default stream (handle 1) cannot be captured: predictions and training steps go on as plain launches."""
    out = []
    for stream in (1, None):
        ctx = aet.Context(0, stream=stream)
        net = cifar(aet, ctx)
        if stream is None:
            net.use_graph(False)
        got = []
        for x, t in batches(net, 12):
            got.append(net.train(x, t))
            got += [net.predict(x).copy(), net.predict_topk(x, 3).copy()]
        got.append(net.layer(0).read(aet.P_WEIGHTS))
        out.append(got)
        net.close()
        ctx.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_blocking_stream_is_not_captured_unasked(aet):
    """While a stream that synchronises with the legacy default stream is captured, no other thread may use that one."""
    import torch
    handle = ctypes.c_void_p()
    torch.cuda.init()
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
    ctx = aet.Context(0, stream=handle.value)
    net = cifar(aet, ctx, batch=2, train=0)
    x, _ = next(batches(net, 1))
    want = net.predict_topk(x, 4).copy()
    stop, failed = threading.Event(), []

    def other():
        a = torch.zeros(64, device="cuda")
        try:
            while not stop.is_set():
                a.add_(1.0)
        except RuntimeError as e:
            failed.append(e)

    worker = threading.Thread(target=other)
    worker.start()
    try:
        for i in range(300):   # a new k is a new pass
            k = 1 + i // 3 % 4
            assert np.array_equal(net.predict_topk(x, k), want[:, :k])
    finally:
        stop.set()
        worker.join()
        net.close()
        ctx.close()
        torch.cuda.synchronize()
        torch.cuda.cudart().cudaStreamDestroy(handle.value)
    assert not failed, failed


def test_prediction_reports_an_expired_wait(aet):
    """A bounded wait that ran out is reported by the prediction that follows or contains it, once."""
    ctx = aet.Context(0)
    net = cifar(aet, ctx)
    (x, _), = batches(net, 1)
    want, best = net.predict(x).copy(), net.predict_topk(x, 3).copy()
    ids = np.arange(net.batch, dtype=np.int32) % 10
    share = net.validate(x, ids, 3)
    try:
        for call in (lambda: net.predict(x), lambda: net.predict_topk(x, 3), lambda: net.validate(x, ids, 3)):
            ctx.set_wait_limit(1000000)
            ctx.wait_probe()
            with pytest.raises(aet.AetError, match="wait"):
                call()
            ctx.set_wait_limit(1000000000)
            assert np.array_equal(net.predict(x), want) and np.array_equal(net.predict_topk(x, 3), best)
            assert net.validate(x, ids, 3) == share
    finally:
        ctx.set_wait_limit(1000000000)
    ctx.check()
    net.close()
    ctx.close()


def test_passes_that_keep_changing_are_not_captured_each_time(aet, ctx):
    """Capturing costs two plain passes of this network: list lengths in turn run as plain launches."""
    net = cifar(aet, ctx, batch=2, train=0)
    x, _ = next(batches(net, 1))

    def median(calls):
        took = []
        for i in range(60):
            t = time.perf_counter()
            calls[i % len(calls)]()
            took.append(time.perf_counter() - t)
        return sorted(took[10:])[25]

    net.use_graph(False)
    plain = median([lambda: net.predict_topk(x, 3)])
    net.use_graph(True)
    assert median([lambda k=k: net.predict_topk(x, k) for k in (3, 4, 5)]) <= 1.7 * plain
    assert median([lambda: net.predict_topk(x, 3)]) <= 1.2 * plain
    net.close()


def test_host_data_is_refused_while_the_stream_is_captured(aet):
    """A captured upload would read its staging memory again at every replay, long after that holds something else."""
    import torch
    stream = torch.cuda.Stream()
    ctx = aet.Context(0, stream=stream.cuda_stream)
    net = cifar(aet, ctx, batch=2)
    (x, t), = batches(net, 1)
    for _ in range(2):
        net.train(x, t)
    layer = net.layer(0)
    w, b = layer.read(aet.P_WEIGHTS), layer.read(aet.P_BIASES)
    net.input.write(x)
    net.truth.write(t)
    ctx.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for call in (lambda: net.input.write(x), lambda: layer.write(aet.P_WEIGHTS, w), lambda: layer.write(aet.P_BIASES, b), lambda: net.train(x, t),
                     lambda: net.augment_input(x, [{}] * 2)):
            with pytest.raises(aet.AetError, match="captured"):
                call()
        net.train_device(want_loss=False)
    w = layer.read(aet.P_WEIGHTS)
    graph.replay()
    torch.cuda.synchronize()
    assert not np.array_equal(layer.read(aet.P_WEIGHTS), w)
    del graph
    net.close()
    ctx.close()
