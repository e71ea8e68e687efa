"""Passes replayed as CUDA graphs against the same passes issued launch by launch: same bits, and every change on the host
that a pass depends on is taken up. GPU."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(fmt, record, dtype=np.float32):
    from pydtnn_b200 import nets
    from pydtnn_b200.model import Model
    np.random.seed(0)
    m = Model(batch_size=4, tensor_format=fmt, dtype=dtype, enable_fused_bn_relu=True, enable_fused_conv_bn=True, enable_fused_conv_bn_relu=True)
    nets.create_resnet50_imagenet(m, input_hw=32, nclasses=10, layout=[[8, 2, 1], [16, 2, 2]])
    m.record_passes = record
    return m


def _state(m):
    out = [m.arena.chunks[0].w, m.arena.chunks[0].dw]
    out += [t.ary.t for l in m.get_all_layers() if l.canonical_name == "BatchNormalization" for t in (l.running_mean, l.running_var)]
    return [t.clone() for t in out]


@pytest.mark.parametrize("fmt", ["NHWC", "NCHW"])
def test_replayed_passes_equal_issued_ones(fmt):
    from pydtnn_b200 import _lib
    from pydtnn_b200.optimizers import SGD
    a, b = _model(fmt, True), _model(fmt, False)
    oa, ob = SGD(0.05, 0.9), SGD(0.05, 0.9)
    rng = np.random.Generator(np.random.PCG64(2))

    def step(gbs=None):
        x, y = rng.standard_normal((4, *a.layers[0].shape)).astype(np.float32), rng.integers(0, 10, 4)
        counts = []
        for m, o in ((a, oa), (b, ob)):
            n = _lib.lib().b2c_launch_count()
            m.train_batch(x, y, o, gbs)
            counts.append(_lib.lib().b2c_launch_count() - n)
        assert counts[0] == counts[1]
        assert a.loss_func.loss() == b.loss_func.loss() and a.loss_func.accuracy() == b.loss_func.accuracy()
        for p, q in zip(_state(a), _state(b)):
            assert torch.equal(p, q)

    def evaluate():
        x = rng.standard_normal((4, *a.layers[0].shape)).astype(np.float32)
        assert np.array_equal(a.evaluate_batch(x).ary.get(), b.evaluate_batch(x).ary.get())

    for _ in range(5):
        step()
    assert a._train_recorder.graph is not None and b._train_recorder.graph is None
    for _ in range(5):
        evaluate()
    assert a._eval_recorder.graph is not None
    # a step changes the running statistics that evaluation uses, without the layers' hooks being called
    for _ in range(2):
        step(), evaluate()
    oa.learning_rate = ob.learning_rate = 0.01
    step()
    # a layer's and the step's own numbers
    for m in (a, b):
        next(l for l in m.get_all_layers() if l.canonical_name == "BatchNormalization").momentum = 0.5
    for _ in range(4):
        step()
    assert a._train_recorder.graph is not None
    for _ in range(4):
        step(8)
    evaluate()
    # parameters written from outside, and another model growing the shared workspaces
    for m in (a, b):
        m.arena.chunks[0].w.mul_(1.5)
    from pydtnn_b200.layers import Conv2D, Input
    from pydtnn_b200.model import Model
    big = Model(batch_size=32)
    big.add(Input(shape=(40, 40, 256)))
    big.add(Conv2D(nfilters=512, filter_shape=(3, 3), padding=1))
    for _ in range(4):
        step(), evaluate()
    # a first look at an activation, and a write through it
    la, lb = a.layers[3].y.ary, b.layers[3].y.ary
    for _ in range(4):
        step()
        assert np.array_equal(la.get(), lb.get())
    assert a._train_recorder.graph is not None
    a.tracer.enable_tracing(ops=True), b.tracer.enable_tracing(ops=True)
    step()


def test_a_callers_own_layer_is_never_recorded():
    from pydtnn_b200.optimizers import SGD
    m = _model("NHWC", True)
    calls, layer = [], m.layers[2]
    forward = layer.forward
    layer.forward = lambda x: (calls.append(1), forward(x))[1]
    x, y = np.ones((4, *m.layers[0].shape), np.float32), np.zeros(4, np.int64)
    for _ in range(6):
        m.train_batch(x, y, SGD(0.01))
    assert len(calls) == 6 and m._train_recorder.graph is None


def _batch(m):
    rng = np.random.Generator(np.random.PCG64(3))
    return rng.standard_normal((4, *m.layers[0].shape)).astype(np.float32), rng.integers(0, 10, 4)


@pytest.mark.parametrize("evaluate", [False, True])
def test_a_changed_descriptor_is_taken_up(evaluate):
    from pydtnn_b200 import _lib
    from pydtnn_b200.layers import FC, Conv2D, Flatten, Input
    from pydtnn_b200.model import Model
    from pydtnn_b200.optimizers import SGD
    out = []
    for record in (True, False):
        np.random.seed(0)
        m = Model(batch_size=4)
        m.record_passes = record
        for layer in (Input(shape=(9, 9, 32)), Conv2D(nfilters=32, filter_shape=(3, 3)), Conv2D(nfilters=64, filter_shape=(3, 3), activation="relu"),
                      Flatten(), FC(shape=(10,), activation="softmax")):
            m.add(layer)
        x, y = _batch(m)
        o = SGD(0.0, 0.0)
        run = (lambda: m.evaluate_batch(x)) if evaluate else (lambda: m.train_batch(x, y, o))
        for _ in range(5):
            run()
        assert ((m._eval_recorder if evaluate else m._train_recorder).graph is not None) == record
        conv = [l for l in m.get_all_layers() if l.canonical_name == "Conv2D"][1]
        conv.desc.engine = _lib.ENGINE_FMA
        run()
        out.append([conv.dw.ary.t.clone(), m.layers[-1].y.ary.t.clone()])
    for p, q in zip(*out):
        assert torch.equal(p, q)


@pytest.mark.parametrize("inside", [False, True])
def test_a_replaced_layer_is_called(inside):
    from pydtnn_b200.optimizers import SGD

    class Spy:
        def __init__(self, layer):
            self.layer, self.calls = layer, 0

        def forward(self, x):
            self.calls += 1
            return self.layer.forward(x)

        def __getattr__(self, name):
            return getattr(self.layer, name)
    m = _model("NHWC", True)
    x, y = _batch(m)
    for _ in range(5):
        m.train_batch(x, y, SGD(0.01))
    assert m._train_recorder.graph is not None
    seq = next(l for l in m.layers if l.paths).paths[0] if inside else m.layers
    seq[1] = spy = Spy(seq[1])
    for n in range(4):
        m.train_batch(x, y, SGD(0.01))
        assert spy.calls == n + 1


def test_a_look_into_one_model_leaves_the_others_recordings():
    from pydtnn_b200.optimizers import SGD
    a, b = _model("NCHW", True), _model("NCHW", True)
    x, y = _batch(a)
    for _ in range(5):
        a.train_batch(x, y, SGD(0.01)), b.train_batch(x, y, SGD(0.01))
    ga, gb = a._train_recorder.graph, b._train_recorder.graph
    assert ga is not None and gb is not None
    look = b.layers[3].y.ary
    a.train_batch(x, y, SGD(0.01)), b.train_batch(x, y, SGD(0.01))
    assert a._train_recorder.graph is ga and b._train_recorder.graph is not gb
    # memory that both models use is everybody's
    shared = next(l for l in a.get_all_layers() if l.canonical_name == "Conv2D").weights
    next(l for l in b.get_all_layers() if l.canonical_name == "Conv2D").weights = shared
    for _ in range(4):
        a.train_batch(x, y, SGD(0.0)), b.train_batch(x, y, SGD(0.0))
    ga, gb = a._train_recorder.graph, b._train_recorder.graph
    assert ga is not None and gb is not None
    shared.ary.t = shared.ary.t.clone()
    a.train_batch(x, y, SGD(0.0)), b.train_batch(x, y, SGD(0.0))
    assert a._train_recorder.graph is not ga and b._train_recorder.graph is not gb
    assert look.shape == b.layers[3].y.dims


def test_a_pass_that_cannot_be_recorded_says_why(monkeypatch):
    from pydtnn_b200.backends.gpu.layers.fc_gpu import FCGPU
    from pydtnn_b200.optimizers import SGD
    backward = FCGPU.backward

    def refuses(self, dy):
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("looks at the host here")
        return backward(self, dy)
    monkeypatch.setattr(FCGPU, "backward", refuses)
    a, b = _model("NHWC", True), _model("NHWC", False)
    x, y = _batch(a)
    with pytest.warns(RuntimeWarning, match="looks at the host here"):
        for _ in range(5):
            a.train_batch(x, y, SGD(0.01)), b.train_batch(x, y, SGD(0.01))
    assert a._train_recorder.graph is None
    for p, q in zip(_state(a), _state(b)):
        assert torch.equal(p, q)


def test_a_callers_own_recording_takes_the_launches():
    m = _model("NHWC", True)
    x, y = _batch(m)
    from pydtnn_b200.optimizers import SGD
    for _ in range(5):
        m.train_batch(x, y, SGD(0.0, 0.0))
    assert m._train_recorder.graph is not None
    want = m.arena.chunks[0].dw.clone()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        with torch.cuda.graph(g):
            m.forward_backward()
            m.join_side_stream()
    del m._train_recorder.graph
    m._train_recorder.graph = None           # the caller's recording does not need the model's
    m.arena.chunks[0].dw.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(m.arena.chunks[0].dw, want)
