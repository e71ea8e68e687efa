"""Activations of NCHW models are stored channel-last until somebody looks at them (``ChannelLastTensor``): a look must
show the NCHW values, keep showing the current ones, and change no result; writes through it must be read. GPU."""
import numpy as np
import pytest
import torch

from pydtnn_b200 import _lib
from tests.gpu_util import DEV, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,rows,cols", [(1, 1, 1), (3, 3, 49), (2, 49, 3), (2, 33, 31), (2, 8, 9), (1, 257, 64), (66000, 3, 4),
                                         (40, 68, 130), (40, 65, 132), (40, 67, 129), (80, 33, 64), (1, 1000, 901)])
def test_transpose(dtype, n, rows, cols):
    x = torch.randn(n, rows, cols, dtype=getattr(torch, dtype), device=DEV)
    y = torch.full((n, cols, rows), float("nan"), dtype=x.dtype, device=DEV)
    _lib.check(_lib.lib().b2c_transpose(_lib.dtype_code(np.dtype(dtype)), n, rows, cols, x.data_ptr(), y.data_ptr(), stream()))
    assert torch.equal(y, x.transpose(1, 2).contiguous())


def _model(dtype):
    from pydtnn_b200 import nets
    from pydtnn_b200.model import Model
    np.random.seed(0)
    m = Model(batch_size=3, tensor_format="NCHW", dtype=dtype, enable_fused_bn_relu=True)
    nets.create_resnet50_imagenet(m, input_hw=36, nclasses=10, layout=[[8, 2, 1], [12, 1, 2]])
    return m


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_looking_at_activations_changes_nothing(dtype):
    from pydtnn_b200.optimizers import SGD
    a, b = _model(np.dtype(dtype).type), _model(np.dtype(dtype).type)
    oa, ob = SGD(0.05, 0.9), SGD(0.05, 0.9)
    rng = np.random.Generator(np.random.PCG64(1))
    handles = None
    for step in range(3):
        x = rng.standard_normal((3, *a.layers[0].shape)).astype(dtype)
        labels = rng.integers(0, 10, 3)
        assert a.train_batch(x, labels, oa).loss() == b.train_batch(x, labels, ob).loss()
        if step == 0:
            handles = {l: l.y.ary for l in b.get_all_layers()[1:]}
        for la, lb in zip(a.get_all_layers()[1:], b.get_all_layers()[1:]):
            # b's handles were taken after the first step and must show every later one; a is looked at only at the end
            # (batch norms and absorbed ReLUs may leave their own buffer to the layer they are fused with)
            if step == 2 and (la.canonical_name in ("Conv2D", "MaxPool2D", "AveragePool2D") or getattr(la, "fed_by_block", False)):
                assert np.array_equal(la.y.ary.get(), handles[lb].get()), lb
            for k in la.grad_vars:
                assert np.array_equal(getattr(la, k).ary.get(), getattr(lb, k).ary.get()), (la, k)


def test_values_written_through_a_look_are_read():
    from pydtnn_b200.layers import Conv2D, Input, Relu
    from pydtnn_b200.model import Model
    m = Model(batch_size=2, tensor_format="NCHW")
    m.add(Input(shape=(5, 7, 3)))
    m.add(Conv2D(nfilters=4, filter_shape=(3, 3), padding=1))
    m.add(Relu())
    m.mode = "train"
    y = m.layers[1].forward(m.layers[0].y)
    v = np.random.default_rng(0).standard_normal((2, 4, 5, 7)).astype(np.float32)
    y.ary.set(v)
    assert np.array_equal(m.layers[2].forward(y).ary.get(), np.maximum(v, 0))


@pytest.mark.parametrize("n,rows,cols", [(1, 65535 * 32 + 5, 9), (2, 65535 * 32 + 33, 33), (1, 65535 * 32 + 1, 3)])
def test_transpose_of_many_rows(n, rows, cols):
    x = torch.randn(n, rows, cols, device=DEV)
    y = torch.full((n, cols, rows), float("nan"), device=DEV)
    _lib.check(_lib.lib().b2c_transpose(_lib.F32, n, rows, cols, x.data_ptr(), y.data_ptr(), stream()))
    assert torch.equal(y, x.transpose(1, 2))


def test_large_nchw_images():
    """Images of more pixels than 32 times a grid axis: the copies of y and dx are cut, or not on that axis at all."""
    from oracle import conv_oracle as co
    from tests.gpu_util import rel_l2, run_conv
    g = co.Geom(1, 1449, 1449, 3, 8, 3, 3, 1, 1, 1, 1)
    rng = np.random.Generator(np.random.PCG64(4))
    x, w, dy = (rng.standard_normal(s).astype(np.float32) for s in ((1, 3, 1449, 1449), (8, 3, 3, 3), (1, 8, 1449, 1449)))
    got = run_conv(g, "NCHW", np.float32, x, w, None, dy)
    fma = run_conv(g, "NCHW", np.float32, x, w, None, dy, engine=_lib.ENGINE_FMA)
    for k in ("y", "dw", "dx"):
        assert rel_l2(got[k], fma[k]) <= 1e-5, k


@pytest.mark.parametrize("fmt", ["NCHW", "NHWC"])
@pytest.mark.parametrize("replaced", [False, True])
def test_backward_reads_x_as_it_is_then(fmt, replaced):
    from pydtnn_b200.layers import BatchNormalization, Conv2D, Input
    from pydtnn_b200.model import Model
    from pydtnn_b200.tensor_gpu import DeviceArray, TensorGPU
    from tests.gpu_util import rel_l2
    rng = np.random.default_rng(0)
    for layer, name in ((Conv2D(nfilters=6, filter_shape=(3, 3), padding=1), "dw"), (BatchNormalization(), "dgamma")):
        m = Model(batch_size=2, tensor_format=fmt)
        m.add(Input(shape=(5, 7, 20)))
        m.add(Conv2D(nfilters=20, filter_shape=(1, 1)))
        m.add(layer)
        m.mode = "train"
        m.overlap_wgrad = False
        shape, grad = m.layers[1].y.dims, layer.y.dims
        x0, x1, dy = (torch.from_numpy(rng.standard_normal(s).astype(np.float32)).to(DEV) for s in (shape, shape, grad))
        x, out = TensorGPU(DeviceArray(x0.clone()), m.tensor_format), []
        for second in (x0, x1):
            layer.forward(x)
            if replaced:
                x.ary = DeviceArray(second.clone())
            else:
                x.ary.t.copy_(second)
            layer.backward(TensorGPU(DeviceArray(dy.clone()), m.tensor_format))
            out.append(getattr(layer, name).ary.t.clone())
            x.ary.t.copy_(x0)
        # the gradient of the weights (of gamma) is linear in the x that backward reads: x1's is not x0's
        assert rel_l2(out[1].cpu().numpy(), out[0].cpu().numpy()) > 0.5
