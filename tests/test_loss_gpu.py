"""Loss, softmax backward and batch totals in one launch: the same bits as the three launches it stands for, at the edges
of a block's columns and rows, with labels out of range, and with the counter back at zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from pydtnn_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 10), (64, 255), (255, 257), (257, 1000), (600, 2)])
def test_one_launch_equals_three(rows, cols, dtype):
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    dt = _lib.dtype_code("float32" if dtype == torch.float32 else "float64")
    rng = np.random.Generator(np.random.PCG64(rows * 1000 + cols))
    probs = torch.softmax(torch.from_numpy(rng.standard_normal((rows, cols)) * 4).to("cuda", dtype), 1)
    labels = torch.from_numpy(rng.integers(-1, cols + 1, rows).astype(np.int32)).cuda()
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")

    def outputs():
        return [torch.full((rows,), 7, dtype=dtype, device="cuda"), torch.full((rows,), 7, dtype=torch.int32, device="cuda"),
                torch.full_like(probs, 7), torch.full_like(probs, 7), torch.full((2,), 7, dtype=torch.float64, device="cuda")]

    a = outputs()
    _lib.check(L.b2c_cce_forward_backward(dt, rows, cols, probs.data_ptr(), labels.data_ptr(), 2 * rows, 1e-8, a[0].data_ptr(),
                                          a[1].data_ptr(), a[2].data_ptr(), st))
    _lib.check(L.b2c_softmax_backward(dt, rows, cols, a[2].data_ptr(), probs.data_ptr(), a[3].data_ptr(), st))
    _lib.check(L.b2c_cce_totals(dt, rows, a[0].data_ptr(), a[1].data_ptr(), a[4].data_ptr(), st))
    for _ in range(3):
        b = outputs()
        _lib.check(L.b2c_cce_softmax_backward(dt, rows, cols, probs.data_ptr(), labels.data_ptr(), 2 * rows, 1e-8, b[0].data_ptr(),
                                              b[1].data_ptr(), b[2].data_ptr(), b[3].data_ptr(), b[4].data_ptr(),
                                              counter.data_ptr(), st))
        for name, u, v in zip(("row loss", "hit", "dx", "softmax dx", "totals"), a, b):
            assert torch.equal(u, v), name
        assert counter.item() == 0


def test_a_step_that_was_cut_short_leaves_nothing_for_the_next_backward():
    from pydtnn_b200.layers import Input, Softmax
    from pydtnn_b200.losses import CategoricalCrossEntropy
    from pydtnn_b200.model import Model
    from pydtnn_b200.tensor_gpu import TensorGPU, to_gpu
    m = Model(batch_size=4)
    m.add(Input(shape=(6,)))
    m.add(Softmax())
    layer = m.layers[1]
    layer.need_dx = True
    rng = np.random.default_rng(0)
    x, dy = (TensorGPU(to_gpu(rng.standard_normal((4, 6)).astype(np.float32)), m.tensor_format) for _ in "xy")
    layer.dx = TensorGPU(to_gpu(np.zeros((4, 6), np.float32)), m.tensor_format)
    y = layer.forward(x)
    CategoricalCrossEntropy((4, 6), m)(y, to_gpu(np.zeros(4, np.int32)), 4, softmax=layer)
    p, d = layer.forward(x).ary.get().astype(np.float64), dy.ary.get().astype(np.float64)
    got = layer.backward(dy).ary.get()
    assert np.allclose(got, p * (d - (d * p).sum(1, keepdims=True)), atol=1e-6)
