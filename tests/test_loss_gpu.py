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
