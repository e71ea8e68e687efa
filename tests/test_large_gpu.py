"""Batch norm and pooling over more elements than 31 bits count (their kernels then divide 64-bit indices): 43 images of three 4096 x 4096
planes, NCHW, against torch image by image. GPU."""
import pytest
import torch

from pydtnn_b200 import _lib
from tests.gpu_util import DEV, stream

pytestmark = pytest.mark.gpu

N, C, HW = 43, 3, 4096


@pytest.fixture(autouse=True)
def room():
    if torch.cuda.mem_get_info()[1] < 64 << 30:
        pytest.skip("needs 35 GB of device memory")
    yield
    torch.cuda.empty_cache()


def _vec(*v):
    return torch.tensor(v, device=DEV)


def test_batch_norm():
    L = _lib.lib()
    gen = torch.Generator(device=DEV).manual_seed(1)
    x = torch.empty(N, C, HW, HW, device=DEV).normal_(generator=gen)
    assert x.numel() > 2 ** 31
    mean, inv, gamma, beta = _vec(0.1, -0.2, 0.3), _vec(1.1, 0.9, 1.3), _vec(0.7, -1.2, 1.5), _vec(0.2, 0.1, -0.4)
    y = torch.full_like(x, float("nan"))
    _lib.check(L.b2c_bn_inference(_lib.F32, _lib.LAYOUT_NCHW, N, C, HW * HW, x.data_ptr(), mean.data_ptr(), inv.data_ptr(), gamma.data_ptr(),
                                  beta.data_ptr(), 0, y.data_ptr(), stream()))
    col = lambda t: t.double().view(C, 1, 1)
    eps = 2.0 ** -24
    for i in range(N):
        xn = (x[i].double() - col(mean)) * col(inv)
        # a rounding each for the difference, the two products and the sum
        assert bool(((y[i].double() - (xn * col(gamma) + col(beta))).abs() <= 4 * eps * ((xn * col(gamma)).abs() + col(beta).abs())).all())
    dy, dx = y, torch.full_like(x, float("nan"))
    dy.normal_(generator=gen)
    dgamma, dbeta = torch.empty(C, device=DEV), torch.empty(C, device=DEV)
    scratch = torch.empty(1200 * C, dtype=torch.float64, device=DEV)
    _lib.check(L.b2c_bn_train_backward(_lib.F32, _lib.LAYOUT_NCHW, N, C, HW * HW, x.data_ptr(), dy.data_ptr(), None, None, gamma.data_ptr(),
                                       mean.data_ptr(), inv.data_ptr(), dgamma.data_ptr(), dbeta.data_ptr(), dx.data_ptr(), scratch.data_ptr(),
                                       scratch.numel() * 8, stream()))
    sums, size = torch.zeros(2, C, dtype=torch.float64, device=DEV), torch.zeros(2, C, dtype=torch.float64, device=DEV)
    for i in range(N):
        g, gx = dy[i].double(), dy[i].double() * ((x[i].double() - col(mean)) * col(inv))
        sums += torch.stack((gx.sum((1, 2)), g.sum((1, 2))))
        size += torch.stack((gx.abs().sum((1, 2)), g.abs().sum((1, 2))))
    # each xn and each product is rounded once or twice, the sums are taken in double
    assert bool(((torch.stack((dgamma, dbeta)).double() - sums).abs() <= 4 * eps * size).all())
    count = N * HW * HW
    for i in range(N):
        xn, g = (x[i].double() - col(mean)) * col(inv), dy[i].double()
        k = col(gamma) * col(inv) / count
        ref = k * (count * g - xn * col(dgamma) - col(dbeta))
        assert bool(((dx[i].double() - ref).abs() <= 8 * eps * k.abs() * (count * g.abs() + (xn * col(dgamma)).abs() + col(dbeta).abs())).all())


@pytest.mark.parametrize("is_max", [1, 0])
def test_pooling_backward(is_max):
    L = _lib.lib()
    gen = torch.Generator(device=DEV).manual_seed(2)
    half = HW // 2
    dy = torch.empty(N, C, half, half, device=DEV).normal_(generator=gen)
    idx = torch.randint(0, 4, dy.shape, dtype=torch.int32, device=DEV, generator=gen)
    dx = torch.full((N, C, HW, HW), float("nan"), device=DEV)
    assert dx.numel() > 2 ** 31
    _lib.check(L.b2c_pool_backward(_lib.F32, _lib.LAYOUT_NCHW, is_max, N, HW, HW, C, 2, 2, 0, 0, 2, 2, 1, 1, dy.data_ptr(), idx.data_ptr(),
                                   dx.data_ptr(), stream()))
    for i in range(N):
        for tap in range(4):
            want = torch.where(idx[i] == tap, dy[i], torch.zeros_like(dy[i])) if is_max else dy[i] / 4
            assert torch.equal(dx[i, :, tap // 2::2, tap % 2::2], want)
