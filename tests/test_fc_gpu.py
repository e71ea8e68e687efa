"""FC layers over the range of their routes (dot products, dense tiles written straight to dw, split sums, small batch with a
large matrix, generic): forward and backward against NumPy in float64, with and without each output. GPU."""
import numpy as np
import pytest
import torch

from pydtnn_b200 import _lib
from tests.gpu_util import DEV, assert_parity, dev, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,i,o", [(1, 1, 1), (64, 128, 10), (9, 33, 31), (512, 16, 1000), (513, 16, 1000), (5, 129, 127), (1, 4096, 1000), (64, 1568, 128),
                                   (128, 300, 100), (33, 2048, 1004), (64, 257, 130), (130, 640, 72), (32, 4096, 1024), (97, 520, 1001)])
def test_fc_routes(n, i, o, dtype):
    L, dt = _lib.lib(), _lib.dtype_code(np.dtype(dtype))
    rng = np.random.Generator(np.random.PCG64(n + i + o))
    x, w, b, dy = (rng.standard_normal(s).astype(dtype) for s in ((n, i), (i, o), (o,), (n, o)))
    X, W, B, D = (a.astype(np.float64) for a in (x, w, b, dy))
    xd, wd, bd, dyd = (dev(a) for a in (x, w, b, dy))
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(dt, n, i, o, 0)), dtype=torch.uint8, device=DEV)

    def out(*shape):
        return torch.full(shape, float("nan"), dtype=xd.dtype, device=DEV)
    for bias in (bd, None):
        y = out(n, o)
        _lib.check(L.b2c_fc_forward(dt, 0, n, i, o, xd.data_ptr(), wd.data_ptr(), bias.data_ptr() if bias is not None else None, y.data_ptr(),
                                    ws.data_ptr(), ws.numel(), stream()))
        assert_parity(y.cpu().numpy(), X @ W + (B if bias is not None else 0), dtype, "y")
    for which in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1)):
        t = (out(i, o), out(o), out(n, i))
        _lib.check(L.b2c_fc_backward(dt, 0, n, i, o, xd.data_ptr(), dyd.data_ptr(), wd.data_ptr(),
                                     *(u.data_ptr() if k else None for u, k in zip(t, which)), ws.data_ptr(), ws.numel(), stream()))
        for u, k, ref in zip(t, which, (X.T @ D, D.sum(0), D @ W.T)):
            if k:
                assert_parity(u.cpu().numpy(), ref, dtype, str(which))
            else:
                assert bool(torch.isnan(u).all())


@pytest.mark.parametrize("n,i,o", [(5, 151, 11), (42, 163, 59), (64, 128, 10), (512, 4, 4096), (3, 16384, 1)])
def test_small_layers_round_once(n, i, o):
    L = _lib.lib()
    rng = np.random.Generator(np.random.PCG64(n))
    x, w, b, dy = (rng.standard_normal(s).astype(np.float32) for s in ((n, i), (i, o), (o,), (n, o)))
    xd, wd, bd, dyd = (dev(a) for a in (x, w, b, dy))
    y, dw, db, dx = (torch.empty(s, device=DEV) for s in ((n, o), (i, o), (o,), (n, i)))
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(0, n, i, o, 0)), dtype=torch.uint8, device=DEV)
    _lib.check(L.b2c_fc_forward(0, 0, n, i, o, xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    _lib.check(L.b2c_fc_backward(0, 0, n, i, o, xd.data_ptr(), dyd.data_ptr(), wd.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(),
                                 ws.data_ptr(), ws.numel(), stream()))
    X, W, B, D = (a.astype(np.float64) for a in (x, w, b, dy))
    # one rounding to float32, and what the sums in double leave of 16384 terms at most (2^-53 each of their magnitudes)
    for got, ref, mag in ((y, X @ W + B, abs(X) @ abs(W) + abs(B)), (dw, X.T @ D, abs(X.T) @ abs(D)), (db, D.sum(0), abs(D).sum(0)), (dx, D @ W.T, abs(D) @ abs(W.T))):
        assert (abs(got.cpu().numpy() - ref) <= 2.0 ** -24 * abs(ref) + 2.0 ** -38 * mag).all()


@pytest.mark.parametrize("n,i,o", [(2048, 64, 16384), (1056, 64, 32000), (1025, 32, 16384)])
def test_bias_gradient_of_wide_layers_with_many_rows(n, i, o):
    L = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(n)
    x, dy, w = (torch.randn(s, device=DEV, generator=g) for s in ((n, i), (n, o), (i, o)))
    dw, db, dx = (torch.full(s, float("nan"), device=DEV) for s in ((i, o), (o,), (n, i)))
    ws = torch.empty(L.b2c_fc_workspace_bytes(0, n, i, o, 0), dtype=torch.uint8, device=DEV)
    _lib.check(L.b2c_fc_backward(0, 0, n, i, o, x.data_ptr(), dy.data_ptr(), w.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(),
                                 ws.data_ptr(), ws.numel(), stream()))
    X, D, W = (a.cpu().numpy().astype(np.float64) for a in (x, dy, w))
    for got, ref, what in ((dw, X.T @ D, "dw"), (db, D.sum(0), "db"), (dx, D @ W.T, "dx")):
        assert_parity(got.cpu().numpy(), ref, np.float32, what)


@pytest.mark.parametrize("n,i,o", [(1, 2048, 1000), (16, 256, 257), (17, 65, 260), (32, 1568, 128), (47, 640, 64), (48, 640, 47), (49, 201, 131), (64, 1568, 128),
                                   (65, 320, 100), (128, 320, 48), (250, 100, 203)])
@pytest.mark.parametrize("shift", [0, 1])
def test_passes_in_one_launch(n, i, o, shift):
    """Edges of the row tiles (16, 32, 64), of the steps of 32 products and of the sums in plain FMAs (47, 48), shares of a K loop
    without any product, filters on any alignment, an infinity and its row."""
    L = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(n + i + o)

    def buf(s, off):
        return torch.full((int(np.prod(s)) + off,), float("nan"), device=DEV)[off:].view(s)
    x, dy, y, dx = (buf(s, 0) for s in ((n, i), (n, o), (n, o), (n, i)))
    w, b, dw, db = (buf(s, shift) for s in ((i, o), (o,), (i, o), (o,)))
    for t in (x, w, b, dy):
        t.copy_(torch.randn(t.shape, device=DEV, generator=g))
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(0, n, i, o, 0)), dtype=torch.uint8, device=DEV)

    def run():
        _lib.check(L.b2c_fc_forward(0, 0, n, i, o, x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
        _lib.check(L.b2c_fc_backward(0, 0, n, i, o, x.data_ptr(), dy.data_ptr(), w.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(),
                                     ws.data_ptr(), ws.numel(), stream()))
    run()
    X, W, B, D = (t.double() for t in (x, w, b, dy))
    for got, ref in ((y, X @ W + B), (dw, X.T @ D), (db, D.sum(0)), (dx, D @ W.T)):
        # float32 sums of up to 2048 random terms: 2^-24 each, growing with the root of their number at most
        assert float((got.double() - ref).norm() / ref.norm()) <= 3e-7
    first = [t.clone() for t in (y, dw, db, dx)]
    run()
    assert all(torch.equal(a, t) for a, t in zip(first, (y, dw, db, dx)))
    x[0, i - 1] = float("inf")
    run()
    assert torch.equal(y[0], torch.where(w[i - 1] > 0, float("inf"), float("-inf")))
    assert bool(torch.isfinite(y[1:]).all()) and bool(torch.isfinite(dw[: i - 1]).all())


@pytest.mark.parametrize("n,i,o", [(3, 1, 17000), (16, 40, 512), (17, 47, 4096), (24, 33, 1000), (64, 16, 2048), (64, 17, 1000), (64, 40, 1000), (200, 47, 400), (250, 33, 515)])
def test_short_forward_sums_are_fmas(n, i, o):
    """Fewer than 48 features, more than 16 K weights: one launch, and as precise as FMAs.  Where one product of a sum is not zero
    an FMA rounds once, so the result is the float32 product (a split product misses it by up to 2^-22)."""
    L = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(n + i + o)
    w, b, v = (torch.randn(s, device=DEV, generator=g) for s in ((i, o), (o,), (n, i)))
    one = torch.zeros(n, i, device=DEV)
    hot = torch.arange(n, device=DEV) % i
    one[torch.arange(n, device=DEV), hot] = v[:, 0]
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(0, n, i, o, 0)), dtype=torch.uint8, device=DEV)

    def forward(x, bias):
        y = torch.full((n, o), float("nan"), device=DEV)
        before = L.b2c_launch_count()
        _lib.check(L.b2c_fc_forward(0, 0, n, i, o, x.data_ptr(), w.data_ptr(), bias.data_ptr() if bias is not None else None, y.data_ptr(),
                                    ws.data_ptr(), ws.numel(), stream()))
        assert L.b2c_launch_count() - before == 1
        return y
    assert torch.equal(forward(one, None), v[:, :1] * w[hot])
    ref = v.double() @ w.double() + b.double()
    assert float((forward(v, b).double() - ref).norm() / ref.norm()) <= 3e-7       # at most 47 roundings of 2^-24, of either sign


@pytest.mark.parametrize("n,i,o", [(16, 256, 257), (24, 512, 100), (64, 777, 333), (64, 256, 256), (100, 300, 203), (48, 512, 130)])
def test_values_that_are_not_finite_come_out_as_from_fmas(n, i, o):
    """Infinities times infinities, tiny values and zeros, NaN, sums with infinities of both signs, values next to the largest one:
    forward, dw (48 to 100 rows, out no multiple of 4 among them) and dx."""
    L = _lib.lib()
    rng = np.random.Generator(np.random.PCG64(n + i + o))
    x, w, dy = (rng.standard_normal(s).astype(np.float32) for s in ((n, i), (i, o), (n, o)))
    inf, big, tiny = np.float32(np.inf), np.finfo(np.float32).max, np.float32(1e-42)
    # x and w meet in y (over i), x and dy in dw (over n), dy and w in dx (over o): planted at indices of their own in each
    x[0, 5] = inf
    x[1, 7], x[1, 9], x[2, 9], x[3, 11] = inf, -inf, np.nan, big * np.float32(2.0) ** -60
    def small(count):
        return np.ldexp(rng.standard_normal(count), -100).astype(np.float32)
    x[4, 13], w[13, :], dy[4, :] = big, small(o), small(o)
    dy[0, 6], dy[5, 8], dy[6, 4], dy[7, 4], dy[8, 10] = inf, -inf, inf, -inf, np.nan
    dy[9, 12], w[:, 12], x[9, :] = -big, small(i), small(i)
    w[5, :4] = inf, -inf, tiny, 0.0
    X, W, D, B = (dev(a) for a in (x, w, dy, np.zeros(o, np.float32)))
    y, dw, db, dx = (torch.full(s, 3.0, device=DEV) for s in ((n, o), (i, o), (o,), (n, i)))
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(0, n, i, o, 0)), dtype=torch.uint8, device=DEV)
    count = [L.b2c_launch_count()]
    _lib.check(L.b2c_fc_forward(0, 0, n, i, o, X.data_ptr(), W.data_ptr(), B.data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    count.append(L.b2c_launch_count())
    _lib.check(L.b2c_fc_backward(0, 0, n, i, o, X.data_ptr(), D.data_ptr(), W.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(), ws.data_ptr(),
                                 ws.numel(), stream()))
    count.append(L.b2c_launch_count())
    assert count[2] - count[1] == 1
    passes = [(dw, x.T, dy, "dw"), (dx, dy, w.T, "dx")]
    if i < 777:                                     # a wide forward pass is the convolution engine's, where infinities meet as NaN
        assert count[1] - count[0] == 1
        passes.append((y, x, w, "y"))
    with np.errstate(all="ignore"):
        for got, a, b, what in passes:
            products = [a[r].astype(np.float64)[:, None] * b.astype(np.float64) for r in range(len(a))]      # exact, or not finite
            ref, size = (np.stack([f(p) for p in products]) for f in (lambda p: p.sum(0), lambda p: np.abs(p).sum(0)))
            got = got.cpu().numpy()
            assert np.array_equal(np.isnan(got), np.isnan(ref)), what
            assert np.array_equal(np.isinf(got), np.isinf(ref)) and np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)].astype(np.float32)), what
            ok = np.isfinite(ref)
            assert ok.sum() > 0.5 * ok.size and size[ok].max() < big, what
            # lo * lo and the bits of either lo past tf32 are 2^-22 of a product each, the tensor core's four truncating sums of a step
            # 2^-23, the float32 sums of up to 25 steps 2^-24 each: 2.7e-6 together; a product of tiny values may vanish below 2^-126, in
            # each of its three parts, up to 777 times
            assert np.all(np.abs(got[ok] - ref[ok]) <= 2.0 ** -18 * size[ok] + 2.0 ** -114), what


@pytest.mark.parametrize("n,i,o", [(16, 256, 257), (64, 256, 256), (64, 777, 333), (8, 1024, 40)])
def test_input_gradient_on_the_buffer_of_the_input(n, i, o):
    """dw is finished before dx is written over x: not in the launch that makes both; the same where dx only reaches into x."""
    L = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(i)
    w, dy, x = (torch.randn(s, device=DEV, generator=g) for s in ((i, o), (n, o), (n, i)))
    X, W, D = (t.double() for t in (x, w, dy))
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(0, n, i, o, 0)), dtype=torch.uint8, device=DEV)
    for shift, at_once in ((0, False), (4 * (n * i // 8), False), (n * i, True)):
        both = torch.zeros(2 * n * i, device=DEV)
        both[:n * i] = x.flatten()
        dx, dw, db = both[shift:shift + n * i], torch.full_like(w, float("nan")), torch.full((o,), float("nan"), device=DEV)
        before = L.b2c_launch_count()
        _lib.check(L.b2c_fc_backward(0, 0, n, i, o, both.data_ptr(), dy.data_ptr(), w.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(),
                                     ws.data_ptr(), ws.numel(), stream()))
        assert (L.b2c_launch_count() - before == 1) == at_once
        for got, ref in ((dw, X.T @ D), (db, D.sum(0)), (dx.view(n, i), D @ W.T)):
            assert float((got.double() - ref).norm() / ref.norm()) <= 2e-6      # the bar of sums of 256 products


@pytest.mark.parametrize("n,i,o,one", [(256, 512, 512, False), (256, 1024, 256, False), (256, 100, 4000, False), (256, 256, 256, True), (192, 512, 512, True),
                                       (129, 333, 777, True)])
def test_gradients_of_more_than_128_rows(n, i, o, one):
    """One launch only where it is the faster route; the same results either way."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes chosen for 148 SMs")
    L = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(n + i + o)
    x, w, dy = (torch.randn(s, device=DEV, generator=g) for s in ((n, i), (i, o), (n, o)))
    dx, dw, db = torch.full_like(x, float("nan")), torch.full_like(w, float("nan")), torch.full((o,), float("nan"), device=DEV)
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(0, n, i, o, 0)), dtype=torch.uint8, device=DEV)
    before = L.b2c_launch_count()
    _lib.check(L.b2c_fc_backward(0, 0, n, i, o, x.data_ptr(), dy.data_ptr(), w.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(),
                                 ws.data_ptr(), ws.numel(), stream()))
    assert (L.b2c_launch_count() - before == 1) == one
    for got, ref in ((dw, x.T.double() @ dy.double()), (db, dy.double().sum(0)), (dx, dy.double() @ w.T.double())):
        assert_parity(got.cpu().numpy(), ref.cpu().numpy(), np.float32)


@pytest.mark.parametrize("n,i,o", [(8, 1024, 40), (16, 516, 100), (15, 513, 101), (24, 1024, 33), (24, 1024, 36), (32, 512, 100), (20, 515, 131), (64, 256, 256),
                                   (64, 131, 203), (48, 512, 44), (40, 300, 203)])
def test_every_form_of_the_one_launch_kernels(n, i, o):
    """Row tiles of 16, 32 and 64, float4 and scalar loads, sums over out in FMAs and in products: one launch a direction, so it is
    these kernels that ran."""
    L = _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(n + i + o)
    x, w, b, dy = (torch.randn(s, device=DEV, generator=g) for s in ((n, i), (i, o), (o,), (n, o)))
    y, dx, dw, db = (torch.full_like(t, float("nan")) for t in (dy, x, w, b))
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(0, n, i, o, 0)), dtype=torch.uint8, device=DEV)
    count = [L.b2c_launch_count()]
    _lib.check(L.b2c_fc_forward(0, 0, n, i, o, x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    count.append(L.b2c_launch_count())
    _lib.check(L.b2c_fc_backward(0, 0, n, i, o, x.data_ptr(), dy.data_ptr(), w.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(),
                                 ws.data_ptr(), ws.numel(), stream()))
    count.append(L.b2c_launch_count())
    assert [count[1] - count[0], count[2] - count[1]] == [1, 1]
    X, W, B, D = (t.double() for t in (x, w, b, dy))
    for got, ref in ((y, X @ W + B), (dw, X.T @ D), (db, D.sum(0)), (dx, D @ W.T)):
        # float32 sums of up to 1024 random terms: 2^-24 each, growing with the root of their number at most
        assert float((got.double() - ref).norm() / ref.norm()) <= 3e-7
