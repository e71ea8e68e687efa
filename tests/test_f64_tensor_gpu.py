"""The generic engine at the edges of its tiles: rows, columns and k-slices that end inside a tile, split sums, every layout,
strided and dilated classes, fully connected layers and unaligned (8-byte) pointers, against the CPU oracle. GPU."""
import numpy as np
import pytest
import torch

from oracle import conv_oracle as co
from pydtnn_b200 import _lib
from tests.gpu_util import DEV, assert_parity, run_conv, stream

pytestmark = pytest.mark.gpu

SHAPES = [(1, 3, 3, 1, 1, 1, 0, 1), (2, 9, 7, 3, 5, 3, 1, 1), (1, 16, 8, 16, 64, 1, 0, 1), (2, 13, 11, 15, 65, 3, 1, 2),
          (1, 12, 12, 17, 130, 5, 2, 1), (3, 6, 6, 128, 24, 3, 1, 1), (2, 14, 14, 33, 129, 1, 0, 2), (4, 5, 5, 96, 9, 3, 0, 1)]
# strides with dilations that share and do not share a factor with them, and taps that reach only some residues
GEOMS = [co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st) for n, h, w, ci, cout, k, pad, st in SHAPES] + [
    co.Geom(2, 13, 12, 4, 6, 3, 3, 2, 1, 2, 3, 2, 1), co.Geom(1, 17, 16, 6, 4, 3, 4, 1, 2, 4, 2, 2, 3), co.Geom(1, 11, 9, 5, 8, 2, 2, 0, 0, 3, 3, 1, 2)]


@pytest.mark.parametrize("layout,w_layout", [("NHWC", "KRSC"), ("NHWC", "CRSK"), ("NCHW", "KCRS")])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("g", GEOMS, ids=lambda g: "x".join(map(str, (g.n, g.h, g.w, g.ci, g.co, g.kh, g.vstr, g.vdil))))
def test_generic_engine(g, layout, w_layout, dtype):
    n, h, w, ci, cout, k = g.n, g.h, g.w, g.ci, g.co, g.kh
    rng = np.random.Generator(np.random.PCG64(ci + 7 * cout))
    nchw = layout == "NCHW"
    x = rng.standard_normal((n, ci, h, w) if nchw else (n, h, w, ci))
    wt = rng.standard_normal((cout, ci, k, g.kw) if nchw else (ci, k, g.kw, cout)) * np.sqrt(2.0 / (ci * k * k))
    b = rng.standard_normal(cout)
    dy = rng.standard_normal((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout))
    y = co.conv2d_forward(x, wt, b, g, layout)
    dw, db, dx = co.conv2d_backward(x, dy, wt, g, layout)
    out = run_conv(g, layout, np.dtype(dtype), x, wt, b, dy, w_layout=w_layout, engine=_lib.ENGINE_FMA)
    for name, ref in (("y", y), ("dw", dw), ("db", db), ("dx", dx)):
        assert_parity(out[name].reshape(ref.shape), ref, dtype, f"{name} {layout} {w_layout}")


@pytest.mark.parametrize("n,i,o", [(1, 64, 10), (3, 129, 65), (200, 300, 257)])
def test_float64_fc_on_8_byte_pointers(n, i, o):
    L = _lib.lib()

    def odd(*shape):                              # a tensor that starts 8 bytes past a 16-byte boundary
        count = int(np.prod(shape))
        return torch.randn(count + 1, dtype=torch.float64, device=DEV)[1:].view(*shape)
    x, w, b, dy = odd(n, i), odd(i, o), odd(o), odd(n, o)
    y, dw, db, dx = odd(n, o), odd(i, o), odd(o), odd(n, i)
    ws = torch.empty(max(256, L.b2c_fc_workspace_bytes(_lib.F64, n, i, o, 0)), dtype=torch.uint8, device=DEV)
    a = (_lib.F64, 0, n, i, o)
    _lib.check(L.b2c_fc_forward(*a, x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    _lib.check(L.b2c_fc_backward(*a, x.data_ptr(), dy.data_ptr(), w.data_ptr(), dw.data_ptr(), db.data_ptr(), dx.data_ptr(), ws.data_ptr(),
                                 ws.numel(), stream()))
    xs, wn, bn, dn = (t.cpu().numpy() for t in (x, w, b, dy))
    for got, ref in ((y, xs @ wn + bn), (dw, xs.T @ dn), (db, dn.sum(0)), (dx, dn @ wn.T)):
        assert_parity(got.cpu().numpy(), ref, np.float64)


@pytest.mark.parametrize("n,h,w,ci,cout", [(3, 83, 79, 300, 40), (1, 90, 85, 200, 300), (2, 98, 97, 131, 129), (1, 20, 19, 2500, 1030)])
@pytest.mark.parametrize("room", [True, False])
def test_float64_last_round_of_tiles_is_split(n, h, w, ci, cout, room):
    """More tiles than SMs: those past whole rounds share their K loops; without workspace for it they stay whole."""
    L = _lib.lib()
    gen = torch.Generator(device=DEV).manual_seed(ci)
    x, f, b, dy = (torch.randn(s, dtype=torch.float64, device=DEV, generator=gen) for s in ((n * h * w, ci), (ci, cout), (cout,), (n * h * w, cout)))
    y, df, dx = (torch.full_like(t, float("nan")) for t in (dy, f, x))
    d = _lib.ConvDesc(_lib.LAYOUT_NHWC, _lib.F64, _lib.W_CRSK, 0, n, h, w, ci, cout, 1, 1, 0, 0, 1, 1, 1, 1)
    need = [L.b2c_conv_workspace_bytes(d, p) for p in (_lib.PASS_FPROP, _lib.PASS_DGRAD, _lib.PASS_WGRAD)]
    tiles = [-(-m // 128) * -(-c // (64 if c <= 64 else 128)) for m, c in ((n * h * w, cout), (n * h * w, ci), (ci, cout))]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert any(t > sms and need[i] > 0 for i, t in enumerate(tiles))
    ws = torch.empty(max(need), dtype=torch.uint8, device=DEV)
    size = [ws.numel() if room or tiles[i] <= sms else 0 for i in range(3)]
    _lib.check(L.b2c_conv_fprop(d, x.data_ptr(), f.data_ptr(), b.data_ptr(), None, 0, y.data_ptr(), ws.data_ptr(), size[0], stream()))
    _lib.check(L.b2c_conv_dgrad(d, dy.data_ptr(), f.data_ptr(), dx.data_ptr(), ws.data_ptr(), size[1], stream()))
    _lib.check(L.b2c_conv_wgrad(d, x.data_ptr(), dy.data_ptr(), df.data_ptr(), None, ws.data_ptr(), size[2], stream()))
    for got, ref in ((y, x @ f + b), (dx, dy @ f.T), (df, x.T @ dy)):
        assert_parity(got.cpu().numpy(), ref.cpu().numpy(), np.float64)


@pytest.mark.parametrize("n,h,w,ci,cout", [(1, 20, 19, 2500, 1030)])
def test_float64_weight_and_bias_gradient_share_the_workspace(n, h, w, ci, cout):
    """The partial sums of a weight gradient's tail lie before the bias gradient's; with room for the latter only, tiles stay whole."""
    L = _lib.lib()
    gen = torch.Generator(device=DEV).manual_seed(ci)
    x, dy = (torch.randn(s, dtype=torch.float64, device=DEV, generator=gen) for s in ((n * h * w, ci), (n * h * w, cout)))
    d = _lib.ConvDesc(_lib.LAYOUT_NHWC, _lib.F64, _lib.W_CRSK, 0, n, h, w, ci, cout, 1, 1, 0, 0, 1, 1, 1, 1)
    full = L.b2c_conv_workspace_bytes(d, _lib.PASS_WGRAD)
    ws = torch.empty(full, dtype=torch.uint8, device=DEV)

    def run(size):
        df, db = torch.full((ci, cout), float("nan"), dtype=torch.float64, device=DEV), torch.full((cout,), float("nan"), dtype=torch.float64, device=DEV)
        ws.fill_(255)
        return L.b2c_conv_wgrad(d, x.data_ptr(), dy.data_ptr(), df.data_ptr(), db.data_ptr(), ws.data_ptr(), size, stream()), df, db
    least, most = 0, full
    while least < most:
        mid = (least + most) // 2
        least, most = (least, mid) if run(mid)[0] == 0 else (mid + 1, most)
    assert least < full // 4                                  # what the bias gradient alone asks for
    for size in (full, full - 1, least):
        rc, df, db = run(size)
        assert rc == 0
        assert_parity(df.cpu().numpy(), (x.T @ dy).cpu().numpy(), np.float64)
        assert_parity(db.cpu().numpy(), dy.sum(0).cpu().numpy(), np.float64)


@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
@pytest.mark.parametrize("n,h,w,ci,cout,k,st,which", [(1, 90, 85, 24, 300, 3, 1, _lib.PASS_FPROP), (1, 90, 85, 300, 24, 3, 1, _lib.PASS_DGRAD),
                                                      (1, 176, 176, 300, 60, 3, 2, _lib.PASS_DGRAD)])
def test_float64_tails_of_filters_with_taps(n, h, w, ci, cout, k, st, which, layout):
    """Padding, several taps, pixel classes of a strided input gradient; both orders of the gathered operand."""
    L = _lib.lib()
    nhwc = layout == "NHWC"
    gen = torch.Generator(device=DEV).manual_seed(ci)
    x, f, b = (torch.randn(s, dtype=torch.float64, device=DEV, generator=gen) for s in ((n, ci, h, w), (cout, ci, k, k), (cout,)))
    x.requires_grad_(True)
    y = torch.nn.functional.conv2d(x, f, b, stride=st, padding=k // 2)
    dy = torch.randn(y.shape, dtype=torch.float64, device=DEV, generator=gen)
    y.backward(dy)
    order = (lambda t: t.detach().permute(0, 2, 3, 1).contiguous()) if nhwc else (lambda t: t.detach().contiguous())
    d = _lib.ConvDesc(_lib.LAYOUT_NHWC if nhwc else _lib.LAYOUT_NCHW, _lib.F64, _lib.W_KRSC if nhwc else _lib.W_KCRS, 0,
                      n, h, w, ci, cout, k, k, k // 2, k // 2, st, st, 1, 1)
    need = L.b2c_conv_workspace_bytes(d, which)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert need > 0                                       # a tail
    xs, ds, fs = order(x), order(dy), order(f)
    for size in (need, 0):
        ws = torch.empty(max(size, 256), dtype=torch.uint8, device=DEV)
        if which == _lib.PASS_FPROP:
            out, ref = torch.full_like(ds, float("nan")), order(y)
            _lib.check(L.b2c_conv_fprop(d, xs.data_ptr(), fs.data_ptr(), b.data_ptr(), None, 0, out.data_ptr(), ws.data_ptr(), size, stream()))
        else:
            out, ref = torch.full_like(xs, float("nan")), order(x.grad)
            _lib.check(L.b2c_conv_dgrad(d, ds.data_ptr(), fs.data_ptr(), out.data_ptr(), ws.data_ptr(), size, stream()))
        assert_parity(out.cpu().numpy(), ref.cpu().numpy(), np.float64)


def test_float64_tails_are_split_where_that_pays():
    """Partial sums are asked for where the K loops past whole rounds are long, not where a tail costs more than it saves."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes chosen for 148 SMs")
    L = _lib.lib()
    for n, h, w, ci, cout, k, which, split in ((1, 88, 80, 512, 128, 1, _lib.PASS_DGRAD, False), (13, 72, 70, 3, 128, 7, _lib.PASS_FPROP, False),
                                               (14, 48, 48, 256, 256, 1, _lib.PASS_FPROP, False), (32, 28, 28, 256, 256, 3, _lib.PASS_FPROP, True),
                                               (32, 28, 28, 256, 256, 3, _lib.PASS_DGRAD, True), (1, 90, 85, 200, 300, 3, _lib.PASS_FPROP, True)):
        d = _lib.ConvDesc(_lib.LAYOUT_NHWC, _lib.F64, _lib.W_KRSC, 0, n, h, w, ci, cout, k, k, k // 2, k // 2, 1, 1, 1, 1)
        assert (L.b2c_conv_workspace_bytes(d, which) > 0) == split, (n, h, w, ci, cout, k)


@pytest.mark.parametrize("n,h,w,ci,cout,kh,kw,st", [(2, 13, 11, 1, 16, 3, 3, 1), (1, 16, 16, 64, 33, 1, 1, 1), (3, 17, 9, 3, 31, 4, 5, 2), (1, 23, 23, 16, 32, 2, 2, 1), (5, 8, 8, 5, 100, 3, 3, 2)])
@pytest.mark.parametrize("layout,w_layout", [("NHWC", "KRSC"), ("NHWC", "CRSK"), ("NCHW", "KCRS")])
def test_float32_forward_of_short_sums(n, h, w, ci, cout, kh, kw, st, layout, w_layout):
    """Up to 64 products an output: 16, 32 and more channels, rows past the last block, padding and strides, fused ReLU."""
    g = co.Geom(n, h, w, ci, cout, kh, kw, 1, 1, st, st, 1, 1)
    rng = np.random.Generator(np.random.PCG64(cout))
    nchw = layout == "NCHW"
    x = rng.standard_normal((n, ci, h, w) if nchw else (n, h, w, ci))
    wt = rng.standard_normal((cout, ci, kh, kw) if nchw else (ci, kh, kw, cout))
    b = rng.standard_normal(cout)
    y = co.conv2d_forward(x, wt, b, g, layout)
    out = run_conv(g, layout, np.float32, x, wt, b, np.zeros(1), w_layout=w_layout, engine=_lib.ENGINE_FMA, passes=("fprop",), relu=True)
    assert_parity(out["y"].reshape(y.shape), np.maximum(y, 0), np.float32)


@pytest.mark.parametrize("n,hw,ci,cout", [(4, 28, 17, 64), (16, 28, 44, 47), (16, 28, 17, 96), (64, 28, 8, 16), (64, 28, 44, 512), (8, 28, 64, 96), (3, 29, 33, 130)])
@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
def test_float32_forward_of_short_sums_by_threads_and_by_tiles(n, hw, ci, cout, layout):
    """1x1 layers on both sides of the rule, at sizes where it is decided by rounds of the chip."""
    L = _lib.lib()
    gen = torch.Generator(device=DEV).manual_seed(ci)
    nhwc = layout == "NHWC"
    x, f, b = (torch.randn(s, device=DEV, generator=gen) for s in ((n, hw * hw, ci), (cout, ci), (cout,)))
    ref = x.double() @ f.double().T + b.double()
    xin = x if nhwc else x.transpose(1, 2).contiguous()
    y = torch.full((n, hw * hw, cout) if nhwc else (n, cout, hw * hw), float("nan"), device=DEV)
    d = _lib.ConvDesc(_lib.LAYOUT_NHWC if nhwc else _lib.LAYOUT_NCHW, _lib.F32, _lib.W_KRSC if nhwc else _lib.W_KCRS, _lib.ENGINE_FMA,
                      n, hw, hw, ci, cout, 1, 1, 0, 0, 1, 1, 1, 1)
    ws = torch.empty(max(256, L.b2c_conv_workspace_bytes(d, _lib.PASS_FPROP)), dtype=torch.uint8, device=DEV)
    _lib.check(L.b2c_conv_fprop(d, xin.data_ptr(), f.data_ptr(), b.data_ptr(), None, 0, y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    got = (y if nhwc else y.transpose(1, 2)).double()
    assert float((got - ref).abs().max()) <= (ci + 1) * 2.0 ** -24 * float((x.abs().double() @ f.abs().double().T + b.abs().double()).max())


@pytest.mark.parametrize("c", [20, 40, 60])
def test_float32_forward_in_place(c):
    """A 1x1 layer that writes y over x: every output of a pixel is stored after its inputs have been read."""
    L = _lib.lib()
    gen = torch.Generator(device=DEV).manual_seed(c)
    x, f = (torch.randn(s, device=DEV, generator=gen) for s in ((16 * 28 * 28, c), (c, c)))
    ref = x.double() @ f.double().T
    d = _lib.ConvDesc(_lib.LAYOUT_NHWC, _lib.F32, _lib.W_KRSC, _lib.ENGINE_FMA, 16, 28, 28, c, c, 1, 1, 0, 0, 1, 1, 1, 1)
    ws = torch.empty(max(256, L.b2c_conv_workspace_bytes(d, _lib.PASS_FPROP)), dtype=torch.uint8, device=DEV)
    _lib.check(L.b2c_conv_fprop(d, x.data_ptr(), f.data_ptr(), None, None, 0, x.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    assert_parity(x.cpu().numpy(), ref.cpu().numpy(), np.float32)


# Sums of 1 to 33 slices of 16 (the ring's stages, the eight slices that are decoded at once, and one more and less of each), an odd channel
# count (single doubles are copied), outputs of one and of several tiles of 64 or 128 columns that end inside them, rows that end inside 32
@pytest.mark.parametrize("ci,cout,n", [(16, 65, 3), (48, 130, 5), (64, 128, 2), (80, 30, 7), (128, 96, 4), (129, 257, 1), (144, 64, 9), (271, 192, 2), (528, 140, 40)])
@pytest.mark.parametrize("layout,w_layout", [("NHWC", "KRSC"), ("NHWC", "CRSK"), ("NCHW", "KCRS")])
def test_float64_tiles_slices_and_stores(ci, cout, n, layout, w_layout):
    g = co.Geom(n, 7, 9, ci, cout, 1, 1, 0, 0, 1, 1)
    rng = np.random.Generator(np.random.PCG64(ci + cout))
    nchw = layout == "NCHW"
    x = rng.standard_normal((n, ci, 7, 9) if nchw else (n, 7, 9, ci))
    wt = rng.standard_normal((cout, ci, 1, 1) if nchw else (ci, 1, 1, cout)) / np.sqrt(ci)
    b = rng.standard_normal(cout)
    dy = rng.standard_normal((n, cout, 7, 9) if nchw else (n, 7, 9, cout))
    y = co.conv2d_forward(x, wt, b, g, layout)
    dw, db, dx = co.conv2d_backward(x, dy, wt, g, layout)
    out = run_conv(g, layout, np.float64, x, wt, b, dy, w_layout=w_layout)
    for name, ref in (("y", y), ("dw", dw), ("db", db), ("dx", dx)):
        assert_parity(out[name].reshape(ref.shape), ref, np.float64, f"{name} {layout} {w_layout}")
    bn = {k: rng.uniform(0.5, 1.5, cout) for k in ("running_mean", "inv_std", "gamma", "beta")}
    v = {k: a.reshape((1, cout, 1, 1) if nchw else (1, 1, 1, cout)) for k, a in bn.items()}
    fused = np.maximum((y - v["running_mean"]) * v["inv_std"] * v["gamma"] + v["beta"], 0)
    got = run_conv(g, layout, np.float64, x, wt, b, None, w_layout=w_layout, bn=bn, relu=True, passes=("fprop",))
    assert_parity(got["y"], fused, np.float64, f"fused {layout}")
