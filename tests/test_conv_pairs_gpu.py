"""Launches whose CTAs work in pairs on 256 rows (conv_tc_kernel, PAIR): row tiles that do not fill the last pair, a last column
tile of few columns, every filter layout, whole tiles, balanced ranges, split K loops, the classes of a strided input gradient,
the weight gradient, batch sums. GPU."""
import ctypes
import re

import numpy as np
import pytest
import torch

from oracle import conv_oracle as co
from pydtnn_b200 import _lib
from tests.gpu_util import DEV, assert_parity, make_desc, run_conv, stream, workspace

pytestmark = pytest.mark.gpu

# (n, h, w, ci, co, k, stride): what the forward pass (input gradient) is cut into on 148 SMs, row tiles of 128
SHAPES = [
    (13, 41, 41, 128, 200, 3, 1),       # whole tiles in several rounds, 171 row tiles (the last pair has one), second column tile of 72
    (55, 17, 17, 128, 128, 3, 1),       # whole tiles in one round, 125 row tiles
    (63, 14, 14, 256, 256, 3, 1),       # balanced ranges, 97 row tiles
    (50, 4, 4, 512, 512, 3, 1),         # split K loops by single CTAs: 7 row tiles (the last of 32 rows) in five parts, more pairs than fit
    (5, 56, 56, 128, 256, 5, 2),        # input gradient: four classes of 31 row tiles
    (20, 27, 27, 96, 200, 5, 1),        # weight gradient with fine sums (200 channels), by single CTAs
    (3, 45, 33, 256, 384, 1, 1),        # weight gradient of a 1x1 layer with two row tiles, by single CTAs
    (23, 9, 9, 512, 200, 3, 1),         # split K loops, 15 row tiles (the last of 71 rows), second column tile of 72
    (24, 27, 27, 96, 224, 5, 1),        # weight gradient: 19 row tiles of (tap, channel), ranges of the pixels, second column tile of 96
    (49, 23, 23, 512, 224, 1, 1),       # weight gradient of a 1x1 layer, two pairs of row tiles
]


def _forms(launch, names=None):
    """Template arguments of the tensor-core kernels that `launch` runs: (weight gradient, columns, balanced, several classes, fine sums, pairs)."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        launch()
        torch.cuda.synchronize()
    out = []
    for e in prof.events():
        if names is not None:
            names.append(e.name)
        if "conv_tc_kernel" in e.name:
            v = [int({"true": 1, "false": 0}.get(a, a)) for a in re.sub(r"\(\w+\)", "", re.search(r"conv_tc_kernel<(.*?)>", e.name).group(1)).split(", ")]
            assert len(v) == 12, e.name
            out.append((v[0], v[1], v[3], v[7], v[9], v[11]))
    return out


def _pairs(launch):
    forms = _forms(launch)
    assert len(forms) == 1
    return bool(forms[0][-1])


def _layer(shape, layout, w_layout):
    n, h, w, ci, cout, k, st = shape
    g = co.Geom(n, h, w, ci, cout, k, k, k // 2, k // 2, st, st)
    desc = make_desc(g, layout, np.float32, w_layout)
    gen = torch.Generator(device=DEV).manual_seed(ci + cout)
    rnd = lambda *s: torch.randn(s, device=DEV, generator=gen)
    x, dy, b = rnd(n, ci, h, w), rnd(n, cout, g.ho, g.wo), rnd(cout)
    wt = rnd(cout, ci, k, k) * float(np.sqrt(2.0 / (ci * k * k)))
    act = (lambda t: t.permute(0, 2, 3, 1).contiguous()) if layout == "NHWC" else (lambda t: t)
    order = {"KCRS": (0, 1, 2, 3), "KRSC": (0, 2, 3, 1), "CRSK": (1, 2, 3, 0)}[w_layout]
    return g, desc, (x, dy, wt, b), (act(x), act(dy), wt.permute(*order).contiguous()), act, order


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout,w_layout", [("NHWC", "KRSC"), ("NHWC", "CRSK"), ("NCHW", "KCRS")])
def test_pairs_of_ctas(shape, layout, w_layout):
    n, h, w, ci, cout, k, st = shape
    L = _lib.lib()
    g, desc, (x, dy, wt, b), (xd, dyd, wd), act, order = _layer(shape, layout, w_layout)
    ws = workspace(desc)
    d = ctypes.byref(desc)

    def passes():
        out = [torch.full_like(t, float("nan")) for t in (dyd, wd, b, xd)]
        y, dw, db, dx = out
        _lib.check(L.b2c_conv_fprop(d, xd.data_ptr(), wd.data_ptr(), b.data_ptr(), None, 1, y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
        _lib.check(L.b2c_conv_wgrad(d, xd.data_ptr(), dyd.data_ptr(), dw.data_ptr(), db.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
        _lib.check(L.b2c_conv_dgrad(d, dyd.data_ptr(), wd.data_ptr(), dx.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
        return out

    y, dw, db, dx = passes()
    x64, w64, dy64 = (t.double() for t in (x, wt, dy))
    x64.requires_grad_(), w64.requires_grad_()
    y64 = torch.nn.functional.conv2d(x64, w64, b.double(), stride=st, padding=k // 2)
    y64.backward(dy64)
    refs = (act(torch.relu(y64.detach())), w64.grad.permute(*order), dy64.sum((0, 2, 3)), act(x64.grad))
    for name, got, ref in zip(("y", "dw", "db", "dx"), (y, dw, db, dx), refs):
        assert_parity(got.cpu().numpy(), ref.cpu().numpy(), np.float32, f"{name} {shape} {layout} {w_layout}")
    for _ in range(5):
        for first, again in zip((y, dw, db, dx), passes()):
            assert torch.equal(first, again)
    status = ctypes.c_int()
    _lib.check(L.b2c_check_device_status(ctypes.byref(status)))
    assert status.value == 0


# (shape, (pass, balanced, several classes, split K loop)): the passes above that are there for pairs
FORMS = [(SHAPES[0], ("fprop", 0, 0, 0)), (SHAPES[1], ("fprop", 0, 0, 0)), (SHAPES[2], ("fprop", 1, 0, 0)), (SHAPES[4], ("dgrad", 0, 1, 0)),
         (SHAPES[7], ("fprop", 0, 0, 1)), (SHAPES[8], ("wgrad", 0, 0, 0)), (SHAPES[9], ("wgrad", 0, 0, 0))]


@pytest.mark.parametrize("shape,form", FORMS)
def test_the_shapes_run_in_pairs(shape, form):
    what, balanced, classes, split = form
    L = _lib.lib()
    _, desc, _, (xd, dyd, wd), _, _ = _layer(shape, "NHWC", "KRSC")
    d, ws = ctypes.byref(desc), workspace(desc)
    y, dw, dx = torch.empty_like(dyd), torch.empty_like(wd), torch.empty_like(xd)
    tail = (ws.data_ptr(), ws.numel(), stream())
    names = []

    def launch():
        if what == "fprop":
            _lib.check(L.b2c_conv_fprop(d, xd.data_ptr(), wd.data_ptr(), None, None, 0, y.data_ptr(), *tail))
        elif what == "wgrad":
            _lib.check(L.b2c_conv_wgrad(d, xd.data_ptr(), dyd.data_ptr(), dw.data_ptr(), None, *tail))
        else:
            _lib.check(L.b2c_conv_dgrad(d, dyd.data_ptr(), wd.data_ptr(), dx.data_ptr(), *tail))

    forms = _forms(launch, names)
    assert forms == [(int(what == "wgrad"), 128, balanced, classes, 0, 1)]
    assert any("tc_split_finish" in n for n in names) == bool(split)


@pytest.mark.parametrize("shape", [(55, 17, 17, 128, 128, 3, 1), (13, 41, 41, 128, 200, 3, 1), (63, 14, 14, 256, 256, 3, 1),
                                   # eight column tiles: 72 of 74 pairs, 48 row tiles (the last of 60 rows) in more pairs than that
                                   (31, 28, 28, 512, 1024, 1, 2)])
def test_batch_sums_of_pairs(shape):
    """The sums a pair leaves for a batch norm, and that the last pair of an odd count of row tiles leaves none for rows there are not."""
    L = _lib.lib()
    g, desc, _, (xd, dyd, wd), _, _ = _layer(shape, "NHWC", "KRSC")
    cout = shape[4]
    nbytes = L.b2c_conv_stats_bytes(ctypes.byref(desc))
    rows, pixels = nbytes // (8 * cout), g.n * g.ho * g.wo
    assert nbytes and rows <= (pixels + 127) // 128 * 4
    stats = torch.full((rows + 8, 2, cout), float("nan"), device=DEV)
    y = torch.full_like(dyd, float("nan"))
    ws = workspace(desc)
    assert _pairs(lambda: _lib.check(L.b2c_conv_fprop_stats(ctypes.byref(desc), xd.data_ptr(), wd.data_ptr(), None, y.data_ptr(), stats.data_ptr(), nbytes,
                                                            ws.data_ptr(), ws.numel(), stream())))
    assert bool(torch.isnan(stats[rows:]).all())
    v = y.double().view(-1, cout)
    # a row holds the sums of at most pixels / rows values and a tile's 32 more, one float32 addition each
    adds = pixels // rows + 64
    for got, ref, mag in ((stats[:rows, 0], v, v.abs()), (stats[:rows, 1], v * v, v * v)):
        err = (got.double().sum(0) - ref.sum(0)).abs()
        assert bool((err <= adds * 2.0 ** -24 * mag.sum(0)).all())


@pytest.mark.parametrize("shape", [(64, 7, 7, 512, 2048, 1, 1), (64, 14, 14, 1024, 2048, 1, 2)])
def test_no_pairs_where_batch_sums_leave_them_too_few_ctas(shape):
    """16 column tiles: 144 of 148 CTAs hold whole groups of them, but only 64 of 74 pairs: four rounds of pairs instead of three."""
    L = _lib.lib()
    _, desc, _, (xd, dyd, wd), _, _ = _layer(shape, "NHWC", "KRSC")
    d, ws, y = ctypes.byref(desc), workspace(desc), torch.empty_like(dyd)
    nbytes = L.b2c_conv_stats_bytes(d)
    stats = torch.empty(nbytes, dtype=torch.uint8, device=DEV)
    args = (ws.data_ptr(), ws.numel(), stream())
    with_sums = lambda: _lib.check(L.b2c_conv_fprop_stats(d, xd.data_ptr(), wd.data_ptr(), None, y.data_ptr(), stats.data_ptr(), nbytes, *args))
    without = lambda: _lib.check(L.b2c_conv_fprop(d, xd.data_ptr(), wd.data_ptr(), None, None, 0, y.data_ptr(), *args))
    assert not _pairs(with_sums)
    first = y.clone()
    assert _pairs(without)
    assert torch.equal(first, y)


@pytest.mark.parametrize("shape,pairs", [((32, 36, 36, 256, 132, 3, 1), False), ((34, 41, 41, 256, 172, 5, 1), False), ((53, 25, 25, 512, 188, 3, 1), True),
                                         ((7, 79, 51, 512, 112, 3, 1), True), ((4, 76, 40, 128, 88, 5, 1), True)])
def test_no_pairs_where_the_last_column_tile_is_narrow(shape, pairs):
    """Balanced ranges of many tiles with a last column tile of 4, 44 and 60 channels: a single CTA does not multiply past them, a pair does.
    (An only column tile costs nearly what a whole one does.)"""
    L = _lib.lib()
    _, desc, _, (xd, dyd, wd), _, _ = _layer(shape, "NHWC", "KRSC")
    ws, y = workspace(desc), torch.empty_like(dyd)
    assert _pairs(lambda: _lib.check(L.b2c_conv_fprop(ctypes.byref(desc), xd.data_ptr(), wd.data_ptr(), None, None, 0, y.data_ptr(),
                                                      ws.data_ptr(), ws.numel(), stream()))) == pairs


@pytest.mark.parametrize("shape", [SHAPES[0], SHAPES[2], SHAPES[7]])
@pytest.mark.parametrize("with_bias", [True, False])
def test_folded_batch_norm_of_pairs(shape, with_bias):
    """Bias, batch norm of the running averages and ReLU in a pair's epilogue: whole tiles with a last column tile of 72, balanced ranges, a split."""
    L = _lib.lib()
    g, desc, (x, _, wt, b), (xd, dyd, wd), act, _ = _layer(shape, "NHWC", "KRSC")
    gen = torch.Generator(device=DEV).manual_seed(9)
    mean, gamma, beta = (torch.randn(shape[4], device=DEV, generator=gen) for _ in range(3))
    inv = torch.rand(shape[4], device=DEV, generator=gen) + 0.5
    bn = _lib.BnParams(*[v.data_ptr() for v in (mean, inv, gamma, beta)])
    ws, y = workspace(desc), torch.full_like(dyd, float("nan"))
    assert _pairs(lambda: _lib.check(L.b2c_conv_fprop(ctypes.byref(desc), xd.data_ptr(), wd.data_ptr(), b.data_ptr() if with_bias else None, ctypes.byref(bn), 1,
                                                      y.data_ptr(), ws.data_ptr(), ws.numel(), stream())))
    ref = act(torch.nn.functional.conv2d(x.double(), wt.double(), b.double() if with_bias else None, padding=shape[5] // 2))
    ref = torch.relu((ref - mean.double()) * inv.double() * gamma.double() + beta.double())
    assert_parity(y.cpu().numpy(), ref.cpu().numpy(), np.float32, f"{shape}")


@pytest.mark.parametrize("shape", [(55, 17, 17, 128, 128, 3, 1), (16, 56, 56, 256, 256, 3, 1)])
@pytest.mark.parametrize("where", ["x", "w", "dy"])
def test_values_that_are_not_finite_in_pairs(shape, where):
    """An infinity of each sign and a NaN touch the outputs that they touch in FMAs and no others (a pair's CTAs each hold half of the B tile);
    in the filter of a long launch, whose high halves are rounded in place, they also come out as from FMAs."""
    n, h, w, ci, cout, k, _ = shape
    g = co.Geom(n, h, w, ci, cout, k, k, k // 2, k // 2, 1, 1)
    rng = np.random.Generator(np.random.PCG64(4))
    t = {"x": rng.standard_normal((n, h, w, ci)).astype(np.float32), "w": rng.standard_normal((ci, k, k, cout)).astype(np.float32),
         "dy": rng.standard_normal((n, h, w, cout)).astype(np.float32)}
    bad = t[where].reshape(-1)
    bad[bad.size // 3], bad[bad.size // 2 + 1], bad[bad.size - 2] = np.inf, -np.inf, np.nan
    a, b = (run_conv(g, "NHWC", np.float32, t["x"], t["w"], None, t["dy"], w_layout="KRSC", engine=e) for e in (_lib.ENGINE_AUTO, _lib.ENGINE_FMA))
    for name in ("y", "dw", "dx"):
        finite = np.isfinite(b[name])
        assert np.array_equal(np.isfinite(a[name]), finite), name
        assert_parity(a[name][finite], b[name][finite], np.float32, name)
        if where == "w" and n == 16:
            assert np.array_equal(np.isnan(a[name]), np.isnan(b[name])), name
            assert np.array_equal(a[name][np.isinf(b[name])], b[name][np.isinf(b[name])]), name
