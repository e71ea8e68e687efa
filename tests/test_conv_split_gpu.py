"""Forward-shaped launches with few tiles, whose K loop is split over CTAs and finished by a second kernel: every epilogue,
batch sums, scattered rows (strided input gradients), ragged channels and fully connected layers. GPU."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import conv_oracle as co
from pydtnn_b200 import _lib
from tests.gpu_util import DEV, assert_parity, dev, make_desc, run_conv, stream, workspace

pytestmark = pytest.mark.gpu

# (n, h, w, ci, co, k, pad, stride): one tile, one k-block per split and a short last one; two column tiles with a narrow
# last one; several row tiles with a ragged last one; a strided layer with scattered input gradient rows
SHAPES = [(1, 14, 14, 256, 256, 3, 1, 1), (1, 7, 7, 512, 520, 3, 1, 1), (2, 10, 9, 130, 68, 3, 1, 1), (1, 14, 14, 1024, 256, 1, 0, 1),
          (3, 12, 12, 96, 64, 5, 2, 2), (1, 15, 15, 256, 100, 3, 1, 2), (5, 1, 1, 4096, 1000, 1, 0, 1)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout,w_layout", [("NHWC", "KRSC"), ("NHWC", "CRSK"), ("NCHW", "KCRS")])
def test_split_launches(shape, layout, w_layout):
    n, h, w, ci, cout, k, pad, st = shape
    g = co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st)
    rng = np.random.Generator(np.random.PCG64(ci + cout))
    nchw = layout == "NCHW"
    x = rng.standard_normal((n, ci, h, w) if nchw else (n, h, w, ci)).astype(np.float32)
    wt = rng.standard_normal((cout, ci, k, k) if nchw else (ci, k, k, cout)).astype(np.float32) * np.float32(np.sqrt(2.0 / (ci * k * k)))
    b = rng.standard_normal(cout).astype(np.float32)
    dy = rng.standard_normal((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout)).astype(np.float32)
    x64, w64, b64, dy64 = (a.astype(np.float64) for a in (x, wt, b, dy))
    y = co.conv2d_forward(x64, w64, b64, g, layout)
    dw, db, dx = co.conv2d_backward(x64, dy64, w64, g, layout)
    out = run_conv(g, layout, np.float32, x, wt, b, dy, w_layout=w_layout, engine=_lib.ENGINE_TENSOR)
    for name, ref in (("y", y), ("dw", dw), ("db", db), ("dx", dx)):
        assert_parity(out[name].reshape(ref.shape), ref, np.float32, f"{name} {shape} {layout}")
    bn = {k_: rng.uniform(0.5, 1.5, cout).astype(np.float32) for k_ in ("running_mean", "inv_std", "gamma", "beta")}
    sh = (1, cout, 1, 1) if nchw else (1, 1, 1, cout)
    v = {k_: a.astype(np.float64).reshape(sh) for k_, a in bn.items()}
    fused = np.maximum((y - v["running_mean"]) * v["inv_std"] * v["gamma"] + v["beta"], 0)
    got = run_conv(g, layout, np.float32, x, wt, b, None, w_layout=w_layout, engine=_lib.ENGINE_TENSOR, bn=bn, relu=True, passes=("fprop",))
    assert_parity(got["y"], fused, np.float32, f"fused {shape} {layout}")


@pytest.mark.parametrize("shape", [(4, 4, 4, 512, 512, 3, 1, 1), (2, 7, 7, 256, 1024, 1, 0, 1), (1, 5, 5, 128, 36, 3, 1, 1)])
def test_batch_sums_of_split_launches(shape):
    n, h, w, ci, cout, k, pad, st = shape
    L = _lib.lib()
    g = co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st)
    desc = make_desc(g, "NHWC", np.float32, "KRSC")
    rng = np.random.Generator(np.random.PCG64(3))
    x = dev(rng.standard_normal((n, h, w, ci)).astype(np.float32))
    wt = dev((rng.standard_normal((cout, k, k, ci)) * np.sqrt(2.0 / (ci * k * k))).astype(np.float32))
    b = dev(rng.standard_normal(cout).astype(np.float32))
    nbytes = L.b2c_conv_stats_bytes(ctypes.byref(desc))
    rows = nbytes // (8 * cout)
    assert rows == (g.n * g.ho * g.wo + 31) // 32
    stats = torch.full((rows, 2, cout), float("nan"), device=DEV)
    y, y2 = (torch.full((n, g.ho, g.wo, cout), float("nan"), device=DEV) for _ in range(2))
    ws = workspace(desc)
    _lib.check(L.b2c_conv_fprop_stats(ctypes.byref(desc), x.data_ptr(), wt.data_ptr(), b.data_ptr(), y.data_ptr(), stats.data_ptr(),
                                      nbytes, ws.data_ptr(), ws.numel(), stream()))
    _lib.check(L.b2c_conv_fprop(ctypes.byref(desc), x.data_ptr(), wt.data_ptr(), b.data_ptr(), None, 0, y2.data_ptr(), ws.data_ptr(),
                                ws.numel(), stream()))
    assert torch.equal(y, y2)
    v = y.double().view(-1, cout)
    # a row of sums is at most 32 float32 additions per channel: 32 * 2^-24 of the sum of magnitudes
    for got, ref, mag in ((stats[:, 0], v, v.abs()), (stats[:, 1], v * v, v * v)):
        err = (got.double().sum(0) - ref.sum(0)).abs()
        assert bool((err <= 34 * 2.0 ** -24 * mag.sum(0)).all())


@pytest.mark.parametrize("n,hw,ci,cout,k,st,launches", [(33, 29, 128, 128, 3, 2, 1), (12, 28, 64, 64, 3, 1, 1), (2, 28, 128, 512, 3, 1, 1), (33, 15, 1024, 96, 1, 1, 1),
                                                        (1, 28, 512, 128, 1, 1, 2), (1, 7, 512, 2048, 1, 1, 2), (1, 56, 64, 64, 3, 1, 2),
                                                        (6, 28, 40, 128, 3, 1, 2), (12, 28, 100, 100, 3, 1, 2)])
def test_k_loops_are_split_where_that_pays(n, hw, ci, cout, k, st, launches):
    """Tiles on half of the chip or more with K loops of 18 to 36 k-blocks stay whole (one launch); the few tiles of one image are split."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes chosen for 148 SMs")
    L = _lib.lib()
    g = co.Geom(n, hw, hw, ci, cout, k, k, k // 2, k // 2, st, st)
    desc = make_desc(g, "NHWC", np.float32, "KRSC")
    gen = torch.Generator(device=DEV).manual_seed(ci)
    x, wt, b = (torch.randn(s, device=DEV, generator=gen) for s in ((n, hw, hw, ci), (cout, k, k, ci), (cout,)))
    y = torch.full((n, g.ho, g.wo, cout), float("nan"), device=DEV)
    ws = workspace(desc)
    before = L.b2c_launch_count()
    _lib.check(L.b2c_conv_fprop(ctypes.byref(desc), x.data_ptr(), wt.data_ptr(), b.data_ptr(), None, 0, y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    assert L.b2c_launch_count() - before == launches
    ref = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), wt.permute(0, 3, 1, 2).double(), b.double(), stride=st, padding=k // 2).permute(0, 2, 3, 1)
    assert_parity(y.cpu().numpy(), ref.cpu().numpy(), np.float32)
