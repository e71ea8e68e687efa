"""Channel counts that fill no block of 32, no 16-byte pixel or neither, on the tensor-core engine: all three passes
against the CPU oracle, both layouts and every filter layout, at the float32 bar. GPU."""
import ctypes

import numpy as np
import pytest

from oracle import conv_oracle as co
from pydtnn_b200 import _lib
from tests.gpu_util import assert_parity, make_desc, run_conv

pytestmark = pytest.mark.gpu

# (n, h, w, ci, co, k, pad, stride): one channel; one to three channels past a block; one short of a block; several blocks
# and a remainder of each length; column tiles of 64 and 128 with few columns left; even images, strides and 1x1 / 2
SHAPES = [(2, 9, 7, 1, 1, 3, 1, 1), (2, 9, 7, 4, 4, 3, 1, 1), (3, 8, 8, 8, 36, 3, 1, 1), (2, 11, 6, 17, 33, 3, 1, 2),
          (2, 12, 12, 20, 12, 5, 2, 1), (1, 10, 9, 30, 31, 3, 1, 1), (2, 7, 9, 33, 130, 1, 0, 1), (3, 15, 11, 40, 72, 3, 1, 1),
          (2, 9, 9, 36, 1, 3, 1, 2), (2, 13, 13, 65, 100, 1, 0, 2), (2, 14, 14, 48, 80, 5, 2, 2), (1, 9, 30, 129, 67, 3, 1, 1),
          (2, 6, 6, 100, 260, 3, 1, 1), (2, 17, 17, 3, 10, 7, 3, 2), (40, 5, 5, 12, 24, 3, 0, 1), (2, 8, 8, 16, 16, 3, 1, 1),
          (4, 61, 53, 12, 192, 3, 1, 1), (8, 61, 53, 4, 64, 3, 1, 1)]      # whole 16-byte pixels, large enough to be lowered

@pytest.mark.parametrize("layout,w_layout", [("NHWC", "KRSC"), ("NHWC", "CRSK"), ("NCHW", "KCRS")])
@pytest.mark.parametrize("shape", SHAPES)
def test_ragged_channels(shape, layout, w_layout):
    n, h, w, ci, cout, k, pad, st = shape
    g = co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st)
    desc = make_desc(g, layout, np.float32, w_layout, engine=_lib.ENGINE_TENSOR)
    assert all(_lib.lib().b2c_conv_engine_for(ctypes.byref(desc), p) == _lib.ENGINE_TENSOR for p in range(3))
    rng = np.random.Generator(np.random.PCG64(ci * 1000 + cout))
    nchw = layout == "NCHW"
    x = rng.standard_normal((n, ci, h, w) if nchw else (n, h, w, ci)).astype(np.float32)
    wt = rng.standard_normal((cout, ci, k, k) if nchw else (ci, k, k, cout)).astype(np.float32) * np.float32(np.sqrt(2.0 / (ci * k * k)))
    b = rng.standard_normal(cout).astype(np.float32)
    dy = rng.standard_normal((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout)).astype(np.float32)
    x64, w64, b64, dy64 = (a.astype(np.float64) for a in (x, wt, b, dy))
    y = co.conv2d_forward(x64, w64, b64, g, layout)
    dw, db, dx = co.conv2d_backward(x64, dy64, w64, g, layout)
    bn = {k_: rng.uniform(0.5, 1.5, cout).astype(np.float32) for k_ in ("running_mean", "inv_std", "gamma", "beta")}
    out = run_conv(g, layout, np.float32, x, wt, b, dy, w_layout=w_layout, engine=_lib.ENGINE_TENSOR)
    for name, ref in (("y", y), ("dw", dw), ("db", db), ("dx", dx)):
        assert_parity(out[name].reshape(ref.shape), ref, np.float32, f"{name} {shape} {layout} {w_layout}")
    sh = (1, cout, 1, 1) if nchw else (1, 1, 1, cout)
    v = {k_: a.astype(np.float64).reshape(sh) for k_, a in bn.items()}
    fused = np.maximum((y - v["running_mean"]) * v["inv_std"] * v["gamma"] + v["beta"], 0)
    got = run_conv(g, layout, np.float32, x, wt, b, None, w_layout=w_layout, engine=_lib.ENGINE_TENSOR, bn=bn, relu=True, passes=("fprop",))
    assert_parity(got["y"], fused, np.float32, f"fused {shape} {layout}")


@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
@pytest.mark.parametrize("n,h,w,ci,cout,kh,kw", [(1, 7, 6, 203, 190, 3, 2), (2, 6, 5, 64, 600, 1, 3), (1, 9, 9, 130, 300, 5, 5), (1, 9, 8, 33, 1070, 8, 8)])
def test_weight_gradient_of_wide_kcrs_filters(n, h, w, ci, cout, kh, kw, layout):
    """(co, ci, kh, kw) filters large enough for the second stage that takes all taps of four channels: 2 to 64 taps, channel
    counts that end inside its blocks."""
    g = co.Geom(n, h, w, ci, cout, kh, kw, 1, 1, 1, 1)
    rng = np.random.Generator(np.random.PCG64(ci))
    nchw = layout == "NCHW"
    x = rng.standard_normal((n, ci, h, w) if nchw else (n, h, w, ci)).astype(np.float32)
    wt = np.zeros((cout, ci, kh, kw) if nchw else (ci, kh, kw, cout), np.float32)
    dy = rng.standard_normal((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout)).astype(np.float32)
    dw, db, _ = co.conv2d_backward(x.astype(np.float64), dy.astype(np.float64), wt.astype(np.float64), g, layout)
    out = run_conv(g, layout, np.float32, x, wt, np.zeros(cout, np.float32), dy, w_layout="KCRS", engine=_lib.ENGINE_TENSOR, passes=("wgrad",))
    for name, ref in (("dw", dw), ("db", db)):
        assert_parity(out[name].reshape(ref.shape), ref, np.float32, name)
