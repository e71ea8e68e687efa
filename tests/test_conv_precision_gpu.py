"""What the tensor-core engine loses of float32 products and sums. GPU."""
import ctypes

import numpy as np
import pytest

from oracle import conv_oracle as co
from pydtnn_b200 import _lib
from tests.gpu_util import make_desc, run_conv

pytestmark = pytest.mark.gpu


# (n, h, w, ci, co, k, pad, stride): resident filters, streamed ones, the split K loop, classes in one launch, class (0, 0) alone,
# a launch per class
INNER = [(9, 13, 13, 64, 64, 1, 0, 1), (2, 8, 8, 64, 128, 3, 1, 1), (1, 7, 7, 256, 64, 3, 1, 1), (2, 9, 9, 64, 64, 3, 1, 2),
         (2, 9, 9, 64, 96, 1, 0, 2), (2, 9, 9, 64, 64, 2, 0, 3), (16, 20, 20, 256, 128, 1, 0, 1)]
# few channels, read in place and lowered
FEW = [(8, 20, 20, 16, 36, 1, 0, 1), (8, 20, 20, 12, 20, 3, 1, 2), (8, 20, 20, 3, 20, 3, 1, 1)]


@pytest.mark.parametrize("shape,layout,w_layout", [(s, l, "KCRS") for s in INNER for l in ("NHWC", "NCHW")] + [(s, "NHWC", l) for s in FEW for l in ("KRSC", "CRSK")])
def test_filters_are_split_by_rounding(shape, layout, w_layout):
    """One product per output, both factors 1 + 2^-10 - 2^-23: with the filter's upper half rounded the dropped product of the
    lower halves is nothing, with a truncated one it is 2^-20."""
    n, h, w, ci, cout, k, pad, st = shape
    g = co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st)
    desc = make_desc(g, layout, np.float32, w_layout, engine=_lib.ENGINE_TENSOR)
    assert _lib.lib().b2c_conv_engine_for(ctypes.byref(desc), _lib.PASS_FPROP) == _lib.ENGINE_TENSOR
    v = np.float32(1 + 2.0 ** -10 - 2.0 ** -23)
    nchw = layout == "NCHW"
    wt = np.zeros((ci, k, k, cout), np.float32)
    m = min(ci, cout)
    wt[np.arange(m), k // 2, k // 2, np.arange(m)] = v
    x = np.full((n, ci, h, w) if nchw else (n, h, w, ci), v)
    dy = np.full((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout), v)
    out = run_conv(g, layout, np.float32, x, wt.transpose(3, 0, 1, 2) if nchw else wt, None, dy, w_layout=w_layout, engine=_lib.ENGINE_TENSOR,
                   passes=("fprop", "dgrad"))
    want = float(v) ** 2
    for name in ("y", "dx") if w_layout == "KCRS" else ("y",):
        got = out[name].astype(np.float64)
        got = got[got != 0]
        assert got.size
        # the other operand's lower half loses its last two bits (3 * 2^-23 at most), each of the two sums at most one more
        assert np.abs(got / want - 1).max() <= 5 * 2.0 ** -23, (name, np.abs(got / want - 1).max())


def _errors(out, refs):
    return {k: float(np.linalg.norm(out[k].astype(np.float64).reshape(r.shape) - r) / np.linalg.norm(r)) for k, r in refs.items()}


# (layout, n, h, w, ci, co, k, pad, stride): channel counts that are no whole blocks (lowered, one to several blocks, strided: all
# classes in one launch, one class, a launch per class), whole blocks on NCHW images too small for the copies, one-pixel images
@pytest.mark.parametrize("shape", [("NHWC", 9, 30, 17, 40, 72, 3, 1, 1), ("NCHW", 3, 16, 16, 3, 20, 3, 1, 1), ("NHWC", 2, 14, 14, 132, 70, 5, 2, 2),
                                   ("NCHW", 5, 9, 9, 36, 100, 3, 1, 2), ("NHWC", 4, 9, 9, 40, 48, 1, 0, 2), ("NHWC", 4, 11, 11, 50, 24, 2, 0, 3),
                                   ("NCHW", 1, 14, 14, 256, 256, 1, 0, 2), ("NHWC", 96, 1, 1, 520, 384, 1, 0, 1), ("NHWC", 8, 8, 8, 423, 512, 3, 1, 1),
                                   ("NCHW", 12, 10, 10, 256, 9, 3, 1, 1), ("NCHW", 6, 28, 28, 1, 16, 3, 1, 1)])
def test_passes_that_sum_like_the_fma_engine(shape):
    """Where the tensor-core engine takes over from the FMA engine it is no further from float64.  On top of the FMA engine's own
    error on the same inputs: one rounding (2^-24) for its shorter chains on the smallest sums."""
    layout, n, h, w, ci, cout, k, pad, st = shape
    g = co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st)
    rng = np.random.Generator(np.random.PCG64(ci + cout))
    nchw = layout == "NCHW"
    x = rng.standard_normal((n, ci, h, w) if nchw else (n, h, w, ci)).astype(np.float32)
    wt = rng.standard_normal((cout, ci, k, k) if nchw else (ci, k, k, cout)).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    dy = rng.standard_normal((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout)).astype(np.float32)
    x64, w64, b64, dy64 = (a.astype(np.float64) for a in (x, wt, b, dy))
    refs = dict(zip(("y", "dw", "db", "dx"), (co.conv2d_forward(x64, w64, b64, g, layout), *co.conv2d_backward(x64, dy64, w64, g, layout))))
    w_layout = "KCRS" if nchw else "KRSC"
    desc = make_desc(g, layout, np.float32, w_layout)
    assert any(_lib.lib().b2c_conv_engine_for(ctypes.byref(desc), p) == _lib.ENGINE_TENSOR for p in range(3))
    got = _errors(run_conv(g, layout, np.float32, x, wt, b, dy, w_layout=w_layout), refs)
    fma = _errors(run_conv(g, layout, np.float32, x, wt, b, dy, w_layout=w_layout, engine=_lib.ENGINE_FMA), refs)
    for name in refs:
        assert got[name] <= fma[name] + 2.0 ** -24, (name, got, fma)


def test_short_ranges_are_not_made_longer():
    """A launch that balanced ranges cut into 5.4 k-blocks per CTA keeps that advantage (6 of 8 products per sum in tensor memory, and
    an error in proportion) over one large enough for whole tiles, whose sums are all of 8 k-blocks."""
    rng = np.random.Generator(np.random.PCG64(7))
    wt = (rng.standard_normal((256, 5, 5, 128)) / 80).astype(np.float32)
    err = []
    for n in (2, 40):
        g = co.Geom(n, 15, 15, 256, 128, 5, 5, 2, 2, 1, 1)
        x = rng.standard_normal((n, 15, 15, 256)).astype(np.float32)
        y = run_conv(g, "NHWC", np.float32, x, wt, None, None, w_layout="KRSC", passes=("fprop",))["y"][:2]
        ref = co.conv2d_forward(x[:2].astype(np.float64), wt.astype(np.float64), np.zeros(128), co.Geom(2, 15, 15, 256, 128, 5, 5, 2, 2, 1, 1), "NHWC")
        err.append(np.linalg.norm(y - ref) / np.linalg.norm(ref))
    assert err[0] <= 0.9 * err[1], err


@pytest.mark.parametrize("shape", [("NHWC", 2, 12, 9, 40, 72, 3, 1, 1), ("NCHW", 2, 11, 11, 36, 100, 3, 1, 2), ("NHWC", 64, 1, 1, 520, 384, 1, 0, 1),
                                   ("NCHW", 2, 16, 16, 3, 21, 5, 2, 1), ("NHWC", 1, 8, 8, 423, 130, 3, 1, 1)])
@pytest.mark.parametrize("where", ["x", "w", "dy"])
def test_infinities_come_out_as_from_fmas(shape, where):
    """Passes that came from the FMA engine answer infinities and NaNs in the same places."""
    layout, n, h, w, ci, cout, k, pad, st = shape
    g = co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st)
    rng = np.random.Generator(np.random.PCG64(ci))
    nchw = layout == "NCHW"
    t = {"x": rng.standard_normal((n, ci, h, w) if nchw else (n, h, w, ci)).astype(np.float32),
         "w": rng.standard_normal((cout, ci, k, k) if nchw else (ci, k, k, cout)).astype(np.float32),
         "dy": rng.standard_normal((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout)).astype(np.float32)}
    # operands that tf32 holds exactly (no lower half), zeros among them, and those that it does not
    for name in t:
        t[name].flat[::3] = np.float32(1.5) * np.sign(t[name].flat[::3])
        t[name].flat[::50] = 0
    bad = t[where].reshape(-1)
    bad[bad.size // 3], bad[bad.size // 2 + 1], bad[bad.size - 2] = np.inf, -np.inf, np.nan
    w_layout = "KCRS" if nchw else "KRSC"
    a, b = (run_conv(g, layout, np.float32, t["x"], t["w"], None, t["dy"], w_layout=w_layout, engine=e) for e in (_lib.ENGINE_AUTO, _lib.ENGINE_FMA))
    for name in ("y", "dw", "dx"):
        assert np.array_equal(np.isnan(a[name]), np.isnan(b[name])), name
        assert np.array_equal(np.isinf(a[name]), np.isinf(b[name])), name
        assert np.array_equal(a[name][np.isinf(b[name])], b[name][np.isinf(b[name])]), name
