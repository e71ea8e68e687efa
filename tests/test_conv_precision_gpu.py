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
@pytest.mark.parametrize("shape", [(9, 13, 13, 64, 64, 1, 0, 1), (2, 8, 8, 64, 128, 3, 1, 1), (1, 7, 7, 256, 64, 3, 1, 1), (2, 9, 9, 64, 64, 3, 1, 2),
                                   (2, 9, 9, 64, 96, 1, 0, 2), (2, 9, 9, 64, 64, 2, 0, 3), (16, 20, 20, 256, 128, 1, 0, 1)])
@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
def test_filters_with_inner_taps_are_split_by_rounding(shape, layout):
    """One product per output, both factors 1 + 2^-10 - 2^-23: with the filter's upper half rounded the dropped product of the
    lower halves is nothing, with a truncated one it is 2^-20."""
    n, h, w, ci, cout, k, pad, st = shape
    g = co.Geom(n, h, w, ci, cout, k, k, pad, pad, st, st)
    desc = make_desc(g, layout, np.float32, "KCRS", engine=_lib.ENGINE_TENSOR)
    assert _lib.lib().b2c_conv_engine_for(ctypes.byref(desc), _lib.PASS_FPROP) == _lib.ENGINE_TENSOR
    v = np.float32(1 + 2.0 ** -10 - 2.0 ** -23)
    nchw = layout == "NCHW"
    wt = np.zeros((ci, k, k, cout), np.float32)
    m = min(ci, cout)
    wt[np.arange(m), k // 2, k // 2, np.arange(m)] = v
    x = np.full((n, ci, h, w) if nchw else (n, h, w, ci), v)
    dy = np.full((n, cout, g.ho, g.wo) if nchw else (n, g.ho, g.wo, cout), v)
    out = run_conv(g, layout, np.float32, x, wt.transpose(3, 0, 1, 2) if nchw else wt, None, dy, w_layout="KCRS", engine=_lib.ENGINE_TENSOR,
                   passes=("fprop", "dgrad"))
    want = float(v) ** 2
    for name in ("y", "dx"):
        got = out[name].astype(np.float64)
        got = got[got != 0]
        assert got.size
        # the other operand's lower half loses its last two bits (3 * 2^-23 at most), each of the two sums at most one more
        assert np.abs(got / want - 1).max() <= 5 * 2.0 ** -23, (name, np.abs(got / want - 1).max())
