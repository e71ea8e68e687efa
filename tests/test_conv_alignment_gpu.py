"""Few-channel layers on pointers that are not 16-byte aligned, and the lowered input that their forward pass leaves. GPU."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import conv_oracle as co
from pydtnn_b200 import _lib
from tests.gpu_util import DEV, make_desc, rel_l2, stream, workspace

pytestmark = pytest.mark.gpu


def _at(t, off):
    """A copy of ``t`` that starts ``off`` floats behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, device=DEV)
    v = buf[off:off + t.numel()].view(t.shape)
    v.copy_(t)
    return v


def _case(cout):
    g = co.Geom(4, 40, 40, 3, cout, 7, 7, 3, 3, 2, 2)
    gen = torch.Generator(device=DEV).manual_seed(5)
    x, w, b, dy = (torch.randn(s, device=DEV, generator=gen) for s in ((g.n, g.h, g.w, g.ci), (g.co, 7, 7, g.ci), (g.co,), (g.n, g.ho, g.wo, g.co)))
    return g, make_desc(g, "NHWC", np.float32, "KRSC"), x, w, b, dy


@pytest.mark.parametrize("cout", [64, 20, 18])
@pytest.mark.parametrize("off_x,off_y,off_dy", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (3, 2, 0)])
def test_weight_gradient_from_the_lowered_input(cout, off_x, off_y, off_dy):
    L = _lib.lib()
    g, desc, x, w, b, dy = _case(cout)
    assert L.b2c_conv_keeps_lowered_input(ctypes.byref(desc)) == 1
    ref = co.conv2d_backward(*(a.cpu().numpy().astype(np.float64) for a in (x, dy)), w.permute(3, 1, 2, 0).contiguous().cpu().numpy().astype(np.float64),
                             g, "NHWC")[0].transpose(3, 1, 2, 0)
    x, dy, y = _at(x, off_x), _at(dy, off_dy), _at(torch.empty_like(dy), off_y)
    ws = workspace(desc)
    ws.view(torch.float32).fill_(float("nan"))
    dw, db = torch.full_like(w, float("nan")), torch.empty_like(b)
    _lib.check(L.b2c_conv_fprop(ctypes.byref(desc), x.data_ptr(), w.data_ptr(), b.data_ptr(), None, 0, y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    rc = L.b2c_conv_wgrad_lowered(ctypes.byref(desc), x.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(), ws.data_ptr(), ws.numel(), stream())
    if rc == 0:
        assert rel_l2(dw.cpu().numpy(), ref) <= 1e-5
    else:
        assert off_dy and bool(torch.isnan(dw).all())           # dy is the one operand that may be refused


def test_forward_on_an_unaligned_y_needs_no_room_for_the_lowered_input():
    L = _lib.lib()
    g, desc, x, w, b, dy = _case(64)
    y, want = _at(torch.zeros_like(dy), 1), torch.empty_like(dy)
    fma = make_desc(g, "NHWC", np.float32, "KRSC", engine=_lib.ENGINE_FMA)
    ws = torch.empty(max(256, L.b2c_conv_workspace_bytes(ctypes.byref(fma), _lib.PASS_FPROP)), dtype=torch.uint8, device=DEV)
    for d, out in ((desc, y), (fma, want)):
        _lib.check(L.b2c_conv_fprop(ctypes.byref(d), x.data_ptr(), w.data_ptr(), b.data_ptr(), None, 0, out.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    assert torch.equal(y, want)
    dw = torch.empty_like(w)
    assert L.b2c_conv_wgrad_lowered(ctypes.byref(desc), x.data_ptr(), dy.data_ptr(), dw.data_ptr(), None, ws.data_ptr(), ws.numel(), stream()) != 0


def test_forward_with_batch_sums_reads_x_anywhere():
    L = _lib.lib()
    g, desc, x, w, b, dy = _case(64)
    ws, out = workspace(desc), []
    nbytes = L.b2c_conv_stats_bytes(ctypes.byref(desc))
    for off in (0, 1):
        xo, y, st = _at(x, off), torch.empty_like(dy), torch.zeros(nbytes // 4, device=DEV)
        _lib.check(L.b2c_conv_fprop_stats(ctypes.byref(desc), xo.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), st.data_ptr(), nbytes,
                                          ws.data_ptr(), ws.numel(), stream()))
        out.append((y, st))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
