"""The residual sum + ReLU folded into the convolution that ends a branch (evaluation): the same bits as the convolution followed
by the add + ReLU kernel, on every epilogue it can run in. GPU."""
import ctypes

import numpy as np
import pytest
import torch

from pydtnn_b200 import _lib
from tests.gpu_util import DEV, stream

pytestmark = pytest.mark.gpu

# resident filters with 2 and 4 k-blocks and 64 columns; 8 k-blocks in one chunk; long K; balanced ranges; split with the plain
# and the deep second stage; ragged channels; a stem on the lowered matrix
SHAPES = [(2, 56, 56, 64, 256, 1), (3, 28, 28, 128, 512, 1), (8, 56, 56, 64, 64, 1), (40, 14, 14, 256, 1024, 1), (32, 28, 28, 128, 128, 3),
          (64, 14, 14, 256, 256, 3), (1, 14, 14, 1024, 256, 1), (4, 14, 14, 512, 512, 3), (3, 17, 13, 40, 72, 3), (2, 20, 20, 3, 12, 5)]


@pytest.mark.parametrize("n,h,w,ci,co,k", SHAPES)
@pytest.mark.parametrize("bn,relu", [(True, 1), (False, 1), (True, 0)])
def test_residual_epilogue_is_bit_identical(n, h, w, ci, co, k, bn, relu):
    L = _lib.lib()
    gen = torch.Generator(device=DEV).manual_seed(ci + co)
    d = _lib.ConvDesc(_lib.LAYOUT_NHWC, _lib.F32, _lib.W_KRSC, _lib.ENGINE_AUTO, n, h, w, ci, co, k, k, k // 2, k // 2, 1, 1, 1, 1)
    assert L.b2c_conv_takes_addend(ctypes.byref(d)) == 1

    def rnd(*s):
        return torch.randn(s, generator=gen, device=DEV)
    x, wt, b, other = rnd(n, h, w, ci), rnd(co, k, k, ci) * (2.0 / (ci * k * k)) ** 0.5, rnd(co), rnd(n, h, w, co)
    vecs = [rnd(co), rnd(co).abs() + 0.5, rnd(co), rnd(co)]
    p = ctypes.byref(_lib.BnParams(*[v.data_ptr() for v in vecs])) if bn else None
    ws = torch.empty(max(256, L.b2c_conv_workspace_bytes(ctypes.byref(d), 0)), dtype=torch.uint8, device=DEV)
    y, want, got = (torch.full((n, h, w, co), float("nan"), device=DEV) for _ in range(3))
    a = (ctypes.byref(d), x.data_ptr(), wt.data_ptr(), b.data_ptr(), p)
    _lib.check(L.b2c_conv_fprop(*a, 0, y.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    if relu:
        _lib.check(L.b2c_add_relu(_lib.F32, y.numel(), y.data_ptr(), other.data_ptr(), want.data_ptr(), stream()))
    else:
        want = y + other
    _lib.check(L.b2c_conv_fprop_residual(*a, other.data_ptr(), relu, got.data_ptr(), ws.data_ptr(), ws.numel(), stream()))
    assert torch.equal(got, want)


def test_paths_that_cannot_say_so():
    L = _lib.lib()
    t = torch.zeros(4096, device=DEV)
    for layout, dt, co in ((_lib.LAYOUT_NCHW, _lib.F32, 32), (_lib.LAYOUT_NHWC, _lib.F64, 32), (_lib.LAYOUT_NHWC, _lib.F32, 30)):
        d = _lib.ConvDesc(layout, dt, _lib.W_KRSC, _lib.ENGINE_AUTO, 1, 4, 4, 32, co, 1, 1, 0, 0, 1, 1, 1, 1)
        assert L.b2c_conv_takes_addend(ctypes.byref(d)) == 0
        q = t.data_ptr()
        assert L.b2c_conv_fprop_residual(ctypes.byref(d), q, q, None, None, q, 1, q, q, 16384, stream()) == -6


@pytest.mark.parametrize("fmt", ["NHWC", "NCHW"])
def test_evaluation_with_folded_sums_is_bit_identical(fmt):
    from pydtnn_b200 import nets
    from pydtnn_b200.model import Model
    outs = []
    for fold in (True, False):
        np.random.seed(3)
        m = Model(batch_size=3, tensor_format=fmt, enable_fused_conv_bn=True, enable_fused_conv_bn_relu=True)
        nets.create_resnet50_imagenet(m, input_hw=40, nclasses=10, layout=[[16, 2, 1], [32, 2, 2]])
        for layer in m.layers:
            if layer.canonical_name == "AdditionBlock":
                layer.fold_sum = fold
        for layer in m.get_all_layers():
            if layer.canonical_name == "BatchNormalization":
                layer.running_var.ary.t.fill_(1.3)
        x = np.random.standard_normal((3, *m.layers[0].shape)).astype(np.float32)
        outs.append([m.evaluate_batch(x).ary.get().copy() for _ in range(4)])
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
