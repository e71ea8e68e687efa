"""The float4 pooling kernel where its windows leave the image (padding, dilation, ragged strides), with several blocks per row,
more rows than a grid axis has, and without the tap numbers, against the general kernel on channels it takes (c not a
multiple of 4 runs there): bit for bit. GPU."""
import pytest
import torch

from pydtnn_b200 import _lib
from tests.gpu_util import DEV, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("is_max", [1, 0])
@pytest.mark.parametrize("n,h,w,c,k,pad,st,dil", [(2, 9, 7, 8, (3, 3), (1, 1), (2, 2), (1, 1)), (3, 8, 13, 4, (2, 3), (0, 1), (1, 2), (2, 3)),
                                                  (1, 7, 7, 2048, (7, 7), (0, 0), (1, 1), (1, 1)), (2, 5, 300, 16, (3, 2), (1, 0), (1, 1), (1, 1)),
                                                  (2, 6, 6, 12, (5, 5), (2, 2), (3, 3), (1, 1)), (1100, 60, 3, 4, (1, 3), (0, 1), (1, 1), (1, 1))])
def test_forward_equals_the_general_kernel(n, h, w, c, k, pad, st, dil, is_max):
    L = _lib.lib()
    ho, wo = ((s + 2 * p - d * (kk - 1) - 1) // t + 1 for s, p, d, kk, t in ((h, pad[0], dil[0], k[0], st[0]), (w, pad[1], dil[1], k[1], st[1])))
    gen = torch.Generator(device=DEV).manual_seed(h * w)
    x = torch.randn(n, h, w, c, device=DEV, generator=gen)

    def run(xt, with_idx=True):
        ch = xt.shape[3]
        y = torch.full((n, ho, wo, ch), float("nan"), device=DEV)
        idx = torch.full((n, ho, wo, ch), -1, dtype=torch.int32, device=DEV) if with_idx and is_max else None
        _lib.check(L.b2c_pool_forward(_lib.F32, _lib.LAYOUT_NHWC, is_max, n, h, w, ch, *k, *pad, *st, *dil, xt.data_ptr(), y.data_ptr(),
                                      idx.data_ptr() if idx is not None else None, stream()))
        return y, idx
    y, idx = run(x)
    wide = torch.cat([x, x[..., :1]], dim=3).contiguous()          # c + 1 channels: the general kernel
    y2, idx2 = run(wide)
    assert torch.equal(y, y2[..., :c]) and torch.equal(run(x, False)[0], y)
    if is_max:
        assert torch.equal(idx, idx2[..., :c])
