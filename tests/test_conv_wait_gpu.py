"""Bounded waits of the tensor-core convolution behind a kernel that lets its dependents start at once and then runs longer than the
waits' limit of about a second: the launch must not count that time as its own. GPU."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import conv_oracle as co
from pydtnn_b200 import _lib
from tests.gpu_util import DEV, assert_parity, make_desc, stream, workspace

pytestmark = pytest.mark.gpu

# One thread that has its dependents started and then sleeps for `ns` nanoseconds (the loop also ends by itself)
HOLD = r"""
extern "C" __global__ void hold(long long ns)
{
    long long t0, t;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (int i = 0; i < (1 << 24); i++) {
        __nanosleep(1000);
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t - t0 > ns) break;
    }
}
"""
HOLD_NS = 1_400_000_000          # the limit is 2e9 cycles, 1.02 s at the boost clock

# (n, h, w, ci, co, k): the roles that wait differ in these forms of the kernel
CASES = [
    ("fprop", (55, 17, 17, 128, 128, 3)),       # pairs of CTAs
    ("fprop", (8, 14, 14, 256, 256, 3)),        # single CTAs, B tiles split by warps of their own
    ("fprop", (16, 28, 28, 64, 256, 1)),        # filter tiles resident for the launch
    ("fprop", (4, 20, 20, 40, 72, 3)),          # fine sums
    ("wgrad", (16, 28, 28, 128, 128, 3)),       # with the bias gradient
]


@pytest.mark.parametrize("what,shape", CASES)
def test_waits_do_not_count_the_kernel_in_front(what, shape):
    n, h, w, ci, cout, k = shape
    L = _lib.lib()
    g = co.Geom(n, h, w, ci, cout, k, k, k // 2, k // 2, 1, 1)
    desc = make_desc(g, "NHWC", np.float32, "KRSC")
    gen = torch.Generator(device=DEV).manual_seed(k + ci)
    rnd = lambda *s: torch.randn(s, device=DEV, generator=gen)
    x, dy, wt, b = rnd(n, h, w, ci), rnd(n, h, w, cout), rnd(cout, k, k, ci), rnd(cout)
    ws = workspace(desc)

    def run(out):
        d = ctypes.byref(desc)
        if what == "fprop":
            _lib.check(L.b2c_conv_fprop(d, x.data_ptr(), wt.data_ptr(), b.data_ptr(), None, 0, out[0].data_ptr(), ws.data_ptr(), ws.numel(), stream()))
        else:
            _lib.check(L.b2c_conv_wgrad(d, x.data_ptr(), dy.data_ptr(), out[0].data_ptr(), out[1].data_ptr(), ws.data_ptr(), ws.numel(), stream()))

    want, out = ([torch.full_like(t, float("nan")) for t in ((dy,) if what == "fprop" else (wt, b))] for _ in range(2))
    run(want)
    hold = torch.cuda._compile_kernel(HOLD, "hold")
    torch.cuda.synchronize()
    a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    hold((1, 1, 1), (1, 1, 1), (HOLD_NS,))
    run(out)                         # right behind it in the stream
    e.record()
    torch.cuda.synchronize()
    status = ctypes.c_int()
    _lib.check(L.b2c_check_device_status(ctypes.byref(status)))
    assert status.value == 0
    assert a.elapsed_time(e) > 1100.0
    for first, again in zip(want, out):
        assert torch.equal(first, again)
    if what == "fprop":
        ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double().permute(0, 3, 1, 2), b.double(), padding=k // 2).permute(0, 2, 3, 1)
        assert_parity(want[0].cpu().numpy(), ref.cpu().numpy(), np.float32, f"{shape}")
