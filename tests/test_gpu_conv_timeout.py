"""The time-out path of the fused convolution: every wait gives up at once, with the copies of the weights and of
the first boxes in flight. The call returns, reports it, and the next one gives what the one before gave."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,w", [(1, 8, 8), (5, 70, 70)])  # fewer tiles than SMs, several to an SM
def test_waits_that_give_up_end_the_kernel_with_a_status(cuda_lib, b, h, w):
    import torch

    def p(t):
        return ctypes.c_void_p(t.data_ptr())

    g = torch.Generator(device="cuda").manual_seed(1)
    act = torch.randn((b * h * w, 64), device="cuda", generator=g).to(torch.bfloat16)
    wgt = (torch.randn((64, 576), device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    none = ctypes.c_void_p(0)

    def conv():
        out = torch.empty((b * h * w, 64), device="cuda", dtype=torch.bfloat16)
        st = torch.zeros(4, device="cuda", dtype=torch.int32)
        assert cuda_lib.wg_pc_conv(0, p(act), b, h, w, 1, p(wgt), 576, none, none, none, p(out), p(st), None) == 0
        torch.cuda.synchronize()
        assert int(st[0]) == 0
        return out

    before = conv()
    st = torch.zeros(4, device="cuda", dtype=torch.int32)
    scratch = torch.empty_like(before)
    assert cuda_lib.wg_selftest_conv_timeout(p(act), b, h, w, p(wgt), p(scratch), p(st), None) == 0
    torch.cuda.synchronize()
    assert int(st[0]) != 0
    assert torch.equal(conv(), before)
