"""The update network's separate passes (transposes, casts, sums, ReLU masks, one layer's Adam) against their
definitions, and as the unfused route that the fused convolutions equal bit for bit: im2col columns, the
tensor-core GEMM and these passes only."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


NONE = ctypes.c_void_p(0)


def _bf16(*shape, g, scale=1.0):
    import torch

    return (torch.randn(shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 13), (64, 64), (129, 72), (33, 576)])
def test_transpose(cuda_lib, rows, cols):
    import torch

    x = _bf16(rows, cols, g=torch.Generator(device="cuda").manual_seed(rows))
    out = torch.empty((cols, rows), device="cuda", dtype=torch.bfloat16)
    assert cuda_lib.wg_pc_transpose_bf16(_p(x), rows, cols, _p(out), None) == 0
    assert torch.equal(out, x.t())


@pytest.mark.parametrize("rows,ld,cols", [(1, 1, 1), (37, 64, 64), (50, 64, 16), (9, 5, 3)])
def test_cast_add_and_mask(cuda_lib, rows, ld, cols):
    import torch

    g = torch.Generator(device="cuda").manual_seed(rows)
    x, y = (torch.randn((rows, ld), device="cuda", generator=g) for _ in range(2))
    for relu in (0, 1):
        out = torch.empty((rows, cols), device="cuda", dtype=torch.bfloat16)
        assert cuda_lib.wg_pc_cast_bf16(_p(x), rows, ld, cols, relu, _p(out), None) == 0
        want = x[:, :cols].clamp_min(0.0) if relu else x[:, :cols]
        assert torch.equal(out, want.to(torch.bfloat16))
    total, t16 = torch.empty_like(x), torch.empty((rows, ld), device="cuda", dtype=torch.bfloat16)
    assert cuda_lib.wg_pc_add(_p(x), _p(y), rows * ld, _p(total), _p(t16), None) == 0
    assert torch.equal(total, x + y) and torch.equal(t16, (x + y).to(torch.bfloat16))
    assert cuda_lib.wg_pc_add(_p(x), _p(y), rows * ld, _p(total), NONE, None) == 0
    mask = y.to(torch.bfloat16)
    assert cuda_lib.wg_pc_relu_grad(_p(x), _p(mask), rows * ld, _p(total), None) == 0
    assert torch.equal(total, torch.where(mask.float() > 0, x, 0.0))


def test_adam_of_one_layer_is_that_of_the_layers_call(cuda_lib):
    import torch

    n, kp, splits = 64, 128, 5
    g = torch.Generator(device="cuda").manual_seed(4)
    part = torch.randn((splits, kp, n), device="cuda", generator=g)
    start = [torch.randn((n, kp), device="cuda", generator=g) for _ in range(2)] + [torch.rand((n, kp), device="cuda", generator=g)]
    runs = []
    for layers in (False, True):
        w, m, v = (t.clone() for t in start)
        q, qt = torch.empty((n, kp), device="cuda", dtype=torch.bfloat16), torch.empty((kp, n), device="cuda", dtype=torch.bfloat16)
        if layers:
            def one(t):
                return (ctypes.c_void_p * 1)(t.data_ptr())

            def num(i):
                return (ctypes.c_int * 1)(i)

            assert cuda_lib.wg_pc_adam_layers(1, one(part), num(splits), num(n), num(kp), one(w), one(m), one(v), None, one(q), one(qt),
                                              1e-3, 0.9, 0.999, 1e-8, 2, None) == 0
        else:
            assert cuda_lib.wg_pc_adam(_p(part), splits, n, kp, _p(w), _p(m), _p(v), 1e-3, 0.9, 0.999, 1e-8, 2, _p(q), _p(qt), None) == 0
        torch.cuda.synchronize()
        runs.append((w, m, v, q, qt))
    assert not torch.equal(runs[0][0], start[0])
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("b,h,w,dil", [(1, 3, 5, 8), (3, 7, 13, 2), (2, 16, 12, 1), (5, 70, 70, 4)])
def test_the_unfused_route_equals_the_fused_convolutions(cuda_lib, b, h, w, dil):
    import torch

    lib, M = cuda_lib, b * h * w
    g = torch.Generator(device="cuda").manual_seed(M)
    act, mask, wgt = _bf16(M, 64, g=g), _bf16(M, 64, g=g), _bf16(64, 576, g=g, scale=0.05)
    add = torch.randn((M, 64), device="cuda", generator=g)
    st = torch.zeros(4, device="cuda", dtype=torch.int32)

    def f32(*shape):
        return torch.full(shape, float("nan"), device="cuda")

    def b16(*shape):
        return torch.full(shape, float("nan"), device="cuda", dtype=torch.bfloat16)

    def conv(mode, weights, add=None, mask=None):
        o32, o16 = f32(M, 64), b16(M, 64)
        assert lib.wg_pc_conv(mode, _p(act), b, h, w, dil, _p(weights), 576, _p(add) if add is not None else NONE,
                              _p(mask) if mask is not None else NONE, _p(o32), _p(o16), _p(st), None) == 0
        return o32, o16

    # forward: columns, product, then a cast with ReLU or the residual sum with its bf16 copy
    col, y = b16(M, 576), f32(M, 64)
    assert lib.wg_pc_im2col(_p(act), b, h, w, 64, dil, 576, _p(col), None) == 0
    assert lib.wg_gemm_bf16_dev(_p(col), _p(wgt), _p(y), M, 64, 576, 1, _p(st), None) == 0
    u32, u16 = f32(M, 64), b16(M, 64)
    assert lib.wg_pc_cast_bf16(_p(y), M, 64, 64, 1, _p(u16), None) == 0
    assert torch.equal(conv(0, wgt)[1], u16)
    assert lib.wg_pc_add(_p(add), _p(y), M * 64, _p(u32), _p(u16), None) == 0
    o32, o16 = conv(2, wgt, add=add)
    assert torch.equal(o32, u32) and torch.equal(o16, u16)
    # data gradient: the transposed weights' product, scattered back over the taps, then sum and mask
    wt, dcol, dx = b16(576, 64), f32(M, 576), f32(M, 64)
    assert lib.wg_pc_transpose_bf16(_p(wgt), 64, 576, _p(wt), None) == 0
    assert lib.wg_gemm_bf16_dev(_p(act), _p(wt), _p(dcol), M, 576, 64, 1, _p(st), None) == 0
    assert lib.wg_pc_col2im(_p(dcol), b, h, w, 64, dil, 576, _p(dx), 0, None) == 0
    assert lib.wg_pc_relu_grad(_p(dx), _p(mask), M * 64, _p(u32), None) == 0
    assert lib.wg_pc_cast_bf16(_p(u32), M, 64, 64, 0, _p(u16), None) == 0
    assert torch.equal(conv(4, wt, mask=mask)[1], u16)
    assert lib.wg_pc_add(_p(add), _p(dx), M * 64, _p(u32), _p(u16), None) == 0
    o32, o16 = conv(5, wt, add=add)
    assert torch.equal(o32, u32) and torch.equal(o16, u16)
    assert lib.wg_pc_relu_grad(_p(u32), _p(mask), M * 64, _p(dx), None) == 0
    assert lib.wg_pc_cast_bf16(_p(dx), M, 64, 64, 0, _p(u16), None) == 0
    assert torch.equal(conv(6, wt, add=add, mask=mask)[1], u16)
    # weight gradient: transposed columns times transposed dL/dy, where pixels fill tiles of 64
    if M % 64 == 0:
        colT, dyT, dy = b16(576, M), b16(64, M), mask
        assert lib.wg_pc_transpose_bf16(_p(col), M, 576, _p(colT), None) == 0
        assert lib.wg_pc_transpose_bf16(_p(dy), M, 64, _p(dyT), None) == 0
        n = lib.wg_pc_wgrad_partials(b, h, w, 3)
        ref, part = f32(n, 576, 64), f32(n, 576, 64)
        assert lib.wg_gemm_bf16_dev(_p(colT), _p(dyT), _p(ref), 576, 64, M, 3, _p(st), None) == 0
        assert lib.wg_pc_conv_wgrad(_p(act), 0, _p(dy), b, h, w, dil, 3, _p(part), _p(st), None) == 0
        assert torch.equal(part, ref)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
