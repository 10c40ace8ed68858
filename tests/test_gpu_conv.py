"""The fused convolutions of the update network against the unfused route (im2col columns, the
tensor-core GEMM, separate elementwise passes): the same operations in the same order, so every
output is equal bit for bit. Sizes: one pixel, rows shorter than the dilation, ragged last tiles of
128 pixels, one tile, several tiles per SM."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1), (1, 3, 5, 8), (2, 8, 8, 1), (3, 7, 13, 2), (1, 64, 2, 4), (5, 70, 70, 8), (33, 70, 70, 2)]


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _case(shape, cin=64, seed=0):
    import torch

    B, H, W, dil = shape
    g = torch.Generator(device="cuda").manual_seed(seed + B * H * W)
    M = B * H * W
    act = torch.randn((M, cin), device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn((64, 576), device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    add = torch.randn((M, 64), device="cuda", generator=g)
    mask = torch.randn((M, 64), device="cuda", generator=g).to(torch.bfloat16)
    return M, act, w, add, mask


def _gemm(lib, a, b, splits=1):
    import torch

    m, k = a.shape
    n = b.shape[0]
    kt = k // 64
    nz = -(-kt // -(-kt // splits))
    d = torch.empty((nz, m, n), device="cuda")
    st = torch.zeros(4, device="cuda", dtype=torch.int32)
    assert lib.wg_gemm_bf16_dev(_p(a), _p(b), _p(d), m, n, k, splits, _p(st), None) == 0
    assert int(st[0]) == 0
    return d


def _columns(lib, act, shape, cin=64, kp=576):
    import torch

    B, H, W, dil = shape
    col = torch.empty((B * H * W, kp), device="cuda", dtype=torch.bfloat16)
    assert lib.wg_pc_im2col(_p(act), B, H, W, cin, dil, kp, _p(col), None) == 0
    return col


def _conv(lib, mode, act, shape, w, kp=576, add=None, mask=None):
    import torch

    B, H, W, dil = shape
    M = B * H * W
    out32 = torch.full((M,) if mode == 3 else (M, 64), float("nan"), device="cuda")
    out16 = torch.full((M, 64), float("nan"), device="cuda", dtype=torch.bfloat16)
    st = torch.zeros(4, device="cuda", dtype=torch.int32)
    none = ctypes.c_void_p(0)
    assert lib.wg_pc_conv(mode, _p(act), B, H, W, dil, _p(w), kp, _p(add) if add is not None else none,
                          _p(mask) if mask is not None else none, _p(out32), _p(out16), _p(st), None) == 0
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    return out32, out16


@pytest.mark.parametrize("shape", SHAPES)
def test_forward_modes_equal_the_unfused_route(cuda_lib, shape):
    import torch

    M, act, w, add, _ = _case(shape)
    y = _gemm(cuda_lib, _columns(cuda_lib, act, shape), w)[0]
    _, o16 = _conv(cuda_lib, 0, act, shape, w)
    assert torch.equal(o16, y.clamp_min(0.0).to(torch.bfloat16))
    o32, o16 = _conv(cuda_lib, 2, act, shape, w, add=add)
    assert torch.equal(o32, add + y) and torch.equal(o16, (add + y).to(torch.bfloat16))
    one = w.clone()
    one[1:] = 0
    o32, _ = _conv(cuda_lib, 3, act, shape, one)
    assert torch.equal(o32, y[:, 0])
    # the input layer: 8 channels through columns of 128
    x0 = act[:, :8].contiguous()
    w0 = w[:, :128].contiguous()
    w0[:, 72:] = 0
    col = _columns(cuda_lib, x0, shape, cin=8, kp=128)
    y = _gemm(cuda_lib, col, w0)[0]
    o32, o16 = _conv(cuda_lib, 1, col, shape, w0, kp=128)
    ref16 = y.clamp_min(0.0).to(torch.bfloat16)
    assert torch.equal(o16, ref16) and torch.equal(o32, torch.where(ref16 > 0, y, 0.0))


@pytest.mark.parametrize("shape", SHAPES)
def test_data_gradient_modes_equal_the_unfused_route(cuda_lib, shape):
    import torch

    B, H, W, dil = shape
    M, dy, w, add, mask = _case(shape, seed=1)
    wt = w.t().contiguous()
    dcol = _gemm(cuda_lib, dy, wt)[0]
    dx = torch.empty((M, 64), device="cuda")
    assert cuda_lib.wg_pc_col2im(_p(dcol), B, H, W, 64, dil, 576, _p(dx), 0, None) == 0
    keep = mask.float() > 0
    _, o16 = _conv(cuda_lib, 4, dy, shape, wt, mask=mask)
    assert torch.equal(o16, torch.where(keep, dx, 0.0).to(torch.bfloat16))
    o32, o16 = _conv(cuda_lib, 5, dy, shape, wt, add=add)
    assert torch.equal(o32, add + dx) and torch.equal(o16, (add + dx).to(torch.bfloat16))
    _, o16 = _conv(cuda_lib, 6, dy, shape, wt, add=add, mask=mask)
    assert torch.equal(o16, torch.where(keep, add + dx, 0.0).to(torch.bfloat16))
    # the output layer: dL/dy in channel 0 only
    if dil == 1:
        dout = dy[:, 0].float() * 1.001  # not a bf16 value
        full = torch.zeros((M, 64), device="cuda", dtype=torch.bfloat16)
        full[:, 0] = dout.to(torch.bfloat16)
        wt0 = wt.clone()
        wt0[:, 1:] = 0
        dcol = _gemm(cuda_lib, full, wt0)[0]
        assert cuda_lib.wg_pc_col2im(_p(dcol), B, H, W, 64, 1, 576, _p(dx), 0, None) == 0
        dh, dh16 = torch.empty_like(dx), torch.empty((M, 64), device="cuda", dtype=torch.bfloat16)
        d16 = torch.zeros_like(dh16)
        assert cuda_lib.wg_pc_out_dgrad(_p(dout), _p(wt0), B, H, W, _p(dh), _p(dh16), _p(d16), None) == 0
        assert torch.equal(dh, dx) and torch.equal(dh16, dx.to(torch.bfloat16)) and torch.equal(d16, full)


@pytest.mark.parametrize("shape,splits", [((1, 8, 8, 1), 1), ((1, 8, 8, 8), 64), ((4, 16, 12, 2), 5), ((16, 70, 70, 4), 64)])
def test_weight_gradient_partials_equal_the_unfused_route(cuda_lib, shape, splits):
    import torch

    B, H, W, dil = shape
    M, act, _, _, _ = _case(shape, seed=2)
    dy = _case(shape, seed=3)[1]
    st = torch.zeros(4, device="cuda", dtype=torch.int32)
    for x, cols in ((act, 0), (_columns(cuda_lib, act[:, :8].contiguous(), shape, cin=8, kp=128), 128)):
        col = x if cols else _columns(cuda_lib, x, shape)
        ref = _gemm(cuda_lib, col.t().contiguous(), dy.t().contiguous(), splits)
        part = torch.full_like(ref, float("nan"))
        assert cuda_lib.wg_pc_conv_wgrad(_p(x), cols, _p(dy), B, H, W, dil, splits, _p(part), _p(st), None) == 0
        torch.cuda.synchronize()
        assert int(st[0]) == 0 and torch.equal(part, ref)


def test_bad_arguments_are_refused(cuda_lib):
    import torch

    M, act, w, add, mask = _case((1, 8, 9, 1))
    st = torch.zeros(4, device="cuda", dtype=torch.int32)
    z = ctypes.c_void_p(0)
    out = torch.empty((72, 64), device="cuda", dtype=torch.bfloat16)
    for mode, kp, dil, o16 in ((7, 576, 1, out), (0, 128, 1, out), (0, 576, 0, out), (0, 576, 11, out), (2, 576, 1, out)):
        assert cuda_lib.wg_pc_conv(mode, _p(act), 1, 8, 9, dil, _p(w), kp, z, z, z, _p(o16), _p(st), None) != 0
    part = torch.empty((1, 576, 64), device="cuda")
    assert cuda_lib.wg_pc_conv_wgrad(_p(act), 0, _p(act), 1, 8, 9, 1, 1, _p(part), _p(st), None) != 0  # 72 pixels
