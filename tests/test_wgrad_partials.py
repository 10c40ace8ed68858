"""How many partials the convolution's weight gradient writes for a number of splits: fewer than asked for when
fewer cover the pixels' tiles. A buffer of `splits` partials keeps what it held beyond them, so the count
is what a caller sums."""

from __future__ import annotations

import ctypes

import pytest

# batch, h, w, splits -> partials: one tile; more splits than tiles; an even split; the update network's step
# (2450 tiles, 39 per split, 63 of 64 used)
CASES = [(1, 8, 8, 1, 1), (1, 8, 8, 64, 1), (4, 16, 12, 5, 4), (2, 32, 32, 8, 8), (32, 70, 70, 64, 63)]


@pytest.fixture(scope="module")
def lib():
    from wgnet_gb300 import _lib, build

    if not _lib.LIB_PATH.exists():
        build.build()
    return _lib.load()


@pytest.mark.parametrize("b,h,w,splits,want", CASES)
def test_count(lib, b, h, w, splits, want):
    assert lib.wg_pc_wgrad_partials(b, h, w, splits) == want


def test_count_of_bad_arguments_is_zero(lib):
    for args in ((1, 8, 9, 1), (0, 8, 8, 1), (1, 8, 8, 0), (1, -8, 8, 1)):
        assert lib.wg_pc_wgrad_partials(*args) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("b,h,w,splits,want", CASES)
def test_exactly_so_many_are_written(lib, b, h, w, splits, want):
    import torch

    def p(t):
        return ctypes.c_void_p(t.data_ptr())

    g = torch.Generator(device="cuda").manual_seed(b)
    x, dy = (torch.randn((b * h * w, 64), device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    part = torch.full((splits, 576, 64), float("nan"), device="cuda")
    st = torch.zeros(4, device="cuda", dtype=torch.int32)
    assert lib.wg_pc_conv_wgrad(p(x), 0, p(dy), b, h, w, 1, splits, p(part), p(st), None) == 0
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    assert not part[:want].isnan().any() and part[want:].isnan().all()
