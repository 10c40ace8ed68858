"""The update network's elementwise passes at the edges of their tiles: Adam over ragged layers (sizes that
no tile divides, several layers in one launch), im2col of odd images, the per-sample RMS."""

from __future__ import annotations

import ctypes

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("layers", [[(64, 576, 63)], [(33, 9, 3), (1, 1, 1), (64, 128, 17)], [(32, 8, 16)] * 16])
@pytest.mark.parametrize("with_grad", [False, True])
def test_adam_layers_match_the_formula(cuda_lib, layers, with_grad):
    g = torch.Generator().manual_seed(5)
    lr, b1, b2, eps, step = 1e-3, 0.9, 0.999, 1e-8, 3
    L = []
    for n, kp, s in layers:
        L.append({"p": torch.randn((s, kp, n), generator=g).cuda(), "w": torch.randn((n, kp), generator=g).cuda(),
                  "m": torch.randn((n, kp), generator=g).cuda(), "v": torch.rand((n, kp), generator=g).cuda(),
                  "g": torch.empty((n, kp), device="cuda"), "q": torch.empty((n, kp), device="cuda", dtype=torch.bfloat16),
                  "qt": torch.empty((kp, n), device="cuda", dtype=torch.bfloat16)})
    want = []
    for d in L:
        t = torch.zeros_like(d["p"][0])
        for part in d["p"]:  # in split order: the same FP32 sum
            t = t + part
        gr = t.t().contiguous()
        m, v = b1 * d["m"].double() + (1 - b1) * gr.double(), b2 * d["v"].double() + (1 - b2) * gr.double() ** 2
        w = d["w"].double() - lr * (m / (1 - b1 ** step)) / ((v / (1 - b2 ** step)).sqrt() + eps)
        want.append((gr, m, v, w))

    def ptrs(key):
        return (ctypes.c_void_p * len(L))(*[d[key].data_ptr() for d in L])

    def ints(i):
        return (ctypes.c_int * len(L))(*[x[i] for x in layers])

    args = [len(L), ptrs("p"), ints(2), ints(0), ints(1), ptrs("w"), ptrs("m"), ptrs("v"),
            ptrs("g") if with_grad else None, ptrs("q"), ptrs("qt"), lr, b1, b2, eps, step, None]
    assert cuda_lib.wg_pc_adam_layers(*args) == 0
    torch.cuda.synchronize()
    for d, (gr, m, v, w) in zip(L, want):
        if with_grad:
            assert torch.equal(d["g"], gr)
        # FP32: a few roundings (6e-8 each) of terms up to the largest m or v; 1 - b2 and 1 - b2^step carry
        # those of b2 = 0.999 amplified by 1000, so that share of v and the step have 1e-4 relative
        assert ((d["m"] - m).abs() <= 4e-7 * (1 + m.abs().max())).all()
        assert ((d["v"] - v).abs() <= 4e-7 * (1 + v) + 1e-7 * gr.double() ** 2).all()
        move = lr * (m / (1 - b1 ** step)).abs() / (v / (1 - b2 ** step)).sqrt()
        assert ((d["w"] - w).abs() <= 4e-7 * (1 + w.abs()) + 1e-4 * move).all()
        assert torch.equal(d["q"], d["w"].bfloat16()) and torch.equal(d["qt"], d["q"].t())
    args[0] = 17
    assert cuda_lib.wg_pc_adam_layers(*args) != 0


@pytest.mark.parametrize("B,H,W,C,dil,kp", [(1, 1, 1, 8, 1, 128), (2, 7, 5, 8, 1, 128), (3, 6, 37, 16, 3, 192)])
def test_im2col_of_odd_images(cuda_lib, B, H, W, C, dil, kp):
    act = torch.randn((B, H, W, C), generator=torch.Generator().manual_seed(2)).cuda().bfloat16()
    col = torch.full((B, H, W, kp), 7.0, device="cuda", dtype=torch.bfloat16)
    assert cuda_lib.wg_pc_im2col(_p(act), B, H, W, C, dil, kp, _p(col), None) == 0
    pad = torch.nn.functional.pad(act, (0, 0, dil, dil, dil, dil))
    want = torch.zeros_like(col)
    for t in range(9):
        y, x = (t // 3) * dil, (t % 3) * dil
        want[..., t * C:(t + 1) * C] = pad[:, y:y + H, x:x + W]
    torch.cuda.synchronize()
    assert torch.equal(col, want)


@pytest.mark.parametrize("H,W", [(1, 1), (3, 11), (32, 32), (70, 71)])
def test_features_rms(cuda_lib, H, W):
    g = torch.randn((3, H, W), generator=torch.Generator().manual_seed(3)).cuda()
    v, band = torch.full_like(g, 3.5), torch.zeros(3, device="cuda", dtype=torch.int32)
    rms = torch.empty(3, device="cuda")
    out = torch.empty((3, H, W, 8), device="cuda", dtype=torch.bfloat16)
    assert cuda_lib.wg_pc_features(_p(v), _p(g), _p(band), 3, H, W, _p(rms), _p(out), None) == 0
    want = g.double().pow(2).mean((1, 2)).sqrt()
    torch.cuda.synchronize()
    assert ((rms - want).abs() <= 1.2e-7 * want).all()  # one rounding to FP32 of the 64-bit value
