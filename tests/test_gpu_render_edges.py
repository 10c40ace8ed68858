"""The renderer's gradient at the ends of its parameters' ranges (widest and narrowest Gaussians, full
offsets and rotations, equal scales where the angle's gradient vanishes) and with cotangents on corner and
border pixels only, against the f64 oracle. Tolerance: sums of at most 625 f32 terms whose exponent has a
few roundings of at most 2^-24 relative on |exponent| < 90, i.e. 1e-5 of the slot's largest gradient
scale where terms matter; per parameter, relative to the norm over all slots."""

from __future__ import annotations

import math

import numpy as np
import pytest

from oracle import render_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_sx,log_sz,angle,off", [(0.5, 0.5, 0.0, 0.0), (6.0, 0.5, math.pi / 2, 2.0), (0.5, 6.0, -math.pi / 2, -2.0),
                                                     (6.0, 6.0, 0.7, 2.0), (1.3, 2.1, -0.4, 0.5)])
@pytest.mark.parametrize("where", ["all", "corners", "border"])
def test_gradient_matches_the_f64_oracle(cuda_lib, log_sx, log_sz, angle, off, where):
    import torch

    from wgnet_gb300.render import render_residual

    rng = np.random.default_rng(5)
    p = np.empty((2, 1225, 6), np.float32)
    p[..., 0], p[..., 1] = off, -off
    p[..., 2], p[..., 3], p[..., 4] = math.log(log_sx), math.log(log_sz), angle
    p[..., 5] = rng.uniform(-1.0, 1.0, (2, 1225))
    cot = rng.standard_normal((2, 70, 70)).astype(np.float32)
    keep = np.zeros((70, 70), np.float32)
    if where == "corners":
        keep[0, 0] = keep[0, 69] = keep[69, 0] = keep[69, 69] = 1
    elif where == "border":
        keep[0] = keep[69] = 1
        keep[:, 0] = keep[:, 69] = 1
    else:
        keep[:] = 1
    cot *= keep
    t = torch.from_numpy(p).cuda().requires_grad_(True)
    field = render_residual(t)
    (grad,) = torch.autograd.grad(field, [t], torch.from_numpy(cot).cuda())
    got = grad.cpu().numpy().astype(np.float64)
    ref = render_np.render_vjp(p.astype(np.float64), cot.astype(np.float64))
    scale = np.linalg.norm(ref.reshape(-1, 6), axis=0)
    err = np.linalg.norm((got - ref).reshape(-1, 6), axis=0)
    # equal scales: the angle's gradient is zero up to the f32 difference of the two log scales
    scale[4] = max(scale[4], 1e-3 * scale[:4].max())
    assert (err <= 1e-5 * scale + 1e-12).all(), (err / scale).tolist()
