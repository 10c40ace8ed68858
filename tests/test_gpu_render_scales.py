"""The renderer's gradient for log scales outside the activation's bounds, up to where an inverse scale or the
ratio of the two leaves the f32 range, against the f64 oracle: no parameter's gradient is lost to an overflow.
Offsets are multiples of 1/64 and the narrow Gaussians unrotated, so that distances are exact in f32 (a
rounding of theirs would be a finite part of so small a scale). Tolerance: sums of at most 625 f32 terms whose
exponent has a few roundings of at most 2^-24 relative on |exponent| < 40 where terms matter, i.e. 1e-5 of the
parameter's norm over all slots."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import render_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_sx,log_sz,angle", [(-40.0, 49.0, 0.0), (49.0, -40.0, 0.0), (0.0, 89.0, 0.3), (89.0, 0.5, -0.3),
                                                 (-4.25, 4.25, 0.0), (4.25, -4.25, 0.0), (-3.75, 3.75, 0.0),
                                                 (20.0, 30.0, 1.0), (1.0, 45.0, 0.7)])
def test_gradient_matches_the_f64_oracle(cuda_lib, log_sx, log_sz, angle):
    import torch

    from wgnet_gb300.render import render_residual

    rng = np.random.default_rng(11)
    p = np.empty((1, 1225, 6), np.float32)
    p[..., :2] = rng.integers(-128, 129, (1, 1225, 2)) / 64.0
    p[..., 2], p[..., 3], p[..., 4] = log_sx, log_sz, angle
    p[..., 5] = rng.uniform(-1.0, 1.0, (1, 1225))
    cot = rng.standard_normal((1, 70, 70)).astype(np.float32)
    t = torch.from_numpy(p).cuda().requires_grad_(True)
    (grad,) = torch.autograd.grad(render_residual(t), [t], torch.from_numpy(cot).cuda())
    got = grad.cpu().numpy().astype(np.float64)
    ref = render_np.render_vjp(p.astype(np.float64), cot.astype(np.float64))
    assert np.isfinite(got).all()
    scale = np.linalg.norm(ref.reshape(-1, 6), axis=0)
    err = np.linalg.norm((got - ref).reshape(-1, 6), axis=0)
    assert (err <= 1e-5 * scale + 1e-12).all(), (err / np.maximum(scale, 1e-300)).tolist()
