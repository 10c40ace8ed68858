"""The causal FIR's two blockings (4 samples per thread for small calls, 16 for the others) at the edges of the
larger one, and on both sides of the line between them: against the same sum in numpy f32 in the same tap
order, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(x, ker):
    out = np.zeros_like(x)
    nt, n = x.shape[1], len(ker)
    for t in range(nt):
        for k in range(max(0, n - 1 - t), n):
            out[:, t] = out[:, t] + ker[k] * x[:, t - (n - 1) + k]
    return out


# more than 128 taps of an output: records that end inside, at and after a block of 16, taps likewise; then
# many traces: records shorter than a block, and outputs x taps either side of 2^23
@pytest.mark.parametrize("series,nt,nrec,klen", [(1, 129, 3, 129), (2, 144, 70, 143), (2, 145, 43, 144), (1, 150, 129, 145), (3, 177, 20, 160),
                                                 (700, 15, 64, 15), (700, 15, 64, 40), (700, 16, 64, 31), (64, 64, 32, 64),
                                                 (64, 65, 32, 64), (1, 128, 70, 128), (1, 129, 70, 128)])
def test_bandlimit_matches_the_sum_in_tap_order(cuda_lib, series, nt, nrec, klen):
    import torch

    from wgnet_gb300.physics import bandlimit_torch

    rng = np.random.default_rng(klen * 1000 + nt)
    x = rng.standard_normal((series, nt, nrec)).astype(np.float32)
    ker = rng.standard_normal(klen).astype(np.float32)
    x[0, 9, nrec - 1] = np.nan
    with np.errstate(invalid="ignore"):
        ref = _reference(x, ker)
    got = bandlimit_torch(torch.from_numpy(x).cuda(), torch.from_numpy(ker)).cpu().numpy()
    np.testing.assert_array_equal(got, ref)
