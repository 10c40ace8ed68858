"""The causal FIR at the edges of its blocking (16 samples per thread, 128 traces per block): filters
shorter than, equal to and longer than the block and the record, against the same sum in numpy f32 in
the same tap order, bit for bit (times before the record are left out, so a NaN in the record reaches
only the samples whose taps hold it)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(x, ker):
    out = np.zeros_like(x)
    nt, n = x.shape[1], len(ker)
    for t in range(nt):
        for k in range(n):
            ts = t - (n - 1) + k
            if ts >= 0:
                out[:, t] = out[:, t] + ker[k] * x[:, ts]
    return out


@pytest.mark.parametrize("klen", [1, 2, 15, 16, 17, 31, 33, 64])
@pytest.mark.parametrize("series,nt,nrec", [(1, 1, 1), (3, 15, 70), (2, 16, 64), (2, 17, 43), (1, 50, 129)])
def test_bandlimit_matches_the_sum_in_tap_order(cuda_lib, klen, series, nt, nrec):
    import torch

    from wgnet_gb300.physics import bandlimit_torch

    rng = np.random.default_rng(klen * 1000 + nt)
    x = rng.standard_normal((series, nt, nrec)).astype(np.float32)
    ker = rng.standard_normal(klen).astype(np.float32)
    if nt > 20:
        x[0, 20, 3] = np.nan
        x[0, 5, 7] = np.inf
    with np.errstate(invalid="ignore"):
        ref = _reference(x, ker)
    got = bandlimit_torch(torch.from_numpy(x).cuda(), torch.from_numpy(ker)).cpu().numpy()
    np.testing.assert_array_equal(got, ref)
