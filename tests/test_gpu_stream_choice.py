"""The streamed forward's choice between one step and four steps per launch, left to the engine: equal to
both explicit settings and to the f32 oracle, on grids of one to several tiles per SM, with widths that end
inside a tile, step counts that are no multiple of four, and with checkpoints (which take one step per
launch)."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import native as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxv,nzv,shots,nt,ck", [(40, 36, 3, 41, None), (152, 90, 4, 37, None), (152, 90, 4, 37, 10),
                                                 (244, 118, 9, 30, None)])
def test_default_equals_both_settings(cuda_lib, nxv, nzv, shots, nt, ck):
    from wgnet_gb300.engine import WaveEngine

    pml = 6 if nxv < 100 else 20
    sv = o.Survey(shots=shots, nt=nt, dt=0.0005, h=5.0, nx_vis=nxv, nz_vis=nzv, pml=pml)
    rng = np.random.default_rng(nxv)
    vel = (1700.0 + 2500.0 * rng.random((1, nzv, nxv))).astype(np.float32)
    eng = WaveEngine(shots=shots, nt=nt, dt=sv.dt, peak_hz=sv.peak_hz, pml=pml, vmin=sv.vmin, vmax=sv.vmax, nx_vis=nxv,
                     nz_vis=nzv, h=sv.h, checkpoint_every=ck)
    eng.set_option("streamed", 1)
    if ck is None:
        eng.checkpoint_every = 0
    src, wav = sv.default_sources(), eng.wavelet()
    ref = o.forward(sv, vel, src, wav)
    obs = o.forward(sv, vel * np.float32(1.03), src, wav)
    _, rg = o.evaluate_adjoint(sv, vel, src, wav, obs)
    assert eng.get_option("temporal_block") == 0
    for setting in (None, 0, 1):
        if setting is not None:
            eng.set_option("temporal_block", setting)
        np.testing.assert_array_equal(eng.simulate(vel), ref, err_msg=str(setting))
        np.testing.assert_array_equal(eng.evaluate_adjoint(vel, obs)[1], rg, err_msg=str(setting))
