"""Grids of widths that no launch shape was compiled for, odd ones included, on the resident kernels'
ragged variant, and launch choices that depend on the batch: traces and gradients equal the f32 oracle
bit for bit for every launch shape that fits."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import native as o

pytestmark = pytest.mark.gpu


def _case(nxv, nzv, pml, shots=2, nt=90):
    sv = o.Survey(shots=shots, nt=nt, dt=0.001, nx_vis=nxv, nz_vis=nzv, pml=pml)
    rng = np.random.default_rng(nxv * 1000 + nzv)
    cur = (1700.0 + 2500.0 * rng.random((2, nzv, nxv))).astype(np.float32)
    src = np.float32([[0.0, 10.0], [(nxv - 1) * 10.0, 15.0]])[:shots]
    return sv, cur, src


def _engine(sv, src, **kw):
    from wgnet_gb300.engine import WaveEngine

    eng = WaveEngine(shots=sv.shots, nt=sv.nt, dt=sv.dt, peak_hz=sv.peak_hz, pml=sv.pml, vmin=sv.vmin, vmax=sv.vmax,
                     nx_vis=sv.nx_vis, nz_vis=sv.nz_vis, h=sv.h, **kw)
    eng.set_sources(src)
    return eng


# padded widths: narrowest that fits (even, odd), either side of one interior warp, of the strides 116,
# 144 and 184, and small C-PMLs; odd heights on compiled widths as well (70, 100)
@pytest.mark.parametrize("nxv,nzv,pml", [(14, 76, 20), (15, 70, 20), (40, 71, 20), (71, 77, 20), (72, 70, 20), (73, 99, 20),
                                         (93, 77, 20), (99, 100, 20), (101, 128, 20), (139, 131, 20), (138, 140, 20),
                                         (61, 70, 8), (64, 64, 4), (70, 69, 20), (100, 71, 20)])
def test_every_shape_is_bitexact(cuda_lib, nxv, nzv, pml):
    sv, cur, src = _case(nxv, nzv, pml)
    eng = _engine(sv, src, checkpoint_every=40)
    wav = eng.wavelet()
    obs = o.forward(sv, cur[::-1] * np.float32(1.02), src, wav)
    ref = o.forward(sv, cur, src, wav)
    rl, rg = o.evaluate_adjoint(sv, cur, src, wav, obs)
    for shape in eng.shape_candidates("forward"):
        eng.set_launch_shape("forward", shape)
        np.testing.assert_array_equal(eng.simulate(cur), ref, err_msg=f"forward shape {shape}")
    ashapes = eng.shape_candidates("adjoint")
    if not ashapes:
        pytest.skip("no resident adjoint for this grid")
    for prefetch in (1, 0):
        eng.set_option("adjoint_prefetch", prefetch)
        for shape in ashapes:
            eng.set_launch_shape("adjoint", shape)
            loss, grad = eng.evaluate_adjoint(cur, obs)
            np.testing.assert_array_equal(grad, rg, err_msg=f"adjoint shape {shape}")
            np.testing.assert_allclose(loss, rl, rtol=1e-12)


def test_a_nan_cell_on_an_odd_width(cuda_lib):
    """The frame column inside the last pair of an odd row stays out of the wavefield."""
    sv, cur, src = _case(75, 73, 20, nt=60)
    cur[0, 30, -1] = np.nan
    eng = _engine(sv, src)
    wav = eng.wavelet()
    obs = o.forward(sv, np.nan_to_num(cur, nan=2000.0), src, wav)
    np.testing.assert_array_equal(eng.simulate(cur), o.forward(sv, cur, src, wav))
    np.testing.assert_array_equal(eng.evaluate_adjoint(cur, obs)[1], o.evaluate_adjoint(sv, cur, src, wav, obs)[1])


@pytest.mark.parametrize("models,shots", [(1, 5), (2, 2), (18, 2), (8, 5), (23, 2), (24, 2), (16, 5)])
def test_small_batches_take_other_shapes_and_no_checkpoints_with_equal_results(cuda_lib, models, shots):
    """Up to 36 units fit the chip in clusters of four, 46 of three, 76 of two (and 80 to 92 take two
    waves of three), so the default shapes differ; an engine with default checkpointing keeps every
    term of a small batch."""
    sv = o.Survey(shots=shots, nt=130, dt=0.001)
    rng = np.random.default_rng(models)
    cur = (1700.0 + 2500.0 * rng.random((models, 70, 70))).astype(np.float32)
    src = sv.default_sources()
    eng, fixed = _engine(sv, src), _engine(sv, src, checkpoint_every=50)
    fixed.set_launch_shape("forward", (2, 704, 10))
    fixed.set_launch_shape("adjoint", (2, 704, 10))
    obs = fixed.simulate(cur[::-1].copy())
    np.testing.assert_array_equal(eng.simulate(cur[::-1].copy()), obs)
    l0, g0 = eng.evaluate_adjoint(cur, obs)
    l1, g1 = fixed.evaluate_adjoint(cur, obs)
    np.testing.assert_array_equal(g0, g1)
    np.testing.assert_array_equal(l0, l1)
    k = min(models, 2)
    np.testing.assert_array_equal(g0[:k], o.evaluate_adjoint(sv, cur[:k], src, eng.wavelet(), obs[:k])[1])
    assert eng.checkpoint_every == 50
