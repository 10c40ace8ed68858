"""Which way the default choices go, by the kernels that a call launches: results are equal bit for bit either
way, so only the counts tell a choice that is never taken, or always."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launches(eng, call):
    """(kernels launched, {kind: launches}) of `call`."""
    from wgnet_gb300 import _lib

    eng.profile(True)
    _lib.launch_count(reset=True)
    call()
    n = _lib.launch_count(reset=True)
    kinds = {k: v[1] for k, v in eng.profile_read().items()}
    eng.profile(False)
    return n, kinds


def _vel(n, nz, nx):
    import torch

    rng = np.random.default_rng(nx + n)
    return torch.from_numpy((1700.0 + 2500.0 * rng.random((n, nz, nx))).astype(np.float32)).cuda()


@pytest.mark.parametrize("models,blocked", [(1, True), (4, True), (9, True), (10, False), (12, False)])
def test_streamed_forward_takes_four_steps_per_launch_up_to_three_tiles_per_sm(cuda_lib, models, blocked):
    """284 x 154 cells are 25 tiles: 2 shots of 9 models 450 (of at most 456), of 10 models 500."""
    import torch

    from wgnet_gb300.engine import WaveEngine

    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the counts are for 152 SMs")
    nt = 26
    eng = WaveEngine(shots=2, nt=nt, dt=0.0005, h=5.0, nx_vis=240, nz_vis=110)
    eng.set_option("streamed", 1)
    vel = _vel(models, 110, 240)
    n, _ = _launches(eng, lambda: eng.simulate_torch(vel))
    assert n == 1 + (-(-nt // 4) if blocked else nt)  # the padding, then the steps


@pytest.mark.parametrize("models,checkpoint,kept", [(2, None, True), (40, None, True), (42, None, False), (2, 50, False), (2, 400, True)])
def test_a_default_engine_recomputes_only_where_its_terms_are_large(cuda_lib, models, checkpoint, kept):
    """5 shots x 400 steps are 104 MB of terms a model: 40 models stay below 4 GiB, 42 do not. A set interval is kept to."""
    from wgnet_gb300.engine import WaveEngine

    eng = WaveEngine(shots=5, nt=400, dt=0.001, checkpoint_every=checkpoint)
    vel = _vel(models, 70, 70)
    obs = eng.simulate_torch(vel * 1.02)
    _, kinds = _launches(eng, lambda: eng.evaluate_adjoint_torch(vel, obs))
    assert kinds["recompute"] == (0 if kept else 7)  # of 8 segments the last keeps its terms in the first pass
    assert kinds["forward"] == (1 if kept else 2) and kinds["adjoint"] == (1 if kept else 8)
