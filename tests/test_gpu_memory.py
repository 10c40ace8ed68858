"""What a call does when little device memory is left, or none may be allocated: the same results, by the
same launches where the engine's workspaces already hold the batch."""

from __future__ import annotations

import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _all_held_but(leave: int):
    """The device's free memory but `leave` bytes is taken; gives what was left."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty((torch.cuda.mem_get_info()[0] - leave) >> 21 << 21, dtype=torch.uint8, device="cuda")
    try:
        yield torch.cuda.mem_get_info()[0]
    finally:
        held.untyped_storage().resize_(0)
        torch.cuda.empty_cache()


def _models(n, nz=70, nx=70, seed=3):
    import torch

    rng = np.random.default_rng(seed)
    return torch.from_numpy((1700.0 + 2500.0 * rng.random((n, nz, nx))).astype(np.float32)).cuda()


def test_a_batch_that_the_workspaces_hold_is_not_cut_up(cuda_lib):
    """8 models x 5 shots x 1000 steps keep 2.1 GB of gradient terms. With 0.6 GB left to the next call it takes as
    many launches as the first, and gives the same bits."""
    from wgnet_gb300 import _lib
    from wgnet_gb300.engine import WaveEngine

    eng = WaveEngine(shots=5, nt=1000, dt=0.001)
    vel = _models(8)
    obs = eng.simulate_torch(vel * 1.02)
    runs = []
    for memory in (contextlib.nullcontext(), _all_held_but(600 << 20)):
        with memory:
            _lib.launch_count(reset=True)
            loss, grad = eng.evaluate_adjoint_torch(vel, obs)
            runs.append((_lib.launch_count(reset=True), loss.cpu().numpy(), grad.cpu().numpy()))
    assert runs[1][0] == runs[0][0]
    np.testing.assert_array_equal(runs[1][1], runs[0][1])
    np.testing.assert_array_equal(runs[1][2], runs[0][2])


def _survey(shots, nt=24):
    from wgnet_gb300.engine import WaveEngine

    eng = WaveEngine(shots=shots, nt=nt, dt=0.0005, h=5.0, nx_vis=276, nz_vis=116)
    eng.set_option("streamed", 1)
    return eng


def test_the_streamed_forward_needs_no_memory_beyond_one_step_per_launch(cuda_lib):
    """18 shots of 320 x 160 cells are 450 tiles: by default four steps per launch, whose two state sets take 22 MiB.
    Where these do not fit but one step's state (17 MiB, in pages of two) does, the call takes one step per launch."""
    import torch

    vel = _models(1, 116, 276)
    warm = _survey(2)  # every kernel of both ways is loaded before memory is short
    warm.simulate_torch(vel)
    warm.set_option("temporal_block", 0)
    warm.simulate_torch(vel)
    ref = _survey(18)
    want = ref.simulate_torch(vel)
    torch.cuda.synchronize()
    eng = _survey(18)
    spare = torch.empty_like(want)  # the call's own output comes from here
    with _all_held_but(20 << 20) as left:
        if not 18 << 20 <= left <= 21 << 20:
            pytest.skip(f"{left} bytes free")
        del spare
        got = eng.simulate_torch(vel)
    assert torch.equal(got, want)
