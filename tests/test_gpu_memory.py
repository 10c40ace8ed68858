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


def _captured(call):
    """The results of `call`, captured into a graph on the stream it runs on, from a replay."""
    import torch

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = call()
    g.replay()
    torch.cuda.synchronize()
    return g, out


def test_a_smaller_batch_than_the_warm_up_can_be_captured(cuda_lib):
    """48 models x 5 shots x 400 steps checkpoint (5 GB of terms); 7 of them would keep their terms by default, in a
    buffer that the warm-up did not allocate. Captured, they take the checkpoints; a later call that does keep
    terms leaves the captured one's buffers where they are."""
    import torch

    from wgnet_gb300.engine import WaveEngine

    eng = WaveEngine(shots=5, nt=400, dt=0.001)
    vel = _models(48)
    obs = eng.simulate_torch(vel * 1.02)
    few, few_obs = vel[:7].contiguous(), obs[:7].contiguous()
    loss, grad = eng.evaluate_adjoint_torch(vel, obs)
    g, got = _captured(lambda: eng.evaluate_adjoint_torch(few, few_obs, check_status=False))
    assert torch.equal(got[0], loss[:7]) and torch.equal(got[1], grad[:7])
    for n in (7, 12):  # eager calls that keep their terms
        again = eng.evaluate_adjoint_torch(vel[:n], obs[:n])
        assert torch.equal(again[1], grad[:n])
    got[1].zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got[1], grad[:7])
    # captured with kept terms: the buffer does not move for a larger batch
    g2, got2 = _captured(lambda: eng.evaluate_adjoint_torch(few, few_obs, check_status=False))
    assert torch.equal(eng.evaluate_adjoint_torch(vel[:20], obs[:20])[1], grad[:20])
    got2[1].zero_()
    g2.replay()
    torch.cuda.synchronize()
    assert torch.equal(got2[1], grad[:7])


def test_fewer_streamed_models_than_the_warm_up_can_be_captured(cuda_lib):
    """10 models x 2 shots are 500 tiles (one step per launch), 2 models 100 (four by default, from a state that the
    warm-up did not allocate)."""
    import torch

    eng = _survey(2)
    vel = _models(10, 116, 276)
    want = eng.simulate_torch(vel)
    few = vel[:2].contiguous()
    g, got = _captured(lambda: eng.simulate_torch(few, check_status=False))
    assert torch.equal(got, want[:2])
    assert torch.equal(eng.simulate_torch(few), want[:2])  # four steps per launch
    g2, got2 = _captured(lambda: eng.simulate_torch(few, check_status=False))
    assert torch.equal(eng.simulate_torch(vel[:4]), want[:4])  # its state would not fit the captured call's
    for graph, out in ((g, got), (g2, got2)):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[:2])
