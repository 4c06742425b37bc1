"""Which steps run their prediction as one call."""
import pytest
import torch


@pytest.fixture
def ops():
    from moddit_b200 import ops as _ops
    was = _ops._TIMING["nvtx"]
    _ops.nvtx_ranges(False)
    yield _ops
    _ops.stage_timing(False)
    _ops.nvtx_ranges(was)


def test_watched_stages_run_as_calls_of_their_own(ops):
    """NVTX ranges and per-stage timing need the single stages; timing of other entry points and of whole predictions
    leaves the step on the path that it takes unwatched."""
    from MoD.mod.attn_mask import _predicts_in_one_call
    H, N, n = 2, 1024, 16
    state = dict(model_type="wan", block_size=64, video_token_num=N, text_token_num=0, warmup_steps=2)
    query = torch.zeros(1, H, N, 64)
    history = [{"c": torch.zeros(H, n), "d": torch.zeros(H, 2 * n - 1)}]
    one_call = lambda: _predicts_in_one_call(query, state, history, 2)      # noqa: E731
    assert one_call()
    ops.nvtx_ranges(True)
    assert not one_call()
    ops.nvtx_ranges(False)
    ops.stage_timing(True)
    assert not one_call()
    ops.stage_timing(True, only=("moddit_sparse_attn_fwd",))
    assert one_call()
    ops.stage_timing(True, by_stage=False)
    assert one_call()
    ops.stage_timing(False)
    assert one_call() and not _predicts_in_one_call(query, state, [], 2) and not _predicts_in_one_call(query, state, history, 0)
