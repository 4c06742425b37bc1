"""The mask prediction in one call against its stages."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from moddit_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("model,D,bs,grid,text", [("wan", 64, 64, (4, 32, 32), 0), ("hunyuan", 128, 128, (6, 32, 48), 200),
                                                  ("cogvideox", 64, 64, (3, 33, 41), 130),
                                                  # past the sizes of the small solve: n = 96, 120 and 106
                                                  ("wan", 128, 64, (6, 32, 32), 0), ("hunyuan", 128, 128, (10, 32, 48), 200),
                                                  ("cogvideox", 64, 64, (5, 33, 41), 130)])
def test_prediction_in_one_call_equals_the_stages(ops, model, D, bs, grid, text):
    from moddit_b200 import _lib, synth
    from MoD.mod.attn_mask import block_geometry
    H, video = 3, grid[0] * grid[1] * grid[2]
    q, k, _ = synth.make_qkv(heads=H, grid=grid, head_dim=D, text_tokens=text, text_first=model == "cogvideox", seed=4,
                             device="cuda")
    q, k = q.contiguous(), k.contiguous()
    N = video + text
    nb, n, first = block_geometry(model, bs, video, text, N)
    bpf = max(1, grid[1] * grid[2] // bs)
    kw = dict(q_block_offset=first, k_block_offset=first, video_blocks=n, scale=D ** -0.5)
    dark = ops.pooled_map(ops.pool_blocks(q, bs), ops.pool_blocks(k, bs), **kw).squeeze(0)
    X = ops.solve(ops.mts(dark, bpf)[0], n, bpf, 1.0)
    feats, modes = ops.split_solution(X, n, 1.0)
    assert torch.equal(feats['d'], X[:, :2 * n - 1]) and torch.equal(feats['c'], X[:, 2 * n - 1:3 * n - 1] / 2)
    assert torch.equal(feats['b_d'], X[:, -1]) and torch.equal(modes, ops.head_modes(X[:, -1], 1.0))
    last = {'c': feats['c'] * 1.01, 'd': feats['d'] * 0.99}
    lines = ops.select_lines(feats['c'], feats['d'], last['c'], last['d'], n // 3, 5)
    mask = ops.mask_from_lines(lines, modes, n=n, blocks_per_frame=bpf, model_type=model,
                               text_blocks=first if model == "cogvideox" else nb - n, total_blocks=nb)
    lists = ops.tile_lists(mask, bs, N)
    got = ops.predict_lines(q, k, bs, first=first, n=n, blocks_per_frame=bpf, model_type=model, last=last, top_k=n // 3,
                            predict_T=5)
    assert torch.equal(got[0], dark) and all(torch.equal(got[1][key], feats[key]) for key in feats)
    assert torch.equal(got[2], modes) and torch.equal(got[3], mask)
    assert torch.equal(got[4].counts, lists.counts) and torch.equal(got[4].order, lists.order)
    live = torch.arange(lists.entries.shape[-1], device="cuda") < lists.counts[..., None]
    assert torch.equal(got[4].entries[live], lists.entries[live])


@pytest.mark.parametrize("model,grid,text", [("wan", (4, 32, 32), 0), ("cogvideox", (5, 33, 41), 130)])
def test_watched_step_equals_the_unwatched_one(ops, model, grid, text):
    """A layer's step gives the same output and state whether its prediction is one call or, under timing, single ones."""
    import logging
    from moddit_b200 import synth
    from MoD.mod.attn_mask import SparseAttentionWithMap
    from MoD.mod.state import create_adaptive_mask_state
    H, video = 2, grid[0] * grid[1] * grid[2]
    got = []
    for watched in (False, True):
        state = create_adaptive_mask_state(model, H, video, text, grid[1] * grid[2], grid[0], warmup_steps=2, top_k=12,
                                           predict_T=5, block_size=64)
        state["score_producer"] = "pooled"
        ops.stage_timing(watched)
        for step in range(4):
            q, k, v = synth.make_qkv(heads=H, grid=grid, head_dim=64, text_tokens=text, text_first=model == "cogvideox",
                                     seed=20 + step, device="cuda")
            out, _ = SparseAttentionWithMap(q, k, v, state, logging.getLogger("test"), current_step=step)
        names = [name for name, _ in ops.stage_records()]
        ops.stage_timing(False)
        assert watched == ("moddit_pool_blocks" in names)
        got.append((out, state["mask"], state["prev_full_maps"], state["mode"], *state["features_history"][-1].values()))
    assert all(torch.equal(a, b) for a, b in zip(*got))
