"""Launches of the forward that run at the same time, one per group of heads: each is told of the others' work items."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,bs", [(128, 128), (64, 64)])
@pytest.mark.parametrize("H,N,groups", [(4, 8448, 2), (5, 1300, 3), (6, 2000, 2)])
def test_groups_of_heads_know_of_each_other(monkeypatch, D, bs, H, N, groups):
    import MoD.mod.attn_mask as am
    from moddit_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(1, H, N, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    nb = (N + bs - 1) // bs
    mask = torch.rand(H, nb, nb, device="cuda", generator=g) < 0.2
    lists = ops.tile_lists(mask, bs, N, heads_per_group=-(-H // groups))
    want = ops.sparse_attn_fwd(q, k, v, lists.counts, lists.entries)
    forward, seen = ops.sparse_attn_fwd, []

    def spy(query, key, value, counts, entries, **kw):
        seen.append((counts.numel(), kw.get("pairs_beside", 0)))
        return forward(query, key, value, counts, entries, **kw)

    monkeypatch.setattr(am._ops, "sparse_attn_fwd", spy)
    out = am.AttentionSparseEngine(q, k, v, mask, block_size=bs, _lists=lists, _group_ready=[None] * groups)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert sum(own for own, _ in seen) == lists.counts.numel() and len(seen) == groups
    assert all(own + beside == lists.counts.numel() for own, beside in seen)
    ops.raise_on_status(q.device)


def test_a_launch_beside_others_into_row_shards():
    """The same bits whatever runs beside it, in one tensor and in row shards (here all of them on one GPU)."""
    from moddit_b200 import ops
    H, D, bs, peers, rows = 3, 128, 128, 2, 650
    N = peers * rows
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(1, H, N, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    mask = torch.rand(H, 11, 11, device="cuda", generator=g) < 0.4
    lists = ops.tile_lists(mask, bs, N)
    want = ops.sparse_attn_fwd(q, k, v, lists.counts, lists.entries)
    for beside in (1, 120, 100000):
        assert torch.equal(ops.sparse_attn_fwd(q, k, v, lists.counts, lists.entries, pairs_beside=beside), want)
        shards = torch.zeros(peers, H, rows, D, device="cuda", dtype=torch.bfloat16)
        ops.sparse_attn_fwd(q, k, v, lists.counts, lists.entries, pairs_beside=beside,
                            scatter=([s.data_ptr() for s in shards], 0))
        assert torch.equal(shards, want.reshape(H, peers, rows, D).transpose(0, 1))
