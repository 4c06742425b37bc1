"""The forward's two forms of a block - a pair of query tiles, or one tile of it, which is what launches with fewer pairs than
SMs run - over masks, key limits and scores that are hard on the order of their products, each against fp32 masked attention
(bounds of the forward's own tests: max-abs 2e-2, relative L2 1e-2, log-sum-exp 5e-3) and one against the other bit for bit.
The form follows from the number of pairs times batches, so a batch is repeated until the launch has the form that is wanted."""
import pytest
import torch

from oracle import moddit_oracle as orc

pytestmark = pytest.mark.gpu

# block (i, j) of a mask; t = number of blocks in a 128-row tile
MASKS = {
    "dense": lambda i, j, t: i >= 0,
    "first tile of a pair empty": lambda i, j, t: (i // t) % 2 == 1,
    "second tile of a pair empty": lambda i, j, t: (i // t) % 2 == 0,
    "rows without blocks": lambda i, j, t: (i % 3 == 1) & (j % 2 == 0),
    "tiles take turns": lambda i, j, t: (i // t + j // t) % 2 == 0,
    "tiles take turns by twos": lambda i, j, t: (i // t + j // (2 * t)) % 2 == 0,
    "first tile ends early": lambda i, j, t: ((i // t) % 2 == 1) | (j < 2 * t),
    "second tile starts late": lambda i, j, t: ((i // t) % 2 == 0) | (j >= 3 * t),
    "diagonals": lambda i, j, t: ((i - j) % 5 == 0) | ((i + j) % 7 == 0),
    "first halves only": lambda i, j, t: j % 2 == 0,
    "second halves only": lambda i, j, t: j % 2 == 1,
    "row halves keep different halves": lambda i, j, t: (i + j) % 2 == 0,
    "nothing for a row half": lambda i, j, t: i % 2 == 0,
    "one block": lambda i, j, t: j == 0,
}


def _inputs(H, N, D, dtype):
    g = torch.Generator().manual_seed(N + D)
    q, k, v = (torch.randn(1, H, N, D, generator=g) for _ in range(3))
    k = k * (1.0 + 3.0 * (torch.arange(N) // 64 % 3))[:, None]            # maxima that jump from half tile to half tile
    return [t.to(dtype) for t in (q, k, v)]


def _batches(items):
    """Numbers of batches at which `items` pairs a batch run as pairs, as pairs and single tiles, as single tiles."""
    from moddit_b200 import _lib
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    forms = -(-sms // items), sms // (items + 1), 1
    pairs, some, single = (_lib.lib.moddit_sparse_attn_single_pairs(sms, items, b, 0) for b in forms)
    assert pairs == 0 and 0 < some < items and single == items
    return forms


def _check(out, lse, ref, ref_lse):
    out, lse = out.float().cpu(), lse.cpu()
    assert torch.isfinite(out).all()
    assert (out - ref).abs().max().item() <= 2e-2
    assert (out - ref).norm().item() <= 1e-2 * ref.norm().item()
    fin = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse), fin)
    assert not fin.any() or (lse[fin] - ref_lse[fin]).abs().max().item() <= 5e-3


@pytest.mark.parametrize("name", list(MASKS))
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("D,bs", [(128, 128), (128, 64), (64, 64), (64, 128)])
def test_pairs_and_single_tiles(D, bs, dtype, name):
    """1,169 tokens: ten tiles, the last with 17 rows; 1,100: nine tiles, a pair with one, under two key limits."""
    from moddit_b200 import ops
    H = 2
    for N, kw in ((1169, {}), (1100, dict(q_split=700, kv_len_lo=1100 - 63, kv_len_hi=900))):
        q, k, v = _inputs(H, N, D, dtype)
        nb = (N + bs - 1) // bs
        i, j = torch.meshgrid(torch.arange(nb), torch.arange(nb), indexing="ij")
        mask = MASKS[name](i, j, 128 // bs).expand(H, nb, nb).clone()
        mask[1] = mask[0].flip(1)                                # another mask for the second head
        ref, ref_lse = orc.masked_attention(q, k, v, mask, bs, return_lse=True, **kw)
        lists = ops.tile_lists(mask.cuda(), bs, N)
        got = []
        for batches, order in zip(_batches(lists.counts.numel()), (lists.order, None, lists.order)):
            out, lse = ops.sparse_attn_fwd(*(t.cuda().repeat(batches, 1, 1, 1) for t in (q, k, v)), lists.counts, lists.entries,
                                           order=order, return_lse=True, **kw)
            for t in (out, lse):
                assert torch.equal(t, t[:1].expand_as(t))
            _check(out[:1], lse[:1], ref, ref_lse)
            got.append((out[:1], lse[:1]))
        for out, lse in got[1:]:
            assert torch.equal(out, got[0][0]) and torch.equal(lse, got[0][1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("D,bs", [(128, 128), (64, 64)])
def test_batches_share_the_idle_sms(D, bs, dtype):
    """56 pairs a batch: all as single tiles in one batch, some in two batches of different data, none in three."""
    from moddit_b200 import _lib, ops
    H, N = 4, 3500
    kw = dict(q_split=3000, kv_len_lo=3490, kv_len_hi=3407, return_lse=True)
    g = torch.Generator(device="cuda").manual_seed(N + D)
    q, k, v = (torch.randn(3, H, N, D, device="cuda", generator=g).to(dtype) for _ in range(3))
    nb = (N + bs - 1) // bs
    mask = torch.rand(H, nb, nb, device="cuda", generator=g) < 0.3
    mask[:, -1] = True
    lists = ops.tile_lists(mask, bs, N)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    single = [_lib.lib.moddit_sparse_attn_single_pairs(sms, lists.counts.numel(), b, 0) for b in (1, 2, 3)]
    assert single[0] == 56 and 0 < single[1] < 56 and single[2] == 0
    out, lse = ops.sparse_attn_fwd(q, k, v, lists.counts, lists.entries, order=lists.order, **kw)
    for b in (1, 2):
        part, part_lse = ops.sparse_attn_fwd(q[:b], k[:b], v[:b], lists.counts, lists.entries, order=lists.order, **kw)
        assert torch.equal(part, out[:b]) and torch.equal(part_lse, lse[:b])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("D,bs", [(128, 128), (64, 64)])
@pytest.mark.parametrize("peers,rows", [(1, 1169), (2, 600), (4, 321)])
def test_rows_of_both_forms_go_to_their_shard(D, bs, dtype, peers, rows):
    """The output in row shards (here all of them on one GPU) equals the output in one tensor; the heads around it stay."""
    from moddit_b200 import ops
    H, N, base = 2, peers * rows, 1
    q, k, v = (t.cuda() for t in _inputs(H, N, D, dtype))
    nb = (N + bs - 1) // bs
    g = torch.Generator(device="cuda").manual_seed(N)
    mask = torch.rand(H, nb, nb, device="cuda", generator=g) < 0.4
    lists = ops.tile_lists(mask, bs, N)
    for batches in _batches(lists.counts.numel()):
        qb, kb, vb = (t.repeat(batches, 1, 1, 1) for t in (q, k, v))
        want, want_lse = ops.sparse_attn_fwd(qb, kb, vb, lists.counts, lists.entries, order=lists.order, return_lse=True)
        shards = torch.full((peers, H * batches + 2 * base, rows, D), 7.0, device="cuda", dtype=dtype)
        none, lse = ops.sparse_attn_fwd(qb, kb, vb, lists.counts, lists.entries, order=lists.order, return_lse=True,
                                        scatter=([s.data_ptr() for s in shards], base))
        assert none is None and torch.equal(lse, want_lse)
        whole = want.reshape(H * batches, peers, rows, D).transpose(0, 1)
        assert torch.equal(shards[:, base:-base], whole)
        assert (shards[:, :base] == 7).all() and (shards[:, -base:] == 7).all()
