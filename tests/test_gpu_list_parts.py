"""Long key-tile lists walked in parts."""
import pytest
import torch

from oracle import moddit_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from moddit_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("D,bs", [(128, 128), (64, 64), (128, 64), (64, 128)])
@pytest.mark.parametrize("N,Hm", [(2304, 1), (4013, 1), (4600, 3)])
def test_long_lists_in_parts(ops, D, bs, N, Hm):
    """Text-like rows that keep everything beside sparse rows: divided lists against fp32 masked attention (16-bit inputs:
    2e-2 / 1e-2 as in test_gpu_sparse_attn.py), rows of undivided lists bit for bit, scattered rows like local ones."""
    g = torch.Generator().manual_seed(N + D)
    H, nb, per = 3, (N + bs - 1) // bs, 256 // bs
    q, k, v = ((torch.randn(1, H, N, D, generator=g) * s).to(torch.bfloat16) for s in (1.0, 1.0, 1.0))
    mask = torch.rand(Hm, nb, nb, generator=g) < (0.15 if bs == 128 else 0.02)
    mask[:, :, 0] = True
    mask[:, -1] = True                                      # the last rows keep every key: a divided list
    mask[0, per:2 * per] = True                             # and a second one in the first head only
    valid = N - 200
    kw = dict(q_split=N // 2, kv_len_lo=min(N, (valid + 63) // 64 * 64), kv_len_hi=valid, return_lse=True)
    lists = ops.tile_lists(mask.cuda(), bs, N)
    dev = [t.cuda() for t in (q, k, v)]
    out, lse = ops.sparse_attn_fwd(*dev, lists.counts, lists.entries, order=lists.order, **kw)
    ref, ref_lse = orc.masked_attention(q, k, v, mask.repeat(H // Hm, 1, 1) if Hm != H else mask, bs, **kw)
    assert (out.float().cpu() - ref).abs().max().item() <= 2e-2
    assert ((out.float().cpu() - ref).norm() / ref.norm()).item() <= 1e-2
    fin = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse.cpu()), fin) and (lse.cpu()[fin] - ref_lse[fin]).abs().max().item() <= 5e-3
    whole, whole_lse = ops.sparse_attn_fwd(*dev, lists.counts, lists.entries, split=False, **kw)
    cnt = lists.counts.repeat(H // Hm, 1).float()
    row_pair = torch.arange(N, device="cuda") // 256
    divided = (cnt > 1.4 * cnt.mean(1, keepdim=True))[:, row_pair]        # every list that may be divided
    assert divided.any() and not divided.all()
    same = (out == whole).all(-1)[0]
    assert bool(same[~divided].all())
    if (cnt.max(1).values > 2 * cnt.mean(1)).any():
        assert not torch.equal(lse, whole_lse) or not bool(same[divided].all())       # the parts were really walked
    peers = [torch.zeros(H + 1, N // 2, D, device="cuda", dtype=torch.bfloat16) for _ in range(2)] if N % 2 == 0 else \
        [torch.zeros(H + 1, N, D, device="cuda", dtype=torch.bfloat16)]
    ops.sparse_attn_fwd(*dev, lists.counts, lists.entries, scatter=([t.data_ptr() for t in peers], 1), **kw)
    assert torch.equal(torch.cat(peers, 1)[1:], out[0]) and not torch.cat(peers, 1)[0].any()
