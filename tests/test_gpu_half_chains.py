"""Head dimension 64: every query tile runs two independent softmax chains, one for either 64-key half of its key tiles,
put together at the end.  Masks in which one chain has nothing, in which the two halves of a tile's rows keep different
halves, and scores whose row maximum jumps from tile to tile, against fp32 masked attention (bounds of the forward's own
tests: max-abs 2e-2, relative L2 1e-2, log-sum-exp 5e-3)."""
import pytest
import torch

from oracle import moddit_oracle as orc

pytestmark = pytest.mark.gpu

PATTERNS = {
    "first halves only": lambda i, j: j % 2 == 0,
    "second halves only": lambda i, j: j % 2 == 1,
    "row halves keep different halves": lambda i, j: (i + j) % 2 == 0,
    "one block": lambda i, j: j == 0,
    "one half longer": lambda i, j: (j % 2 == 0) | (j < 3),
    "nothing for a row half": lambda i, j: i % 2 == 0,
}


@pytest.mark.parametrize("pattern", list(PATTERNS))
@pytest.mark.parametrize("N,kv_lo,kv_hi", [(64, None, None), (64 * 9 + 17, None, None), (640, 577, 300)])
def test_masks_that_starve_a_chain(pattern, N, kv_lo, kv_hi):
    from moddit_b200 import ops
    H, D, bs = 2, 64, 64
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(1, H, N, D, generator=g) for _ in range(3))
    k = k * (1.0 + 3.0 * (torch.arange(N) // 64 % 3))[:, None]            # maxima that jump from half to half
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    nb = (N + bs - 1) // bs
    i, j = torch.meshgrid(torch.arange(nb), torch.arange(nb), indexing="ij")
    mask = PATTERNS[pattern](i, j).expand(H, nb, nb).clone()
    lists = ops.tile_lists(mask.cuda(), bs, N)
    kw = dict(q_split=None if kv_lo is None else N // 2, kv_len_lo=kv_lo, kv_len_hi=kv_hi)
    out, lse = ops.sparse_attn_fwd(q.cuda(), k.cuda(), v.cuda(), lists.counts, lists.entries, order=lists.order,
                                   return_lse=True, **kw)
    ref, ref_lse = orc.masked_attention(q, k, v, mask, bs, return_lse=True, **kw)
    out, lse = out.float().cpu(), lse.cpu()
    assert torch.isfinite(out).all()
    assert (out - ref).abs().max().item() <= 2e-2
    assert (out - ref).norm().item() <= 1e-2 * ref.norm().item()
    fin = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse), fin)
    assert not fin.any() or (lse[fin] - ref_lse[fin]).abs().max().item() <= 5e-3
