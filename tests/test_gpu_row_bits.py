"""A row of the sparse forward depends on its own list of key tiles and on nothing else in the launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from moddit_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,bs,N", [(128, 128, 4013), (64, 64, 4013), (128, 64, 8448), (64, 128, 600)])
def test_rows_do_not_depend_on_other_lists(ops, D, bs, N, dtype):
    """Text-like rows that keep every key, once beside sparse rows (their list is then several times the average one) and
    once beside rows that keep as much: the same bits, and the same as in a launch of that head alone."""
    g = torch.Generator().manual_seed(N + D)
    H, nb = 3, (N + bs - 1) // bs
    q, k, v = (torch.randn(1, H, N, D, generator=g).to(dtype).cuda() for _ in range(3))
    sparse = torch.rand(H, nb, nb, generator=g) < 0.1
    sparse[:, :, 0] = True
    first = (N - 1) // 256 * 256                     # rows of the last pair of query tiles
    sparse[:, first // bs:] = True
    full = torch.ones_like(sparse)
    kw = dict(q_split=N // 2, kv_len_lo=N - 64, kv_len_hi=N - 70, return_lse=True)

    def run(mask, heads=slice(None)):
        lists = ops.tile_lists(mask[heads].cuda(), bs, N)
        return ops.sparse_attn_fwd(*(t[:, heads].contiguous() for t in (q, k, v)), lists.counts, lists.entries,
                                   order=lists.order, **kw)

    out, lse = run(sparse)
    dense, dense_lse = run(full)
    assert torch.equal(out[:, :, first:], dense[:, :, first:]) and torch.equal(lse[:, :, first:], dense_lse[:, :, first:])
    for h in range(H):
        alone, alone_lse = run(sparse, slice(h, h + 1))
        assert torch.equal(alone, out[:, h:h + 1]) and torch.equal(alone_lse, lse[:, h:h + 1])
