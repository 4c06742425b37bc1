"""Launches with fewer query-tile pairs than SMs run the two tiles of a pair as blocks of their own: same bits as the pair."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,bs", [(128, 128), (128, 64), (64, 64), (64, 128)])
@pytest.mark.parametrize("N,H", [(128, 1), (300, 1), (1000, 2), (1280, 3), (3500, 8), (4096, 9)])
def test_a_tile_by_itself_equals_its_half_of_the_pair(D, bs, N, H):
    """H heads alone (some or all pairs as single tiles) against the same heads among copies that fill the chip (none)."""
    from moddit_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = (N + 255) // 256
    copies = sms // (pairs * H) + 2
    g = torch.Generator(device="cuda").manual_seed(N + H)
    q, k, v = (torch.randn(1, H, N, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    k = k * (1.0 + torch.arange(N, device="cuda") // 128 % 3)[:, None].bfloat16()
    nb = (N + bs - 1) // bs
    mask = torch.rand(H, nb, nb, device="cuda", generator=g) < 0.35
    mask[:, -1] = True

    def run(c, ordered):
        lists = ops.tile_lists(mask.repeat(c, 1, 1), bs, N)
        return ops.sparse_attn_fwd(*[t.repeat(1, c, 1, 1) for t in (q, k, v)], lists.counts, lists.entries,
                                   order=lists.order if ordered else None, kv_len_lo=N - 3, return_lse=True)

    want, want_lse = (t[:, :H] for t in run(copies, True))
    for ordered in (True, False):
        out, lse = run(1, ordered)
        assert torch.equal(out, want) and torch.equal(lse, want_lse)
