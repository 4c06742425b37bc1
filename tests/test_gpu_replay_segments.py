"""Segments of the replay map."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from moddit_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("bs,n,H", [(128, 1, 1), (128, 2, 3), (128, 31, 5), (64, 63, 4), (128, 259, 1)])
def test_replay_segments(ops, bs, n, H):
    """Runs that start and end inside a query tile, sweeps longer than one segment, odd tile counts: against the second,
    independently written kernel (the bound both share with the oracle: 2.1 elements per block)."""
    torch.manual_seed(n)
    N, D = n * bs, 64
    q, k = ((torch.randn(1, H, N, D, device="cuda") * 1.5).half() for _ in range(2))
    lse = torch.full((1, H, N), 5.0, device="cuda")
    kw = dict(softmax_scale=D ** -0.5, log_threshold=-6.0, q_video_offset=0, k_video_offset=0, video_blocks=n, block_size=bs)
    got, want = (ops.replay_map(q, k, lse, kernel=name, **kw).float() for name in ("tcgen05", "mma"))
    assert ops.replay_status(torch.device("cuda")) == (0, 0, 0, 0)
    assert 0.05 < want.mean().item() < 0.95
    assert ((got - want).abs() * bs * bs).max().item() <= 2.1


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,bs,n,H,q_off,k_off,text", [(128, 128, 9, 14, 0, 0, 100), (128, 128, 9, 5, 128, 128, 0),
                                                       (128, 64, 37, 8, 100, 36, 200), (128, 128, 33, 9, 0, 0, 0),
                                                       (128, 128, 258, 1, 64, 64, 0), (64, 64, 33, 7, 226, 226, 30)])
def test_replay_segments_two_query_buffers(ops, D, bs, n, H, q_off, k_off, text, dtype):
    """Head dimension 128 (query buffers twice as large), left-over tiles dealt out (5 x 9, 8 x 19, 9 x 33, 258 and
    7 x 17 items on 148 SMs) and as a round of their own (14 x 9), offsets inside a tile: same bound as above."""
    torch.manual_seed(n + D)
    N = max(q_off, k_off) + n * bs + text
    q, k = (torch.randn(1, H, N, D, device="cuda").to(dtype) for _ in range(2))
    lse = torch.randn(1, H, N, device="cuda") * 0.1 + 5.0
    kw = dict(softmax_scale=D ** -0.5, log_threshold=-5.5, q_video_offset=q_off, k_video_offset=k_off, video_blocks=n,
              block_size=bs)
    got, want = (ops.replay_map(q, k, lse, kernel=name, **kw).float() for name in ("tcgen05", "mma"))
    assert ops.replay_status(torch.device("cuda")) == (0, 0, 0, 0)
    assert 0.05 < want.mean().item() < 0.95
    assert ((got - want).abs() * bs * bs).max().item() <= 2.1
