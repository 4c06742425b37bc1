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
