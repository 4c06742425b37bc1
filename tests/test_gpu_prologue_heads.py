"""Head groups of the attention prologue."""
import pytest
import torch

from oracle import moddit_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from moddit_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("norm,H,D,bs", [("rms_head", 1, 128, 128), ("rms_all_heads", 3, 64, 64), ("layer", 5, 64, 64),
                                         (None, 4, 128, 96), ("layer", 2, 128, 64)])
def test_prologue_head_groups(ops, norm, H, D, bs):
    """Odd and even head counts, one head, block means of every head, inputs that are absent: against one head at a time
    (a head's rows do not depend on the others except through the norm that spans them)."""
    g = torch.Generator().manual_seed(H * D)
    S = 4 * bs + 40
    proj = [torch.randn(1, S, H * D, generator=g).bfloat16() for _ in range(3)]
    width = H * D if norm == "rms_all_heads" else D
    w = [(1 + 0.1 * torch.randn(width, generator=g)).bfloat16() for _ in range(2)]
    bias = [(0.1 * torch.randn(D, generator=g)).bfloat16() for _ in range(2)] if norm == "layer" else [None, None]
    ang = torch.rand(S - 30, D // 2, generator=g) * 6.28
    cos, sin = ang.cos().repeat_interleave(2, 1).contiguous(), ang.sin().repeat_interleave(2, 1).contiguous()
    kw = dict(num_heads=H, norm=norm, rope_cos=cos, rope_sin=sin, rope_range=(10, S - 20))
    if norm is not None:
        kw.update(q_weight=w[0], k_weight=w[1], q_bias=bias[0], k_bias=bias[1])
    dev = {key: val.cuda() if torch.is_tensor(val) else val for key, val in kw.items()}
    got, pools = ops.qkv_prologue(*[t.cuda() for t in proj], pool_block_size=bs, **dev)
    ref = orc.qkv_prologue(*proj, **kw)
    for a, b in zip(got, ref):
        diff = (a.float().cpu() - b.float()).abs()
        assert diff.max().item() <= 4 * 2.0 ** -8 * b.float().abs().max().item()      # two ulp of the pair's magnitude
        assert (diff == 0).float().mean().item() > 0.97
    assert torch.equal(got[2].cpu(), ref[2])
    if bs in (64, 128):
        assert torch.equal(pools[0], ops.pool_blocks(got[0], bs)) and torch.equal(pools[1], ops.pool_blocks(got[1], bs))
    only_k, _ = ops.qkv_prologue(None, proj[1].cuda(), None, **dev)
    assert torch.equal(only_k[1], got[1])
    only_v, _ = ops.qkv_prologue(None, None, proj[2].cuda(), **dev)
    assert torch.equal(only_v[2], got[2])
