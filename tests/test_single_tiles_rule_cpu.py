"""How many pairs of query tiles a launch of the forward runs as two blocks (`moddit_sparse_attn_single_pairs`)."""
import ctypes
import random

from moddit_b200 import _lib

SMS = 148
rule = _lib.lib.moddit_sparse_attn_single_pairs


def test_idle_sms_of_a_launch_alone():
    for pairs, batches, want in ((1, 1, 1), (74, 1, 74), (75, 1, 73), (132, 1, 16), (147, 1, 1), (148, 1, 0), (5000, 1, 0),
                                 (56, 1, 56), (56, 2, 18), (56, 3, 0), (1, 148, 0), (1, 74, 1), (1, 200, 0)):
        assert rule(SMS, pairs, batches, 0) == want, (pairs, batches)


def test_launches_at_a_time_share_the_idle_sms():
    """No more blocks than SMs, and no more single tiles than one launch of everything would have."""
    rng = random.Random(0)
    for _ in range(2000):
        groups = [rng.randint(1, 100) for _ in range(rng.randint(1, 8))]
        total = sum(groups)
        split = [rule(SMS, g, 1, total - g) for g in groups]
        assert all(0 <= n <= g for n, g in zip(split, groups))
        assert sum(split) <= rule(SMS, total, 1, 0) and sum(split) >= rule(SMS, total, 1, 0) - len(groups)
        assert total >= SMS or total + sum(split) <= SMS
    assert [rule(SMS, 66, 1, 66), rule(SMS, 66, 1, 132), rule(SMS, 32, 1, 32)] == [8, 0, 32]
    assert rule(SMS, 66, 1, 2**31 - 1) == 0 and rule(SMS, 10, 2, 20) == 10 and rule(0, 1, 1, 0) == rule(SMS, 0, 1, 0) == 0


def test_one_destination():
    buf = ctypes.cast(ctypes.create_string_buffer(64), ctypes.c_void_p)
    table = (ctypes.c_void_p * 1)(buf.value)
    fwd = lambda beside, out, peers: _lib.lib.moddit_sparse_attn_fwd_beside(      # noqa: E731
        buf, buf, buf, 0, 1, 128, 64, buf, buf, None, 1, 0.125, 128, 128, 128, beside, out, peers, 1, 0, None, buf, None)
    assert fwd(1, None, None) == fwd(1, buf, table) == -1
    assert b"destination" in _lib.lib.moddit_last_error_string()
    assert fwd(-1, buf, None) == -1 and b"pairs_beside" in _lib.lib.moddit_last_error_string()
