"""The small least-squares solve against a float64 solve of the same system."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from moddit_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("n,bpf,H", [(1, 1, 1), (11, 3, 5), (64, 16, 4), (74, 30, 9)])
def test_small_solve_is_exact_to_float32(ops, n, bpf, H):
    """The inverse is kept to about 48 bits and the sums are float64: what is left is the rounding of the result
    (2^-24) and the cancellation of its terms (condition number of the system below 4 n^2)."""
    g = torch.Generator().manual_seed(n)
    b = torch.rand(H, 3 * n, generator=g) * n
    A = ops.mtm(n, bpf, 1.0, "cuda").double().cpu()
    want = torch.linalg.solve(A, b.double().T).T
    got = ops.solve(b.cuda(), n, bpf, 1.0, method="small").double().cpu()
    assert ((got - want).abs().max() / want.abs().max()).item() <= 2.0 ** -24 + 4 * n * n * 2.0 ** -47
