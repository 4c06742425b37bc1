"""Splitting a least-squares solution into its features."""
import pytest
import torch


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16])
@pytest.mark.parametrize("n", [1, 5])
def test_features_of_any_solution_tensor(n, dtype):
    """Slicing takes every kind of tensor: on the host, in any float type, not contiguous, with a column too many."""
    from MoD.mod.cuda_lstsq import features_from_solution
    X = torch.arange(4 * (3 * n + 1), dtype=dtype).view(2, -1)[:, ::2]
    assert X.shape == (2, 3 * n + 1) and not X.is_contiguous()
    nd = 2 * n - 1
    got = features_from_solution(X[:, :3 * n], n)
    assert torch.equal(got['d'], X[:, :nd]) and torch.equal(got['c'], X[:, nd:nd + n] / 2)
    assert torch.equal(got['b_d'], X[:, 3 * n - 1]) and torch.equal(features_from_solution(X, n)['b_d'], X[:, -1])
