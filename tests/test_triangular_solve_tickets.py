"""A thread block of the triangular solves whose ticket lies past the last block (what a
solve meets when another one overlaps on its workspace) does nothing."""
import pytest
import torch

import fml_b200
from fml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 128, 129, 1000, 20001])
def test_block_too_many(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, 8), dtype=torch.float64, device="cuda", generator=g)
    A = A @ A.t()
    A.diagonal().add_(float(n))
    y = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    x = fml_b200.cho_solve(A.clone(), y)
    try:
        _lib.call("fmlb_tc_test_hooks", 0, 2)
        many = fml_b200.cho_solve(A.clone(), y)
        torch.cuda.synchronize()
    finally:
        _lib.call("fmlb_tc_test_hooks", 0, 0)
    assert torch.equal(x, many)
