"""The triangular solves whose blocks wait for one another: block counts around
the number of SMs, a ragged last block, right-hand sides with NaN."""
import time

import numpy as np
import pytest
import torch

import fml_b200

pytestmark = pytest.mark.gpu


def _system(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B = torch.randn((n, 24), dtype=torch.float64, device="cuda", generator=g)
    A = B @ B.t()
    A.diagonal().add_(float(n))
    return A, torch.randn(n, dtype=torch.float64, device="cuda", generator=g)


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 256, 1000, 148 * 128, 149 * 128 + 5,
                               20001])
def test_solution_and_repeatability(n):
    A, y = _system(n, n)
    x = fml_b200.cho_solve(A.clone(), y)
    # the condition number is below 1 + |B|^2 / n < 40 and the factor's backward
    # error below n u |A|: n u cond with a margin
    r = torch.linalg.vector_norm(A @ x - y) / torch.linalg.vector_norm(y)
    assert float(r) < 40 * max(n, 32) * 2.0 ** -53
    assert torch.equal(x, fml_b200.cho_solve(A.clone(), y))


def test_nan_right_hand_side_is_not_waited_for():
    """A NaN of any payload, the pattern that marks an unset value among them,
    comes out as NaN at once (a wait that ran out would take two seconds)."""
    A, y = _system(700, 3)
    bits = y.cpu().numpy().view(np.uint64).copy()
    bits[300] = np.uint64(0xFFFFFFFFFFFFFFFF)
    bad = torch.from_numpy(bits.view(np.float64)).cuda()
    fml_b200.cho_solve(A.clone(), y)
    torch.cuda.synchronize()
    t = time.perf_counter()
    x = fml_b200.cho_solve(A, bad)
    torch.cuda.synchronize()
    assert time.perf_counter() - t < 1.0
    assert torch.isnan(x).all()
