"""Atomic vector kernels over padded arrays of more than 2^31 atom rows."""
import math

import numpy as np
import pytest
import torch

from fml_b200.kernels import _vector_kernels

pytestmark = pytest.mark.gpu


def test_rows_past_32_bits():
    """2^24 + 1 molecules of up to 128 atoms, one feature each: the last molecule's rows
    start at 2^31."""
    nm = 2 ** 24 + 1
    if torch.cuda.mem_get_info()[0] < 24 * 2 ** 30:
        pytest.skip("needs 24 GB of device memory")
    x1 = torch.zeros((nm, 128, 1), dtype=torch.float64, device="cuda")
    x1[0, :3, 0] = torch.tensor([0.5, 1.0, -1.0], dtype=torch.float64)
    x1[-1, :2, 0] = torch.tensor([2.0, -0.25], dtype=torch.float64)
    x2 = torch.tensor([[[0.75]]], dtype=torch.float64, device="cuda")
    n1 = np.zeros(nm, dtype=np.int32)
    n1[0], n1[-1] = 3, 2
    K = _vector_kernels(0, x1, x2, n1, np.array([1]), [1.0])[0, :, 0]
    ref = [sum(math.exp(-0.5 * (v - 0.75) ** 2) for v in row)
           for row in ([0.5, 1.0, -1.0], [2.0, -0.25])]
    assert abs(K[0].item() - ref[0]) < 1e-15 and abs(K[-1].item() - ref[1]) < 1e-15
    assert torch.count_nonzero(K).item() == 2
