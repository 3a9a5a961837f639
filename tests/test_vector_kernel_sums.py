"""The rounding of the atomic kernels' sums over atom pairs."""
import math

import numpy as np
import pytest

import fml_b200

pytestmark = pytest.mark.gpu


def test_mean_error_of_a_sum():
    """3600 exponentials a kernel, against their exact sum. With an ulp between two
    exponential functions, rows and then columns summed one after the other leave a mean
    relative error of 1.7e-16, in four partial sums each 7.5e-17 (computed from 576 such
    pairs in numpy); the line is between the two."""
    rng = np.random.default_rng(1)
    x1, x2 = rng.normal(size=(1, 60, 24)), rng.normal(size=(1, 60, 24))
    n = np.full(24, 60)
    K = fml_b200.fget_vector_kernels_gaussian(x1, x2, n, n, [1.0], 24, 24, 1)[0]
    err = 0.0
    for i in range(24):
        for j in range(24):
            e = np.exp(-0.5 * (x1[0, :, i][:, None] - x2[0, :, j]) ** 2)
            exact = math.fsum(e.ravel())
            err += abs(K[i, j] - exact) / exact / 576
    assert err < 1.1e-16
