"""FP64 ARAD kernels of the fast kernel and of a warp per molecule pair: the same bits."""
import numpy as np
import pytest

import fml_b200
from fml_b200 import synthetic

pytestmark = pytest.mark.gpu

SIG = [0.1, 0.5, 2.0]


def _set(nm, size, pad=0):
    b = synthetic.generate(nm, nmax=size, nmin=min(4, size), seed=size)
    X = fml_b200.generate_arad_descriptors(b.charges, b.coords, b.offsets, size=size + pad,
                                           cut=1e6)
    return X, [b.molecule(i)[0] for i in range(nm)]


@pytest.mark.parametrize("size", [7, 23])
def test_padding_past_the_fast_kernel(size):
    """The same molecules padded past 32 atoms (a warp per pair): the same bits."""
    X, Z = _set(30, size)
    Xp, _ = _set(30, size, pad=33 - size)
    np.testing.assert_array_equal(fml_b200.get_atomic_symmetric_kernels_arad(X, Z, SIG),
                                  fml_b200.get_atomic_symmetric_kernels_arad(Xp, Z, SIG))
