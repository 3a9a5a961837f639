"""FP64 ARAD kernels of small molecules: a warp per molecule pair or the fast kernel by
the atoms and the number of pairs, with the same bits either way."""
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


@pytest.mark.parametrize("size,nm", [(4, 40), (5, 40), (6, 24), (7, 70), (8, 200), (9, 60)])
def test_any_number_of_pairs_gives_a_pairs_bits(oracle_mod, size, nm):
    """Calls below and above the number of pairs at which the route changes (6 atoms: 2^8, 7:
    2^11, 8: 2^14), symmetric and not; and against the oracle."""
    X, Z = _set(nm, size)
    K = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, SIG)
    few = fml_b200.get_atomic_symmetric_kernels_arad(X[3:8], Z[3:8], SIG)
    np.testing.assert_array_equal(K[:, 3:8, 3:8], few)
    np.testing.assert_allclose(few, oracle_mod.get_atomic_symmetric_kernels_arad(X[3:8], Z[3:8], SIG),
                               rtol=1e-12, atol=1e-300)
    R = fml_b200.get_atomic_kernels_arad(X, X, Z, Z, SIG)
    np.testing.assert_array_equal(R[:, 2:4, 1:9],
                                  fml_b200.get_atomic_kernels_arad(X[2:4], X[1:9], Z[2:4], Z[1:9],
                                                                   SIG))


@pytest.mark.parametrize("size", [7, 23])
def test_padding_past_the_fast_kernel(size):
    """The same molecules padded past 32 atoms (a warp per pair): the same bits."""
    X, Z = _set(30, size)
    Xp, _ = _set(30, size, pad=33 - size)
    np.testing.assert_array_equal(fml_b200.get_atomic_symmetric_kernels_arad(X, Z, SIG),
                                  fml_b200.get_atomic_symmetric_kernels_arad(Xp, Z, SIG))
