"""The tiled FP32 ARAD kernel at the edges of its tiles: molecules of 1 to 32
atoms, more and fewer molecules than a tile holds, full groups of records,
several sigma chunks, up to and above the classes of the paired path."""
import numpy as np
import pytest

import fml_b200
from fml_b200 import synthetic

pytestmark = pytest.mark.gpu


def _mols(oracle_mod, sizes, size, charges, seed=11):
    rng = np.random.default_rng(seed)
    big = synthetic.generate(64, nmax=max(max(sizes), 4), nmin=max(max(sizes), 4), seed=seed)
    X = np.zeros((len(sizes), size, 5, size))
    Z = []
    for m, n in enumerate(sizes):
        z, r = big.molecule(m % 64)
        z = rng.choice(np.array(charges, dtype=np.float64), size=n)
        X[m] = oracle_mod.arad_descriptors(z, r[:n], np.array([0, n], dtype=np.int32), size,
                                           1e6)[0]
        Z.append(z)
    return X, Z


@pytest.mark.parametrize("nsig", [1, 9])
@pytest.mark.parametrize("charges", [(1, 6, 7, 8, 16), (1, 3, 5, 6, 7, 8, 9, 11, 14, 15, 16, 17)])
@pytest.mark.parametrize("size,sizes", [
    (4, [1, 4, 2, 3]), (23, [1, 23, 9, 2, 16, 8, 17, 3, 21, 22, 10]),
    (32, [32, 31, 32, 5, 32, 32, 1, 29, 32, 30, 32])])
def test_any_tile_gives_a_pairs_value(oracle_mod, size, sizes, charges, nsig):
    """A kernel value depends on its two molecules alone: bit for bit the same
    from a call with other molecules around it, and for a molecule with itself
    the number of equal atoms' pairs. Against FP64: l2 is a difference of sums of
    up to 32 * 32 terms below 4 in FP32, each with a relative error of some ulps."""
    X, Z = _mols(oracle_mod, sizes, size, charges)
    sig = list(np.linspace(1.0, 3.0, nsig))
    K = fml_b200.get_atomic_kernels_arad(X, X, Z, Z, sig, precision="fp32")
    back = fml_b200.get_atomic_kernels_arad(X[::-1].copy(), X[3:], Z[::-1], Z[3:], sig,
                                            precision="fp32")
    np.testing.assert_array_equal(K[:, ::-1, 3:], back)
    S = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, sig, precision="fp32")
    np.testing.assert_array_equal(S, S.transpose(0, 2, 1))
    sub = fml_b200.get_atomic_symmetric_kernels_arad(X[2:4], Z[2:4], sig, precision="fp32")
    np.testing.assert_array_equal(S[:, 2:4, 2:4], sub)
    D = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, sig)
    # an atom pair's exponential changes by at most l2's error / sigma^2
    err = 4 * 32 * 32 * 8 * 2.0 ** -24
    atoms = np.outer(sizes, sizes)
    assert (np.abs(S - D) <= err * atoms).all()
