"""The fast FP64 ARAD path (descriptors of at most 32 atoms and 16 element
classes) against the oracle and the generic path, at the edges of its range:
one atom, 32 and 33 atoms, neighbour lists that do not ascend, more classes
than the table holds, empty molecules, chunks of atoms."""
import numpy as np
import pytest

import fml_b200
from fml_b200 import synthetic

pytestmark = pytest.mark.gpu

SIG = [0.5, 1.0, 2.0]


def _mols(oracle_mod, sizes, size, cut=1e6, seed=7, charges=(1, 6, 7, 8, 16)):
    """ARAD descriptors and charges of molecules with the given atom counts."""
    rng = np.random.default_rng(seed)
    big = synthetic.generate(64, nmax=max(max(sizes), 4), nmin=max(max(sizes), 4), seed=seed)
    X = np.zeros((len(sizes), size, 5, size))
    Z = []
    for m, n in enumerate(sizes):
        z, r = big.molecule(m % 64)
        z = rng.choice(np.array(charges, dtype=np.float64), size=n)
        off = np.array([0, n], dtype=np.int32)
        X[m] = oracle_mod.arad_descriptors(z, r[:n], off, size, cut)[0]
        Z.append(z)
    return X, Z


def _check(K, ref):
    np.testing.assert_allclose(K, ref, rtol=1e-12, atol=1e-300)


@pytest.mark.parametrize("size,sizes", [
    (1, [1, 1, 1]), (4, [1, 4, 2, 3]), (23, [1, 23, 22, 2, 16, 17]), (32, [32, 31, 5, 32]),
    (33, [33, 32, 4])])  # 33: the generic path
@pytest.mark.parametrize("symmetric", [True, False])
def test_edges_of_the_atom_range(oracle_mod, size, sizes, symmetric):
    X, Z = _mols(oracle_mod, sizes, size)
    if symmetric:
        K = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, SIG)
        ref = oracle_mod.get_atomic_symmetric_kernels_arad(X, Z, SIG)
    else:
        K = fml_b200.get_atomic_kernels_arad(X, X[::-1].copy(), Z, Z[::-1], SIG)
        ref = oracle_mod.get_atomic_kernels_arad(X, X[::-1].copy(), Z, Z[::-1], SIG)
    _check(K, ref)


def test_lists_that_do_not_ascend(oracle_mod):
    """Neighbour records in any order: the window is tested on every term. One
    molecule keeps ascending lists, so both forms meet in a call."""
    X, Z = _mols(oracle_mod, [9, 14, 23, 6], 23)
    rng = np.random.default_rng(3)
    for m, z in enumerate(Z[1:], start=1):
        n = len(z)
        for a in range(n):
            X[m, a, :, :n] = X[m, a, :, rng.permutation(n)].T
    _check(fml_b200.get_atomic_symmetric_kernels_arad(X, Z, SIG),
           oracle_mod.get_atomic_symmetric_kernels_arad(X, Z, SIG))


def test_more_classes_than_the_table_holds(oracle_mod):
    X, Z = _mols(oracle_mod, [20, 18, 12], 23, charges=tuple(range(1, 31)))
    _check(fml_b200.get_atomic_symmetric_kernels_arad(X, Z, SIG),
           oracle_mod.get_atomic_symmetric_kernels_arad(X, Z, SIG))


def test_empty_molecules_many_sigmas_and_block_sizes(oracle_mod):
    """Molecules without atoms give zeros; 17 sigmas take two passes; 130
    molecules reach the 2 x 2 blocks."""
    rng = np.random.default_rng(5)
    X, Z = _mols(oracle_mod, [int(v) for v in rng.integers(1, 8, size=130)], 7)
    Z[3] = Z[3][:0]
    Z[129] = Z[129][:0]
    X[3] = X[129] = 0.0
    sig = list(np.linspace(0.5, 2.0, 17))
    K = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, sig)
    _check(K, oracle_mod.get_atomic_symmetric_kernels_arad(X, Z, sig))
    assert (K[:, 3] == 0.0).all() and (K[:, :, 129] == 0.0).all()


def test_fast_and_generic_paths_agree(oracle_mod):
    """Padding the arrays past 32 atoms takes the generic path: the same l2 bit
    for bit, so the kernels differ by the order of at most 529 exponentials
    (529 * 2^-53 relative)."""
    X, Z = _mols(oracle_mod, [23, 17, 9], 23)
    Xp = np.full((3, 33, 5, 33), 0.0)
    Xp[:, :23, :, :23] = X
    sig = [0.1, 1.0]
    K = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, sig)
    Kp = fml_b200.get_atomic_symmetric_kernels_arad(Xp, Z, sig)
    np.testing.assert_allclose(K, Kp, rtol=529 * 2.0 ** -53, atol=0.0)
