"""FP32 ARAD kernels against FP64 with the error that FP32 arithmetic allows each atom
pair, and the exact zero of an atom's distance to itself."""
import numpy as np
import pytest

import fml_b200
from fml_b200 import synthetic

WIDTH, CUT = 0.2, 6.0


def _mols(oracle_mod, sizes, size, seed):
    big = synthetic.generate(len(sizes), nmax=max(sizes), nmin=max(sizes), seed=seed)
    rng = np.random.default_rng(seed)
    X, Z = np.zeros((len(sizes), size, 5, size)), []
    for m, n in enumerate(sizes):
        r = big.molecule(m)[1][:n]
        Z.append(rng.choice(np.array([1.0, 6.0, 7.0, 8.0, 16.0]), size=n))
        X[m] = oracle_mod.arad_descriptors(Z[m], r, np.array([0, n], dtype=np.int32), size, 1e6)[0]
    return X, Z


def _sums(x, y):
    """(S, sum of |terms|) of two atoms' records x, y (5, n): farad_kernels.f90:58-88."""
    def side(v):
        k = np.argmax(v[0] > CUT) if (v[0] > CUT).any() else v.shape[1]
        return v[:, :k], 1.0 - np.sin(v[0, :k] * np.pi / (2.0 * CUT))
    (x, ex), (y, ey) = side(x), side(y)
    t = (x[0][:, None] - y[0]) ** 2
    v = np.exp(-t / (4.0 * WIDTH ** 2)) * (t < (8.0 * WIDTH) ** 2) * ex[:, None] * ey
    v = v / (1.0 + (x[1][:, None] - y[1]) ** 2) * 0.25 / (0.25 + (x[2][:, None] - y[2]) ** 2)
    v = v * (1.0 + x[3][:, None] * y[3] + x[4][:, None] * y[4])
    return v.sum(), np.abs(v).sum()


def _bound(X, Z, ptp, sig):
    """Exact kernels and the most that FP32 may move them: a term's relative error is below
    2e-5 (its exponent: distances scaled to at most 18.1 rounded to 24 bits, differences
    below 4.81 of them squared, times ln 2: 1.8e-5; a dozen roundings and the hardware's
    exponential: 1e-6), an l2 takes that from each of its sums, and the sum of at most
    1024 exponentials in FP32 lanes of 4 another 4e-6."""
    nm = len(Z)
    S = {}
    for i in range(nm):
        for a in range(len(Z[i])):
            n = len(Z[i])
            S[i, a] = _sums(X[i, a, :, :n], X[i, a, :, :n])
    K, E = np.zeros((len(sig), nm, nm)), np.zeros((len(sig), nm, nm))
    for i in range(nm):
        for j in range(i, nm):
            for a in range(len(Z[i])):
                for b in range(len(Z[j])):
                    s, m = _sums(X[i, a, :, :len(Z[i])], X[j, b, :, :len(Z[j])])
                    dz = ptp[i][a] - ptp[j][b]
                    st = 1.0 / (1.0 + dz[0] ** 2) * 0.25 / (0.25 + dz[1] ** 2)
                    l2 = S[i, a][0] + S[j, b][0] - 2.0 * s * st
                    d = 2.0e-5 * (S[i, a][1] + S[j, b][1] + 2.0 * m * st)
                    for k, g in enumerate(sig):
                        e = np.exp(-l2 / g ** 2)
                        K[k, i, j] += e
                        E[k, i, j] += e * np.expm1(d / g ** 2)
            K[:, j, i], E[:, j, i] = K[:, i, j], E[:, i, j]
    return K, E + 4.0e-6 * K


@pytest.mark.gpu
@pytest.mark.parametrize("size,sizes", [(9, [1, 9, 4, 7, 2]), (23, [23, 17, 5]), (32, [32, 31])])
def test_against_the_exact_sums(oracle_mod, size, sizes):
    X, Z = _mols(oracle_mod, sizes, size, 5)
    sig = [0.5, 1.0, 3.0]
    ptp, _ = fml_b200.kernels._ptp_arrays(Z, size)[:2]
    K, E = _bound(X, Z, ptp, sig)
    got = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, sig, precision="fp32")
    assert (np.abs(got - K) <= E).all()
    assert (E[1:] < 0.02 * K[1:]).all()  # a bound that says something


@pytest.mark.gpu
@pytest.mark.parametrize("size,sizes", [(23, [1, 23, 22, 16, 2, 9]), (32, [32, 31, 17])])
def test_an_atom_and_itself(oracle_mod, size, sizes):
    """At a small sigma only the atoms of equal environments count: each with itself, whose
    l2 cancels exactly (and the two of a molecule of two equal atoms)."""
    X, Z = _mols(oracle_mod, sizes, size, 6)
    K = fml_b200.get_atomic_symmetric_kernels_arad(X, Z, [0.003], precision="fp32")[0]
    ref = np.diag(oracle_mod.get_atomic_symmetric_kernels_arad(X, Z, [0.003])[0])
    assert (ref >= np.array(sizes)).all() and (ref == np.rint(ref)).all()
    np.testing.assert_array_equal(np.diag(K), ref)
