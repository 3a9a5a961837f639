"""Atomic vector kernels of small sets with short descriptors (a CTA per molecule pair) and
the calls just past that route's limits: 128 atom pairs, 128 features, 24 molecule pairs
per SM."""
import numpy as np
import pytest
import torch

import fml_b200
from fml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a1,a2,nm1,nm2,d,nsig", [
    (1, 1, 1, 1, 1, 1), (8, 16, 59, 60, 128, 32), (8, 16, 60, 60, 128, 2), (8, 16, 10, 9, 129, 1),
    (11, 11, 30, 31, 66, 3), (128, 1, 20, 9, 33, 2), (1, 128, 9, 20, 64, 2), (43, 3, 12, 12, 40, 1),
    (7, 7, 5, 4, 31, 32)])
@pytest.mark.parametrize("kind", ["gaussian", "laplacian"])
def test_against_the_oracle(oracle_mod, kind, a1, a2, nm1, nm2, d, nsig):
    rng = np.random.default_rng(a1 + d)
    n1, n2 = rng.integers(0, a1 + 1, nm1), rng.integers(0, a2 + 1, nm2)
    n1[0], n2[0] = a1, a2
    x1, x2 = rng.normal(size=(d, a1, nm1)), rng.normal(size=(d, a2, nm2))
    sig = list(np.linspace(2.0, 30.0, nsig))
    if kind == "gaussian":
        K = fml_b200.fget_vector_kernels_gaussian(x1, x2, n1, n2, sig, nm1, nm2, nsig)
    else:
        K = fml_b200.get_atomic_kernels_laplacian(x1, x2, n1, n2, sig)
    ref = oracle_mod.vector_kernels(kind, x1.transpose(2, 1, 0), x2.transpose(2, 1, 0), n1, n2, sig)
    # distances bit for bit; exponentials of arguments above -200 within 2 ulp of one
    # another, at most 128 of them in another order
    np.testing.assert_allclose(K, ref, rtol=128 * 2.0 ** -53 + 4.5e-16, atol=1e-300)


def test_packed_rows_and_a_molecule_too_large():
    """The packed form gives the padded form's values; a molecule of more atoms than stated
    sets the status and counts as cut off."""
    rng = np.random.default_rng(4)
    off = np.array([0, 3, 3, 7, 12], dtype=np.int32)
    X = torch.from_numpy(rng.normal(size=(12, 20))).cuda()
    O = torch.from_numpy(off).cuda()
    sp, keep = _lib.host_doubles([3.0, 8.0])

    def packed(amax):
        K = torch.empty((2, 4, 4), dtype=torch.float64, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call("fmlb_vector_kernels_packed_f64", 1, _lib.ptr(X), _lib.ptr(O), 4, amax,
                  _lib.ptr(X), _lib.ptr(O), 4, amax, 20, sp, 2, _lib.ptr(K), _lib.ptr(status),
                  _lib.stream_handle())
        return K.cpu().numpy(), int(status.item())

    def padded(counts):
        x = np.zeros((20, 5, 4))
        for m in range(4):
            x[:, :counts[m], m] = X.cpu().numpy()[off[m]:off[m] + counts[m]].T
        return fml_b200.get_atomic_kernels_laplacian(x, x, counts, counts, [3.0, 8.0])

    K, status = packed(5)
    assert status == 0
    np.testing.assert_array_equal(K, padded([3, 0, 4, 5]))
    K, status = packed(4)
    assert status == 1
    np.testing.assert_array_equal(K, padded([3, 0, 4, 4]))
    del keep
