"""FP64 ARAD kernels of more molecules than one launch takes (65535 in the first set)."""
import numpy as np
import pytest
import torch

import fml_b200
from fml_b200 import synthetic

pytestmark = pytest.mark.gpu


def test_rows_past_one_launch(oracle_mod):
    """65535 + 70 molecules against three: the same bits as calls of parts of them, and
    the oracle's values on both sides of the boundary."""
    nm, size = 65535 + 70, 2
    b = synthetic.generate(64, nmax=4, nmin=4, seed=2)
    off = np.arange(0, 2 * 64 + 1, 2, dtype=np.int32)
    z = np.concatenate([b.molecule(m)[0][:2] for m in range(64)])
    r = np.concatenate([b.molecule(m)[1][:2] for m in range(64)])
    X = oracle_mod.arad_descriptors(z, r, off, size, 1e6)
    at = np.arange(nm) * 7 % 64
    Z = [z[2 * m:2 * m + 2] for m in at]
    sig = [0.5, 2.0]
    K = fml_b200.get_atomic_kernels_arad(torch.from_numpy(X[at]).cuda(),
                                         torch.from_numpy(X[:3]).cuda(), Z,
                                         [z[2 * m:2 * m + 2] for m in range(3)], sig)
    K = K.cpu().numpy() if torch.is_tensor(K) else K
    assert K.shape == (2, nm, 3)
    ref = oracle_mod.get_atomic_kernels_arad(X, X[:3], [z[2 * m:2 * m + 2] for m in range(64)],
                                             [z[2 * m:2 * m + 2] for m in range(3)], sig)
    np.testing.assert_allclose(K, ref[:, at], rtol=1e-12)
    part = fml_b200.get_atomic_kernels_arad(X[at[65500:]], X[:3], Z[65500:],
                                            [z[2 * m:2 * m + 2] for m in range(3)], sig)
    np.testing.assert_array_equal(K[:, 65500:], part)
