"""An infinite diagonal entry: the factor holds its infinite root and zeros below it, as
LAPACK's dpotrf leaves them, and the solution a zero in its place."""
import numpy as np
import pytest
import torch

from fml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cols", [(4, [1]), (40, [0, 39]), (150, [31, 32, 127, 128, 149]),
                                    (300, [5, 64, 200])])
def test_infinite_diagonal(n, cols):
    B = np.random.default_rng(n).normal(size=(n, n + 3))
    M = B @ B.T / n + np.eye(n)
    M[cols, cols] = np.inf
    keep = np.setdiff1d(np.arange(n), cols)
    y = np.random.default_rng(1).normal(size=n)
    A, x = torch.from_numpy(M).cuda(), torch.from_numpy(y).cuda()
    ws = torch.empty(_lib.load().fmlb_potrf_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("fmlb_potrf_f64", _lib.ptr(A), n, n, _lib.ptr(ws), _lib.ptr(info),
              _lib.stream_handle())
    _lib.call("fmlb_potrs_f64", _lib.ptr(A), n, n, _lib.ptr(ws), _lib.ptr(x), _lib.stream_handle())
    assert int(info.item()) == 0
    L = np.tril(A.cpu().numpy())
    assert np.isposinf(L[cols, cols]).all()
    for c in cols:
        assert (L[c + 1:, c] == 0.0).all()
    # without the infinite rows and columns, an ordinary system (condition below 40)
    sub = M[np.ix_(keep, keep)]
    ref = np.linalg.solve(sub, y[keep])
    got = x.cpu().numpy()
    assert (got[cols] == 0.0).all()
    assert np.abs(got[keep] - ref).max() <= 40 * 8 * n * 2.0 ** -53 * np.abs(ref).max()
