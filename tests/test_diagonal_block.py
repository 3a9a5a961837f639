"""The factorisation's diagonal block: sizes around its sub-blocks, bases and row
strides that 16-byte copies cannot take, the failing column, pivots outside the
normal numbers."""
import numpy as np
import pytest
import torch

from fml_b200 import _lib

pytestmark = pytest.mark.gpu


def _factor(A, n):
    ws = torch.empty(_lib.load().fmlb_potrf_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("fmlb_potrf_f64", _lib.ptr(A), A.stride(0), n, _lib.ptr(ws), _lib.ptr(info),
              _lib.stream_handle())
    return int(info.item())


def _spd(n, seed):
    B = np.random.default_rng(seed).normal(size=(n, n + 3))
    return B @ B.T / n + np.eye(n)


@pytest.mark.parametrize("ld_extra,shift", [(0, 0), (1, 0), (2, 1), (3, 1)])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 160, 255, 300])
def test_factor(n, ld_extra, shift):
    M = _spd(n, n)
    ld = n + ld_extra
    buf = torch.full((n * ld + shift,), -7.0, dtype=torch.float64, device="cuda")
    A = buf[shift:].view(n, ld)
    A[:, :n] = torch.from_numpy(M).cuda()
    assert _factor(A, n) == 0
    out = A.cpu().numpy()
    L = np.tril(out[:, :n])
    # the factor's backward error, and the blocks' inverses times a few ulps
    assert np.abs(L @ L.T - M).max() <= 8 * n * 2.0 ** -53 * np.abs(M).max()
    np.testing.assert_array_equal(np.triu(out[:, :n], 1), np.triu(M, 1))
    assert (out[:, n:] == -7.0).all()


@pytest.mark.parametrize("col", [0, 1, 7, 8, 30, 31, 32, 33, 63, 64, 100, 127, 128, 140])
@pytest.mark.parametrize("value", [0.0, -1.0, float("nan")])
def test_failing_column(col, value):
    M = _spd(150, 3)
    M[col, col] = value
    assert _factor(torch.from_numpy(M).cuda(), 150) == col + 1


@pytest.mark.parametrize("scale", [1e-309, 1e-300, 1e300])
@pytest.mark.parametrize("n", [5, 40, 128])
def test_pivots_at_the_ends_of_the_range(n, scale):
    """A few pivots far from the others, below the normal numbers among them; the
    off-diagonal entries are small enough that no column overflows."""
    d = np.ones(n)
    d[2::7] = scale
    M = np.diag(d)
    assert _factor(A := torch.from_numpy(M).cuda(), n) == 0
    got = np.diag(A.cpu().numpy())
    # a subnormal has fewer digits; its root is formed from it exactly rounded
    np.testing.assert_allclose(got, np.sqrt(d), rtol=4 * 2.0 ** -53)


def test_infinite_pivot_is_no_failure():
    M = np.diag(np.array([1.0, np.inf, 4.0, 9.0]))
    assert _factor(A := torch.from_numpy(M).cuda(), 4) == 0
    assert torch.diagonal(A).cpu()[[0, 2, 3]].tolist() == [1.0, 2.0, 3.0]
