"""The FP64 distance tile where its columns or rows run out: every number of columns
up to a tile's 64, 32-row tiles of 4 x 4 pairs with a last block of one or two tiles,
and the sizes around the change between 32- and 64-row tiles."""
import ctypes

import numpy as np
import pytest
import torch

import fml_b200
from fml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [641, 672, 673, 704, 1025, 1300, 1312, 1313, 1659, 1787, 2043, 2427])
@pytest.mark.parametrize("fn", ["gaussian_kernel", "laplacian_kernel"])
def test_symmetric_blocks(n, fn):
    """Any tile height, symmetric or not, gives an entry the same bits; its value against
    plain 64-bit distances."""
    g = torch.Generator(device="cuda").manual_seed(n)
    X = torch.rand((n, 21), dtype=torch.float64, device="cuda", generator=g)
    kernel = getattr(fml_b200, fn)
    K = kernel(X.t(), X.t(), [0.8, 2.0])
    assert torch.equal(K, kernel(X.t(), X.clone().t(), [0.8, 2.0]))
    assert torch.equal(K[:, -40:], kernel(X[-40:].t(), X.t(), [0.8, 2.0]))
    D = torch.cdist(X, X, p=1.0) if fn[0] == "l" else \
        (X[:, None] - X[None]).square().sum(-1)
    for k, s in enumerate([0.8, 2.0]):
        ref = torch.exp(D * (-1.0 / s if fn[0] == "l" else -0.5 / s ** 2))
        # 21 terms below 1 in two orders: |dD| <= 2 * 21 * 21 * 2^-53; exponent below 33
        torch.testing.assert_close(K[k], ref, rtol=2.5e-13, atol=0)


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 33, 64])
@pytest.mark.parametrize("kind", ["gaussian", "laplacian"])
def test_every_number_of_columns(oracle_mod, kind, rows):
    """A molecule of `rows` atoms against molecules of 1 .. 64 atoms, one to a tile."""
    rng = np.random.default_rng(rows)
    n1, n2 = np.array([rows, 1]), np.arange(1, 65)
    x1, x2 = rng.normal(size=(9, 64, 2)), rng.normal(size=(9, 64, 64))
    sig = [1.5, 4.0]
    if kind == "gaussian":
        K = fml_b200.fget_vector_kernels_gaussian(x1, x2, n1, n2, sig, 2, 64, 2)
    else:
        K = fml_b200.get_atomic_kernels_laplacian(x1, x2, n1, n2, sig)
    ref = oracle_mod.vector_kernels(kind, x1.transpose(2, 1, 0), x2.transpose(2, 1, 0), n1, n2, sig)
    # the distances bit for bit; sums of at most 4096 exponentials in two orders
    np.testing.assert_allclose(K, ref, rtol=4096 * 2.0 ** -53 + 4e-16, atol=1e-300)


@pytest.mark.parametrize("nq", [1, 40, 700])
def test_prediction_with_every_number_of_columns(nq):
    """Training sets of 1 .. 64 points (and 65 .. 72): the last tile's columns."""
    rng = np.random.default_rng(nq)
    Q, T = rng.normal(size=(nq, 19)), rng.normal(size=(72, 19))
    w = rng.normal(size=72)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    Qd, Td, wd = dev(Q), dev(T), dev(w)
    K = np.exp(-0.5 * ((Q[:, None] - T[None]) ** 2).sum(-1) / 2.25)
    sp, keep = _lib.host_doubles([1.5])
    y = torch.empty(nq, dtype=torch.float64, device="cuda")
    for nt in range(1, 73):
        nb = _lib.load().fmlb_kernel_predict_workspace_bytes(nq, nt, 1)
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        _lib.call("fmlb_kernel_predict_f64", 0, _lib.ptr(Qd), nq, 19, _lib.ptr(Td), nt, 19, 19,
                  ctypes.cast(sp, ctypes.POINTER(ctypes.c_double)), 1, _lib.ptr(wd), nt,
                  _lib.ptr(y), nq, _lib.ptr(ws), nb, _lib.stream_handle())
        # 72 products in two orders, exponents below 100 from 19 terms in two orders
        tol = (2 * 72 + 64 + 100 * 40) * 2.0 ** -53 * (K[:, :nt] @ np.abs(w[:nt])).max()
        np.testing.assert_allclose(y.cpu().numpy(), K[:, :nt] @ w[:nt], rtol=0, atol=tol)
    del keep
