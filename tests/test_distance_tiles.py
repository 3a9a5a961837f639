"""The FP64 distance tile (kernel matrices, fused prediction, atomic vector
kernels) at the edges of its tiles: 16- and 64-row tiles, 8-feature chunks,
groups of molecules."""
import ctypes

import numpy as np
import pytest
import torch

import fml_b200
from fml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb,d", [
    (1, 1, 1), (16, 64, 7), (17, 65, 8), (63, 127, 9), (64, 64, 31), (65, 129, 33), (3, 1000, 276),
    (1500, 9, 24), (1601, 1030, 17)])
@pytest.mark.parametrize("fn", ["gaussian_kernel", "laplacian_kernel"])
def test_kernel_tiles_vs_oracle(oracle_mod, fn, na, nb, d):
    rng = np.random.default_rng(na + nb)
    A, B = rng.normal(size=(d, na)), rng.normal(size=(d, nb))
    K = getattr(fml_b200, fn)(A, B, 2.0)
    np.testing.assert_allclose(K, getattr(oracle_mod, fn)(A, B, 2.0), rtol=1e-12)


@pytest.mark.parametrize("n", [5, 64, 300, 700, 1601])
def test_small_and_large_routes_are_the_same_bits(n):
    """A symmetric build, the same build of two arrays and a slice of it (the
    16-row tiles) agree bit for bit."""
    A = np.random.default_rng(n).normal(size=(45, n))
    sig = [0.7, 3.0]
    K = fml_b200.gaussian_kernel(A, A, sig)
    assert np.array_equal(K, fml_b200.gaussian_kernel(A, A.copy(), sig))
    assert np.array_equal(K, K.transpose(0, 2, 1))
    assert np.array_equal(K[:, :7], fml_b200.gaussian_kernel(A[:, :7].copy(), A, sig))
    assert (np.diagonal(K, axis1=1, axis2=2) == 1.0).all()


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("nq,nt,nsig", [(1, 1, 1), (15, 129, 3), (17, 1024, 8), (65, 1025, 2),
                                        (700, 2311, 3)])
def test_prediction_chunks(oracle_mod, kind, nq, nt, nsig):
    """Fused prediction against the stored kernel times the weights; a query's
    value does not depend on the queries beside it."""
    rng = np.random.default_rng(nq + nt)
    d = 21
    Q, T = rng.normal(size=(nq, d)), rng.normal(size=(nt, d))
    alpha = rng.normal(size=(nsig, nt))
    sig = [1.0 + 0.5 * k for k in range(nsig)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    lib = _lib.load()
    sp = (ctypes.c_double * nsig)(*sig)
    Td, ad = dev(T), dev(alpha)

    def predict(q):
        n = len(q)
        y = torch.empty((nsig, n), dtype=torch.float64, device="cuda")
        ws = torch.empty(lib.fmlb_kernel_predict_workspace_bytes(n, nt, nsig), dtype=torch.uint8,
                         device="cuda")
        qd = dev(q)
        _lib.call("fmlb_kernel_predict_f64", kind, _lib.ptr(qd), n, d, _lib.ptr(Td), nt, d, d,
                  ctypes.cast(sp, ctypes.POINTER(ctypes.c_double)), nsig, _lib.ptr(ad), nt,
                  _lib.ptr(y), n, _lib.ptr(ws), ws.numel(), _lib.stream_handle())
        return y.cpu().numpy()

    y = predict(Q)
    fn = oracle_mod.gaussian_kernel if kind == 0 else oracle_mod.laplacian_kernel
    for k in range(nsig):
        K = fn(Q.T, T.T, sig[k])
        # two sums of nt terms in different orders, a few ulp of each kernel entry
        tol = (2 * nt + 64) * 2.0 ** -53 * (K @ np.abs(alpha[k])).max()
        np.testing.assert_allclose(y[k], K @ alpha[k], rtol=0, atol=tol)
    assert np.array_equal(y[:, nq // 2:nq // 2 + 1], predict(Q[nq // 2:nq // 2 + 1]))


@pytest.mark.parametrize("amax,nm1,nm2,d,nsig", [(1, 3, 200, 5, 1), (7, 40, 33, 16, 32),
                                                 (23, 9, 70, 9, 2), (65, 5, 4, 8, 3),
                                                 (128, 2, 3, 17, 1)])
@pytest.mark.parametrize("kind", ["gaussian", "laplacian"])
def test_vector_kernel_groups(oracle_mod, kind, amax, nm1, nm2, d, nsig):
    """Groups of molecules of every size, with empty and full molecules."""
    rng = np.random.default_rng(amax)
    n1, n2 = rng.integers(0, amax + 1, nm1), rng.integers(0, amax + 1, nm2)
    n1[0], n2[-1] = amax, 0
    x1, x2 = rng.normal(size=(d, amax, nm1)), rng.normal(size=(d, amax, nm2))
    sig = list(np.linspace(1.0, 4.0, nsig))
    if kind == "gaussian":
        K = fml_b200.fget_vector_kernels_gaussian(x1, x2, n1, n2, sig, nm1, nm2, nsig)
    else:
        K = fml_b200.get_atomic_kernels_laplacian(x1, x2, n1, n2, sig)
    ref = oracle_mod.vector_kernels(kind, x1.transpose(2, 1, 0), x2.transpose(2, 1, 0), n1, n2, sig)
    np.testing.assert_allclose(K, ref, rtol=1e-13, atol=1e-300)
    assert (K[:, :, -1] == 0.0).all()
