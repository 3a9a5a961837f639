"""The FP64 distance tiles of 16, 32 and 64 rows: an entry is summed by one thread
in the features' order, so it is the same, bit for bit, whichever the size of the
call selects, in the symmetric form too; a prediction likewise."""
import pytest
import torch

import fml_b200
from fml_b200 import _lib

pytestmark = pytest.mark.gpu


def _rows(n, d, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((n, d), dtype=torch.float64, device="cuda", generator=g)


@pytest.mark.parametrize("kernel", [fml_b200.gaussian_kernel, fml_b200.laplacian_kernel])
@pytest.mark.parametrize("na,nb", [(1, 65), (16, 2367), (17, 2369), (63, 3000), (96, 1025),
                                   (97, 1000), (161, 1200)])
def test_rows_of_a_larger_call(kernel, na, nb):
    X = _rows(4096, 37, na)
    full = kernel(X.t(), X[:nb].t(), [3.0, 9.0])  # 64-row tiles
    part = kernel(X[:na].t(), X[:nb].t(), [3.0, 9.0])
    assert torch.equal(part, full[:, :na])


@pytest.mark.parametrize("n", [33, 449, 500, 544, 993, 1025, 1536, 1537])
def test_symmetric_form(n):
    X = _rows(n, 37, n)
    a = X.t()
    K = fml_b200.laplacian_kernel(a, a, 5.0)
    assert torch.equal(K, K.t())
    assert torch.equal(K, fml_b200.laplacian_kernel(a, X.clone().t(), 5.0))


@pytest.mark.parametrize("nq,nt", [(1, 1000), (511, 1000), (577, 1000), (33, 8200), (641, 2300)])
def test_predictions_of_a_larger_call(nq, nt):
    Q, T = _rows(4096, 37, nq), _rows(nt, 37, nt + 1)
    w = _rows(1, nt, 5)[0]
    sp, keep = _lib.host_doubles([4.0])

    def predict(n):
        y = torch.empty(n, dtype=torch.float64, device="cuda")
        ws = torch.empty(_lib.load().fmlb_kernel_predict_workspace_bytes(n, nt, 1),
                         dtype=torch.uint8, device="cuda")
        _lib.call("fmlb_kernel_predict_f64", 1, _lib.ptr(Q), n, 37, _lib.ptr(T), nt, 37, 37, sp, 1,
                  _lib.ptr(w), nt, _lib.ptr(y), n, _lib.ptr(ws), ws.numel(), _lib.stream_handle())
        return y

    assert torch.equal(predict(nq), predict(4096)[:nq])
    del keep
