"""Waits of the triangular solves that run out: NaN in the solution after a short time,
no hang, and the next solve on the same workspace is right."""
import time

import pytest
import torch

from fml_b200 import _lib, cho_solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 1000, 148 * 128 + 300])
def test_waits_run_out(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, 8), dtype=torch.float64, device="cuda", generator=g)
    A = A @ A.t()
    A.diagonal().add_(float(n))
    y = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    ws = torch.empty(_lib.load().fmlb_potrf_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    L = A.clone()
    _lib.call("fmlb_potrf_f64", _lib.ptr(L), n, n, _lib.ptr(ws), _lib.ptr(info),
              _lib.stream_handle())

    def solve():
        x = y.clone()
        _lib.call("fmlb_potrs_f64", _lib.ptr(L), n, n, _lib.ptr(ws), _lib.ptr(x),
                  _lib.stream_handle())
        torch.cuda.synchronize()
        return x

    solve()
    try:
        _lib.call("fmlb_tc_test_hooks", 20000, 4)  # waits of about 10 us
        t = time.perf_counter()
        x = solve()
        # a wait per thread and block chain, not one for each block
        assert time.perf_counter() - t < 1.0
    finally:
        _lib.call("fmlb_tc_test_hooks", 0, 0)
    assert torch.isnan(x).all()
    assert torch.equal(solve(), cho_solve(A, y))
