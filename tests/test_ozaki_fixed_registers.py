"""The int8 update in the form that moves no registers between its warps (for builds
whose compiler grants another number): the same bits as the usual one."""
import numpy as np
import pytest
import torch

from fml_b200 import _lib

pytestmark = pytest.mark.gpu


def _syrk(C, P, s, hook):
    m, k = P.shape
    lib = _lib.load()
    Cd, Pd = torch.from_numpy(C.copy()).cuda(), torch.from_numpy(P).cuda()
    nb = lib.fmlb_syrk_ozaki_workspace_bytes(m, k, s)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        _lib.call("fmlb_tc_test_hooks", 0, hook)
        _lib.call("fmlb_syrk_lower_ozaki", _lib.ptr(Cd), m, m, _lib.ptr(Pd), k, k, 0, s,
                  _lib.ptr(ws), nb, _lib.ptr(info), _lib.stream_handle())
    finally:
        _lib.call("fmlb_tc_test_hooks", 0, 0)
    assert int(info.item()) == 0
    return Cd.cpu().numpy()


@pytest.mark.parametrize("m,k", [(1, 32), (129, 96), (700, 256)])
@pytest.mark.parametrize("s", [1, 2, 3, 4, 5, 6, 7, 8])
def test_same_bits(m, k, s):
    rng = np.random.default_rng(m + s)
    P, C = rng.standard_normal((m, k)), rng.standard_normal((m, m))
    np.testing.assert_array_equal(_syrk(C, P, s, 8), _syrk(C, P, s, 0))
