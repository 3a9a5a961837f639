"""Workspaces that a pipeline lays side by side stay aligned (no GPU needed)."""
import pytest

from fml_b200 import _lib


@pytest.mark.parametrize("n", [1, 127, 128, 1001, 12001, 16384, 32767])
@pytest.mark.parametrize("slices", [1, 6, 8])
def test_factor_workspaces_are_multiples_of_256(n, slices):
    lib = _lib.load(require_cuda=False)
    assert lib.fmlb_potrf_workspace_bytes(n) % 256 == 0
    assert lib.fmlb_potrf_ozaki_workspace_bytes(n, slices) % 256 == 0
