"""Atomic vector kernels with several molecules to a CTA on both sides: many
sigmas beside the largest groups, ragged last groups, empty and full molecules,
groups of more than one 64-row tile."""
import numpy as np
import pytest
import torch

import fml_b200

pytestmark = pytest.mark.gpu


def _groups(nm1, nm2, amax):
    """Molecules of a CTA per side (the rule of vector_kernels.cu, same amax)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = [max(1, min(8, 160 // amax))] * 2
    while True:
        q = 0 if g[0] >= g[1] else 1
        if g[q] == 1 or -(-nm1 // g[0]) * -(-nm2 // g[1]) >= (8 if g[q] * amax > 64 else 2) * sms:
            return tuple(g)
        g[q] = (g[q] + 1) // 2


@pytest.mark.parametrize("amax,nm1,nm2,d,nsig,groups", [
    (7, 300, 290, 5, 3, (8, 8)), (20, 290, 283, 5, 1, (8, 8)), (20, 300, 300, 3, 19, (8, 8)),
    (8, 300, 300, 3, 32, (8, 8)), (22, 260, 250, 3, 24, (7, 7)), (23, 220, 230, 9, 2, (6, 6)),
    (50, 110, 109, 7, 2, (3, 3)), (23, 40, 43, 9, 2, (2, 2)), (23, 30, 31, 5, 1, (1, 2)),
    (7, 100, 99, 5, 2, (4, 8)), (10, 80, 75, 5, 1, (4, 4))])
@pytest.mark.parametrize("kind", ["gaussian", "laplacian"])
def test_groups_of_several_molecules(oracle_mod, kind, amax, nm1, nm2, d, nsig, groups):
    assert _groups(nm1, nm2, amax) == groups
    rng = np.random.default_rng(amax + nsig)
    n1, n2 = rng.integers(0, amax + 1, nm1), rng.integers(0, amax + 1, nm2)
    n1[:8] = n2[-5:] = amax
    n1[9], n2[3] = 0, 0
    x1, x2 = rng.normal(size=(d, amax, nm1)), rng.normal(size=(d, amax, nm2))
    sig = list(np.linspace(1.0, 4.0, nsig))
    if kind == "gaussian":
        K = fml_b200.fget_vector_kernels_gaussian(x1, x2, n1, n2, sig, nm1, nm2, nsig)
    else:
        K = fml_b200.get_atomic_kernels_laplacian(x1, x2, n1, n2, sig)
    ref = oracle_mod.vector_kernels(kind, x1.transpose(2, 1, 0), x2.transpose(2, 1, 0), n1, n2, sig)
    # the same distances bit for bit; exponentials of arguments above -200 within 2 ulp of
    # one another, sums of at most 2500 of them in another order: below 2500 * 2^-53 + 4e-16
    np.testing.assert_allclose(K, ref, rtol=3e-13, atol=1e-300)
    assert (K[:, 9] == 0.0).all() and (K[:, :, 3] == 0.0).all()
