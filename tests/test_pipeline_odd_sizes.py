"""KRRPipeline with an odd number of training points and several sigmas.

A sigma's kernel matrix, weights and factor workspace then start 8 bytes off a
16-byte boundary in every second place of the pipeline's stacked arrays. The
same sigma in three places has to give the same bits as one pipeline with that
sigma alone (kernels, factors, solves and predictions are formed in one order
whatever the alignment), which needs no tolerance.
"""

import pytest
import torch

from fml_b200 import synthetic
from fml_b200.krr import KRRPipeline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("factor", ["fp64", "ozaki"])
@pytest.mark.parametrize("n", [129, 1001, 2177])
def test_sigmas_side_by_side_give_the_bits_of_one(factor, n):
    b = synthetic.generate(n + 33, nmax=11, seed=5)
    args = [torch.from_numpy(v).cuda() for v in (b.charges, b.coords, b.offsets, b.energies[:n])]
    one = KRRPipeline(b.nmol, n, 11, [400.0], 1e-6, factor=factor)
    ref = one.run(*args).clone()
    three = KRRPipeline(b.nmol, n, 11, [400.0] * 3, 1e-6, factor=factor)
    got = three.run(*args)
    assert (one.info.cpu() == 0).all() and (three.info.cpu() == 0).all()
    assert torch.isfinite(ref).all()
    for q in range(3):
        assert torch.equal(got[q], ref[0]), q
