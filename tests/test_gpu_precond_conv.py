"""The FP32 training kernels of the network at batch sizes on both sides of each slab height (1, 2
and 5 planes per item) and with more items than SMs, against the FP64 oracle.

Tolerances as in the other tests of these kernels: gradients are FP32 sums of up to 77,000
random-signed products, whose roundings random-walk to 2^-24 sqrt(N / 2) ~ 1.2e-5 of the sum at
most: 1e-4 of the largest entry; outputs are sums of 864 products: 1e-5."""
import numpy as np
import pytest

import amps_gb300 as A
from oracle import precond_oracle as PO
from tests.gpu_cases import rel_err
from tests.test_gpu_precond import random_samples, small_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 20, 77])
def test_training_kernels_match_oracle_across_slab_heights(S):
    rng = np.random.default_rng(S)
    wl, ctx = small_ctx(nb=(1, 1, 1), ppc=1)
    with ctx:
        w = A.init_precond_weights(seed=S, out_scale=0.5)
        ctx.precond_load(*w)
        x, e = random_samples(rng, S)
        loss, g = ctx.precond_loss_grad(x, e)
        y = ctx.precond_forward(x, tensor_cores=False)
    lref, gref = PO.loss_grad(x, e, *w)
    assert loss == pytest.approx(lref, rel=1e-5)
    for a, b in zip(g, gref):
        assert rel_err(a, b) < 1e-4
    assert rel_err(y, PO.owned(PO.forward(x, *w)[3])) < 1e-5
