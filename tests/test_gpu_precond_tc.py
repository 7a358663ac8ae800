"""The tensor-core network on values that BF16 and FP32 hold exactly: one dense
layer, two that move a single voxel and channel each, so every tap, both CTAs'
halves, the plane between them and the ring must be right to the last bit.

The inputs are whole numbers up to 2 and the weights -1, 0 or 1; as long as the
activations stay below 256 (asserted; BF16 has 8 bits) nothing is rounded, and the
FP32 sums (below 2^24) don't depend on their order.
"""
import numpy as np
import pytest

import amps_gb300 as A
from oracle import precond_oracle as PO

pytestmark = pytest.mark.gpu

SHAPES = ((27, 3, 32), (27, 32, 32), (27, 32, 3))


@pytest.mark.parametrize("dense", [0, 1, 2])
@pytest.mark.parametrize("samples", [1, 2, 77])  # one cluster; an odd tail beyond one wave of 152 SMs
def test_whole_numbers_are_exact(dense, samples):
    rng = np.random.default_rng(10 * dense + samples)
    ws = []
    for layer, (taps, cin, cout) in enumerate(SHAPES):
        w = np.zeros((taps, cin, cout), np.float32)
        if layer == dense:
            keep = rng.random(w.shape) < (0.1 if layer == 1 else 1.0)
            w[:] = np.where(keep, rng.integers(-1, 2, w.shape), 0)
        else:
            for n in range(cout):
                w[rng.integers(taps), rng.integers(cin), n] = rng.choice([-1, 1])
        ws.append(w)
    x = rng.integers(-2, 3, (samples, 1000, 3)).astype(np.float32)
    _, h1, h2, y = PO.forward(x, *ws)
    ref = PO.owned(y)
    with A.EcsimContext(A.electron_proton_plasma("pc", 1, 1, 1, 1, 3), capacity=4096, track_ids=False) as ctx:
        ctx.precond_load(*ws)
        got = ctx.precond_forward(x, tensor_cores=True)
    assert max(np.abs(h1).max(), np.abs(h2).max()) < 256
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(got, ref.astype(np.float32))
