"""A step limit that means none: the largest values are accepted, and particles
that leave end as they do at any limit above their steps."""
import numpy as np
import pytest

from amps_gb300 import tracer as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("max_steps", [1 << 60, 9 * 10 ** 18, 2 ** 63 - 1])
def test_any_step_limit(precision, max_steps):
    # 10^5 GV, outward: hardly bent on the way to 10 Earth radii
    x, p = T.sphere_starts(300, 3, rig_gv=(1e5, 2e5))
    p = np.linalg.norm(p, axis=1, keepdims=True) * x / np.linalg.norm(x, axis=1, keepdims=True)
    ref = T.trace_cutoff(300, precision=precision, max_steps=100000, starts=(x, p))
    assert (ref[2] == 2).all()
    got = T.trace_cutoff(300, precision=precision, max_steps=max_steps, starts=(x, p))
    for k in range(5):
        np.testing.assert_array_equal(got[k], ref[k])
