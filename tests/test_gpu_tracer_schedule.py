"""The tracer's result is one trajectory per particle: it must not depend on which lane, warp or CTA
a particle runs in, nor on when states are packed or refilled.  A batch that fills the chip several
times over, parts of it, and single particles give the same bits."""
import numpy as np
import pytest

from amps_gb300 import tracer as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n", [(0, 60001), (1, 300007)])
def test_results_do_not_depend_on_the_batch(precision, n):
    starts = T.sphere_starts(n, 5)
    whole = T.trace_cutoff(n, precision=precision, max_steps=150, starts=starts)
    assert whole[4] == int(whole[3].sum())
    rng = np.random.default_rng(1)
    for idx in (np.arange(33), rng.permutation(n)[:1025], np.array([n - 1])):
        part = T.trace_cutoff(len(idx), precision=precision, max_steps=150,
                              starts=tuple(a[idx] for a in starts))
        for k in range(4):
            assert np.array_equal(part[k], whole[k][idx])
