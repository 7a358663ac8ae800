"""What a tracing call holds on the device: 36 (FP32) or 60 (FP64) bytes per
particle (6 components, the step count and the status) and a staging area that
does not grow with the batch; and batches on either side of the staged chunks
(2^18 particles) give each particle its own trajectory."""
import threading
import time

import numpy as np
import pytest
import torch

from amps_gb300 import tracer as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,per_particle", [(0, 60), (1, 36)])
def test_device_memory_of_a_large_batch(precision, per_particle):
    n = 6_000_000
    x, p = (np.tile(a, (n // 60_000, 1)) for a in T.sphere_starts(60_000, 5))
    T.trace_cutoff(1000, precision=precision, max_steps=5)  # modules loaded
    free0 = torch.cuda.mem_get_info()[0]
    low, done = [free0], threading.Event()

    def watch():
        while not done.is_set():
            low[0] = min(low[0], torch.cuda.mem_get_info()[0])
            time.sleep(1e-3)

    t = threading.Thread(target=watch)
    t.start()
    try:
        T.trace_cutoff(n, precision=precision, max_steps=50, starts=(x, p))
    finally:
        done.set()
        t.join()
    used = free0 - low[0]
    # the call was seen; 12.6 MB of staging and the allocator's granularity (2 MB)
    assert per_particle * n <= used <= per_particle * n + (32 << 20)


@pytest.mark.parametrize("precision", [0, 1])
def test_chunks_keep_their_particles(precision):
    n = (1 << 19) + 5
    starts = T.sphere_starts(n, 9)
    whole = T.trace_cutoff(n, precision=precision, max_steps=20, starts=starts)
    for idx in (np.arange(1 << 18), np.arange((1 << 18) - 3, (1 << 18) + 3), np.arange(1 << 19, n)):
        part = T.trace_cutoff(len(idx), precision=precision, max_steps=20, starts=tuple(a[idx] for a in starts))
        for k in range(4):
            np.testing.assert_array_equal(part[k], whole[k][idx])
