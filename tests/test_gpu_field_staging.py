"""Pageable fields that together pass the staging bound: they arrive as smaller
ones do, and the staging that the context keeps is one field's (or 64 MB)."""
import numpy as np
import pytest
import torch

import amps_gb300 as A

pytestmark = pytest.mark.gpu

KEYS = ("E_n", "E_half", "B_center", "B_corner_prev", "B_corner_cur")


# 884,736 points of 21 MB a field: three in the batch, two after it; 2,097,152 of 50 MB: one, four
@pytest.mark.parametrize("nb", [(12, 12, 12), (16, 16, 16)])
def test_large_pageable_fields(nb):
    wl = A.electron_proton_plasma("t", *nb, 1, 1)
    rng = np.random.default_rng(nb[0])
    n = wl.mesh.ncells
    field = 24 * n
    pin = A.PinnedArrays()
    f = {k: rng.standard_normal((n, 3)) for k in KEYS}
    with A.EcsimContext(wl, capacity=16, track_ids=False) as ctx:
        ctx.import_fields(E_n=np.zeros((n, 3)))  # its staging: one field
        free0 = torch.cuda.mem_get_info()[0]
        ctx.import_fields(**f)
        out = ctx.export_fields()
        for k in KEYS:
            np.testing.assert_array_equal(out[k], f[k])
        # one field's staging was there before; 64 MB and the allocator's granularity
        assert free0 - torch.cuda.mem_get_info()[0] + field <= max(field, 64 << 20) + (4 << 20)
        mixed = {k: pin.empty((n, 3)) if q % 2 else np.empty((n, 3)) for q, k in enumerate(KEYS)}
        ctx.export_fields(out=mixed)
        for k in KEYS:
            np.testing.assert_array_equal(mixed[k], f[k])
    pin.free()
