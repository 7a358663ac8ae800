"""Field import and export with page-locked, pageable and absent arrays in one call."""
import numpy as np
import pytest

import amps_gb300 as A
from tests import gpu_cases as G

pytestmark = pytest.mark.gpu

KEYS = ("E_n", "E_half", "B_center", "B_corner_prev", "B_corner_cur")


@pytest.mark.parametrize("pinned", [(), ("E_n",), ("E_half", "B_corner_cur"), KEYS])
def test_round_trip_with_mixed_host_memory(pinned):
    wl = A.electron_proton_plasma("t", 1, 2, 3, 1, 1)
    rng = np.random.default_rng(len(pinned))
    n = wl.mesh.ncells
    pin = A.PinnedArrays()

    def arr(k):
        return pin.empty((n, 3)) if k in pinned else np.empty((n, 3))
    f = {k: arr(k) for k in KEYS}
    for a in f.values():
        a[:] = rng.standard_normal((n, 3))
    with A.EcsimContext(wl, capacity=16, track_ids=False) as ctx:
        ctx.import_fields(**f)
        out = {k: arr(k) for k in KEYS}
        ctx.export_fields(out=out)
        assert all(np.array_equal(out[k], f[k]) for k in KEYS)
        new = rng.standard_normal((n, 3))
        ctx.import_fields(B_center=new)
        part = {k: arr(k) if k in ("E_half", "B_center") else None for k in KEYS}
        ctx.export_fields(out=part)
        assert np.array_equal(part["E_half"], f["E_half"]) and np.array_equal(part["B_center"], new)
    pin.free()
