"""The current-only corner export of an AMR context against the export of J and M."""
import numpy as np
import pytest

import amps_gb300 as A
from amps_gb300 import amr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb0,lmax,mode,frac", [((2, 2, 2), 0, 0, 0.5), ((4, 4, 4), 1, 0, 0.5),
                                                ((4, 4, 4), 2, 1, 0.4)])
def test_current_alone_equals_current_with_mass_matrix(nb0, lmax, mode, frac):
    """The same sums in the same order: equal bit for bit, into pageable and page-locked arrays."""
    wl = amr.AmrWorkload("j", nb0, lmax, mode, frac, 16)
    mesh = wl.mesh()
    ic = wl.initial_condition(mesh, seed=3)
    pin = A.PinnedArrays()
    with A.EcsimContext(wl.plasma, capacity=len(ic["spec"]), track_ids=False, amr_mesh=mesh) as ctx:
        ctx.import_particles_local(ic["u"], ic["v"], ic["spec"], ic["block"])
        ctx.import_fields(**amr.amr_initial_fields(mesh, wl.b0))
        ctx.UpdateJMassMatrix()
        J0, _ = ctx.export_moments(with_m=False)
        J1, _ = ctx.export_moments()
        J2, _ = ctx.export_moments(out=(pin.empty((ctx.ncorners, 3)), None))
        assert np.any(J0 != 0.0)
        assert np.array_equal(J0, J1) and np.array_equal(J2, J1)
    pin.free()
