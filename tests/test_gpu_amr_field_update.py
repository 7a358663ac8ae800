"""The AMR field update after the solve (B^{n+1} from the curl, corner B from cell B,
E^{n+1}, wave energy) against the oracle, without hanging corners and with one and
two levels of them (edges and faces of blocks, corners of one block's own lattice).

Tolerance: E^{n+theta} is solved to a relative residual of 1e-11 with a condition
below 30 (theta = 1/2, dt = 1/2, finest cell 1/4): 1e-11 x 30 x 15 for the largest
component = 5e-9.  E^{n+1} = 2 E^{n+theta} - E^n doubles it: 1e-8.  B changes by
dt curl E, |E| below |B|: 1e-8.  The energy is quadratic in both: 2e-8."""
import pytest

from tests import gpu_cases as G
from tests.test_gpu_amr import amr_case, gpu_for, oracle_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb0,lmax", [((1, 1, 1), 0), ((2, 1, 3), 0), ((3, 3, 3), 1), ((4, 4, 4), 2)])
def test_update_matches_oracle(nb0, lmax):
    mesh, wl, ic, x, f = amr_case(nb0=nb0, lmax=lmax, ppc=2, seed=41)
    wl.dt = 0.5
    with gpu_for(mesh, wl, ic, x, f) as ctx:
        ctx.UpdateJMassMatrix()
        st = ctx.TimeStep(tol=1e-11, maxit=600, precond=1)
        assert st.converged
        g = ctx.export_fields()
        cJ, cM = ctx.export_cell_moments()
    ao = oracle_for(mesh, wl, ic, x, f)
    ao.cellJ[:], ao.cellM[:] = cJ.reshape(-1), cM.reshape(-1)
    ref = ao.field_solve(tol=1e-12, maxit=3000)
    assert G.rel_err(g["E_n"], ao.E_n) < 1e-8
    assert G.rel_err(g["B_center"], ao.Bcen) < 1e-8
    assert G.rel_err(g["B_corner_cur"], ao.Bcur) < 1e-8
    assert st.wave_energy == pytest.approx(ref[-1], rel=2e-8)
