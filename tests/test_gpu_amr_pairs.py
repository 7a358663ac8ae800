"""The AMR operator and right-hand side in FP32 pairs, at numbers of 16-cell tiles
below one per resident CTA, between one and two, and beyond (tiles claimed one by
one), with and without hanging corners: a solve's E^{n+theta} against the oracle's
FP64 GMRES(30) from the same moments.

Tolerance: the solution error is at most the condition number times the relative
residual (1e-11), on top of the operator's own error (~1e-13 in pairs; FP32 would
leave 1e-7).  With theta = 1/2, dt = 1/2 and a finest cell of 1/2 the curl-curl part
lies below (dt/2)^2 12 / dx^2 = 3 and the mass term below that of the plasma
frequency, so the condition is below 10; a factor 15 for the largest component
leaves 1.5e-9: 1e-8."""
import pytest

from tests import gpu_cases as G
from tests.test_gpu_amr import amr_case, gpu_for, oracle_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb0,lmax,tiles", [((2, 2, 2), 0, 256), ((3, 3, 3), 1, 1088), ((4, 4, 4), 1, 3840)])
def test_solve_matches_oracle(nb0, lmax, tiles):
    mesh, wl, ic, x, f = amr_case(nb0=nb0, lmax=lmax, ppc=2, seed=31)
    assert mesh.ncells == 16 * tiles
    wl.dt = 0.5
    with gpu_for(mesh, wl, ic, x, f) as ctx:
        ctx.UpdateJMassMatrix()
        st = ctx.TimeStep(tol=1e-11, maxit=600, precond=0)
        assert st.converged and st.rel_residual <= 1e-11
        g = ctx.export_fields()
        cJ, cM = ctx.export_cell_moments()
    ao = oracle_for(mesh, wl, ic, x, f)
    ao.cellJ[:], ao.cellM[:] = cJ.reshape(-1), cM.reshape(-1)
    ao.field_solve(tol=1e-12, maxit=3000)
    assert G.rel_err(g["E_half"], ao.E_half) < 1e-8
