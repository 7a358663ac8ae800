"""The Arnoldi step of the field solve at the sizes where its tiling changes:
one CTA's worth of tiles kept on chip, more tiles than stages (large bases
included: the solves run through whole restart cycles), a vector length that is
no multiple of the stream alignment.  Each solve must reach a residual of 1e-11
and agree with the oracle's FP64 GMRES(30) from the same moments.

Tolerance: the solution error is at most the condition number times the
residual.  With theta = 1/2, dx = 1 the operator's eigenvalues lie between 1
and 1 + (dt/2)^2 (12 + 1) ~ 60 at dt = 4 (60 x 1e-11 = 6e-10 in the 2-norm; a
factor 15 for the largest component): 1e-8."""
import ctypes as C

import numpy as np
import pytest

from amps_gb300 import amr
import amps_gb300 as A
from tests import gpu_cases as G
from tests.oracle_lib import p
from tests.test_gpu_amr import gpu_for, oracle_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,dt", [((1, 1, 1), 0.1), ((2, 1, 3), 4.0), ((5, 5, 4), 4.0)])
def test_uniform_solve_matches_oracle(nb, dt):
    wl, ic, x, f = G.make_case(nb=nb, ppc=2, seed=7)
    wl.dt = dt
    with G.gpu_ctx(wl, ic, x, f) as ctx:
        ctx.UpdateJMassMatrix()
        st = ctx.TimeStep(tol=1e-11, maxit=600, precond=0)
        assert st.converged and st.rel_residual <= 1e-11
        g = ctx.export_fields()
        J, M = ctx.export_moments()
    o = G.oracle_state(wl, ic, x, f)
    o.J[:], o.M[:] = J, M
    b = o.rhs()
    dE, res = np.zeros_like(b), np.zeros(1)
    o.lib.orc_gmres(C.byref(o.m), p(o.M), p(b), p(dE), 1e-12, 3000, 30, 0, p(res))
    assert G.rel_err(g["E_half"], o.E_n + dE) < 1e-8


def test_vector_length_off_the_stream_alignment():
    nb0 = (4, 4, 4)
    mesh = amr.AmrMesh(nb0, 1, amr.nested_leaves(nb0, 1, 0, 0.5), open_axes=(True, True, True))
    assert 3 * mesh.ncorners % 4 == 3
    wl = A.electron_proton_plasma("odd", 1, 1, 1, 2, 1, dt=0.5)
    ic = amr.amr_initial_condition(mesh, wl.species, 2, seed=5)
    x = mesh.block_origins()[ic["block"]] + ic["u"].astype(np.float64) * mesh.block_dx()[ic["block"]][:, None]
    rng = np.random.default_rng(5)
    nc, ncell = mesh.ncorners, mesh.ncells
    f = {k: 2e-3 * rng.standard_normal((nc, 3)) for k in ("E_n", "E_half")}
    f["B_center"] = np.array(wl.b0) + 0.05 * rng.standard_normal((ncell, 3))
    f["B_corner_prev"] = f["B_corner_cur"] = np.array(wl.b0) + 0.05 * rng.standard_normal((nc, 3))
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
