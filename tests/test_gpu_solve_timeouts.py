"""A wait of the solve's Arnoldi step that gives up: the kernels end, the solve
reports DEVICE_TIMEOUT on every mesh and launch path and leaves E^n and B alone,
and with the limit restored the context solves as one that never saw it.

A limit of 0 lets every wait give up at once, whatever the copies do; the step
then computes on tiles that may not have landed, inside its own buffers, takes
part in every barrier and ends when its copies have."""
import numpy as np
import pytest

from amps_gb300 import _capi
from tests import gpu_cases as G
from tests.test_gpu_amr import amr_case, gpu_for

pytestmark = pytest.mark.gpu

LIMIT = 1 << 24


def uniform(nb, dt):
    wl, ic, x, f = G.make_case(nb=nb, ppc=2, seed=7)
    wl.dt = dt
    return lambda: G.gpu_ctx(wl, ic, x, f), f


def refined():
    mesh, wl, ic, x, f = amr_case(ppc=2, seed=7)
    wl.dt = 2.0
    return lambda: gpu_for(mesh, wl, ic, x, f), f


# one tile per CTA; several tiles per CTA, kept on chip and (at 26 vectors and more) streamed
@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("precond", [0, 1])
@pytest.mark.parametrize("case", [lambda: uniform((1, 1, 1), 0.5), lambda: uniform((5, 5, 4), 4.0), refined],
                         ids=["one_block", "100_blocks", "refined"])
def test_timeouts_are_reported(case, precond, graphs):
    make, f = case()

    def solve(ctx):
        ctx.import_fields(**f)
        return ctx.TimeStep(tol=1e-11, maxit=600, precond=precond)

    with make() as ctx, make() as ref:
        for c in (ctx, ref):
            c.set_graphs(graphs)
            c.UpdateJMassMatrix()
        for _ in range(2):  # the second as a captured cycle
            solve(ctx)
            solve(ref)
        ctx.set_wait_limit(0)
        for _ in range(2):
            with pytest.raises(_capi.AmpsGpuError) as e:
                solve(ctx)
            assert e.value.status == 4 and "bounded waits" in str(e.value)
            g = ctx.export_fields()
            for k in ("E_n", "B_center", "B_corner_cur"):
                np.testing.assert_array_equal(g[k], f[k])
        ctx.set_wait_limit(LIMIT)
        st, sr = solve(ctx), solve(ref)
        assert st.converged and st.rel_residual <= 1e-11
        assert abs(st.iterations - sr.iterations) <= 1
        a, b = ctx.export_fields(), ref.export_fields()
        # both to a residual of 1e-11 (the refined operator adds atomically): as in test_gpu_arnoldi
        assert G.rel_err(a["E_half"], b["E_half"]) < 1e-8
