"""A captured first cycle serves any tolerance: solves of one system whose
tolerance changes from call to call take the iterations and give the field that
a stream solve at that tolerance does, whatever cycles are kept from before."""
import pytest

from tests import gpu_cases as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [0, 1])
def test_kept_cycles_take_the_tolerance_of_the_call(precond):
    wl, ic, x, f = G.make_case(nb=(2, 2, 2), ppc=4, seed=19)
    wl.dt = 0.5
    with G.gpu_ctx(wl, ic, x, f) as ctx:
        ctx.UpdateJMassMatrix()

        def solve(tol):
            ctx.import_fields(**f)
            st = ctx.TimeStep(tol=tol, maxit=200, precond=precond)
            assert st.converged and st.rel_residual <= tol
            return st.iterations, ctx.export_fields()["E_half"]

        tight, loose = 1e-10, 1e-4
        its, E = solve(tight)  # graphs off
        assert solve(loose)[0] < its <= 30
        ctx.set_graphs(True)
        # a cycle of `its` steps captured at the loose tolerance, then as many at the
        # tight one: the first of those starts from the loose solve's step count
        # (a restart), the later ones from their own
        solve(tight)
        solve(loose)
        solve(tight)
        for _ in range(3):
            n, e = solve(tight)
            assert n == its
            # residuals of 1e-10 of an operator with eigenvalues in [1, 2]
            assert G.rel_err(e, E) < 15 * tight
