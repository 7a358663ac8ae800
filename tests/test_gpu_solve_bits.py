"""A uniform solve gives the same bits at every CTA size of the operator kernels
(what the autotuner chooses by time), on the FP32 and the FP64 inner operator."""
import numpy as np
import pytest

from amps_gb300 import _capi
from tests import gpu_cases as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner_fp64", [False, True])
@pytest.mark.parametrize("nb", [(1, 1, 1), (3, 2, 2)])
def test_bits_do_not_depend_on_the_cta_size(nb, inner_fp64):
    wl, ic, x, f = G.make_case(nb=nb, ppc=4, seed=31)
    with G.gpu_ctx(wl, ic, x, f) as ctx:
        ctx.set_inner_fp64(inner_fp64)
        ctx.UpdateJMassMatrix()
        out = []
        for tb in (64, 128, 256):
            ctx.set_tuning(tb, 304)
            ctx.import_fields(**f)
            st = ctx.TimeStep(tol=1e-10, maxit=200, precond=1)
            assert st.converged
            out.append((st.iterations, st.rel_residual, ctx.export_fields()))
    for its, rel, e in out[1:]:
        assert (its, rel) == out[0][:2]
        for k, v in e.items():
            np.testing.assert_array_equal(v, out[0][2][k])


def test_refused_tuning():
    wl, ic, x, f = G.make_case(nb=(1, 1, 1), ppc=1)
    with G.gpu_ctx(wl, ic, x, f) as ctx:
        for tb, red in ((32, 304), (512, 304), (256, 0), (256, 305)):
            with pytest.raises(_capi.AmpsGpuError):
                ctx.set_tuning(tb, red)
