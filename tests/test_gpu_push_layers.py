"""Push and deposit with particles on the edges of a layer's staged slab (cell corners,
faces, the last FP32 offset below a face, in every layer of a block) and with velocities
whose components vanish, tie or swap order, against the oracle.

Tolerances: those of the push and deposit tests (FP32 positions and partial sums).  The
energy: squares, weights and sums are carried in FP32 pairs, whose error per particle is
below 2^-45; v itself is compared, so the reference energy is taken from the exported
FP32 velocities: 1e-12."""
import numpy as np
import pytest

import amps_gb300 as A
from tests import gpu_cases as G
from tests import oracle_lib as O
from tests.test_gpu_ecsim import compare_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("centre", [False, True])
@pytest.mark.parametrize("nb", [(1, 1, 1), (2, 1, 3), (3, 3, 1), (5, 2, 1)])  # rows in parts up to 9 blocks
def test_slab_edges_and_velocity_orders(nb, centre):
    wl, _, _, f = G.make_case(nb=nb, ppc=1, seed=51)
    n3 = np.array(wl.mesh.shape)
    cells = np.stack(np.meshgrid(*[np.arange(n) for n in n3], indexing="ij"), -1).reshape(-1, 3)
    below = float(np.nextafter(np.float32(1), np.float32(0)))
    off = np.array([[0, 0, 0], [0.5, 0, 0.5], [below, below, 0], [0.25, 0.75, 1 - 2.0 ** -20]])
    x = (cells[:, None, :] + off[None]).reshape(-1, 3) * wl.mesh.dx
    kinds = 0.03 * np.array([[0, 0, 0], [1, 0, 0], [0, -1, 0], [0, 0, 1], [1, 1, 1], [-1, 2, -3], [3, -2, 1],
                             [2, 2, -1], [1e-3, 1, -1e3]])
    v = kinds[np.arange(len(x)) % len(kinds)].astype(np.float32)
    ic = {"v": v, "spec": (np.arange(len(x)) % 2).astype(np.uint8)}
    with A.EcsimContext(wl, capacity=4 * len(x), track_ids=True) as ctx:
        ctx.import_particles(x, v.astype(np.float64), ic["spec"])
        ctx.import_fields(**f)
        ctx.set_b_center(centre)
        st = O.OracleState(wl, x, v.astype(np.float64), ic["spec"], f, b_center=centre)
        eg = ctx.push_deposit()
        st.push()
        st.deposit()
        compare_particles(ctx, st)
        e = ctx.export_particles()
        J, M = ctx.export_moments()
    assert G.rel_err(J, st.J) <= 1e-5 and G.rel_err(M, st.M) <= 1e-5
    ke = np.array([0.5 * s.mass * s.weight for s in wl.species])
    assert eg == pytest.approx(np.sum(ke[e["spec"]] * np.sum(e["v"] ** 2, axis=1)), rel=1e-12)
