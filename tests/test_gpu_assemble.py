"""The corner assembly of the uniform deposit and of the no-allocation entry point against a numpy
flush of the exported per-cell sums, on boxes whose periodic wrap meets every side of a tile.

Tolerance: a corner entry is an FP32 sum of at most 8 cells, 7 roundings of 2^-24 of its partial
sums (each at most the sum of the magnitudes, itself at most a few times the largest entry):
1e-6 of the largest entry."""
import ctypes as C

import numpy as np
import pytest

import amps_gb300 as A
from tests import gpu_cases as G

pytestmark = pytest.mark.gpu

OFF = np.array([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)])


def flush(mesh, cJ, cM):
    NX, NY, NZ = mesh.shape
    b, l = np.divmod(np.arange(mesh.ncells), 512)
    lo = np.stack([8 * (b % mesh.nbx) + l % 8, 8 * ((b // mesh.nbx) % mesh.nby) + (l // 8) % 8,
                   8 * (b // (mesh.nbx * mesh.nby)) + l // 64], 1)
    cor = []
    for o in OFF:
        p = (lo + o) % np.array([NX, NY, NZ])
        cor.append(p[:, 0] + NX * (p[:, 1] + NY * p[:, 2]))
    J, M = np.zeros((mesh.ncells, 3)), np.zeros((mesh.ncells, 27, 9))
    dig = {0: 0, -1: 1, 1: 2}
    pr = 0
    for c1 in range(8):
        np.add.at(J, cor[c1], cJ[:, 3 * c1:3 * c1 + 3])
        for c2 in range(c1 + 1):
            for a, e in {(c1, c2), (c2, c1)}:
                d = OFF[e] - OFF[a]
                slot = dig[d[0]] + 3 * dig[d[1]] + 9 * dig[d[2]]
                np.add.at(M, (cor[a], slot), cM[:, 9 * pr:9 * pr + 9])
            pr += 1
    return J / mesh.dx ** 3, M.reshape(-1, 243)


@pytest.mark.parametrize("nb", [(1, 1, 1), (1, 2, 1), (3, 1, 2)])
def test_assembly_equals_flush_of_the_cell_sums(nb):
    torch = pytest.importorskip("torch")
    wl, ic, x, f = G.make_case(nb=nb, ppc=3, seed=9)
    with G.gpu_ctx(wl, ic, x, f) as ctx:
        ctx.UpdateJMassMatrix()
        J, M = ctx.export_moments()
        cJ, cM = ctx.export_cell_moments()
        ex = ctx.export_particles()
        J0, M0 = flush(wl.mesh, cJ, cM)
        assert G.rel_err(J, J0) <= 1e-6 and G.rel_err(M, M0) <= 1e-6
        # the same particles through the entry point on caller-owned buffers
        key = ex["block"].astype(np.int64) * 512 + ex["cell"]
        start = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=wl.mesh.ncells))]).astype(np.int32)
        u = ((ex["x"] - A.block_origins(wl.mesh, ex["block"])) / wl.mesh.dx).astype(np.float32)
        t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
             (start, u.T, ex["v"].astype(np.float32).T, ex["spec"], f["B_corner_cur"])]
        dJ = torch.full((wl.mesh.ncells, 3), 7.0, dtype=torch.float64, device="cuda")
        dM = torch.full((wl.mesh.ncells, 243), 7.0, dtype=torch.float64, device="cuda")
        en = torch.zeros(1, dtype=torch.float64, device="cuda")
        ptr = [C.c_void_p(q.data_ptr()) for q in (*t, dJ, dM, en)]
        assert A.load().amps_gpu_update_j_mass_matrix_noalloc(C.byref(ctx.cfg), len(key), *ptr, None) == 0
        torch.cuda.synchronize()
        # the FP32 cell sums of the two paths differ by the particles' order within a cell: 27
        # particles at most per cell, sums of 2^-24 roundings as above
        assert G.rel_err(dJ.cpu().numpy(), J0) <= 1e-5 and G.rel_err(dM.cpu().numpy(), M0) <= 1e-5
