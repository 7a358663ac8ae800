"""The relativistic Boris mover over exactly one gyro period: every particle's
remaining time equals its sub-step limit to within rounding, whichever side the
rounding of the limit falls on.  On a periodic mesh none may be lost.

The particles sit at rest on the corners (gamma = 1, interpolation weight 1) of
a field of one magnitude and random directions, so |B|^2 differs by rounding
alone; the magnitudes are ones at which 2 pi / |B| rounds to above 2 pi / B0 for
a part of the directions."""
import numpy as np
import pytest

import amps_gb300 as A
from tests.gpu_cases import make_case
from tests.test_gpu_amr import amr_case, gpu_for

pytestmark = pytest.mark.gpu

MAGNITUDES = (0.465609570169658, 0.5258696623555813, 0.7215675499372012, 0.7993580754603049)


def fields_of(f, b0, seed):
    """no E, corner B of magnitude b0 in random directions"""
    rng = np.random.default_rng(seed)
    out = {k: np.zeros_like(v) for k, v in f.items()}
    d = rng.standard_normal(f["B_corner_cur"].shape)
    out["B_corner_cur"] = b0 * (d / np.linalg.norm(d, axis=-1, keepdims=True))
    return out


def gyrate(ctx, x, f):
    for q, b0 in enumerate(MAGNITUDES):
        ctx.import_fields(**fields_of(f, b0, q))
        for spec in (0, 1):
            s = ctx.wl.species[spec]
            period = 2.0 * np.pi / (abs(s.charge) / s.mass) / b0
            ctx.import_particles(x, np.zeros_like(x), np.full(len(x), spec, np.uint8))
            ctx.MoveParticlesRelativistic(period, 1.0)
            assert ctx.num_particles() == len(x)
            assert ctx.deleted_particles() == 0
            e = ctx.export_particles()
            assert not e["v"].any()


def test_uniform_mesh_keeps_every_particle():
    wl, _, _, f = make_case(nb=(2, 2, 2), ppc=1)
    i = np.indices(wl.mesh.shape).reshape(3, -1).T.astype(np.float64)
    x = np.array(wl.mesh.x0) + i * np.array(wl.mesh.dx)
    with A.EcsimContext(wl, capacity=len(x) + 1024, track_ids=True) as ctx:
        gyrate(ctx, x, f)


def test_refined_mesh_keeps_every_particle():
    mesh, wl, ic, x, f = amr_case(ppc=1)
    i = np.indices((8, 8, 8)).reshape(3, -1).T.astype(np.float64)
    x = (mesh.block_origins()[:, None] + i[None] * mesh.block_dx()[:, None, None]).reshape(-1, 3)
    ic = {"v": np.zeros_like(x), "spec": np.zeros(len(x), np.uint8)}
    with gpu_for(mesh, wl, ic, x, f) as ctx:
        gyrate(ctx, x, f)
