"""What the speed of this framework is measured on: the calls a plasma run makes, through the
package's public entry points, over the range of meshes, fillings, precisions and options they are
used at.

A case is one of these kinds of work (`kind`):
  step     one PIC::TimeStep of the ECSIM track (field solve, move, deposit), then what a run
           writes out: corner E, centre B, the corner current, and the two energies it prints
  push     the particle half alone (push, re-bin, deposit), then the corner current
  deposit  UpdateJMassMatrix on device buffers that the caller owns, J and M handed on in FP32
  solve    the implicit field solve for a host code that keeps E and B itself
  tracks   test particles moved on the mesh fields, their states filed by particle id
  net      loss and weight gradients of the preconditioner network (one training mini-batch)
  trace    batched cutoff-rigidity tracing in a dipole

Everything is seeded; sizes come from the configurations of the package, its tests and its bench.
"""
import ctypes as C
import math

import numpy as np
import torch

import amps_gb300 as A
from amps_gb300 import _capi, amr

MASS_RATIO, VTH_E, B0, THETA = 25.0, 0.05, 0.5, 0.5
R_E, Q_P, C_LIGHT = 6371.2e3, 1.602176634e-19, 299792458.0
M_P = 1.007276466621 * 1.66053906660e-27
B_EQ, B_SOUTH, DPHI, DT_MAX = 3.1e-5, 5e-9, 0.15, 10.0


def listed():
    return [
        # the smallest run the tests make: one block, 4 particles per species and cell; launches,
        # synchronisations and copies are all of it
        {"name": "step_8c_4ppc", "kind": "step", "nbx": 1, "nby": 1, "nbz": 1, "lmax": 0,
         "ppc": 4, "dt": 0.1, "precond": 0, "graphs": True},
        # the plain ECSIM plasma: 32^3 cells, 64 particles per species and cell, Jacobi GMRES to 1e-8
        {"name": "step_32c_64ppc", "kind": "step", "nbx": 4, "nby": 4, "nbz": 4, "lmax": 0,
         "ppc": 64, "dt": 0.1, "precond": 1, "graphs": True},
        # the headline plasma: 64^3 base cells, central 1/8 refined, 67.1M particles
        {"name": "step_amr_64c_128ppc", "kind": "step", "nbx": 8, "nby": 8, "nbz": 8, "lmax": 1,
         "sphere": False, "frac": 0.5, "per_cell": False, "ppc": 128, "dt": 0.1, "precond": 1,
         "graphs": True},
        # three levels nested around a sphere, the same few weighted particles in cells of every
        # level, the reference's unpreconditioned solve, stream launches
        {"name": "step_amr3_128e_16ppc", "kind": "step", "nbx": 4, "nby": 4, "nbz": 4, "lmax": 2,
         "sphere": True, "frac": 0.4, "per_cell": True, "ppc": 16, "dt": 0.1, "precond": 0,
         "graphs": False},
        # the reference's default build: B at the cell centres; ragged box, chunks with a remainder
        {"name": "push_centre_b_5x3x4_27ppc", "kind": "push", "nbx": 5, "nby": 3, "nbz": 4,
         "centre": True, "ppc": 27, "dt": 0.1},
        # a host framework that owns all device memory: 12 blocks, the range of that entry point
        {"name": "deposit_2x2x3_24ppc", "kind": "deposit", "nbx": 2, "nby": 2, "nbz": 3, "ppc": 24,
         "dt": 0.1},
        # field solve with the learned preconditioner (BF16 tensor cores) on the plain plasma's mesh
        {"name": "solve_learned_32c", "kind": "solve", "nbx": 4, "nby": 4, "nbz": 4, "lmax": 0,
         "ppc": 8, "dt": 0.1, "precond": 2},
        # field solve at a time step an implicit scheme is chosen for, two levels, no preconditioner
        {"name": "solve_amr_64c_dt05", "kind": "solve", "nbx": 8, "nby": 8, "nbz": 8, "lmax": 1,
         "sphere": False, "frac": 0.5, "per_cell": False, "ppc": 8, "dt": 0.5, "precond": 0},
        # relativistic test particles on the mesh, FP64 sub-steps, trajectories kept by id
        {"name": "tracks_rel_24c_36ppc", "kind": "tracks", "nbx": 3, "nby": 3, "nbz": 3, "ppc": 36,
         "dt": 2.0, "rel": True},
        # one large mini-batch of the preconditioner's training
        {"name": "net_grad_256", "kind": "net", "samples": 256},
        # cutoff rigidity, FP32 and FP64, uneven lifetimes
        {"name": "trace_fp32_256k", "kind": "trace", "n": 262144, "max_steps": 2000, "precision": 1},
        {"name": "trace_fp64_20k", "kind": "trace", "n": 20000, "max_steps": 500, "precision": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "push", "push", "deposit", "solve", "solve", "tracks",
                       "net", "trace", "trace"])
    if kind == "net":
        return {"kind": kind, "samples": _log(rng, 8, 512)}
    if kind == "trace":
        fp32 = rng.random() < 0.5
        return {"kind": kind, "n": _log(rng, 1000, 300000) if fp32 else _log(rng, 500, 30000),
                "max_steps": _log(rng, 200, 2000) if fp32 else _log(rng, 100, 600),
                "precision": 1 if fp32 else 0}
    nb = {"nbx": rng.randint(1, 5), "nby": rng.randint(1, 5), "nbz": rng.randint(1, 5)}
    if kind == "deposit":
        nb = {"nbx": rng.randint(1, 2), "nby": rng.randint(1, 4), "nbz": rng.randint(1, 2)}
        return {"kind": kind, **nb, "ppc": _log(rng, 2, 64), "dt": rng.choice([0.1, 0.25])}
    if kind == "tracks":
        return {"kind": kind, **nb, "ppc": _log(rng, 2, 40), "dt": rng.choice([0.5, 2.0, 6.0]),
                "rel": rng.random() < 0.6}
    if kind == "push":
        return {"kind": kind, **nb, "centre": rng.random() < 0.5, "ppc": _log(rng, 3, 150), "dt": 0.1}
    c = {"kind": kind, **nb, "lmax": rng.choice([0, 0, 1, 2]), "dt": rng.choice([0.1, 0.2, 0.5]),
         "precond": rng.choice([0, 1, 2] if kind == "solve" else [0, 1])}
    c["ppc"] = _log(rng, 4, 12) if kind == "solve" else _log(rng, 3, 100)
    if c["lmax"]:
        c.update(nbx=rng.randint(4, 6), nby=rng.randint(4, 6), nbz=4, sphere=c["lmax"] == 2,
                 frac=0.4 if c["lmax"] == 2 else 0.5, per_cell=c["lmax"] == 2)
        if c["per_cell"]:
            c["ppc"] = min(c["ppc"], 20)
    if kind == "step":
        c["graphs"] = rng.random() < 0.5
    return c


# ---------------------------------------------------------------------------- inputs
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _plasma(case, seed, mesh=None):
    """Electrons and protons drawn together, uniform in every cell, Maxwellian: FP32 block-local
    offsets u, velocities v, species, block, weight corrections or None (tensors on the GPU)."""
    g, ppc = _gen(seed), case["ppc"]
    nb = mesh.nblocks if mesh is not None else case["nbx"] * case["nby"] * case["nbz"]
    level = torch.as_tensor(mesh.level, device="cuda").long() if mesh is not None else torch.zeros(
        nb, dtype=torch.int64, device="cuda")
    per_block = torch.full_like(level, ppc) if case.get("per_cell") else (ppc // 8 ** level).clamp(min=1)
    cell = torch.repeat_interleave(torch.arange(nb * 512, device="cuda"), per_block.repeat_interleave(512))
    l = cell % 512
    low = torch.stack([l % 8, (l // 8) % 8, l // 64], 1).float()
    u = (low + torch.rand(len(cell), 3, generator=g, device="cuda")).clamp(max=7.9999995)
    vth = torch.tensor([VTH_E, VTH_E / math.sqrt(MASS_RATIO)], device="cuda")
    v = torch.randn(len(cell), 2, 3, generator=g, device="cuda") * vth[:, None]
    spec = torch.tensor([0, 1], dtype=torch.uint8, device="cuda").repeat(len(cell))
    block = (cell // 512).int().repeat_interleave(2)
    wc = 0.125 ** level.float()[block.long()] if case.get("per_cell") else None
    return u.repeat_interleave(2, 0), v.reshape(-1, 3), spec, block, wc


def _waves(x, box, seed, salt, amp, mean):
    """A few periodic modes of the box at positions x (n, 3), FP64: (n, 3)."""
    g = _gen(seed, salt)
    f = torch.zeros_like(x) + torch.tensor(mean, dtype=torch.float64, device="cuda")
    for _ in range(4):
        k = torch.randint(-3, 4, (3,), generator=g, device="cuda").double() * (2 * math.pi / box)
        ph = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
        a = torch.randn(3, generator=g, device="cuda", dtype=torch.float64) * amp
        f += a * torch.sin((x @ k)[:, None] + ph)
    return f


def _lattice(case, off=0.0):
    n = [8 * case[k] for k in ("nbx", "nby", "nbz")]
    K, J, I = torch.meshgrid(*(torch.arange(m, device="cuda") for m in (n[2], n[1], n[0])), indexing="ij")
    return torch.stack([I, J, K], -1).reshape(-1, 3).double() + off, torch.tensor(n, device="cuda").double()


def _wave_fields(case, seed, e_amp=5e-3, b_amp=0.02):
    xc, box = _lattice(case)
    xm, _ = _lattice(case, 0.5)
    e = _waves(xc, box, seed, 1, e_amp, (0.0, 0.0, 0.0))
    b = [_waves(x, box, seed, 2, b_amp, (0.0, 0.0, B0)) for x in (xc, xm)]
    return {"E_n": e, "E_half": e, "B_center": b[1], "B_corner_prev": b[0], "B_corner_cur": b[0]}


def _noise_fields(case, seed, ncor, ncell):
    """E and B of the solve cases: the uniform field and the noise a particle run has in it."""
    g = _gen(seed, 3)
    e = 1e-3 * torch.randn(ncor, 3, generator=g, device="cuda", dtype=torch.float64)
    b0 = torch.tensor([0.0, 0.0, B0], dtype=torch.float64, device="cuda")
    bm = b0 + 0.02 * torch.randn(ncell, 3, generator=g, device="cuda", dtype=torch.float64)
    bc = b0 + 0.02 * torch.randn(ncor, 3, generator=g, device="cuda", dtype=torch.float64)
    return {"E_n": e, "E_half": e, "B_center": bm, "B_corner_prev": bc, "B_corner_cur": bc}


def _samples(case, seed):
    """Residual and correction pairs of the network, normalised to unit RMS as the harvest does."""
    g = _gen(seed, 4)
    x = torch.randn(case["samples"], 1000, 3, generator=g, device="cuda")
    e = x.reshape(-1, 10, 10, 10, 3)[:, 1:9, 1:9, 1:9].reshape(-1, 512, 3)
    return x, e * 0.9 + 0.1 * torch.randn(e.shape, generator=g, device="cuda")


def _weights(seed):
    return A.init_precond_weights(seed=int(seed) % 1000, out_scale=0.05)


def _starts(case, seed):
    """Protons on a sphere of 1.1 R_E, isotropic, rigidity log-uniform in 0.1-20 GV."""
    r = np.random.default_rng(seed)
    n = case["n"]
    out = []
    for _ in range(2):
        mu, ph = r.uniform(-1, 1, n), r.uniform(0, 2 * np.pi, n)
        s = np.sqrt(1 - mu ** 2)
        out.append(np.stack([s * np.cos(ph), s * np.sin(ph), mu], 1))
    rig = 10 ** r.uniform(8, math.log10(20e9), n)
    return 1.1 * R_E * out[0], (rig * Q_P / C_LIGHT)[:, None] * out[1]


def _pinned(*shape, dtype=torch.float64):
    return torch.empty(*shape, dtype=dtype, pin_memory=True)


def _context(case, seed, fields=None, track_ids=False):
    wl = A.electron_proton_plasma("case", case["nbx"], case["nby"], case["nbz"], case["ppc"], 1,
                                  dt=case["dt"])
    mesh = None
    if case.get("lmax"):
        nb0 = (case["nbx"], case["nby"], case["nbz"])
        mesh = amr.AmrMesh(nb0, case["lmax"], amr.nested_leaves(nb0, case["lmax"], int(case["sphere"]),
                                                                case["frac"]))
    u, v, spec, block, wc = _plasma(case, seed, mesh)
    ctx = A.EcsimContext(wl, capacity=len(spec), track_ids=track_ids, amr_mesh=mesh)
    if case.get("centre"):
        ctx.set_b_center(True)
    ctx.import_particles_local(*(t.cpu().numpy() for t in (u, v, spec, block)),
                               wcorr=None if wc is None else wc.cpu().numpy())
    if fields is None:
        fields = amr.amr_initial_fields(mesh, wl.b0) if mesh is not None else A.initial_fields(wl)
    else:
        fields = {k: t.cpu().numpy() for k, t in fields(ctx).items()}
    ctx.import_fields(**fields)
    return wl, ctx, len(spec)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "step":
        wl, ctx, s["n"] = _context(case, seed)
        ctx.set_graphs(case["graphs"])
        ctx.UpdateJMassMatrix()
        s.update(ctx=ctx, tol=wl.tol, out={"E_n": _pinned(ctx.ncorners, 3), "B_center": _pinned(ctx.ncells, 3)},
                 J=_pinned(ctx.ncorners, 3))
    elif kind == "push":
        wl, ctx, s["n"] = _context(case, seed, lambda c: _wave_fields(case, seed))
        s.update(ctx=ctx, J=_pinned(ctx.ncorners, 3))
    elif kind == "solve":
        host = {}

        def keep(ctx):
            f = _noise_fields(case, seed, ctx.ncorners, ctx.ncells)
            for k, t in f.items():
                host[k] = _pinned(*t.shape).copy_(t)
            return f
        wl, ctx, s["n"] = _context(case, seed, keep)
        if case["precond"] == 2:
            for k in range(ctx.precond_num_sets()):
                ctx.precond_select(k)
                ctx.precond_load(*_weights(seed + k))
            ctx.precond_select(0)
            ctx.precond_use_tensor_cores(True)
        ctx.UpdateJMassMatrix()
        s.update(ctx=ctx, tol=wl.tol, fields={k: t.numpy() for k, t in host.items()}, hold=host,
                 out={"E_n": _pinned(ctx.ncorners, 3), "B_center": _pinned(ctx.ncells, 3)})
    elif kind == "tracks":
        wl, ctx, n = _context(case, seed, lambda c: _wave_fields(case, seed), track_ids=True)
        s.update(ctx=ctx, x=_pinned(n, 3), v=_pinned(n, 3), id=_pinned(n, dtype=torch.int32),
                 tracks=torch.zeros(n, 6, device="cuda"))
    elif kind == "deposit":
        wl = A.electron_proton_plasma("case", case["nbx"], case["nby"], case["nbz"], case["ppc"], 1,
                                      dt=case["dt"])
        cfg = _capi.Config()
        cfg.nbx, cfg.nby, cfg.nbz = case["nbx"], case["nby"], case["nbz"]
        for d in range(3):
            cfg.x0[d], cfg.dx[d] = 0.0, 1.0
        cfg.nspec = 2
        for i, sp in enumerate(wl.species):
            cfg.charge[i], cfg.mass[i], cfg.weight[i] = sp.charge, sp.mass, sp.weight
        cfg.dt, cfg.theta = wl.dt, wl.theta
        u, v, spec, block, _ = _plasma(case, seed)
        ncell = wl.mesh.ncells
        start = torch.arange(ncell + 1, device="cuda", dtype=torch.int32) * (2 * case["ppc"])
        s.update(cfg=cfg, n=len(spec), start=start, u=u.T.contiguous(), v=v.T.contiguous(), spec=spec,
                 B=_wave_fields(case, seed)["B_corner_cur"].contiguous(), lib=A.load(),
                 J=torch.empty(ncell, 3, device="cuda", dtype=torch.float64),
                 M=torch.empty(ncell, 243, device="cuda", dtype=torch.float64),
                 e=torch.empty(1, device="cuda", dtype=torch.float64))
    elif kind == "net":
        wl = A.electron_proton_plasma("case", 1, 1, 1, 1, 1)
        ctx = A.EcsimContext(wl, capacity=16, track_ids=False)
        ctx.precond_load(*_weights(seed))
        x, e = _samples(case, seed)
        s.update(ctx=ctx, x=_pinned(*x.shape, dtype=torch.float32).copy_(x),
                 e=_pinned(*e.shape, dtype=torch.float32).copy_(e))
    else:
        s["x"], s["p"] = _starts(case, seed)
    return s


# ---------------------------------------------------------------------------- one pass
def _field_state(ctx, out):
    """The corner E and centre B a run writes out, in single precision."""
    host = {k: out[k].numpy() if k in out else None
            for k in ("E_n", "E_half", "B_center", "B_corner_prev", "B_corner_cur")}
    ctx.export_fields(out=host)
    return {k: t.float() for k, t in out.items()}


def run(state):
    kind = state["case"]["kind"]
    if kind == "step":
        st = state["ctx"].PicTimeStep(tol=state["tol"], maxit=400, precond=state["case"]["precond"])
        state["ctx"].export_moments(out=(state["J"].numpy(), None))
        return {"energy": torch.tensor([st.particle_energy, st.solve.wave_energy], dtype=torch.float32),
                "J": state["J"].float(), **_field_state(state["ctx"], state["out"])}
    if kind == "push":
        ctx = state["ctx"]
        energy = ctx.push_deposit()
        ctx.export_moments(out=(state["J"].numpy(), None))
        return {"energy": torch.tensor(energy, dtype=torch.float32), "J": state["J"].float()}
    if kind == "solve":
        ctx = state["ctx"]
        ctx.import_fields(**state["fields"])
        st = ctx.TimeStep(tol=state["tol"], maxit=400, precond=state["case"]["precond"])
        return {"energy": torch.tensor(st.wave_energy, dtype=torch.float32),
                **_field_state(ctx, state["out"])}
    if kind == "tracks":
        ctx, x, v, ids = state["ctx"], state["x"], state["v"], state["id"]
        if state["case"]["rel"]:
            ctx.MoveParticlesRelativistic(state["case"]["dt"])
        else:
            ctx.MoveParticlesBoris(state["case"]["dt"])
        n = C.c_longlong()
        f64 = C.POINTER(C.c_double)
        if ctx.lib.amps_gpu_export_particles(ctx.h, C.cast(x.data_ptr(), f64), C.cast(v.data_ptr(), f64), None,
                                             None, None, C.cast(ids.data_ptr(), C.POINTER(C.c_uint32)),
                                             C.byref(n)):
            raise RuntimeError("export_particles failed")
        at = ids.cuda(non_blocking=True).long()
        state["tracks"][at, :3] = x.cuda(non_blocking=True).float()
        state["tracks"][at, 3:] = v.cuda(non_blocking=True).float()
        return state["tracks"]
    if kind == "deposit":
        p = {k: C.c_void_p(state[k].data_ptr()) for k in ("start", "u", "v", "spec", "B", "J", "M", "e")}
        if state["lib"].amps_gpu_update_j_mass_matrix_noalloc(
                C.byref(state["cfg"]), state["n"], p["start"], p["u"], p["v"], p["spec"], p["B"], p["J"],
                p["M"], p["e"], C.c_void_p(torch.cuda.current_stream().cuda_stream)):
            raise RuntimeError("the deposit failed")
        return {"J": state["J"].float(), "M": state["M"].float(), "energy": state["e"].float()}
    if kind == "net":
        loss, g = state["ctx"].precond_loss_grad(state["x"].numpy(), state["e"].numpy())
        return {"loss": torch.tensor(loss, dtype=torch.float32), "g": g}
    x, p = state["x"].copy(), state["p"].copy()
    status, steps, total, _ = A.trace_dipole(x, p, Q_P, M_P, B_EQ, R_E, np.array([0.0, 0.0, -B_SOUTH]), R_E,
                                             10.0 * R_E, state["case"]["max_steps"], DPHI, DT_MAX,
                                             state["case"]["precision"])
    return {"x": x, "p": p, "status": status, "steps": steps, "total": total}


# ---------------------------------------------------------------------------- least work
def _sizes(case):
    """Cells and particles (AMR: of the refinement's nominal volume)."""
    base = 512 * case["nbx"] * case["nby"] * case["nbz"]
    if not case.get("lmax"):
        return base, 2 * case["ppc"] * base
    cells, vol, part = 0.0, 1.0, 0.0
    for lev in range(case["lmax"] + 1):
        h = case["frac"] / 2 ** lev
        inner = 0.0 if lev == case["lmax"] else (4.0 / 3.0 * math.pi * h ** 3 if case["sphere"] else h ** 3)
        here = base * 8 ** lev * (vol - min(inner, vol))
        cells += here
        part += here * (case["ppc"] if case["per_cell"] else max(1, case["ppc"] // 8 ** lev))
        vol = min(inner, vol)
    return int(cells), int(2 * part)


def work(case):
    kind = case["kind"]
    if kind == "net":
        s = case["samples"]
        macs = 27 * (1000 * 3 * 32 + 1000 * 32 * 32 + 512 * 32 * 3)
        return {"bytes": s * (1000 + 512) * 12 + 2 * 4 * 27 * (96 + 1024 + 96), "flops": s * 2 * macs * 3}
    if kind == "trace":
        return {"bytes": case["n"] * (2 * 48 + 12), "flops": 90.0 * case["n"] * case["max_steps"] * 0.3}
    cells, n = _sizes(case)
    part, mass, fields = 49.0 * n, 4.0 * 243 * cells, 24.0 * cells
    if kind == "step":  # state in and out, M written and read, E and B in and out; 8 operator products
        return {"bytes": part + 2 * mass + 8 * fields, "flops": 816.0 * n + 8 * 2 * 243 * cells}
    if kind == "push":
        return {"bytes": part + mass + 4 * fields, "flops": 816.0 * n}
    if kind == "deposit":
        return {"bytes": 25.0 * n + 2 * mass + 2 * fields, "flops": 600.0 * n}
    if kind == "solve":
        return {"bytes": mass + 8 * fields, "flops": 10 * 2.0 * 243 * cells}
    return {"bytes": 24.0 * n * 2 + 28.0 * n + 2 * fields, "flops": 260.0 * n}


# ---------------------------------------------------------------------------- 64-bit values
_D = dict(dtype=torch.float64, device="cuda")
_OFF = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _species64(case):
    w = 1.0 / (4.0 * math.pi * case["ppc"])
    return torch.tensor([-1.0, 1.0], **_D), torch.tensor([1.0, MASS_RATIO], **_D), w


def _n3(case):
    return torch.tensor([8 * case[k] for k in ("nbx", "nby", "nbz")], device="cuda")


def _index(ijk, n3):
    ijk = ijk % n3
    return ijk[..., 0] + n3[0] * (ijk[..., 1] + n3[1] * ijk[..., 2])


def _corners(x, n3):
    """The 8 corners' indices and trilinear weights at positions x (n, 3), cell size 1."""
    i = torch.floor(x)
    f = x - i
    for o in _OFF:
        w = torch.ones(len(x), **_D)
        for d in range(3):
            w = w * (f[:, d] if o[d] else 1.0 - f[:, d])
        yield _index(i.long() + torch.tensor(o, device="cuda"), n3), w


def _gather(x, field, n3):
    s = torch.zeros_like(x)
    for c, w in _corners(x, n3):
        s += w[:, None] * field[c]
    return s


def _alpha(h, B):
    c0 = 1.0 / (1.0 + h * h * (B * B).sum(1))
    hb = h[:, None] * B
    a = hb[:, :, None] * hb[:, None, :] + torch.eye(3, **_D)
    P = -hb
    z = torch.zeros_like(c0)
    a += torch.stack([torch.stack([z, -P[:, 2], P[:, 1]], 1), torch.stack([P[:, 2], z, -P[:, 0]], 1),
                      torch.stack([-P[:, 1], P[:, 0], z], 1)], 1)
    return c0[:, None, None] * a


def _positions(case, u, block):
    b = block.long()
    o = torch.stack([b % case["nbx"], (b // case["nbx"]) % case["nby"], b // (case["nbx"] * case["nby"])], 1)
    return 8.0 * o.double() + u.double()


def _push64(case, x, v, spec, E, B, centre):
    q, m, _ = _species64(case)
    n3 = _n3(case)
    h = (0.5 * case["dt"] * q / m)[spec.long()]
    Bp = _gather((x - 0.5) if centre else x, B, n3)
    vp = (_alpha(h, Bp) @ (v + h[:, None] * _gather(x, E, n3))[:, :, None])[:, :, 0]
    v = 2.0 * vp - v
    return (x + case["dt"] * v) % n3.double(), v


def _slot(d):
    dig = [0 if o == 0 else (1 if o < 0 else 2) for o in d]
    return dig[0] + 3 * dig[1] + 9 * dig[2]


def _deposit64(case, x, v, spec, B, centre=False, mass=True):
    """Corner J (n, 3) and M (n, 243), and the kinetic energy."""
    q, m, w0 = _species64(case)
    n3 = _n3(case)
    nc = int(n3.prod())
    J, M, en = torch.zeros(nc, 3, **_D), torch.zeros(nc * 27, 9, **_D) if mass else None, 0.0
    for p0 in range(0, len(x), 1 << 20):
        s = slice(p0, p0 + (1 << 20))
        X, V, sp = x[s], v[s], spec[s].long()
        h = (0.5 * case["dt"] * q / m)[sp]
        al = _alpha(h, _gather((X - 0.5) if centre else X, B, n3))
        qav = (q * w0)[sp][:, None] * (al @ V[:, :, None])[:, :, 0]
        en += float((0.5 * (m * w0)[sp] * (V * V).sum(1)).sum())
        cw = list(_corners(X, n3))
        for c, w in cw:
            J.index_add_(0, c, w[:, None] * qav)
        if mass:
            ka = ((q * w0)[sp] * h)[:, None] * al.reshape(-1, 9)
            for (c1, w1), o1 in zip(cw, _OFF):
                for (_, w2), o2 in zip(cw, _OFF):
                    M.index_add_(0, c1 * 27 + _slot([b - a for a, b in zip(o1, o2)]), (w1 * w2)[:, None] * ka)
    return J, M.reshape(nc, 243) if mass else None, en


def _roll(f, n, d):
    """f at index + d on the periodic lattice (n = (NX, NY, NZ))."""
    g = f.reshape(n[2], n[1], n[0], -1)
    return torch.roll(g, (-d[2], -d[1], -d[0]), (0, 1, 2)).reshape(f.shape)


def _solve64(case, E, Bm, J, M):
    """E^{n+1}, centre B^{n+1} and the wave energy of one implicit field update."""
    n = [8 * case[k] for k in ("nbx", "nby", "nbz")]
    dt, cth = case["dt"], case["dt"] * THETA
    f = 4.0 * math.pi * cth
    S, D1, D2 = {-1: .25, 0: .5, 1: .25}, {-1: -.5, 0: 0., 1: .5}, {-1: 1., 0: -2., 1: 1.}
    offs = [(i, j, k) for k in (-1, 0, 1) for j in (-1, 0, 1) for i in (-1, 0, 1)]
    taps = {}
    for o in offs:
        lap = [math.prod((D2 if d == a else S)[o[d]] for d in range(3)) for a in range(3)]
        K = torch.zeros(3, 3, **_D)
        for p in range(3):
            for r in range(3):
                gd = lap[p] if p == r else math.prod((D1 if d in (p, r) else S)[o[d]] for d in range(3))
                K[p, r] = gd - (sum(lap) if p == r else 0.0)
        taps[o] = cth * cth * K

    def curl_mass(x):  # (theta dt)^2 curl curl x + 4 pi theta dt M x
        y = torch.zeros_like(x)
        for o in offs:
            xs = _roll(x, n, o)
            y += xs @ taps[o].T + f * (M[:, 9 * _slot(o):9 * _slot(o) + 9].reshape(-1, 3, 3) @ xs[:, :, None])[:, :, 0]
        return y

    def diff(F, d, back):  # average over the two other axes of the difference along d
        e = [0, 0, 0]
        e[d] = -1 if back else 1
        g = F - _roll(F, n, e) if back else _roll(F, n, e) - F
        for a in range(3):
            if a != d:
                e = [0, 0, 0]
                e[a] = -1 if back else 1
                g = 0.5 * (g + _roll(g, n, e))
        return g

    def curl(F, back):
        d = [diff(F, a, back) for a in range(3)]
        return torch.stack([d[1][:, 2] - d[2][:, 1], d[2][:, 0] - d[0][:, 2], d[0][:, 1] - d[1][:, 0]], 1)

    b = cth * curl(Bm, True) - f * J - curl_mass(E)
    x, r = torch.zeros_like(b), b.clone()  # BiCGStab to the rounding of 64 bits
    r0, p = r.clone(), r.clone()
    rho, nb = (r0 * r).sum(), b.norm()
    for _ in range(300):
        v = p + curl_mass(p)
        al = rho / (r0 * v).sum()
        s = r - al * v
        t = s + curl_mass(s)
        om = (t * s).sum() / (t * t).sum()
        x = x + al * p + om * s
        r = s - om * t
        if r.norm() <= 1e-14 * nb:
            break
        rho, old = (r0 * r).sum(), rho
        p = r + (rho / old) * (al / om) * (p - om * v)
    Eh = E + x
    Bn = Bm - dt * curl(Eh, False)
    En = (Eh - (1.0 - THETA) * E) / THETA
    return En, Bn, Eh, float(((En * En).sum() + (Bn * Bn).sum()) / (8.0 * math.pi))


def _c2n(B, n):
    s = torch.zeros_like(B)
    for o in _OFF:
        s += _roll(B, n, [-k for k in o])
    return s / 8.0


def _tracks64(case, x, v, spec, f):
    q, m, _ = _species64(case)
    n3 = _n3(case)
    qm, rel = (q / m)[spec.long()], case["rel"]
    rem = torch.full((len(x),), float(case["dt"]), **_D)
    while bool((rem > 0).any()):
        E, B = _gather(x, f["E_n"], n3), _gather(x, f["B_corner_cur"], n3)
        dt = rem
        if rel:
            gam = 1.0 / (1.0 - (v * v).sum(1)).sqrt()
            dt = torch.minimum(rem, 2.0 * math.pi * gam / (qm.abs() * B.norm(dim=1)))
        h = (0.5 * qm * dt)[:, None]
        um = (v * gam[:, None] if rel else v) + h * E
        t = h * B / ((1.0 + (um * um).sum(1)).sqrt()[:, None] if rel else 1.0)
        up = um + torch.linalg.cross(um, t)
        uf = um + torch.linalg.cross(up, 2.0 * t / (1.0 + (t * t).sum(1))[:, None]) + h * E
        vn = uf / (1.0 + (uf * uf).sum(1)).sqrt()[:, None] if rel else uf
        go = (rem > 0)[:, None]
        v = torch.where(go, vn, v)
        x = torch.where(go, (x + vn * dt[:, None]) % n3.double(), x)
        rem = torch.where(rem > 0, rem - dt, rem)
    return torch.cat([x, v], 1)


def _net64(case, seed):
    x, e = _samples(case, seed)
    ws = [torch.tensor(w, **_D).requires_grad_(True) for w in _weights(seed)]
    total = torch.zeros((), **_D)
    for s in range(0, len(x), 32):
        xx, ee = x[s:s + 32].double(), e[s:s + 32].double()
        a = xx.reshape(-1, 10, 10, 10, 3)
        for w in ws:
            pad = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
            a = sum(pad[:, t // 9:t // 9 + 10, (t // 3) % 3:(t // 3) % 3 + 10, t % 3:t % 3 + 10] @ w[t]
                    for t in range(27))
        z = (a + xx.reshape(a.shape[:4] + (3,)))[:, 1:9, 1:9, 1:9].reshape(-1, 512, 3)
        loss = ((z - ee) ** 2).sum() / (len(x) * 512 * 3)
        loss.backward()
        total += loss.detach()
    return {"loss": total, "g": [w.grad for w in ws]}


def _trace64(case, seed):
    x0, p0 = _starts(case, seed)
    x, p = torch.tensor(x0 / R_E, **_D), torch.tensor(p0 / (M_P * C_LIGHT), **_D)
    kq, ext = Q_P * B_EQ * R_E / (M_P * C_LIGHT), torch.tensor([0.0, 0.0, -B_SOUTH / B_EQ], **_D)
    live = torch.ones(len(x), dtype=torch.bool, device="cuda")
    ez = torch.tensor([0.0, 0.0, 1.0], **_D)
    for _ in range(case["max_steps"]):
        r = x.norm(dim=1, keepdim=True)
        B = 3.0 * x * x[:, 2:] / r ** 5 - ez / r ** 3 + ext
        g = (1.0 + (p * p).sum(1, keepdim=True)).sqrt()
        dt = torch.clamp(DPHI * g / (kq * B.norm(dim=1, keepdim=True)), max=DT_MAX * C_LIGHT / R_E)
        xn = x + 0.5 * dt * p / g
        t = 0.5 * kq * dt / g * B
        pn = p + torch.linalg.cross(p + torch.linalg.cross(p, t), 2.0 * t / (1.0 + (t * t).sum(1, keepdim=True)))
        xn = xn + 0.5 * dt * pn / (1.0 + (pn * pn).sum(1, keepdim=True)).sqrt()
        x, p = torch.where(live[:, None], xn, x), torch.where(live[:, None], pn, p)
        rr = (x * x).sum(1)
        live = live & (rr >= 1.0) & (rr <= 100.0)
        if not bool(live.any()):
            break
    return {"x": x * R_E, "p": p * (M_P * C_LIGHT), "status": None, "steps": None, "total": None}


def exact(case, seed):
    kind = case["kind"]
    if case.get("lmax"):
        return None  # the refined meshes' operator has no short form
    if kind == "net":
        return _net64(case, seed)
    if kind == "trace":
        # near the cutoff FP32 trajectories part from any other arithmetic's exponentially
        return None if case["precision"] else _trace64(case, seed)
    n = [8 * case[k] for k in ("nbx", "nby", "nbz")]
    u, v, spec, block, _ = _plasma(case, seed)
    x, v = _positions(case, u, block), v.double()
    if kind == "tracks":
        return _tracks64(case, x, v, spec, _wave_fields(case, seed))
    if kind == "push":
        f, c = _wave_fields(case, seed), case["centre"]
        B = f["B_center"] if c else f["B_corner_cur"]
        x, v = _push64(case, x, v, spec, f["E_half"], B, c)
        J, _, en = _deposit64(case, x, v, spec, B, c, mass=False)
        return {"energy": en, "J": J}
    if kind == "deposit":
        J, M, en = _deposit64(case, x, v, spec, _wave_fields(case, seed)["B_corner_cur"])
        return {"J": J, "M": M, "energy": torch.tensor([en], **_D)}
    ncell = n[0] * n[1] * n[2]
    if kind == "solve":
        f = _noise_fields(case, seed, ncell, ncell)
    else:
        z, b = torch.zeros(ncell, 3, **_D), torch.tensor([0.0, 0.0, B0], **_D).repeat(ncell, 1)
        f = {"E_n": z, "B_center": b, "B_corner_prev": b, "B_corner_cur": b}
    J, M, _ = _deposit64(case, x, v, spec, f["B_corner_cur"])
    En, Bn, Eh, wave = _solve64(case, f["E_n"], f["B_center"], J, M)
    if kind == "solve":
        return {"energy": wave, "E_n": En, "B_center": Bn}
    x, v = _push64(case, x, v, spec, Eh, f["B_corner_cur"], False)
    J, _, kin = _deposit64(case, x, v, spec, _c2n(Bn, n), mass=False)
    return {"energy": torch.tensor([kin, wave], **_D), "E_n": En, "B_center": Bn, "J": J}
