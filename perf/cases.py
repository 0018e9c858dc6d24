"""What this framework is timed on: the calls a PeriX user makes, from a 64x64 Poisson system to the 44-million-bond slab.

A case is a dict of plain values with a "kind"; the kinds are the framework's paths:

  scalar    Poisson / diffusion Jacobian values on a mesh that is set up once (every Newton iteration calls it)
  dynfrac   implicit dynamic fracture Jacobian values (dim unknowns a node, frozen bond health)
  stress    stress-coupled Cahn-Hilliard Jacobian values (dim + 2 unknowns a node: battery particles)
  chrun     an implicit Cahn-Hilliard run on the device: assembly, BiCGStab and Newton per step
  setup     a new mesh: families, operators, matrix pattern and the first system
  run       the explicit fracture loop between two output times, from a saved state, state read back
  rate      one per-step call of the explicit element with host buffers (what the reference's interface asks for)
  clouds    operators of many 2D and 3D point clouds in one batch and all derivatives of a field on them
  field     all derivatives of a field through torch, forward and backward
  inverse   the explicit loop and its adjoint through torch (an inverse problem's gradient)

Meshes are lattices with one mirrored ghost layer a face, as PeriX's decks use them, or jittered clouds; the horizon
is 3.015 spacings.  ``exact`` restates the mathematics in plain torch, 64 bits, with none of this package's code.
"""
import ctypes as C
import math

import numpy as np
import torch

import perix_b200 as px
from perix_b200.autograd import explicit_run, pddo_apply

DEV = "cuda"
HORIZON = 3.015
PRECISION = {"fp64": px.FP64, "mixed": px.MIXED}


# ------------------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest system in use, one Newton iteration's values: launches and latency count
        dict(name="poisson_64", kind="scalar", dim=2, nx=64, ny=64, nz=1, precision="fp64", transient=False),
        # implicit fracture on the 400x200 plate
        dict(name="dynfrac_plate", kind="dynfrac", dim=2, nx=400, ny=200, nz=1),
        # a 3D battery particle with fracturing bonds, five unknowns a node
        dict(name="stress_ch_3d", kind="stress", dim=3, nx=32, ny=32, nz=32, fracture=True),
        # spinodal decomposition, 256x256, ten backward-Euler steps as one call
        dict(name="ch_run_256", kind="chrun", nx=256, ny=256, steps=10),
        # a new 3D mesh up to its first Poisson system
        dict(name="setup_3d", kind="setup", dim=3, nx=40, ny=40, nz=40),
        # the notched plate between outputs; its streams stay in L2
        dict(name="plate_run_mixed", kind="run", dim=2, nx=400, ny=200, nz=1, precision="mixed", steps=50,
             tension_only=True),
        # the notched slab between outputs, both precisions: the largest explicit runs
        dict(name="slab_run_fp64", kind="run", dim=3, nx=120, ny=120, nz=24, precision="fp64", steps=20,
             tension_only=True),
        dict(name="slab_run_mixed", kind="run", dim=3, nx=120, ny=120, nz=24, precision="mixed", steps=20,
             tension_only=True),
        # the reference interface: displacement in, acceleration out, every step
        dict(name="plate_rate", kind="rate", dim=2, nx=400, ny=200, nz=1, precision="fp64"),
        # 32 clouds, 2D and 3D, log-uniform sizes
        dict(name="clouds_fp64", kind="clouds", count=32, smallest=1000, largest=50000, precision="fp64", layout=1),
        # derivatives of a field on a 3D mesh inside a torch program
        dict(name="field_3d", kind="field", dim=3, nx=48, ny=48, nz=48, precision="fp64"),
        # the gradient of an explicit run, every state kept
        dict(name="inverse_slab", kind="inverse", dim=3, nx=60, ny=60, nz=24, precision="fp64", steps=20, keep=0),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _grid(rng, dim, lo2, hi2, lo3, hi3):
    if dim == 2:
        return dict(dim=2, nx=_log_int(rng, lo2, hi2), ny=_log_int(rng, lo2, hi2), nz=1)
    return dict(dim=3, nx=_log_int(rng, lo3, hi3), ny=_log_int(rng, lo3, hi3), nz=_log_int(rng, lo3, hi3))


def draw(rng):
    kind = rng.choice(["scalar", "dynfrac", "stress", "chrun", "setup", "run", "run", "rate", "clouds", "field",
                       "inverse"])
    dim = rng.choice([2, 3])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "scalar":
        return dict(kind=kind, **_grid(rng, dim, 32, 512, 10, 56), precision=precision, transient=rng.random() < 0.5)
    if kind == "dynfrac":
        return dict(kind=kind, **_grid(rng, dim, 32, 400, 10, 40))
    if kind == "stress":
        return dict(kind=kind, **_grid(rng, dim, 32, 300, 10, 32), fracture=rng.random() < 0.5)
    if kind == "chrun":
        return dict(kind=kind, nx=_log_int(rng, 32, 256), ny=_log_int(rng, 32, 256), steps=rng.randint(2, 10))
    if kind == "setup":
        return dict(kind=kind, **_grid(rng, dim, 32, 300, 10, 40))
    if kind == "run":
        if dim == 2:
            return dict(kind=kind, dim=2, nx=_log_int(rng, 40, 400), ny=_log_int(rng, 30, 200), nz=1,
                        precision=precision, steps=rng.randint(5, 50), tension_only=rng.random() < 0.7)
        return dict(kind=kind, dim=3, nx=_log_int(rng, 20, 120), ny=_log_int(rng, 20, 120), nz=_log_int(rng, 6, 24),
                    precision=precision, steps=rng.randint(5, 20), tension_only=rng.random() < 0.7)
    if kind == "rate":
        if dim == 2:
            return dict(kind=kind, dim=2, nx=_log_int(rng, 40, 400), ny=_log_int(rng, 30, 200), nz=1,
                        precision=precision)
        return dict(kind=kind, dim=3, nx=_log_int(rng, 20, 120), ny=_log_int(rng, 20, 120), nz=_log_int(rng, 6, 24),
                    precision=precision)
    if kind == "clouds":
        return dict(kind=kind, count=rng.randint(2, 32), smallest=1000, largest=_log_int(rng, 4000, 50000),
                    precision=precision, layout=rng.randint(2, 1 << 20))
    if kind == "field":
        return dict(kind=kind, **_grid(rng, dim, 32, 400, 10, 48), precision=precision)
    return dict(kind="inverse", **_grid(rng, dim, 40, 300, 12, 44), precision="fp64", steps=rng.randint(5, 20),
                keep=rng.choice([0, 4]))


# ----------------------------------------------------------------------------------------------------------- meshes
def _spacing(case):
    """1 mm in mechanics, the unit interval along x elsewhere."""
    return 1.0e-3 if case["kind"] in ("run", "rate", "inverse", "dynfrac") else 1.0 / case["nx"]


def _lattice(case):
    """Cell centres, x fastest, then one mirrored ghost a face cell (left, right, bottom, top[, back, front])."""
    dim, m = case["dim"], (case["nx"], case["ny"], case["nz"])
    h = _spacing(case)
    idx = np.indices(m[::-1]).reshape(3, -1)[::-1].T[:, :3]  # (i, j, k) with i fastest
    bulk = idx.astype(np.int64)
    number = lambda q: q[:, 0] + m[0] * (q[:, 1] + m[1] * q[:, 2])  # noqa: E731
    sites, mirror, faces = [bulk], [np.zeros(len(bulk), np.int64)], []
    at = len(bulk)
    for d in range(dim):
        for side in (0, 1):
            b = bulk[bulk[:, d] == (0 if side == 0 else m[d] - 1)]
            g = b.copy()
            g[:, d] += -1 if side == 0 else 1
            sites.append(g)
            mirror.append(number(b) + 1)
            faces.append(np.arange(at, at + len(b)) + 1)
            at += len(b)
    q = np.concatenate(sites)
    x = (q + 0.5) * h
    if dim == 2:
        x[:, 2] = 0.0
    n = len(x)
    return dict(x=np.ascontiguousarray(x), n=n, dim=dim, h=h, vol=np.full(n, h ** dim), delta=HORIZON * h * (1 + 1e-6),
                mirror=np.concatenate(mirror).astype(np.int32), faces=faces, nbulk=len(bulk), m=m)


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _smooth(x, seed, count, slope):
    """`count` smooth fields at the nodes x (n, 3), sums of four waves, with slopes of about `slope`."""
    r = np.random.default_rng(int(seed))
    span = (x.max(dim=0).values - x.min(dim=0).values).clamp_min(1e-30)
    live = (span > 1e-20).double()
    out = []
    for _ in range(count):
        f = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
        for _ in range(4):
            k = torch.tensor(r.uniform(-3.0, 3.0, 3), device=x.device) * 2 * math.pi / span * live
            a = slope * r.uniform(0.3, 0.7) / max(float(k.norm()), 1e-30)
            f += a * torch.sin(x @ k + r.uniform(0, 2 * math.pi))
        out.append(f)
    return torch.stack(out, 1)


def _xyz(L):
    return torch.from_numpy(L["x"]).to(DEV)


def _broken(L, i, j, seed, notch):
    """Bonds that start broken: those across the edge notch (between bulk cells, ghosts through their mirrors) and about
    one in fifty of the rest, chosen symmetrically."""
    own = torch.from_numpy(np.where(L["mirror"] > 0, L["mirror"] - 1, np.arange(L["n"])).astype(np.int64)).to(DEV)
    a, b = own[i], own[j]
    m = L["m"]
    xa, ya, xb, yb = a % m[0], (a // m[0]) % m[1], b % m[0], (b // m[0]) % m[1]
    cut = m[1] // 2  # the notch lies between cell rows cut - 1 and cut
    cross = (ya < cut) != (yb < cut)
    s = torch.where(ya == yb, torch.zeros_like(ya).double(),
                    (cut - 0.5 - ya).double() / torch.where(ya == yb, torch.ones_like(ya), yb - ya).double())
    dead = cross & (xa + s * (xb - xa) < notch - 0.5)
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    lot = (lo * 73856093 + hi * 19349663 + seed * 83492791) % 1009
    return dead | ((lot < 20) & (a != b))


def _material(dim):
    E, nu, rho = (72e9, 0.22, 2440.0) if dim == 3 else (190e9, 0.3, 8000.0)
    d = (1 + nu) * (1 - 2 * nu)
    return (E * (1 - nu) / d, E * nu / d, E / (2 * (1 + nu))), rho, (0.004 if dim == 3 else 0.01)


def _boundary(L):
    """Ghosts copy their mirrors; then the two outermost y layers (bulk and ghosts) are pulled apart at +-2 m/s."""
    y = L["x"][:, 1]
    top = np.nonzero(y > (L["m"][1] - 3) * L["h"])[0] + 1
    bottom = np.nonzero(y < 3 * L["h"])[0] + 1
    return top.astype(np.int32), bottom.astype(np.int32)


def _dt(L, Cs, rho):
    return 0.8 * L["h"] / math.sqrt(Cs[0] / rho)


# ---------------------------------------------------------------------------------------------------------- prepare
def _context(L, precision=None, order=2):
    ctx = px.Context(0)
    ctx.set_geometry_points(L["x"], L["vol"], L["delta"], L["delta"], L["h"], L["dim"], mirror=L["mirror"])
    if precision is not None:
        ctx.gbuild(order, PRECISION[precision])
    return ctx


def _on_torch(ctx):
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)


def _bonds_of(ctx):
    off, ids = ctx.get_families()
    off = torch.from_numpy(off.astype(np.int64)).to(DEV)
    i = torch.repeat_interleave(torch.arange(off.numel() - 1, device=DEV), off.diff())
    return i, torch.from_numpy(ids).to(DEV).long() - 1


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _zeros(n):
    return torch.zeros(int(n), dtype=torch.float64, device=DEV)


def _explicit(case, seed, sc_on=True):
    """A context with the explicit element, its boundary conditions and a seeded displacement near breaking."""
    L = _lattice(case)
    Cs, rho, sc = _material(L["dim"])
    ctx = _context(L)
    i, j = _bonds_of(ctx)
    health = (~_broken(L, i, j, seed, L["m"][0] // 6)).to(torch.uint8).cpu().numpy()
    ctx.epf_setup(*Cs, rho, (0.0, 0.0, 0.0), sc if sc_on else 0.0, case.get("tension_only", True), health0=health,
                  precision=PRECISION[case["precision"]])
    comps = list(range(L["dim"]))
    top, bottom = _boundary(L)
    ctx.epf_set_bcs([px.BC("neumann", comps, f) for f in L["faces"]] +
                    [px.BC("dirichlet", [1], top, velocity=[0, 2.0, 0], direct=True),
                     px.BC("dirichlet", [1], bottom, velocity=[0, -2.0, 0], direct=True)])
    u0 = _smooth(_xyz(L), seed, L["dim"], 0.7 * sc).reshape(-1)
    return L, ctx, Cs, rho, sc, u0


def _cloud_list(case, seed):
    """The clouds' sizes are the case's own (`layout`), their jitter and field the seed's."""
    sizes = np.random.default_rng(case["layout"])
    r = np.random.default_rng(seed)
    clouds = []
    for k in range(case["count"]):
        dim = 2 + k % 2
        n = math.exp(sizes.uniform(math.log(case["smallest"]), math.log(case["largest"])))
        m = max(6, int(round(n ** (1.0 / dim))))
        h = 1.0 / m
        q = np.indices((m,) * dim).reshape(dim, -1)[::-1].T
        x = np.zeros((len(q), 3))
        x[:, :dim] = (q + 0.5) * h + r.uniform(-0.2 * h, 0.2 * h, q.shape)
        clouds.append(dict(dim=dim, coords3=x, vols=np.full(len(x), h ** dim), delta=HORIZON * h, dx_char=h))
    return clouds


def _cloud_fields(clouds, seed):
    return [_smooth(torch.from_numpy(c["coords3"]).to(DEV), seed * 1000 + k, 1, 1.0)[:, 0]
            for k, c in enumerate(clouds)]


def _stress_inputs(L, seed):
    """State (c, mu, u), previous state, mobility, velocity of the stress-coupled element."""
    n, dim = L["n"], L["dim"]
    g = _generator(seed)
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64, device=DEV)  # noqa: E731
    u = torch.empty(n, dim + 2, dtype=torch.float64, device=DEV)
    u[:, 0] = 0.5 + 0.2 * (rnd(n) - 0.5)
    u[:, 1] = 0.1 * (rnd(n) - 0.5)
    u[:, 2:] = _smooth(_xyz(L), seed, dim, 1e-3)
    uold = u.clone()
    uold[:, 0] += 0.01 * (rnd(n) - 0.5)
    return u, uold, u[:, 0] * (1 - u[:, 0]), 1e-3 * (rnd(n, dim) - 0.5)


def _stress_params(fracture):
    return dict(C11=1.35, C12=0.58, C66=0.385, A=0.3, Kh=0.9, Ch=-0.25, Omega=0.06, cref=0.5, chi=2.5, kappa=1e-4,
                dt=1e-4, kres=1e-6, rho=1e-6 if fracture else 0.0)


CH = dict(chi=2.5, kappa=1e-4, M0=1.0, dt=1e-6)


def _dynfrac_inputs(L, seed):
    Cs, rho, sc = _material(L["dim"])
    g = _generator(seed)
    u = _smooth(_xyz(L), seed, L["dim"], 0.5 * sc)
    du = 1e-2 * sc * L["h"] * (torch.rand(u.shape, generator=g, dtype=torch.float64, device=DEV) - 0.5)
    vel = torch.rand(u.shape, generator=g, dtype=torch.float64, device=DEV) - 0.5
    return Cs, rho, 20 * _dt(L, Cs, rho), u, u - du, vel


class _CachedParams(C.Structure):
    _fields_ = [("C11", C.c_double), ("C12", C.c_double), ("C66", C.c_double), ("rho", C.c_double),
                ("dt", C.c_double), ("b", C.c_double * 3)]


def _ok(ctx, status):
    if status:
        raise px.PxbError(status, ctx.L.pxb_last_error().decode(errors="replace"))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind in ("scalar", "setup"):
        L = _lattice(case)
        u = _smooth(_xyz(L), seed, 1, 1.0)[:, 0].contiguous()
        s.update(u=u, uold=(u * 0.99).contiguous(), f=_smooth(_xyz(L), seed + 1, 1, 10.0)[:, 0].contiguous())
        if kind == "setup":
            ctx = px.Context(0)
            _on_torch(ctx)
            s.update(ctx=ctx, L=L, rhs=_zeros(L["n"]))
            return s
        ctx = _context(L, case["precision"])
        _on_torch(ctx)
        nnz = ctx.csr_build_pattern(1)
        s.update(ctx=ctx, kvals=_zeros(nnz), rhs=_zeros(L["n"]))
        t = case["transient"]
        s["args"] = (ctx.h, 1 if t else 0, C.c_double(0.7), C.c_double(0.0), _ptr(s["f"]),
                     C.c_double(1e-3 if t else 0.0), _ptr(u), _ptr(s["uold"]) if t else None, _ptr(s["kvals"]),
                     _ptr(s["rhs"]))
    elif kind == "dynfrac":
        L = _lattice(case)
        Cs, rho, dt, u, uold, vel = _dynfrac_inputs(L, seed)
        ctx = _context(L, "fp64")
        _on_torch(ctx)
        i, j = _bonds_of(ctx)
        nnz = ctx.csr_build_pattern(L["dim"])
        s.update(ctx=ctx, u=u.contiguous(), uold=uold.contiguous(), vel=vel.contiguous(),
                 health=(~_broken(L, i, j, seed, L["m"][0] // 6)).double(), kvals=_zeros(nnz),
                 rhs=_zeros(L["n"] * L["dim"]),
                 prm=_CachedParams(*Cs, rho, dt, (C.c_double * 3)(0.0, -9.81 * rho, 0.0)))
        s["args"] = (ctx.h, C.byref(s["prm"]), _ptr(s["vel"]), L["dim"], _ptr(s["health"]), 1, _ptr(s["u"]),
                     _ptr(s["uold"]), _ptr(s["kvals"]), _ptr(s["rhs"]))
    elif kind == "stress":
        L = _lattice(case)
        u, uold, mob, vel = _stress_inputs(L, seed)
        ctx = _context(L, "fp64")
        _on_torch(ctx)
        ctx.ch_build_geometry()
        nnz = ctx.csr_build_pattern(L["dim"] + 2)
        s.update(ctx=ctx, u=u, uold=uold, mob=mob.contiguous(), vel=vel, prm=_stress_params(case["fracture"]),
                 kvals=_zeros(nnz), rhs=_zeros(u.numel()), health=None)
        if case["fracture"]:
            i, j = _bonds_of(ctx)
            s["health"] = (~_broken(L, i, j, seed, L["m"][0] // 6)).double()
    elif kind == "chrun":
        L = _lattice(dict(case, dim=2, nz=1))
        ctx = _context(L, "fp64")
        ctx.ch_build_geometry()
        ctx.csr_build_pattern(2)
        c0 = 0.5 + np.random.default_rng(seed).uniform(-0.01, 0.01, L["n"])
        s.update(ctx=ctx, c0=c0, steps=case["steps"])
    elif kind == "run":
        L, ctx, Cs, rho, sc, u0 = _explicit(case, seed)
        ctx.epf_start(u0.cpu().numpy(), None, _dt(L, Cs, rho))
        ctx.epf_autotune(steps=8, use_cache=True)
        _ok(ctx, ctx.L.pxb_epf_snapshot(ctx.h))
        pin = lambda k, t: torch.zeros(int(k), dtype=t, pin_memory=True)  # noqa: E731
        s.update(ctx=ctx, steps=case["steps"], u=pin(u0.numel(), torch.float64), up=pin(u0.numel(), torch.float64),
                 health=pin(ctx.nb, torch.uint8), t=C.c_double(0.0))
    elif kind == "rate":
        L, ctx, Cs, rho, sc, u0 = _explicit(case, seed)
        u = torch.empty(u0.numel(), dtype=torch.float64, pin_memory=True)
        u.copy_(u0)
        torch.cuda.synchronize()
        _ok(ctx, ctx.L.pxb_epf_autotune_rate(ctx.h, _ptr(u), 5, 1, None, None))
        s.update(ctx=ctx, u=u, a=torch.zeros(u0.numel(), dtype=torch.float64, pin_memory=True), broken=C.c_longlong(0))
        s["args"] = (ctx.h, _ptr(s["u"]), _ptr(s["a"]), C.byref(s["broken"]))
    elif kind == "clouds":
        clouds = _cloud_list(case, seed)
        u = torch.cat(_cloud_fields(clouds, seed))
        ctx = px.Context(0)
        ctx.batch_set_points(clouds)
        _on_torch(ctx)
        out = _zeros(ctx.batch_out_len)
        p = PRECISION[case["precision"]]
        ctx.batch_gbuild(p)
        ctx.batch_autotune(0, reps=2)
        ctx.batch_autotune(1, reps=2, u_ptr=u.data_ptr(), out_ptr=out.data_ptr())
        s.update(ctx=ctx, u=u, out=out, precision=p)
    elif kind == "field":
        L = _lattice(case)
        ctx = _context(L, case["precision"])
        nop = 5 if L["dim"] == 2 else 9
        u = _smooth(_xyz(L), seed, 1, 1.0)[:, 0].contiguous().requires_grad_(True)
        w = torch.randn(L["n"], nop, generator=_generator(seed), dtype=torch.float64, device=DEV)
        s.update(ctx=ctx, u=u, w=w, slots=list(range(nop)))
    else:
        L, ctx, Cs, rho, sc, u0 = _explicit(case, seed, sc_on=False)
        ctx.epf_start(u0.cpu().numpy(), None, _dt(L, Cs, rho))
        ctx.epf_autotune(steps=8, use_cache=True)
        s.update(ctx=ctx, u0=u0.requires_grad_(True), dt=_dt(L, Cs, rho), steps=case["steps"], keep=case["keep"],
                 C=torch.tensor(Cs, dtype=torch.float64, device=DEV, requires_grad=True),
                 w=torch.randn(u0.numel(), generator=_generator(seed), dtype=torch.float64, device=DEV))
    return s


# -------------------------------------------------------------------------------------------------------------- run
def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "scalar":
        _ok(ctx, ctx.L.pxb_assemble_scalar_d(*s["args"]))
        return [s["kvals"], s["rhs"]]
    if kind == "dynfrac":
        _ok(ctx, ctx.L.pxb_assemble_cached_d(*s["args"]))
        return [s["kvals"], s["rhs"]]
    if kind == "stress":
        h = s["health"]
        ctx.assemble_stress_ch_d(s["prm"], s["mob"].data_ptr(), s["u"].data_ptr(), s["uold"].data_ptr(),
                                 s["kvals"].data_ptr(), s["rhs"].data_ptr(),
                                 health_ptr=None if h is None else h.data_ptr(), vel_ptr=s["vel"].data_ptr())
        return [s["kvals"], s["rhs"]]
    if kind == "chrun":
        u, E, _ = ctx.ch_run(s["c0"], CH["chi"], CH["kappa"], CH["M0"], CH["dt"], s["steps"])
        return [u, E]
    if kind == "setup":
        L = s["L"]
        ctx.set_geometry_points(L["x"], L["vol"], L["delta"], L["delta"], L["h"], L["dim"], mirror=L["mirror"])
        ctx.gbuild(2, px.FP64)
        kvals = torch.empty(ctx.csr_build_pattern(1), dtype=torch.float64, device=DEV)
        _ok(ctx, ctx.L.pxb_assemble_scalar_d(ctx.h, 0, C.c_double(0.7), C.c_double(0.0), _ptr(s["f"]),
                                             C.c_double(0.0), _ptr(s["u"]), None, _ptr(kvals), _ptr(s["rhs"])))
        return [kvals, s["rhs"]]
    if kind == "run":
        _ok(ctx, ctx.L.pxb_epf_restore(ctx.h))
        ctx.epf_advance(s["steps"])
        _ok(ctx, ctx.L.pxb_epf_get_state(ctx.h, _ptr(s["u"]), _ptr(s["up"]), _ptr(s["health"]), C.byref(s["t"])))
        return [s["u"], s["up"], s["health"]]
    if kind == "rate":
        _ok(ctx, ctx.L.pxb_epf_rate(*s["args"]))
        return s["a"]
    if kind == "clouds":
        ctx.batch_gbuild(s["precision"])
        ctx.batch_apply_d(s["u"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    if kind == "field":
        d = pddo_apply(ctx, s["u"], s["slots"])
        return [d.detach(), torch.autograd.grad(d, s["u"], s["w"])[0]]
    uN, _ = explicit_run(ctx, s["u0"], None, s["C"], s["dt"], s["steps"], checkpoint_every=s["keep"])
    g = torch.autograd.grad(uN, [s["u0"], s["C"]], s["w"])
    return [uN.detach(), g[0], g[1]]


# ------------------------------------------------------------------------------------------------------------- work
def _bond_count(case):
    """Directed bonds of the lattice with its ghosts: occupied sites a horizon apart."""
    dim, m = case["dim"], (case["nx"], case["ny"], case["nz"])
    occ = np.zeros(tuple(k + 2 for k in m), bool)
    occ[1:-1, 1:-1, 1:-1] = True
    occ[[0, -1], 1:-1, 1:-1] = True
    occ[1:-1, [0, -1], 1:-1] = True
    if dim == 3:
        occ[1:-1, 1:-1, [0, -1]] = True
    r = range(-3, 4)
    nb = 0
    for a in r:
        for b in r:
            for c in (r if dim == 3 else (0,)):
                if 0 < a * a + b * b + c * c <= 9 and all(abs(o) < e for o, e in zip((a, b, c), occ.shape)):
                    here = tuple(slice(max(0, -o), e - max(0, o)) for o, e in zip((a, b, c), occ.shape))
                    there = tuple(slice(max(0, o), e - max(0, -o)) for o, e in zip((a, b, c), occ.shape))
                    nb += int(np.count_nonzero(occ[here] & occ[there]))
    return int(np.count_nonzero(occ)), nb


def work(case):
    kind = case["kind"]
    if kind == "clouds":
        sizes = np.random.default_rng(case["layout"])
        B = F = 0.0
        for k in range(case["count"]):
            dim = 2 + k % 2
            n = math.exp(sizes.uniform(math.log(case["smallest"]), math.log(case["largest"])))
            n, nop, fam = max(6, int(round(n ** (1.0 / dim)))) ** dim, (5, 9)[dim - 2], (27, 100)[dim - 2]
            e = 8 if case["precision"] == "fp64" else 4
            B += n * (fam * (2 * 4 + 2 * nop * e) + 8 * dim + 8 + 8 + 8 * nop)
            F += n * (fam * (2.0 * nop * nop * 2 + 4 * nop) + nop ** 3)
        return dict(bytes=B, flops=F)
    c = dict(case, dim=case.get("dim", 2), nz=case.get("nz", 1))
    n, nb = _bond_count(c)
    dim, e = c["dim"], 4 if case.get("precision") == "mixed" else 8
    nc, nop = (6, 9) if dim == 3 else (3, 5)
    if kind == "scalar":
        return dict(bytes=nb * (4 + dim * e + 8 + 4) + n * (8 * 5), flops=nb * 6)
    if kind == "dynfrac":
        return dict(bytes=nb * (4 + 8 * nc + 8 + 8 * dim * dim + 4) + n * 8 * (5 * dim + dim * dim),
                    flops=nb * (4 * nc + 4 * dim * dim))
    if kind == "stress":
        nd = dim + 2
        return dict(bytes=nb * (4 + 8 * nop + 8 + 4 + 8 + 8 * nd * nd + 4) + n * 8 * (3 * nd + nd * nd + dim + 2),
                    flops=nb * (6 * nd * nd))
    if kind == "chrun":  # three Newton iterations a step, ten BiCGStab iterations each: two products over the bonds
        its = case["steps"] * 3 * 10
        return dict(bytes=its * 2 * (nb * (4 + 16) + n * 2 * 8 * 5) + case["steps"] * 3 * nb * 60, flops=its * 2 * nb * 8)
    if kind == "setup":
        return dict(bytes=n * (8 * 4 + 8) + nb * (4 * 4 + 8 * nop * 2 + 8) + n * 40,
                    flops=nb * (4.0 * nop * nop + 4 * nop) + n * nop ** 3)
    if kind == "run":
        return dict(bytes=case["steps"] * (nb * (4 + nc * e + 1) + n * 4 * dim * 8) + nb + n * dim * 16,
                    flops=case["steps"] * nb * (24 if dim == 2 else 40))
    if kind == "rate":
        return dict(bytes=nb * (4 + nc * e + 1) + n * dim * 8 * 3, flops=nb * (24 if dim == 2 else 40))
    if kind == "field":
        return dict(bytes=2 * (nb * (4 + nop * e) + n * (8 + 8 * nop)), flops=4 * nb * nop)
    # inverse: per step one pass over the operators forward and one backward
    return dict(bytes=case["steps"] * 2 * (nb * (4 + nc * e + 1) + n * 5 * dim * 8),
                flops=case["steps"] * nb * (24 if dim == 2 else 40) * 2.5)


# ------------------------------------------------------------------------------------- the same in plain torch, 64 bits
def _pairs(x, radius, dim):
    """All directed pairs within the radius, sorted by (i, j)."""
    lo = x.min(dim=0).values
    cell = ((x - lo) / radius).floor().long()
    if dim == 2:
        cell[:, 2] = 0
    size = cell.max(dim=0).values + 1
    number = (cell[:, 2] * size[1] + cell[:, 1]) * size[0] + cell[:, 0]
    order = torch.argsort(number)
    count = torch.bincount(number, minlength=int(size.prod()))
    start = count.cumsum(0) - count
    out = []
    node = torch.arange(len(x), device=x.device)
    for dz in ((-1, 0, 1) if dim == 3 else (0,)):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                q = cell + torch.tensor([dx, dy, dz], device=x.device)
                inside = ((q >= 0) & (q < size)).all(1)
                a = node[inside]
                k = ((q[:, 2] * size[1] + q[:, 1]) * size[0] + q[:, 0])[inside]
                c = count[k]
                i = torch.repeat_interleave(a, c)
                within = torch.arange(i.numel(), device=x.device) - torch.repeat_interleave(c.cumsum(0) - c, c)
                j = order[torch.repeat_interleave(start[k], c) + within]
                near = ((x[i] - x[j]).square().sum(1) <= radius * radius * (1 + 1e-14)) & (i != j)
                out.append(i[near] * len(x) + j[near])
    key = torch.cat(out).sort().values
    return key // len(x), key % len(x)


def _index(dim):
    if dim == 2:
        return [(1, 0, 0), (0, 1, 0), (2, 0, 0), (1, 1, 0), (0, 2, 0)]
    return [(1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (1, 1, 0), (1, 0, 1), (0, 2, 0), (0, 1, 1), (0, 0, 2)]


def _operators(x, vol, i, j, delta, dxc, dim):
    """Order-2 PDDO g-functions of every bond (Madenci's moment systems with the Gaussian weight and the rim volumes)."""
    pqr = _index(dim)
    n, k = len(x), len(pqr)
    fact = torch.tensor([math.prod(math.factorial(v) for v in t) for t in pqr], dtype=torch.float64, device=x.device)
    deg = torch.tensor([sum(t) for t in pqr], dtype=torch.float64, device=x.device)
    fam = torch.bincount(i, minlength=n)
    first = fam.cumsum(0) - fam
    g = torch.empty(len(i), k, dtype=torch.float64, device=x.device)
    width = int(fam.max())
    step = max(1, 40_000_000 // (width * k))
    for a in range(0, n, step):
        b = min(n, a + step)
        t0, t1 = int(first[a]), int(first[b - 1] + fam[b - 1])
        ii, jj = i[t0:t1], j[t0:t1]
        xi = x[jj] - x[ii]
        r = xi.norm(dim=1)
        rim = torch.where(r > delta - 0.5 * dxc, ((delta - r + 0.5 * dxc) / dxc).clamp(0, 1), torch.ones_like(r))
        w = torch.exp(-(2 * r / delta).square()) * rim * vol[jj]
        e = xi / delta
        M = torch.stack([e[:, 0] ** p * e[:, 1] ** q * e[:, 2] ** s for p, q, s in pqr], 1)
        pad = torch.zeros(b - a, width, k, dtype=torch.float64, device=x.device)
        wpad = torch.zeros_like(pad)
        at = torch.arange(t0, t1, device=x.device) - first[ii]
        pad[ii - a, at] = M
        wpad[ii - a, at] = M * w[:, None]
        X = torch.linalg.solve(wpad.transpose(1, 2) @ pad, torch.diag(fact).expand(b - a, k, k))
        g[t0:t1] = ((pad @ X)[ii - a, at]) * w[:, None] / delta ** deg
    return g


def _plain_mesh(case):
    L = _lattice(case)
    x, vol = _xyz(L), torch.from_numpy(L["vol"]).to(DEV)
    i, j = _pairs(x, L["delta"], L["dim"])
    return L, x, vol, i, j, _operators(x, vol, i, j, L["delta"], L["h"], L["dim"])


def _sum(n, i, v):
    return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add_(0, i, v)


def _csr_values(n, i, j, blocks, diag):
    """Block values in a CSR with sorted columns, rows of a node one after another."""
    nd = diag.shape[1]
    key = torch.cat([i * n + j, torch.arange(n, device=DEV) * (n + 1)])
    order = key.argsort()
    row = key[order] // n
    m = torch.bincount(row, minlength=n)
    first = m.cumsum(0) - m
    k = torch.arange(len(order), device=DEV) - first[row]
    a = torch.arange(nd, device=DEV)
    at = (nd * nd * first[row] + k * nd)[:, None, None] + (a[:, None] * (m[row] * nd)[:, None, None]) + a
    out = torch.empty(len(order) * nd * nd, dtype=torch.float64, device=DEV)
    out[at.reshape(-1)] = torch.cat([blocks, diag])[order].reshape(-1)
    return out


def _navier(g, dim, Cs):
    """Symmetric Navier block of every bond (nb, dim, dim)."""
    C11, C12, C66 = Cs
    s = {t: k for k, t in enumerate(_index(dim))}
    unit = torch.eye(3, dtype=torch.int64).tolist()
    second = lambda a, b: g[:, s[tuple(u + v for u, v in zip(unit[a], unit[b]))]]  # noqa: E731
    K = torch.empty(len(g), dim, dim, dtype=torch.float64, device=g.device)
    trace = sum(second(a, a) for a in range(dim))
    for a in range(dim):
        for b in range(dim):
            K[:, a, b] = C11 * second(a, a) + C66 * (trace - second(a, a)) if a == b else (C12 + C66) * second(a, b)
    return K


def _laplacian(g, dim):
    s = {t: k for k, t in enumerate(_index(dim))}
    out = g[:, s[(2, 0, 0)]] + g[:, s[(0, 2, 0)]]
    return out + g[:, s[(0, 0, 2)]] if dim == 3 else out


def _ch_laplacian(L, x, i, j, g):
    """The lambda-corrected Laplacian of the Cahn-Hilliard elements, its reverse bonds' values, the ghosts."""
    dim, n = L["dim"], L["n"]
    ghost = torch.from_numpy(L["mirror"] > 0).to(DEV)
    lap = _laplacian(g, dim)
    q = x.square().sum(1)
    lapq = _sum(n, i, torch.where(ghost[j], torch.zeros_like(lap), lap * (q[j] - q[i])))
    lam = torch.where(lapq > 1e-12, 2.0 * dim / lapq, torch.ones_like(lapq))
    lap = torch.where(ghost[j], lap, lap * lam[i])
    back = torch.searchsorted(i * n + j, j * n + i)
    return lap, lap[back], ghost


def _exact_scalar(case, seed):
    L, x, vol, i, j, g = _plain_mesh(case)
    n = L["n"]
    u = _smooth(x, seed, 1, 1.0)[:, 0]
    f = _smooth(x, seed + 1, 1, 10.0)[:, 0]
    t = case.get("transient", False)
    c = (-0.7 if t else 0.7) * _laplacian(g, L["dim"])
    rhs = _sum(n, i, c * (u[j] - u[i])) + ((u - 0.99 * u) / 1e-3 - f if t else f)
    diag = _sum(n, i, c) - (1e3 if t else 0.0)
    return [_csr_values(n, i, j, -c[:, None, None], diag[:, None, None]), rhs]


def _exact_dynfrac(case, seed):
    L, x, vol, i, j, g = _plain_mesh(case)
    n, dim = L["n"], L["dim"]
    Cs, rho, dt, u, uold, vel = _dynfrac_inputs(L, seed)
    K = _navier(g, dim, Cs) * (~_broken(L, i, j, seed, L["m"][0] // 6)).double()[:, None, None]
    b = torch.tensor([0.0, -9.81 * rho, 0.0][:dim], dtype=torch.float64, device=DEV)
    c0 = rho / (dt * dt)
    rhs = b - c0 * (u - uold - vel * dt) + _sum(n, i, torch.einsum("tab,tb->ta", K, u[j] - u[i]))
    diag = _sum(n, i, K) + c0 * torch.eye(dim, dtype=torch.float64, device=DEV)
    return [_csr_values(n, i, j, -K, diag), rhs.reshape(-1)]


def _exact_stress(case, seed):
    L, x, vol, i, j, g = _plain_mesh(case)
    n, dim = L["n"], L["dim"]
    nd = dim + 2
    u, uold, mob, vel = _stress_inputs(L, seed)
    p = _stress_params(case["fracture"])
    lap, back, ghost = _ch_laplacian(L, x, i, j, g)
    gate = torch.ones(len(i), dtype=torch.float64, device=DEV)
    if case["fracture"]:
        gate = torch.where(_broken(L, i, j, seed, L["m"][0] // 6), torch.full_like(gate, p["kres"]), gate)
    G = g * gate[:, None]
    zero = torch.zeros_like(lap)
    K = torch.zeros(len(i), nd, nd, dtype=torch.float64, device=DEV)
    K[:, 0, 1] = torch.where(ghost[j], zero, -0.5 * (mob[i] * lap + vol[j] / vol[i] * mob[j] * back))
    K[:, 1, 0] = torch.where(ghost[j], zero, p["kappa"] * lap)
    for d in range(dim):
        K[:, 1, 2 + d] = p["Omega"] * p["Kh"] * G[:, d]
        K[:, 2 + d, 0] = -p["A"] * G[:, d]
    K[:, 2:, 2:] = _navier(G, dim, (p["C11"], p["C12"], p["C66"]))
    c, mu = u[:, 0], u[:, 1]
    r = torch.zeros(n, nd, dtype=torch.float64, device=DEV)
    kii = torch.zeros(n, nd, nd, dtype=torch.float64, device=DEV)
    r[:, 0] = (c - uold[:, 0]) / p["dt"]
    r[:, 1] = mu - torch.log(c / (1 - c)) - p["chi"] * (1 - 2 * c) + p["Omega"] * p["Ch"] * (c - p["cref"])
    kii[:, 0, 0] = -1 / p["dt"]
    kii[:, 1, 0] = 1 / (c * (1 - c)) - 2 * p["chi"] - p["Omega"] * p["Ch"]
    kii[:, 1, 1] = -1.0
    if p["rho"] > 0:
        c0 = p["rho"] / p["dt"] ** 2
        r[:, 2:] -= c0 * (u[:, 2:] - uold[:, 2:] - vel * p["dt"])
        for d in range(dim):
            kii[:, 2 + d, 2 + d] += c0
    r += _sum(n, i, torch.einsum("tab,tb->ta", K, u[j] - u[i]))
    return [_csr_values(n, i, j, -K, kii + _sum(n, i, K)), r.reshape(-1)]


def _bicgstab(A, b, diag, tol=1e-15, most=400):
    """Jacobi-preconditioned BiCGStab, the best iterate seen."""
    x = torch.zeros_like(b)
    r = b.clone()
    r0, rho, al, om = r.clone(), 1.0, 1.0, 1.0
    v = p = torch.zeros_like(b)
    scale, best = float(b.norm()), (math.inf, x)
    for _ in range(most):
        rho1 = float(r0 @ r)
        if rho1 == 0.0 or scale == 0.0:
            break
        p = r + (rho1 / rho) * (al / om) * (p - om * v)
        y = p / diag
        v = A(y)
        al = rho1 / float(r0 @ v)
        s = r - al * v
        z = s / diag
        t = A(z)
        om = float(t @ s) / max(float(t @ t), 1e-300)
        x = x + al * y + om * z
        r = s - om * t
        rho = rho1
        e = float(r.norm())
        if e < best[0]:
            best = (e, x)
        if e <= tol * scale:
            break
    return best[1]


def _exact_chrun(case, seed):
    L, x, vol, i, j, g = _plain_mesh(dict(case, dim=2, nz=1))
    n, nbulk = L["n"], L["nbulk"]
    lap, back, ghost = _ch_laplacian(L, x, i, j, g)
    chi, kappa, M0, dt = CH["chi"], CH["kappa"], CH["M0"], CH["dt"]
    keep = ~ghost[i] & ~ghost[j]  # bonds to ghosts carry nothing, ghosts follow their mirrors
    bi, bj, l2, lb = i[keep], j[keep], lap[keep], back[keep]
    vr = vol[bj] / vol[bi]
    c = torch.from_numpy(0.5 + np.random.default_rng(seed).uniform(-0.01, 0.01, n)).to(DEV)[:nbulk]
    mu = torch.zeros_like(c)
    Lc = lambda v: _sum(nbulk, bi, l2 * (v[bj] - v[bi]))  # noqa: E731
    for _ in range(case["steps"]):
        old = c
        for _ in range(40):
            k = c.clamp(1e-8, 1 - 1e-8)
            mob = M0 * k * (1 - k)
            w = 0.5 * (mob[bi] * l2 + vr * mob[bj] * lb)
            A = lambda v: -_sum(nbulk, bi, w * (v[bj] - v[bi]))  # noqa: E731, B023
            fp, fpp = torch.log(k / (1 - k)) + chi * (1 - 2 * k), 1 / (k * (1 - k)) - 2 * chi
            target = fp - kappa * Lc(c)  # mu of this c
            rhs = -((c - old) / dt + A(target))
            S = lambda v: v / dt + A(fpp * v - kappa * Lc(v))  # noqa: E731, B023
            diag = 1 / dt + _sum(nbulk, bi, w) * (fpp + kappa * _sum(nbulk, bi, l2))
            dc = _bicgstab(S, rhs, diag)
            c = c + dc
            mu = target + fpp * dc - kappa * Lc(dc)
            if float(dc.norm()) <= 1e-15 * float(c.norm()):
                break
    k = c.clamp(1e-8, 1 - 1e-8)
    mu = torch.log(k / (1 - k)) + chi * (1 - 2 * k) - kappa * Lc(c)
    full = torch.from_numpy(np.where(L["mirror"] > 0, L["mirror"] - 1, np.arange(n)).astype(np.int64)).to(DEV)
    c, mu = c[full], mu[full]
    grad = _sum(n, i, g[:, :2] * (c[j] - c[i])[:, None])
    dens = c * torch.log(c) + (1 - c) * torch.log(1 - c) + chi * c * (1 - c) + 0.5 * kappa * grad.square().sum(1)
    return [torch.stack([c, mu], 1).reshape(-1), float((vol * dens)[:nbulk].sum())]


def _break(alive, K, x, i, j, u, sc, tension_only):
    """One damage pass over bonds that are alive."""
    xi = x[j, :u.shape[1]] - x[i, :u.shape[1]]
    r = xi.square().sum(1).sqrt()
    s = ((xi + u[j] - u[i]).square().sum(1).sqrt() - r) / r
    return alive & ~((s if tension_only else s.abs()) > sc)


def _force(n, K, alive, i, j, u, rho):
    return _sum(n, i, torch.einsum("tab,tb->ta", K, u[j] - u[i]) * alive.double()[:, None]) / rho


def _preset(L):
    """The boundary pass as a function of (u, t)."""
    top, bottom = (torch.from_numpy(v.astype(np.int64)).to(DEV) - 1 for v in _boundary(L))
    g = torch.arange(L["nbulk"], L["n"], device=DEV)
    b = torch.from_numpy(L["mirror"][L["nbulk"]:].astype(np.int64)).to(DEV) - 1

    def apply(u, t):
        u = u.index_copy(0, g, u[b])
        y = u[:, 1].index_fill(0, top, 2.0 * t).index_fill(0, bottom, -2.0 * t)
        return torch.cat([u[:, :1], y[:, None], u[:, 2:]], 1)
    return apply


def _exact_explicit(case, seed):
    L, x, vol, i, j, g = _plain_mesh(case)
    n, dim = L["n"], L["dim"]
    Cs, rho, sc = _material(dim)
    K = _navier(g, dim, Cs)
    del g
    alive = ~_broken(L, i, j, seed, L["m"][0] // 6)
    u = _smooth(x, seed, dim, 0.7 * sc)
    to = case.get("tension_only", True)
    alive = _break(alive, K, x, i, j, u, sc, to)
    a = _force(n, K, alive, i, j, u, rho)
    if case["kind"] == "rate":
        return a.reshape(-1)
    dt, preset, t = _dt(L, Cs, rho), _preset(L), 0.0
    up = u + 0.5 * dt * dt * a
    for _ in range(case["steps"]):
        alive = _break(alive, K, x, i, j, u, sc, to)
        t = t + dt
        up, u = u, preset(2 * u - up + dt * dt * _force(n, K, alive, i, j, u, rho), t)
    return [u.reshape(-1), up.reshape(-1), None]


def _exact_inverse(case, seed):
    L, x, vol, i, j, g = _plain_mesh(case)
    n, dim = L["n"], L["dim"]
    Cs, rho, sc = _material(dim)
    alive = (~_broken(L, i, j, seed, L["m"][0] // 6)).double()
    u0 = _smooth(x, seed, dim, 0.7 * sc).reshape(-1)
    dt, preset = _dt(L, Cs, rho), _preset(L)
    Ct = torch.tensor(Cs, dtype=torch.float64, device=DEV, requires_grad=True)
    u0 = u0.requires_grad_(True)
    # the force is linear in C: its three parts, bond blocks kept once
    parts = [_navier(g, dim, c) * alive[:, None, None] / rho for c in ((1.0, 0, 0), (0, 1.0, 0), (0, 0, 1.0))]
    back = torch.searchsorted(i * n + j, j * n + i)

    class Force(torch.autograd.Function):
        @staticmethod
        def forward(ctx, u, c):
            e = u[j] - u[i]
            ctx.save_for_backward(u, c)
            return sum(_sum(n, i, torch.einsum("tab,tb->ta", P, e)) * c[k] for k, P in enumerate(parts))

        @staticmethod
        def backward(ctx, w):
            u, c = ctx.saved_tensors
            e, wi, wj = u[j] - u[i], w[i], w[j]
            gu, gc = torch.zeros_like(u), []
            for k, P in enumerate(parts):
                own = torch.einsum("tab,ta->tb", P, wi)
                gc.append((own * e).sum())
                gu += c[k] * _sum(n, i, torch.einsum("tab,ta->tb", P[back], wj) - own)
            return gu, torch.stack(gc)

    u = u0.reshape(n, dim)
    up, t = u + 0.5 * dt * dt * Force.apply(u, Ct), 0.0
    for _ in range(case["steps"]):
        t = t + dt
        up, u = u, preset(2 * u - up + dt * dt * Force.apply(u, Ct), t)
    w = torch.randn(u0.numel(), generator=_generator(seed), dtype=torch.float64, device=DEV)
    gu, gc = torch.autograd.grad(u.reshape(-1), [u0, Ct], w)
    return [u.detach().reshape(-1), gu, gc]


def _exact_field(case, seed):
    L, x, vol, i, j, g = _plain_mesh(case)
    n = L["n"]
    u = _smooth(x, seed, 1, 1.0)[:, 0]
    w = torch.randn(n, g.shape[1], generator=_generator(seed), dtype=torch.float64, device=DEV)
    s = (g * w[i]).sum(1)
    return [_sum(n, i, g * (u[j] - u[i])[:, None]), _sum(n, j, s) - _sum(n, i, s)]


def _exact_clouds(case, seed):
    clouds = _cloud_list(case, seed)
    out = []
    for c, u in zip(clouds, _cloud_fields(clouds, seed)):
        x, vol = torch.from_numpy(c["coords3"]).to(DEV), torch.from_numpy(c["vols"]).to(DEV)
        i, j = _pairs(x, c["delta"], c["dim"])
        g = _operators(x, vol, i, j, c["delta"], c["dx_char"], c["dim"])
        out.append(_sum(len(x), i, g * (u[j] - u[i])[:, None]).reshape(-1))
    return torch.cat(out)


def exact(case, seed):
    return {"scalar": _exact_scalar, "setup": _exact_scalar, "dynfrac": _exact_dynfrac, "stress": _exact_stress,
            "chrun": _exact_chrun, "run": _exact_explicit, "rate": _exact_explicit, "clouds": _exact_clouds,
            "field": _exact_field, "inverse": _exact_inverse}[case["kind"]](case, seed)
