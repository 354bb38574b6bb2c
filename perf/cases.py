"""What this library's performance is measured on.

Each case is a piece of work that a program using the library has it do through
its public entry points: a driver hands a state in from pinned host columns,
has it advanced some steps (or has one density and one force evaluation made of
it) and reads the new state back.  The two ``device_density`` cases call the
allocation-free entry point on caller-owned device arrays instead.

The workloads are the library's own configurations (``spearhed_b200.setups``:
Sod tube, Orszag-Tang slab, Kelvin-Helmholtz cube, MHD rotor, Brio-Wu ensemble)
and the reference's walled channel with tracers, at sizes from a few thousand
to two million particles.  Lattices are jittered by the seed, as particles are
after their first steps.

``exact`` evaluates the same equations in 64 bits with plain torch operations.
"""
import ctypes as C
import math

import numpy as np
import torch

import spearhed_b200 as sb
from spearhed_b200 import abi, flops, setups

FLUID, WALL, TRACER = abi.SPECIES_DEFAULT, abi.SPECIES_BOUNDARY, abi.SPECIES_TRACER
PRECISION = {"fp32": abi.PREC_FP32_COMP, "fp64": abi.PREC_FP64}
KERNEL = {"cubic": abi.KERNEL_CUBIC, "quintic": abi.KERNEL_QUINTIC, "wendland": abi.KERNEL_WENDLAND_C2}


def listed():
    return [
        # a tube small enough that a step's launches and its longest rows are all there is
        {"name": "sod_tiny_fp64", "kind": "sod", "prec": "fp64", "scale": 0.5, "steps": 20},
        # the Sod configuration as it stands (18,432 particles): AV, CFL, adaptive h, two cell levels
        {"name": "sod_fp32", "kind": "sod", "prec": "fp32", "scale": 1.0, "steps": 20},
        # the Orszag-Tang configuration at its full 512 x 512 x 4: one level, one h, full SPMHD
        {"name": "orszag_tang_fp32", "kind": "orszag_tang", "prec": "fp32", "nx": 512, "nz": 4, "steps": 10},
        # the FP64 path on an odd slab
        {"name": "orszag_tang_fp64", "kind": "orszag_tang", "prec": "fp64", "nx": 203, "nz": 5, "steps": 10},
        # shear flow in a periodic cube: adaptive h over a factor 1.26, one level, 1.4 M particles
        {"name": "kelvin_helmholtz_fp32", "kind": "kelvin_helmholtz", "prec": "fp32", "n_outer": 96, "n_band": 122,
         "steps": 8},
        # a ten-fold density contrast: two cell levels, uneven cells
        {"name": "rotor_fp32", "kind": "rotor", "prec": "fp32", "nxy": 417, "nz": 4, "steps": 8},
        # the headline's batched path: independent Brio-Wu tubes, a time step each, two levels
        {"name": "tubes_fp32", "kind": "tubes", "prec": "fp32", "nbox": 32, "n_lo": 4096, "n_hi": 262144, "steps": 8},
        # a few small tubes in FP64
        {"name": "tubes_fp64", "kind": "tubes", "prec": "fp64", "nbox": 8, "n_lo": 4096, "n_hi": 65536, "steps": 8},
        # the reference's own physics, stage by stage (UpdateDensity, UpdateHydroForces), quintic spline
        {"name": "hydro_stages_fp32", "kind": "stages", "prec": "fp32", "kernel": "quintic", "nx": 61, "ny": 53,
         "nz": 47},
        # walls and tracers beside the fluid: the three species of the reference's time-step test
        {"name": "channel_fp32", "kind": "channel", "prec": "fp32", "nx": 120, "ny": 40, "tracers": 4001, "steps": 10},
        # density of device arrays without allocation, near the entry point's limit
        {"name": "device_density_fp32", "kind": "device", "prec": "fp32", "kernel": "cubic", "n": 250007},
        # and a small call, where launches count
        {"name": "device_density_fp64", "kind": "device", "prec": "fp64", "kernel": "wendland", "n": 6007},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(["sod", "orszag_tang", "kelvin_helmholtz", "rotor", "tubes", "stages", "channel", "device"])
    c = {"kind": kind, "prec": rng.choice(["fp32", "fp32", "fp64"])}
    if kind == "sod":
        c |= {"scale": round(_log(rng, 0.5, 2.5), 3), "steps": rng.randint(6, 20)}
    elif kind == "orszag_tang":
        # at most 0.4 M particles in FP64, 1.0 M in FP32
        c |= {"nx": int(_log(rng, 40, 280 if c["prec"] == "fp64" else 450)), "nz": rng.randint(4, 5),
              "steps": rng.randint(3, 10)}
    elif kind == "kelvin_helmholtz":
        m = int(_log(rng, 8, 17 if c["prec"] == "fp64" else 24))
        c |= {"n_outer": 4 * m, "n_band": 2 * round(4 * m * 2 ** (1 / 3) / 2), "steps": rng.randint(3, 8)}
    elif kind == "rotor":
        c |= {"nxy": int(_log(rng, 64, 250 if c["prec"] == "fp64" else 400)), "nz": 4, "steps": rng.randint(3, 8)}
    elif kind == "tubes":
        nbox = int(_log(rng, 1, 25))
        c |= {"nbox": nbox, "n_lo": 4096, "n_hi": int(_log(rng, 8192, 65536 if c["prec"] == "fp64" else 200000)),
              "steps": rng.randint(3, 8)}
    elif kind == "stages":
        c |= {"kernel": rng.choice(["cubic", "quintic", "wendland"]), "nx": int(_log(rng, 12, 70)),
              "ny": int(_log(rng, 12, 70)), "nz": int(_log(rng, 12, 60))}
    elif kind == "channel":
        c |= {"nx": int(_log(rng, 30, 160)), "ny": int(_log(rng, 10, 44)), "tracers": int(_log(rng, 11, 9000)),
              "steps": rng.randint(3, 10)}
    else:
        c |= {"kernel": rng.choice(["cubic", "quintic", "wendland"]), "n": int(_log(rng, 500, 262144))}
    return c


# ---------------------------------------------------------------- inputs
def _perturb(s, lo, hi, periodic, amplitude, rng):
    """Displaces every particle by up to amplitude x h / 1.2 per axis, inside its box, and
    adds a velocity noise of 1e-2 (the seed's own disturbance of an exact lattice)."""
    d = amplitude * s.h / 1.2
    for a in range(3):
        x = s.pos[a] + d * rng.uniform(-1.0, 1.0, s.n)
        L = np.asarray(hi[a]) - np.asarray(lo[a])
        s.pos[a] = lo[a] + (x - lo[a]) % L if periodic[a] else np.clip(x, lo[a], hi[a])
        s.vel[a] += 1e-2 * rng.uniform(-1.0, 1.0, s.n)


def _disturb_field(s, amplitude, rng):
    """Adds a divergence-free disturbance to B, as a flow has after its first steps."""
    ph = rng.uniform(0.0, 2.0 * math.pi, 2)
    s.B[0] += amplitude * np.sin(4 * math.pi * s.pos[1] + ph[0])
    s.B[1] += amplitude * np.sin(4 * math.pi * s.pos[0] + ph[1])


def _channel(case, rng):
    """A fluid between two frozen walls of four layers, periodic in y and z, with tracers."""
    prec = PRECISION[case["prec"]]
    nx, ny = case["nx"], case["ny"]
    dx = 1.0 / (nx + 8)

    def species(pos, jitter):
        s = abi.Species(pos.shape[1])
        s.pos[:] = pos
        s.mass[:] = dx ** 3
        s.h[:] = 1.2 * dx
        s.density[:] = 1.0
        s.u[:] = 1.5
        if jitter:
            s.pos += jitter * dx * rng.uniform(-1.0, 1.0, s.pos.shape)
            for a in (1, 2):
                s.pos[a] %= ny * dx
        return s

    lat = lambda x0, n: setups.lattice((x0, 0.0, 0.0), (x0 + n * dx, ny * dx, ny * dx), (n, ny, ny))  # noqa: E731
    fluid = species(lat(4 * dx, nx), 0.05)
    fluid.vel[0] = 0.2 * np.sin(2 * math.pi * (fluid.pos[0] - 4 * dx) / (nx * dx))
    fluid.vel[1] = 0.3 * np.cos(2 * math.pi * fluid.pos[0])
    walls = species(np.concatenate([lat(0.0, 4), lat((nx + 4) * dx, 4)], axis=1), 0.0)
    tr = species(rng.uniform((0.2, 0.0, 0.0), (0.8, ny * dx, ny * dx), size=(case["tracers"], 3)).T.copy(), 0.0)
    tr.vel[:] = 0.05 * rng.standard_normal(tr.vel.shape)
    params = abi.default_params(kernel=abi.KERNEL_CUBIC, precision=prec, physics=abi.PHYS_AV | abi.PHYS_CFL,
                                h0=1.2 * dx, gamma=1.4, dt=0.05 * dx)
    # room beyond the walls: nothing reaches it
    box = abi.make_box((-0.5, 0.0, 0.0), (1.5, ny * dx, ny * dx), (0, 1, 1))
    return params, [box], {FLUID: fluid, WALL: walls, TRACER: tr}


def _inputs(case, seed):
    """(params, boxes, {species id: host columns}) of a case, from the seed alone."""
    rng = np.random.default_rng(seed)
    kind, prec = case["kind"], PRECISION[case["prec"]]
    if kind == "sod":
        w = setups.sod_small(precision=prec, scale=case["scale"])
        _perturb(w.species[FLUID], (-0.75, 0, 0), (0.75, 0.125, 0.125), (0, 1, 1), 0.05, rng)
    elif kind == "orszag_tang":
        w = setups.orszag_tang(nx=case["nx"], nz=case["nz"], precision=prec, jitter=0.05, seed=seed)
    elif kind == "kelvin_helmholtz":
        w = setups.kelvin_helmholtz(case["n_outer"], case["n_band"], precision=prec, seed=seed)
        _disturb_field(w.species[FLUID], 0.02, rng)
    elif kind == "rotor":
        w = setups.mhd_rotor(case["nxy"], case["nz"], precision=prec, seed=seed)
        _disturb_field(w.species[FLUID], 0.05, rng)
    elif kind == "tubes":
        w = setups.brio_wu_ensemble(case["nbox"], precision=prec, n_lo=case["n_lo"], n_hi=case["n_hi"])
        s = w.species[FLUID]
        L = np.array([b.hi[1] for b in w.boxes])[s.box_id]
        _perturb(s, (-0.75, 0.0, 0.0), (0.75, L, L), (0, 1, 1), 0.05, rng)
    elif kind == "channel":
        return _channel(case, rng)
    elif kind == "stages":
        # an open block of fluid under the reference's inviscid hydro, one h
        n = (case["nx"], case["ny"], case["nz"])
        dx = 1.0 / max(n)
        s = abi.Species(n[0] * n[1] * n[2])
        hi = tuple(k * dx for k in n)
        s.pos[:] = setups.lattice((0.0, 0.0, 0.0), hi, n)
        s.mass[:] = dx ** 3
        s.h[:] = 1.2 * dx
        s.u[:] = 1.5 + 0.5 * np.sin(2 * math.pi * s.pos[0])
        s.vel[:] = 0.3 * np.sin(2 * math.pi * s.pos[[1, 2, 0]])
        _perturb(s, (0, 0, 0), hi, (0, 0, 0), 0.1, rng)
        params = abi.default_params(kernel=KERNEL[case["kernel"]], precision=prec, h0=1.2 * dx)
        return params, [abi.make_box((0, 0, 0), hi)], {FLUID: s}
    return w.params, w.boxes, w.species


def _cloud(case, seed):
    """Random positions in the unit box (periodic in y and z), about 40 neighbours each."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    sup = 3 if case["kernel"] == "quintic" else 2
    h0 = min((40.0 / n * 3.0 / (4.0 * math.pi)) ** (1.0 / 3.0) / sup, 0.3)
    x = rng.uniform(0.0, 1.0, (3, n))
    mass = rng.uniform(0.5, 1.5, n) / n
    h = np.full(n, h0) * rng.uniform(0.9, 1.0, n)
    params = abi.default_params(kernel=KERNEL[case["kernel"]], precision=PRECISION[case["prec"]], h0=h0)
    return params, abi.make_box((0, 0, 0), (1, 1, 1), (0, 1, 1)), x, mass, h


# ---------------------------------------------------------------- the program under measurement
_DP = C.POINTER(C.c_double)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    out = t.numpy()
    out[...] = a
    return out


def _view(columns):
    v = abi.SphSoAView()
    for name, a in columns.items():
        if a.ndim == 2:
            for k in range(3):
                getattr(v, name)[k] = a[k].ctypes.data_as(_DP)
        else:
            setattr(v, name, a.ctypes.data_as(_DP))
    return v


def _columns(params, sid):
    """Input and output columns of one species."""
    mhd = bool(params.physics & abi.PHYS_MHD)
    cin = ["pos", "vel", "mass", "h", "u"] + (["B", "psi"] if mhd else [])
    if sid == WALL:
        return cin + ["density"], []
    if sid == TRACER:
        return cin, ["pos"]
    out = ["pos", "vel", "density", "u"] + (["B", "psi"] if mhd else [])
    return cin, out + (["h"] if params.physics & abi.PHYS_ADAPTIVE_H else [])


def prepare(case, seed):
    if case["kind"] == "device":
        params, box, x, mass, h = _cloud(case, seed)
        cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x[0], x[1], x[2], mass, h)]
        rho = torch.empty(case["n"], dtype=torch.float64, device="cuda")
        return {"params": params, "box": box, "cols": cols, "rho": rho, "n": case["n"],
                "stream": torch.cuda.current_stream().cuda_stream}
    params, boxes, species = _inputs(case, seed)
    ctx = sb.Context(params, boxes)
    st = {"ctx": ctx, "in": {}, "out": {}, "keep": {}, "steps": case.get("steps", 0), "dt": params.dt}
    for sid, s in species.items():
        ctx.set_species(sid, s)
        cin, cout = _columns(params, sid)
        if case["kind"] == "stages":
            cout = ["density", "dvdt", "dudt"]
        host = {c: _pinned(getattr(s, c)) for c in cin}
        back = {c: _pinned(np.zeros_like(getattr(s, c))) for c in cout}
        st["keep"][sid], st["out"][sid] = host, back
        st["in"][sid] = (s.n, _view(host), _view(back))
    if st["steps"]:
        ctx.use_graph(True)
        ctx.prepare_graph()
    else:
        ctx.density()
    return st


def run(st):
    L = abi.lib()
    if "rho" in st:
        abi.check(L.sph_density_noalloc(C.byref(st["params"]), C.byref(st["box"]), st["n"],
                                        *[c.data_ptr() for c in st["cols"]], st["rho"].data_ptr(), st["stream"]))
        return {"rho": st["rho"]}
    ctx = st["ctx"]
    for sid, (n, vin, _) in st["in"].items():
        abi.check(L.sph_set_species(ctx._p, sid, abi.SPECIES_ROLES[sid], n, C.byref(vin)))
    clock = None
    if st["steps"]:
        ctx.set_clock(0.0, st["dt"])
        ctx.step(st["steps"])
        # (time, next dt) per box, as a run's log holds it: the time step is one particle's
        # signal speed, which FP32 cases know to 32 bits
        clock = np.stack(ctx.clock()).astype(np.float32)
    else:
        sb.UpdateDensity(ctx)
        sb.UpdateHydroForces(ctx)
    for sid, (_, _, vout) in st["in"].items():
        if st["out"][sid]:
            abi.check(L.sph_get_species(ctx._p, sid, C.byref(vout)))
    out = {f"species{sid}": cols for sid, cols in st["out"].items() if cols}
    if clock is not None:
        out["clock"] = clock
    return out


def _counts(case):
    """(fluid, wall, tracer) particles of a case."""
    k = case["kind"]
    if k == "sod":
        a, b = int(64 * case["scale"]), int(16 * case["scale"])
        return a * b * b + int(32 * case["scale"]) * int(8 * case["scale"]) ** 2, 0, 0
    if k == "orszag_tang":
        return case["nx"] ** 2 * case["nz"], 0, 0
    if k == "kelvin_helmholtz":
        return (case["n_outer"] ** 3 + case["n_band"] ** 3) // 2, 0, 0
    if k == "rotor":
        return int(case["nxy"] ** 2 * case["nz"] * (1.0 + 9.0 * math.pi * 0.01)), 0, 0
    if k == "tubes":
        return int(setups.brio_wu_sizes(case["nbox"], n_lo=case["n_lo"], n_hi=case["n_hi"]).sum()), 0, 0
    if k == "channel":
        return case["nx"] * case["ny"] ** 2, 8 * case["ny"] ** 2, case["tracers"]
    if k == "stages":
        return case["nx"] * case["ny"] * case["nz"], 0, 0
    return case["n"], 0, 0


def work(case):
    """Each input column read and each output column written once; the pair terms of
    every step (spearhed_b200.flops), at the lattice's mean neighbour count."""
    fluid, wall, tracer = _counts(case)
    k = case["kind"]
    if k == "device":
        kern = {"cubic": "cubic", "quintic": "quintic", "wendland": "wendland_c2"}[case["kernel"]]
        return {"bytes": 8.0 * 6 * fluid, "flops": 40.0 * fluid * flops.DENSITY_FLOPS[kern]}
    wide = k in ("orszag_tang", "kelvin_helmholtz", "rotor")  # Wendland C2 at 1.45 spacings
    mhd = wide or k == "tubes"
    radius = 2.9 if wide else 3.6 if case.get("kernel") == "quintic" else 2.4
    pairs = (4.0 / 3.0 * math.pi * radius ** 3 - 1.0) * fluid
    per = flops.DENSITY_FLOPS["cubic"] + flops.FORCE_FLOPS["mhd" if mhd else "hydro"]
    ins = 13 if mhd else 9
    outs = 5 if k == "stages" else 12 if mhd else 8
    return {"bytes": 8.0 * (ins * (fluid + wall + tracer) + outs * fluid + 3 * tracer),
            "flops": pairs * per * case.get("steps", 1)}


# ---------------------------------------------------------------- the same equations in 64 bits
_CHUNK = 12_000_000  # candidate pairs at once


def _support(kernel):
    return 3.0 if kernel == abi.KERNEL_QUINTIC else 2.0


def _shape(kernel, q):
    """Kernel shape w(q) and dw/dq without the norm."""
    p = lambda c: torch.clamp(c - q, min=0.0)  # noqa: E731
    if kernel == abi.KERNEL_CUBIC:
        a, b = p(2.0), p(1.0)
        return 0.25 * a ** 3 - b ** 3, -0.75 * a ** 2 + 3.0 * b ** 2
    if kernel == abi.KERNEL_QUINTIC:
        a, b, c = p(3.0), p(2.0), p(1.0)
        return a ** 5 - 6 * b ** 5 + 15 * c ** 5, -5 * a ** 4 + 30 * b ** 4 - 75 * c ** 4
    t = torch.clamp(1.0 - 0.5 * q, min=0.0)
    return t ** 4 * (1.0 + 2.0 * q), -5.0 * q * t ** 3


_NORM = {abi.KERNEL_CUBIC: 1.0 / math.pi, abi.KERNEL_QUINTIC: 1.0 / (120.0 * math.pi),
         abi.KERNEL_WENDLAND_C2: 21.0 / (16.0 * math.pi)}


def _pairs(x, lo, L, periodic, R, pair_max, target, source):
    """Chunks (i, j, r_i - r_j) of every pair of a target i and a source j (or an image of
    it) nearer than R (one number, or max(R_i, R_j) with pair_max); not the particle itself."""
    dev = x[0].device
    rmax = float(R.max()) if pair_max else float(R)
    n = [max(1, min(1024, int(L[a] / (rmax * (1 + 1e-5))))) for a in range(3)]
    cell = [torch.clamp(((x[a] - lo[a]) / (L[a] / n[a])).floor().long(), 0, n[a] - 1) for a in range(3)]
    js = torch.nonzero(source).flatten()
    key = ((cell[2] * n[1] + cell[1]) * n[0] + cell[0])[js]
    key, order = torch.sort(key)
    js = js[order]
    start = torch.searchsorted(key, torch.arange(n[0] * n[1] * n[2] + 1, device=dev))
    o = torch.tensor([[a, b, c] for c in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)], device=dev)
    ts = torch.nonzero(target).flatten()
    # targets in cell order share their candidates' memory
    ts = ts[torch.argsort((cell[2] * n[1] + cell[1])[ts] * n[0] + cell[0][ts])]
    cnt = start[1:] - start[:-1]
    for part in torch.split(ts, max(1, int(_CHUNK / max(1.0, 27.0 * float(cnt.double().mean()) * 4.0)))):
        id_, img, ok = 0, [], None
        for a in (2, 1, 0):
            c = cell[a][part][:, None] + o[None, :, a]
            w = c % n[a] if periodic[a] else torch.clamp(c, 0, n[a] - 1)
            good = torch.ones_like(c, dtype=torch.bool) if periodic[a] else c == w
            ok = good if ok is None else ok & good
            img.append(((c - w) // n[a]).double() * L[a] if periodic[a] else None)
            id_ = id_ * n[a] + w
        img = img[::-1]
        k = torch.where(ok, cnt[id_], 0).flatten()
        first = start[id_].flatten()
        total = int(k.sum())
        for lo_row, hi_row in _row_blocks(k, total):
            kk = k[lo_row:hi_row]
            row = torch.repeat_interleave(torch.arange(lo_row, hi_row, device=dev), kk)
            base = torch.cumsum(kk, 0) - kk
            j = js[first[row] + torch.arange(row.numel(), device=dev) - base[row - lo_row]]
            i = part[row // 27]
            d, r2, moved = [], 0.0, torch.zeros_like(i, dtype=torch.bool)
            for a in range(3):
                xj = x[a][j]
                if img[a] is not None:
                    s = img[a].flatten()[row]
                    xj = xj + s
                    moved |= s != 0.0
                d.append(x[a][i] - xj)
                r2 = r2 + d[a] * d[a]
            rr = torch.maximum(R[i], R[j]) if pair_max else R
            keep = (r2 < rr * rr) & ((i != j) | moved)
            yield i[keep], j[keep], [q[keep] for q in d]


def _row_blocks(k, total):
    """Ranges of rows holding at most about _CHUNK candidates each."""
    if total <= _CHUNK:
        yield 0, k.numel()
        return
    ends = torch.cumsum(k, 0)
    lo = 0
    while lo < k.numel():
        done = int(ends[lo - 1]) if lo else 0
        hi = max(lo + 1, int(torch.searchsorted(ends, done + _CHUNK, right=True)))
        yield lo, min(hi, k.numel())
        lo = min(hi, k.numel())


class _Box:
    """One box of particles under the library's equations, in 64 bits."""

    def __init__(self, p, box, cols, roles, dev):
        self.p, self.dev = p, dev
        self.lo, self.L = list(box.lo), [box.hi[a] - box.lo[a] for a in range(3)]
        self.periodic = [bool(v) for v in box.periodic]
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.x, self.v, self.B = ([t(cols[c][a]) for a in range(3)] for c in ("pos", "vel", "B"))
        self.m, self.h, self.u, self.psi, self.rho = (t(cols[c]) for c in ("mass", "h", "u", "psi", "density"))
        roles = t(roles)
        self.movable = (roles & abi.ROLE_MOVABLE) != 0
        self.source = (roles & abi.ROLE_SOURCE) != 0
        self.target = self.movable & ((roles & abi.ROLE_THERMODYNAMIC) != 0)
        self.dt, self.time = p.dt, 0.0
        self.cap = p.h_max if p.h_max > 0 else 1e300
        if p.h_max <= 0 and p.physics & abi.PHYS_ADAPTIVE_H:
            for a in range(3):
                if self.periodic[a]:
                    lim = self.L[a] / (_support(p.kernel) * (1.0 + 1.0 / 262144.0))
                    self.cap = min(self.cap, max(lim, float(self.h.max())))

    def pairs(self):
        pm = self.p.cull == abi.CULL_PAIR_MAX
        R = _support(self.p.kernel) * (self.h if pm else self.p.h0)
        return _pairs(self.x, self.lo, self.L, self.periodic, R, pm, self.target, self.source)

    def density(self):
        k = self.p.kernel
        norm = _NORM[k] / self.h ** 3
        acc = self.m * norm * _shape(k, torch.zeros_like(self.h))[0]
        for i, j, d in self.pairs():
            r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
            acc.index_add_(0, i, self.m[j] * norm[i] * _shape(k, r / self.h[i])[0])
        self.rho = torch.where(self.target, acc, self.rho)

    def force(self):
        p, k = self.p, self.p.kernel
        av, mhd = bool(p.physics & abi.PHYS_AV), bool(p.physics & abi.PHYS_MHD)
        dedner, tensile = mhd and bool(p.physics & abi.PHYS_DEDNER), mhd and bool(p.physics & abi.PHYS_TENSILE)
        x, v, B, h, m, psi = self.x, self.v, self.B, self.h, self.m, self.psi
        rho = torch.where(self.rho > 0, self.rho, 1.0)
        P = (p.gamma - 1.0) * rho * self.u
        B2 = B[0] ** 2 + B[1] ** 2 + B[2] ** 2 if mhd else torch.zeros_like(rho)
        c = torch.sqrt(p.gamma * P / rho + B2 / (p.mu0 * rho))
        pt = (P + 0.5 * B2 / p.mu0) / rho ** 2
        z = lambda: torch.zeros_like(rho)  # noqa: E731
        a, T, gp = [z(), z(), z()], [z(), z(), z()], [z(), z(), z()]
        D, heat, div, tens, vsig = z(), z(), z(), z(), c.clone()
        for i, j, r in self.pairs():
            r2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2
            dist = torch.sqrt(r2)
            inv = torch.where(r2 > 0, 1.0 / torch.where(r2 > 0, dist, 1.0), 0.0)
            si = _NORM[k] / h[i] ** 4 * _shape(k, dist / h[i])[1] * inv
            sj = _NORM[k] / h[j] ** 4 * _shape(k, dist / h[j])[1] * inv
            mj = m[j]
            dv = [v[q][i] - v[q][j] for q in range(3)]
            vr = dv[0] * r[0] + dv[1] * r[1] + dv[2] * r[2]
            f = -mj * (pt[i] * si + pt[j] * sj)
            if av:
                hb = 0.5 * (h[i] + h[j])
                mu = hb * torch.clamp(vr, max=0.0) / (r2 + p.av_eps * hb * hb)
                Pi = (-p.alpha * 0.5 * (c[i] + c[j]) * mu + p.beta * mu * mu) / (0.5 * (rho[i] + rho[j]))
                g = mj * Pi * 0.5 * (si + sj)
                f = f - g
                heat.index_add_(0, i, 0.5 * g * vr)
            D.index_add_(0, i, mj * si * vr)
            vsig.index_reduce_(0, i, c[i] + c[j] - p.beta * torch.clamp(vr * inv, max=0.0), "amax")
            F = [f * r[q] for q in range(3)]
            if mhd:
                Bi = B[0][i] * r[0] + B[1][i] * r[1] + B[2][i] * r[2]
                Bj = B[0][j] * r[0] + B[1][j] * r[1] + B[2][j] * r[2]
                ci, cj = mj * si * Bi / (p.mu0 * rho[i] ** 2), mj * sj * Bj / (p.mu0 * rho[j] ** 2)
                tens.index_add_(0, i, ci + cj)
                div.index_add_(0, i, mj * si * (Bi - Bj))
                for q in range(3):
                    F[q] = F[q] + ci * B[q][i] + cj * B[q][j]
                    T[q].index_add_(0, i, mj * si * Bi * dv[q])
                if dedner:
                    g = mj * (psi[i] / rho[i] ** 2 * si + psi[j] / rho[j] ** 2 * sj)
                    for q in range(3):
                        gp[q].index_add_(0, i, g * r[q])
            for q in range(3):
                a[q].index_add_(0, i, F[q])
        t = self.target
        if tensile:
            a = [a[q] - B[q] * tens for q in range(3)]
        self.a = [torch.where(t, a[q], 0.0) for q in range(3)]
        self.du = torch.where(t, P / rho ** 2 * D + heat, 0.0)
        self.dB, self.dpsi = None, None
        if mhd:
            divB, divv = -div / rho, -D / rho
            self.dB = [torch.where(t, -(T[q] - B[q] * D) / rho - rho * gp[q], 0.0) for q in range(3)]
            if dedner:
                ch = c[t].max()
                self.dpsi = torch.where(t, -ch * ch * divB - psi * p.dedner_sigma * ch / h - 0.5 * psi * divv, 0.0)
        lim = p.cfl * h / vsig
        amag = torch.sqrt(a[0] ** 2 + a[1] ** 2 + a[2] ** 2)
        some = (amag > 0) & (p.cfl_force > 0)
        lim = torch.where(some, torch.minimum(lim, p.cfl_force * torch.sqrt(h / torch.where(some, amag, 1.0))), lim)
        self.dt_next = float(lim[t].min())

    def step(self):
        p, dt = self.p, self.dt
        for a in range(3):
            self.x[a] = torch.where(self.movable, self.x[a] + self.v[a] * dt, self.x[a])
            if self.periodic[a]:
                hi = self.lo[a] + self.L[a]
                self.x[a] = torch.where(self.movable & (self.x[a] >= hi), self.x[a] - self.L[a], self.x[a])
                self.x[a] = torch.where(self.movable & (self.x[a] < self.lo[a]), self.x[a] + self.L[a], self.x[a])
        self.density()
        self.force()
        self.v = [self.v[q] + self.a[q] * dt for q in range(3)]
        self.u = self.u + self.du * dt
        if self.dB is not None:
            self.B = [self.B[q] + self.dB[q] * dt for q in range(3)]
        if self.dpsi is not None:
            self.psi = self.psi + self.dpsi * dt
        if p.physics & abi.PHYS_ADAPTIVE_H:
            hn = p.hfact * (self.m / self.rho) ** (1.0 / 3.0)
            self.h = torch.where(self.target, torch.clamp(hn, max=self.cap), self.h)
        self.time += dt
        if p.physics & abi.PHYS_CFL:
            self.dt = self.dt_next


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if case["kind"] == "device":
        params, box, x, mass, h = _cloud(case, seed)
        zero = np.zeros_like(mass)
        b = _Box(params, box, {"pos": x, "vel": [zero] * 3, "B": [zero] * 3, "mass": mass, "h": h, "u": zero,
                               "psi": zero, "density": zero}, np.full(case["n"], abi.ROLES_DEFAULT, np.int64), dev)
        b.density()
        return {"rho": b.rho.cpu().numpy()}
    params, boxes, species = _inputs(case, seed)
    ids = sorted(species)
    every = abi.Species.concat([species[s] for s in ids])
    sid = np.concatenate([np.full(species[s].n, s) for s in ids])
    roles = np.array([abi.SPECIES_ROLES[s] for s in range(3)], dtype=np.int64)[sid]
    at = {c: getattr(every, c) for c in ("pos", "vel", "B", "mass", "h", "u", "psi", "density")}
    got = {c: np.zeros_like(a) for c, a in at.items()}
    got |= {"dvdt": np.zeros_like(every.pos), "dudt": np.zeros_like(every.u)}
    clock = np.zeros((2, len(boxes)))
    # the box's particles, found once: boxes of an ensemble are independent
    order = np.argsort(every.box_id, kind="stable")
    ends = np.searchsorted(every.box_id[order], np.arange(len(boxes) + 1))
    for k, box in enumerate(boxes):
        mine = order[ends[k]:ends[k + 1]]
        b = _Box(params, box, {c: a[..., mine] for c, a in at.items()}, roles[mine], dev)
        if case["kind"] == "stages":
            b.density()
            b.force()
            for q in range(3):
                got["dvdt"][q, mine] = b.a[q].cpu().numpy()
            got["dudt"][mine] = b.du.cpu().numpy()
        for _ in range(case.get("steps", 0)):
            b.step()
        for c, t in (("pos", b.x), ("vel", b.v), ("B", b.B)):
            for q in range(3):
                got[c][q, mine] = t[q].cpu().numpy()
        for c, t in (("h", b.h), ("u", b.u), ("psi", b.psi), ("density", b.rho)):
            got[c][mine] = t.cpu().numpy()
        clock[:, k] = b.time, b.dt
    out = {}
    for s in ids:
        cout = ["density", "dvdt", "dudt"] if case["kind"] == "stages" else _columns(params, s)[1]
        if cout:
            out[f"species{s}"] = {c: np.ascontiguousarray(got[c][..., sid == s]) for c in cout}
    if case["kind"] != "stages":
        out["clock"] = clock
    return out
