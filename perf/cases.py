"""The work a user of this library has it do, as timed cases.

Each case is one kind of program around the C ABI, at one size:

    fx        a block of steps of the FP32 / fixed-point form (push, zigzag
              current, CIC charge, tile sort), rho and J to the host after it
    host      the same with the field solver on the host: eb up and rho / J
              down every step
    em        the electromagnetic loop on the device (bfield, step, efield)
    es        the electrostatic loop on the device (step without the current,
              Poisson solve for any face type, E from phi)
    body      a plasma streaming past a charged box: inflow, photoemission,
              absorption with surface counts, background charge
    ensemble  many small independent runs replayed from one graph
    adjoint   gradients of a current probe through K steps
    dropin    the FP64 drop-in of the reference's records: grdcrt, psolve1,
              charge, the guard folds, spsort
    dropin_es the FP64 drop-in of its electrostatic loop (psolve2 + charge)
    init      the start of an FP64 run: load, positn, compaction of the
              particles that left through the open faces, spsort, charge

A pass goes on from where the pass before it ended, as a run does.  The
particles stay on the device (they do in a run; 64 bytes each would be most of
a pass): their state shows in every value of rho and J, in the energies, and
in the next pass.  Grid outputs are the nodes 0..n that a field solver takes:
the guard layers outside hold partial sums that depend on which side of a
periodic face a particle is stored.

`exact` is a 64-bit restatement in torch of the same equations from the same
seeds.  J of the FP32 form has none: the zigzag current jumps where an end
point crosses a cell face, so the few particles that rounding puts on the
other side of one decide its distance from 64 bits, not the sums.
"""
import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

from ctca_b200 import inputs
from ctca_b200.emses import FIELDS, PARTICLE_DTYPE, Batch, Emses, field_shape

USTEP = 2
TCS = 0.125          # c^2 dt^2 of the field step in internal units
RENV, RENE, RENB, RENQ, QM1 = 0.25, -0.0625, -0.25, -0.0625, -1.0  # inputs.units(dt = 0.5)
FX_KINDS = ("fx", "host", "em", "es")


# ---------------------------------------------------------------- cases
def listed():
    return [
        # the CPU-sized test case: small enough that launches count
        dict(name="fx_32cube", kind="fx", nx=32, ny=32, nz=32, ppc_e=16, ppc_i=16, ratio=100.0, walls="ppp", tile=8,
             steps=17, sort=4, graph=True),
        # odd sizes, partial tiles, reflecting walls in z, unequal species
        dict(name="fx_walls_ragged", kind="fx", nx=75, ny=42, nz=61, ppc_e=40, ppc_i=20, ratio=100.0, walls="ppw",
             tile=8, steps=8, sort=4, graph=False),
        # the headline particle step
        dict(name="fx_128cube", kind="fx", nx=128, ny=128, nz=128, ppc_e=64, ppc_i=64, ratio=1836.0, walls="ppp",
             tile=8, steps=8, sort=4, graph=False),
        # the same plasma at half the edge under a field solver on the host
        dict(name="host_64cube", kind="host", nx=64, ny=64, nz=64, ppc_e=64, ppc_i=64, ratio=1836.0, walls="ppp",
             tile=8, steps=8, sort=4, graph=False),
        dict(name="em_80x64x96", kind="em", nx=80, ny=64, nz=96, ppc_e=32, ppc_i=32, ratio=100.0, walls="ppp", tile=8,
             steps=8, sort=4, graph=False),
        # phi = 0 plates in z
        dict(name="es_plates_64x64x70", kind="es", nx=64, ny=64, nz=70, ppc_e=32, ppc_i=32, ratio=1836.0,
             walls="ppw", face=1, tile=8, steps=8, sort=4, graph=False),
        # the body workload at a quarter of its edge
        dict(name="body_64x64x128", kind="body", nx=64, ny=64, nz=128, ppc_e=24, ppc_i=24, ratio=100.0, walls="ppo",
             tile=8, steps=4, sort=4, graph=False),
        dict(name="ensemble_12", kind="ensemble", runs=12, side=48, ppc_e=64, ppc_i=64, ratio=100.0, steps=16, sort=4,
             tile=8),
        # the adjoint workload's plasma at half its edge
        dict(name="adjoint_32cube", kind="adjoint", nx=32, ny=32, nz=32, ppc_e=32, ppc_i=32, ratio=100.0, walls="ppp",
             tile=8, steps=16, sort=4, ckpt=8),
        dict(name="dropin_64cube", kind="dropin", nx=64, ny=64, nz=64, ppc_e=64, ppc_i=64, ratio=1836.0, walls="ppp",
             tile=8, steps=4, sort=4, dump=False),
        # the smallest run of the reference's own kind, records to the host (a restart file)
        dict(name="dropin_20x16x12", kind="dropin", nx=20, ny=16, nz=12, ppc_e=16, ppc_i=16, ratio=100.0, walls="pwp",
             tile=0, steps=4, sort=2, dump=True),
        dict(name="init_70x45x38", kind="init", nx=70, ny=45, nz=38, ppc_e=30, ppc_i=30, ratio=100.0, walls="ppo",
             tile=8),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kinds above over their ranges (grids of 12 to 128
    cells an axis, odd ones among them, 4 to 96 particles a cell)."""
    kind = rng.choice(["fx", "fx", "host", "em", "es", "body", "ensemble", "adjoint", "dropin", "dropin",
                       "dropin_es", "init"])
    ratio = rng.choice([25.0, 100.0, 1836.0])
    sort = rng.choice([2, 4, 4, 8])
    if kind == "ensemble":
        return dict(kind=kind, runs=rng.randint(4, 16), side=rng.choice([24, 32, 48]), ppc_e=rng.randint(16, 64),
                    ppc_i=rng.randint(16, 64), ratio=ratio, steps=16, sort=rng.choice([2, 4]), tile=8)
    most = {"fx": 128, "host": 96, "em": 112, "es": 112, "body": 80, "adjoint": 40, "dropin": 64, "dropin_es": 72,
            "init": 80}[kind]
    n = [_size(rng, 12, most) for _ in range(3)]
    if kind == "body":
        n = [max(24, x) for x in n]
    # at most these particles a species
    cap = {"fx": 120e6, "adjoint": 1e6, "dropin": 12e6, "dropin_es": 12e6, "init": 12e6}.get(kind, 24e6)
    top = max(4, min(96, int(cap / (n[0] * n[1] * n[2]))))
    ppc = [_size(rng, 4, top) for _ in range(2)]
    c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], ppc_e=ppc[0], ppc_i=ppc[1], ratio=ratio, walls="ppp", tile=8)
    if kind in ("fx", "es", "dropin", "dropin_es"):
        c["walls"] = rng.choice(["ppp", "ppp", "ppw", "pwp", "wpw"])
    if kind in ("body", "init"):
        c["walls"] = "ppo"
    if kind == "es":
        c["face"] = rng.choice([1, 2])
    if kind == "init":
        return c
    if kind == "adjoint":
        c.update(steps=16, sort=4, ckpt=rng.choice([4, 8, 16]))
        return c
    if kind in ("dropin", "dropin_es"):
        c.update(steps=4, sort=rng.choice([2, 4]), dump=False, tile=rng.choice([0, 8]))
        return c
    graph = kind == "fx" and rng.random() < 0.4
    c.update(steps=2 * sort + 1 if graph else max(4, sort), sort=sort, graph=graph)
    return c


# ---------------------------------------------------------------- inputs
def _species(c):
    """[(ppc, qm, vth, drift)] in normalised units."""
    vz = -0.08 if c["kind"] == "body" else 0.0
    vx = 0.01 if c["kind"] in FX_KINDS else 0.0
    out = [(c["ppc_e"], -1.0, 0.05, (0.0, 0.0, vz)),
           (c["ppc_i"], 1.0 / c["ratio"], 0.05 / math.sqrt(c["ratio"]), (vx, 0.0, vz))]
    if c["kind"] == "body":
        out.append((0, -1.0, 0.01, (0.0, 0.0, 0.0)))  # photoelectrons
    return out


def _numbers(c):
    """Internal q, qm, vth, drift of each species, e0 and b0."""
    sp = _species(c)
    qe = -1.0 / sp[0][0]
    q = [qe * RENQ if qm < 0 else -qe * sp[0][0] / ppc * RENQ for ppc, qm, _, _ in sp]
    b0 = (0.05, 0.0, 0.1) if c["kind"] == "body" else (0.0, 0.0, 0.1)
    return dict(q=q, qm=[s[1] / QM1 for s in sp], vth=[s[2] * RENV for s in sp],
                drift=[tuple(d * RENV for d in s[3]) for s in sp], ppc=[s[0] for s in sp],
                e0=(1e-3 * RENE, 0.0, 0.0), b0=tuple(b * RENB for b in b0))


def _grid(c):
    return c["nx"], c["ny"], c["nz"]


def _bounds(c):
    """Particle and field boundary types per axis."""
    np_ = [{"p": 0, "w": 1, "o": 2}[w] for w in c["walls"]]
    return np_, [0 if p == 0 else 1 for p in np_]


def _plates(c):
    return [c.get("face", 0) if f else 0 for f in _bounds(c)[1]]


def _box(c):
    n, b = _grid(c), (max(2, c["nx"] // 8), max(2, c["ny"] // 8), max(2, c["nz"] // 32))
    lo = [(n[d] - b[d]) // 2 for d in range(3)]
    return lo, [lo[d] + b[d] for d in range(3)]


def _config(c):
    num, (npb, nfb) = _numbers(c), _bounds(c)
    sp = [inputs.Species(ppc, qm, vth, drift, tuple(npb)) for ppc, qm, vth, drift in _species(c)]
    case = inputs.Case(n=_grid(c), species=sp, b0=tuple(b / RENB for b in num["b0"]),
                       e0=tuple(e / RENE for e in num["e0"]), nfbnd=tuple(nfb), sort_tile=(c["tile"],) * 3)
    cells = c["nx"] * c["ny"] * c["nz"]
    capacity = [max(1, cells * s.ppc) for s in sp]
    if c["kind"] == "body":  # room for the particles a long run injects
        lo, hi = _box(c)
        case.bodies = [dict(geotype=0, ncond=1, xlpc=float(lo[0]), xupc=float(hi[0]), ylpc=float(lo[1]),
                            yupc=float(hi[1]), zlpc=float(lo[2]), zupc=float(hi[2]), sqdscaled=1.0)]
        capacity = [3 * x + (8 << 20) for x in capacity[:2]] + [8 << 20]
    cfg = inputs.make_config(case, capacity)
    cfg.flags = 1 if c["kind"] in FX_KINDS + ("body",) else 0  # FP32-only where no FP64 record is used
    return cfg


def _plasma(c, cfg, seed):
    from ctca_b200.emses import Plasma
    pl, num = Plasma(), _numbers(c)
    for i in range(cfg.nspec):
        pl.ppc[i], pl.vth[i] = num["ppc"][i], num["vth"][i]
        for d in range(3):
            pl.vdrift[i][d] = num["drift"][i][d]
    pl.seed = seed
    return pl


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _eb(c, seed):
    """eb (6, -1:n+1 per axis) as (nz+3, ny+3, nx+3, 6): four E and four
    transverse B modes of amplitude 1e-3, periodic guards."""
    n, dev, rng = _grid(c), _dev(), np.random.default_rng([seed, 7])
    ax = [torch.arange(-1, n[d] + 2, device=dev, dtype=torch.float64) % n[d] for d in range(3)]
    out = torch.zeros((n[2] + 3, n[1] + 3, n[0] + 3, 6), device=dev, dtype=torch.float64)
    h = 0.5
    offs = ((h, 0, 0), (0, h, 0), (0, 0, h), (0, h, h), (h, 0, h), (h, h, 0))
    for kind in range(2):
        for _ in range(4):
            m = rng.integers(-3, 4, 3)
            m[rng.integers(3)] = rng.integers(1, 4)
            k = 2 * math.pi * m / np.array(n, dtype=float)
            pol = rng.normal(size=3)
            if kind == 1:
                pol -= pol.dot(k) / k.dot(k) * k
            pol *= 1e-3 / np.linalg.norm(pol) * (RENE, RENB)[kind]
            ph = rng.uniform(0, 2 * math.pi)
            for d in range(3):
                o = offs[3 * kind + d]
                arg = [float(k[a]) * (ax[a] + o[a]) for a in range(3)]
                out[..., 3 * kind + d] += float(pol[d]) * torch.cos(
                    arg[2][:, None, None] + arg[1][None, :, None] + arg[0][None, None, :] + ph)
    return out


class State:
    """What the user's program holds: the runs, its pinned host arrays."""

    def __init__(self, c):
        self.c, self.runs, self.bufs, self.batch = c, [], {}, None

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for g in self.runs:
            g.close()


def _pinned(count, dtype=torch.float64):
    return torch.empty(count, dtype=dtype, pin_memory=True)


def _open(s, c, seed, key=0):
    g = Emses(_config(c))
    s.runs.append(g)
    eb = _eb(c, seed).cpu().numpy()
    g.upload_field("eb", eb)
    names = {"em": ("eb", "rho"), "es": ("phi", "rho"), "dropin_es": ("rho",), "init": ("rho",)}.get(
        c["kind"], ("rho", "aj"))
    for name in names:
        s.bufs[name, key] = _pinned(g.field_size(name)).numpy()
    pl = _plasma(c, g.cfg, seed)
    if g.cfg.flags:
        g.fx_load_plasma(pl)
    else:
        g.load_plasma(pl)
    return g, eb, pl


def _sub_cases(c):
    """The runs of an ensemble: sides and particles a cell up to the case's."""
    out = []
    for r in range(c["runs"]):
        side = (16, 24, c["side"])[r % 3] if c["side"] > 24 else (16, c["side"])[r % 2]
        out.append(dict(kind="fx", nx=side, ny=side, nz=side, ppc_e=max(4, c["ppc_e"] - 3 * r),
                        ppc_i=max(4, c["ppc_i"] - 2 * r), ratio=c["ratio"], walls="ppp", tile=c["tile"],
                        steps=c["steps"], sort=c["sort"], graph=True))
    return out


def _probe(c):
    n = _grid(c)
    return [x // 2 - 2 for x in n], [x // 2 + 2 for x in n]


def prepare(case, seed):
    c = dict(case)
    s = State(c)
    if c["kind"] == "ensemble":
        for r, sub in enumerate(_sub_cases(c)):
            _open(s, sub, seed + 1000 * r, r)
        s.batch = Batch(s.runs, USTEP, 2 * c["sort"], [c["sort"]] * c["runs"])
        return s
    g, eb, pl = _open(s, c, seed)
    s.plasma, s.step = pl, 0
    if c["kind"] == "host":
        s.eb = _pinned(eb.size).numpy()
        s.eb[:] = eb.reshape(-1)
    if c["kind"] == "adjoint":
        s.n = (c["ppc_e"] + c["ppc_i"]) * c["nx"] * c["ny"] * c["nz"]
        s.gv = _pinned((s.n, 3)).numpy()
    if c.get("dump"):
        n = (c["ppc_e"] + c["ppc_i"]) * c["nx"] * c["ny"] * c["nz"]
        s.records = _pinned(n * PARTICLE_DTYPE.itemsize, torch.uint8).numpy().view(PARTICLE_DTYPE)
    if c["kind"] == "body":
        rng, num = np.random.default_rng([seed, 9]), _numbers(c)
        npr = 4096

        def flux(vd, vt):  # speeds through a face, |v| f(v)
            x = np.abs(rng.normal(vd, vt, 16 * npr))
            return np.sort(rng.choice(x, npr, p=x / x.sum()))

        s.tables = []
        for i in range(2):
            vt, vd = num["vth"][i], num["drift"][i][2]
            s.tables.append((-flux(vd, vt), rng.normal(0, vt, npr), rng.normal(0, vt, npr)))
        s.emit = (num["vth"][2] * np.sqrt(-2 * np.log(1 - rng.random(npr))), rng.normal(0, num["vth"][2], npr))
    return s


# ---------------------------------------------------------------- passes
def _inner(s, name, key=0):
    """Nodes 0..n of a downloaded field."""
    g = s.runs[key]
    a = s.bufs[name, key].reshape(field_shape(g.cfg, name))
    lo = 4 if name == "aj" else 1
    n = g.cfg
    return a[lo:lo + n.nz + 1, lo:lo + n.ny + 1, lo:lo + n.nx + 1]


def _down(s, *names, key=0):
    g = s.runs[key]
    for name in names:
        g._check(g.lib.emsesg_download_field(g.h, FIELDS[name], s.bufs[name, key].ctypes.data))
    return {name: _inner(s, name, key) for name in names}


def _run_body(s, g, c):
    lo, hi = _box(c)
    nemit = max(16, c["nx"] * c["ny"] // 64)
    nflow = int(0.08 * 0.5 * c["nx"] * c["ny"] * c["ppc_e"])
    for k in range(c["steps"]):
        for i in range(2):
            vn, va, vb = s.tables[i]
            g.fx_inflow_z(i + 1, False, nflow, vn, va, vb, 2.0, 5, 10 + i, s.step * nflow)
        g.fx_emit(3, 1, float(hi[0]), (lo[1], hi[1]), (lo[2], hi[2]), nemit, *s.emit, 5, 1, s.step * nemit)
        g.fx_step(USTEP, (k + 1) % c["sort"] == 0)
        g.fx_background()
        s.step += 1
    return dict(_down(s, "rho", "aj"), surface=g.fx_surface(), energy=g.fx_energy())


def run(state):
    s, c = state, state.c
    g, kind = s.runs[0], c["kind"]
    if kind == "ensemble":
        s.batch.launch(c["steps"] // (2 * c["sort"]))
        return [_down(s, "rho", "aj", key=r) for r in range(c["runs"])]
    if kind == "body":
        return _run_body(s, g, c)
    sorts = [(k + 1) % c["sort"] == 0 for k in range(c["steps"])] if "steps" in c else []
    if kind == "fx":
        if c["graph"]:
            g.fx_run(USTEP, c["steps"] - 1, c["sort"], True)
        else:
            for do_sort in sorts[:-1]:
                g.fx_step(USTEP, do_sort)
        g.fx_step_download(USTEP, False if c["graph"] else sorts[-1], s.bufs["rho", 0], s.bufs["aj", 0])
        return dict(rho=_inner(s, "rho"), aj=_inner(s, "aj"), energy=g.fx_energy())
    if kind == "host":
        for do_sort in sorts:
            g.upload_eb_async(s.eb)
            g.fx_step_download(USTEP, do_sort, s.bufs["rho", 0], s.bufs["aj", 0])
        return dict(rho=_inner(s, "rho"), aj=_inner(s, "aj"), energy=g.fx_energy())
    if kind == "em":
        for do_sort in sorts:
            g.fx_em_step(USTEP, do_sort, TCS)
        return dict(_down(s, "eb", "rho"), energy=g.fx_energy())
    if kind == "es":
        for do_sort in sorts:
            g.fx_step_es(USTEP, do_sort)
            g.esfield(1, check=False, mtd_vbnd=_plates(c))
        return dict(_down(s, "phi", "rho"), energy=g.fx_energy())
    if kind == "adjoint":
        g.fx_load()
        lo, hi = _probe(c)
        loss, gE, gB, g0, gv = g.fx_adjoint(c["steps"], USTEP, c["ckpt"], c["sort"], lo, hi, s.n, gv_out=s.gv)
        return dict(loss=float(loss), gE=gE, gB=gB, g0=g0, gv=gv)
    if kind == "init":
        g.load_plasma(s.plasma)
        g.positn(1, USTEP)
        counts = g.compact(1)
        g.spsort(1)
        g.charge(1, 0)
        g.reduce_rho("rho")
        return dict(_down(s, "rho"), counts=counts, energy=g.energy())
    # the FP64 drop-in, in the order of the reference's main loops
    for do_sort in sorts:
        g.grdcrt(1)
        if kind == "dropin":
            g.zero_field("aj")
            g.psolve1(1, USTEP, 0)
            g.reduce_aj()
        else:
            g.psolve2(1, USTEP)
        if do_sort:
            g.spsort(1)
        g.charge(1, 0)
        g.reduce_rho("rho")
    out = dict(_down(s, "rho"), energy=g.energy())
    if kind == "dropin":
        out.update(_down(s, "aj"))
    if c.get("dump"):
        tp = (ctypes.c_int64 * 10)()
        g._check(g.lib.emsesg_download_particles(g.h, 1, s.records.ctypes.data, tp))
        out["records"] = s.records.view(np.float64).reshape(-1, 8)[:, :6]
        out["marks"] = s.records.view(np.int32).reshape(-1, 16)[:, 12:]
    return out


# ---------------------------------------------------------------- work
def work(case):
    """Bytes: every particle record read and written once a step (28 bytes in
    the FP32 form, 64 in the FP64 one) and once a sort, the grid arrays a step
    reads and writes, the outputs; charge alone reads the 64-byte records once
    more.  Flops: about 250 a particle-step (gather 96, Boris and move 60,
    zigzag and charge 94), without the current 170."""
    c = dict(case)
    if c["kind"] == "ensemble":
        w = [work(x) for x in _sub_cases(c)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    cells = c["nx"] * c["ny"] * c["nz"]
    n = (c["ppc_e"] + c["ppc_i"]) * cells
    if c["kind"] == "init":  # written by the load, moved, compacted and sorted once each, read by charge
        return {"bytes": 64.0 * n * 7 + 16.0 * cells, "flops": 150.0 * n}
    steps, sorts = c["steps"], c["steps"] // c["sort"]
    f64 = c["kind"].startswith("dropin")
    rec = 64 if f64 else 28
    b = n * (2.0 * rec * (steps + sorts) + (64.0 * steps if f64 else 0.0))
    b += cells * steps * (48.0 + 8.0 + (24.0 if c["kind"] not in ("es", "dropin_es") else 8.0))
    if c["kind"] == "em":
        b += cells * steps * 96.0
    if c["kind"] == "adjoint":  # forward, recompute, and 24 bytes of adjoint state read and written a step
        b += n * steps * (56.0 + 28.0 + 48.0) + cells * 48.0
    flops = n * steps * (170.0 if c["kind"] in ("es", "dropin_es") else 250.0) * (4 if c["kind"] == "adjoint" else 1)
    return {"bytes": b, "flops": flops}


def tolerance(case):
    k = case["kind"]
    if k in ("dropin", "dropin_es", "init"):
        return {"rel": 1e-11, "max": 1e-9}
    # a particle that rounding puts on the other side of a face moves current
    # between nodes: a few of them set the error of J, and of the fields that
    # follow from it (four times the 2e-5 and 2.5e-3 seen over drawn cases)
    return {"rel": 8e-5, "max": 1e-2, "differ": 1e-2}


# ---------------------------------------------------------------- 64 bits
_M = (1 << 64) - 1


def _s64(x):
    x &= _M
    return x - (1 << 64) if x >> 63 else x


def _mix_int(z):
    z = (z + 0x9E3779B97F4A7C15) & _M
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _M
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M
    return z ^ (z >> 31)


def _shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _mix(z):
    z = z + _s64(0x9E3779B97F4A7C15)
    z = (z ^ _shr(z, 30)) * _s64(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _s64(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _uniform(seed, stream, index):
    a = _mix_int(seed ^ _mix_int((stream + 0x632BE59BD9B4E019) & _M))
    b = _mix((index * _s64(0xD1B54A32D192ED03)) ^ _s64(a))
    return _shr(b, 11).to(torch.float64) * (1.0 / 9007199254740992.0)


def _particles(c, seed, sp, m0, m1):
    """Particles m0..m1-1 of species sp of the seeded plasma: x, v [n, 3]."""
    num, n = _numbers(c), _grid(c)
    m = torch.arange(m0, m1, device=_dev(), dtype=torch.int64)
    u = [_uniform(seed, 1000 + sp, m * 8 + k) for k in range(7)]
    cell = m // num["ppc"][sp]
    x = torch.stack((cell % n[0] + u[0], cell // n[0] % n[1] + u[1], cell // (n[0] * n[1]) + u[2]), 1)
    r1, r2 = torch.sqrt(-2 * torch.log(1 - u[3])), torch.sqrt(-2 * torch.log(1 - u[5]))
    t, d, tau = num["vth"][sp], num["drift"][sp], 2 * math.pi
    v = torch.stack((t * r1 * torch.cos(tau * u[4]) + d[0], t * r1 * torch.sin(tau * u[4]) + d[1],
                     t * r2 * torch.cos(tau * u[6]) + d[2]), 1)
    return x, v


def _nodes(c, eb):
    """E and B on the nodes 0..n: (nz+1, ny+1, nx+1, 6)."""
    num, n = _numbers(c), _grid(c)

    def at(comp, di, dj, dk):
        return eb[1 - dk:2 - dk + n[2], 1 - dj:2 - dj + n[1], 1 - di:2 - di + n[0], comp]

    out = [0.5 * (at(0, 0, 0, 0) + at(0, 1, 0, 0)), 0.5 * (at(1, 0, 0, 0) + at(1, 0, 1, 0)),
           0.5 * (at(2, 0, 0, 0) + at(2, 0, 0, 1)),
           0.25 * (at(3, 0, 0, 0) + at(3, 0, 1, 0) + at(3, 0, 0, 1) + at(3, 0, 1, 1)),
           0.25 * (at(4, 0, 0, 0) + at(4, 1, 0, 0) + at(4, 0, 0, 1) + at(4, 1, 0, 1)),
           0.25 * (at(5, 0, 0, 0) + at(5, 1, 0, 0) + at(5, 0, 1, 0) + at(5, 1, 1, 0))]
    add = num["e0"] + num["b0"]
    return torch.stack([o + a for o, a in zip(out, add)], -1)


def _kick(n, nodes, x, v, qm):
    cell = [torch.clamp(torch.floor(x[:, d]), 0, n[d]).to(torch.int64) for d in range(3)]
    f = [x[:, d] - cell[d] for d in range(3)]
    flat, sy, sz = nodes.reshape(-1, 6), n[0] + 1, (n[0] + 1) * (n[1] + 1)
    eb = 0
    for dk in range(2):
        for dj in range(2):
            for di in range(2):
                w = (f[0] if di else 1 - f[0]) * (f[1] if dj else 1 - f[1]) * (f[2] if dk else 1 - f[2])
                at = torch.clamp(cell[0] + di, max=n[0]) + sy * torch.clamp(cell[1] + dj, max=n[1]) + \
                    sz * torch.clamp(cell[2] + dk, max=n[2])
                eb = eb + flat[at] * w[:, None]
    e, b = eb[:, :3] * (qm * USTEP * 0.5), eb[:, 3:] * (qm * USTEP * 0.5)
    v = v + e
    s = 2.0 / (1.0 + (b * b).sum(1, keepdim=True))
    v = v + s * torch.linalg.cross(v + torch.linalg.cross(v, b), b)
    return v + e, cell


def _scatter(n, grid, at, value, pad):
    """grid[k + pad, j + pad, i + pad] += value at the nodes at = (i, j, k)."""
    ex, ey = n[0] + 1 + 2 * pad, n[1] + 1 + 2 * pad
    return grid.index_add(0, (at[0] + pad) + ex * ((at[1] + pad) + ey * (at[2] + pad)), value)


def _push(c, nodes, x, v, sp, current, only=None):
    """One step: new x, v and the raw current on the nodes -1..n+1 (three
    flat arrays, or component `only`)."""
    num, n, (npb, _) = _numbers(c), _grid(c), _bounds(c)
    v, ib = _kick(n, nodes, x, v, num["qm"][sp])
    a, ia, r, xs, vs = [], [], [], [], []
    for d in range(3):
        p = x[:, d] + v[:, d] * USTEP
        low, high, w = p < 0, p >= n[d], v[:, d]
        f = torch.clamp(torch.floor(p), -1, n[d]).to(torch.int64)
        mid = torch.where(ib[d] == f, (x[:, d] + p) * 0.5, torch.maximum(ib[d], f).to(p.dtype))
        if npb[d] == 0:
            a.append(p)
            ia.append(f)
            xs.append(torch.where(low, p + n[d], torch.where(high, p - n[d], p)))
        else:
            p = torch.where(low, -p, torch.where(high, 2 * n[d] - p, p))
            w = torch.where(low | high, -w, w)
            a.append(p)
            ia.append(torch.where(low, 0, torch.where(high, n[d] - 1, f)))
            xs.append(p)
        r.append(torch.where(low, 0.0, torch.where(high, float(n[d]), mid)))
        vs.append(w)
    J = None
    if current:
        J = [None] * 3
        for comp in range(3) if only is None else (only,):
            p, q = [d for d in range(3) if d != comp]
            flat = torch.zeros((n[0] + 3) * (n[1] + 3) * (n[2] + 3), device=x.device, dtype=x.dtype)
            for cell, s, e in ((ib, [x[:, d] for d in range(3)], r), (ia, r, a)):
                fl = (e[comp] - s[comp]) / USTEP
                u, w = (s[p] + e[p]) * 0.5 - cell[p], (s[q] + e[q]) * 0.5 - cell[q]
                for dp in range(2):
                    for dq in range(2):
                        at = list(cell)
                        at[p], at[q] = at[p] + dp, at[q] + dq
                        flat = _scatter(n, flat, at, fl * (u if dp else 1 - u) * (w if dq else 1 - w), 1)
            J[comp] = flat
    return torch.stack(xs, 1), torch.stack(vs, 1), J


def _charge(c, x, grid):
    n = _grid(c)
    cell = [torch.floor(x[:, d]).to(torch.int64) for d in range(3)]
    f = [x[:, d] - cell[d] for d in range(3)]
    for dk in range(2):
        for dj in range(2):
            for di in range(2):
                w = (f[0] if di else 1 - f[0]) * (f[1] if dj else 1 - f[1]) * (f[2] if dk else 1 - f[2])
                grid = _scatter(n, grid, (cell[0] + di, cell[1] + dj, cell[2] + dk), w, 1)
    return grid


def _fold(c, flat, comp=None):
    """Guard folds: raw values on -1..n+1 to the nodes 0..n."""
    n, (_, nfb) = _grid(c), _bounds(c)
    g = flat.reshape(n[2] + 3, n[1] + 3, n[0] + 3)
    for d in (2, 1, 0):
        a = [g.select(2 - d, m) for m in range(n[d] + 3)]  # a[m] holds node m - 1
        if nfb[d] == 0:
            raw = list(a)
            for m in range(3):
                a[m], a[n[d] + m] = raw[m] + raw[n[d] + m], raw[m] + raw[n[d] + m]
        elif comp == d:
            a[n[d] + 1] = -a[n[d]]
        else:
            a[1], a[n[d] + 1] = a[1] * 2, a[n[d] + 1] * 2
        g = torch.stack(a, 2 - d)
    return g[1:-1, 1:-1, 1:-1]


def _energy(c, v2):
    num, n = _numbers(c), _grid(c)
    return np.array([[0.5 * (num["q"][s] / num["qm"][s]) * float(t) / (n[0] * n[1] * n[2]) for t in row]
                     for s, row in enumerate(v2)])


def _solve(c, rho):
    """phi on the nodes 0..n: rho extended to a periodic array (oddly over
    phi = 0 faces, evenly over Neumann ones), divided by the eigenvalues."""
    n, t = _grid(c), _plates(c)
    r = rho
    for d in range(3):
        ax = 2 - d
        if t[d] == 0:
            r = r.narrow(ax, 0, n[d])
        else:
            inner = r.narrow(ax, 1, n[d] - 1)
            z = torch.zeros_like(r.narrow(ax, 0, 1))
            ends = (z, z) if t[d] == 1 else (r.narrow(ax, 0, 1), r.narrow(ax, n[d], 1))
            r = torch.cat((ends[0], inner, ends[1], (-1 if t[d] == 1 else 1) * inner.flip(ax)), ax)
    lam = 0
    for d in range(3):
        m = r.shape[2 - d]
        e = (2 * torch.sin(math.pi * torch.arange(m, device=r.device, dtype=r.dtype) / m)) ** 2
        lam = lam + e.reshape([-1 if a == 2 - d else 1 for a in range(3)])
    s = torch.fft.fftn(r)
    lam[0, 0, 0] = 1.0
    s = s / lam
    s[0, 0, 0] = 0.0
    p = torch.fft.ifftn(s).real
    for d in range(3):
        ax = 2 - d
        p = torch.cat((p, p.narrow(ax, 0, 1)), ax) if t[d] == 0 else p.narrow(ax, 0, n[d] + 1)
    return p


def _e_of_phi(c, phi, eb):
    """EX..EZ of eb from phi, the faces' normal components copied or negated."""
    n, t = _grid(c), _plates(c)
    eb = eb.clone()
    eb[..., :3] = 0.0
    for d in range(3):
        ax = 2 - d
        e = phi.narrow(ax, 0, n[d]) - phi.narrow(ax, 1, n[d])  # 0..n-1
        lo, hi = e.narrow(ax, n[d] - 1, 1), e.narrow(ax, 0, 1)  # -1 and n of a periodic axis
        if t[d]:
            sign = 1.0 if t[d] == 1 else -1.0
            lo, hi = sign * e.narrow(ax, 0, 1), sign * e.narrow(ax, n[d] - 1, 1)
        e = torch.cat((lo, e, hi), ax)
        sl = [slice(1, n[2] + 2), slice(1, n[1] + 2), slice(1, n[0] + 2)]
        sl[ax] = slice(0, n[d] + 2)
        eb[tuple(sl) + (d,)] = e
    return eb


def _guards(c, inner):
    """Periodic guards -1..n+1 around the nodes 0..n-1."""
    n = _grid(c)
    for d in range(3):
        at = torch.arange(-1, n[d] + 2, device=inner.device) % n[d]
        inner = inner.index_select(2 - d, at)
    return inner


def _loop(c, seed, all_species=True):
    """The states and the fields through the steps of the field loops, whose
    steps depend on each other's deposits, or of any drop-in block."""
    num, n, kind = _numbers(c), _grid(c), c["kind"]
    cells = n[0] * n[1] * n[2]
    parts = [_particles(c, seed, sp, 0, num["ppc"][sp] * cells) for sp in range(2)]
    eb = _eb(c, seed)
    size = (n[0] + 3) * (n[1] + 3) * (n[2] + 3)
    out = {}
    for _ in range(c["steps"]):
        if kind == "em":
            eb = _bfield(c, eb)
        nodes = _nodes(c, eb)
        rho, J = 0, [0, 0, 0]
        for sp in range(2):
            x, v, j = _push(c, nodes, *parts[sp], sp, kind in ("em", "dropin"))
            parts[sp] = (x, v)
            rho = rho + num["q"][sp] * _charge(c, x, torch.zeros(size, device=x.device, dtype=x.dtype))
            if j:
                J = [J[d] + num["q"][sp] * j[d] for d in range(3)]
        rho = _fold(c, rho)
        if kind in ("em", "dropin"):
            J = torch.stack([_fold(c, J[d], d) for d in range(3)], -1)
        if kind == "em":
            eb = _efield(c, _bfield(c, eb), J)
        if kind == "es":
            out["phi"] = _solve(c, rho)
            eb = _e_of_phi(c, out["phi"], eb)
            out["phi"] = out["phi"][..., None]
    out["rho"] = rho[..., None]
    if kind == "dropin":
        out["aj"] = J
    if kind == "em":
        out["eb"] = eb[1:-1, 1:-1, 1:-1]
    out["energy"] = _energy(c, [(v * v).sum(0) for _, v in parts])
    return out


def _bfield(c, eb):
    n = _grid(c)
    f = eb[1:n[2] + 1, 1:n[1] + 1, 1:n[0] + 1].clone()
    e = [f[..., d].clone() for d in range(3)]

    def up(a, d):
        return torch.roll(a, -1, 2 - d)

    f[..., 3] += up(e[1], 2) - e[1] - up(e[2], 1) + e[2]
    f[..., 4] += up(e[2], 0) - e[2] - up(e[0], 2) + e[0]
    f[..., 5] += up(e[0], 1) - e[0] - up(e[1], 0) + e[1]
    return _guards(c, f)


def _efield(c, eb, J):
    n = _grid(c)
    f = eb[1:n[2] + 1, 1:n[1] + 1, 1:n[0] + 1].clone()
    b = [f[..., 3 + d].clone() for d in range(3)]
    j = J[:n[2], :n[1], :n[0]]

    def dn(a, d):
        return a - torch.roll(a, 1, 2 - d)

    f[..., 0] += TCS * (dn(b[2], 1) - dn(b[1], 2)) - 2.0 * j[..., 0]
    f[..., 1] += TCS * (dn(b[0], 2) - dn(b[2], 0)) - 2.0 * j[..., 1]
    f[..., 2] += TCS * (dn(b[1], 0) - dn(b[0], 1)) - 2.0 * j[..., 2]
    return _guards(c, f)


def _block(c, seed):
    """Steps in a static field: chunk by chunk through all of them, the
    charge of the last one."""
    num, n = _numbers(c), _grid(c)
    cells, chunk = n[0] * n[1] * n[2], 1 << 23
    nodes = _nodes(c, _eb(c, seed))
    rho, v2 = 0, []
    for sp in range(2):
        grid = torch.zeros((n[0] + 3) * (n[1] + 3) * (n[2] + 3), device=_dev(), dtype=torch.float64)
        s = torch.zeros(3, device=_dev(), dtype=torch.float64)
        for m in range(0, num["ppc"][sp] * cells, chunk):
            x, v = _particles(c, seed, sp, m, min(m + chunk, num["ppc"][sp] * cells))
            for _ in range(c["steps"]):
                x, v, _ = _push(c, nodes, x, v, sp, False)
            grid = _charge(c, x, grid)
            s += (v * v).sum(0)
        rho = rho + num["q"][sp] * grid
        v2.append(s)
    return dict(rho=_fold(c, rho)[..., None], aj=None, energy=_energy(c, v2))


def _sorted(c, x):
    """The canonical order: tile-major cell key, stable."""
    n = _grid(c)
    t = [min(c["tile"], n[d]) if c["tile"] else n[d] for d in range(3)]
    nt = [(n[d] + t[d] - 1) // t[d] for d in range(3)]
    i = [torch.clamp(torch.floor(x[:, d]), 0, n[d] - 1).to(torch.int64) for d in range(3)]
    key = (i[0] // t[0] + nt[0] * (i[1] // t[1] + nt[1] * (i[2] // t[2]))) * (t[0] * t[1] * t[2])
    key = key + i[0] % t[0] + t[0] * (i[1] % t[1] + t[1] * (i[2] % t[2]))
    return torch.sort(key, stable=True).indices


def _exact_init(c, seed):
    num, n = _numbers(c), _grid(c)
    rho, counts, v2 = 0, [], []
    for sp in range(2):
        x, v = _particles(c, seed, sp, 0, num["ppc"][sp] * n[0] * n[1] * n[2])
        x = x + v * USTEP
        live = (x[:, 2] >= 0) & (x[:, 2] < n[2])
        x, v = x[live], v[live]
        for d in range(2):
            x[:, d] = torch.where(x[:, d] < 0, x[:, d] + n[d], torch.where(x[:, d] >= n[d], x[:, d] - n[d], x[:, d]))
        x = torch.minimum(x, torch.tensor(n, device=x.device) * (1 - 1e-16))
        rho = rho + num["q"][sp] * _charge(c, x, torch.zeros((n[0] + 3) * (n[1] + 3) * (n[2] + 3), device=x.device,
                                                             dtype=x.dtype))
        counts.append(len(x))
        v2.append((v * v).sum(0))
    return dict(rho=_fold(c, rho)[..., None], counts=np.array(counts), energy=_energy(c, v2))


def _exact_adjoint(c, seed):
    num, n = _numbers(c), _grid(c)
    lo, hi = _probe(c)
    cells = n[0] * n[1] * n[2]
    inner = _nodes(c, _eb(c, seed))[:-1, :-1, :-1].contiguous().requires_grad_(True)
    parts, v0 = [], []
    for sp in range(2):
        x, v = _particles(c, seed, sp, 0, num["ppc"][sp] * cells)
        o = _sorted(c, x)
        v0.append(v[o].requires_grad_(True))
        parts.append((x[o], v0[-1]))

    def step(nodes, x0, w0, x1, w1):
        out, J = [], 0
        for sp, (x, w) in enumerate(((x0, w0), (x1, w1))):
            x, w, j = _push(c, nodes, x, w, sp, True, only=0)
            out += [x, w]
            J = J + num["q"][sp] * j[0]
        J = _fold(c, J, 0)[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]]
        return (*out, (J * J).sum())

    nodes = inner
    for d in range(3):
        nodes = torch.cat((nodes, nodes.narrow(2 - d, 0, 1)), 2 - d)
    s, loss = [*parts[0], *parts[1]], 0
    for _ in range(c["steps"]):
        *s, part = torch.utils.checkpoint.checkpoint(step, nodes, *s, use_reentrant=False)
        loss = loss + part
    loss.backward()
    g = inner.grad.reshape(-1, 6)
    return dict(loss=float(loss.detach()), gE=g[:, :3], gB=g[:, 3:], g0=g.sum(0), gv=torch.cat([v.grad for v in v0]))


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "ensemble":
        return [{"rho": _block(sub, seed + 1000 * r)["rho"], "aj": None} for r, sub in enumerate(_sub_cases(c))]
    if c["kind"] == "body":  # its injected records come from the device's own draws
        return None
    if c["kind"] == "init":
        return _exact_init(c, seed)
    if c["kind"] == "adjoint":
        return _exact_adjoint(c, seed)
    if c["kind"] in ("fx", "host"):
        return _block(c, seed)
    out = _loop(c, seed)
    if c.get("dump"):
        out.update(records=None, marks=None)
    return out
