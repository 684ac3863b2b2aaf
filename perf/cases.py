"""The work a user of this library has it do, as cases that can be timed and compared.

Six kinds of work, each through the library's public entry points (the classes of
`tpic_b200` or the C ABI of include/tpicb200.h, as an external caller binds it):

  cycle     whole ECSIM cycles of a shipped deck (Simulation.run), at the deck's size or another
  push      the particle stage: implicit mover, then the stable sort of the moved records
  deposit   the moment stage: clear, implicit current and mass matrix of two species, periodic fold
  solve     the field solve (GMRES on the mass-matrix-augmented Maxwell system)
  backward  the adjoint of two cycles: energy gradient, then two cycle backwards on their tapes
  moments   the snapshot's output moments (rho, J, P_ij) of two species

`exact` restates each kind in plain torch FP64 on periodic unique-node arrays.
"""
import ctypes as C
import math
from pathlib import Path

import numpy as np
import torch

from tpic_b200 import _lib, deck
from tpic_b200.adjoint import AdjointBuffers, TapeBuffers
from tpic_b200.plasma import Case, GridSpec, SpeciesSpec
from tpic_b200.simulation import Simulation

DEV = "cuda"
F64 = torch.float64
DECKS = Path(__file__).resolve().parent.parent / "tpic_b200" / "decks"

# Cell size, time step, electron q/m and thermal speeds of the shipped decks, by dimension: the stage
# kinds use the deck whose grid they look like (3-D thermal plasma, 2-D sheet/anisotropy, 1-D beams).
PLASMA = {3: dict(d=0.15625, dt=0.15, qe=-64.0, ve=0.045, vi=0.0056, b=(0.0, 0.0, 0.0195)),
          2: dict(d=0.1, dt=0.125, qe=-100.0, ve=0.05, vi=0.003, b=(0.0195, 0.0, 0.0)),
          1: dict(d=0.006135923151542565, dt=0.1, qe=-1.0, ve=0.01, vi=0.0, b=(0.0, 0.0, 0.0))}


def listed():
    return [
        # The headline workload: 3-D thermal plasma, 268M records, BF16x3 assembly, tiled mass (bench.py's choice).
        dict(name="cycle 128^3 bf16x3", kind="cycle", deck="uniform3d_128", nx=128, ny=128, nz=128, npx=4, npy=4, npz=4,
             precision="mixed", mass="bf16x3", layout="tiled", smooth=0),
        # A 2-D production run: Harris sheets, four species, TF32 assembly.
        dict(name="cycle harris 256x128 tf32", kind="cycle", deck="harris2d_256x128", nx=256, ny=128, nz=1, npx=10, npy=10,
             npz=1, precision="mixed", mass="tf32", layout="tiled", smooth=0),
        # A 1-D run, the default scalar assembly and the driver's layout: many GMRES steps on little data.
        dict(name="cycle two-stream 1024", kind="cycle", deck="twostream1d_1024", nx=1024, ny=1, nz=1, npx=128, npy=1,
             npz=1, precision="mixed", mass="scalar", layout="stencil-major", smooth=0),
        # The smallest run, all defaults of Simulation (FP64, scalar): what a first user and the tests run.
        dict(name="cycle 16^3 double", kind="cycle", deck="uniform3d_16", nx=16, ny=16, nz=16, npx=3, npy=3, npz=3,
             precision="double", mass="scalar", layout="stencil-major", smooth=0),
        # The default assembly on an odd 3-D grid, ragged cells.
        dict(name="deposit scalar 61x47x53", kind="deposit", nx=61, ny=47, nz=53, ppc=27, precision="mixed", mass="scalar",
             layout="stencil-major"),
        # The double-precision assembly of an accurate 3-D run.
        dict(name="deposit moments-f64 64^3", kind="deposit", nx=64, ny=64, nz=64, ppc=64, precision="double",
             mass="moments-f64", layout="stencil-major"),
        # The particle stage of a mid-size 3-D species.
        dict(name="push mixed 80x64x48", kind="push", nx=80, ny=64, nz=48, ppc=64, precision="mixed"),
        # The particle stage of a small 2-D species in double.
        dict(name="push double 127x65", kind="push", nx=127, ny=65, nz=1, ppc=100, precision="double"),
        # Field solve with the default six smoothing passes on the 2-D grid.
        dict(name="solve smoothed 256x128", kind="solve", nx=256, ny=128, nz=1, precision="mixed", layout="stencil-major",
             smooth=6, alpha=0.5, op=0),
        # Field solve of an accurate 3-D run.
        dict(name="solve double 64^3", kind="solve", nx=64, ny=64, nz=64, precision="double", layout="stencil-major",
             smooth=0, alpha=1.0, op=0),
        # The gradient direction: two cycle backwards of a 2-D run.
        dict(name="backward 192x160", kind="backward", nx=192, ny=160, nz=1, ppc=64, precision="mixed", mass="bf16x3",
             layout="stencil-major"),
        # A field snapshot of a 3-D run.
        dict(name="moments 64^3", kind="moments", nx=64, ny=64, nz=64, ppc=64, precision="mixed"),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def grid(dim, small, large):
        if dim == 3:
            n = (log(small, large), log(small, large), log(small, large))
        elif dim == 2:
            n = (log(4 * small, 6 * large), log(4 * small, 4 * large), 1)
        else:
            n = (log(128, 1024), 1, 1)
        return dict(nx=n[0], ny=n[1], nz=n[2])

    kind = rng.choice(["cycle", "cycle", "push", "deposit", "deposit", "solve", "solve", "backward", "moments"])
    dim = rng.choice([3, 3, 2, 2, 1] if kind in ("cycle", "solve") else [3, 3, 2])
    layout = rng.choice(["stencil-major", "stencil-major", "tiled", "records"])
    precision = rng.choice(["mixed", "mixed", "double"])
    mass = rng.choice(["scalar", "scalar", "tf32", "bf16x3"] if precision == "mixed" else
                      ["scalar", "moments-f64", "scalar-f64"])
    ppc = log(16, 100)
    if kind == "cycle":
        g = grid(dim, 12, 72)
        name = {3: rng.choice(["uniform3d_16", "uniform3d_128"]), 2: rng.choice(["harris2d_256x128", "anisotropy2d_512"]),
                1: "twostream1d_1024"}[dim]
        a = {3: (rng.randint(2, 4), rng.randint(2, 4), rng.randint(2, 4)), 2: (rng.randint(4, 10), rng.randint(4, 10), 1),
             1: (log(32, 128), 1, 1)}[dim]
        return dict(kind=kind, deck=name, **g, npx=a[0], npy=a[1], npz=a[2], precision=precision, mass=mass, layout=layout,
                    smooth=rng.choice([0, 0, 0, 6]) if dim > 1 else 0)
    if kind == "push":
        return dict(kind=kind, **grid(dim, 12, 80), ppc=ppc, precision=precision)
    if kind == "deposit":
        return dict(kind=kind, **grid(dim, 12, 72), ppc=ppc, precision=precision, mass=mass, layout=layout)
    if kind == "solve":
        smooth = rng.choice([0, 0, 6]) if dim > 1 else 0
        return dict(kind=kind, **grid(dim, 12, 80), precision=precision, layout=layout, smooth=smooth,
                    alpha=rng.choice([0.5, 0.75]) if smooth else 1.0, op=rng.choice([0, 0, 1]) if smooth else 0)
    if kind == "backward":
        return dict(kind=kind, **grid(dim, 10, 40), ppc=min(ppc, 64), precision=precision, mass=mass, layout=layout)
    return dict(kind=kind, **grid(dim, 12, 72), ppc=ppc, precision=precision)


# -- inputs ------------------------------------------------------------------------------------------


def dimension(case):
    return sum(n > 1 for n in (case["nx"], case["ny"], case["nz"])) or 1


def plasma(case):
    return PLASMA[dimension(case)]


def grid_of(case):
    p = plasma(case)
    n = (case["nx"], case["ny"], case["nz"])
    return GridSpec(*n, *(m * p["d"] for m in n))


def stage_simulation(case, species, **more):
    """A Simulation that owns the context and buffers of a stage case; the records and fields are ours."""
    p = plasma(case)
    c = Case(grid_of(case), species, dt=p["dt"], theta=0.5, gmres_tol=1e-8)
    # The 1-D grid's light-crossing number needs more GMRES steps than the default hundred.
    return Simulation(c, precision=case["precision"], mass_kind=case.get("mass", "scalar"),
                      mass_layout=case.get("layout", "stencil-major"), generate=False, gmres_max_iterations=300, **more)


def wrap_index(n, first, count):
    return (torch.arange(count, device=DEV) + first) % n


def spread(case, unique, nodes):
    """A unique-node (or cell) field [3, nz, ny, nx] in the stored layout with its periodic copies."""
    extra = 3 if nodes else 2
    iz, iy, ix = (wrap_index(n, -1, n + extra) for n in (case["nz"], case["ny"], case["nx"]))
    return unique[:, iz][:, :, iy][:, :, :, ix].reshape(-1).contiguous()


def random_fields(case, g, e_amplitude):
    """Unique-node E and cell B: noise at the amplitude of a thermal run over the background field."""
    p = plasma(case)
    shape = (3, case["nz"], case["ny"], case["nx"])
    e = e_amplitude * torch.randn(shape, generator=g, device=DEV, dtype=F64)
    b = 5e-4 * torch.randn(shape, generator=g, device=DEV, dtype=F64)
    b -= b.mean((1, 2, 3), keepdim=True)
    return e, b + torch.tensor(p["b"], device=DEV, dtype=F64).view(3, 1, 1, 1)


def random_records(case, g, ppc, qom, vth, ids=False, base=None):
    """Records of one species sorted by cell with the Poisson occupancy a run has after its first cycles."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz * ppc
    ext = torch.tensor([nx, ny, nz], device=DEV, dtype=F64).view(3, 1)
    if base is None:
        pos = torch.rand((3, n), generator=g, device=DEV, dtype=F64) * ext
        vel = vth * torch.randn((3, n), generator=g, device=DEV, dtype=F64)
        ident = None
    else:  # the same records some cycles later: moved by about a cell
        ident, pos, vel = base["id"], base["pos"] + 0.7 * torch.randn((3, n), generator=g, device=DEV, dtype=F64), base["vel"]
        pos = torch.remainder(pos, ext)
    pos = torch.minimum(pos, ext * (1 - 1e-12))
    cell = pos.floor()
    lin = (cell[0] + nx * (cell[1] + ny * cell[2])).to(torch.int64)
    lin, order = torch.sort(lin, stable=True)
    pos, vel, cell = pos[:, order], vel[:, order], cell[:, order]
    frac = torch.clamp(pos - cell, 0.0, 1 - 1e-12)
    c = cell.to(torch.int64)
    key = ((c[0] + 2) + (nx + 4) * ((c[1] + 2) + (ny + 4) * (c[2] + 2))).to(torch.int32)
    d = plasma(case)["d"]
    q = torch.full((n,), math.copysign(d**3 / ppc / (4 * math.pi), qom), device=DEV, dtype=F64)
    vdt = F64 if case["precision"] == "double" else torch.float32
    r = dict(rx=frac[0].contiguous(), ry=frac[1].contiguous(), rz=frac[2].contiguous(), u=vel[0].to(vdt), v=vel[1].to(vdt),
             w=vel[2].to(vdt), q=q, cell=key)
    bins = (nx + 4) * (ny + 4) * (nz + 4)
    counts = torch.bincount(key.long(), minlength=bins).to(torch.int32)
    offsets = torch.zeros(bins + 1, dtype=torch.int32, device=DEV)
    offsets[1:] = torch.cumsum(counts, 0)
    out = dict(rec=r, counts=counts, offsets=offsets, n=n, qom=qom)
    if ids:
        r["id"] = torch.arange(n, device=DEV) if ident is None else ident[order]
        out.update(id=r["id"], pos=pos, vel=vel)
    return out


def species_of(case, ids=False):
    p = plasma(case)
    ppc = case["ppc"]
    return [SpeciesSpec(qom=p["qe"], npcel=(ppc, 1, 1)), SpeciesSpec(qom=1.0, npcel=(ppc, 1, 1))]


def struct_of(r, n):
    return Simulation._particles(r, n)


def loaded_deck(case, seed):
    """The shipped deck with this case's cells and particles per cell, the cell size kept."""
    text = (DECKS / (case["deck"] + ".inp")).read_text()
    d = deck.parse(text)
    lengths = [length / cells * n for length, cells, n in ((d.grid.lx, d.grid.nx, case["nx"]), (d.grid.ly, d.grid.ny, case["ny"]),
                                                           (d.grid.lz, d.grid.nz, case["nz"]))]
    text += "".join(f"\n{k} = {v!r}" for k, v in zip(("nxc", "nyc", "nzc", "Lx", "Ly", "Lz"),
                                                     (case["nx"], case["ny"], case["nz"], *lengths)))
    for k, key in (("npcelx", "npx"), ("npcely", "npy"), ("npcelz", "npz")):
        text += f"\n{k} = " + " ".join([str(case[key])] * d.ns)
    if case["smooth"]:
        text += f"\nECSimSmoothing = energy_conserving\nSmoothNiter = {case['smooth']}\nSmooth = 0.5"
    return deck.to_case(deck.parse(text + "\n"), seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    if kind == "cycle":
        sim = Simulation(loaded_deck(case, seed), precision=case["precision"], mass_kind=case["mass"],
                         mass_layout=case["layout"], gmres_max_iterations=300, generate_on_device=True)
        sim.prepare()
        return dict(kind=kind, case=case, sim=sim)
    p = plasma(case)
    if kind == "push":
        s = random_records(case, g, case["ppc"], p["qe"], p["ve"])
        sim = stage_simulation(case, [SpeciesSpec(qom=p["qe"], npcel=(case["ppc"], 1, 1))])
        e, b = random_fields(case, g, 2e-5)
        sim.e_theta.copy_(spread(case, e, True))
        sim.b_node.copy_(spread(case, cell_to_node(b), True))
        for k, t in s["rec"].items():
            sim.slots[0][0][k].copy_(t)
        sim.bins[0][0].copy_(s["counts"])
        sim.bins[0][1].copy_(s["offsets"])
        return dict(kind=kind, case=case, sim=sim, live=0, qom=p["qe"], invalid=torch.zeros(1, dtype=torch.int32, device=DEV))
    if kind in ("deposit", "moments"):
        sets = [random_records(case, g, case["ppc"], *sv) for sv in ((p["qe"], p["ve"]), (1.0, p["vi"]))]
        sim = stage_simulation(case, species_of(case))
        _, b = random_fields(case, g, 1e-3)
        sim.b_node.copy_(spread(case, cell_to_node(b), True))
        state = dict(kind=kind, case=case, sim=sim, sets=sets)
        state["parts"] = (_lib.Particles * 2)(*[struct_of(s["rec"], s["n"]) for s in sets])
        state["qom"] = (C.c_double * 2)(*[s["qom"] for s in sets])
        state["counts"] = (C.c_void_p * 2)(*[s["counts"].data_ptr() for s in sets])
        state["offsets"] = (C.c_void_p * 2)(*[s["offsets"].data_ptr() for s in sets])
        if kind == "moments":
            cells = case["nx"] * case["ny"] * case["nz"]
            state["out"] = [[torch.zeros(m * cells, dtype=F64, device=DEV) for m in (1, 3, 6)] for _ in sets]
        return state
    if kind == "solve":
        # J and the mass of a quiet two-species plasma, eight jittered records per cell and species.
        one = SpeciesSpec(qom=p["qe"], npcel=(1, 1, 1))
        sim = stage_simulation(case, [one], smoothing=(case["smooth"], case["alpha"], case["op"]))
        e, b = random_fields(case, g, 1e-4)
        bn = cell_to_node(b)
        j, m = 0, 0
        for qom, vth in ((p["qe"], p["ve"]), (1.0, p["vi"])):
            jj, mm = deposit_exact(case, quiet_records(case, g, qom, vth), qom, bn)
            j, m = j + jj, m + mm
        sim.e.copy_(spread(case, e, True))
        sim.b_cell.copy_(spread(case, b, False))
        sim.j.copy_(spread(case, j, True))
        sim.mass.copy_(mass_layout(case, m))
        return dict(kind=kind, case=case, sim=sim, result=_lib.GmresResult())
    if kind == "backward":
        sim = stage_simulation(case, species_of(case), keep_ids=True)
        adj = AdjointBuffers(sim)
        tapes = []
        base = [random_records(case, g, case["ppc"], qom, vth, ids=True) for qom, vth in ((p["qe"], p["ve"]), (1.0, p["vi"]))]
        for _ in range(2):
            t = TapeBuffers(sim)
            base = [random_records(case, g, case["ppc"], s["qom"], 0.0, ids=True, base=s) for s in base]
            for k, s in enumerate(base):
                for a, v in s["rec"].items():
                    t.species[k][a].copy_(v)
                t.bins[k][0].copy_(s["counts"])
                t.bins[k][1].copy_(s["offsets"])
            e, b = random_fields(case, g, 1e-3)
            t.e.copy_(spread(case, e, True))
            t.b_cell.copy_(spread(case, b, False))
            t.e_theta.copy_(spread(case, 1e-3 * torch.randn(e.shape, generator=g, device=DEV, dtype=F64), True))
            tapes.append(t)
        e, b = random_fields(case, g, 1e-3)
        sim.e.copy_(spread(case, e, True))
        sim.b_cell.copy_(spread(case, b, False))
        return dict(kind=kind, case=case, sim=sim, adj=adj, tapes=tapes, result=_lib.GmresResult())
    raise ValueError(kind)


# -- one pass ----------------------------------------------------------------------------------------


def run(state):
    sim, kind = state["sim"], state["kind"]
    lib, ctx, stream = sim.lib, sim.ctx, sim._stream()
    if kind == "cycle":
        r = sim.run(1)[0]
        scalars = np.array([*r.field_energy, r.total_energy, *(v for s in r.species_scalars for v in s)])
        return dict(e=sim.field("e"), b=sim.field("b_cell"), j=sim.field("j"), mass=sim.field("mass"), scalars=scalars)
    if kind == "push":
        live = state["live"]
        src, dst = sim.slots[0][live], sim.slots[0][1 - live]
        n = src["rx"].numel()
        p, out = struct_of(src, n), struct_of(dst, n)
        cnt, off = (t.data_ptr() for t in sim.bins[0])
        inv = state["invalid"].data_ptr()
        _lib.check(lib.tpicb200_mover(ctx, state["qom"], C.byref(p), sim.e_theta.data_ptr(), sim.b_node.data_ptr(), inv, stream))
        _lib.check(lib.tpicb200_sort_binned(ctx, C.byref(p), cnt, off, C.byref(out), cnt, off, inv, stream))
        state["live"] = 1 - live
        return dict(rec=dst, counts=sim.bins[0][0], offsets=sim.bins[0][1])
    if kind == "deposit":
        _lib.check(lib.tpicb200_clear_moments(ctx, sim.j.data_ptr(), sim.mass.data_ptr(), stream))
        _lib.check(lib.tpicb200_deposit_species(ctx, 2, state["qom"], state["parts"], state["counts"], state["offsets"],
                                                sim.b_node.data_ptr(), sim.j.data_ptr(), sim.mass.data_ptr(), sim.mass_kind,
                                                0, stream))
        _lib.check(lib.tpicb200_fold_periodic(ctx, sim.j.data_ptr(), sim.mass.data_ptr(), stream))
        return dict(j=sim.j, mass=sim.mass)
    if kind == "moments":
        for s in range(2):
            rho, j, pr = state["out"][s]
            rho.zero_(), j.zero_(), pr.zero_()
            _lib.check(lib.tpicb200_output_moments(ctx, state["qom"][s], C.byref(state["parts"][s]), rho.data_ptr(),
                                                   j.data_ptr(), pr.data_ptr(), stream))
        return state["out"]
    if kind == "solve":
        _lib.check(lib.tpicb200_field_solve(ctx, sim.e.data_ptr(), sim.b_cell.data_ptr(), sim.j.data_ptr(), sim.mass.data_ptr(),
                                            sim.e_theta.data_ptr(), C.byref(state["result"]), stream))
        return dict(e_theta=sim.e_theta)
    adj = state["adj"]
    _lib.check(lib.tpicb200_adjoint_energy(ctx, sim.e.data_ptr(), sim.b_cell.data_ptr(), 1.0, 1.0, C.byref(adj.struct), stream))
    for t in reversed(state["tapes"]):
        _lib.check(lib.tpicb200_cycle_backward(ctx, C.byref(t.struct), C.byref(adj.struct), C.byref(state["result"]), stream))
    return dict(e=adj.e_bar, b=adj.b_bar, x=adj.x_bar, v=adj.v_bar, q=adj.q_bar)


# -- what a pass cannot do without -------------------------------------------------------------------


def work(case):
    cells = case["nx"] * case["ny"] * case["nz"]
    word = 8 if case["precision"] == "double" else 4
    record = 24 + 3 * word + 8 + 4
    kind = case["kind"]
    if kind == "cycle":
        n = cells * case["npx"] * case["npy"] * case["npz"] * {"harris2d_256x128": 4, "twostream1d_1024": 3}.get(case["deck"], 2)
        # Records read and written, J and the mass written; 27 pair classes x 12 entries and the push per record.
        return dict(bytes=n * 2 * record + cells * word * (2 * 129 + 24), flops=n * 1000.0 + cells * 12 * 700.0)
    if kind == "solve":
        return dict(bytes=cells * (word * (126 + 9) + 24), flops=cells * 12 * 700.0)
    n = cells * case["ppc"] * (1 if kind == "push" else 2)
    if kind == "push":
        return dict(bytes=n * 2 * record + cells * (24 + 3 * word), flops=n * 250.0)
    if kind == "deposit":
        return dict(bytes=n * record + cells * word * 132, flops=n * 800.0)
    if kind == "moments":
        return dict(bytes=n * record + 2 * cells * 80, flops=n * 200.0)
    # Two tapes read, the record gradients read and written twice, the mass formed and read.
    return dict(bytes=n * 2 * (record + 8 + 2 * 56) + cells * word * 4 * 129, flops=n * 2 * 2500.0 + cells * 24 * 700.0)


def tolerance(case):
    # Measured against `exact` and between two runs of the same inputs, times about four.
    kind, mixed = case["kind"], case["precision"] == "mixed"
    form = case.get("mass", "scalar")
    if kind == "push":
        return "exact"  # every product of the mover is rounded by itself and the sort is stable
    if kind == "moments":
        return {"rel": 4e-15, "max": 4e-14}
    if kind == "solve":  # two solutions that both meet the GMRES tolerance of 1e-8
        return {"rel": 4e-7, "max": 4e-6} if mixed else {"rel": 4e-8, "max": 4e-7}
    if form == "tf32":
        return {"rel": 1e-3, "max": 1e-2}
    if form == "bf16x3":
        return {"rel": 2e-5, "max": 4e-4}
    if kind == "deposit":
        return {"rel": 6e-7, "max": 6e-6} if mixed else {"rel": 4e-15, "max": 4e-14}
    return {"rel": 5e-6, "max": 5e-5} if mixed else {"rel": 2e-7, "max": 2e-6}


# -- the same in plain torch FP64 --------------------------------------------------------------------
# Periodic unique-node and cell arrays [3, nz, ny, nx]; at(f, di, dj, dk) is f at (i + di, j + dj, k + dk).

STENCIL = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1),
           (1, -1, 1), (1, 1, -1), (-1, 1, 1), (1, 1, 1)]
CORNERS = [(a & 1, (a >> 1) & 1, (a >> 2) & 1) for a in range(8)]
PAIRS = [(a, b, STENCIL.index(tuple(y - x for x, y in zip(CORNERS[a], CORNERS[b])))) for a in range(8) for b in range(8)
         if tuple(y - x for x, y in zip(CORNERS[a], CORNERS[b])) in STENCIL]


def at(f, di, dj, dk):
    return torch.roll(f, (-dk, -dj, -di), (-3, -2, -1))


def cell_to_node(b):
    return sum(at(b, -i, -j, -k) for i, j, k in CORNERS) / 8


def derivative(f, axis, d, sign):
    return sum((1 if a[axis] else -1) * sign * at(f, *(sign * x for x in a)) for a in CORNERS) / (4 * d)


def curl(f, d, sign):
    """curl N2C (sign +1: a cell from its corner nodes) or C2N (sign -1: a node from its cells)."""
    return torch.stack([derivative(f[q], p, d[p], sign) - derivative(f[p], q, d[q], sign) for p, q in ((1, 2), (2, 0), (0, 1))])


def smoothed(f, case):
    for _ in range(case["smooth"]):
        if case["op"] == 0:
            faces = sum(at(f, *(s if a == c else 0 for c in range(3))) for a in range(3) for s in (-1, 1))
            f = case["alpha"] * f + (1 - case["alpha"]) / 6 * faces
        else:
            for a in range(3):
                f = 0.5 * f + 0.25 * sum(at(f, *(s if a == c else 0 for c in range(3))) for s in (-1, 1))
    return f


def mass_apply(m, v, transpose=False):
    """M v, M [14, 3, 3, nz, ny, nx]."""
    eq = "rczyx,rzyx->czyx" if transpose else "rczyx,czyx->rzyx"
    out = torch.einsum(eq, m[0], v)
    for s in range(1, 14):
        o = STENCIL[s]
        out = out + torch.einsum(eq, m[s], at(v, *o))
        n = tuple(-x for x in o)
        out = out + torch.einsum(eq, at(m[s], *n), at(v, *n))
    return out


def solve_linear(apply, b, x):
    """Restarted GMRES in FP64 to the rounding of the residual."""
    scale = float(b.norm()) or 1.0
    last = math.inf
    for _ in range(12):
        r = b - apply(x)
        beta = float(r.norm())
        if beta <= 2e-15 * scale or beta > 0.5 * last:
            break
        last = beta
        m = 200
        v, h = [r / beta], np.zeros((m + 1, m))
        used = 0
        for c in range(m):
            w = apply(v[c])
            basis = torch.stack([t.reshape(-1) for t in v])
            for _ in range(2):
                dots = basis @ w.reshape(-1)
                w = w - (dots @ basis).reshape(w.shape)
                h[:c + 1, c] += dots.cpu().numpy()
            h[c + 1, c] = float(w.norm())
            used = c + 1
            e1 = np.zeros(used + 1)
            e1[0] = beta
            y, _, _, _ = np.linalg.lstsq(h[:used + 1, :used], e1, rcond=None)
            if np.linalg.norm(h[:used + 1, :used] @ y - e1) <= 1e-9 * beta or h[c + 1, c] < 1e-300:
                break
            v.append(w / h[c + 1, c])
        x = x + sum(float(t) * u for t, u in zip(y, v))
    return x


def quiet_records(case, g, qom, vth):
    """Eight records per cell, one in each octant of it, in cell order."""
    cells = case["nx"] * case["ny"] * case["nz"]
    sub = torch.tensor(CORNERS, device=DEV, dtype=F64).T.repeat(1, cells)
    frac = (sub + torch.rand((3, 8 * cells), generator=g, device=DEV, dtype=F64)) / 2
    vel = vth * torch.randn((3, 8 * cells), generator=g, device=DEV, dtype=F64)
    cell = torch.arange(cells, device=DEV).repeat_interleave(8)
    d = plasma(case)["d"]
    q = torch.full((8 * cells,), math.copysign(d**3 / 8 / (4 * math.pi), qom), device=DEV, dtype=F64)
    return dict(lin=cell, frac=frac, vel=vel, q=q)


def records_of(case, r, n=None):
    """Linear cell, fractions, velocities and charges (FP64) of stored records."""
    key = r["cell"].long() if n is None else r["cell"][:n].long()
    ex, ey = case["nx"] + 4, case["ny"] + 4
    i, j, k = key % ex - 2, (key // ex) % ey - 2, key // (ex * ey) - 2
    return dict(lin=i + case["nx"] * (j + case["ny"] * k), frac=torch.stack([r[a] for a in ("rx", "ry", "rz")]),
                vel=torch.stack([r[a].to(F64) for a in ("u", "v", "w")]), q=r["q"])


def corner_nodes(case, lin):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    i, j, k = lin % nx, (lin // nx) % ny, lin // (nx * ny)
    return torch.stack([(i + a) % nx + nx * ((j + b) % ny + ny * ((k + c) % nz)) for a, b, c in CORNERS], 1)


def weights(frac):
    return torch.stack([math.prod(frac[a] if c[a] else 1 - frac[a] for a in range(3)) for c in CORNERS], 1)


def gathered(field, idx, w):
    """A unique-node field at the records, [n, 3]."""
    return torch.einsum("cna,na->nc", field.reshape(3, -1)[:, idx], w)


def response(b, boc):
    o = boc * b
    x, y, z = o[:, 0], o[:, 1], o[:, 2]
    zero = torch.zeros_like(x)
    k = torch.stack([zero, z, -y, -z, zero, x, y, -x, zero], 1).view(-1, 3, 3)
    eye = torch.eye(3, device=DEV, dtype=F64)
    return (eye + o[:, :, None] * o[:, None, :] + k) / (1 + (o * o).sum(1))[:, None, None]


def chunks(r, size=400_000):
    n = r["q"].numel()
    for a in range(0, n, size):
        b = min(n, a + size)
        yield a, b, r["lin"][a:b], r["frac"][:, a:b], r["vel"][:, a:b], r["q"][a:b]


def spacing_dt(case):
    if case["kind"] == "cycle":
        d = deck.parse((DECKS / (case["deck"] + ".inp")).read_text())
        return [d.grid.lx / d.grid.nx, d.grid.ly / d.grid.ny, d.grid.lz / d.grid.nz], d.dt
    return [plasma(case)["d"]] * 3, plasma(case)["dt"]


def deposit_exact(case, r, qom, bn):
    """J [3, ...] and M [14, 3, 3, ...] of one species' records at the unique nodes."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells = nx * ny * nz
    d, dt = spacing_dt(case)
    boc, volume = qom * dt / 2, d[0] * d[1] * d[2]
    acc = torch.zeros((cells, len(PAIRS) * 9 + 24), device=DEV, dtype=F64)
    pa, pb = ([p[i] for p in PAIRS] for i in (0, 1))
    for _, _, lin, frac, vel, q in chunks(r):
        w = weights(frac)
        alpha = response(gathered(bn, corner_nodes(case, lin), w), boc)
        pair = (w[:, pa] * w[:, pb])[:, :, None] * (alpha.reshape(-1, 1, 9) * (boc * q)[:, None, None])
        cur = torch.einsum("nij,jn->ni", alpha, vel) * (q / volume)[:, None]
        acc.index_add_(0, lin, torch.cat([pair.reshape(-1, len(PAIRS) * 9), (w[:, :, None] * cur[:, None, :]).reshape(-1, 24)], 1))
    acc = acc.T.reshape(-1, nz, ny, nx)
    j = torch.zeros((3, nz, ny, nx), device=DEV, dtype=F64)
    m = torch.zeros((14, 9, nz, ny, nx), device=DEV, dtype=F64)
    for i, (a, _, s) in enumerate(PAIRS):
        m[s] += at(acc[9 * i:9 * i + 9], *(-x for x in CORNERS[a]))
    for a in range(8):
        j += at(acc[9 * len(PAIRS) + 3 * a:][:3], *(-x for x in CORNERS[a]))
    return j, m.view(14, 3, 3, nz, ny, nx)


def mass_layout(case, m):
    """The mass buffer of the case's layout, periodic copies filled."""
    flat = m.reshape(126, case["nz"], case["ny"], case["nx"])
    iz, iy, ix = (wrap_index(n, -1, n + 3) for n in (case["nz"], case["ny"], case["nx"]))
    full = flat[:, iz][:, :, iy][:, :, :, ix]
    if case["layout"] == "records":
        return full.reshape(126, -1).T.reshape(-1).contiguous()
    if case["layout"] == "tiled":
        pad = -full.shape[-1] % 4
        full = torch.nn.functional.pad(full, (0, pad))
    return full.reshape(-1).contiguous()


def push_exact(case, r, qom, theta, bn):
    """Moved velocities [3, n], fractions and linear cells."""
    d, dt = spacing_dt(case)
    ext = (case["nx"], case["ny"], case["nz"])
    vel, frac, lin_out = torch.empty_like(r["vel"]), torch.empty_like(r["frac"]), torch.empty_like(r["lin"])
    for a, b, lin, f, v, _ in chunks(r, 2_000_000):
        idx, w = corner_nodes(case, lin), weights(f)
        alpha = response(gathered(bn, idx, w), qom * dt / 2)
        new = 2 * torch.einsum("nij,jn->in", alpha, v + qom * dt / 2 * gathered(theta, idx, w).T) - v
        out, stride = 0, 1
        cell = (lin % ext[0], (lin // ext[0]) % ext[1], lin // (ext[0] * ext[1]))
        for c in range(3):
            moved = f[c] + dt * new[c] / d[c]
            step = moved.floor()
            part = moved - step
            carry = part >= 1
            frac[c, a:b] = torch.where(carry, 0.0, part)
            out = out + stride * ((cell[c] + step.long() + carry) % ext[c])
            stride *= ext[c]
        vel[:, a:b], lin_out[a:b] = new, out
    return vel, frac, lin_out


def unique(case, field, nodes):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    e = 3 if nodes else 2
    return field.to(F64).view(3, nz + e, ny + e, nx + e)[:, 1:nz + 1, 1:ny + 1, 1:nx + 1].contiguous()


def operator(case, m, transpose=False):
    d, dt = spacing_dt(case)
    delta, kv = 0.5 * dt, 4 * math.pi * 0.5 * dt / (d[0] * d[1] * d[2])
    flat = dict(case, smooth=0) if transpose else case

    def apply(v):
        response_ = smoothed(mass_apply(m, smoothed(v, flat), transpose), flat)
        return v + delta**2 * curl(curl(v, d, 1), d, -1) + kv * response_
    return apply


def field_solve_exact(case, e, b, j, m):
    d, dt = spacing_dt(case)
    rhs = e + 0.5 * dt * curl(b, d, -1) - 4 * math.pi * 0.5 * dt * smoothed(j, case)
    return solve_linear(operator(case, m), rhs, e)


def exact(case, seed):
    kind = case["kind"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "cycle" and (cells > 80_000 or cells * case["npx"] * case["npy"] * case["npz"] > 6_000_000):
        return None
    state = prepare(case, seed)
    sim = state["sim"]
    if kind == "cycle":
        return cycle_exact(case, sim)
    if kind == "push":
        r = records_of(case, sim.slots[0][0])
        vel, frac, lin = push_exact(case, r, state["qom"], unique(case, sim.e_theta, True), unique(case, sim.b_node, True))
        _, order = torch.sort(lin, stable=True)
        rec = {k: v[order] for k, v in zip(("rx", "ry", "rz", "u", "v", "w", "q"), (*frac, *vel, r["q"]))}
        return dict(rec=dict(rec, cell=None), counts=None, offsets=None)
    if kind == "deposit":
        j, m = 0, 0
        for s in state["sets"]:
            jj, mm = deposit_exact(case, records_of(case, s["rec"]), s["qom"], unique(case, sim.b_node, True))
            j, m = j + jj, m + mm
        return dict(j=spread(case, j, True), mass=mass_layout(case, m))
    if kind == "moments":
        return [moments_exact(case, records_of(case, s["rec"]), s["qom"]) for s in state["sets"]]
    if kind == "solve":
        if case["nz"] > 1 and cells > 600_000:
            return None
        f = [unique(case, t, n) for t, n in ((sim.e, True), (sim.b_cell, False), (sim.j, True))]
        return dict(e_theta=spread(case, field_solve_exact(case, *f, unique_mass(case, sim.mass)), True))
    return backward_exact(case, state)


def unique_mass(case, mass):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["layout"] == "records":
        full = mass.to(F64).view(-1, 126).T.reshape(126, nz + 3, ny + 3, nx + 3)
    else:
        full = mass.to(F64).view(126, nz + 3, ny + 3, -1)
    return full[:, 1:nz + 1, 1:ny + 1, 1:nx + 1].contiguous().view(14, 3, 3, nz, ny, nx)


def moments_exact(case, r, qom):
    cells = case["nx"] * case["ny"] * case["nz"]
    volume = plasma(case)["d"]**3
    out = torch.zeros((cells, 10), device=DEV, dtype=F64)
    for _, _, lin, frac, vel, q in chunks(r, 2_000_000):
        c = q / volume
        u, v, w = vel
        amount = torch.stack([4 * math.pi * c, c * u, c * v, c * w, *(c / qom * t for t in (u * u, u * v, u * w, v * v, v * w, w * w))], 1)
        wt, idx = weights(frac), corner_nodes(case, lin)
        for a in range(8):
            out.index_add_(0, idx[:, a], amount * wt[:, a:a + 1])
    return [out[:, 0].contiguous(), out[:, 1:4].T.reshape(-1).contiguous(), out[:, 4:].T.reshape(-1).contiguous()]


def cycle_exact(case, sim):
    full = dict(case, alpha=0.5, op=0)
    d, dt = spacing_dt(full)
    start_e = sim.field("e")
    e, b = unique(full, start_e, True), unique(full, sim.field("b_cell"), False)
    bn = cell_to_node(b)
    species = [(records_of(full, sim.live(s)), sp.qom) for s, sp in enumerate(sim.case.species)]

    def deposits(sets, field):
        j, m = 0, 0
        for r, qom in sets:
            jj, mm = deposit_exact(full, r, qom, field)
            j, m = j + jj, m + mm
        return j, m

    theta = field_solve_exact(full, e, b, *deposits(species, bn))
    e_next, b_next = 2 * theta - e, b - dt * curl(theta, d, 1)
    seen = smoothed(theta, full)
    moved, scalars = [], []
    for r, qom in species:
        vel, frac, lin = push_exact(full, r, qom, seen, bn)
        moved.append((dict(lin=lin, frac=frac, vel=vel, q=r["q"]), qom))
        mass = r["q"] / qom
        scalars += [0.5 * (mass * (vel * vel).sum(0)).sum(), r["q"].sum(), *((mass * vel).sum(1))]
    j, m = deposits(moved, cell_to_node(b_next))
    norm = d[0] * d[1] * d[2] / (8 * math.pi)
    fields = [norm * (e_next**2).sum(), norm * (b_next**2).sum()]
    total = sum(fields) + sum(scalars[5 * s] for s in range(len(species)))
    # The advance writes E at the nodes 0..n; the ghost layer keeps what the run started with.
    stored = start_e.to(F64).clone().view(3, case["nz"] + 3, case["ny"] + 3, case["nx"] + 3)
    inner = (slice(None),) + (slice(1, -1),) * 3
    stored[inner] = spread(full, e_next, True).view_as(stored)[inner]
    return dict(e=stored.reshape(-1), b=spread(full, b_next, False), j=spread(full, j, True), mass=mass_layout(full, m),
                scalars=np.array([float(v) for v in (*fields, total, *scalars)]))


def backward_exact(case, state):
    """The adjoint of two cycles: FP64 reverse mode of each stage, the solve by its transposed operator."""
    full = dict(case, smooth=0)
    sim = state["sim"]
    d, dt = spacing_dt(full)
    volume = d[0] * d[1] * d[2]
    norm = volume / (4 * math.pi)
    eb, bb = norm * unique(full, sim.e, True), norm * unique(full, sim.b_cell, False)
    n = [t.numel() // 3 for t in state["adj"].x_bar]
    xb, vb = ([torch.zeros((3, m), device=DEV, dtype=F64) for m in n] for _ in range(2))
    qb = [torch.zeros(m, device=DEV, dtype=F64) for m in n]
    inv = torch.tensor([1 / s for s in d], device=DEV, dtype=F64)
    kfac = 4 * math.pi * 0.5 * dt
    for tape in reversed(state["tapes"]):
        b, theta = unique(full, tape.b_cell, False), unique(full, tape.e_theta, True)
        bn = cell_to_node(b)
        sets = [(records_of(full, tape.species[s]), tape.species[s]["id"], sim.case.species[s].qom) for s in range(2)]
        m = sum(deposit_exact(full, r, qom, bn)[1] for r, _, qom in sets)
        # theta_bar of the advance (N2C is the transpose of C2N) and of the movers.
        tb = 2 * eb - dt * curl(bb, d, -1)
        for s, (r, ident, qom) in enumerate(sets):
            for i, k, lin, f, v, q in chunks(r):
                p = ident[i:k]
                w, idx = weights(f), corner_nodes(full, lin)
                alpha = response(gathered(bn, idx, w), qom * dt / 2)
                g = 2 * (vb[s][:, p].T + dt * inv * xb[s][:, p].T)
                t = qom * dt / 2 * torch.einsum("nij,ni->nj", alpha, g)
                for a in range(8):
                    tb.view(3, -1).index_add_(1, idx[:, a], (w[:, a:a + 1] * t).T.contiguous())
        lam = solve_linear(operator(full, m, True), tb, torch.zeros_like(tb))
        bnb = torch.zeros_like(bn)
        for s, (r, ident, qom) in enumerate(sets):
            boc = qom * dt / 2
            for i, k, lin, f, v, q in chunks(r, 200_000):
                p = ident[i:k]
                idx = corner_nodes(full, lin)
                f, v, q = (t.clone().requires_grad_() for t in (f, v, q))
                corners = bn.reshape(3, -1)[:, idx].clone().requires_grad_()
                w = weights(f)
                alpha = response(torch.einsum("cna,na->nc", corners, w), boc)
                u, lp = gathered(theta, idx, w), gathered(lam, idx, w)
                new = 2 * torch.einsum("nij,nj->ni", alpha, v.T + boc * u) - v.T
                value = (vb[s][:, p].T * new).sum() + (xb[s][:, p].T * (f.T + dt * inv * new)).sum()
                value = value - kfac / volume * (q * (lp * torch.einsum("nij,jn->ni", alpha, v)).sum(1)).sum()
                value = value - kfac / volume * boc * (q * (lp * torch.einsum("nij,nj->ni", alpha, u)).sum(1)).sum()
                gf, gv, gq, gc = torch.autograd.grad(value, (f, v, q, corners))
                xb[s][:, p], vb[s][:, p] = gf, gv
                qb[s][p] += gq
                for a in range(8):
                    bnb.view(3, -1).index_add_(1, idx[:, a], gc[:, :, a].contiguous())
        eb = lam - eb
        bb = bb + 0.5 * dt * curl(lam, d, 1) + sum(at(bnb, *c) for c in CORNERS) / 8
    return dict(e=spread(full, eb, True), b=spread(full, bb, False), x=[t.reshape(-1) for t in xb], v=[t.reshape(-1) for t in vb], q=qb)
