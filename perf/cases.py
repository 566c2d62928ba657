"""Work that users of this library have it do, as timed cases: MD loops, single-point evaluations of frames that come from
the host, the host-buffer force call of an engine plugin, and radius graphs for machine-learned potentials.

Every case goes through ``deepscalemd_b200.capi`` as a program does that couples the library from Python. Inputs are made
from the seed on the GPU; systems have the shapes, densities, cutoffs and parameters of the repository's own synthetic
systems (``deepscalemd_b200/synthetic.py``), at any atom count: lattices with vacancies where the count does not fill them.
"""
import math

import numpy as np
import torch

from deepscalemd_b200 import capi
from deepscalemd_b200 import synthetic

KCAL = 2390.0574            # A^2 amu / fs^2 -> kcal/mol
KB = 0.0019872041           # kcal / mol / K
FORCE_TO_ACCEL = 4.184e-4   # kcal / mol / A / amu -> A / fs^2
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "fx", "fy", "fz")


def listed():
    return [
        # the smallest box MD users and the test-suite run: every step is a handful of short launches
        {"name": "lj_nve_864", "kind": "nve", "atoms": 864, "steps": 30},
        # the standard small Lennard-Jones benchmark (20^3 FCC cells)
        {"name": "lj_nve_32000", "kind": "nve", "atoms": 32000, "steps": 30},
        # the benchmark's production size (100^3 FCC cells)
        {"name": "lj_nve_4000000", "kind": "nve", "atoms": 4000000, "steps": 12},
        # binary mixture under a velocity-scaling thermostat: the step-by-step entry points the driver calls, with the
        # displacement and the kinetic energy read back every step
        {"name": "mixture_nvt_1048575", "kind": "nvt", "atoms": 1048575, "steps": 5},
        # rigid water with real-space Ewald, exclusions and constraints: a small box and the production size
        {"name": "water_md_3993", "kind": "water", "molecules": 1331, "steps": 10},
        {"name": "water_md_648000", "kind": "water", "molecules": 216000, "steps": 5},
        # flexible chains: every kind of bonded term, exclusions, per-atom charges
        {"name": "chains_md_63504", "kind": "chains", "tiles_x": 6, "tiles_y": 7, "tiles_z": 7, "steps": 10},
        # re-evaluation of a stored frame: upload, list, energy and virial with a switched potential
        {"name": "frame_energy_108000", "kind": "frame", "atoms": 108000, "switched": True},
        # an engine that keeps its atoms on the host and calls the library as a force provider between list rebuilds
        {"name": "host_forces_1000188", "kind": "host", "atoms": 1000188},
        # radius graph of a periodic solid, compact form, atoms numbered at random
        {"name": "graph_periodic_1000000", "kind": "graph", "atoms": 1000000},
        # one call of a machine-learned potential in the framework's own form: image atoms, receiver mask, edges with
        # shifts, forces folded back, virial
        {"name": "mlip_step_125000", "kind": "mlip", "atoms": 125000},
        # radius graph of a small cluster without a box
        {"name": "graph_open_2001", "kind": "open", "atoms": 2001},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nve", "nve", "nvt", "water", "chains", "frame", "host", "graph", "mlip", "open"])
    if kind == "nve":
        n = _log_uniform(rng, 700, 4000000)
        return {"kind": kind, "atoms": n, "steps": 30 if n < 200000 else 12}
    if kind == "nvt":
        return {"kind": kind, "atoms": _log_uniform(rng, 1500, 1048575), "steps": 5}
    if kind == "water":
        m = _log_uniform(rng, 1100, 216000)
        return {"kind": kind, "molecules": m, "steps": 10 if m < 20000 else 5}
    if kind == "chains":
        return {"kind": kind, "tiles_x": rng.randint(1, 7), "tiles_y": rng.randint(1, 7), "tiles_z": rng.randint(1, 7), "steps": 10}
    if kind == "frame":
        return {"kind": kind, "atoms": _log_uniform(rng, 4000, 500000), "switched": rng.random() < 0.5}
    if kind == "host":
        return {"kind": kind, "atoms": _log_uniform(rng, 10000, 4000000)}
    if kind == "graph":
        return {"kind": kind, "atoms": _log_uniform(rng, 2000, 1000000)}
    if kind == "mlip":
        return {"kind": kind, "atoms": _log_uniform(rng, 2000, 125000)}
    return {"kind": kind, "atoms": _log_uniform(rng, 1000, 100000)}


# -- inputs ------------------------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, half_width):
    return (torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0) * half_width


def _sites(n, per_cell=1):
    """A near-cubic block of lattice cells with at least n sites."""
    c = max(1, math.ceil((n / per_cell) ** (1.0 / 3.0) - 1e-9))
    return c, c, math.ceil(n / (per_cell * c * c))


def _lattice(g, n, basis, density):
    """n atoms on a random subset of the sites of a lattice (ascending site order) at the given density; box and spacing."""
    dims = _sites(n, len(basis))
    total = dims[0] * dims[1] * dims[2] * len(basis)
    spacing = (n / (density * dims[0] * dims[1] * dims[2])) ** (1.0 / 3.0)
    site = torch.randperm(total, generator=g, device="cuda")[:n].sort().values if n < total else torch.arange(total, device="cuda")
    cell, b = site // len(basis), site % len(basis)
    idx = torch.stack([cell // (dims[1] * dims[2]), (cell // dims[2]) % dims[1], cell % dims[2]], dim=1).double()
    offsets = torch.tensor(basis, device="cuda", dtype=torch.float64)[b]
    return (idx + offsets + 0.25) * spacing, np.array(dims, dtype=np.float64) * spacing, spacing


def _velocities(g, mass, temperature, kb=1.0):
    v = torch.randn((len(mass), 3), generator=g, device="cuda", dtype=torch.float64) * (kb * temperature / mass)[:, None].sqrt()
    v -= (v * mass[:, None]).sum(0) / mass.sum()
    return v * math.sqrt(temperature * kb * (3 * len(mass) - 3) / float((mass[:, None] * v * v).sum()))


FCC = [[0.0, 0.0, 0.0], [0.5, 0.5, 0.0], [0.5, 0.0, 0.5], [0.0, 0.5, 0.5]]


def _lennard_jones(g, n):
    pos, box, _ = _lattice(g, n, FCC, 0.8442)
    boxes = torch.tensor(box, device="cuda")
    pos = (pos + _uniform(g, pos.shape, 0.05)) % boxes
    vel = _velocities(g, torch.ones(n, device="cuda", dtype=torch.float64), 1.44)
    return pos.cpu().numpy(), box, vel.cpu().numpy()


def _lj_context(case, seed, switch=-1.0):
    g = _generator(seed)
    pos, box, vel = _lennard_jones(g, case["atoms"])
    ctx = capi.Context(case["atoms"])
    ctx.set_box(box)
    ctx.set_pair_params([[1.0]], [[1.0]], 2.5, 0.3, switch)
    return ctx, pos, vel


def _mixture_context(case, seed):
    g = _generator(seed)
    n = case["atoms"]
    pos, box, spacing = _lattice(g, n, [[0.0, 0.0, 0.0]], 1.2)
    pos = (pos + _uniform(g, pos.shape, 0.12)) % torch.tensor(box, device="cuda")
    types = torch.zeros(n, device="cuda", dtype=torch.int32)
    types[torch.randperm(n, generator=g, device="cuda")[: n // 5]] = 1
    vel = _velocities(g, torch.ones(n, device="cuda", dtype=torch.float64), 0.8)
    ctx = capi.Context(n)
    ctx.set_box(box)
    ctx.set_pair_params([[1.0, 1.5], [1.5, 0.5]], [[1.0, 0.8], [0.8, 0.88]], 2.5, 0.3)
    ctx.upload(pos.cpu().numpy(), vel=vel.cpu().numpy(), mass=np.ones(n), types=types.cpu().numpy())
    return ctx


def _water_context(case, seed):
    g = _generator(seed)
    m = case["molecules"]
    centre, box, spacing = _lattice(g, m, [[0.0, 0.0, 0.0]], 1.0 / 29.9151)
    centre = centre + _uniform(g, centre.shape, 0.1)
    q = torch.randn((m, 4), generator=g, device="cuda", dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    # the two columns of the rotation matrix that the O-H vectors need (they lie in the local x-z plane)
    ex = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], dim=1)
    ez = torch.stack([2 * (x * z + y * w), 2 * (y * z - x * w), 1 - 2 * (x * x + y * y)], dim=1)
    half = math.radians(109.47) / 2.0
    pos = torch.stack([centre, centre + math.sin(half) * ex + math.cos(half) * ez,
                       centre - math.sin(half) * ex + math.cos(half) * ez], dim=1).reshape(-1, 3)
    n = 3 * m
    mass = torch.tensor([15.9994, 1.008, 1.008], device="cuda", dtype=torch.float64).repeat(m)
    # rigid molecules: all three atoms start with the velocity of their centre (no component along a constraint)
    vel = _velocities(g, torch.full((m,), 18.0154, device="cuda", dtype=torch.float64), 300.0, KB / KCAL)
    vel = vel.repeat_interleave(3, dim=0)
    o = 3 * np.arange(m, dtype=np.int32)
    pairs = np.stack([np.stack([o, o + 1], 1), np.stack([o, o + 2], 1), np.stack([o + 1, o + 2], 1)], axis=1).reshape(-1, 2)
    rows = np.concatenate([pairs.astype(np.float64), np.tile([1.0, 1.0, 2.0 * math.sin(half)], m)[:, None]], axis=1)
    charges = [-0.8476, 0.4238]
    ctx = capi.Context(n)
    ctx.set_box(box)
    ctx.set_pair_params([[0.1553, 0.0], [0.0, 0.0]], [[3.166, 1.583], [1.583, 0.0]], 10.0, 2.0)
    ctx.set_coulomb(True)
    ctx.set_exclusions(n, pairs)
    ctx.set_constraints(n, rows)
    ctx.upload(pos.cpu().numpy(), vel=vel.cpu().numpy(), mass=mass.cpu().numpy(), types=np.tile(np.array([0, 1, 1], np.int32), m),
               charge=np.tile([charges[0], charges[1], charges[1]], m))
    ctx.set_type_charges(charges)
    return ctx


def _chains_context(case, seed):
    """A cube of 27 chains, repeated along the axes; every copy gets its own velocities."""
    g = _generator(seed)
    s = synthetic.chain_fluid(3, 8, spacing=14.0, seed=int(seed) % (1 << 30))
    tiles = [case["tiles_x"], case["tiles_y"], case["tiles_z"]]
    copies = tiles[0] * tiles[1] * tiles[2]
    shift = np.stack(np.meshgrid(*[np.arange(t) for t in tiles], indexing="ij"), axis=-1).reshape(-1, 1, 3) * s.box
    n = copies * s.n
    pos = (s.pos[None] + shift).reshape(-1, 3)
    mass = np.tile(s.mass, copies)
    vel = _velocities(g, torch.tensor(mass, device="cuda"), 300.0, KB / KCAL).cpu().numpy()

    def repeated(ids):
        ids = np.asarray(ids)
        return (ids[None] + (np.arange(copies) * s.n).reshape(-1, 1, 1)).reshape(-1, ids.shape[1]).astype(np.int32)

    atoms = ("bonds", "angles", "torsions", "specials")
    terms = {k: repeated(v) if k in atoms else np.tile(v, copies) for k, v in s.bonded.items() if k != "n_dihedrals"}
    ctx = capi.Context(n)
    box = s.box * np.array(tiles)
    ctx.set_box(box)
    ctx.set_pair_params(s.eps, s.sig, s.cutoff, s.skin)
    ctx.set_coulomb(True)
    ctx.set_exclusions(n, repeated(s.exclusions))
    ctx.set_bonded(n, terms)
    # chains that cross the face of the cube go on in the neighbouring copy
    first = s.pos.reshape(27, 8, 3)[:, :1]
    jump = np.round((s.pos.reshape(27, 8, 3) - first) / s.box).reshape(-1, 3)
    pos = (pos.reshape(copies, s.n, 3) - jump[None] * s.box).reshape(-1, 3) % box
    ctx.upload(pos, vel=vel, mass=mass, types=np.tile(s.types, copies), charge=np.tile(s.charge, copies))
    return ctx


def _solid(seed, n, shuffled, periodic=True):
    """A disordered solid: jittered cubic lattice at 0.05 atoms / A^3, numbered by site or at random. The seed moves and
    mirrors one solid per size (through the periodic box, or as an open cluster) and numbers its atoms, so that the graph
    has the same number of edges whatever the seed."""
    pos, box, spacing = _lattice(_generator(n), n, [[0.0, 0.0, 0.0]], 0.05)
    pos = pos + _uniform(_generator(n + 1), pos.shape, 0.45)
    g = _generator(seed)
    boxes = torch.tensor(box, device="cuda")
    mirror = torch.randint(0, 2, (3,), generator=g, device="cuda") * 2.0 - 1.0
    pos = pos * mirror + torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * boxes
    if periodic:
        pos = pos % boxes
    if shuffled:
        pos = pos[torch.randperm(n, generator=g, device="cuda")]
    return [pos[:, k].contiguous() for k in range(3)], box, g


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "views": {}, "xi": 0.0}
    if kind == "nve":
        ctx, pos, vel = _lj_context(case, seed)
        ctx.upload(pos, vel=vel)
    elif kind == "nvt":
        ctx = _mixture_context(case, seed)
    elif kind == "water":
        ctx = _water_context(case, seed)
    elif kind == "chains":
        ctx = _chains_context(case, seed)
    elif kind == "frame":
        ctx, pos, _ = _lj_context(case, seed, 2.0 if case["switched"] else -1.0)
        state["frame"] = pos
    elif kind == "host":
        ctx, pos, _ = _lj_context(case, seed)
        ctx.upload(pos)
    if kind in ("nve", "nvt", "water", "chains", "host"):
        ctx.build_neighbor_list()
        ctx.compute_forces()
        ctx.compute_bonded()
    if kind == "host":
        # the engine's buffers, in the context's order, half a skin's way from the list's reference positions at most
        order = ctx.download("global_id")
        moved = pos[order] + _uniform(_generator(seed + 1), pos.shape, 0.08).cpu().numpy()
        state["host"] = [torch.from_numpy(np.ascontiguousarray(moved[:, k])).pin_memory() for k in range(3)]
        state["forces"] = [torch.zeros(len(pos), dtype=torch.float64).pin_memory() for _ in range(3)]
    if kind in ("graph", "mlip", "open"):
        state["graph"] = capi.EdgeBuilder()
        state["xyz"], state["box"], g = _solid(seed, case["atoms"], kind != "mlip", kind != "open")
        if kind == "mlip":
            reach = 5.0 + 1e-8
            state["region"] = (np.full(3, -reach), state["box"] + reach)
            state["types"] = torch.randint(0, 3, (case["atoms"],), generator=g, device="cuda", dtype=torch.int32)
            n_all = state["graph"].images(*state["xyz"], state["types"], state["box"], np.zeros(3), *state["region"], (1, 1, 1))["n_all"]
            # what the model returns for the atoms and their images
            state["model"] = [torch.randn(n_all, generator=g, device="cuda", dtype=torch.float64) for _ in range(3)]
            state["total"] = [torch.zeros(case["atoms"], device="cuda", dtype=torch.float64) for _ in range(3)]
    else:
        state["ctx"] = ctx
    return state


# -- one pass ----------------------------------------------------------------------------------------------------------

def _view(state, name):
    """The context's own device array as a tensor (sorting at a list build swaps between two sets of arrays)."""
    ctx = state["ctx"]
    key = ctx.device_pointer(name)
    if key not in state["views"]:
        n, _ = ctx.counts()
        dtype = torch.int32 if name == "global_id" else torch.float64
        state["views"][key] = capi._tensor_from_ptr(key, (n,), dtype, torch.device("cuda", ctx.device))
    return state["views"][key]


def _by_atom(state, fields):
    """[fields, atoms] in the caller's atom numbering: the arrays of the context are in cell order."""
    rows = torch.stack([_view(state, f) for f in fields])
    out = torch.empty_like(rows)
    out[:, _view(state, "global_id").long()] = rows
    return out


def _held(builder, *tensors):
    """The builder's results are views of its own buffers: whoever holds one holds the builder."""
    for t in tensors:
        t.builder = builder
    return tensors


def _thermostat(state, dt, temperature_now, target, tau):
    state["xi"] += dt / (tau * tau) * (temperature_now / target - 1.0)
    return math.exp(-state["xi"] * dt)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "nve":
        state["ctx"].run_nve(case["steps"], 0.005)
        return _by_atom(state, FIELDS)
    if kind == "nvt":
        ctx, dt = state["ctx"], 0.005
        for _ in range(case["steps"]):
            ctx.integrate(1, dt)
            if ctx.max_displacement_sq() > 0.15 * 0.15:
                ctx.build_neighbor_list()
            ctx.compute_forces()
            ctx.integrate(2, dt)
            kinetic = ctx.kinetic_energy()
            ctx.scale_velocities(_thermostat(state, dt, 2.0 * kinetic / (3 * case["atoms"] - 3), 0.8, 0.05))
        return {"state": _by_atom(state, FIELDS), "kinetic": kinetic}
    if kind == "water":
        ctx = state["ctx"]
        ctx.run_nve(case["steps"], 2.0, FORCE_TO_ACCEL)
        kinetic = ctx.kinetic_energy()
        # velocities rescaled to 300 K between the blocks of steps, as an equilibration run does
        now = 2.0 * kinetic * KCAL / (KB * (6 * case["molecules"] - 3))
        ctx.scale_velocities(math.sqrt(300.0 / now))
        return {"state": _by_atom(state, FIELDS), "kinetic": kinetic}
    if kind == "chains":
        ctx = state["ctx"]
        ctx.run_nve(case["steps"], 0.5, FORCE_TO_ACCEL)
        return _by_atom(state, FIELDS)
    if kind == "frame":
        ctx = state["ctx"]
        ctx.upload(state["frame"])
        ctx.build_neighbor_list()
        ctx.compute_forces(capi.PHASE_FULL, want_energy=True)
        scalars = ctx.read_scalars()
        return {"forces": _by_atom(state, ("fx", "fy", "fz")), **scalars}
    if kind == "host":
        state["ctx"].forces_host(*[t.data_ptr() for t in state["host"]], *[t.data_ptr() for t in state["forces"]])
        return state["forces"]
    graph = state["graph"]
    if kind == "graph":
        return _held(graph, *graph.build_periodic(*state["xyz"], state["box"], 5.0))
    if kind == "open":
        return _held(graph, graph.build(*state["xyz"], 5.0)[0])
    lo, hi = state["region"]
    image = graph.images(*state["xyz"], state["types"], state["box"], np.zeros(3), lo, hi, (1, 1, 1))
    positions = (image["x"], image["y"], image["z"])
    inside = graph.mark_receivers(*[p[: case["atoms"]] for p in positions], np.zeros(3), state["box"], 2.0)
    index, shift = graph.build(*positions, 5.0, lo=lo, hi=hi, n_centers=case["atoms"], owner=image["owner"],
                               shift=image["shift"], receiver_ok=inside, row=1)
    for t in state["total"]:
        t.zero_()
    graph.fold_image_forces(*state["model"], *state["total"])
    virial = graph.virial_from_forces(*positions, *state["model"])
    _held(graph, index, shift)
    return {"index": index, "shift": shift, "forces": state["total"], "virial": virial}


# -- what a pass cannot do without ---------------------------------------------------------------------------------------

def _sphere(density, r):
    return density * 4.0 / 3.0 * math.pi * r ** 3


def work(case):
    """Bytes: the state of the atoms in and out once per pass (an MD pass: positions, velocities and forces; the box is
    small enough to stay on the chip or is streamed again every step, which is not counted), the input and output arrays
    of a graph once. Flops: 8 for every pair of atoms inside the list radius and 19 (28 with Coulomb) for every pair
    inside the cutoff, per force evaluation; 8 per tested neighbour of a graph."""
    kind = case["kind"]
    if kind in ("graph", "open", "mlip"):
        n = case["atoms"]
        edges = n * _sphere(0.05, 5.0)
        if kind == "graph":
            return {"bytes": 24 * n + 23 * edges, "flops": 8 * edges}
        if kind == "open":
            return {"bytes": 24 * n + 16 * edges, "flops": 8 * edges}
        side = (n / 0.05) ** (1.0 / 3.0)
        n_all = n * ((side + 10.0) / side) ** 3
        return {"bytes": 28 * n + 60 * n_all + 40 * edges + 48 * n_all + 72 * n, "flops": 8 * edges + 12 * n_all}
    density, cutoff, skin, flops = {"nve": (0.8442, 2.5, 0.3, 19), "nvt": (1.2, 2.5, 0.3, 19), "water": (0.1003, 10.0, 2.0, 28),
                                    "chains": (0.0029, 9.0, 1.5, 28), "frame": (0.8442, 2.5, 0.3, 19), "host": (0.8442, 2.5, 0.3, 19)}[kind]
    n = {"water": lambda: 3 * case["molecules"], "chains": lambda: 216 * case["tiles_x"] * case["tiles_y"] * case["tiles_z"]}.get(
        kind, lambda: case["atoms"])()
    evaluations = case.get("steps", 1)
    flops = evaluations * n * 0.5 * (8 * _sphere(density, cutoff + skin) + flops * _sphere(density, cutoff))
    return {"bytes": n * {"frame": 24 + 24, "host": 24 + 24}.get(kind, 72 + 72), "flops": flops}


def tolerance(case):
    """Single-precision pair sums: forces agree to some 1e-6; an MD pass adds the growth of such differences along a short
    trajectory of strongly coupled atoms. Graphs are exact; the virial of the folded forces is a sum in double precision."""
    kind = case["kind"]
    if kind in ("graph", "open"):
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "mlip":
        return {"rel": 1e-9, "max": 1e-9}
    if kind in ("frame", "host"):
        return {"rel": 5e-6, "max": 1e-4}
    return {"rel": 5e-5, "max": 5e-3}
