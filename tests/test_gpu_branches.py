"""GPU tests of the branches that a size, a type or the layout of the input picks, at the sizes where they can go wrong,
against the CPU oracle."""
import numpy as np
import pytest

from deepscalemd_b200 import capi
from oracle import cpu_oracle as co

pytestmark = pytest.mark.gpu


# atoms, box, cutoff, skin, types, Coulomb, exclusions: lone atoms and two; rows of one to four atoms; one, two, few and more than
# eight types; Ewald tables in one copy (short rows) and in eight (rows of 240 and more, which have their entries in another order)
ROWS = [
    (1, 20.0, 4.0, 0.5, 1, False, False), (2, 20.0, 4.0, 0.5, 1, True, False), (37, 20.0, 4.0, 0.5, 3, False, False),
    (333, 20.0, 4.0, 0.5, 8, True, True), (334, 20.0, 4.0, 0.5, 9, True, True), (600, 16.0, 3.0, 0.3, 9, False, True),
    (2500, 25.0, 6.0, 0.5, 2, True, True), (2500, 25.0, 6.0, 0.5, 1, False, False), (600, 16.0, 3.0, 0.3, 2, False, True),
    (2500, 25.0, 6.0, 0.5, 2, False, True), (2503, 25.0, 6.0, 0.5, 9, False, True),
]


@pytest.mark.parametrize("n,L,rc,skin,nt,coulomb,excl", ROWS)
@pytest.mark.parametrize("switched", [False, True])
def test_forces_of_every_row_form(cuda_device, n, L, rc, skin, nt, coulomb, excl, switched):
    rng = np.random.default_rng(n + nt)
    side = int(np.ceil(n ** (1 / 3)))
    sites = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(side ** 3)[:n]]
    pos = ((sites + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * (L / side)) % L
    box = np.full(3, L)
    types = rng.integers(0, nt, n).astype(np.int32)
    sig = 0.5 * (rng.uniform(0.8, 1.2, nt)[:, None] + rng.uniform(0.8, 1.2, nt)[None])
    sig, eps = 0.5 * (sig + sig.T), np.full((nt, nt), 0.3)
    charge = rng.uniform(-0.5, 0.5, n) if coulomb else np.zeros(n)
    pairs = co.pairs(*pos.T, n, box, search=rc + skin)
    exclusions = pairs[:: 5] if excl else None
    switch = 0.8 * rc if switched else -1.0
    ctx = capi.Context(n)
    ctx.set_box(box)
    ctx.set_pair_params(eps, sig, rc, skin, switch)
    if coulomb:
        ctx.set_coulomb(True)
    if excl:
        ctx.set_exclusions(n, exclusions)
    ctx.upload(pos, types=types, charge=charge)
    ctx.build_neighbor_list()
    alpha = co.ewald_alpha(rc) if coulomb else 0.0
    c6, c12 = co.lj_tables(eps, sig)
    want, scalars = co.forces(*pos.T, n, box, pairs, c6, c12, rc, charge=charge, types=types, switch=switch, do_coulomb=coulomb,
                              alpha=alpha, exclusions=exclusions)
    scale = max(np.abs(want).max(), 1e-12)
    for energy in (False, True):
        ctx.compute_forces(capi.PHASE_FULL, want_energy=energy)
        assert np.abs(ctx.forces_by_gid(n) - want).max() <= 2e-5 * scale
    got = ctx.read_scalars()
    assert abs(got["pe"] - scalars["pe"]) <= 1e-5 * max(abs(scalars["pe"]), 1.0)
    assert got["pairs_in_cutoff"] == scalars["pairs_in_cutoff"]
    ctx.close()


@pytest.mark.parametrize("n,L,rc,nt,coulomb", [(300, 20.0, 4.0, 1, False), (300, 20.0, 4.0, 3, True), (2500, 25.0, 6.0, 2, True)])
def test_atoms_that_coincide(cuda_device, n, L, rc, nt, coulomb):
    """Pairs at r^2 < 1e-10 exert nothing on each other, and the rest of their rows is as it would be without them."""
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    sites = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(side ** 3)[:n]]
    pos = ((sites + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * (L / side)) % L
    pos[10:20] = pos[:10]
    pos[30:40] = pos[20:30] + [4e-6, 0.0, 0.0]
    pos[50:60] = pos[40:50]   # three at a place, and rows that hold them from elsewhere
    pos[60:70] = pos[40:50]
    box, types = np.full(3, L), rng.integers(0, nt, n).astype(np.int32)
    charge = rng.uniform(-0.5, 0.5, n) if coulomb else np.zeros(n)
    eps, sig = np.full((nt, nt), 0.3), np.ones((nt, nt))
    ctx = capi.Context(n)
    ctx.set_box(box)
    ctx.set_pair_params(eps, sig, rc, 0.5)
    if coulomb:
        ctx.set_coulomb(True)
    ctx.upload(pos, types=types, charge=charge)
    ctx.build_neighbor_list()
    pairs = co.pairs(*pos.T, n, box, search=rc + 0.5)
    c6, c12 = co.lj_tables(eps, sig)
    want, scalars = co.forces(*pos.T, n, box, pairs, c6, c12, rc, charge=charge, types=types, do_coulomb=coulomb,
                              alpha=co.ewald_alpha(rc) if coulomb else 0.0)
    for energy in (False, True):
        ctx.compute_forces(capi.PHASE_FULL, want_energy=energy)
        assert np.abs(ctx.forces_by_gid(n) - want).max() <= 2e-5 * np.abs(want).max()
    got = ctx.read_scalars()
    assert abs(got["pe"] - scalars["pe"]) <= 1e-5 * max(abs(scalars["pe"]), 1.0)
    assert got["pairs_in_cutoff"] == scalars["pairs_in_cutoff"]
    ctx.close()


@pytest.mark.parametrize("n,rc", [(600, 4.0), (2500, 6.0)])
def test_charges_switched_on_and_off_under_one_list(cuda_device, n, rc):
    """The forms with and without Ewald read the rows of a list that either of them was built for (short rows, long rows)."""
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    sites = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(side ** 3)[:n]]
    pos, box, charge = (sites + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * (25.0 / side), np.full(3, 25.0), rng.uniform(-0.5, 0.5, n)
    pairs = co.pairs(*pos.T, n, box, search=rc + 0.5)
    c6, c12 = co.lj_tables([[0.3]], [[1.0]])
    for build_with in (False, True):
        ctx = capi.Context(n)
        ctx.set_box(box)
        ctx.set_pair_params([[0.3]], [[1.0]], rc, 0.5)
        ctx.set_coulomb(build_with)
        ctx.upload(pos, charge=charge)
        ctx.build_neighbor_list()
        for coulomb in (build_with, not build_with, build_with):
            ctx.set_coulomb(coulomb)
            ctx.compute_forces()
            want, _ = co.forces(*pos.T, n, box, pairs, c6, c12, rc, charge=charge, types=np.zeros(n, np.int32), do_coulomb=coulomb,
                                alpha=co.ewald_alpha(rc) if coulomb else 0.0)
            assert np.abs(ctx.forces_by_gid(n) - want).max() <= 2e-5 * np.abs(want).max()
        ctx.close()


@pytest.mark.parametrize("free", [False, True])
@pytest.mark.parametrize("shape", ["bond", "triangle", "chain"])
def test_constraint_shapes(cuda_device, shape, free):
    """Groups that are compiled for (two atoms, three atoms in a ring) and any other, with and without atoms outside every
    group: positions after the drift and velocities after the second half equal the oracle's."""
    ring = {"bond": [(0, 1)], "triangle": [(0, 1), (0, 2), (1, 2)], "chain": [(0, 1), (1, 2), (2, 3)]}[shape]
    size, groups, L, dt = {"bond": 2, "triangle": 3, "chain": 4}[shape], 65, 30.0, 1.0
    rng = np.random.default_rng(size)
    shapes = np.array([[0.0, 0.0, 0.0], [1.0, 0.1, 0.0], [0.3, 0.9, 0.0], [0.4, 1.0, 1.0]])[:size]
    centres = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)[:groups] * 6.0
    pos = (centres[:, None] + shapes[None]).reshape(-1, 3)
    constraints = np.array([(g * size + a, g * size + b, np.linalg.norm(shapes[a] - shapes[b])) for g in range(groups) for a, b in ring])
    if free:
        pos = np.concatenate([pos, rng.uniform(0, L, (7, 3))])
    n, box = len(pos), np.full(3, L)
    pos = pos % L
    mass = rng.uniform(1.0, 16.0, n)
    vel = rng.normal(scale=0.02, size=(n, 3))
    ctx = capi.Context(n)
    ctx.set_box(box)
    ctx.set_pair_params([[0.0]], [[1.0]], 3.0, 0.5)
    ctx.set_constraints(n, constraints)
    ctx.upload(pos, vel=vel, mass=mass)
    ctx.build_neighbor_list()
    gid = ctx.download("global_id", n)

    def fields(names):
        out = np.empty((n, 3))
        out[gid] = np.stack([ctx.download(k, n) for k in names], axis=1)
        return out

    pre = [np.ascontiguousarray(c) for c in pos.T]
    p = [np.ascontiguousarray(c) for c in (pos + dt * vel).T]
    v = [np.ascontiguousarray(c) for c in vel.T]
    ctx.integrate(1, dt)
    assert co.shake(constraints, p, v, mass, pre, box, dt)
    assert np.abs(fields("xyz") - np.stack(p, 1)).max() <= 1e-9
    assert np.abs(fields(("vx", "vy", "vz")) - np.stack(v, 1)).max() <= 1e-9
    ctx.integrate(2, dt)
    assert co.rattle(constraints, p, v, mass, box, dt, 1.0)[0]
    assert np.abs(fields(("vx", "vy", "vz")) - np.stack(v, 1)).max() <= 1e-9
    assert ctx.constraint_failures() == 0
    ctx.close()


# a warp per atom up to 32,768 atoms, a thread per atom beyond; slices of 32; rows of more than 1,024 edges per slice (the flat
# order in pieces); atoms outside the box
@pytest.mark.parametrize("n,density,outside", [(2, 0.05, False), (33, 0.05, True), (2000, 0.05, True), (1000, 0.6, False),
                                               (32768, 0.02, False), (32769, 0.02, True)])
def test_graphs_of_every_search_and_slice_form(cuda_device, n, density, outside):
    import torch
    rng = np.random.default_rng(n)
    cutoff = 4.0
    L = max((n / density) ** (1 / 3), 3.2 * cutoff)
    pos = rng.uniform(0, L, (n, 3))
    x, y, z = (torch.tensor(np.ascontiguousarray(c), device="cuda") for c in pos.T)
    eb = capi.EdgeBuilder()
    want, _ = co.edges(*pos.T, cutoff)
    got = eb.build(x, y, z, cutoff)[0].cpu().numpy()
    assert np.array_equal(got[:, np.lexsort(got[::-1])], want[:, np.lexsort(want[::-1])])
    moved = pos + (rng.integers(-1, 2, (n, 3)) * L if outside else 0.0)
    src, dst, shift, vec = (t.cpu().numpy() for t in eb.build_periodic(*[torch.tensor(np.ascontiguousarray(c), device="cuda") for c in moved.T],
                                                                       np.full(3, L), cutoff))
    half = co.pairs(*pos.T, n, np.full(3, L), search=cutoff)
    both = np.concatenate([half, half[:, ::-1]])
    order, order_want = np.lexsort((dst, src)), np.lexsort((both[:, 1], both[:, 0]))
    assert np.array_equal(np.stack([src, dst], 1)[order], both[order_want])
    assert np.abs(moved[dst] + shift * L - moved[src] - vec).max(initial=0.0) <= 1e-5
    eb.close()


@pytest.mark.parametrize("n,cells", [(500, 5), (256000, 40)])
def test_host_buffers_pinned_and_not(cuda_device, n, cells):
    """The host-buffer call by kernels that read the host's memory (few atoms), by slabs (many), and with memory that kernels
    cannot read: the same forces, bit for bit."""
    import torch
    from deepscalemd_b200 import synthetic as syn
    s = syn.fcc_lj(cells)
    assert s.n == n
    ctx = capi.Context(n)
    ctx.set_box(s.box)
    ctx.set_pair_params(s.eps, s.sig, s.cutoff, s.skin)
    ctx.upload(s.pos)
    ctx.build_neighbor_list()
    order = ctx.download("global_id")
    moved = s.pos[order] + np.random.default_rng(5).uniform(-0.08, 0.08, s.pos.shape)
    plain = [np.ascontiguousarray(c) for c in moved.T]
    ctx.upload_positions_ptr(*[c.ctypes.data for c in plain])
    ctx.pack_positions(0, None)
    ctx.compute_forces()
    want = [ctx.download(k) for k in ("fx", "fy", "fz")]
    pinned = [torch.from_numpy(c).pin_memory() for c in plain]
    out_pinned, out_plain = [torch.zeros(n, dtype=torch.float64).pin_memory() for _ in range(3)], [np.zeros(n) for _ in range(3)]
    ctx.forces_host(*[t.data_ptr() for t in pinned], *[t.data_ptr() for t in out_pinned])
    ctx.forces_host(*[c.ctypes.data for c in plain], *[c.ctypes.data for c in out_plain])
    for k in range(3):
        assert np.array_equal(out_pinned[k].numpy(), want[k]) and np.array_equal(out_plain[k], want[k])
    ctx.close()


@pytest.mark.parametrize("lagged", [False, True])
@pytest.mark.parametrize("n_cells,nt", [(5, 1), (8, 2), (8, 9)])
def test_loop_equals_step_by_step(cuda_device, n_cells, nt, lagged):
    """The MD loop (forces, both velocity halves and the drift in one kernel, the next step queued before the check is read)
    against the same steps through the single entry points."""
    from deepscalemd_b200 import synthetic as syn
    s = syn.fcc_lj(n_cells)
    types = np.arange(s.n, dtype=np.int32) % nt
    eps, sig = np.full((nt, nt), 1.0), np.full((nt, nt), 1.0)
    ends = []
    for loop in (True, False):
        ctx = capi.Context(s.n)
        ctx.set_box(s.box)
        ctx.set_pair_params(eps, sig, s.cutoff, s.skin)
        ctx.upload(s.pos, vel=s.vel, types=types)
        ctx.build_neighbor_list()
        ctx.compute_forces()
        if loop:
            ctx.run_nve(25, 0.004, lagged=lagged)
        else:
            for _ in range(25):
                ctx.integrate(1, 0.004)
                if ctx.max_displacement_sq() > (0.5 * s.skin) ** 2:
                    ctx.build_neighbor_list()
                ctx.compute_forces()
                ctx.integrate(2, 0.004)
        gid = ctx.download("global_id", s.n)
        out = np.empty((s.n, 6))
        out[gid] = np.stack([ctx.download(k, s.n) for k in ("x", "y", "z", "vx", "vy", "vz")], axis=1)
        ends.append(out)
        ctx.close()
    assert np.abs(ends[0] - ends[1]).max() <= 1e-4


# cell tables of one block of the scan, of eight and a few more (sums of blocks), of more than it takes (the library's scan)
@pytest.mark.parametrize("L,cells", [(14.0, 2916), (28.0, 27436), (38.0, 78732), (60.0, 296352), (126.0, 2819876)])
def test_lists_over_cell_tables_of_every_size(cuda_device, L, cells):
    n = 1500 if L > 14.0 else 700
    rng = np.random.default_rng(cells)
    pos, box = rng.uniform(0.0, L, (n, 3)), np.full(3, L)
    ctx = capi.Context(20000)
    ctx.set_box(box)
    ctx.set_pair_params([[1.0]], [[1.0]], 2.5, 0.3)
    for _ in range(2):   # the second build finds the counts as the first one left them
        ctx.upload(pos)
        ctx.build_neighbor_list()
        assert ctx.list_stats()["cells"] == cells
        i, j = ctx.list_pairs()[:2]
        gid = ctx.download("global_id", n)
        got = np.sort(np.stack([gid[np.asarray(i)], gid[np.asarray(j)]], 1), axis=1)
        want = np.sort(co.pairs(*pos.T, n, box, search=2.8), axis=1)
        got, want = np.unique(got, axis=0), np.unique(want, axis=0)
        assert np.array_equal(got, want)
        pos = rng.uniform(0.0, L, (n, 3))
    ctx.close()


def test_rebuild_with_longer_rows_inside_the_loop(cuda_device):
    """Atoms without forces that fall towards the middle of the box: the loop queues a step behind each list build, and where
    the rows turn out too short the step must not have happened."""
    n, L, dt, steps = 4000, 40.0, 0.01, 60
    rng = np.random.default_rng(7)
    pos = rng.uniform(0.0, L, (n, 3))
    vel = (L / 2 - pos) * 1.4
    ctx = capi.Context(n)
    ctx.set_box(np.full(3, L))
    ctx.set_pair_params([[0.0]], [[1.0]], 2.5, 0.6)
    ctx.upload(pos, vel=vel)
    ctx.build_neighbor_list()
    ctx.compute_forces()
    short = ctx.list_stats()["row_stride"]
    ctx.run_nve(steps, dt)
    assert ctx.list_stats()["row_stride"] > short
    gid = ctx.download("global_id", n)
    out = np.empty((n, 3))
    out[gid] = np.stack([ctx.download(k, n) for k in "xyz"], axis=1)
    d = out - (pos + vel * dt * steps)
    assert np.abs(d - L * np.round(d / L)).max() <= 1e-9
    ctx.close()


# the last block reports the check up to 25,000 threads, a launch behind it beyond
@pytest.mark.parametrize("n", [1000, 24999, 25001])
def test_displacement_checks_reported_by_block_and_by_launch(cuda_device, n):
    rng = np.random.default_rng(n)
    L = 60.0
    pos, vel, box = rng.uniform(0.0, L, (n, 3)), rng.normal(size=(n, 3)), np.full(3, L)
    ctx = capi.Context(n)
    ctx.set_box(box)
    ctx.set_pair_params([[0.0]], [[1.0]], 2.0, 0.5)
    ctx.upload(pos, vel=vel)
    ctx.build_neighbor_list()
    ctx.compute_forces()
    for k in range(1, 4):   # each check stands for itself and for the largest so far
        ctx.integrate(1, 0.01)
        want = ((k * 0.01 * vel) ** 2).sum(1).max()
        assert abs(ctx.max_displacement_sq() - want) <= 1e-9 * want
    ctx.close()


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n", [1, 3, 4097, 50000])
def test_uploaded_rows_are_the_callers_again_at_once(cuda_device, n, pinned):
    import torch
    rng = np.random.default_rng(n)
    rows = [rng.uniform(0.0, 20.0, (n, 3)) for _ in range(2)]
    given = [torch.from_numpy(r.copy()).pin_memory().numpy() if pinned else r.copy() for r in rows]
    ctx = capi.Context(n + 5)
    ctx.set_box(np.full(3, 20.0))
    ctx.set_pair_params([[1.0]], [[1.0]], 2.0, 0.5)
    for _ in range(2):   # the second upload goes through the set of arrays that the first one's sort left behind
        for g, r in zip(given, rows):
            g[:] = r
        ctx.upload(given[0], vel=given[1])
        for g in given:
            g[:] = -1.0
        if n > 1:
            ctx.build_neighbor_list()
        gid = ctx.download("global_id", n)
        for names, want in (("xyz", rows[0]), (("vx", "vy", "vz"), rows[1])):
            assert np.array_equal(np.stack([ctx.download(k, n) for k in names], axis=1), want[gid])
    ctx.close()


@pytest.mark.parametrize("n,vel", [(1000, False), (16384, True), (32768, False)])
@pytest.mark.parametrize("pinned", [False, True])
def test_few_rows_are_uploaded_without_waiting_for_the_stream(cuda_device, n, vel, pinned):
    import ctypes
    import torch
    rng = np.random.default_rng(n)
    given = [torch.from_numpy(rng.uniform(0.0, 20.0, (n, 3))) for _ in range(2)]
    given = [(g.pin_memory() if pinned else g).numpy() for g in given]
    want = [g.copy() for g in given]
    ctx = capi.Context(n)
    stream = torch.cuda.Stream()

    def upload():
        pos, velocities = (ctypes.c_void_p(g.ctypes.data) for g in given)
        assert ctx.lib.dsmd_upload_rows(ctx.h, ctypes.c_int64(n), ctypes.c_int64(n), pos, velocities if vel else None, None, None, None, None,
                                        ctypes.c_void_p(stream.cuda_stream)) == 0

    upload()   # allocations
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)   # 0.1 s
    upload()
    assert not stream.query()
    for g in given:
        g[:] = -1.0
    torch.cuda.synchronize()
    for names, rows in (("xyz", want[0]), (("vx", "vy", "vz"), want[1] if vel else np.zeros((n, 3)))):
        assert np.array_equal(np.stack([ctx.download(k, n) for k in names], axis=1), rows)
    ctx.close()


@pytest.mark.parametrize("first,last", [(0.4, 0.6), (0.0, 0.5), (0.5, 1.0), (0.0, 1.0)])
def test_rows_of_memory_registered_in_part(cuda_device, first, last):
    import ctypes
    import mmap
    import torch
    n = 60000
    memory = mmap.mmap(-1, 24 * n)   # whole pages
    rows = np.frombuffer(memory, np.float64).reshape(n, 3)
    want = np.random.default_rng(5).uniform(0.0, 20.0, (n, 3))
    rows[:] = want
    lo, hi = int(first * rows.nbytes) // 4096 * 4096, rows.nbytes if last == 1.0 else int(last * rows.nbytes) // 4096 * 4096
    runtime = torch.cuda.cudart()
    assert int(runtime.cudaHostRegister(rows.ctypes.data + lo, hi - lo, 0)) == 0
    ctx = capi.Context(n)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)
    assert ctx.lib.dsmd_upload_rows(ctx.h, ctypes.c_int64(n), ctypes.c_int64(n), ctypes.c_void_p(rows.ctypes.data), None, None, None, None, None,
                                    ctypes.c_void_p(stream.cuda_stream)) == 0
    rows[:] = -1.0
    torch.cuda.synchronize()
    assert int(runtime.cudaHostUnregister(rows.ctypes.data + lo)) == 0
    assert np.array_equal(np.stack([ctx.download(k, n) for k in "xyz"], axis=1), want)
    ctx.close()


# types, Coulomb, exclusions, atoms at one place, pairs below the Ewald table
LONG_ROWS_WITH_GHOSTS = [(1, False, False, False, False), (2, False, True, False, False), (9, False, False, True, False), (1, True, False, False, True),
                         (2, True, True, False, False), (3, True, False, True, True)]


@pytest.mark.parametrize("dims", [(2, 1, 1), (2, 2, 1)])
@pytest.mark.parametrize("nt,coulomb,excl,coincide,close", LONG_ROWS_WITH_GHOSTS)
def test_long_rows_with_ghosts(cuda_device, nt, coulomb, excl, coincide, close, dims):
    """Rows of 240 entries and more (groups of 16 entries, four lanes and more per row) that end in ghosts: all at once, and first the
    owned partners and then the ghosts, with and without sums, brick by brick against the undivided system."""
    from deepscalemd_b200 import synthetic as syn
    n, L, rc, skin = 3000, 26.0, 6.5, 0.5
    rng = np.random.default_rng(nt + 10 * coulomb)
    side = int(np.ceil(n ** (1 / 3)))
    sites = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(side ** 3)[:n]]
    pos, box = ((sites + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * (L / side)) % L, np.full(3, L)
    near = np.argsort(np.abs(pos[:, 0] - L / 2))   # of the face between the bricks
    touched = np.zeros(n, bool)
    if coincide:
        pos[near[40:48]] = pos[near[:8]]
        touched[near[:8]] = touched[near[40:48]] = True
    if close:
        a, b = near[100:108], near[140:148]
        pos[a, 0] = L / 2 - rng.uniform(0.1, 0.3, 8)
        pos[b] = pos[a] + [0.6, 0.0, 0.0]
        touched[a] = touched[b] = True
    types, charge = rng.integers(0, nt, n).astype(np.int32), rng.uniform(-0.5, 0.5, n) if coulomb else np.zeros(n)
    eps, sig = np.full((nt, nt), 0.3), np.full((nt, nt), 0.5)
    sig += 0.05 * np.add.outer(np.arange(nt), np.arange(nt)) / nt
    pairs = co.pairs(*pos.T, n, box, search=rc + skin)
    exclusions = pairs[:: 7] if excl else None
    c6, c12 = co.lj_tables(eps, sig)
    want, scalars = co.forces(*pos.T, n, box, pairs, c6, c12, rc, charge=charge, types=types, do_coulomb=coulomb,
                              alpha=co.ewald_alpha(rc) if coulomb else 0.0, exclusions=exclusions)

    def check(got, atom):
        for mask in (touched[atom], ~touched[atom]):   # (what touches feels far more than the others)
            if mask.any():
                assert np.abs(got[mask] - want[atom[mask]]).max() <= 2e-5 * np.abs(want[atom[mask]]).max()

    pe = counted = 0.0
    halo = rc + skin + 0.2
    for brick in syn.brick_decompose(pos, box, dims, halo):
        own, src, img = brick["owned"], brick["ghost_src"], brick["ghost_image"]
        place, atom = np.concatenate([pos[own], pos[src] + img * box]), np.concatenate([own, src])
        ctx = capi.Context(len(atom))
        ctx.set_box(box, (1, 1, 1), brick["lo"], brick["hi"], halo)
        ctx.set_pair_params(eps, sig, rc, skin)
        if coulomb:
            ctx.set_coulomb(True)
        if excl:
            ctx.set_exclusions(n, exclusions)
        ctx.upload(place, n_owned=len(own), types=types[atom], charge=charge[atom], gid=atom.astype(np.int32))
        ctx.build_neighbor_list()
        assert ctx.list_stats()["row_stride"] >= 240
        i, j = ctx.list_pairs()[:2]
        here = ctx.download("global_id", len(atom))
        assert ctx.list_stats()["interior_entries"] == int((np.asarray(j) < len(own)).sum()) < len(j)
        for energy in (False, True):
            for phases in ((capi.PHASE_INTERIOR, capi.PHASE_BOUNDARY), (capi.PHASE_FULL,)):
                for phase in phases:
                    ctx.compute_forces(phase, want_energy=energy)
                check(np.stack([ctx.download(k, len(own)) for k in ("fx", "fy", "fz")], axis=1), here[:len(own)])
                if energy:
                    sums = ctx.read_scalars()
                    if len(phases) == 2:
                        parts = sums
        assert abs(parts["pe"] - sums["pe"]) <= 1e-6 * abs(sums["pe"]) and parts["pairs_in_cutoff"] == sums["pairs_in_cutoff"]
        pe += sums["pe"]
        counted += sums["pairs_in_cutoff"]
        ctx.close()
    # charges of either sign all but cancel in the sum: a rounding of single precision per term, of terms of up to 332 / 4 / 1.4
    # at random signs, each counted twice at half
    cancelled = 2.0 ** -24 * 60.0 * np.sqrt(2.0 * counted) if coulomb else 0.0
    assert abs(pe - scalars["pe"]) <= 1e-5 * abs(scalars["pe"]) + cancelled
    # a pair within a rounding of single precision of the cutoff counts or not: 2^-23 of 295,000 pairs, half as many again per unit of
    # ln r^2, are 0.05 per system (one here lies 5e-9 inside)
    assert abs(counted - scalars["pairs_in_cutoff"]) <= 1


def after_steps(make, steps, dt, f2a=1.0, hi_frac=0.5, lagged=None, bonded=False):
    """Places and velocities after some steps, by run_nve or (lagged None) through the single entry points; and the rebuilds."""
    ctx, limit = make()
    ctx.build_neighbor_list()
    ctx.compute_forces()
    if bonded:
        ctx.compute_bonded()
    rebuilds = 0
    if lagged is not None:
        rebuilds = ctx.run_nve(steps, dt, f2a, hi_frac, 0, lagged)["rebuilds"]
    else:
        for _ in range(steps):
            ctx.integrate(1, dt, f2a)
            if ctx.max_displacement_sq() > (hi_frac * limit) ** 2:
                ctx.build_neighbor_list()
                rebuilds += 1
            ctx.compute_forces()
            if bonded:
                ctx.compute_bonded()
            ctx.integrate(2, dt, f2a)
    n = ctx.counts()[0]
    gid = ctx.download("global_id", n)
    out = np.empty((n, 6))
    out[gid] = np.stack([ctx.download(k, n) for k in ("x", "y", "z", "vx", "vy", "vz")], axis=1)
    stride = ctx.list_stats()["row_stride"]
    ctx.close()
    return out[:, :3], out[:, 3:], rebuilds, stride


def assert_same_run(make, steps, dt, rebuilds_least, tolerance=1e-6, **kwargs):
    """The loop sums the same forces in the same order as the single calls, over lists built at the same steps: what is left are
    the roundings of two half kicks against one whole (2^-53), multiplied by the system's own divergence."""
    want, got = after_steps(make, steps, dt, **kwargs), after_steps(make, steps, dt, lagged=False, **kwargs)
    assert got[2] == want[2] >= rebuilds_least
    for g, w in zip(got[:2], want[:2]):
        assert np.abs(g - w).max() <= tolerance * np.abs(w).max()
    return got


def test_longer_rows_inside_the_loop_with_forces(cuda_device):
    """Atoms that interact and fall towards the middle of the box: where the rows turn out too short, the step queued behind the list
    build must not have happened, and the next one must read the places that it would have read."""
    side, L = 14, 40.0
    rng = np.random.default_rng(8)
    pos = (np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(-0.1, 0.1, (side ** 3, 3))) * 1.7 + 8.0
    vel = (L / 2 - pos) * 0.6

    def make():
        ctx = capi.Context(len(pos))
        ctx.set_box(np.full(3, L))
        ctx.set_pair_params([[1.0]], [[0.8]], 2.5, 0.6)
        ctx.upload(pos, vel=vel)
        return ctx, 0.6

    ctx, _ = make()
    ctx.build_neighbor_list()
    short = ctx.list_stats()["row_stride"]
    ctx.close()
    _, _, _, stride = assert_same_run(make, 120, 0.005, 3)
    assert stride > short


@pytest.mark.parametrize("side,free", [(12, False), (12, True), (38, False)])   # 38: more than 25,000 groups
def test_loop_with_constraints_equals_step_by_step(cuda_device, side, free):
    rng = np.random.default_rng(side)
    sites = (np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * 2.2
    u = rng.normal(size=sites.shape)
    u *= 0.45 / np.linalg.norm(u, axis=1, keepdims=True)
    groups = len(sites) * 2 // 3 if free else len(sites)
    pos = np.concatenate([np.stack([sites[:groups] - u[:groups], sites[:groups] + u[:groups]], 1).reshape(-1, 3), sites[groups:]])
    n, box = len(pos), np.full(3, side * 2.2)
    mates = np.arange(2 * groups, dtype=np.int32).reshape(-1, 2)
    vel = rng.normal(scale=1.2, size=(n, 3))
    vel[:2 * groups] = np.repeat(vel[:groups], 2, axis=0)

    def make():
        ctx = capi.Context(n)
        ctx.set_box(box)
        ctx.set_pair_params([[1.0]], [[0.9]], 2.5, 0.4)
        ctx.set_exclusions(n, mates)
        ctx.set_constraints(n, np.concatenate([mates, np.full((groups, 1), 0.9)], axis=1))
        ctx.upload(pos % box, vel=vel)
        return ctx, 0.4

    # SHAKE stops at a relative error of 1e-8 of the squared length, from places that differ by their roundings
    assert_same_run(make, 60, 0.004, 2, tolerance=1e-5)


def test_loop_with_constrained_water_equals_step_by_step(cuda_device):
    from deepscalemd_b200 import synthetic as syn
    s = syn.water_box(11, seed=5)

    def make():
        ctx = capi.Context(s.n)
        ctx.set_box(s.box)
        ctx.set_pair_params(s.eps, s.sig, s.cutoff, s.skin)
        ctx.set_coulomb(True)
        ctx.set_exclusions(s.n, s.exclusions)
        ctx.set_constraints(s.n, s.constraints)
        ctx.upload(s.pos, vel=s.vel, mass=s.mass, types=s.types, charge=s.charge)
        return ctx, s.skin

    assert_same_run(make, 60, 2.0, 2, tolerance=1e-5, f2a=4.184e-4, hi_frac=0.1)


def test_loop_with_bonded_terms_equals_step_by_step(cuda_device):
    from deepscalemd_b200 import synthetic as syn
    s = syn.chain_fluid(4, 8, spacing=14.0, seed=12)   # (closer ones overlap)

    def make():
        ctx = capi.Context(s.n)
        ctx.set_box(s.box)
        ctx.set_pair_params(s.eps, s.sig, s.cutoff, s.skin)
        ctx.set_coulomb(True)
        ctx.set_exclusions(s.n, s.exclusions)
        ctx.set_bonded(s.n, s.bonded)
        ctx.upload(s.pos, vel=s.vel, mass=s.mass, types=s.types, charge=s.charge)
        return ctx, s.skin

    assert_same_run(make, 80, 0.5, 2, f2a=s.force_to_accel, hi_frac=0.1, bonded=True)


def test_loop_of_many_threads_equals_step_by_step(cuda_device):
    """More than 25,000 threads: checks reported by a launch of their own, behind the loop's kernel and behind the single calls'."""
    from deepscalemd_b200 import synthetic as syn
    s = syn.fcc_lj(20)

    def make():
        ctx = capi.Context(s.n)
        ctx.set_box(s.box)
        ctx.set_pair_params(s.eps, s.sig, s.cutoff, s.skin)
        ctx.upload(s.pos, vel=s.vel)
        return ctx, s.skin

    assert_same_run(make, 40, 0.004, 2)


@pytest.mark.parametrize("system", ["lj_864", "lj_32000", "water", "chains"])
def test_captured_steps_equal_the_calls(cuda_device, system):
    """A whole step captured into a graph (kernels that overlap become programmatic edges) and replayed, against the same calls."""
    import torch
    from deepscalemd_b200 import synthetic as syn
    s = {"lj_864": lambda: syn.fcc_lj(6), "lj_32000": lambda: syn.fcc_lj(20), "water": lambda: syn.water_box(11, seed=6),
         "chains": lambda: syn.chain_fluid(4, 8, spacing=14.0, seed=15)}[system]()
    dt, f2a = {"water": (1.0, 4.184e-4), "chains": (0.5, getattr(s, "force_to_accel", 1.0))}.get(system, (0.002, 1.0))
    ends = []
    for captured in (False, True):
        ctx = capi.Context(s.n)
        ctx.set_box(s.box)
        ctx.set_pair_params(s.eps, s.sig, s.cutoff, s.skin)
        if s.coulomb:
            ctx.set_coulomb(True)
        if s.exclusions is not None:
            ctx.set_exclusions(s.n, s.exclusions)
        if system == "water":
            ctx.set_constraints(s.n, s.constraints)
        if system == "chains":
            ctx.set_bonded(s.n, s.bonded)
        ctx.upload(s.pos, vel=s.vel, mass=s.mass, types=s.types, charge=s.charge)
        ctx.build_neighbor_list()
        stream = torch.cuda.Stream()

        def step():
            ctx.integrate(1, dt, f2a, stream=stream)
            ctx.compute_forces(stream=stream)
            if system == "chains":
                ctx.compute_bonded(stream=stream)
            ctx.integrate(2, dt, f2a, stream=stream)

        ctx.compute_forces(stream=stream)
        if system == "chains":
            ctx.compute_bonded(stream=stream)
        step()   # allocations, and the maps from ids to slots
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        if captured:
            with torch.cuda.graph(graph, stream=stream):
                step()
                step()
        for _ in range(4):
            if captured:
                graph.replay()
            else:
                step()
                step()
        torch.cuda.synchronize()
        moved = ctx.max_displacement_sq()
        gid = ctx.download("global_id", s.n)
        out = np.empty((s.n, 9))
        out[gid] = np.stack([ctx.download(k, s.n) for k in ("x", "y", "z", "vx", "vy", "vz", "fx", "fy", "fz")], axis=1)
        ends.append((out, moved))
        del graph
        ctx.close()
    assert np.array_equal(ends[0][0], ends[1][0]) and ends[0][1] == ends[1][1] > 0.0
