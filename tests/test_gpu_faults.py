"""GPU tests of single faults that were found by reading: each one fails with the fault it names."""
import numpy as np
import pytest

from deepscalemd_b200 import capi
from oracle import cpu_oracle as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("owned", [3, 4, 7])
@pytest.mark.parametrize("seed", range(6))
def test_rows_whose_first_stranger_is_a_ghost(cuda_device, owned, seed):
    """A few owned atoms in one cell row, all within each other's reach, and ghosts beyond it: the owned part of a row has no
    atom outside the list radius to fill its last chunk with, the ghost part meets one. Nobody may be counted twice."""
    rng = np.random.default_rng(100 * owned + seed)
    L, rc, skin, face = 40.0, 2.5, 0.3, 20.0
    halo = rc + skin + 0.2
    # spacing 0.9 along x, the last atom close to the face; the seventh atom is the first one's neighbour across
    own = np.stack([face - 0.3 - 0.9 * np.arange(owned)[::-1], np.full(owned, 10.5), np.full(owned, 10.5)], 1)
    if owned == 7:
        own = np.concatenate([own[3:], own[4:] + [0.0, 0.0, 1.0]])
    own += rng.uniform(-0.05, 0.05, own.shape)
    ghosts = np.empty((0, 3))
    while len(ghosts) < 14:
        p = np.array([face, 8.0, 8.0]) + rng.uniform(0.1, 1.0, 3) * [halo, 5.0, 5.0]
        if np.linalg.norm(np.concatenate([own, ghosts]) - p, axis=1).min() > 0.95:
            ghosts = np.concatenate([ghosts, p[None]])
    pos, n, box = np.concatenate([own, ghosts]), len(own), np.full(3, L)
    ctx = capi.Context(len(pos))
    ctx.set_box(box, (1, 1, 1), (0.0, 0.0, 0.0), (face, L, L), halo)
    ctx.set_pair_params([[1.0]], [[1.0]], rc, skin)
    ctx.upload(pos, n_owned=n, gid=np.arange(len(pos), dtype=np.int32))
    ctx.build_neighbor_list()
    pairs = co.pairs(*pos.T, n, box, split=(1, 0, 0), search=rc + skin)
    want, scalars = co.forces(*pos.T, n, box, pairs, *co.lj_tables([[1.0]], [[1.0]]), rc, split=(1, 0, 0))
    for phases in ((capi.PHASE_FULL,), (capi.PHASE_INTERIOR, capi.PHASE_BOUNDARY)):
        for phase in phases:
            ctx.compute_forces(phase, want_energy=True)
        assert np.abs(ctx.forces_by_gid(n) - want).max() <= 1e-5 * np.abs(want).max()
        assert ctx.read_scalars()["pairs_in_cutoff"] == _owned_share(pairs, pos, box, rc, n)
    ctx.close()


def _owned_share(pairs, pos, box, rc, n):
    """Pairs inside the cutoff, those with a ghost counted half."""
    d = pos[pairs[:, 0]] - pos[pairs[:, 1]]
    d[:, 1:] -= box[1:] * np.rint(d[:, 1:] / box[1:])
    inside = (d * d).sum(1) < rc * rc
    return 0.5 * (2 * inside.sum() - (inside & (pairs.max(1) >= n)).sum())
