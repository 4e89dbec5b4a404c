"""F_s shells at the edges of the kernels' blocks against the FP64 oracle: vector
lists are summed in blocks of 32 terms (whole blocks and a remainder), octant
representatives likewise, by one or by two atoms per thread, and octant tables that
do not fit a block with two atoms (or any) take the narrower path.  Tolerance: that
of the normalised F_s everywhere, 1e-6 absolute."""
import numpy as np
import pytest

from amdat_gb300 import synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

BOX = 16.0


def _compare(eng, n_atoms, kv, off, steps=3):
    scheme = synth.TimeScheme.exponential(2, steps, 1.4, 0, 0, 0.005)
    traj = synth.random_walk(n_atoms, BOX, scheme, 0.5, seed=n_atoms)
    eng.upload(traj.unwrapped, traj.box)
    eng.set_scheme(scheme)
    out = eng.disp(0, shells=(kv, off), period=BOX)
    ref = orc.isfs(orc.scheme(scheme), traj.unwrapped, np.arange(n_atoms, dtype=np.int32), kv, off,
                   2.0 * np.pi / BOX, BOX, 0, orc.F64)
    m = out["atom_pairs"] > 0
    got = out["fs_sum"][m] / out["atom_pairs"][m][:, None]
    assert np.abs(got - ref[m]).max() <= 1e-6


@pytest.mark.parametrize("counts", [(1, 31, 32, 33), (64, 65, 95, 96, 97), (2049, 3)])
def test_vector_list_blocks(eng, counts):
    rng = np.random.default_rng(sum(counts))
    kv = rng.integers(-20, 21, (sum(counts), 3)).astype(np.int32)
    kv[:, 0] = 3 + np.arange(len(kv)) % 17  # never closed under the sign of x: list mode
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    _compare(eng, 300, kv, off)


def _closed(reps):
    """All sign images of the representatives."""
    signs = np.array([[x, y, z] for x in (1, -1) for y in (1, -1) for z in (1, -1)])
    return np.unique((np.asarray(reps)[:, None] * signs[None]).reshape(-1, 3), axis=0).astype(np.int32)


# 128 threads a block: items of one step, of one step and a bit, of odd step counts
@pytest.mark.parametrize("n_atoms", [1, 127, 129, 255, 257, 385, 900])
@pytest.mark.parametrize("steps", [2, 12])
def test_octant_blocks(eng, n_atoms, steps):
    rng = np.random.default_rng(n_atoms)
    grid = np.stack(np.meshgrid(np.arange(9), np.arange(9), np.arange(9), indexing="ij"), -1).reshape(-1, 3)
    rng.shuffle(grid)
    cuts = np.cumsum([0, 1, 31, 32, 33, 64, 65])
    shells = [_closed(grid[a:b]) for a, b in zip(cuts[:-1], cuts[1:])] + [np.zeros((1, 3), np.int32)]
    off = np.concatenate([[0], np.cumsum([len(s) for s in shells])]).astype(np.int32)
    _compare(eng, n_atoms, np.concatenate(shells), off, steps)


# the largest component decides the tables' size: two atoms per thread in one to several
# blocks per SM, 2,600 representatives, and the largest octant table
@pytest.mark.parametrize("top,n_rep", [(0, 1), (3, 20), (24, 200), (36, 100), (40, 2600), (48, 2600), (48, 5300)])
def test_octant_tables(eng, top, n_rep):
    rng = np.random.default_rng(top + n_rep)
    reps = np.unique(rng.integers(0, top + 1, (n_rep, 3)), axis=0)
    reps[-1] = top
    kv = _closed(np.unique(reps, axis=0))
    _compare(eng, 600, kv, np.array([0, len(kv)], np.int32))
