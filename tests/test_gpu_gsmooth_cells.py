"""The smoothed histogram's cell kernels and their cell lists against the FP64 oracle:
exactly three and unequal numbers of cells per axis (every pair of cells met once), the
smallest list that uses cells and ragged last blocks, both lane splits, empty cells and
cells of several warps of atoms, an index list, coarse bins (no recurrence) and a cutoff
that leaves some pairs out of every bin.  Tolerances: forward 1e-4 of the largest bin,
gradient 5e-4 of its largest component (those of the kernels' other cases)."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


# box, atoms, (sigma, r_max, bins), layout; the cutoff is r_max + 6 sigma
CASES = [([12.5, 12.5, 12.5], 1024, (0.02, 4.0, 400), "uniform"),
         ([12.5, 17.0, 21.5], 1025, (0.02, 4.0, 400), "uniform"),
         ([30.0, 13.0, 13.0], 1151, (0.02, 4.0, 400), "slab"),
         ([14.0, 14.0, 14.0], 2000, (0.02, 4.0, 37), "uniform"),
         ([9.0, 9.0, 9.0], 3000, (0.05, 2.0, 200), "blob"),
         ([20.0, 20.0, 20.0], 5001, (0.02, 4.0, 400), "list"),
         ([40.0, 40.0, 40.0], 39999, (0.02, 1.5, 150), "uniform"),
         ([40.0, 40.0, 40.0], 40001, (0.02, 1.5, 150), "uniform")]


@pytest.mark.parametrize("box,n,par,layout", CASES)
def test_cells_match_oracle(eng, box, n, par, layout):
    rng = np.random.default_rng(n)
    pos = rng.random((1, n, 3)) * box
    if layout == "slab":  # most cells empty
        pos[..., 0] *= 0.2
    if layout == "blob":  # one cell with hundreds of atoms
        pos[:, ::4] = 1.0 + rng.random((1, len(pos[0, ::4]), 3))
    pos = pos.astype(np.float32)
    eng.upload(pos, box, box_lo=[0.0, 0.0, 0.0], wrapped=pos)
    lst = np.arange(n, dtype=np.int32)
    h = 0
    if layout == "list":
        lst = lst[lst % 3 != 1]
        h = eng.list(lst)
    w = np.random.default_rng(3).standard_normal(par[2])
    assert _rel(eng.gsmooth(h, [0], *par), orc.gsmooth(pos, box, lst, [0], *par)) <= 1e-4
    g = eng.gsmooth_adjoint(h, [0], *par, w, len(lst))
    assert _rel(g, orc.gsmooth_grad(pos, box, lst, [0], *par, w)) <= 5e-4
