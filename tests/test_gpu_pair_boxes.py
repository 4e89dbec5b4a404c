"""The cell pass of ordered pair histograms in boxes that lie anywhere and with wrapped
coordinates that are not quite in the box, and lists too sparse for compact groups: the
counts equal the all-pairs pass's."""
import numpy as np
import pytest

from amdat_gb300 import synth

pytestmark = pytest.mark.gpu


def _both(eng, monkeypatch, l1, l2, max_d, nb):
    monkeypatch.delenv("AMDAT_PAIR_CELLS", raising=False)
    got = eng.vhd(l1, l2, max_d, nb)
    monkeypatch.setenv("AMDAT_PAIR_CELLS", "off")
    want = eng.vhd(l1, l2, max_d, nb)
    monkeypatch.delenv("AMDAT_PAIR_CELLS")
    assert want.sum() > 0
    return got, want


@pytest.mark.parametrize("lo", [(0.0, 0.0, 0.0), (1000.0, -3e3, 2e4), (1e5, -1e5, 3e5), (-1e6, 0.0, 1e6)])
@pytest.mark.parametrize("max_d", [1.9, 4.9])
def test_vhd_cells_far_origin(eng, monkeypatch, lo, max_d):
    """The spacing of FP32 numbers at the origin is up to 2^-4, far above the cutoff's margin."""
    rng = np.random.default_rng(int(max_d))
    L, n = np.array([15.0, 18.0, 30.0], np.float32), 6000
    lo = np.array(lo, np.float32)
    u = (lo + rng.random((3, n, 3)) * L).astype(np.float32)
    eng.upload(u, L, lo)
    eng.set_scheme(synth.TimeScheme.linear(3, 1.0))
    few, many = eng.list(np.arange(0, n, 40)), eng.list(np.setdiff1d(np.arange(n), np.arange(0, n, 40)))
    for l1, l2 in ((0, 0), (few, many), (many, 0)):
        got, want = _both(eng, monkeypatch, l1, l2, max_d, 49)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("out,cells", [(1e-5, True), (1e-2, True), (0.4, True), (1.8, True), (3.5, False)])
def test_vhd_cells_outside_the_box(eng, monkeypatch, out, cells):
    """Wrapped coordinates up to an eighth of the box outside it stay with the cell pass."""
    rng = np.random.default_rng(3)
    L, n = np.array([15.0, 16.0, 27.0], np.float32), 6000
    w = (rng.random((3, n, 3)) * (L + 2 * out) - out).astype(np.float32)
    eng.upload(w, L, wrapped=w)
    eng.set_scheme(synth.TimeScheme.linear(3, 1.0))
    some = eng.list(np.arange(0, n, 2))
    for l1, l2 in ((0, 0), (some, 0), (0, some)):
        eng.profile_reset()
        eng.vhd(l1, l2, 4.9, 49)
        assert (eng.profile_kernel("pair_hist_kernel")[0] == 0) == cells
        got, want = _both(eng, monkeypatch, l1, l2, 4.9, 49)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n,box,max_d", [(40000, 34.0, 1.0), (1024, 300.0, 0.9), (30000, (200.0, 9.5, 3.2), 1.05)])
def test_vhd_cells_many_cells(eng, monkeypatch, n, box, max_d):
    """More cells than the scan takes at a time, and mostly empty ones."""
    rng = np.random.default_rng(n)
    L = np.broadcast_to(np.float32(box), 3).astype(np.float32)
    eng.upload((rng.random((2, n, 3)) * L).astype(np.float32), L)
    eng.set_scheme(synth.TimeScheme.linear(2, 1.0))
    for l1, l2 in ((0, 0), (eng.list(np.arange(1, n, 9)), 0)):
        monkeypatch.delenv("AMDAT_PAIR_CELLS", raising=False)
        got = eng.vhd(l1, l2, max_d, 30)
        monkeypatch.setenv("AMDAT_PAIR_CELLS", "off")
        np.testing.assert_array_equal(got, eng.vhd(l1, l2, max_d, 30))


@pytest.mark.parametrize("frames,n1,max_d,walk", [(2, 2, 3.0, True), (2, 33, 5.0, True), (40, 200, 1.5, True),
                                                  (40, 1100, 1.1, True), (2, 30000, 5.0, False), (2, 1, 5.0, False)])
def test_vhd_few_atoms_to_many(eng, monkeypatch, frames, n1, max_d, walk):
    """A few atoms among many (32, 8 and 1 lanes each) walk the cells around them: groups of
    atoms far apart would gather the whole box."""
    rng = np.random.default_rng(n1)
    n, L = 30000, 33.0
    u = (rng.random((1, n, 3)) * L + np.cumsum(rng.normal(0, 0.05, (frames, n, 3)), 0)).astype(np.float32)
    eng.upload(u, [L] * 3)
    eng.set_scheme(synth.TimeScheme.linear(frames, 1.0))
    perm = rng.permutation(n)
    few, rest = eng.list(np.sort(perm[:n1])), eng.list(np.sort(perm[min(n1, n - 2000):]))
    for l2 in (rest, 0):
        eng.profile_reset()
        eng.vhd(few, l2, max_d, 40)
        assert (eng.profile_kernel("pair_hist_walk_kernel")[0] == 1) == walk or l2 != 0
        got, want = _both(eng, monkeypatch, few, l2, max_d, 40)
        np.testing.assert_array_equal(got, want)


def test_vhd_walk_of_one_list(eng, monkeypatch):
    """One list on both sides: its frames are sorted once; no atom pairs with itself."""
    rng = np.random.default_rng(5)
    n, L = 30000, 54.5
    u = (rng.random((1, n, 3)) * L + np.cumsum(rng.normal(0, 0.1, (2, n, 3)), 0)).astype(np.float32)
    eng.upload(u, [L] * 3)
    eng.set_scheme(synth.TimeScheme.linear(2, 1.0))
    for lst in (0, eng.list(np.arange(0, n, 2))):
        eng.profile_reset()
        eng.vhd(lst, lst, 2.0, 26)
        assert eng.profile_kernel("pair_hist_walk_kernel")[0] == 1
        got, want = _both(eng, monkeypatch, lst, lst, 2.0, 26)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("mb", [0, 1, 3])
@pytest.mark.parametrize("max_d", [1.0, 3.0])
def test_vhd_cells_in_batches_of_frames(eng, monkeypatch, mb, max_d):
    """Cell tables over the limit: the time pairs run in batches of frames, one frame of
    each side at least, and give the same counts."""
    rng = np.random.default_rng(mb)
    n, L, T = 9000, 24.0, 11
    u = (rng.random((1, n, 3)) * L + np.cumsum(rng.normal(0, 0.1, (T, n, 3)), 0)).astype(np.float32)
    eng.upload(u, [L] * 3)
    eng.set_scheme(synth.TimeScheme.linear(T, 1.0))
    half, few = eng.list(np.arange(0, n, 2)), eng.list(np.arange(7, n, 300))
    for l1, l2 in ((0, 0), (half, 0), (few, 0), (half, half)):
        monkeypatch.delenv("AMDAT_PAIR_SCRATCH_MB", raising=False)
        eng.profile_reset()
        want = eng.vhd(l1, l2, max_d, 40)
        assert eng.profile_kernel("pair_hist_cells_kernel")[0] == 1 and want.sum() > 0
        monkeypatch.setenv("AMDAT_PAIR_SCRATCH_MB", str(mb))
        eng.profile_reset()
        np.testing.assert_array_equal(eng.vhd(l1, l2, max_d, 40), want)
        assert mb == 3 or eng.profile_kernel("pair_hist_cells_kernel")[0] > 1


def test_vhd_cells_scratch_is_bounded(engine_mod, monkeypatch):
    import torch
    monkeypatch.setenv("AMDAT_PAIR_SCRATCH_MB", "64")
    rng = np.random.default_rng(1)
    n, L, T = 200000, 62.0, 40
    eng = engine_mod.Engine(0)
    try:
        eng.upload((rng.random((1, n, 3)) * L + rng.normal(0, 0.1, (T, n, 3))).astype(np.float32), [L] * 3)
        eng.set_scheme(synth.TimeScheme.linear(T, 1.0))
        free = torch.cuda.mem_get_info()[0]
        eng.vhd(0, 0, 1.5, 40)
        assert free - torch.cuda.mem_get_info()[0] < 100 << 20
    finally:
        eng.close()
