"""Pair histograms at the edges of the all-pairs pass: lists around its block (256 I
members) and segment sizes, lists that overlap, bins whose edges the distances sit
on, atoms at one place.  Counts equal the reference's FP32 chain (a numpy
restatement of it in the same order of operations) exactly."""
import numpy as np
import pytest

from amdat_gb300 import synth

pytestmark = pytest.mark.gpu


def _counts(wa, wb, ids_a, ids_b, L, max_d, nb):
    out = np.zeros(nb, np.int64)
    bs = np.float32(np.float32(max_d) / np.float32(nb))
    for i in range(len(ids_a)):
        d = np.abs(wb - wa[i])
        m = np.minimum(d, L - d)
        s2 = (m[:, 0] * m[:, 0] + m[:, 1] * m[:, 1]) + m[:, 2] * m[:, 2]
        b = (np.sqrt(s2) / bs).astype(np.int64)
        ok = (b < nb) & (ids_b != ids_a[i])
        out += np.bincount(b[ok], minlength=nb)[:nb]
    return out


def _upload(eng, n, box, frames, seed, lattice=None):
    rng = np.random.default_rng(seed)
    u = (rng.random((frames, n, 3)) * box).astype(np.float32)
    if lattice:  # coordinates on a grid: many distances on bin edges, some atoms at one place
        u = (rng.integers(0, int(box / lattice), (frames, n, 3)) * lattice).astype(np.float32)
    eng.upload(u, [box] * 3)
    return u


@pytest.mark.parametrize("n,nb,max_d,lattice", [(2, 7, 3.0, None), (255, 40, 4.5, None), (257, 333, 4.5, None),
                                                (1025, 500, 4.5, None), (1500, 4096, 4.5, None),
                                                (700, 18, 4.5, 0.25), (1030, 36, 4.5, 0.125)])
def test_rdf_symmetric_units(eng, n, nb, max_d, lattice):
    box = 9.0
    u = _upload(eng, n, box, 2, n, lattice)
    got = eng.rdf(0, 0, [1, 0], max_d, nb)
    ids = np.arange(n)
    for row, f in enumerate((1, 0)):
        np.testing.assert_array_equal(got[row], _counts(u[f], u[f], ids, ids, np.float32(box), max_d, nb))


@pytest.mark.parametrize("n1,n2", [(1, 900), (300, 129), (1100, 1023)])
def test_rdf_two_lists_units(eng, n1, n2):
    box, n = 9.0, 1200
    u = _upload(eng, n, box, 1, n1 + n2)
    rng = np.random.default_rng(n1)
    a, b = (np.sort(rng.permutation(n)[:k]) for k in (n1, n2))
    got = eng.rdf(eng.list(a), eng.list(b), [0], 4.0, 77)
    np.testing.assert_array_equal(got[0], _counts(u[0][a], u[0][b], a, b, np.float32(box), 4.0, 77))


def test_rdf_many_bins_sum_to_few_bins(eng):
    """Large lists take wide units: the counts over 8 x 64 bins add up to those over 64,
    and to the sum over a list's halves and their cross pairs."""
    box, n = 30.0, 23000
    _upload(eng, n, box, 2, 11)
    fr = [0, 1]
    fine, coarse = eng.rdf(0, 0, fr, 8.0, 512), eng.rdf(0, 0, fr, 8.0, 64)
    np.testing.assert_array_equal(fine.reshape(2, 64, 8).sum(2), coarse)
    a, b = eng.list(np.arange(0, n // 2)), eng.list(np.arange(n // 2, n))
    parts = eng.rdf(a, a, fr, 8.0, 64) + eng.rdf(b, b, fr, 8.0, 64) + eng.rdf(a, b, fr, 8.0, 64) + eng.rdf(b, a, fr, 8.0, 64)
    np.testing.assert_array_equal(coarse, parts)


@pytest.mark.parametrize("n,max_d", [(900, 4.0), (1300, 4.0)])
def test_vhd_all_pairs_units(eng, monkeypatch, n, max_d):
    """Different frames: an atom's own pair is left out by its index."""
    monkeypatch.setenv("AMDAT_PAIR_CELLS", "off")
    box = 9.0
    u = _upload(eng, n, box, 4, n)
    sc = synth.TimeScheme.linear(4, 1.0)
    eng.set_scheme(sc)
    got = eng.vhd(0, 0, max_d, 50)
    ids = np.arange(n)
    from amdat_gb300 import engine as E
    g, t0, t1 = E.scheme_pairs(eng.scheme)
    ref = np.zeros_like(got)
    for k in range(len(g)):
        ref[g[k]] += _counts(u[t0[k]], u[t1[k]], ids, ids, np.float32(box), max_d, 50)
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("n,box,max_d,nb,sigma", [(1100, 12.0, 3.9, 60, 0.3), (5000, 18.0, 1.2, 33, 0.5),
                                                  (6001, 40.0, 13.0, 200, 2.0), (3000, 15.0, 4.99, 500, 0.0)])
def test_vhd_cells(eng, monkeypatch, n, box, max_d, nb, sigma):
    """The cell pass against the all-pairs pass: dense and sparse boxes, reaches just
    below a third of the box and far below it, atoms that do not move (every own pair
    at zero distance)."""
    sc = synth.TimeScheme.linear(4, 1.0)
    traj = synth.random_walk(n, box, sc, sigma, seed=n, time_scaled=False)
    eng.upload(traj.unwrapped, traj.box)
    eng.set_scheme(sc)
    third, rest = eng.list(np.arange(0, n, 3)), eng.list(np.arange(0, n))
    half, other = eng.list(np.arange(0, n // 2)), eng.list(np.arange(n // 2, n))
    for l1, l2 in ((0, 0), (third, rest), (third, 0), (half, 0), (0, other), (third, third), (eng.list([5]), rest)):
        monkeypatch.delenv("AMDAT_PAIR_CELLS", raising=False)
        got = eng.vhd(l1, l2, max_d, nb)
        monkeypatch.setenv("AMDAT_PAIR_CELLS", "off")
        np.testing.assert_array_equal(got, eng.vhd(l1, l2, max_d, nb))


def test_vhd_cells_slab_and_outside(eng, monkeypatch):
    """A box of unequal edges and an offset origin, a list gathered in one corner; wrapped
    coordinates that lie outside the box take the all-pairs pass."""
    rng = np.random.default_rng(8)
    L, lo, n = np.array([30.0, 9.5, 14.0], np.float32), np.array([-7.0, 2.0, 100.0], np.float32), 4000
    u = (lo + rng.random((3, n, 3)) * L).astype(np.float32)
    sc = synth.TimeScheme.linear(3, 1.0)
    for wrapped in (None, (u + (rng.random((1, n, 1)) < 0.01) * 2.5 * L).astype(np.float32)):
        eng.upload(u, L, lo, wrapped=wrapped)
        eng.set_scheme(sc)
        corner = eng.list(np.nonzero((u[0] - lo < 0.3 * L).all(1))[0])
        for l1, l2 in ((0, 0), (corner, 0)):
            monkeypatch.delenv("AMDAT_PAIR_CELLS", raising=False)
            got = eng.vhd(l1, l2, 3.0, 40)
            monkeypatch.setenv("AMDAT_PAIR_CELLS", "off")
            np.testing.assert_array_equal(got, eng.vhd(l1, l2, 3.0, 40))
            assert got.sum() > 0
