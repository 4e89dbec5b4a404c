"""Pair histograms with coordinates that are NaN or infinite: their pairs are counted in no
bin (no comparison with the last bin holds), all others as without them, in the all-pairs
pass, the cell groups and the walk."""
import numpy as np
import pytest

from amdat_gb300 import engine as E
from amdat_gb300 import synth

pytestmark = pytest.mark.gpu


def _counts(wa, wb, ids_a, ids_b, L, max_d, nb):
    out = np.zeros(nb, np.int64)
    bs = np.float32(np.float32(max_d) / np.float32(nb))
    fin = np.isfinite(wb).all(1)
    wb, ids_b = wb[fin], ids_b[fin]
    for x, a in zip(wa, ids_a):
        if not np.isfinite(x).all():
            continue
        d = np.abs(wb - x)
        m = np.minimum(d, L - d)
        s2 = (m[:, 0] * m[:, 0] + m[:, 1] * m[:, 1]) + m[:, 2] * m[:, 2]
        b = (np.sqrt(s2) / bs).astype(np.int64)
        out += np.bincount(b[(b < nb) & (ids_b != a)], minlength=nb)[:nb]
    return out


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("whole_groups", [False, True])
def test_nonfinite_coordinates_are_in_no_bin(eng, bad, whole_groups):
    rng = np.random.default_rng(4)
    n, L, T = 1500, np.float32(15.0), 2
    w = (rng.random((T, n, 3)) * L).astype(np.float32)
    hit = np.arange(0, 96) if whole_groups else np.arange(3, n, 37)
    for k, a in enumerate(hit):
        w[k % T, a, k % 3 if not whole_groups else slice(None)] = bad
    eng.upload(w, [L] * 3, wrapped=w)
    eng.set_scheme(synth.TimeScheme.linear(T, 1.0))
    ids, few = np.arange(n), np.arange(0, n, 150)
    got = eng.rdf(0, 0, [0, 1], 7.0, 35)
    for f in range(T):
        np.testing.assert_array_equal(got[f], _counts(w[f], w[f], ids, ids, L, 7.0, 35))
    some = eng.list(few.astype(np.int32))
    g, t0, t1 = E.scheme_pairs(eng.scheme)
    for handle, members, max_d in ((0, ids, 4.0), (some, few, 2.0)):
        ref = np.zeros((eng.n_timegaps, 20), np.int64)
        for k in range(len(g)):
            ref[g[k]] += _counts(w[t0[k]][members], w[t1[k]], members, ids, L, max_d, 20)
        np.testing.assert_array_equal(eng.vhd(handle, 0, max_d, 20), ref)
