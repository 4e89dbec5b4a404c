"""Items of the moments passes: units of up to 4,096 members keep items of at most 4,096
members, several pairs to an item only for units of half of that; larger units take
longer items but never several pairs in one, and sum their terms 16 at a time.  The sums
are the oracle's to 1e-6."""
import numpy as np
import pytest

from amdat_gb300 import engine as E
from amdat_gb300 import synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,frames,chunk,per_item", [(500, 60, 1024, 2), (1000, 200, 4096, 4), (2049, 200, 4096, 1),
                                                     (4000, 200, 4096, 1), (5000, 200, 16384, 1), (8192, 200, 16384, 1)])
def test_items_of_one_unit(eng, n, frames, chunk, per_item):
    sc = synth.TimeScheme.linear(frames, 1.0)
    traj = synth.random_walk(n, 15.0, sc, 0.3, seed=n, time_scaled=False)
    eng.upload(traj.unwrapped, traj.box)
    eng.set_scheme(sc)
    gaps = np.bincount(E.scheme_pairs(eng.scheme)[0])
    plan = eng.plan([0])
    info = plan.info()
    assert info["chunk"] == chunk
    assert info["n_items"] == (-(-gaps // per_item)).sum()  # one chunk of members each
    plan.run()
    out = plan.read()
    d2, d4, cnt = orc.disp_moments(orc.scheme(sc), traj.unwrapped, np.arange(n, dtype=np.int32), 0)
    np.testing.assert_array_equal(out["atom_pairs"][0], cnt)
    np.testing.assert_allclose(out["sum_d2"][0], d2, rtol=1e-6, atol=1e-12)
    np.testing.assert_allclose(out["sum_d4"][0], d4, rtol=1e-6, atol=1e-14)
    plan.close()


@pytest.mark.parametrize("gathered", [False, True])
@pytest.mark.parametrize("bins", [0, 20])
def test_long_items_keep_small_terms(eng, gathered, bins):
    """Items are whole multiples of 4,096 members.  One such round in four moves by 2^-15,
    the others by 1, in every pair of odd gap.  One Kahan sum per thread and item would drop
    small terms (3e-10 of the sum); sums of 16 terms merged error-free keep them."""
    n, T = 64000, 40
    far = np.arange(n) // 4096 % 4 > 0
    u = np.zeros((T, 2 * n if gathered else n, 3), np.float32)
    members = np.arange(n) * 2 if gathered else np.arange(n)
    u[1::2, members, 0] = np.where(far, np.float32(1.0), np.float32(2.0 ** -15))
    eng.upload(u, [40.0] * 3)
    eng.set_scheme(synth.TimeScheme.linear(T, 1.0))
    handle = eng.list(members.astype(np.int32)) if gathered else 0
    plan = eng.plan([handle], n_bins=bins, bin_max=2.0 if bins else 0.0)
    assert plan.info()["chunk"] == 16384
    plan.run()
    out = plan.read()
    plan.close()
    g, t0, t1 = E.scheme_pairs(eng.scheme)
    odd = np.bincount(g, weights=(t1 - t0) % 2)
    exact = odd * (far.sum() + (~far).sum() * 2.0 ** -30)
    np.testing.assert_allclose(out["sum_d2"][0], exact, rtol=3e-11)
    np.testing.assert_allclose(out["sum_d4"][0], odd * far.sum(), rtol=3e-11)
