"""MSD + NGP moments of several gathered units by slabs of members in atom order: the
sums equal the exact sums of the FP32 terms to 1e-9 (the kernel's additions are
error-free but for the last bits of their corrections) and the oracle's to 1e-6, over
slab edges, unit counts on both sides of the
lane groups' rule and up to the route's limit, units of one atom and up, empty lists,
contiguous units among gathered ones and repeated atoms across lists.  A list of all
atoms brings the lists' mean size over the route's lower limit."""
import numpy as np
import pytest

from amdat_gb300 import synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _sets(kind, n, m, rng):
    """Lists over m scattered atoms, then the list of all n."""
    some = np.sort(rng.permutation(n)[:m])
    perm = rng.permutation(some)
    if kind.startswith("types"):
        out = [np.sort(x) for x in np.array_split(perm, int(kind[5:]))]
    elif kind == "nested":
        out = [np.sort(perm[:k]) for k in (1, 3, m // 9 + 1, m // 3 + 1, m)]
    elif kind == "mixed":
        out = [np.arange(m), np.zeros(0, int)] + [m + np.arange(i, n - m, 7) for i in range(6)]
    else:  # overlapping
        out = [np.sort(rng.choice(some, m // 2 + 1, replace=False)) for _ in range(9)]
    return out + [np.arange(n)]


def _exact(scheme, u, fb, members):
    """Per gap the sums of d2 = fma(dz, dz, fma(dy, dy, dx dx)) and d2 d2 in FP32 terms,
    of the engine's coordinates (FP32, relative to frame 0), added in FP64 (where a
    product of FP32 numbers is exact)."""
    u = u - u[:1]
    gap, t0, t1 = orc.pairs(orc.scheme(scheme), fb)
    out = np.zeros((2, gap.max() + 1))
    for a, b, g in zip(t0, t1, gap):
        d = (u[b, members] - u[a, members]).astype(np.float64)
        d2 = (d[:, 0] * d[:, 0]).astype(np.float32)
        for k in (1, 2):
            d2 = (d[:, k] * d[:, k] + d2).astype(np.float32)
        out[0, g] += d2.astype(np.float64).sum()
        out[1, g] += (d2 * d2).astype(np.float64).sum()
    return out


@pytest.mark.parametrize("n,m", [(16383, 5), (16384, 127), (16385, 1023), (16900, 1500)])
@pytest.mark.parametrize("kind", ["types2", "types15", "types16", "types127", "nested", "mixed", "overlap"])
def test_slabs_match_exact_sums(eng, n, m, kind):
    scheme = synth.TimeScheme.exponential(4, 8, 1.4, 0, 0, 0.005)
    traj = synth.random_walk(n, 15.0, scheme, 0.5, seed=n)
    eng.upload(traj.unwrapped, traj.box)
    eng.set_scheme(scheme)
    sets = _sets(kind, n, m, np.random.default_rng(n))
    handles = [eng.list(s.astype(np.int32)) for s in sets]
    for flags, fb in ((0, 0), (2, 1)):  # plain and replayed as a graph; default and full-block pairs
        plan = eng.plan(handles, flags=flags, fullblock=fb)
        for _ in range(2):
            plan.run()
        out = plan.read()
        counts = np.bincount(orc.pairs(orc.scheme(scheme), fb)[0])
        for i, members in enumerate(sets):
            np.testing.assert_array_equal(out["atom_pairs"][i], counts * len(members))
            d2, d4 = _exact(scheme, traj.unwrapped, fb, members)
            np.testing.assert_allclose(out["sum_d2"][i], d2, rtol=1e-9)
            np.testing.assert_allclose(out["sum_d4"][i], d4, rtol=1e-9)
            if len(members) and i in (0, len(sets) - 1):
                d2, d4, _ = orc.disp_moments(orc.scheme(scheme), traj.unwrapped, np.sort(members).astype(np.int32), fb)
                np.testing.assert_allclose(out["sum_d2"][i], d2, rtol=1e-6, atol=1e-12)
                np.testing.assert_allclose(out["sum_d4"][i], d4, rtol=1e-6, atol=1e-14)
        plan.close()
