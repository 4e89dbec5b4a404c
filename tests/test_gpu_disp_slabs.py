"""MSD + NGP moments of several gathered units by slabs of members in atom order: the
sums equal the exact sums of the FP32 terms to 1e-9 (the kernel's additions are
error-free but for the last bits of their corrections) and the oracle's to 1e-6, over
slab edges, unit counts on both sides of the
lane groups' rule and up to the route's limit, empty lists, contiguous
units among gathered ones and repeated atoms across lists."""
import numpy as np
import pytest

from amdat_gb300 import synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _sets(kind, n, rng):
    perm = rng.permutation(n)
    if kind.startswith("types"):
        return [np.sort(x) for x in np.array_split(perm, int(kind[5:]))]
    if kind == "nested":
        return [np.sort(perm[:m]) for m in (1, 3, n // 9, n // 3, n)]
    if kind == "mixed":
        return [np.arange(n // 2), np.zeros(0, int)] + [n // 2 + np.arange(i, n - n // 2, 7) for i in range(7)]
    return [np.sort(rng.choice(n, n // 2, replace=False)) for _ in range(9)]  # overlapping


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


@pytest.mark.parametrize("n", [5, 127, 1023, 1024, 1025, 3000])
@pytest.mark.parametrize("kind", ["types2", "types16", "types17", "types128", "nested", "mixed", "overlap"])
def test_slabs_match_exact_sums(eng, n, kind):
    scheme = synth.TimeScheme.exponential(3, 7, 1.4, 0, 0, 0.005)
    traj = synth.random_walk(n, 15.0, scheme, 0.5, seed=n)
    eng.upload(traj.unwrapped, traj.box)
    eng.set_scheme(scheme)
    sets = _sets(kind, n, np.random.default_rng(n))
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
