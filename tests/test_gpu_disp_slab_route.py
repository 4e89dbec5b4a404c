"""The slab route of moments plans by its own kernel name: up to its limit of 128 units,
units of one atom and of none beside scattered lists that make slabs worth it; over the
limit the units' kernel runs.  The sums are those of the
FP32 terms to 1e-9."""
import numpy as np
import pytest

from amdat_gb300 import synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _exact(scheme, u, members):
    """Per gap the sums of d2 = fma(dz, dz, fma(dy, dy, dx dx)) and d2 d2 in FP32 terms,
    added in FP64 (where a product of FP32 numbers is exact)."""
    u = u - u[:1]
    gap, t0, t1 = orc.pairs(orc.scheme(scheme), 0)
    out = np.zeros((2, gap.max() + 1))
    for a, b, g in zip(t0, t1, gap):
        d = (u[b, members] - u[a, members]).astype(np.float64)
        d2 = (d[:, 0] * d[:, 0]).astype(np.float32)
        for k in (1, 2):
            d2 = (d[:, k] * d[:, k] + d2).astype(np.float32)
        out[0, g] += d2.astype(np.float64).sum()
        out[1, g] += (d2 * d2).astype(np.float64).sum()
    return out


@pytest.mark.parametrize("n", [25600, 30001])
@pytest.mark.parametrize("singles,empties", [(1, 0), (9, 3), (124, 1), (61, 64)])
def test_slabs_with_tiny_units(eng, n, singles, empties):
    scheme = synth.TimeScheme.exponential(4, 8, 1.4, 0, 0, 0.005)
    traj = synth.random_walk(n, 18.0, scheme, 0.5, seed=n)
    eng.upload(traj.unwrapped, traj.box)
    eng.set_scheme(scheme)
    perm = np.random.default_rng(n).permutation(n)
    sets = [perm[i:i + 1] for i in range(singles)] + [perm[:0]] * empties
    sets += [np.sort(x) for x in np.array_split(perm[singles:], 3)]  # scattered thirds
    handles = [eng.list(s.astype(np.int32)) for s in sets]
    assert len(sets) <= 128
    plan = eng.plan(handles, flags=4)  # lists as units
    eng.profile_reset()
    plan.run()
    assert eng.profile_kernel("disp_slab_kernel")[0] == eng.profile_kernel("disp_mixed_kernel")[0] == 1
    out = plan.read()
    counts = np.bincount(orc.pairs(orc.scheme(scheme), 0)[0])
    for i, members in enumerate(sets):
        np.testing.assert_array_equal(out["atom_pairs"][i], counts * len(members))
        d2, d4 = _exact(scheme, traj.unwrapped, members)
        np.testing.assert_allclose(out["sum_d2"][i], d2, rtol=1e-9)
        np.testing.assert_allclose(out["sum_d4"][i], d4, rtol=1e-9)
    plan.close()
    over = eng.plan(handles + handles[-1:] * (129 - len(handles)), flags=4)
    eng.profile_reset()
    over.run()
    assert eng.profile_kernel("disp_slab_kernel")[0] == 0 and eng.profile_kernel("disp_mixed_kernel")[0] == 1
    over.close()
