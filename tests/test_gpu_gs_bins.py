"""G_s bins by estimate and, near an edge, by the exact chain: the counts equal those of
the FP32 chain sqrt((dx dx + dy dy) + dz dz) / bin evaluated with IEEE arithmetic on the
host, exactly, on displacements that lie on bin edges (a dyadic grid along one axis), on
random ones, beyond the last bin and at zero, for one bin to the most bins, contiguous
and gathered lists, and with F_s of both kinds in the same pass."""
import numpy as np
import pytest

from amdat_gb300 import synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

BOX = 8.0


def _counts(scheme, u, members, bin_max, n_bins):
    gap, t0, t1 = orc.pairs(orc.scheme(scheme), 0)
    u = u - u[:1]
    bin_size = np.float32(bin_max) / np.float32(n_bins)
    out = np.zeros((gap.max() + 1, n_bins), np.int64)
    for g, a, b in zip(gap, t0, t1):
        d = u[b, members] - u[a, members]
        s2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
        k = (np.sqrt(s2) / bin_size).astype(np.int64)
        out[g] += np.bincount(k[k < n_bins], minlength=n_bins)
    return out


@pytest.mark.parametrize("n_bins,bin_max", [(1, 0.5), (64, 1.0), (200, 0.7), (16384, 2.0), (16384, 0.01)])
@pytest.mark.parametrize("layout", ["contiguous", "gathered"])
@pytest.mark.parametrize("fs", ["none", "octants", "vectors"])
def test_gs_counts_equal_the_chain(eng, n_bins, bin_max, layout, fs):
    n = 1500
    scheme = synth.TimeScheme.exponential(3, 6, 1.4, 0, 0, 0.005)
    u = synth.random_walk(n, BOX, scheme, 0.3, seed=n_bins).unwrapped.astype(np.float32)
    # a third of the atoms move along x on a grid of 2^-8 (bin edges of the dyadic bins)
    u[:, ::3] = 0.0
    steps = np.random.default_rng(7).integers(-60, 61, (u.shape[0], len(u[0, ::3])))
    u[:, ::3, 0] = np.cumsum(steps, 0) * np.float32(2.0 ** -8)
    members = np.arange(n, dtype=np.int32)
    if layout == "gathered":
        members = members[np.random.default_rng(5).random(n) < 0.4]
    kw = {}
    if fs != "none":
        kv = np.array([[x, y, z] for x in (2, -2) for y in (3, -3) for z in (1, -1)], np.int32)
        if fs == "vectors":
            kv = kv[:5]
        kw = dict(shells=(kv, np.array([0, len(kv)], np.int32)), period=BOX)
    eng.upload(u, np.full(3, BOX, np.float32))
    eng.set_scheme(scheme)
    out = eng.disp(eng.list(members), n_bins=n_bins, bin_max=bin_max, **kw)
    np.testing.assert_array_equal(out["gs_counts"], _counts(scheme, u, members, bin_max, n_bins))
