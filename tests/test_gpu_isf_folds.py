"""The pair-table correlator's folds of four (two, one) gaps' sums and the warp sums over
tiles, at every tile width (set by the number of frames), gap counts on and off the folds'
multiples, shells of one vector, of whole tiles and one more, and an empty shell, against
FP64 sums of the engine's own densities.  Tolerance: each FP32 product of a pair is
rounded twice, 2^-23 of its magnitude, and the compensated sums add nothing above that:
2^-22 of the sum of |rho1| |rho2|."""
import numpy as np
import pytest

from amdat_gb300 import synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks,steps", [(1, 1), (2, 3), (5, 4), (9, 25), (100, 9), (200, 9), (450, 9), (900, 9),
                                          (1500, 9)])
@pytest.mark.parametrize("two", [False, True])
def test_pair_correlator_matches_fp64(eng, monkeypatch, blocks, steps, two):
    scheme = synth.TimeScheme.exponential(blocks, steps, 1.3, 0, 0, 0.005)
    traj = synth.random_walk(24, 9.0, scheme, 0.3, seed=blocks)
    if two and traj.n_frames > 12000:
        pytest.skip("two densities of so many frames do not fit a tile")
    eng.upload(traj.unwrapped, traj.box)
    eng.set_scheme(scheme)
    rng = np.random.default_rng(steps)
    off = np.cumsum([0, 1, 32, 0, 33, 7]).astype(np.int32)
    kv = rng.integers(-6, 7, (off[-1], 3)).astype(np.int32)
    fr = np.arange(traj.n_frames, dtype=np.int32)
    monkeypatch.setenv("AMDAT_ISF_KERNEL", "pairs")
    h1 = eng.wave_density(0, kv, 9.0, fr)
    h2 = eng.wave_density(eng.list(np.arange(0, 24, 2, dtype=np.int32)), kv, 9.0, fr) if two else h1
    corr, pc = eng.isf(h1, h2, off)
    r1, r2 = (np.asarray(eng.wave_density_read(h, len(fr), len(kv)), np.float64).reshape(len(fr), len(kv), 2)
              for h in (h1, h2))
    gap, t0, t1 = orc.pairs(orc.scheme(scheme), 0, loop_order=True)
    mag1, mag2 = np.hypot(r1[..., 0], r1[..., 1]), np.hypot(r2[..., 0], r2[..., 1])
    for g in range(len(pc)):
        a, b = t0[gap == g], t1[gap == g]
        assert pc[g] == len(a)
        per_k = (r1[a] * r2[b]).sum((0, 2))
        bound = (mag1[a] * mag2[b]).sum(0)
        for s in range(len(off) - 1):
            H = max(off[s + 1] - off[s], 1)
            ref, tol = per_k[off[s]:off[s + 1]].sum() / H, bound[off[s]:off[s + 1]].sum() / H * 2.0 ** -22
            assert abs(corr[g, s] - ref) <= tol + 1e-12, (g, s)
    sk = eng.structure_factor(h1, h2, off)
    both = (r1 * r2).sum((0, 2))
    top = (mag1 * mag2).sum(0)
    for s in range(len(off) - 1):
        H = max(off[s + 1] - off[s], 1)
        assert abs(sk[s] - both[off[s]:off[s + 1]].sum() / H) <= top[off[s]:off[s + 1]].sum() / H * 2.0 ** -22 + 1e-12
    eng.wave_density_free(h1)
    if two:
        eng.wave_density_free(h2)
