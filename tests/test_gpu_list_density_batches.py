"""Vector-list densities whose sums of 128 atoms do not fit their buffer at once, and the
kernel without segments on more than one such sum: the same bits as small lists give, in
bounded memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L = 30.0


def _vectors(n, seed):
    return np.random.default_rng(seed).integers(-25, 26, (n, 3)).astype(np.int32)


def _density(eng, kv, frames):
    h = eng.wave_density(0, kv, L, frames)
    rho = eng.wave_density_read(h, len(frames), len(kv))
    eng.wave_density_free(h)
    return rho


@pytest.mark.parametrize("n,nk", [(400_003, 90_001), (7_000_003, 3_000)])
def test_large_lists_in_vector_batches(engine_mod, n, nk):
    """One frame's sums would take 2.2 and 1.3 GB."""
    import torch
    rng = np.random.default_rng(nk)
    kv = _vectors(nk, 1)
    eng = engine_mod.Engine(0)
    try:
        eng.upload((rng.random((2, n, 3)) * L).astype(np.float32), [L] * 3)
        some = np.unique(np.concatenate([[0, nk - 1], rng.integers(0, nk, 60)]))
        want = _density(eng, kv[some], [0, 1])
        free = torch.cuda.mem_get_info()[0]
        got = _density(eng, kv, [0, 1])
        assert free - torch.cuda.mem_get_info()[0] < 1100 << 20
        np.testing.assert_array_equal(got[:, some], want)
    finally:
        eng.close()


@pytest.mark.parametrize("nk,F", [(600, 3700), (300, 3700), (60, 15000)])
def test_without_segments(eng, nk, F):
    """So many frames that no atom segments are cut (24 blocks of 256 threads per SM), with
    three whole sums of 128 atoms and a partial one."""
    n = 401
    rng = np.random.default_rng(nk)
    eng.upload((rng.random((F, n, 3)) * L).astype(np.float32), [L] * 3)
    kv = _vectors(nk, 2)
    pick = [0, 1, F // 2, F - 1]
    got = _density(eng, kv, np.arange(F, dtype=np.int32))[pick]
    np.testing.assert_array_equal(got, _density(eng, kv, pick))
