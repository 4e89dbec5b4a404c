"""Vector-list densities at the edges of the kernel's folds (128 atoms), vector
blocks (64 to 1024) and atom segments, against the FP64 oracle: 2e-6 * sqrt(N) as
for the other list densities.  Segments do not change a bit of the result."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
L = 9.0


def _vectors(n, seed):
    return np.random.default_rng(seed).integers(-25, 26, (n, 3)).astype(np.int32)


@pytest.mark.parametrize("n,nk,F", [(1, 1, 1), (127, 64, 2), (128, 65, 1), (129, 129, 3), (513, 256, 1), (640, 257, 2),
                                    (1000, 512, 1), (1023, 513, 2), (3000, 1100, 1)])
def test_list_density(eng, n, nk, F):
    rng = np.random.default_rng(n)
    u = (rng.random((F, n, 3)) * L).astype(np.float32)
    eng.upload(u, [L] * 3)
    kv = _vectors(nk, nk)
    h = eng.wave_density(0, kv, L, np.arange(F, dtype=np.int32))
    rho = eng.wave_density_read(h, F, nk).astype(np.float64)
    eng.wave_density_free(h)
    ref = orc.rhok_parallel(u, np.arange(F, dtype=np.int32), kv, L, 8)
    assert np.abs(rho - ref).max() <= 2e-6 * np.sqrt(n)


def test_list_density_same_in_segments(eng):
    """A few frames are cut into atom segments, thousands are not: the same bits."""
    n, nk, F = 300, 600, 2000
    rng = np.random.default_rng(2)
    eng.upload((rng.random((F, n, 3)) * L).astype(np.float32), [L] * 3)
    kv = _vectors(nk, 3)
    rows = []
    for frames in (np.arange(F, dtype=np.int32), np.array([0, F - 1], np.int32)):
        h = eng.wave_density(0, kv, L, frames)
        rows.append(eng.wave_density_read(h, len(frames), nk)[[0, -1]])
        eng.wave_density_free(h)
    np.testing.assert_array_equal(rows[0], rows[1])
