"""The cell pass of ordered pair histograms in boxes that lie anywhere and with wrapped
coordinates that are not quite in the box: the counts equal the all-pairs pass's."""
import numpy as np
import pytest

from amdat_gb300 import synth

pytestmark = pytest.mark.gpu


def _both(eng, monkeypatch, l1, l2, max_d, nb):
    monkeypatch.delenv("AMDAT_PAIR_CELLS", raising=False)
    got = eng.vhd(l1, l2, max_d, nb)
    monkeypatch.setenv("AMDAT_PAIR_CELLS", "off")
    want = eng.vhd(l1, l2, max_d, nb)
    monkeypatch.delenv("AMDAT_PAIR_CELLS")
    assert want.sum() > 0
    return got, want


@pytest.mark.parametrize("lo", [(0.0, 0.0, 0.0), (1000.0, -3e3, 2e4), (1e5, -1e5, 3e5), (-1e6, 0.0, 1e6)])
@pytest.mark.parametrize("max_d", [1.9, 4.9])
def test_vhd_cells_far_origin(eng, monkeypatch, lo, max_d):
    """The spacing of FP32 numbers at the origin is up to 2^-4, far above the cutoff's margin."""
    rng = np.random.default_rng(int(max_d))
    L, n = np.array([15.0, 18.0, 30.0], np.float32), 6000
    lo = np.array(lo, np.float32)
    u = (lo + rng.random((3, n, 3)) * L).astype(np.float32)
    eng.upload(u, L, lo)
    eng.set_scheme(synth.TimeScheme.linear(3, 1.0))
    few, many = eng.list(np.arange(0, n, 40)), eng.list(np.setdiff1d(np.arange(n), np.arange(0, n, 40)))
    for l1, l2 in ((0, 0), (few, many), (many, 0)):
        got, want = _both(eng, monkeypatch, l1, l2, max_d, 49)
        np.testing.assert_array_equal(got, want)
