"""Lattice densities at the edges of the tensor-core tiling, every vector against
the FP64 oracle: nz windows at their widest (96) and split just beyond it, four
and two operand stages (64 and 72 nz), ragged atom chunks (32 atoms, two chunks
per accumulation, four per ring cycle).  Tolerance as for the other lattice
densities: 3e-6 * sqrt(N) for the largest and 1e-6 * sqrt(N) for the rms error."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_atoms,radius", [(1, 7.5), (33, 8.5), (64, 63.5), (65, 64.5), (97, 79.5), (129, 95.5),
                                            (161, 97.5), (700, 12.2)])
def test_lattice_tiles(eng, n_atoms, radius):
    box = 8.0
    rng = np.random.default_rng(n_atoms)
    u = (rng.random((2, n_atoms, 3)) * 3 * box - box).astype(np.float32)
    eng.upload(u, [box] * 3)
    frames = np.arange(2, dtype=np.int32)
    h, nk, ns = eng.wave_density_lattice(0, radius * 2 * np.pi / box, 0.5, box, frames)
    kv, _ = eng.wave_density_vectors(h, nk, ns)
    rho = eng.wave_density_read(h, 2, nk).astype(np.float64)
    eng.wave_density_free(h)
    w = (u - np.float32(box) * np.floor(u / np.float32(box))).astype(np.float32)
    ref = orc.rhok_lattice(w, frames, kv, box, 8)
    err = np.abs(rho - ref) / np.sqrt(n_atoms)
    assert err.max() <= 3e-6, err.max()
    assert np.sqrt((err ** 2).mean()) <= 1e-6


def test_lattice_half_plane_images(eng):
    """Both images of a row, (nx, ny, nz) and (-nx, -ny, nz), and the rows nx = 0 or
    ny = 0 carry their own vector's density: mirroring the atoms through the origin
    conjugates every density exactly."""
    box, n = 16.0, 40
    rng = np.random.default_rng(5)
    q = rng.integers(1, 1 << 20, (1, n, 3)).astype(np.float64) * box / (1 << 20)  # exact in FP32, as is box - q
    out = []
    for pos in (q, box - q):
        eng.upload(pos.astype(np.float32), [box] * 3)
        h, nk, ns = eng.wave_density_lattice(0, 9.3 * 2 * np.pi / box, 0.5, box, [0])
        out.append(eng.wave_density_read(h, 1, nk))
        eng.wave_density_free(h)
    np.testing.assert_array_equal(out[0][..., 0], out[1][..., 0])
    np.testing.assert_array_equal(out[0][..., 1], -out[1][..., 1])


@pytest.mark.parametrize("n_atoms,radius", [(1, 3.2), (127, 15.5), (129, 16.5), (300, 31.4), (200, 129.3)])
def test_adjoint_tiles(eng, monkeypatch, n_atoms, radius):
    """S(k) adjoint at the edges of its tiling (atom blocks of 128, nz chunks of 16,
    a second nz window beyond 128) against the FP32 column kernel, 5e-4 of the
    largest component as for the adjoint's other comparisons."""
    box = 8.0
    rng = np.random.default_rng(n_atoms)
    eng.upload((rng.random((2, n_atoms, 3)) * box).astype(np.float32), [box] * 3)
    h, nk, ns = eng.wave_density_lattice(0, radius * 2 * np.pi / box, 0.5, box, [1, 0])
    _, off = eng.wave_density_vectors(h, nk, ns)
    w = rng.standard_normal(ns)
    g = eng.structure_factor_adjoint(h, off, w, 2, n_atoms)
    monkeypatch.setenv("AMDAT_SK_ADJOINT", "columns")
    ref = eng.structure_factor_adjoint(h, off, w, 2, n_atoms)
    eng.wave_density_free(h)
    assert np.isfinite(ref).all()
    scale = np.abs(ref).max() if n_atoms > 1 else float(np.abs(w).sum() * radius)  # one atom: the gradient is zero
    assert np.abs(g - ref).max() <= 5e-4 * scale
