"""The map's sub-sample counts over its range of radii against the FP64 oracle:
exact owners and counts on both sides of the radius where the count changes from
comparing points to one square root per column (mapped radius 2, i.e. R = 2.5),
for radii below a cell, for spheres larger than one classification chunk, and
for cell types that the map leaves out (per-cell link masks) or not."""
import numpy as np
import pytest

from oracle.oracle import OracleGrains, OracleLattice
from tests.gpu_util import HertzContactConfig, make_dem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("radius", [0.7, 1.3, 2.4999, 2.5, 2.5001, 3.1, 5.0, 7.77, 15.2])
def test_counts_over_radii(radius, walls):
    from lbdem_taichi_b200.lbdem.psclattice3d import PSCLattice3D
    nx, ny, nz = 61, 44, 40
    rng = np.random.default_rng(int(1000 * radius) + walls)
    n = 2 if radius > 10 else 24          # overlaps included: the owner rule decides
    pos = rng.uniform(0.0, 1.0, (n, 3)) * (nx, ny, nz)
    pos[0] = np.round(pos[0]) + 0.5       # centre on the 0.1 grid: sub-points exactly on the surface
    rad = radius * np.where(np.arange(n) % 3, 1.0, 1.0 + 1e-7)
    dem = make_dem((0.0, nx, 0.0, ny, 0.0, nz), 0.1, (0, 0, 0), HertzContactConfig(0.3, 0.3, 0.9, 0.9), rad,
                   2.0 * 4 / 3 * np.pi * rad ** 3, pos, np.zeros((n, 3)), periodic=(True, True, True))
    lat = PSCLattice3D(nx, ny, nz, 1 / 0.6, 1.0, 1.0, 1.0, dem)
    o = OracleLattice(nx, ny, nz, 1 / 0.6, psc=True)
    if walls:
        ct = np.ones((nx, ny, nz), np.int32)
        ct[:, :, 0] = ct[:, :, -1] = 8
        ct[20:24, 10:30, 12:15] = 8
        lat.CT.from_numpy(ct)
        o.ct[...] = ct
    lat.initialize()
    o.initialize()
    g = OracleGrains(pos, rad, np.zeros((n, 3)), np.zeros((n, 3)))
    o.grains2lattice(g)
    np.testing.assert_array_equal(lat.id.to_numpy(), o.id)
    np.testing.assert_allclose(lat.volfrac.to_numpy(), o.volfrac, rtol=0, atol=1e-7)   # FP32 of k / 125
    assert (o.id >= 0).any() or radius < 0.6
