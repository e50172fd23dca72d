"""Narrow lattices with more rows than one grid dimension of the step's
two-warp blocks covers (65,535 blocks of one or two rows), which take a kernel
of their own: a flow that repeats every PERIOD rows must stay the small
lattice's, row for row and bit for bit -- populations, lagged state, stress,
with walls and a particle.  Widths of one, two and four x-blocks (four: 97 to
128 cells), the last size of the ordinary kernel and the first beyond."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PERIOD = 16


@pytest.mark.parametrize("nx,ny,storage", [(5, 131088, "f32"), (32, 131056, "f16"), (33, 65552, "f32"),
                                           (97, 65520, "f32"), (97, 65552, "f16"), (64, 131088, "bf16")])
def test_rows_beyond_one_grid_dimension(nx, ny, storage):
    from lbdem_taichi_b200.lbm3d.lattice import BasicLattice3D
    rng = np.random.default_rng(2)
    ct0 = np.ones((nx, PERIOD, 1), np.int32)
    ct0[2, 3] = 8
    v0 = 0.03 * rng.uniform(-1, 1, (nx, PERIOD, 1, 3))
    v0[2, 3] = 0.0
    r0 = 1.0 + 0.01 * rng.uniform(-1, 1, (nx, PERIOD, 1))
    out = []
    for n in (PERIOD, ny):
        rep = n // PERIOD
        lat = BasicLattice3D(nx, n, 1, 1 / 0.6, 1.0, 1.0, 1.0, storage=storage, stress=True)
        lat.CT.from_numpy(np.tile(ct0, (1, rep, 1)))
        lat.vel.from_numpy(np.tile(v0, (1, rep, 1, 1)))
        lat.rho.from_numpy(np.tile(r0, (1, rep, 1)))
        lat.initialize()
        for _ in range(3):
            lat.collide()
            lat.stream()
            lat.compute_stress()       # the next collide() writes it
        lat.collide()
        lat.stream()
        out.append((lat._f[lat._cur].clone(), lat._aux.clone(), lat._stress.clone()))
    for small, tall in zip(*out):
        planes = 7 if small is out[0][2] else 1
        assert (tall.view(planes, ny // PERIOD, -1) == small.view(planes, 1, -1)).all()


def test_particles_beyond_one_grid_dimension():
    """Two equal spheres, one near either end of the rows, drag alike."""
    from lbdem_taichi_b200.lbdem.psclattice3d import PSCLattice3D
    from tests.gpu_util import HertzContactConfig, make_dem
    nx, ny, nz = 33, 65600, 12
    pos = np.array([[16.3, 40.6, 6.2], [16.3, 40.6 + 65504.0, 6.2]])
    rad = np.full(2, 4.0)
    dem = make_dem((0, nx, 0, ny, 0, nz), 0.1, (0, 0, 0), HertzContactConfig(0.3, 0.3, 0.9, 0.9), rad, np.full(2, 500.0),
                   pos, np.zeros((2, 3)), periodic=(True, True, True), freeze=np.ones(2, np.int32))
    lat = PSCLattice3D(nx, ny, nz, 1 / 0.6, 1.0, 1.0, 1.0, dem, body_force=(2e-5, 1e-5, 0))
    lat.initialize()
    lat.run(4, 1, pipeline=False)
    lat.check_status()
    F = dem.gf.force_fluid.to_numpy()
    assert np.abs(F[0]).max() > 0
    # (the centre's rounding at y = 65,544 is 1e-11 of a cell; FP32 sums group the same cells alike)
    np.testing.assert_allclose(F[1], F[0], rtol=1e-6, atol=1e-6 * np.abs(F[0]).max())
