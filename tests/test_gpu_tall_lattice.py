"""Narrow lattices with more rows than one grid dimension of the step's
two-warp blocks covers (65,535 blocks of one or two rows): a flow that repeats
every PERIOD rows must stay the small lattice's, row for row and bit for bit.
Widths of one, two and four x-blocks (four: 97 to 128 cells)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PERIOD = 16


@pytest.mark.parametrize("nx,ny,storage", [(5, 131088, "f32"), (33, 65552, "f32"), (97, 65552, "f16"), (64, 131088, "bf16")])
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
        lat = BasicLattice3D(nx, n, 1, 1 / 0.6, 1.0, 1.0, 1.0, storage=storage)
        lat.CT.from_numpy(np.tile(ct0, (1, rep, 1)))
        lat.vel.from_numpy(np.tile(v0, (1, rep, 1, 1)))
        lat.rho.from_numpy(np.tile(r0, (1, rep, 1)))
        lat.initialize()
        for _ in range(3):
            lat.collide()
            lat.stream()
        out.append(lat._f[lat._cur].clone())
    small, tall = out
    assert (tall.view(ny // PERIOD, -1) == small.view(1, -1)).all()
