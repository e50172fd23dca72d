"""Owner keys cleared other than by the next map: by the step that reads them
(run(), every step form) and by lbdem_psc_map_clear beside the DEM."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.gpu_util import HertzContactConfig, make_dem, rsa_spheres

pytestmark = pytest.mark.gpu


def _system(shape, n, storage, wall=None, seed=4):
    from lbdem_taichi_b200.lbdem.psclattice3d import PSCLattice3D
    rng = np.random.default_rng(seed)
    pos, rad = rsa_spheres(rng, n, shape, 6.0, 10.0, gap=0.5, margin=1.5)
    dem = make_dem((0.0, shape[0], 0.0, shape[1], 0.0, shape[2]), 0.1, (1e-6, 0, 0), HertzContactConfig(0.3, 0.3, 0.9, 0.9),
                   rad, 2.0 * 4 / 3 * np.pi * rad ** 3, pos, rng.normal(0, 5e-2, (n, 3)), periodic=(True, True, wall is None))
    lat = PSCLattice3D(*shape, 1 / 0.6, 1.0, 1.0, 1.0, dem, smagorinsky="reference", body_force=(1e-6, 0, 0),
                       storage=storage)
    if wall is not None:
        ct = np.ones(shape, np.int32)
        ct[:, :, 0] = ct[:, :, -1] = wall
        lat.CT.from_numpy(ct)
    lat.initialize()
    return lat, dem


def _same(a, b, ftol):
    (la, da), (lb, db) = a, b
    assert np.array_equal(la._key.cpu().numpy(), lb._key.cpu().numpy())
    assert (la._f[la._cur].float() - lb._f[lb._cur].float()).abs().max().item() <= ftol
    Fa, Fb = da.gf.force_fluid.to_numpy(), db.gf.force_fluid.to_numpy()
    assert np.abs(Fa - Fb).max() <= 1e-9 * np.abs(Fb).max()
    for k in ("id", "volfrac"):
        np.testing.assert_array_equal(getattr(la, k).to_numpy(), getattr(lb, k).to_numpy())


# bounds of tests/test_gpu_pipeline.py: the runs differ in the order of FP64 force sums
@pytest.mark.parametrize("storage,wall", [("f16", None), ("bf16", 8), ("f16", 32)])
def test_pairs_clear_the_keys_that_they_read(storage, wall):
    """Two cells per thread (16-bit rows of 225 to 256 cells, 8192 rows), whose
    warps beside walls run the one-cell code."""
    a, b = (_system((228, 64, 128), 60, storage, wall) for _ in range(2))
    for n in (5, 1, 4):
        a[0].run(n, 5, pipeline=False)
        for _ in range(n):
            b[0].step(5)
        _same(a, b, 1e-5 * 4096)
    assert np.abs(a[1].gf.position.to_numpy() - b[1].gf.position.to_numpy()).max() <= 1e-9


@pytest.mark.parametrize("n", [2, 40])
def test_clear_beside_the_dem(n):
    """lbdem_psc_map_clear on a second stream after the step: the next map
    starts on clear keys (few particles: several blocks share a box)."""
    from lbdem_taichi_b200 import _native as N
    a, b = (_system((96, 80, 72), n, "f32") for _ in range(2))
    lat, dem = a
    main, side = torch.cuda.current_stream(), torch.cuda.Stream()
    for k in range(6):
        lat.collide()
        lat.stream()
        side.wait_stream(main)
        N.call("lbdem_psc_map_clear", C.byref(lat._lat), C.byref(lat._psc), C.byref(lat._grains), side.cuda_stream)
        assert lat._psc.have_prev == 0
        dem.run_substeps(5)
        main.wait_stream(side)
        if k % 2:
            assert not lat._key.any().item()
        b[0].step(5)
    lat.grains2lattice()
    b[0].grains2lattice()
    _same(a, b, 1e-6)
    assert lat._key.any().item()
