"""run(pipeline=False), which issues its steps from one native call, against
the loop of step() that it stands for."""
import numpy as np
import pytest

from tests.gpu_util import HertzContactConfig, make_dem, rsa_spheres

pytestmark = pytest.mark.gpu


def _system(cls=None, shape=(48, 40, 36), n=8, frozen=False, storage="f32", seed=3, vel=2e-3, **kw):
    from lbdem_taichi_b200.lbdem.psclattice3d import PSCLattice3D
    rng = np.random.default_rng(seed)
    pos, rad = rsa_spheres(rng, n, shape, 6.0, 9.0, gap=1.0, margin=1.0)
    v = np.zeros((n, 3)) if frozen else rng.normal(0, vel, (n, 3))
    dem = make_dem((0.0, shape[0], 0.0, shape[1], 0.0, shape[2]), 0.2, (0, 0, 0), HertzContactConfig(0.3, 0.3, 0.9, 0.9),
                   rad, 2.0 * 4.0 / 3.0 * np.pi * rad ** 3, pos, v, periodic=(True, True, True),
                   freeze=np.ones(n, np.int32) if frozen else None)
    lat = (cls or PSCLattice3D)(*shape, 1 / 0.6, 1.0, 1.0, 1.0, dem, body_force=(2e-5, 0, 0), storage=storage, **kw)
    return lat, dem


@pytest.mark.parametrize("method", ["collide", "stream", "step", "grains2lattice"])
@pytest.mark.parametrize("how", ["subclass", "class", "instance"])
def test_run_calls_overridden_methods(method, how, monkeypatch):
    from lbdem_taichi_b200.lbdem.psclattice3d import PSCLattice3D
    calls, own = [], getattr(PSCLattice3D, method)

    def wrapped(self, *a, **k):
        calls.append(1)
        return own(self, *a, **k)

    if how == "subclass":
        lat, _ = _system(type("Watched", (PSCLattice3D,), {method: wrapped}))
    elif how == "class":
        monkeypatch.setattr(PSCLattice3D, method, wrapped)
        lat, _ = _system()
    else:
        lat, _ = _system()
        setattr(lat, method, lambda *a, **k: wrapped(lat, *a, **k))
    lat.initialize()
    calls.clear()
    lat.run(5, 2, pipeline=False)
    assert len(calls) == 5


def test_run_calls_an_overridden_dem():
    lat, dem = _system()
    lat.initialize()
    own, calls = dem.run_substeps, []
    dem.run_substeps = lambda n: (calls.append(n), own(n))
    lat.run(5, 2, pipeline=False)
    assert calls == [2] * 5


def test_drag_run_calls_an_overridden_collide():
    from lbdem_taichi_b200.lbdem.adjoint import FrozenBedDrag
    lat, _ = _system(frozen=True, solid_fraction="smooth")
    drag = FrozenBedDrag(lat, 4, checkpoint_every=2)
    loss = drag.forward()
    own, calls = lat.collide, []
    lat.collide = lambda: (calls.append(1), own())
    assert drag.forward() == pytest.approx(loss, rel=1e-9)
    assert len(calls) == 4


def test_failed_run_does_not_mark_the_map_current():
    """A native call that fails before its first map leaves the owner keys as
    stale as they were: obstacles set before it lose theirs at the next step."""
    from lbdem_taichi_b200 import _native as N
    from lbdem_taichi_b200.lbm3d.lbmutils import CellType
    lat, _ = _system(frozen=True)
    lat.initialize()
    lat.run(2, 1, pipeline=False)
    assert lat._key.cpu().numpy().reshape(36, 40, 48)[:, :, 20:24].any()
    ct = lat.CT.to_numpy()
    ct[20:24, :, :] = CellType.OBSTACLE
    lat.CT.from_numpy(ct)
    lat._psc.disp_limit = 0.25             # refused by the native loop
    with pytest.raises(N.LbdemError):
        lat.run(2, 1, pipeline=False)
    lat._psc.disp_limit = 0.0
    lat.run(2, 1, pipeline=False)
    assert not lat._key.cpu().numpy().reshape(36, 40, 48)[:, :, 20:24].any()
