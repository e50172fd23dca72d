"""The one-launch DEM form in which a particle waits only for the particles it
can touch (lbdem_dem_substeps_flow) against two launches per sub-step, which
follow the reference phase by phase: same contact sets, histories and states.

Both forms evaluate every contact with the same FP64 operations; only the
order in which a particle's contact forces are summed differs (atomics there,
lane order here), a relative 1e-16 per sum.  Hertz contacts of these moduli
amplify it by less than 1e4 over the runs, so positions are held to 1e-11 and
velocities, forces and histories to 1e-8 of the largest value.
"""
import numpy as np
import pytest

from tests.gpu_util import make_dem

pytestmark = pytest.mark.gpu

STATE = ("position", "velocity", "acceleration", "force", "omega", "omega_dot", "moment", "quaternion")


def _contact(model):
    from lbdem_taichi_b200.dem3d.demconfig import HertzContactConfig, LinearContactConfig
    if model == "linear":
        return LinearContactConfig(stiffness_normal=50.0, stiffness_tangential=30.0, damping_normal=0.2,
                                   damping_tangential=0.1, pp_friction=0.3, pw_friction=0.3)
    return HertzContactConfig(pp_friction=0.3, pw_friction=0.3, pp_restitution=0.9, pw_restitution=0.9)


def _grid(side, spacing, origin=4.0):
    g = np.stack(np.meshgrid(*[np.arange(s) for s in side], indexing="ij"), -1).reshape(-1, 3)
    return origin + g * spacing


def _case(name):
    """(domain, periodic, compat, model, positions, radii, velocities, options)"""
    rng = np.random.default_rng(3)
    if name == "single":          # one particle onto the floor
        return (0, 64, 0, 64, 0, 40), (True, True, False), "reference", "hertz", np.array([[30.0, 30.0, 5.99]]), np.array([6.0]), \
            np.array([[1e-3, 0, -0.01]]), {}
    if name == "pairs":           # a suspension: most alone, some in touching pairs, walls in z
        pos = _grid((9, 9, 9), 6.2)
        pos[1::6, 2] = pos[0::6, 2][:len(pos[1::6])] + 3.999
        pos[2::6, 2] += 1.0
        return (0, 60, 0, 60, 0, 60), (True, True, False), "reference", "hertz", pos, np.full(len(pos), 2.0), \
            rng.normal(0, 0.02, pos.shape), {}
    if name == "loose":           # partners found and lost again, hardly a contact
        pos = _grid((9, 9, 9), 6.5)
        pos = pos + rng.uniform(-1.25, 1.25, pos.shape)
        rad = rng.uniform(1.9, 2.1, len(pos))
        return (0, 60, 0, 60, 0, 60), (True, True, False), "reference", "hertz", pos, rad, rng.normal(0, 0.02, pos.shape), {}
    if name in ("bed", "bed_linear"):    # every sphere touches six, the outer ones the walls
        pos = _grid((7, 7, 6), 3.995, 2.0) + rng.uniform(-2e-3, 2e-3, (294, 3))
        return (0, 27.99, 0, 27.99, 0, 30), (False,) * 3, "reference", "linear" if "linear" in name else "hertz", pos, \
            np.full(len(pos), 2.0), rng.normal(0, 0.01, pos.shape), {}
    if name in ("faces", "faces_wrapped"):   # pairs across the periodic faces, and particles that cross them
        pos = _grid((8, 8, 8), 4.0, 0.02) + rng.uniform(-0.03, 0.03, (512, 3))
        pos = np.mod(pos, 32.0)
        return (0, 32, 0, 32, 0, 32), (True,) * 3, "wrapped" if "wrapped" in name else "reference", "hertz", pos, \
            np.full(len(pos), 2.0), rng.normal(0, 0.03, pos.shape), {}
    if name == "fast":            # beyond the displacement the partner search covers
        pos = _grid((6, 6, 6), 4.5)
        vel = rng.normal(0, 0.02, pos.shape)
        vel[::7, 0] = 1.5
        return (0, 40, 0, 40, 0, 40), (True, True, False), "reference", "hertz", pos, np.full(len(pos), 2.0), vel, {}
    if name == "crowd":           # one large sphere touched by more small ones than a particle may list
        k = np.arange(40)
        th, ph = np.arccos(1 - 2 * (k + 0.5) / 40), np.pi * (1 + 5 ** 0.5) * k
        pos = 16.0 + 4.79 * np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1)
        pos = np.concatenate([np.array([[16.0, 16.0, 16.0]]), pos])
        rad = np.concatenate([[4.0], np.full(40, 0.8)])
        return (0, 40, 0, 40, 0, 40), (False,) * 3, "reference", "hertz", pos, rad, rng.normal(0, 0.01, pos.shape), {"max_coord": 48}
    if name == "frozen":          # frozen and fixed-velocity particles among free ones
        pos = _grid((5, 5, 5), 3.99)
        freeze = np.zeros(len(pos), np.int32)
        freeze[::3] = 1
        return (0, 30, 0, 30, 0, 30), (True, True, False), "reference", "hertz", pos, np.full(len(pos), 2.0), \
            rng.normal(0, 0.02, pos.shape), {"freeze": freeze}
    raise KeyError(name)


def _run(monkeypatch, mode, name, calls):
    dom, per, compat, model, pos, rad, vel, opt = _case(name)
    opt = dict(opt)
    if mode is None:
        monkeypatch.delenv("LBDEM_DEM_KERNELS", raising=False)
    else:
        monkeypatch.setenv("LBDEM_DEM_KERNELS", mode)
    mass = 2.0 * 4.0 / 3.0 * np.pi * rad ** 3
    dem = make_dem(tuple(float(v) for v in dom), 0.05, (0, 0, -1e-3), _contact(model), rad, mass, pos, vel, periodic=per,
                   max_coord=opt.pop("max_coord", 24), E=1e3, wall_E=1e3, model=model, compat=compat, **opt)
    rng = np.random.default_rng(5)
    dem.gf.omega.from_numpy(rng.normal(0, 0.02, pos.shape))
    dem.gf.force_fluid.from_numpy(rng.normal(0, 1e-3, pos.shape))
    dem.gf.moment_fluid.from_numpy(rng.normal(0, 1e-3, pos.shape))
    for n in calls:
        dem.run_substeps(n)
    dem.check_status()
    monkeypatch.delenv("LBDEM_DEM_KERNELS", raising=False)
    return dem


# 37 sub-steps cross the partner search's chunk of 16 twice; an odd count flips the broad phase's half
@pytest.mark.parametrize("calls", [(10, 10), (37, 2, 1)])
@pytest.mark.parametrize("name", ["single", "pairs", "loose", "bed", "bed_linear", "faces", "faces_wrapped", "fast", "crowd", "frozen"])
def test_flow_matches_split_kernels(name, calls, monkeypatch):
    a, b = _run(monkeypatch, "flow", name, calls), _run(monkeypatch, "split", name, calls)
    ca, cb = a.active_contacts(), b.active_contacts()
    assert set(ca) == set(cb)
    if name not in ("single", "loose", "crowd"):      # (the crowd has bounced off by the end)
        assert len(ca) > 3
    for q in range(3):
        x, y = np.array([ca[p][q] for p in sorted(ca)]), np.array([cb[p][q] for p in sorted(cb)])
        if len(ca):
            assert np.abs(x - y).max() <= 1e-8 * max(np.abs(y).max(), 1e-12)
    for k in STATE:
        x, y = getattr(a.gf, k).to_numpy(), getattr(b.gf, k).to_numpy()
        tol = 1e-11 if k == "position" else 1e-8 * np.abs(y).max()
        assert np.abs(x - y).max() <= tol, k
    np.testing.assert_array_equal(a.wcf_active.cpu().numpy(), b.wcf_active.cpu().numpy())
    on = b.wcf_active.cpu().numpy().astype(bool)
    for k in ("wcf_shear", "wcf_force"):
        x, y = getattr(a, k).cpu().numpy()[on], getattr(b, k).cpu().numpy()[on]
        if len(y):
            assert np.abs(x - y).max() <= 1e-8 * max(np.abs(y).max(), 1e-12)
    # what the next call relies on: no pending slots, accumulators and barrier words clear
    assert not a.cf_add.any() and not a.acc_force.any() and not a.acc_moment.any() and not a.sync.any()
    assert not a.flow[:8].any()
    np.testing.assert_array_equal(a.cfn.cpu().numpy(), b.cfn.cpu().numpy())


def test_flow_reports_a_full_contact_list(monkeypatch):
    """More contacts than max_coordinate_number: flagged as by the two-phase form."""
    import lbdem_taichi_b200._native as N
    monkeypatch.delenv("LBDEM_DEM_KERNELS", raising=False)
    pos = np.array([[5.0, 5.0, 5.0], [6.0, 5.0, 5.0], [5.5, 6.0, 5.0]])
    rad = np.ones(3)
    dem = make_dem((0, 10, 0, 10, 0, 10), 1e-3, (0, 0, 0), _contact("hertz"), rad, np.ones(3), pos, np.zeros((3, 3)),
                   max_coord=1)
    dem.run_substeps(4)
    with pytest.raises(N.LbdemError, match="max_coordinate_number"):
        dem.check_status()
