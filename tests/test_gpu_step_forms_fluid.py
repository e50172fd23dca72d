"""The form of the gathered step that the size rule picks for 16-bit storage
without particles, at the rule's edges: which kernel runs, and the same
populations, lagged state and moments as the gathers, bit for bit (the same
arithmetic on the same inputs), with and without walls.  The term of a wall that
moves is contracted into multiply-adds differently from kernel to kernel, a last
FP32 bit: there stored values may round the other way, in each of the three
steps once, so that values of magnitude up to m differ by up to three units of
their last place, 3 x 2^-10 m (FP16) or 3 x 2^-7 m (BF16)."""
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(mode, shape, storage, smag, wall):
    from lbdem_taichi_b200 import _native as N
    from lbdem_taichi_b200.lbm3d.lattice import BasicLattice3D
    os.environ["LBDEM_STEP_KERNEL"] = mode
    try:
        rng = np.random.default_rng(9)
        lat = BasicLattice3D(*shape, 1 / 0.55, 1.0, 1.0, 1.0, storage=storage, smagorinsky=smag)
        if wall:
            ct = np.ones(shape, np.int32)
            ct[:, :, 0] = wall
            ct[7, 5, 9] = 8
            lat.CT.from_numpy(ct)
        lat.vel.from_numpy(0.03 * rng.uniform(-1, 1, (*shape, 3)))
        lat.initialize()
        for _ in range(3):
            lat.collide()
            lat.stream()
        form = N.load().lbdem_psc_step_form_last()
        out = [lat._f[lat._cur].clone(), lat.rho.to_numpy(), lat.vel.to_numpy()]
        if lat._aux is not None:
            out.append(lat._aux.clone())
        return form, out
    finally:
        os.environ.pop("LBDEM_STEP_KERNEL", None)


ONE, ROWS, PAIRS = 0, 1, 2


@pytest.mark.parametrize("shape,storage,smag,form,wall", [
    ((226, 64, 64), "f16", "off", PAIRS, None), ((226, 63, 65), "f16", "off", ONE, None),
    ((256, 128, 192), "bf16", "off", PAIRS, 8), ((252, 128, 193), "f16", "off", ONE, None),
    ((240, 192, 193), "bf16", "off", PAIRS, None), ((256, 192, 193), "f16", "off", ONE, 8),
    ((250, 131, 96), "f16", "local", PAIRS, 32), ((256, 96, 128), "bf16", "reference", PAIRS, 8),
    ((256, 97, 128), "f16", "reference", ONE, None), ((192, 64, 128), "f16", "reference", PAIRS, 32),
    ((192, 63, 130), "f16", "local", ONE, None), ((251, 64, 128), "f16", "local", ROWS, 32),
    ((223, 64, 128), "bf16", "reference", ROWS, 8), ((251, 64, 128), "f16", "off", ONE, None),
    ((251, 128, 193), "f16", "reference", ONE, None), ((128, 64, 128), "bf16", "local", ONE, None),
    ((288, 64, 128), "f16", "local", ONE, None),
])
def test_chosen_form(shape, storage, smag, form, wall):
    ran, got = _run("auto", shape, storage, smag, wall)
    assert ran == form
    _, want = _run("simt", shape, storage, smag, wall)
    for g, w in zip(got, want):
        g, w = torch.as_tensor(g).double(), torch.as_tensor(w).double()
        if wall == 32:
            live = w > -4000.0         # (cells never written keep f = 0)
            ulp = 2.0 ** (-10 if storage == "f16" else -7)
            assert (g - w).abs().max() <= 3 * ulp * w[live].abs().max()
        else:
            assert torch.equal(g, w)
