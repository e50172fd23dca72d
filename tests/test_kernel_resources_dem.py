"""Register and spill budgets of the one-launch DEM form, the adjoint step and the
tall-lattice step, from the ptxas reports (no GPU needed).

- k_dem_flow at two blocks of 128 threads per SM: 255 registers; 8 lanes per
  particle spill at most 128 bytes, 4 lanes 256; at three blocks 168 registers
  and at most 1536 bytes (a particle's eight pairs do not fit);
- k_psc_adjoint: 85 registers (three blocks of 256 threads per SM), no spills;
- k_psc_step_tall: 128 registers, no spills.
"""
import pytest

from tests.test_kernel_resources import _match, _resources


@pytest.fixture(scope="module")
def res():
    return _resources()


@pytest.mark.parametrize("lanes,blocks,regs,spill", [(8, 2, 255, 128), (4, 2, 255, 256), (4, 3, 168, 1536), (2, 3, 168, 1536)])
def test_dem_flow(res, lanes, blocks, regs, spill):
    got = _match(res, rf"k_dem_flowILb[01]ELi{lanes}ELi{blocks}E")
    assert len(got) == 2
    assert all(r <= regs and s <= spill for r, s in got.values()), got


def test_adjoint(res):
    got = _match(res, "k_psc_adjointI")
    assert len(got) == 4
    assert all(r <= 85 and s == 0 for r, s in got.values()), got


def test_tall_step(res):
    got = _match(res, "k_psc_step_tallI")
    assert len(got) == 3 * 2 * 3 * 2
    assert all(r <= 128 and s == 0 for r, s in got.values()), got
