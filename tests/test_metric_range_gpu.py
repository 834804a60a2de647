"""Uniform grids whose x spacing is far from the other axes': the kernels that work in
units of the x metric factor leave them to the general ones, before a square of a y or
z derivative in that unit leaves the double range.  One step against the oracle, 1e-12
of each field's max-norm, the bound of every fused-path comparison.
"""
import pytest

from gpu_util import oracle_for, rel_err
from mhd_gb300.case import STATE_FIELDS, initial_state, small_cases
from mhd_gb300.sim import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xmax", [1e180, 1e58, 1e55, 1e30])
@pytest.mark.parametrize("sw", ["mhd_rot_flux", "hydro_default_bc"])
def test_one_step_with_a_far_x_spacing(sw, xmax):
    case = small_cases()[sw].replace(nPx=17, nPy=9, nPz=8, xMax=xmax)
    st = initial_state(case)
    sim = Simulation(case)
    sim.upload_state(st)
    sim.communicate()
    sim.step(case.dt)
    got = sim.download_state()
    sim.close()
    o = oracle_for(case, st)
    o.steps(1)
    for k in STATE_FIELDS[:case.nfields]:
        assert rel_err(got[k], o.arr[k]) <= 1e-12, (k, rel_err(got[k], o.arr[k]))
