"""Rows of the CFL reduction whose smallest spacing is the x spacing: on a
uniform x grid they are filtered like the others (their DD is the same in every
cell), on a stretched one they are evaluated cell by cell; DT and UMACH equal
the oracle's bit for bit either way, for row lengths around a warp's passes
(32 lanes, groups of 2 and 4 cells, passes of 256)."""
import numpy as np
import pytest

from gpu_util import METRIC_NAMES
from mhd_gb300.case import initial_state, small_cases, tanh_metric
from mhd_gb300.sim import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [2, 31, 33, 128, 129, 257, 300])
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("mag", [True, False])
def test_dt_where_the_x_spacing_is_smallest(nx, stretched, mag):
    import oracle
    # x spacing 0.5/(nx-1) below the z spacings (2/7 in the middle) and y's
    case = small_cases()["mhd_fixedT"].replace(nPx=nx, nPy=5, nPz=8, xMax=0.5, yMax=6.0, lMag=mag, seed=nx)
    st = initial_state(case)
    rng = np.random.default_rng(nx)
    for k in ("RU", "RV", "RW"):
        st[k] += 0.1 * rng.standard_normal(st[k].shape)
    mo = {}
    if stretched:
        mo = dict(zip(("dxxdx", "d2xxdx2", "DDX"), tanh_metric(nx, case.xMax, 0.8)))
    sim = Simulation(case, metric_override=mo or None)
    sim.upload_state(st)
    sim.communicate()
    dt, um = sim.cfl_dt()
    sim.close()
    o = oracle.OracleSim(case, st)
    for n, a in mo.items():
        o._metric_arrays[METRIC_NAMES.index(n)][:] = a
    o.communicate()
    ref_dt, ref_um = o.cfl_dt()
    assert dt == ref_dt and um == ref_um
