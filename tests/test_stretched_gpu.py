"""Stretched x / y grids: second derivatives hold their first-derivative part
apart from the large one, as on every other path, so that a uniform field has
none at all.  (With merged factors b + a and b - a its derivative is b times
the field's rounding instead.)
"""
import numpy as np
import pytest

from mhd_gb300.case import STATE_FIELDS, small_cases, tanh_metric
from mhd_gb300.sim import Batch, Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shr", [False, True])
@pytest.mark.parametrize("form", ["alone", "batch"])
def test_uniform_fields_stay_uniform(form, shr):
    """A gas at rest without gravity in a uniform field, diffusive enough that
    the smallest error of a Laplacian shows in one step: away from the walls
    every bit stays (each of the three substages carries the walls' influence
    by at most three planes, the one-sided wall stencils included)."""
    case = small_cases()["mhd_fixedT"].replace(nPx=20, nPy=18, nPz=28, lShr=shr, THETA=0.0, GRAV=0.0, RM=1e-3, RE=1e-3, dt=1e-3)
    dx, dy = tanh_metric(case.nPx, case.xMax, 1.1), tanh_metric(case.nPy, case.yMax, 0.9)
    mo = dict(zip(("dxxdx", "d2xxdx2", "DDX", "dyydy", "d2yydy2", "DDY"), dx + dy))
    value = {"RU": 0.0, "RV": 0.0, "RW": 0.0, "TT": 0.7, "RO": 1.0, "BX": 0.3, "BY": 1.0 / 3.0, "BZ": 0.1}
    st = {k: np.full(case.shape, v) for k, v in value.items()}
    sim = Simulation(case, metric_override=mo)
    sim.upload_state(st)
    sim.communicate()
    if form == "batch":
        b = Batch([sim])
        b.set_tile(2)
        b.steps(1)
        b.sync()
        b.close()
    else:
        sim.step(case.dt)
    got = sim.download_state()
    sim.close()
    for k in STATE_FIELDS:
        inner = got[k][11:-11, 1:-1, 1:-1]
        assert (inner == value[k]).all(), (k, np.abs(inner - value[k]).max())
