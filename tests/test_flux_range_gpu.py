"""The unfused right-hand sides at the end of the double range: where the
reference's 2 F overflows, so does ours (bit for bit, any NaN counting as any
other)."""
import numpy as np
import pytest

from gpu_util import oracle_for
from mhd_gb300.case import FLUX_FIELDS, initial_state, small_cases
from mhd_gb300.sim import Simulation

pytestmark = pytest.mark.gpu

# below, at and above half of the largest double (2^1023 and its neighbours among them)
VALUES = [np.nextafter(2.0 ** 1023, 0), 2.0 ** 1023, -(2.0 ** 1023), 1e308, -1.7e308, np.finfo(float).max]


@pytest.mark.parametrize("value", VALUES)
@pytest.mark.parametrize("field", ["TT", "BX", "RU"])
@pytest.mark.parametrize("everywhere", [True, False])
def test_second_differences_overflow_as_the_reference(field, value, everywhere):
    case = small_cases()["mhd_rot_flux"].replace(lMag=True, nPx=9, nPy=8, nPz=7, xMax=1e3, yMax=1e3)
    st = initial_state(case)
    if everywhere:
        st[field][:] = value
    else:
        st[field][4, 4, 5] = value
    sim = Simulation(case, path="parity")
    sim.upload_state(st)
    sim.communicate()
    sim.fluxes()
    o = oracle_for(case, st)
    with np.errstate(all="ignore"):
        o.fluxes()
    for k in FLUX_FIELDS:
        got, want = (a[1:-1, 1:-1, 1:-1] for a in (sim.download(k), o.arr[k]))
        assert np.array_equal(got, want, equal_nan=True), (k, int((got != want).sum()))
    sim.close()
