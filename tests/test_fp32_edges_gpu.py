"""The FP32-storage substage at the edges of its tiles (32 columns by 4
or 5 rows) and of its z ranges, on isotropic, unequal and stretched x / y
spacings: one step against the oracle within 1e-5 of each field's max-norm (the bound of the FP32-storage
form: its stencils work on floats, 6e-8, amplified by at most the 1e2 of the
differenced terms), and a non-finite state that stays non-finite where it is
and finite elsewhere.
"""
import numpy as np
import pytest

from gpu_util import METRIC_NAMES, rel_err
from mhd_gb300.case import STATE_FIELDS, initial_state, small_cases, tanh_metric
from mhd_gb300.sim import Simulation

pytestmark = pytest.mark.gpu

SIZES = [(31, 7, 4), (32, 8, 5), (33, 9, 6), (2, 2, 4), (64, 17, 7), (40, 25, 33),
         # large enough for tiles of 5 rows: remainders 1, 4, 0
         (97, 201, 9), (97, 224, 9), (161, 25, 20)]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("grid", ["isotropic", "unequal", "stretched"])
@pytest.mark.parametrize("sw", ["mhd_rot_flux", "mhd_rot_shr", "hydro_default_bc"])
def test_one_step_at_tile_edges(size, grid, sw):
    import oracle
    nx, ny, nz = size
    case = small_cases()[sw].replace(nPx=nx, nPy=ny, nPz=nz, xMax=3.0)
    case = case.replace(yMax=3.0 * (ny - 1) / (nx - 1) if grid == "isotropic" else 2.0)
    mo = {}
    if grid == "stretched":
        dx, dy = tanh_metric(nx, case.xMax, 0.8), tanh_metric(ny, case.yMax, 0.6)
        mo = dict(zip(("dxxdx", "d2xxdx2", "DDX", "dyydy", "d2yydy2", "DDY"), dx + dy))
    st = initial_state(case)
    sim = Simulation(case, precision="fp32", metric_override=mo or None)
    sim.upload_state(st)
    sim.communicate()
    sim.step(case.dt)
    got = sim.download_state()
    sim.close()
    o = oracle.OracleSim(case, st)
    for n, a in mo.items():
        o._metric_arrays[METRIC_NAMES.index(n)][:] = a
    o.communicate()
    o.steps(1)
    for k in STATE_FIELDS[:case.nfields]:
        assert rel_err(got[k], o.arr[k]) <= 1e-5, (k, rel_err(got[k], o.arr[k]))


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_cells_stay_non_finite(value):
    """A non-finite momentum in one cell makes the cells that its step reaches
    non-finite and leaves the others finite (right-hand sides and register
    values outside the ordinary float range take the general conversions)."""
    case = small_cases()["mhd_fixedT"].replace(nPx=40, nPy=20, nPz=16)
    st = initial_state(case)
    st["RU"][8, 10, 12] = value
    sim = Simulation(case, precision="fp32")
    sim.upload_state(st)
    sim.communicate()
    sim.step(case.dt)
    got = sim.download_state()
    d = sim.diagnostics(check=False)
    sim.close()
    assert d["flags"] & 1
    for k in STATE_FIELDS:
        bad = ~np.isfinite(got[k])
        zz, yy, xx = np.nonzero(bad)
        assert bad.any()
        assert np.abs(zz - 8).max() <= 3 and np.abs(yy - 10).max() <= 3 and np.abs(xx - 12).max() <= 3, k


def test_download_widens_every_piece():
    """The state comes back as its stored floats plus the profiles, in pieces:
    a grid of more elements than one piece holds, whole and field by field, is
    what was uploaded to the rounding of one float of the deviation (and
    exactly the same values either way)."""
    case = small_cases()["mhd_fixedT"].replace(nPx=100, nPy=90, nPz=60)
    st = initial_state(case)
    sim = Simulation(case, precision="fp32")
    sim.upload_state(st)
    got = sim.download_state()
    whole = np.empty((8,) + case.shape)
    import ctypes as C
    assert sim.L.mhd_download_state(sim.ctx, whole.ctypes.data_as(C.POINTER(C.c_double))) == 0
    sim.close()
    assert whole.size > 2 << 20  # the piece length, in elements
    for i, k in enumerate(STATE_FIELDS):
        assert np.array_equal(whole[i], got[k]), k
        mean = st[k][:, 1:-1, 1:-1].mean(axis=(1, 2))[:, None, None] if k in ("RO", "TT") else 0.0
        bound = 2.0 ** -24 * np.abs(st[k] - mean) + 2.0 ** -50 * np.abs(st[k]) + 2.0 ** -149
        assert (np.abs(got[k] - st[k]) <= bound).all(), k
