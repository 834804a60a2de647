"""The fused FP64 substage at the edges of its 16 x 8 tile and of its z
ranges: sizes one below, at and one above a tile in x and y (the last tile
then holds one column or row, whose right neighbours are ghost columns of the
same tile or halo points), and the fewest planes, on isotropic and on unequal
x / y spacings, and on a stretched x / y grid.  One step against the oracle;
1e-12 of each field's max-norm, the bound of every fused-path comparison:
regrouped sums of about 200 FP64 operations per cell differ by rounding only.
"""
import numpy as np
import pytest

from gpu_util import METRIC_NAMES, rel_err
from mhd_gb300.case import STATE_FIELDS, initial_state, small_cases, tanh_metric
from mhd_gb300.sim import Batch, Simulation

pytestmark = pytest.mark.gpu

SIZES = [(15, 7, 4), (16, 8, 5), (17, 9, 6), (31, 8, 7), (33, 17, 4), (2, 2, 4), (16, 2, 9), (18, 25, 33),
         # tiles of different numbers of z ranges (25 and 26, 30 and 31, 22 and 23)
         (33, 41, 83), (65, 17, 104), (49, 33, 76)]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("grid", ["isotropic", "unequal", "stretched"])
@pytest.mark.parametrize("sw", ["mhd_rot_flux", "mhd_rot_shr", "hydro_default_bc"])
def test_one_step_at_tile_edges(size, grid, sw):
    nx, ny, nz = size
    case = small_cases()[sw].replace(nPx=nx, nPy=ny, nPz=nz, xMax=3.0)
    # isotropic: equal spacings xMax/(nx-1) = yMax/(ny-1)
    case = case.replace(yMax=3.0 * (ny - 1) / (nx - 1) if grid == "isotropic" else 2.0)
    mo = {}
    if grid == "stretched":
        dx, dy = tanh_metric(nx, case.xMax, 0.8), tanh_metric(ny, case.yMax, 0.6)
        mo = dict(zip(("dxxdx", "d2xxdx2", "DDX", "dyydy", "d2yydy2", "DDY"), dx + dy))
    st = initial_state(case)
    sim = Simulation(case, path="fused", metric_override=mo or None)
    sim.upload_state(st)
    sim.communicate()
    sim.step(case.dt)
    got = sim.download_state()
    sim.close()
    import oracle
    o = oracle.OracleSim(case, st)
    for n, a in mo.items():
        o._metric_arrays[METRIC_NAMES.index(n)][:] = a
    o.communicate()
    o.steps(1)
    for k in STATE_FIELDS[:case.nfields]:
        assert rel_err(got[k], o.arr[k]) <= 1e-12, (k, rel_err(got[k], o.arr[k]))


@pytest.mark.parametrize("zmax", [1, 2, 3, 5])
def test_batch_walls_for_short_z_ranges(zmax):
    """Z ranges of fewer than three planes leave BCON to its own kernel, longer
    ones apply it where the wall cells are computed: the same values either
    way, as each cell's arithmetic does not depend on the range it lies in."""
    base = small_cases()["mhd_fixedT"].replace(izCon=1, iTCon=1)
    cases = [base.replace(nPx=nx, nPy=ny, nPz=nz, seed=i) for i, (nx, ny, nz) in
             enumerate([(20, 12, 4), (17, 9, 7), (32, 8, 11)])]

    def run(z):
        sims = []
        for c in cases:
            s = Simulation(c)
            s.upload_state(initial_state(c))
            s.communicate()
            sims.append(s)
        b = Batch(sims)
        b.set_tile(2)
        b.set_zrange(z)
        b.steps(3)
        b.sync()
        out = [s.download_state() for s in sims]
        b.close()
        for s in sims:
            s.close()
        return out

    for got, ref in zip(run(zmax), run(64)):
        for k in STATE_FIELDS:
            assert np.array_equal(got[k], ref[k]), k
