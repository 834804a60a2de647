"""BCON by its own kernel in FP32-storage batches: z ranges of fewer than three
planes leave the walls to it, longer ones apply BCON where the wall cells are
computed.  The same values either way over several steps: the kernel has to
keep the FP64 register's wall values in step too, or the later steps differ.
"""
import numpy as np
import pytest

from mhd_gb300.case import initial_state, small_cases
from mhd_gb300.sim import Batch, Simulation

pytestmark = pytest.mark.gpu


def run(sw, zmax):
    base = small_cases()[sw]
    cases = [base.replace(nPx=nx, nPy=ny, nPz=nz, seed=i) for i, (nx, ny, nz) in
             enumerate([(20, 12, 4), (17, 9, 7), (32, 8, 11)])]
    sims = []
    for c in cases:
        s = Simulation(c, precision="fp32")
        s.upload_state(initial_state(c))
        s.communicate()
        sims.append(s)
    b = Batch(sims)
    b.set_tile(0)
    b.set_zrange(zmax)
    b.steps(3)
    b.sync()
    b.close()
    for s in sims:  # the register as the single instance's step reads it
        s.step(s.case.dt)
    out = [s.download_state() for s in sims]
    for s in sims:
        s.close()
    return out


@pytest.mark.parametrize("zmax", [1, 2, 3, 5])
@pytest.mark.parametrize("sw", ["mhd_rot_flux", "mhd_rot_shr", "hydro_default_bc"])
def test_fp32_batch_walls_for_short_z_ranges(sw, zmax):
    for got, ref in zip(run(sw, zmax), run(sw, 64)):
        for k in got:
            assert np.array_equal(got[k], ref[k]), k
