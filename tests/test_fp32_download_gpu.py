"""Downloads of an FP32-storage state: they keep no device memory, and stepping
goes on from them as if they had not been made (the values pass through the
buffer that the next step writes, whose z ghost planes no step writes).
"""
import numpy as np
import pytest

from mhd_gb300.case import STATE_FIELDS, initial_state, small_cases
from mhd_gb300.sim import Batch, Simulation

pytestmark = pytest.mark.gpu

# the second has more elements than a piece of the download holds
SIZES = [(20, 12, 9), (100, 90, 60)]


def started(size, sw="mhd_fixedT"):
    nx, ny, nz = size
    case = small_cases()[sw].replace(nPx=nx, nPy=ny, nPz=nz)
    st = initial_state(case)
    for k in STATE_FIELDS[:case.nfields]:  # ghost planes that no neighbour holds
        st[k][0], st[k][-1] = 1.25 * st[k][1] + 0.5, 0.75 * st[k][-2] + 0.25
    sim = Simulation(case, precision="fp32")
    sim.upload_state(st)
    sim.communicate()
    return case, sim


def whole(sim):
    import ctypes as C
    out = np.empty((sim.case.nfields,) + sim.case.shape)
    assert sim.L.mhd_download_state(sim.ctx, out.ctypes.data_as(C.POINTER(C.c_double))) == 0
    return out


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("sw", ["mhd_fixedT", "hydro_default_bc"])
def test_download_keeps_no_memory_and_changes_nothing(size, sw):
    _, ref = started(size, sw)
    case, sim = started(size, sw)
    before = sim.device_bytes()
    assert np.array_equal(whole(sim), whole(ref))
    assert sim.device_bytes() == before
    for n in (1, 2, 3):
        sim.steps(n)
        before = sim.device_bytes()
        state = whole(sim)
        assert sim.device_bytes() == before
        for i, k in enumerate(STATE_FIELDS[:case.nfields]):
            assert np.array_equal(sim.download(k), state[i]), k
    ref.steps(6)
    assert np.array_equal(state, whole(ref))
    sim.close()
    ref.close()


def test_batch_goes_on_after_downloads():
    sizes = [(20, 12, 9), (33, 8, 6)]

    def run(read):
        sims = [started(s)[1] for s in sizes]
        b = Batch(sims)
        b.set_tile(0)
        for _ in range(3):
            b.steps(1)
            if read:
                for s in sims:
                    whole(s)
                    s.download("TT")
        b.sync()
        out = [whole(s) for s in sims]
        b.close()
        for s in sims:
            s.close()
        return out

    for got, ref in zip(run(True), run(False)):
        assert np.array_equal(got, ref)


def test_downloads_of_several_threads():
    """Downloads at the same time, of which one holds the shared buffer and the
    others go through their own contexts: each gets its state, and stepping goes
    on from it."""
    from concurrent.futures import ThreadPoolExecutor
    sizes = [(20, 12, 9), (33, 8, 6), (64, 48, 40), (70, 60, 50)]
    sims = [started(s)[1] for s in sizes]
    refs = [started(s)[1] for s in sizes]
    for s in sims + refs:
        s.steps(2)
    want = [whole(s) for s in refs]

    def often(sim):
        return [whole(sim) for _ in range(20)]

    with ThreadPoolExecutor(len(sims)) as ex:
        got = list(ex.map(often, sims))
    for g, w in zip(got, want):
        for a in g:
            assert np.array_equal(a, w)
    for s, r in zip(sims, refs):
        s.steps(3)
        r.steps(3)
        assert np.array_equal(whole(s), whole(r))
        s.close()
        r.close()
