"""Launches that start while the kernel before them drains, between a caller's
own kernels on a caller's stream and in a captured graph: the results of the
plain calls, bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

from mhd_gb300 import abi
from mhd_gb300.case import STATE_FIELDS, initial_state, metrics, small_cases
from mhd_gb300.sim import Simulation, params_for

pytestmark = pytest.mark.gpu

# a separate BCON launch; equal z ranges; tiles of different numbers of z ranges
SIZES = [(20, 12, 4), (40, 20, 12), (33, 41, 83)]


def case_of(size, sw="mhd_rot_flux"):
    nx, ny, nz = size
    return small_cases()[sw].replace(nPx=nx, nPy=ny, nPz=nz)


def started(case, prec, stream=None):
    if stream is None:
        sim = Simulation(case, precision=prec)
    else:
        sim = Simulation.__new__(Simulation)
        sim.case, sim.L, sim.timt, sim.ctx = case, abi.load(), 0.0, C.c_void_p()
        p, sim._keep = params_for(case, "fused", prec)
        abi.check(sim.L.mhd_create(C.byref(p), stream.cuda_stream, C.byref(sim.ctx)))
    sim.upload_state(initial_state(case))
    sim.communicate()
    return sim


def busy(torch):
    """A caller's kernels: some hundred microseconds of work."""
    a = torch.ones((2048, 2048), device="cuda")
    for _ in range(4):
        a = a @ a * 1e-4
    return a


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_steps_between_a_callers_kernels(size, prec):
    torch = pytest.importorskip("torch")
    case = case_of(size)
    ref = started(case, prec)
    stream = torch.cuda.Stream()
    sim = started(case, prec, stream)
    with torch.cuda.stream(stream):
        busy(torch)
        sim.steps(2)
        busy(torch)
        sim.steps_cfl(3)
        busy(torch)
    ref.steps(2)
    ref.steps_cfl(3)
    got, want = sim.download_state(), ref.download_state()
    for k in STATE_FIELDS:
        assert np.array_equal(got[k], want[k]), k
    sim.close()
    ref.close()


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_captured_steps(size, prec):
    """An even number of steps leaves the buffers as they were, so that its graph can be replayed."""
    torch = pytest.importorskip("torch")
    case = case_of(size)
    ref = started(case, prec)
    stream = torch.cuda.Stream()
    sim = started(case, prec, stream)
    sim.steps(2)  # every buffer is there before the capture
    sim.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sim.steps(2)
    with torch.cuda.stream(stream):
        for _ in range(3):
            graph.replay()
    stream.synchronize()
    ref.steps(8)
    got, want = sim.download_state(), ref.download_state()
    for k in STATE_FIELDS:
        assert np.array_equal(got[k], want[k]), k
    sim.close()
    ref.close()


def noalloc_args(torch, case, state, flux):
    m = metrics(case)
    a = abi.MhdFluxesNoallocArgs()
    a.nPx, a.nPy, a.nPz = case.nPx, case.nPy, case.nPz
    a.switches = (abi.SW_LROT if case.lRot else 0) | (abi.SW_LMAG if case.lMag else 0)
    a.izCon, a.iTCon, a.iBCon = case.izCon, case.iTCon, case.iBCon
    for k in ("RE", "PR", "THETA", "GRAV", "RY", "ANG", "RM", "BETA", "TP", "GAMMA", "SFF"):
        setattr(a, k, float(getattr(case, k)))
    a.TB = case.tb
    keep = [torch.tensor(v, dtype=torch.float64, device="cuda") for v in m.arrays()]
    for n, t in zip(("dxxdx", "d2xxdx2", "DDX", "dyydy", "d2yydy2", "DDY", "dzzdz", "d2zzdz2", "DDZ", "RKAPA", "DKAPA"), keep):
        setattr(a, n, t.data_ptr())
    for f in range(state.shape[0]):
        a.state[f] = state[f].data_ptr()
        a.flux[f] = flux[f].data_ptr()
    return a, keep


@pytest.mark.parametrize("captured", [False, True])
def test_fluxes_between_a_callers_kernels(captured):
    """The state is written by a kernel just before the call, overwritten by
    one just after it, and the right-hand sides are read by the next."""
    torch = pytest.importorskip("torch")
    case = case_of((40, 20, 12))
    lib = abi.load()
    st = initial_state(case)
    src = torch.tensor(np.stack([st[k] for k in STATE_FIELDS]), device="cuda")
    state, flux = src.clone(), torch.zeros_like(src)
    args, keep = noalloc_args(torch, case, state, flux)
    abi.check(lib.mhd_fluxes_noalloc(C.byref(args), None))
    torch.cuda.synchronize()
    want = flux.clone()
    stream = torch.cuda.Stream()
    got = []

    def once():
        state.copy_(src)
        abi.check(lib.mhd_fluxes_noalloc(C.byref(args), torch.cuda.current_stream().cuda_stream))
        copy = flux * 1.0
        state.fill_(1.0)
        flux.zero_()
        return copy

    with torch.cuda.stream(stream):
        state.zero_()
        flux.zero_()
        busy(torch)
    stream.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = once()
        with torch.cuda.stream(stream):
            for _ in range(3):
                busy(torch)
                graph.replay()
                got.append(out.clone())
    else:
        with torch.cuda.stream(stream):
            for _ in range(3):
                busy(torch)
                got.append(once())
    stream.synchronize()
    for g in got:
        assert torch.equal(g, want)
