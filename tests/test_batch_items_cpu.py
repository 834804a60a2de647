"""The check of a batch's work items and arguments, on the host: the function
that the kernels call before they touch memory is compiled for the CPU and fed
arguments that must not pass.
"""
import subprocess

import pytest

from conftest import REPO

PROGRAM = r"""
#include "mhd_common.cuh"
#include <cstdio>
using namespace mhd;
template <class A> A args(int nx, int ny, int nz) {
    A a{};
    a.g.nx = nx; a.g.ny = ny; a.g.nz = nz; a.g.nPz = nz - 2; a.g.sy = nx; a.g.sz = (long long)nx * ny;
    return a;
}
static double mem[3 * 8 * 20000];
static float mem32[2 * 8 * 20000];
int main() {
    const int nx = 34, ny = 18, nz = 9;
    const long long n = (long long)nx * ny * nz;
    FusedArgs good = args<FusedArgs>(nx, ny, nz);
    good.fs = n;
    for (int f = 0; f < 8; f++) {
        good.U.p[f] = mem + f * n;
        good.Uo.p[f] = mem + (8 + f) * n;
        good.Z.p[f] = mem + (16 + f) * n;
    }
    Fused32Args good32 = args<Fused32Args>(nx, ny, nz);
    for (int f = 0; f < 8; f++) {
        good32.U.p[f] = mem32 + f * n;
        good32.Uo.p[f] = mem32 + (8 + f) * n;
        good32.Z.p[f] = mem + f * n;
    }
    const int4 item = make_int4(0, 1, 3, 1 | (8 << 16));
    auto say = [&](const char* what, auto a, int4 it, int nf = 8) {
        printf("%s %d\n", what, batch_item_code(1, &a, it, 16, 4, nf));
    };
    say("good", good, item);
    say("good32", good32, item);
    say("instance", good, make_int4(1, 1, 3, item.w));
    say("tile", good, make_int4(0, 2, 3, item.w));
    say("range", good, make_int4(0, 1, 3, 1 | (9 << 16)));
    { auto a = good; a.g.sz++; say("sizes", a, item); }
    { auto a = good; a.Z.p[7] = nullptr; say("null", a, item); say("null_hydro", a, item, 5); }
    { auto a = good32; a.Uo.p[3] = nullptr; say("null32", a, item); }
    { auto a = good; a.fs = 0; say("distance_unset", a, item); }
    { auto a = good; a.fs = n - 1; say("distance_short", a, item); }
    { auto a = good; a.U.p[2] += 1; say("field_elsewhere", a, item); }
    { auto a = good; a.Uo.p[4] -= n; say("written_field_elsewhere", a, item); }
    { auto a = good; for (int f = 0; f < 8; f++) a.Z.p[f] = mem + f; say("register_elsewhere", a, item); }
}
"""
EXPECT = {"good": 0, "good32": 0, "instance": 1, "tile": 3, "range": 4, "sizes": 2, "null": 5, "null_hydro": 0,
          "null32": 5, "distance_unset": 5, "distance_short": 5, "field_elsewhere": 5, "written_field_elsewhere": 5,
          "register_elsewhere": 5}


@pytest.fixture(scope="module")
def codes(tmp_path_factory):
    import importlib.util
    spec = importlib.util.spec_from_file_location("mhd_build", REPO / "rast-3dmhd-cpp_gb300" / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    d = tmp_path_factory.mktemp("items")
    (d / "items.cu").write_text(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++20", "--expt-relaxed-constexpr", "-I", str(build.CSRC),
                    "-o", str(d / "items"), str(d / "items.cu")], check=True)
    out = subprocess.run([str(d / "items")], check=True, capture_output=True, text=True).stdout
    return {k: int(v) for k, v in (line.split() for line in out.splitlines())}


def test_every_form_is_named(codes):
    assert codes.keys() == EXPECT.keys()


@pytest.mark.parametrize("form", sorted(EXPECT))
def test_item_check(codes, form):
    assert codes[form] == EXPECT[form]
