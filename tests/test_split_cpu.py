"""The cut of a substage launch into blocks (tile, z range): every plane of every
tile is computed by exactly one block, and the sizes of the edge tests reach the
kernels that they are meant for.
"""
import subprocess

import pytest

from conftest import REPO
from test_fp32_edges_gpu import SIZES as SIZES32
from test_fused_edges_gpu import SIZES as SIZES64

SMS = 152
PROGRAM = r"""
#include "mhd_split.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
using namespace mhd;

// the blocks of a split as the kernels take them; 0 when they are as they should be
static int check(int lo, int planes, int nbx, int tiles, long long n) {
    const ZSplit s = make_split(lo, planes, nbx, tiles, n);
    std::vector<int> hits((size_t)tiles * planes, 0);
    int first = planes, last = planes, before = 1 << 30;
    for (int b = 0; b < n; b++) {
        int tile, zb, ze;
        if (s.ranges) {
            const int r = b / tiles;
            tile = b % tiles;
            zb = lo + (int)((long long)planes * r / s.ranges);
            ze = lo + (int)((long long)planes * (r + 1) / s.ranges);
        } else {
            int j = b;
            const ZSplit::Class k = block_class(s, j);
            if (j >= k.blocks) return 1;
            tile = k.tile0 + j % k.tiles;
            zb = lo + k.z0 + j / k.tiles * k.len;
            ze = zb + k.len;
            if (k.len > before || k.len != range_length(s, b)) return 2;
            before = k.len;
        }
        if (tile < 0 || tile >= tiles || zb < lo || ze > lo + planes || zb >= ze) return 3;
        for (int z = zb; z < ze; z++) hits[(size_t)tile * planes + z - lo]++;
        if (zb == lo && ze - zb < first) first = ze - zb;
        if (ze == lo + planes && ze - zb < last) last = ze - zb;
    }
    for (int h : hits)
        if (h != 1) return 4;
    return s.first == first && s.last == last ? 0 : 5;
}

int main(int argc, char** argv) {
    if (argc == 2) {
        long long bad = 0, all = 0;
        for (int planes = 1; planes <= 34; planes++)
            for (int tiles = 1; tiles <= 23; tiles++)
                for (long long n = tiles; n <= (long long)tiles * planes; n++, all++)
                    bad += check(planes % 3 + 1, planes, 1 + tiles % 5, tiles, n) != 0;
        for (int planes : {61, 83, 104, 129, 256})
            for (int tiles : {1, 7, 18, 30, 98, 152, 455, 457})
                for (long long n : {(long long)tiles, 304LL, 456LL, 3LL * tiles, 500LL, (long long)tiles * planes})
                    if (n >= tiles && n <= (long long)tiles * planes) all++, bad += check(1, planes, 1, tiles, n) != 0;
        printf("%lld %lld\n", all, bad);
        return 0;
    }
    const int nx = atoi(argv[2]), ny = atoi(argv[3]), planes = atoi(argv[4]), sms = atoi(argv[5]);
    if (!strcmp(argv[1], "64")) {
        const int nbx = (nx + 15) / 16, tiles = nbx * ((ny + 7) / 8);
        const long long n = choose_blocks(planes + 2, true, 3, nbx, tiles, sms, 1, planes);
        const ZSplit s = make_split(1, planes, nbx, tiles, n);
        printf("%d %d %d\n", check(1, planes, nbx, tiles, n), s.ranges == 0, split_walls(planes + 2, s));
    } else {
        const Split32 s = split32(nx, ny, planes, sms);
        printf("%d %d %d\n", s.chunks >= 1 && s.chunks <= planes ? 0 : 1, s.ty, split32_walls(planes, s.chunks));
    }
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "split.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++20", "-I", str(REPO / "rast-3dmhd-cpp_gb300" / "csrc"), "-o", str(d / "split"),
                    str(d / "split.cpp")], check=True)

    def run(*args):
        out = subprocess.run([str(d / "split"), *map(str, args)], check=True, capture_output=True, text=True).stdout
        return [int(v) for v in out.split()]

    return run


def test_every_plane_of_every_tile_once(split):
    cases, bad = split("all")
    assert cases > 100_000 and bad == 0


def test_sizes_of_the_fp64_edge_tests_reach_both_kernels(split):
    """The last three were chosen for tiles of different numbers of z ranges; BCON
    runs inside the launch and outside it."""
    got = [split("64", *s, SMS) for s in SIZES64]
    assert all(ok == 0 for ok, _, _ in got)
    assert [mixed for _, mixed, _ in got] == [0] * (len(got) - 3) + [1] * 3
    assert {walls for _, _, walls in got} >= {0, 3}


def test_sizes_of_the_fp32_edge_tests_reach_both_tiles(split):
    """The last three were chosen for tiles of five rows."""
    got = [split("32", *s, SMS) for s in SIZES32]
    assert all(ok == 0 for ok, _, _ in got)
    assert [rows for _, rows, _ in got[-3:]] == [5] * 3 and 4 in [rows for _, rows, _ in got]
    assert {walls for _, _, walls in got} >= {0, 3}
