// mhd_fused.cu -- launches of the fused FP64 RK3 substage for one instance
// (the per-tile work is in mhd_fused_tile.cuh) and of the wall kernel.
//
// Splitting every column into z ranges spreads a small grid over the SMs and turns
// the tail wave of a large one into many short work units (choose_blocks).
#include "mhd_fused_tile.cuh"

#include <algorithm>

namespace mhd {
namespace {

using namespace fused;
// tile of the single-instance kernel (MHD_FUSED_TILE_X x MHD_FUSED_TILE_Y threads):
// 16 x 8 loads 18 x 10 ring points per 128 cells (32 x 4: 34 x 6), and each
// warp still reads whole 128-byte rows (measured: 71.7 vs 72.9 ms per step at
// 512 x 512 x 256; 32 x 6, 32 x 8 and 16 x 12 run fewer CTAs per SM and are slower)
#ifndef MHD_FUSED_TILE_X
#define MHD_FUSED_TILE_X 16
#endif
#ifndef MHD_FUSED_TILE_Y
#define MHD_FUSED_TILE_Y 8
#endif
// This file is compiled twice: MHD_FUSED_XP=0 gives the kernels without the
// optional temperature terms (and the dispatcher and the wall kernels),
// MHD_FUSED_XP=1 the ones with the iTCon 2 heat sink and lRem.
#ifndef MHD_FUSED_XP
#define MHD_FUSED_XP 0
#endif
constexpr bool kExtra = MHD_FUSED_XP != 0;
using DefaultTile = Tile<MHD_FUSED_TILE_X, MHD_FUSED_TILE_Y>;
constexpr int kMinBlocks = DefaultTile::kThreads >= 256 ? 2 : 3;

// grid (x tiles, y tiles, z ranges)
template <class SW, bool UXY, bool ISO>
__global__ void __launch_bounds__(DefaultTile::kThreads, kMinBlocks) k_substage(FusedArgs a) {
    extern __shared__ double ring[];
    const int lo = a.zhi > 0 ? a.zlo : 1;
    const int nz = (a.zhi > 0 ? a.zhi : a.g.nz - 1) - lo;
    const int zb = lo + (int)((long long)nz * blockIdx.z / gridDim.z);
    const int ze = lo + (int)((long long)nz * (blockIdx.z + 1) / gridDim.z);
    substage_tile<SW, DefaultTile, UXY, kExtra, ISO>(a, blockIdx.x, blockIdx.y, zb, ze, ring);
    launch_next();
}

// tiles of different numbers of z ranges
template <class SW, bool UXY, bool ISO>
__global__ void __launch_bounds__(DefaultTile::kThreads, kMinBlocks) k_substage_mixed(FusedArgs a, ZSplit s) {
    extern __shared__ double ring[];
    int j = blockIdx.x;
    ZSplit::Class k = s.cls[0];
#pragma unroll
    for (int c = 1; c < 4; c++) {
        if (j < k.blocks) continue;
        j -= k.blocks;
        k = s.cls[c];
    }
    const int t = __shfl_sync(0xffffffffu, k.tile0 + j % k.tiles, 0);
    const int zb = __shfl_sync(0xffffffffu, s.lo + k.z0 + j / k.tiles * k.len, 0);
    substage_tile<SW, DefaultTile, UXY, kExtra, ISO>(a, t % s.nbx, t / s.nbx, zb, zb + __shfl_sync(0xffffffffu, k.len, 0), ring);
    launch_next();
}

template <class SW>
__global__ void k_bcon_ghost(Grid g, Consts c, Fields8 U, double timt, int wall0, int nwalls) {
    wait_previous();
    launch_next();
    const int nPx = g.nx - 2, nPy = g.ny - 2;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nwalls * nPx * nPy) return;
    const int r = t % (nPx * nPy);
    bcon_cell<SW>(g, c, U, timt, wall0 + t / (nPx * nPy), 1 + r % nPx, 1 + r / nPx);
}

// First plane of z range k of n over `planes` planes (the kernel's split).
int chunk_begin(int planes, int k, int n) { return (int)((long long)planes * k / n); }

// Split of `planes` planes from lo on, of `tiles` tiles in rows of nbx, into n blocks:
// where n is no multiple of the tiles, the first n % tiles of them have one range
// more than the others, a tile's longer ranges come first, and the blocks are numbered
// by falling length.
ZSplit make_split(int lo, int planes, int nbx, int tiles, long long n) {
    ZSplit s = {};
    s.lo = lo;
    s.planes = planes;
    s.nbx = nbx;
    s.tiles = tiles;
    const int r = (int)(n / tiles), more = (int)(n % tiles);
    if (more == 0) {
        s.ranges = r;
        s.first = chunk_begin(planes, 1, r);
        s.last = planes - chunk_begin(planes, r - 1, r);
        return s;
    }
    s.first = (planes + r) / (r + 1);
    s.last = planes / (r + 1);
    auto set = [&](int c, int tile0, int count, int ranges, bool longer) {
        const int q = planes / ranges, m = planes % ranges;
        s.cls[c] = {count * (longer ? m : ranges - m), tile0, count, longer ? 0 : m * (q + 1), longer ? q + 1 : q};
    };
    set(0, more, tiles - more, r, true);
    set(1, 0, more, r + 1, true);
    set(2, more, tiles - more, r, false);
    set(3, 0, more, r + 1, false);
    if (s.cls[1].len < s.cls[2].len) std::swap(s.cls[1], s.cls[2]);
    return s;
}

// Length of block `block` of a split into unequal numbers of ranges.
int range_length(const ZSplit& s, long long block) {
    int c = 0;
    while (c < 3 && block >= s.cls[c].blocks) block -= s.cls[c++].blocks;
    return s.cls[c].len;
}

// Whether the z ranges next to the walls hold the planes of BCON.
int fused_walls(const FusedArgs& a, const ZSplit& s) {
    return (s.lo == 1 && s.first >= kWallPlanes ? 1 : 0) |
           (s.lo + s.planes == a.g.nz - 1 && s.last >= kWallPlanes ? 2 : 0);
}

// Number of blocks, (tile, z range) each.  In units of the time the SM's one FP64 unit
// takes for a plane of a tile (6.2 us with lMag), a launch of n CTAs with P
// planes each lasts, measured at 16^3 .. 300x256x40 for 1 .. 64 ranges:
//   n <= 152 (one per SM)          1.5 + 1.24 P   one CTA alone does not keep the unit busy
//   n <= 304                       1.5 + 2.1 P
//   n <= 456 (all resident)        1.5 + 2.95 P
//   more                           1.0 + ceil(n / 456) (1.4 + 2.95 P)
// with the constants for the planes around a range and its start-up; the last
// wave counts in full because its CTAs are not spread evenly over the SMs.  A
// range too short for BCON at the walls adds a launch (0.6).  The choice is within
// 2 % of the fastest on those 19 grids.  Against at most eight ranges of four
// planes, us per step, launches not overlapped: 32x32x32 138 -> 87 (32 ranges of
// one plane), 97x45x61 (no field) 344 -> 272, 128x128x64 1146 -> 1094 (BCON inside
// the launch included).
long long choose_blocks(const FusedArgs& a, int nbx, long long tiles, int sms, int lo, int planes) {
    long long best = tiles;
    double best_cost = 1e300;
    const int need = (lo == 1 ? 1 : 0) | (lo + planes == a.g.nz - 1 ? 2 : 0);
    const long long wave = (long long)kMinBlocks * sms;
    // A slab of a host-to-host step runs beside the slabs of other substages,
    // which fill its last wave: where a plane has a wave of tiles, about two waves
    // of long ranges (256x256x128: 8.65 ms per step with 2 ranges, 9.24 with the 8
    // of the model below; 512x512x256: 57.3 ms with 1)
    if (planes < a.g.nz - 2 && tiles >= wave)
        return tiles * std::max(1LL, std::min<long long>(planes, (2 * wave + tiles / 2) / tiles));
    for (int c = 1; c <= planes; c++) {
        const long long n = tiles * c;
        const double most = (planes + c - 1) / c, avg = (double)planes / c;
        double cost = n <= sms       ? 1.5 + 1.24 * most
                      : n <= 2 * sms ? 1.5 + 2.1 * most
                      : n <= wave    ? 1.5 + 2.95 * most
                                     : 1.0 + (double)((n + wave - 1) / wave) * (1.4 + 2.95 * avg);
        if (fused_walls(a, make_split(lo, planes, nbx, (int)tiles, n)) != need) cost += 0.6;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = n;
        }
    }
    // ... or one wave that fills every SM, with tiles of c and of c + 1 ranges: an SM's
    // blocks (i, i + 152 and i + 304) are then of different lengths, the longest first.
    // us per step without and with: 97x45x61 (no field) 263, 246; 72^3 488, 434;
    // 33x65x129 486, 449; 80x64x48 300, 288; 96x96x64 618, 608; but where the ranges get
    // too short for BCON at the walls 64x64x32 178, 181 and 128x64x16 188, 211.
    // Two blocks per SM that way are not spread evenly (64x64x32 200).  Not built for
    // the optional temperature terms.
    if (kMinBlocks == 3 && a.c.pl_mode != 3 && !a.c.lrem && wave >= tiles && wave <= tiles * planes && wave % tiles != 0) {
        const ZSplit s = make_split(lo, planes, nbx, (int)tiles, wave);
        const int l1 = range_length(s, 0), l2 = range_length(s, sms), l3 = range_length(s, 2LL * sms);
        double cost = 1.7 + 2.95 * l3 + 2.1 * (l2 - l3) + 1.24 * (l1 - l2);
        if (fused_walls(a, s) != need) cost += 1.3;
        if (1.02 * cost < best_cost) best = wave;
    }
    return best;
}

int sm_count() {
    static const int n = [] {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return sms > 0 ? sms : 1;
    }();
    return n;
}

template <class SW, bool UXY, bool ISO>
int launch_t(const FusedArgs& a, const ZSplit& s, int blocks, cudaStream_t st) {
    using T = DefaultTile;
    const size_t smem = ring_bytes<SW, T>();
    if (kExtra || s.ranges) {
        static const cudaError_t set =
            cudaFuncSetAttribute(k_substage<SW, UXY, ISO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (set != cudaSuccess) return (int)set;
        return launch_overlapped(k_substage<SW, UXY, ISO>, dim3(s.nbx, s.tiles / s.nbx, s.ranges), T::kThreads, smem, st, a);
    }
    if constexpr (!kExtra) {
        static const cudaError_t set =
            cudaFuncSetAttribute(k_substage_mixed<SW, UXY, ISO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (set != cudaSuccess) return (int)set;
        return launch_overlapped(k_substage_mixed<SW, UXY, ISO>, dim3(blocks), T::kThreads, smem, st, a, s);
    }
    return (int)cudaErrorInvalidValue;
}

template <class SW>
void launch_substage(const FusedArgs& a, const ZSplit& s, int blocks, cudaStream_t st, int* rc) {
    // the instantiation with the optional temperature terms has no isotropic variant
    if (!kExtra && a.k.uniform_xy && a.k.isotropic_xy) *rc = launch_t<SW, true, !kExtra>(a, s, blocks, st);
    else *rc = a.k.uniform_xy ? launch_t<SW, true, false>(a, s, blocks, st) : launch_t<SW, false, false>(a, s, blocks, st);
}

template <class SW>
void launch_bcon_ghost(const FusedArgs& a, int wall0, int nwalls, cudaStream_t st, int* rc) {
    const int n = nwalls * (a.g.nx - 2) * (a.g.ny - 2);
    *rc = launch_overlapped(k_bcon_ghost<SW>, (n + 127) / 128, 128, 0, st, a.g, a.c, a.Uo, a.timt, wall0, nwalls);
}

}  // namespace

#if MHD_FUSED_XP
int fused_substage_xp(unsigned sw, const FusedArgs& a, const ZSplit& s, int blocks, cudaStream_t st) {
    int rc = 0;
    MHD_DISPATCH_SW(sw, launch_substage, a, s, blocks, st, &rc);
    return rc;
}
#else
int fused_substage(unsigned sw, const FusedArgs& args, cudaStream_t st) {
    FusedArgs a = args;
    const int lo = a.zhi > 0 ? a.zlo : 1, planes = (a.zhi > 0 ? a.zhi : a.g.nz - 1) - lo;
    const int nbx = (a.g.nx - 2 + DefaultTile::kTX - 1) / DefaultTile::kTX;
    const long long tiles = (long long)nbx * ((a.g.ny - 2 + DefaultTile::kTY - 1) / DefaultTile::kTY);
    const long long n = choose_blocks(a, nbx, tiles, sm_count(), lo, planes);
    const ZSplit s = make_split(lo, planes, nbx, (int)tiles, n);
    a.walls = fused_walls(a, s);
    int rc = 0;
    if (a.c.pl_mode == 3 || a.c.lrem) rc = fused_substage_xp(sw, a, s, (int)n, st);
    else MHD_DISPATCH_SW(sw, launch_substage, a, s, (int)n, st, &rc);
    if (rc) return rc;
    // the walls that the substage left
    const bool first = lo == 1 && !(a.walls & 1), last = lo + planes == a.g.nz - 1 && !(a.walls & 2);
    if (first || last) MHD_DISPATCH_SW(sw, launch_bcon_ghost, a, first ? 0 : 1, (first ? 1 : 0) + (last ? 1 : 0), st, &rc);
    return rc;
}
#endif

}  // namespace mhd
