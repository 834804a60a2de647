// mhd_fused.cu -- launches of the fused FP64 RK3 substage for one instance
// (the per-tile work is in mhd_fused_tile.cuh) and of the wall kernel.
//
// The grid is (x tiles, y tiles, z chunks): splitting every column into z
// ranges spreads a small grid over the SMs and turns the tail wave of a large
// one into many short work units (choose_chunks).
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

// Whether the z ranges next to the walls hold the planes of BCON.
int fused_walls(const FusedArgs& a, int lo, int planes, int chunks) {
    int w = 0;
    if (lo == 1 && chunk_begin(planes, 1, chunks) >= kWallPlanes) w |= 1;
    if (lo + planes == a.g.nz - 1 && planes - chunk_begin(planes, chunks - 1, chunks) >= kWallPlanes) w |= 2;
    return w;
}

// Number of z ranges per column.  In units of the time the SM's one FP64 unit
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
int choose_chunks(const FusedArgs& a, long long tiles, int sms, int lo, int planes) {
    int best = 1;
    double best_cost = 1e300;
    const int need = (lo == 1 ? 1 : 0) | (lo + planes == a.g.nz - 1 ? 2 : 0);
    const long long wave = (long long)kMinBlocks * sms;
    // A slab of a host-to-host step runs beside the slabs of other substages,
    // which fill its last wave: where a plane has a wave of tiles, about two waves
    // of long ranges (256x256x128: 8.65 ms per step with 2 ranges, 9.24 with the 8
    // of the model below; 512x512x256: 57.3 ms with 1)
    if (planes < a.g.nz - 2 && tiles >= wave) return (int)std::max(1LL, std::min<long long>(planes, (2 * wave + tiles / 2) / tiles));
    for (int c = 1; c <= planes; c++) {
        const long long n = tiles * c;
        const double most = (planes + c - 1) / c, avg = (double)planes / c;
        double cost = n <= sms       ? 1.5 + 1.24 * most
                      : n <= 2 * sms ? 1.5 + 2.1 * most
                      : n <= wave    ? 1.5 + 2.95 * most
                                     : 1.0 + (double)((n + wave - 1) / wave) * (1.4 + 2.95 * avg);
        if (fused_walls(a, lo, planes, c) != need) cost += 0.6;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = c;
        }
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
int launch_t(const FusedArgs& a, int chunks, cudaStream_t st) {
    using T = DefaultTile;
    const size_t smem = ring_bytes<SW, T>();
    static const cudaError_t set =
        cudaFuncSetAttribute(k_substage<SW, UXY, ISO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (set != cudaSuccess) return (int)set;
    const int nbx = (a.g.nx - 2 + T::kTX - 1) / T::kTX, nby = (a.g.ny - 2 + T::kTY - 1) / T::kTY;
    return launch_overlapped(k_substage<SW, UXY, ISO>, dim3(nbx, nby, chunks), T::kThreads, smem, st, a);
}

template <class SW>
void launch_substage(const FusedArgs& a, int chunks, cudaStream_t st, int* rc) {
    // the instantiation with the optional temperature terms has no isotropic variant
    if (!kExtra && a.k.uniform_xy && a.k.isotropic_xy) *rc = launch_t<SW, true, !kExtra>(a, chunks, st);
    else *rc = a.k.uniform_xy ? launch_t<SW, true, false>(a, chunks, st) : launch_t<SW, false, false>(a, chunks, st);
}

template <class SW>
void launch_bcon_ghost(const FusedArgs& a, int wall0, int nwalls, cudaStream_t st, int* rc) {
    const int n = nwalls * (a.g.nx - 2) * (a.g.ny - 2);
    *rc = launch_overlapped(k_bcon_ghost<SW>, (n + 127) / 128, 128, 0, st, a.g, a.c, a.Uo, a.timt, wall0, nwalls);
}

}  // namespace

#if MHD_FUSED_XP
int fused_substage_xp(unsigned sw, const FusedArgs& a, int chunks, cudaStream_t st) {
    int rc = 0;
    MHD_DISPATCH_SW(sw, launch_substage, a, chunks, st, &rc);
    return rc;
}
#else
int fused_substage(unsigned sw, const FusedArgs& args, cudaStream_t st) {
    FusedArgs a = args;
    const int lo = a.zhi > 0 ? a.zlo : 1, planes = (a.zhi > 0 ? a.zhi : a.g.nz - 1) - lo;
    const long long tiles = (long long)((a.g.nx - 2 + DefaultTile::kTX - 1) / DefaultTile::kTX) *
                            ((a.g.ny - 2 + DefaultTile::kTY - 1) / DefaultTile::kTY);
    const int chunks = choose_chunks(a, tiles, sm_count(), lo, planes);
    a.walls = fused_walls(a, lo, planes, chunks);
    int rc = 0;
    if (a.c.pl_mode == 3 || a.c.lrem) rc = fused_substage_xp(sw, a, chunks, st);
    else MHD_DISPATCH_SW(sw, launch_substage, a, chunks, st, &rc);
    if (rc) return rc;
    // the walls that the substage left
    const bool first = lo == 1 && !(a.walls & 1), last = lo + planes == a.g.nz - 1 && !(a.walls & 2);
    if (first || last) MHD_DISPATCH_SW(sw, launch_bcon_ghost, a, first ? 0 : 1, (first ? 1 : 0) + (last ? 1 : 0), st, &rc);
    return rc;
}
#endif

}  // namespace mhd
