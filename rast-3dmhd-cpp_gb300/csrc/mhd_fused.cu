// mhd_fused.cu -- launches of the fused FP64 RK3 substage for one instance
// (the per-tile work is in mhd_fused_tile.cuh) and of the wall kernel.
//
// Splitting every column into z ranges spreads a small grid over the SMs and turns
// the tail wave of a large one into many short work units (choose_blocks in mhd_split.h).
#include "mhd_fused_tile.cuh"

namespace mhd {
namespace {

using namespace fused;
// tile of the single-instance kernel (MHD_FUSED_TILE_X x MHD_FUSED_TILE_Y threads):
// 16 x 8 loads 18 x 10 ring points per 128 cells (32 x 4: 34 x 6), and each warp still
// reads whole 128-byte rows.  ms per step at 512 x 512 x 256, with lMag, lRot and lShr
// and with lMag alone: 16 x 8 53.9 and 59.1; 8 x 16 55.4, 60.1; 32 x 4 56.5, 62.0; with
// more threads and so fewer CTAs per SM 32 x 6 61.5, 69.1; 16 x 12 62.3, 70.9; 32 x 8
// 65.9, 71.4.
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
// three CTAs per SM: 168 registers, of which some kernels spill 4 to 56 bytes
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
    const ZSplit::Class k = block_class(s, j);
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
    const long long n = choose_blocks(a.g.nz, a.c.pl_mode != 3 && !a.c.lrem, kMinBlocks, nbx, tiles, sm_count(), lo, planes);
    const ZSplit s = make_split(lo, planes, nbx, (int)tiles, n);
    a.walls = split_walls(a.g.nz, s);
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
