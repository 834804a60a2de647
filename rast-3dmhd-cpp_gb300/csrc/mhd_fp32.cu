// mhd_fp32.cu -- launches of the FP32-storage substage (the per-tile work is in
// mhd_fp32_tile.cuh) for one instance and for ragged batches, of its wall
// kernel, and the FP32-storage ghost fill, lRem means and diagnostics.
#include "mhd_fp32_tile.cuh"

namespace mhd {
namespace {

using namespace fp32;

// CTAs per SM: four, with 128 registers a thread in tiles of 4 rows (16 warps) and
// 96 in tiles of 5 rows (20 warps).  Neither spills, but for 4 bytes in one kernel.
// Many small CTAs wait less at the barrier of a plane than few large ones.  With lMag,
// us per step at 200x150x100 and at 256x256x128, us per step of a batch of 24 instances
// (all before points beyond the grid were left out, which takes 8 % off the first and
// 5 % off the batches, and before the ring held the pressure deviation, 1 to 3 %):
//   two CTAs of 8 rows (128 registers)     680  1364  1983
//   two of 10 rows (96)                    670  1335  2019
//   four of 4 rows (128)                   651  1357  1867
//   four of 5 rows (96)                    617  1275  2018
//   five of 4 rows (96)                    687  1515  1980
// Batches therefore run tiles of 4 rows, one instance the better of the two by
// split32 (mhd_split.h).
constexpr int kResident = kResident32;
using BatchTile = Tile<kBatch32TY>;

// one instance: grid (tiles, x fastest; 1; z chunks)
template <class SW, class T, bool EXTRA>
__global__ void __launch_bounds__(T::kThreads, kResident) k_substage32(Fused32Args a) {
    extern __shared__ double smem32[];
    const int nPz = a.g.nz - 2;
    const int zb = 1 + (int)((long long)nPz * blockIdx.z / gridDim.z);
    const int ze = 1 + (int)((long long)nPz * (blockIdx.z + 1) / gridDim.z);
    const int nbx = (a.g.nx - 2 + kTX - 1) / kTX;
    substage32_tile<SW, T, EXTRA>(a, blockIdx.x % nbx, blockIdx.x / nbx, zb, ze, smem32);
    launch_next();
}

// ragged batch: persistent CTAs take (instance, tile x, tile y, z range) items
// (w = first plane | end plane << 16) from a counter that is zero at launch
template <class SW>
__global__ void __launch_bounds__(BatchTile::kThreads, kResident)
    k_substage32_batch(const Fused32Args* __restrict__ args, const int4* __restrict__ items, int nitems, int* counter,
                       BatchCtl ctl) {
    extern __shared__ double smem32[];
    constexpr int kArgWords = sizeof(Fused32Args) / sizeof(int);
    __shared__ __align__(16) int s_args[kArgWords];
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int t = s_item;
        __syncthreads();
        if (t >= nitems) break;
        const int4 it = items[t];
        // a malformed item, or an instance that has taken its steps (both uniform over the CTA)
        if (!batch_item_ok(ctl, args, it, kBatch32TX, kBatch32TY, SW::lMag ? 8 : 5) || ctl.left[it.x] <= 0) continue;
        // the instance's arguments in shared memory: every access to a field reads
        // its pointer there
        for (int k = threadIdx.x; k < kArgWords; k += BatchTile::kThreads)
            s_args[k] = reinterpret_cast<const int*>(args + it.x)[k];
        __syncthreads();
        substage32_tile<SW, BatchTile>(*reinterpret_cast<const Fused32Args*>(s_args), it.y, it.z, it.w & 0xffff,
                                       it.w >> 16, smem32);
        __syncthreads();
    }
}

template <class SW>
__global__ void k_bcon_ghost32(Fused32Args a, int wall0, int nwalls) {
    wait_previous();
    launch_next();
    const int nPx = a.g.nx - 2, nPy = a.g.ny - 2;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nwalls * nPx * nPy) return;
    const int r = t % (nPx * nPy);
    bcon32_cell<SW>(a.g, a.c, a.Uo, a.Z, a.bgR, a.bgT, a.timt, wall0 + t / (nPx * nPy), 1 + r % nPx, 1 + r / nPx);
}

// BCON for a ragged batch: block b covers 128 wall cells of instance items[b].x from cell items[b].y
template <class SW>
__global__ void k_bcon_ghost32_batch(const Fused32Args* __restrict__ args, const int2* __restrict__ items,
                                     BatchCtl ctl) {
    const int2 it = items[blockIdx.x];
    if (it.x < 0 || it.x >= ctl.n) {
        if (threadIdx.x == 0 && atomicCAS(ctl.err, 0, 1) == 0) ctl.err[1] = it.x;
        return;
    }
    if (ctl.left[it.x] <= 0) return;
    const Fused32Args& a = args[it.x];
    const int nPx = a.g.nx - 2, nPy = a.g.ny - 2;
    const int t = it.y + threadIdx.x;
    if (t >= 2 * nPx * nPy) return;
    const int r = t % (nPx * nPy);
    bcon32_cell<SW>(a.g, a.c, a.Uo, a.Z, a.bgR, a.bgT, a.timt, t / (nPx * nPy), 1 + r % nPx, 1 + r / nPx);
}

// periodic ghost fill of FP32 fields (communicate(), 3dmhdmpi.h:11-143)
__global__ void k_comm32(int nf, Grid g, Fields8f U) {
    const long long per_plane = 2LL * g.nx + 2LL * (g.ny - 2);
    const long long n = per_plane * g.nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const int z = (int)(t / per_plane);
        long long r = t % per_plane;
        int y, x;
        if (r < g.nx) {
            y = 0;
            x = (int)r;
        } else if (r < 2LL * g.nx) {
            y = g.ny - 1;
            x = (int)(r - g.nx);
        } else {
            r -= 2LL * g.nx;
            y = 1 + (int)(r / 2);
            x = (r % 2) ? g.nx - 1 : 0;
        }
        const int ys = (y == 0) ? g.ny - 2 : (y == g.ny - 1 ? 1 : y);
        const int xs = (x == 0) ? g.nx - 2 : (x == g.nx - 1 ? 1 : x);
        const long long d = z * g.sz + y * g.sy + x, s = z * g.sz + ys * g.sy + xs;
        for (int f = 0; f < nf; f++) U.p[f][d] = U.p[f][s];
    }
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

template <class SW, class T, bool EXTRA>
int launch32_t(const Fused32Args& a, dim3 grid, cudaStream_t st) {
    const size_t smem = smem_bytes<SW, T>();
    static const cudaError_t set =
        cudaFuncSetAttribute(k_substage32<SW, T, EXTRA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (set != cudaSuccess) return (int)set;
    return launch_overlapped(k_substage32<SW, T, EXTRA>, grid, T::kThreads, smem, st, a);
}

template <class SW>
void launch32(const Fused32Args& args, cudaStream_t st, int* rc) {
    Fused32Args a = args;
    const int planes = a.g.nz - 2;
    const Split32 s = split32(a.g.nx - 2, a.g.ny - 2, planes, sm_count());
    a.walls = split32_walls(planes, s.chunks);
    // (y tiles of few rows could exceed the y extent of a grid)
    const dim3 grid((a.g.nx - 2 + kTX - 1) / kTX * ((a.g.ny - 2 + s.ty - 1) / s.ty), 1, s.chunks);
    const bool extra = a.c.pl_mode == 3 || a.c.lrem;
    if (s.ty == 4) {
        *rc = extra ? launch32_t<SW, Tile<4>, true>(a, grid, st) : launch32_t<SW, Tile<4>, false>(a, grid, st);
    } else {
        *rc = extra ? launch32_t<SW, Tile<5>, true>(a, grid, st) : launch32_t<SW, Tile<5>, false>(a, grid, st);
    }
    if (*rc || a.walls == 3) return;
    // the walls that the substage left
    const int first = a.walls & 1 ? 1 : 0, n = a.walls ? 1 : 2;
    const int cells = n * (a.g.nx - 2) * (a.g.ny - 2);
    *rc = launch_overlapped(k_bcon_ghost32<SW>, (cells + 127) / 128, 128, 0, st, a, first, n);
}

template <class SW>
void batch32_launch(const Fused32Args* args, const int4* items, int nitems, int* counter, BatchCtl ctl, int grid,
                    cudaStream_t st, int* rc) {
    k_substage32_batch<SW><<<grid, BatchTile::kThreads, smem_bytes<SW, BatchTile>(), st>>>(args, items, nitems, counter, ctl);
    *rc = (int)cudaGetLastError();
}

template <class SW>
void batch32_occupancy(int* blocks, int* rc) {
    const size_t smem = smem_bytes<SW, BatchTile>();
    cudaFuncSetAttribute(k_substage32_batch<SW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    *rc = (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_substage32_batch<SW>, BatchTile::kThreads,
                                                             smem);
}

template <class SW>
void batch32_bcon(const Fused32Args* args, const int2* items, BatchCtl ctl, int nblocks, cudaStream_t st) {
    k_bcon_ghost32_batch<SW><<<nblocks, 128, 0, st>>>(args, items, ctl);
}

}  // namespace

int fused32_batch_substage(unsigned sw, const Fused32Args* args, const int4* items, int nitems, int* counter,
                           BatchCtl ctl, int grid, cudaStream_t st) {
    int rc = 0;
    MHD_DISPATCH_SW(sw, batch32_launch, args, items, nitems, counter, ctl, grid, st, &rc);
    return rc;
}

int fused32_batch_occupancy(unsigned sw, int* blocks_per_sm) {
    int rc = 0;
    MHD_DISPATCH_SW(sw, batch32_occupancy, blocks_per_sm, &rc);
    return rc;
}

int fused32_batch_bcon(unsigned sw, const Fused32Args* args, const int2* items, BatchCtl ctl, int nblocks,
                       cudaStream_t st) {
    MHD_DISPATCH_SW(sw, batch32_bcon, args, items, ctl, nblocks, st);
    return (int)cudaGetLastError();
}

int fused32_substage(unsigned sw, const Fused32Args& a, cudaStream_t st) {
    int rc = 0;
    MHD_DISPATCH_SW(sw, launch32, a, st, &rc);
    return rc;
}

namespace {

// plane means of T = T0(z) + dT over the interior (y, x), the deviations summed
// in FP64 by a block reduction per plane
__global__ void k_lrem_ttm32(Grid g, const float* dT, const double* bgT, double* ttm) {
    __shared__ double s[256];
    const int z = blockIdx.x;
    const int n = (g.nx - 2) * (g.ny - 2);
    double w = 0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int y = 1 + k / (g.nx - 2), x = 1 + k % (g.nx - 2);
        w += (double)dT[(long long)z * g.sz + (long long)y * g.sy + x];
    }
    s[threadIdx.x] = w;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) ttm[z] = bgT[z] + s[0] / (double)n;
}

}  // namespace

namespace {

// Elements [first, first + n) of the state, fields one after another, as FP64:
// the stored deviation plus its profile (rho0, T0; zero for the other fields).
__global__ void k_widen32(Grid g, const float* U, const double* bgR, const double* bgT, long long first, int n,
                          double* out) {
    const long long ncell = g.sz * g.nz;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const long long e = first + k;
        const int f = (int)(e / ncell);
        const int z = (int)((e - f * ncell) / g.sz);
        out[k] = widen_f32(U[e]) + (f == S_RO ? bgR[z] : f == S_TT ? bgT[z] : 0.0);
    }
}

// planes 0 and nz - 1 of eight fields
__global__ void k_zghosts32(Grid g, const float* from, float* to) {
    const long long n = 16 * g.sz, stride = (long long)gridDim.x * blockDim.x;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += stride) {
        const int k = (int)(t / g.sz);  // field and side
        const long long i = ((long long)(k >> 1) * g.nz + (k & 1 ? g.nz - 1 : 0)) * g.sz + t % g.sz;
        to[i] = from[i];
    }
}

}  // namespace

int widen32(const Grid& g, const float* U, const double* bgR, const double* bgT, long long first, int n, double* out,
            cudaStream_t st) {
    const int b = (n + 255) / 256;
    k_widen32<<<b < 152 * 16 ? b : 152 * 16, 256, 0, st>>>(g, U, bgR, bgT, first, n, out);
    return (int)cudaGetLastError();
}

int zghosts32(const Grid& g, const float* from, float* to, cudaStream_t st) {
    const long long b = (16 * g.sz + 255) / 256;
    k_zghosts32<<<(int)(b < 152 * 8 ? b : 152 * 8), 256, 0, st>>>(g, from, to);
    return (int)cudaGetLastError();
}

int lrem_profiles32(const Grid& g, const Consts& c, const float* dT, const double* bgT, double* buf, cudaStream_t st) {
    k_lrem_ttm32<<<g.nz, 256, 0, st>>>(g, dT, bgT, buf);
    const int e = (int)cudaGetLastError();
    return e ? e : lrem_hrad_from_means(g, c, buf, st);
}

int communicate32(int nf, const Grid& g, Fields8f U, cudaStream_t st) {
    const long long n = (2LL * g.nx + 2LL * (g.ny - 2)) * g.nz;
    long long b = (n + 255) / 256;
    if (b > 152 * 16) b = 152 * 16;
    k_comm32<<<(int)b, 256, 0, st>>>(nf, g, U);
    return (int)cudaGetLastError();
}

namespace {

constexpr int kRedThreads = 256;

__device__ __forceinline__ double rec(const Fields8f& U, const double* bg, int f, long long i, int z) {
    const double v = (double)U.p[f][i];
    return bg ? v + bg[z] : v;
}

// Mass, energy, max |div B| and flags in FP64 from the reconstructed state
// (same definitions as the FP64 diagnostics in mhd_diag.cu).
template <bool MAG>
__global__ void k_diag32(Grid g, Consts c, Fields8f U, const double* bgR, const double* bgT, double* part) {
    const int nPx = g.nx - 2, nPy = g.ny - 2, nPz = g.nz - 2;
    const long long ncell = (long long)nPx * nPy * nPz;
    double mass = 0, energy = 0, divb = 0;
    int flags = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < ncell;
         t += (long long)gridDim.x * blockDim.x) {
        const int x = 1 + (int)(t % nPx);
        const int y = 1 + (int)((t / nPx) % nPy);
        const int z = 1 + (int)(t / ((long long)nPx * nPy));
        const long long i = z * g.sz + y * g.sy + x;
        const double ro = rec(U, bgR, S_RO, i, z), tt = rec(U, bgT, S_TT, i, z);
        const double ru = U.p[S_RU][i], rv = U.p[S_RV][i], rw = U.p[S_RW][i];
        const double dv = c.DDX[x] * c.DDY[y] * c.DDZ[z];
        double e = 0.5 * (ru * ru + rv * rv + rw * rw) / ro + c.CV * ro * tt;
        if (!(ro > 0.0)) flags |= 2;
        if (!(tt > 0.0)) flags |= 4;
        if constexpr (MAG) {
            const double bx = U.p[S_BX][i], by = U.p[S_BY][i], bz = U.p[S_BZ][i];
            e += 0.5 * c.OBETA * (bx * bx + by * by + bz * bz);
            if (z > 1 && z < g.nz - 2) {
                const double d = ((double)U.p[S_BX][i + 1] - (double)U.p[S_BX][i - 1]) * c.dxxdx[x] * c.hx +
                                 ((double)U.p[S_BY][i + g.sy] - (double)U.p[S_BY][i - g.sy]) * c.dyydy[y] * c.hy +
                                 ((double)U.p[S_BZ][i + g.sz] - (double)U.p[S_BZ][i - g.sz]) * c.dzzdz[z] * c.hz;
                divb = fmax(divb, fabs(d));
            }
            if (!isfinite(bx) || !isfinite(by) || !isfinite(bz)) flags |= 1;
        }
        if (!isfinite(ro) || !isfinite(tt) || !isfinite(ru) || !isfinite(rv) || !isfinite(rw)) flags |= 1;
        mass += ro * dv;
        energy += e * dv;
    }
    __shared__ double s[4][kRedThreads];
    s[0][threadIdx.x] = mass;
    s[1][threadIdx.x] = energy;
    s[2][threadIdx.x] = divb;
    s[3][threadIdx.x] = (double)flags;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            s[0][threadIdx.x] += s[0][threadIdx.x + h];
            s[1][threadIdx.x] += s[1][threadIdx.x + h];
            s[2][threadIdx.x] = fmax(s[2][threadIdx.x], s[2][threadIdx.x + h]);
            s[3][threadIdx.x] = (double)((int)s[3][threadIdx.x] | (int)s[3][threadIdx.x + h]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; k++) part[(long long)k * gridDim.x + blockIdx.x] = s[k][0];
}

__global__ void k_diag32_finish(const double* part, int nb, double* out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double m = 0, e = 0, d = 0;
    int f = 0;
    for (int b = 0; b < nb; b++) {
        m += part[b];
        e += part[nb + b];
        d = fmax(d, part[2LL * nb + b]);
        f |= (int)part[3LL * nb + b];
    }
    out[0] = m;
    out[1] = e;
    out[2] = d;
    out[3] = (double)f;
}

int red_blocks(const Grid& g, int cap) {
    const long long ncell = (long long)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
    long long nb = (ncell + kRedThreads - 1) / kRedThreads;
    if (nb > cap) nb = cap;
    return nb < 1 ? 1 : (int)nb;
}

}  // namespace


int diag32(bool mag, const Grid& g, const Consts& c, Fields8f U, const double* bgR, const double* bgT,
           double* partials, int max_blocks, double* out4, cudaStream_t st) {
    const int nb = red_blocks(g, max_blocks);
    if (mag) k_diag32<true><<<nb, kRedThreads, 0, st>>>(g, c, U, bgR, bgT, partials);
    else k_diag32<false><<<nb, kRedThreads, 0, st>>>(g, c, U, bgR, bgT, partials);
    k_diag32_finish<<<1, 32, 0, st>>>(partials, nb, out4);
    return (int)cudaGetLastError();
}

}  // namespace mhd
