// mhd_common.cuh -- device-side definitions shared by the 3dmhd kernels.
//
// Layout of every field: double (or float) [nz][ny][nx], x fastest, one ghost
// cell per side, exactly the reference's `data` type (3dmhddata.h:8) on one
// global domain.  Strides: sy = nx, sz = nx*ny (elements).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "mhd_split.h"

namespace mhd {

// Compile-time physics switches, the reference's 3dmhdparam.h:8-17 and
// :86-107 macros as template parameters.  Horizontal boundaries are periodic
// only (fluxes() exits otherwise, 3dmhdsub.h:204-209); lPot is never read by
// the reference; lRem is out of scope.
template <bool MAG, bool ROT, bool SHR>
struct Switches {
    static constexpr bool lMag = MAG;
    static constexpr bool lRot = ROT;
    static constexpr bool lShr = SHR;
    static constexpr bool lPot = false;
    static constexpr bool lRem = false;
    static constexpr int ixCon = 0;
    static constexpr int iyCon = 0;
};

// field slots of the state (dump record order, 3dmhdio.h:23-33)
enum StateSlot { S_RU = 0, S_RV, S_RW, S_TT, S_RO, S_BX, S_BY, S_BZ };
// field slots of the right-hand sides
enum FluxSlot { F_FU = 0, F_FV, F_FW, F_FR, F_FT, F_WW1, F_WW2, F_WW3 };

struct Grid {
    int nx, ny, nz;  // full sizes, ghosts included
    int nPz;
    long long sy, sz;
};

// Scalars of set()/main() (3dmhd.cpp:144-145,354-369,401-459) and device
// pointers to the 1-D metric arrays (3dmhddata.h:21-23).
struct Consts {
    double C13, C23, C43;
    double hx, h2x, hy, h2y, hz, h2z;
    double GRAV, THETA, RE, REPR, ORE, OCV, CV, GAMMA, OMX, OMZ, RM, ORM, OBETA, TB, TP, SFF;
    double DDXmin;  // min of DDX over interior x (NaN skipped), for the CFL reduction
    int DDXsame, DDXpad_;  // every interior DDX equals DDXmin
    // Plume terms (3dmhdsub.h:443-459,750-778): pl_mode 0 none, 1 cooling spot
    // on the top wall with iTCon 0, 2 the same with iTCon 1, 3 internal heat
    // sink (iTCon 2).  plx/ply/plz are the host-computed Gaussian factors per
    // x, y, z; pl_tpr (top spot) and pl_s (sink amplitude) depend on TIMT and
    // are refreshed by the host before every step.
    int pl_mode, pl_pad_;
    const double *plx, *ply, *plz;
    double pl_hh, pl_tpr, pl_s;
    // lRem (3dmhdsub.h:229-238,297-313,783-802,852-854): per-substage arrays
    // filled before the right-hand side: lrem_ttm = horizontal mean of T per
    // z, lrem_hrad = HRAD, lrem_g = HRAD minus the z second derivative of the
    // mean (the fused kernels' form); TU, DZTU, DZTB for BCON
    int lrem, lrem_pad_;
    const double *lrem_ttm, *lrem_hrad, *lrem_g;
    double TU, DZTU, DZTB;
    int izCon, iTCon, iBCon, pad_;
    const double *dxxdx, *d2xxdx2, *DDX;
    const double *dyydy, *d2yydy2, *DDY;
    const double *dzzdz, *d2zzdz2, *DDZ;
    const double *RKAPA, *DKAPA;
};

// Programmatic dependent launch: a kernel launched with launch_overlapped may start
// while the one before it on its stream drains; it reaches the memory of earlier
// work only after wait_previous(), which returns when that work is complete and
// visible.  launch_next() lets the next such kernel start as soon as every block of
// this one has called it; without it (k_flux, and the kernels launched plainly before
// one of these) that happens when this one ends.  The substage, CFL and k_prep kernels
// call it last: called first, the next kernel's blocks crowd onto the SMs that are free
// then (a step at 64x64x32: 187 us without overlap, 253 so, 178 called last; 32x32x32
// 87, 99, 72; FP32 storage at 64x64x32 67, 84, 59).  The wall kernels, a few short
// blocks, call it after their own wait.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
int launch_overlapped(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchAttribute overlap = {};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &overlap;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) cudaGetLastError();  // returned, not left behind
    return (int)e;
}

struct Fields8 {
    double* p[8];
};

// Coefficients of the fused FP64 kernels.  The kernels for uniform x and y
// grids work in units of kappa = cx1 (the x metric factor duudu*hu, the same
// in every column): every equation is divided by it and the RK coefficients
// multiplied by it, except the temperature's with lShr, whose right-hand side
// is kept from call to call in true units.  `sT` below is the scale of the
// temperature equation, 1/kappa or (lShr) 1.  On other grids kappa = 1.
//
// One row per z (kZt rows follow one another, ZR_N doubles each):
enum ZRow {
    ZR_CZ = 0,    // cz1 / kappa (cz1 = dzzdz*hz)
    ZR_SZ0,       // z second-derivative factors of the planes above and below, b + a and b - a
                  // (a = d2zzdz2*hz, b = dzzdz^2*h2z), other grids b and a, scaled by ORE, ORE*C43, ORM,
                  // over kappa: 6 entries
    ZR_KZP = ZR_SZ0 + 6,  // conduction: the factors of T(z+1) and T(z-1), kapz (b +- a) +- dkapz cz1, with
    ZR_KZM,               // kapz, dkapz = OCV/REPR * (RKAPA, DKAPA), times sT; other grids: kapz and dkapz cz1
    ZR_KX, ZR_KY,         // kapz cx2b, kapz cy2b (cx2b = duudu^2*h2u), times sT
    ZR_SU, ZR_SV, ZR_SW,  // centre coefficients 2 (sx + sy + sz) of the Laplacians of u, v, w,
    ZR_ST, ZR_SB, ZR_SBW, // T (kapz and sT included) and B, and 2 (sx + sy) of B for the wall planes
    ZR_KQZ,               // C13*ORE*cz1
    ZR_OCZ,               // OBETA*cz1 / kappa
    ZR_TZP, ZR_TZM, ZR_STL,  // the unscaled Laplacian's b + a, b - a and centre coefficient (lRem); other grids b, a
    ZR_WD2, ZR_WD1,          // ORM a and ORM b over kappa: the one-sided d2B/dz2 on the walls
    ZR_N
};
// Scalars, read through shared memory (a constant-bank operand makes a DFMA
// slower); SC_ONE and SC_NZ are the 1 and -0 of the sums and products.
enum Scalar {
    SC_ONE = 0, SC_NZ,
    SC_KAPPA, SC_ST,
    SC_CY,                   // cy1 / kappa
    SC_SX0,                  // cx2b scaled by ORE, ORE*C43, ORM, over kappa: 3 entries
    SC_SY0 = SC_SX0 + 3,     // the same of y
    SC_KQX = SC_SY0 + 3, SC_KQY,  // C13*ORE*cx1, C13*ORE*cy1; other grids: C13*ORE
    SC_GRAV, SC_OMZ, SC_OMX,      // over kappa
    SC_HQ,                   // OCV*ORE*kappa^2*sT, viscous heating
    SC_MOCV,                 // -OCV*kappa*sT, pdV work
    SC_C43, SC_C43X3,        // C43 and 3*C43
    SC_OB,                   // OBETA
    SC_OHM,                  // ORM*OCV*kappa^2*sT/OBETA (0 for OBETA = 0), Ohmic heating of OBETA j
    SC_TX, SC_TY,            // cx2b, cy2b (lRem)
    SC_TMPC,                 // OCV/REPR*sT (lRem)
    SC_G, SC_Z, SC_GT, SC_ZT,  // filled by the kernel: gamma dt and zeta dt times kappa; of the temperature
    SC_N
};
struct Coefs {
    const double* zt[2];  // [nz][ZR_N]: any grid, uniform x / y
    const double* sc[2];  // [SC_N]
    // per column (any grid): first-derivative factors duudu*hu
    const double *cx1, *cy1;
    // per column (any grid): second-derivative coefficients c2b = duudu^2*h2u and
    // c2a = d2uudu2*hu, scaled by ORE, ORE*C43, ORM and unscaled
    const double *xt[8], *yt[8];
    // for the FP32 kernels: c2b and c2a as floats, scaled alike
    const float *xf[8], *yf[8];
    // uniform x and y grids: d2xxdx2 and d2yydy2 vanish and the x / y
    // coefficients are the same in every interior column
    int uniform_xy;
    // with uniform_xy: the same first-derivative coefficient on x and y (equal spacings)
    int isotropic_xy;
};

// ---- launchers implemented in the .cu files ----------------------------
// Parity path (compiled with -fmad=false, bit-exact with the reference).
int parity_fluxes(unsigned sw, const Grid& g, const Consts& c, Fields8 U, Fields8 F, double* P, double* UU,
                  double* VV, double* WW, cudaStream_t st);
// The same right-hand sides with 1/rho written to RI instead of RO (RO is
// only read); every scratch array is fully written before it is read.
int parity_fluxes_ext(unsigned sw, const Grid& g, const Consts& c, Fields8 U, Fields8 F, double* RI, double* P,
                      double* UU, double* VV, double* WW, cudaStream_t st);
int parity_rk(int kind, int nf, const Grid& g, Fields8 U, Fields8 Z, Fields8 F, double coef, cudaStream_t st);
int parity_bcon(unsigned sw, const Grid& g, const Consts& c, Fields8 U, double timt, cudaStream_t st);
int parity_communicate(int nf, const Grid& g, Fields8 U, cudaStream_t st);
// lRem: horizontal means of T per z (in the reference's summation order when
// `exact`, else by a parallel reduction), then HRAD and the fused form
// G = HRAD - d2(TTM)/dz2, into buf = [TTM | HRAD | G] (3 x nz doubles).
int lrem_profiles(const Grid& g, const Consts& c, const double* TT, double* buf, bool exact, cudaStream_t st);
// HRAD and G from the plane means already in buf[0, nz) (buf as lrem_profiles)
int lrem_hrad_from_means(const Grid& g, const Consts& c, double* buf, cudaStream_t st);
// CFL partial minima/maxima; out[0..4] = UMACH^2-candidate max, w0..w3 minima.
int parity_cfl(bool mag, const Grid& g, const Consts& c, Fields8 U, double* partials, int max_blocks,
               double* out5, cudaStream_t st);
// Conserved totals and max |div B|; out[0..3] = mass, energy, max divB, flags.
int diag_reduce(bool mag, const Grid& g, const Consts& c, Fields8 U, double* partials, int max_blocks, double* out4,
                cudaStream_t st);

// Measured FP64 FMA throughput of the current device (TFLOP/s, 2 flops per FMA).
int fp64_peak(double* tflops);

// Fused FP64 path.
struct FusedArgs {
    Grid g;
    Consts c;
    Coefs k;
    Fields8 U;     // state read (with ghosts)
    Fields8 Uo;    // state written (interior + x/y ghost images)
    Fields8 Z;     // RK register (read when substage > 0, written when substage < 2)
    long long fs;  // the fields of U, Uo and Z each follow one another at this distance (elements)
    double* FT;    // persistent temperature right-hand side (lShr only)
    double gdt;    // GAM_k * dt
    double zdt;    // ZETA_k * dt
    double timt;   // simulation time seen by BCON
    int substage;  // 0, 1, 2
    // device-resident time step (adaptive CFL without a host round trip):
    // when dtp is set, gdt = gam * dtp[0] and zdt = zet * dtp[0]
    const double* dtp;
    double gam, zet;
    // interior z planes [zlo, zhi) of a single-instance launch (zhi = 0: all)
    int zlo, zhi;
    // BCON of the wall cells by the thread that computed them (bit 0: plane 1,
    // bit 1: plane nz - 2): only where the z range next to that wall holds the
    // kWallPlanes planes that BCON involves
    int walls;
};
// Device time-step record of mhd_steps_cfl: [0] DT in use (0 once halted),
// [1] TIMT, [2] UMACH, [3] halt flag (DT < 1e-8), [4] the CFL DT computed
// last, [5] completed steps, [6] TIMI, [7] TIMC.
constexpr int kDtRecord = 8;
int cfl_dt_on_device(bool mag, const Grid& g, const Consts& c, Fields8 U, double* partials, int max_blocks,
                     double* rec, cudaStream_t st);
// One substage over planes [zlo, zhi) and BCON of the walls they touch (a.walls is set here).
int fused_substage(unsigned sw, const FusedArgs& a, cudaStream_t st);
// the instantiation with the optional temperature terms (fused_substage calls it)
int fused_substage_xp(unsigned sw, const FusedArgs& a, const ZSplit& s, int blocks, cudaStream_t st);
// Ragged batches: persistent CTAs take (instance, tile x, tile y) items from a
// counter that must be zero at launch.  Tile shapes: 0 = 32x4, 1 = 32x8, 2 = 16x8.
constexpr int kBatchTiles = 3;
void batch_tile_dims(int tile, int* tx, int* ty);
// Per-call control of a ragged batch (device pointers): left[i] = the steps
// instance i still takes in this call (its items are skipped at 0); err[0] =
// the first failed item check (0 = none), err[1..3] = that item (instance,
// tile x | tile y << 16, z range); n = the number of instances.
struct BatchCtl {
    int* left;
    int* err;
    int n;
};

// _uxy: uniform x/y grids (d2xxdx2 = d2yydy2 = 0); _gen: any grid.
// Item w = first z plane | (end plane << 16).
int fused_batch_substage_uxy(unsigned sw, int tile, const FusedArgs* args, const int4* items, int nitems, int* counter,
                             BatchCtl ctl, int grid, cudaStream_t st);
int fused_batch_substage_gen(unsigned sw, int tile, const FusedArgs* args, const int4* items, int nitems, int* counter,
                             BatchCtl ctl, int grid, cudaStream_t st);
int fused_batch_occupancy_uxy(unsigned sw, int tile, int* blocks_per_sm);
int fused_batch_occupancy_gen(unsigned sw, int tile, int* blocks_per_sm);
int fused_batch_bcon(unsigned sw, const FusedArgs* args, const int2* items, BatchCtl ctl, int nblocks,
                     cudaStream_t st);
// end of a batched step: left[i] -= 1 where positive
int batch_tick(int* left, int n, cudaStream_t st);

// FP32-storage path (fields stored in FP32, RO and TT as deviations from FP64
// reference profiles rho0(z), T0(z)).
struct Fields8f {
    float* p[8];
};
// the FP32 kernels' per-z coefficients, one row of ZF_N floats per z
enum ZFloat {
    ZF_CZ = 0, ZF_NCZ,   // +-cz1
    ZF_SZ0,              // b and a of the z second derivative, scaled by ORE, ORE*C43, ORM and unscaled: 8 entries
    ZF_KQZ = ZF_SZ0 + 8, // C13*ORE*cz1
    ZF_KAP, ZF_DKAP,     // OCV/REPR * (RKAPA, DKAPA)
    // from the profiles: their hydrostatic residual rho0 GRAV - D_z(rho0 T0), T0's first and second z
    // derivatives, and rho0, T0 as float pairs hi, lo
    ZF_HZ, ZF_DZT, ZF_D2T, ZF_RH, ZF_RL, ZF_TH, ZF_TL,
    ZF_N
};
struct Fused32Args {
    Grid g;
    Consts c;
    Coefs k;
    Fields8f U;    // state read (deviation form, with ghosts)
    Fields8f Uo;   // state written
    Fields8 Z;     // FP64 RK register (full values)
    double* FT;    // FP64 persistent temperature right-hand side (lShr only)
    const double *bgR, *bgT;     // reference profiles rho0(z), T0(z)
    const float* zf;             // [nz][ZF_N]
    double gdt, zdt;
    double timt;
    int substage;
    // device time-step record of mhd_steps_cfl (as FusedArgs)
    const double* dtp;
    double gam, zet;
    int walls;  // as FusedArgs
};
// Whether the arguments hold nf fields where the kernels look for them: the FP64
// substage addresses field f at p[0] + f * fs.
__host__ __device__ __forceinline__ bool fields_ok(const FusedArgs& a, int nf) {
    bool ok = a.fs >= a.g.sz * a.g.nz;
    auto placed = [&](const Fields8& q, int f) { return q.p[f] && q.p[f] == q.p[0] + f * a.fs; };
    for (int f = 0; f < nf; f++) ok = ok && placed(a.U, f) && placed(a.Uo, f) && placed(a.Z, f);
    return ok;
}
__host__ __device__ __forceinline__ bool fields_ok(const Fused32Args& a, int nf) {
    bool ok = true;
    for (int f = 0; f < nf; f++) ok = ok && a.U.p[f] && a.Uo.p[f] && a.Z.p[f];
    return ok;
}

// Check of a work item and of its instance's arguments before a kernel uses
// them: an item that fails records its code in ctl.err and is skipped, so a
// malformed work list shows up as an error status instead of a stray access.
// Codes: 0 valid, 1 instance index, 2 grid sizes, 3 tile position, 4 z range, 5 a
// field is missing or not where the kernel looks for it.
template <class A>
__host__ __device__ __forceinline__ int batch_item_code(int n, const A* args, int4 it, int tx, int ty, int nf) {
    if (it.x < 0 || it.x >= n) return 1;
    const A& a = args[it.x];
    const int zb = it.w & 0xffff, ze = it.w >> 16;
    if (a.g.nx < 3 || a.g.ny < 3 || a.g.nz < 6 || a.g.sy != a.g.nx || a.g.sz != (long long)a.g.nx * a.g.ny) return 2;
    if (it.y < 0 || it.z < 0 || 1 + it.y * tx > a.g.nx - 2 || 1 + it.z * ty > a.g.ny - 2) return 3;
    if (zb < 1 || ze > a.g.nz - 1 || zb >= ze) return 4;
    return fields_ok(a, nf) ? 0 : 5;
}
template <class A>
__device__ __forceinline__ bool batch_item_ok(const BatchCtl& ctl, const A* args, int4 it, int tx, int ty, int nf) {
    const int code = batch_item_code(ctl.n, args, it, tx, ty, nf);
    if (code && atomicCAS(ctl.err, 0, code) == 0) {
        ctl.err[1] = it.x;
        ctl.err[2] = it.y | (it.z << 16);
        ctl.err[3] = it.w;
    }
    return code == 0;
}

// One substage and BCON (a.walls is set here).
int fused32_substage(unsigned sw, const Fused32Args& a, cudaStream_t st);
int communicate32(int nf, const Grid& g, Fields8f U, cudaStream_t st);
// the z ghost planes of all eight fields of `from` into those of `to`
int zghosts32(const Grid& g, const float* from, float* to, cudaStream_t st);
// elements [first, first + n) of an FP32-storage state (fields one after another) as FP64 values in out
int widen32(const Grid& g, const float* U, const double* bgR, const double* bgT, long long first, int n, double* out,
            cudaStream_t st);
// lRem profiles (as lrem_profiles) of an FP32-storage temperature: the plane
// means T0(z) + mean(dT) summed in FP64
int lrem_profiles32(const Grid& g, const Consts& c, const float* dT, const double* bgT, double* buf, cudaStream_t st);
// ragged batches of FP32-storage instances (tile 32x4; same item and counter
// conventions as the FP64 batch)
constexpr int kBatch32TX = 32, kBatch32TY = 4;
int fused32_batch_substage(unsigned sw, const Fused32Args* args, const int4* items, int nitems, int* counter,
                           BatchCtl ctl, int grid, cudaStream_t st);
int fused32_batch_occupancy(unsigned sw, int* blocks_per_sm);
int fused32_batch_bcon(unsigned sw, const Fused32Args* args, const int2* items, BatchCtl ctl, int nblocks,
                       cudaStream_t st);
// CFL reduction of an FP32-storage state (the FP64 row kernel on the widened
// fields): out5 as parity_cfl, or the device time-step record as cfl_dt_on_device
int cfl32_rows(bool mag, const Grid& g, const Consts& c, Fields8f U, const double* bgR, const double* bgT,
               double* partials, int max_blocks, double* out5, cudaStream_t st);
int cfl32_dt_on_device(bool mag, const Grid& g, const Consts& c, Fields8f U, const double* bgR, const double* bgT,
                       double* partials, int max_blocks, double* rec, cudaStream_t st);
int diag32(bool mag, const Grid& g, const Consts& c, Fields8f U, const double* bgR, const double* bgT,
           double* partials, int max_blocks, double* out4, cudaStream_t st);

constexpr unsigned kSwRot = 0x1u, kSwMag = 0x2u, kSwShr = 0x10u;

}  // namespace mhd

// Dispatch a runtime switch word to Switches<MAG,ROT,SHR> template instances.
#define MHD_DISPATCH_SW(sw, FN, ...)                                                  \
    do {                                                                              \
        const bool m_ = ((sw) & ::mhd::kSwMag) != 0;                                  \
        const bool r_ = ((sw) & ::mhd::kSwRot) != 0;                                  \
        const bool s_ = ((sw) & ::mhd::kSwShr) != 0;                                  \
        if (m_ && r_ && s_) FN<::mhd::Switches<true, true, true>>(__VA_ARGS__);       \
        else if (m_ && r_) FN<::mhd::Switches<true, true, false>>(__VA_ARGS__);       \
        else if (m_ && s_) FN<::mhd::Switches<true, false, true>>(__VA_ARGS__);       \
        else if (m_) FN<::mhd::Switches<true, false, false>>(__VA_ARGS__);            \
        else if (r_ && s_) FN<::mhd::Switches<false, true, true>>(__VA_ARGS__);       \
        else if (r_) FN<::mhd::Switches<false, true, false>>(__VA_ARGS__);            \
        else if (s_) FN<::mhd::Switches<false, false, true>>(__VA_ARGS__);            \
        else FN<::mhd::Switches<false, false, false>>(__VA_ARGS__);                   \
    } while (0)
