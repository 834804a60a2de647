// mhd_fp32_tile.cuh -- the fused RK3 substage with FP32 field storage for one
// tile of columns.
//
// Storage: every state field is an FP32 array.  RO and TT are stored as
// deviations from an FP64 reference profile rho0(z), T0(z) (the horizontal
// mean of the uploaded state), so the large hydrostatic part of rho and T
// never passes through FP32; the other six fields have a zero profile.
// Arithmetic:
//   FP32: every stencil of fluxes() (3dmhdsub.h:204-695), with the pressure as
//         its deviation dp = p - rho0 T0 (compensated, see point_values): the
//         large parts that cancel in hydrostatic balance enter as the
//         profiles' residual rho0 GRAV - D_z(rho0 T0), per z on the host;
//   FP64: the RK3 register Z (U' = Z + gamma dt F, Z' = U' + zeta dt F,
//         3dmhdsub.h:168-192), which also carries the state from one step to
//         the next (the last substage writes U' into it, BCON keeps its wall
//         values), so FP32 rounding enters only through the stencil inputs.
//
// What bounds it: HBM (448 + 128 bytes per cell and step) and the FP64 unit
// (about 20 instructions per cell and substage, 12 in the last), 0.24 ms each
// per substage at 256x256x128, if the instructions issued per cell and the
// latencies stay below that.  The march, the sums Q1, Q2, Q3 of 1-D differences
// (z neighbours are then read in the own column only) and the single barrier per
// plane are those of the FP64 kernel (mhd_fused_tile.cuh).  Field addresses are
// one multiply-add each (32-bit element indices on pointers in the constant
// bank), and the conversions between float and double run on the integer pipe
// in 3 and 11 instructions (mhd_convert.cuh): 1040 instructions per cell and
// substage with lMag, against 1470 for the version before it, which read the z
// neighbours' halos and had two barriers per plane.  Measured, with BCON inside:
// a step at 256x256x128 1630 -> 1262 us, at 64x64x32 98 -> 57 us, a batch of 24
// instances 2400 -> 1815 us (see the CTA sizes in mhd_fp32.cu).  Two cells per
// thread packed into f32x2 operations need 730 instructions per cell but 168
// registers, 12 warps per SM: 620 us per substage against 425; updating the fields
// of a plane in four groups, each where its right-hand sides are complete, was 2 %
// slower than all at the plane's end.
#pragma once

#include "mhd_common.cuh"
#include "mhd_convert.cuh"

#include <type_traits>

namespace mhd {
namespace fp32 {

// 32 columns per row: a warp's shared-memory accesses touch every bank once
constexpr int kTX = kTX32, kPX = kTX + 2;
template <int TY>
struct Tile {
    static constexpr int kTY = TY;
    static constexpr int kThreads = kTX * kTY;
    static constexpr int kPlane = kPX * (kTY + 2);
    static constexpr int kHalo = kPlane - kThreads;
    static_assert(kHalo <= kThreads, "one halo point per thread at most");
};

// quantities of a ring plane, with halo
enum QF { F_RU = 0, F_RV, F_DT, F_U, F_V, F_W, F_DP, F_BX, F_BY, F_BZ, F_NQ };
// quantities of the own column only
enum OF { G_RW = 0, G_N };
// scalars
enum SF { K_GRAV = 0, K_OMZ, K_NOMZ, K_OMX, K_NOMX, K_HQ, K_C43, K_OCV, K_OB, K_OHM, K_TMPC, K_C13ORE, K_N };

// gamma dt and zeta dt, and those of the temperature's equation
enum RF { R_G = 0, R_Z, R_GT, R_ZT, R_N };

constexpr int kZRing = 4;
// column coefficients of the second derivative, b and a, scaled by ORE, ORE*C43, ORM and unscaled
constexpr int kCoef = 8;

template <class SW>
constexpr int nqf() {
    return SW::lMag ? F_NQ : F_BX;
}
template <class SW>
constexpr int nraw() {
    return SW::lMag ? 8 : 5;
}
// floats: ring [3][nq][plane], Q1 and Q2 [2][2][plane], raw staging [nraw][plane], own columns [3][G_N][threads],
// coefficient rows, x and y second-derivative coefficients [kCoef][kTX], [kCoef][kTY], scalars; before them the RK
// coefficients (doubles)
template <class SW, class T>
constexpr size_t smem_bytes() {
    constexpr int kPlane = T::kPlane, kThreads = T::kThreads, kTY = T::kTY;
    return ((size_t)(3 * nqf<SW>() + 4 + nraw<SW>()) * kPlane + 3 * G_N * kThreads + kZRing * ZF_N +
            kCoef * (kTX + kTY) + K_N) * sizeof(float) + R_N * sizeof(double);
}

// the _rn forms are not contracted: what a sum or product rounds to does not
// depend on where it stands
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }

__device__ __forceinline__ void store32_with_images(float* F, const Grid& g, int z, int y, int x, float v) {
    const long long zo = (long long)z * g.sz;
    const int yb = (y == 1) ? g.ny - 1 : (y == g.ny - 2 ? 0 : -1);
    const int xb = (x == 1) ? g.nx - 1 : (x == g.nx - 2 ? 0 : -1);
    F[zo + (long long)y * g.sy + x] = v;
    if (xb >= 0) F[zo + (long long)y * g.sy + xb] = v;
    if (yb >= 0) {
        F[zo + (long long)yb * g.sy + x] = v;
        if (xb >= 0) F[zo + (long long)yb * g.sy + xb] = v;
    }
}

// BCON (3dmhdsub.h:720-873) on the FP32 wall planes, evaluated in FP64 from
// the reconstructed fields, plus the periodic ghost images.
template <class SW>
__device__ __forceinline__ void bcon32_cell(const Grid& g, const Consts& c, const Fields8f& U, const Fields8& Z,
                                            const double* bgR, const double* bgT, double timt, int wall, int x, int y) {
    const long long sz = g.sz;
    const int z = wall == 0 ? 1 : g.nz - 2;
    const int s = wall == 0 ? 1 : -1;
    const long long i = (long long)z * sz + (long long)y * g.sy + x;
    const long long i1 = i + s * sz, i2 = i + 2 * s * sz;
    const float *RU = U.p[S_RU], *RV = U.p[S_RV], *TT = U.p[S_TT], *RO = U.p[S_RO];
    const double ro = bgR[z] + (double)RO[i];
    const double ro1 = bgR[z + s] + (double)RO[i1], ro2 = bgR[z + 2 * s] + (double)RO[i2];
    const double t1 = bgT[z + s] + (double)TT[i1], t2 = bgT[z + 2 * s] + (double)TT[i2];
    double ru, rv, tt;
    if constexpr (SW::lShr) {
        ru = 0.0;
        rv = (wall == 0 ? 1.0 : -1.0) * cos(0.0 * timt) * ro;
    } else {
        ru = ro * (c.C43 * (double)RU[i1] / ro1 - c.C13 * (double)RU[i2] / ro2);
        rv = ro * (c.C43 * (double)RV[i1] / ro1 - c.C13 * (double)RV[i2] / ro2);
    }
    if (wall == 0) {
        if (c.pl_mode == 1) {
            // cooling spot on the top wall (3dmhdsub.h:750-766)
            tt = 1.0f - (1.0f - c.pl_tpr) * c.plx[x] / c.pl_hh * c.ply[y] / c.pl_hh;
        } else if (c.pl_mode == 2) {
            const double DZ = 1.0f / (double)(g.nPz - 1) / c.dzzdz[z];
            tt = c.C43 * t1 - c.C13 * t2 -
                 c.C23 * DZ * (c.THETA - (c.THETA - c.pl_tpr) * c.plx[x] / c.pl_hh * c.ply[y] / c.pl_hh);
        } else if (c.iTCon == 1) {
            const double DZ = 1.0f / (float)(g.nPz - 1) / c.dzzdz[z];
            tt = c.lrem ? c.C43 * t1 - c.C13 * t2 + c.DZTU : c.C43 * t1 - c.C13 * t2 - c.C23 * DZ * c.THETA;
        } else if (c.lrem) {
            tt = c.TU;
        } else {
            tt = 1.0;
            if (c.iTCon == 4 && x < g.nx / 2) tt = 1.0f - c.TP;
        }
    } else {
        if (c.izCon == 0) {
            tt = c.TB;
        } else if (c.lrem) {
            tt = c.C43 * t1 - c.C13 * t2 + c.DZTB;
        } else {
            const double DZ = 1.0f / (float)(g.nPz - 1) / c.dzzdz[z];
            tt = c.C43 * t1 - c.C13 * t2 - c.C23 * DZ * c.THETA / c.RKAPA[z];
        }
    }
    store32_with_images(U.p[S_RU], g, z, y, x, (float)ru);
    store32_with_images(U.p[S_RV], g, z, y, x, (float)rv);
    store32_with_images(U.p[S_RW], g, z, y, x, 0.0f);
    store32_with_images(U.p[S_TT], g, z, y, x, (float)(tt - bgT[z]));
    // the FP64 register holds the state between steps: keep its wall values in step
    Z.p[S_RU][i] = ru;
    Z.p[S_RV][i] = rv;
    Z.p[S_RW][i] = 0.0;
    Z.p[S_TT][i] = tt;
    if constexpr (SW::lMag) {
        if (c.iBCon == 0) {
            store32_with_images(U.p[S_BZ], g, z, y, x, 0.0f);
            Z.p[S_BZ][i] = 0.0;
        }
    }
}

// 1/x: one Newton-Raphson step from the hardware estimate, which is good to one
// unit in the last place: the error stays within 2^-24 + 2^-43 of the value (a
// rounded quotient's is 2^-24).  Where x or the estimate is no normal number (|x|
// below 2^-126 or above 2^126, infinity, NaN) the residual is 1 or no number: there
// the estimate that knows subnormal numbers, alone (a division spills registers).
__device__ __forceinline__ float recip32(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float e = fmaf(-x, r, 1.0f);
    r = fmaf(r, e, r);
    if (!(fabsf(e) < 0.5f)) asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The derived quantities of a point: 1/rho, the velocities, and the
// equation of state as the deviation dp = rho0 dT + drho T0 + drho dT of p from
// the plane's rho0 T0.  rho0 and T0 come as float pairs hi + lo (about 48
// significant bits); error-free transformations give rho = rh + drho as s + e
// (two-sum), plus rl, and recover every product's rounding error by fma, so dp
// keeps about one float rounding where its terms cancel (near pressure
// balance; measured against 80-bit sums: <= 0.6 ulp up to a 1e6 cancellation
// ratio).
struct Point {
    float ri, u, v, w, dp;
};
__device__ __forceinline__ Point point_values(const float* row, float ru, float rv, float rw, float dt,
                                               float dro) {
    const float rh = row[ZF_RH], rl = row[ZF_RL], th = row[ZF_TH], tl = row[ZF_TL];
    auto two_sum = [](float a, float b, float& e) {
        const float s = add(a, b), bb = sub(s, a);
        e = add(sub(a, sub(s, bb)), sub(b, bb));
        return s;
    };
    Point p;
    float se;
    const float s = two_sum(rh, dro, se);
    p.ri = recip32(add(s, add(se, rl)));
    const float p1 = mul(rh, dt), e1 = fmaf(rh, dt, -p1);
    const float p2 = mul(th, dro), e2 = fmaf(th, dro, -p2);
    const float p3 = mul(dro, dt), e3 = fmaf(dro, dt, -p3);
    float qe, qe2;
    const float q = two_sum(p1, p2, qe);
    const float q2 = two_sum(q, p3, qe2);
    const float tail = add(add(add(qe, qe2), add(e1, e2)), add(e3, fmaf(rl, dt, mul(tl, dro))));
    p.dp = add(q2, tail);
    p.u = mul(ru, p.ri);
    p.v = mul(rv, p.ri);
    p.w = mul(rw, p.ri);
    return p;
}

// One tile (bx, by) of one instance, interior z planes [zb, ze).  EXTRA: the
// instantiation with the iTCon 2 plume heat sink and lRem.  `smem` begins with
// the RK coefficients, so the kernels declare it as doubles (8-byte aligned).
template <class SW, class T, bool EXTRA = false>
__device__ __forceinline__ void substage32_tile(const Fused32Args& a, int bx, int by, int zb, int ze, double* smem) {
    constexpr int kTY = T::kTY, kThreads = T::kThreads, kPlane = T::kPlane;
    constexpr int NQ = nqf<SW>(), NRAW = nraw<SW>();
    constexpr int kOwn = NQ * kPlane;
    constexpr int kSlot = NQ * kPlane + G_N * kThreads;  // a plane's arrays, then its own-column ones
    const Grid& g = a.g;
    const Consts& c = a.c;
    double* rk = smem;                         // [R_N]
    float* ring = reinterpret_cast<float*>(smem + R_N);
    float* qbuf = ring + 3 * kSlot;            // [parity][Q1, Q2][plane]
    float* stage = qbuf + 4 * kPlane;          // [nraw][plane]
    float* zrow = stage + NRAW * kPlane;       // [kZRing][ZF_N]
    float* xtab = zrow + kZRing * ZF_N;        // [kCoef][kTX]
    float* ytab = xtab + kCoef * kTX;          // [kCoef][kTY]
    float* sc = ytab + kCoef * kTY;            // [K_N]
    const int tid = threadIdx.x;
    const int x0 = 1 + bx * kTX, y0 = 1 + by * kTY;
    const int tx = tid % kTX, ty = tid / kTX;
    const int x = x0 + tx, y = y0 + ty;
    const bool active = x <= g.nx - 2 && y <= g.ny - 2;
    const int zl = 1, zr = g.nz - 1;

    // this thread's points of a plane, as in the FP64 kernel: its own column and
    // one halo point of the rows, then the columns, then the corners
    const int pc = (ty + 1) * kPX + (tx + 1);
    int hk = 0, hkind = -1;  // 0: row halo (needs Q2), 1: column halo (Q1), 2: corner
    if (tid < 2 * kTX) {
        hk = (tid < kTX ? 0 : (kTY + 1) * kPX) + 1 + tid % kTX;
        hkind = 0;
    } else if (tid < 2 * kTX + 2 * kTY) {
        const int r = tid - 2 * kTX;
        hk = (1 + r % kTY) * kPX + (r < kTY ? 0 : kPX - 1);
        hkind = 1;
    } else if (tid < T::kHalo) {
        const int r = tid - 2 * kTX - 2 * kTY;
        hk = ((r & 2) ? (kTY + 1) * kPX : 0) + ((r & 1) ? kPX - 1 : 0);
        hkind = 2;
    }
    const int hx = x0 - 1 + hk % kPX, hy = y0 - 1 + hk / kPX;
    // Points beyond the grid, which no active cell uses, are not read: those of the
    // halo are left out and the columns filled with zeros (reading the last column in
    // their stead, lanes with one address, made a step at 33x300x61 306 us instead of 197)
    const bool own_in = x < g.nx && y < g.ny;
    if (hx >= g.nx || hy >= g.ny) hkind = -1;
    // element indices of the points in plane 0 (a field has fewer than 2^31 elements)
    const int sz = (int)g.sz;
    const int oc = own_in ? y * (int)g.sy + x : 0, ohc = hy * (int)g.sy + hx;
    const int own_bytes = own_in ? 4 : 0;

    // Copy the raw fields of this thread's points of plane z into an [nraw][plane]
    // area (cp.async of 4 bytes: the rows of an unpadded FP32 field are not
    // 16-byte aligned, which rules out TMA and wider copies).  Every thread copies
    // the points it later derives itself, so its own wait is the only one needed.
    auto copy_plane = [&](float* to, int z) {
        const int i = z * sz + oc;
#pragma unroll
        for (int f = 0; f < NRAW; f++) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(to + f * kPlane + pc);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(a.U.p[f] + i), "r"(own_bytes) : "memory");
        }
        if (hkind >= 0) {
            const int j = z * sz + ohc;
#pragma unroll
            for (int f = 0; f < NRAW; f++) {
                const unsigned dst = (unsigned)__cvta_generic_to_shared(to + f * kPlane + hk);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(a.U.p[f] + j) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the tile's rows of a plane of the register and FT into L2: 32 doubles lie in
    // two or three 128-byte lines, the last of which the next tile's rows share
    const bool fetch = (tx & 15) == 0 && own_in;
    auto prefetch = [&](int z) {
        if (fetch && z < g.nz - 1) {
#pragma unroll
            for (int f = 0; f < NRAW; f++) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.Z.p[f] + (z * sz + oc)));
            if constexpr (SW::lShr) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.FT + (z * sz + oc)));
        }
    };
    auto put_row = [&](int z) {
        if (tid < ZF_N) zrow[(z & (kZRing - 1)) * ZF_N + tid] = a.zf[(size_t)z * ZF_N + tid];
    };
    auto row = [&](int z) { return zrow + (z & (kZRing - 1)) * ZF_N; };

    float *Pm = ring + (size_t)((zb - 1) % 3) * kSlot, *P0 = ring + (size_t)(zb % 3) * kSlot,
          *Pp = ring + (size_t)((zb + 1) % 3) * kSlot;
    // coefficients: rows zb - 1 .. zb + 2, columns, scalars (no kernel writes them)
    for (int z = zb - 1; z <= zb + 2 && z <= ze; z++) put_row(z);
    for (int k = tid; k < kCoef * kTX; k += kThreads) xtab[k] = a.k.xf[k / kTX][min(x0 + k % kTX, g.nx - 1)];
    for (int k = tid; k < kCoef * kTY; k += kThreads) ytab[k] = a.k.yf[k / kTY][min(y0 + k % kTY, g.ny - 1)];
    if (tid < K_N) {
        double v = 0.0;
        switch (tid) {
            case K_GRAV: v = c.GRAV; break;
            case K_OMZ: v = c.OMZ; break;
            case K_NOMZ: v = -c.OMZ; break;
            case K_OMX: v = c.OMX; break;
            case K_NOMX: v = -c.OMX; break;
            case K_HQ: v = c.OCV * c.ORE; break;
            case K_C43: v = c.C43; break;
            case K_OCV: v = c.OCV; break;
            case K_OB: v = c.OBETA; break;
            case K_OHM: v = c.OBETA * c.ORM * c.OCV; break;
            case K_TMPC: v = c.OCV / c.REPR; break;
            case K_C13ORE: v = c.C13 * c.ORE; break;
        }
        sc[tid] = (float)v;
    }
    // the first three planes, each into its own slot, where it is derived
    wait_previous();
    copy_plane(Pm, zb - 1);
    copy_plane(P0, zb);
    copy_plane(Pp, zb + 1);
    const int ym = g.ny - 1;
    const float cx = (float)a.k.cx1[min(x, g.nx - 1)], cy = (float)a.k.cy1[min(y, ym)];
    const float ncx = -cx, ncy = -cy;
    // RK coefficients: from the host, or from the device time-step record; a
    // halted record (dt below 1e-8) turns the substage into a copy of the state
    // (scaled by 2^896, see below, but for the temperature's with lShr)
    if (tid == 0) {
        const double gdt = a.dtp ? a.gam * a.dtp[0] : a.gdt, zdt = a.dtp ? a.zet * a.dtp[0] : a.zdt;
        rk[R_G] = gdt * 0x1p896;
        rk[R_Z] = zdt * 0x1p896;
        rk[R_GT] = SW::lShr ? gdt : gdt * 0x1p896;
        rk[R_ZT] = SW::lShr ? zdt : zdt * 0x1p896;
    }
    const bool halted = a.dtp && a.dtp[3] != 0.0;
    __syncthreads();

    float dro0, ri0, dro1, ri1;  // drho, 1/rho of planes z, z + 1
    // ring quantities of a copied point (the copy may lie in P itself: all of it is
    // read first); returns w, and leaves RW and dp + RW w of the own column too
    auto put_point = [&](const float* zr_, const float* from, int k, float* P, bool own, float& dro, float& ri) {
        float r[NRAW];
#pragma unroll
        for (int f = 0; f < NRAW; f++) r[f] = from[f * kPlane + k];
        const Point p = point_values(zr_, r[S_RU], r[S_RV], r[S_RW], r[S_TT], r[S_RO]);
        P[F_RU * kPlane + k] = r[S_RU];
        P[F_RV * kPlane + k] = r[S_RV];
        P[F_DT * kPlane + k] = r[S_TT];
        P[F_U * kPlane + k] = p.u;
        P[F_V * kPlane + k] = p.v;
        P[F_W * kPlane + k] = p.w;
        P[F_DP * kPlane + k] = p.dp;
        if (own) P[kOwn + G_RW * kThreads + tid] = r[S_RW];
        if constexpr (SW::lMag) {
            P[F_BX * kPlane + k] = r[S_BX];
            P[F_BY * kPlane + k] = r[S_BY];
            P[F_BZ * kPlane + k] = r[S_BZ];
        }
        dro = r[S_RO];
        ri = p.ri;
        return p.w;
    };
    float ux, vy, wz;                      // the own column's D_x u, D_y v, D_z w of plane z
    float q3m, q3c, q3p;                   // Q3 of planes z - 1, z, z + 1
    auto own_q3 = [&](const float* P, float& du, float& dv) {
        du = mul(cx, sub(P[F_U * kPlane + pc + 1], P[F_U * kPlane + pc - 1]));
        dv = mul(cy, sub(P[F_V * kPlane + pc + kPX], P[F_V * kPlane + pc - kPX]));
        return add(du, dv);
    };
    // the halo point's metric factor
    const float hc = hkind == 0 ? (float)a.k.cx1[min(hx, g.nx - 1)] : (float)a.k.cy1[min(hy, ym)];
    auto put_q = [&](const float* P, int z, float du, float dv, float wp, float wm, float hwp, float hwm) {
        float* q1 = qbuf + (z & 1) * 2 * kPlane;
        float* q2 = q1 + kPlane;
        const float cz = row(z)[ZF_CZ];
        ux = du;
        vy = dv;
        wz = mul(cz, sub(wp, wm));
        q1[pc] = add(dv, wz);
        q2[pc] = add(du, wz);
        if (hkind == 0)
            q2[hk] = fmaf(cz, sub(hwp, hwm), mul(hc, sub(P[F_U * kPlane + hk + 1], P[F_U * kPlane + hk - 1])));
        else if (hkind == 1)
            q1[hk] = fmaf(cz, sub(hwp, hwm), mul(hc, sub(P[F_V * kPlane + hk + kPX], P[F_V * kPlane + hk - kPX])));
    };

    {
        asm volatile("cp.async.wait_all;" ::: "memory");
        float wm, wp, hwm = 0.0f, hwp = 0.0f, t0, t1;
        wm = put_point(row(zb - 1), Pm, pc, Pm, true, t0, t1);
        put_point(row(zb), P0, pc, P0, true, dro0, ri0);
        wp = put_point(row(zb + 1), Pp, pc, Pp, true, dro1, ri1);
        if (hkind >= 0) {
            hwm = put_point(row(zb - 1), Pm, hk, Pm, false, t0, t1);
            put_point(row(zb), P0, hk, P0, false, t0, t1);
            hwp = put_point(row(zb + 1), Pp, hk, Pp, false, t0, t1);
        }
        __syncthreads();
        if (zb + 2 <= ze) copy_plane(stage, zb + 2);
        float du, dv;
        q3m = own_q3(Pm, du, dv);
        q3c = own_q3(P0, du, dv);
        put_q(P0, zb, du, dv, wp, wm, hwp, hwm);
    }
    for (int z = zb; z < ze; z++) {
        __syncthreads();
        if (z + 1 < ze) prefetch(z + 1);
        if (z + 3 <= ze) put_row(z + 3);
        float ux1, vy1;
        q3p = own_q3(Pp, ux1, vy1);
        if (active) {
            const float* R = row(z);
            // the register: its loads (L2 hits, prefetched) are under way meanwhile; without
            // lMag and with the optional terms from after the momentum terms on (before them
            // the 5-row tile spills, without lMag a step at 256x256x128 1101 us instead of 894)
            const int i = z * sz + oc;
            double zf[NRAW];
            auto load_register = [&] {
#pragma unroll
                for (int f = 0; f < NRAW; f++) zf[f] = a.Z.p[f][i];
            };
            if constexpr (SW::lMag && !EXTRA) load_register();
            const double t0z = a.bgT[z], r0z = a.bgR[z];
            // (constant offsets from one pointer per plane)
            const float *c0 = P0 + pc, *cp = Pp + pc, *cm = Pm + pc;
            const float *w0 = P0 + kOwn + tid, *wp_ = Pp + kOwn + tid, *wm_ = Pm + kOwn + tid;
            auto C0 = [&](int q) { return c0[q * kPlane]; };
            auto XP = [&](int q) { return c0[q * kPlane + 1]; };
            auto XM = [&](int q) { return c0[q * kPlane - 1]; };
            auto YP = [&](int q) { return c0[q * kPlane + kPX]; };
            auto YM = [&](int q) { return c0[q * kPlane - kPX]; };
            auto ZP = [&](int q) { return cp[q * kPlane]; };
            auto ZM = [&](int q) { return cm[q * kPlane]; };
            const float *xt = xtab + tx, *yt = ytab + ty;
            // acc + b_k (p + m - 2 c), the second derivative without its a_k (p - m) part,
            // along x, y and z (with that part), for the scale k
            auto lapx = [&](int q, int k, float acc) {
                return fmaf(xt[2 * k * kTX], fmaf(-2.0f, C0(q), add(XP(q), XM(q))), acc);
            };
            auto lapy = [&](int q, int k, float acc) {
                return fmaf(yt[2 * k * kTY], fmaf(-2.0f, C0(q), add(YP(q), YM(q))), acc);
            };
            auto lapz = [&](int q, int k, float dz, float acc) {
                acc = fmaf(R[ZF_SZ0 + 2 * k], fmaf(-2.0f, C0(q), add(ZP(q), ZM(q))), acc);
                return fmaf(R[ZF_SZ0 + 2 * k + 1], dz, acc);
            };
            // ... and the a_k (p - m) parts of x and y on stretched grids
            auto skew = [&](int q, int kx, int ky, float acc) {
                acc = fmaf(xt[(2 * kx + 1) * kTX], sub(XP(q), XM(q)), acc);
                return fmaf(yt[(2 * ky + 1) * kTY], sub(YP(q), YM(q)), acc);
            };
            const bool stretched = !a.k.uniform_xy;
            const float cz = R[ZF_CZ], ncz = R[ZF_NCZ];
            const bool wall = (z == zl || z == zr - 1);
            const int wz2 = z == zl ? 2 : -2;  // planes to the one-sided stencils' second point
            // a field of the second (third) point behind a wall
            auto far = [&](int f, int dz) {
                return a.U.p[f][(z + dz) * sz + oc];
            };
            const float rwp = wp_[G_RW * kThreads], rwm = wm_[G_RW * kThreads];
            const float u = C0(F_U), v = C0(F_V), w = C0(F_W), dt0 = C0(F_DT);

            // ---- continuity (3dmhdsub.h:204-227), one-sided dRW/dz on the walls
            const float rup = XP(F_RU), rum = XM(F_RU), rvp = YP(F_RV), rvm = YM(F_RV);
            float nrwz = sub(rwm, rwp);
            if (wall) {
                const float q = far(S_RW, wz2);
                nrwz = z == zl ? fmaf(-4.0f, rwp, q) : sub(mul(4.0f, rwm), q);
            }
            const float fr = fmaf(cz, nrwz, fmaf(cy, sub(rvm, rvp), mul(cx, sub(rum, rup))));

            // ---- momentum: pressure deviation and gravity (3dmhdsub.h:266-272),
            // advection (3dmhdsub.h:279-289), viscous Laplacians (3dmhdsub.h:462-472)
            const float up = XP(F_U), um = XM(F_U), vp = YP(F_V), vm = YM(F_V), wp = ZP(F_W), wm = ZM(F_W);
            const float dUz = sub(ZP(F_U), ZM(F_U)), dVz = sub(ZP(F_V), ZM(F_V)), dWz = sub(wp, wm);
            float fu = mul(cx, sub(XM(F_DP), XP(F_DP)));
            float fv = mul(cy, sub(YM(F_DP), YP(F_DP)));
            float fw = fmaf(dro0, sc[K_GRAV], fmaf(cz, sub(ZM(F_DP), ZP(F_DP)), R[ZF_HZ]));
            // (each momentum flux by itself: added to dp at the points first, it would carry
            // dp's rounding; a difference rounds one of its two products)
            fu = fmaf(ncx, fmaf(rup, up, -mul(rum, um)), fu);
            fv = fmaf(ncy, fmaf(rvp, vp, -mul(rvm, vm)), fv);
            fw = fmaf(ncz, fmaf(rwp, wp, -mul(rwm, wm)), fw);
            fu = fmaf(ncy, fmaf(rvp, YP(F_U), -mul(rvm, YM(F_U))), fu);
            fu = fmaf(ncz, fmaf(rwp, ZP(F_U), -mul(rwm, ZM(F_U))), fu);
            fv = fmaf(ncx, fmaf(rup, XP(F_V), -mul(rum, XM(F_V))), fv);
            fv = fmaf(ncz, fmaf(rwp, ZP(F_V), -mul(rwm, ZM(F_V))), fv);
            fw = fmaf(ncx, fmaf(rup, XP(F_W), -mul(rum, XM(F_W))), fw);
            fw = fmaf(ncy, fmaf(rvp, YP(F_W), -mul(rvm, YM(F_W))), fw);
            fu = lapx(F_U, 1, lapy(F_U, 0, lapz(F_U, 0, dUz, fu)));
            fv = lapx(F_V, 0, lapy(F_V, 1, lapz(F_V, 0, dVz, fv)));
            fw = lapx(F_W, 0, lapy(F_W, 0, lapz(F_W, 1, dWz, fw)));
            if (stretched) {
                fu = skew(F_U, 1, 0, fu);
                fv = skew(F_V, 0, 1, fv);
                fw = skew(F_W, 0, 0, fw);
            }

            // ---- viscous cross terms (3dmhdsub.h:486-487,517-518,531-532)
            {
                const float* q1 = qbuf + (z & 1) * 2 * kPlane + pc;
                const float* q2 = q1 + kPlane;
                const float k13 = sc[K_C13ORE];
                fu = fmaf(mul(k13, cx), sub(q1[1], q1[-1]), fu);
                fv = fmaf(mul(k13, cy), sub(q2[kPX], q2[-kPX]), fv);
                fw = fmaf(R[ZF_KQZ], sub(q3p, q3m), fw);
            }

            if constexpr (!SW::lMag || EXTRA) load_register();
            // ---- temperature (deviation stencils plus the profile's derivatives):
            // nadv collects what is subtracted, qr the terms proportional to 1/rho
            const float dTz = sub(ZP(F_DT), ZM(F_DT)), Tz = fmaf(cz, dTz, R[ZF_DZT]);
            float nadv = 0.0f;
            if constexpr (!SW::lShr) {
                nadv = mul(u, mul(cx, sub(XP(F_DT), XM(F_DT))));
                nadv = fmaf(v, mul(cy, sub(YP(F_DT), YM(F_DT))), nadv);
                nadv = fmaf(w, Tz, nadv);
            }
            float lapT = lapx(F_DT, 3, lapy(F_DT, 3, lapz(F_DT, 3, dTz, R[ZF_D2T])));
            if (stretched) lapT = skew(F_DT, 3, 3, lapT);
            float qr;
            if (EXTRA && c.lrem && !SW::lShr) {
                // lRem (3dmhdsub.h:297-313): conduction of T - TTM(z) plus HRAD, as
                // lap T + G(z) with G = HRAD - d2 TTM/dz2 from the FP64 plane means
                qr = mul(sc[K_TMPC], add(lapT, (float)c.lrem_g[z]));
            } else {
                qr = fmaf(R[ZF_KAP], lapT, mul(R[ZF_DKAP], Tz));
            }
            // internal plume heat sink (iTCon 2, 3dmhdsub.h:443-459)
            if constexpr (EXTRA) {
                if (c.pl_mode == 3) {
                    qr = add(qr, (float)(-c.pl_s * (c.plx[x] * c.ply[y] * c.plz[z])));
                }
            }

            // velocity gradients (heating and induction)
            float uy, vx, wx, wy, uz, vz;
            if constexpr (!SW::lShr || SW::lMag) {
                vx = mul(cx, sub(XP(F_V), XM(F_V)));
                wx = mul(cx, sub(XP(F_W), XM(F_W)));
                uy = mul(cy, sub(YP(F_U), YM(F_U)));
                wy = mul(cy, sub(YP(F_W), YM(F_W)));
                uz = mul(cz, dUz);
                vz = mul(cz, dVz);
            }
            // ---- viscous heating and pdV work (3dmhdsub.h:477-538, not with lShr)
            if constexpr (!SW::lShr) {
                const float div = add(q3c, wz);
                const float s1 = add(uy, vx), s2 = add(uz, wx), s3 = add(vz, wy);
                float dg = mul(ux, ux);
                dg = fmaf(vy, vy, dg);
                dg = fmaf(wz, wz, dg);
                dg = sub(dg, fmaf(wz, q3c, mul(ux, vy)));
                const float sh = fmaf(s1, s1, fmaf(s2, s2, mul(s3, s3)));
                qr = fmaf(sc[K_HQ], fmaf(sc[K_C43], dg, sh), qr);
                nadv = fmaf(mul(sc[K_OCV], add(R[ZF_TH], dt0)), div, nadv);  // float(T0) + dT
            }
            // ---- Coriolis (3dmhdsub.h:540-545)
            if constexpr (SW::lRot) {
                const float rv = C0(F_RV);
                fu = fmaf(sc[K_OMZ], rv, fu);
                fv = fmaf(sc[K_NOMZ], C0(F_RU), fv);
                fv = fmaf(sc[K_OMX], w0[G_RW * kThreads], fv);
                fw = fmaf(sc[K_NOMX], rv, fw);
            }

            // ---- induction, Lorentz force, Ohmic heating (3dmhdsub.h:547-695)
            float w1, w2, w3;
            if constexpr (SW::lMag) {
                const float bx = C0(F_BX), by = C0(F_BY), bz = C0(F_BZ);
                // stretching; one-sided dw/dz on the walls (3dmhdsub.h:572-584)
                float wzm = wz;
                if (wall) {
                    const float rq = far(S_RW, wz2), dq = far(S_RO, wz2);
                    const float q = rq / (float)(a.bgR[z + wz2] + (double)dq);
                    wzm = z == zl ? mul(cz, sub(mul(4.0f, ZP(F_W)), q)) : mul(cz, fmaf(-4.0f, ZM(F_W), q));
                }
                const float nbx = -bx, nby = -by, nbz = -bz;
                w1 = fmaf(by, uy, fmaf(bz, uz, mul(nbx, add(vy, wzm))));
                w2 = fmaf(bx, vx, fmaf(bz, vz, mul(nby, add(ux, wzm))));
                w3 = fmaf(bx, wx, fmaf(by, wy, mul(nbz, q3c)));
                // advection
                const float dBYx = sub(XP(F_BY), XM(F_BY)), dBZx = sub(XP(F_BZ), XM(F_BZ));
                const float dBXy = sub(YP(F_BX), YM(F_BX)), dBZy = sub(YP(F_BZ), YM(F_BZ));
                const float dBXz = sub(ZP(F_BX), ZM(F_BX)), dBYz = sub(ZP(F_BY), ZM(F_BY));
                const float dBZz = sub(ZP(F_BZ), ZM(F_BZ));
                const float ncxu = mul(ncx, u), ncyv = mul(ncy, v), nczw = mul(ncz, w);
                w1 = fmaf(ncxu, sub(XP(F_BX), XM(F_BX)), fmaf(ncyv, dBXy, fmaf(nczw, dBXz, w1)));
                w2 = fmaf(ncxu, dBYx, fmaf(ncyv, sub(YP(F_BY), YM(F_BY)), fmaf(nczw, dBYz, w2)));
                w3 = fmaf(ncxu, dBZx, fmaf(ncyv, dBZy, fmaf(nczw, dBZz, w3)));
                // resistive Laplacians
                w1 = lapx(F_BX, 2, lapy(F_BX, 2, w1));
                w2 = lapx(F_BY, 2, lapy(F_BY, 2, w2));
                w3 = lapx(F_BZ, 2, lapy(F_BZ, 2, lapz(F_BZ, 2, dBZz, w3)));
                if (stretched) {
                    w1 = skew(F_BX, 2, 2, w1);
                    w2 = skew(F_BY, 2, 2, w2);
                    w3 = skew(F_BZ, 2, 2, w3);
                }
                if (!wall) {
                    w1 = lapz(F_BX, 2, dBXz, w1);
                    w2 = lapz(F_BY, 2, dBYz, w2);
                } else {
                    // d2B/dz2 with the one-sided wall stencils (3dmhdsub.h:640-654,673-687)
                    const int s = (z == zl) ? 1 : -1;
                    const float d2 = mul((float)s, R[ZF_SZ0 + 5]), d1 = R[ZF_SZ0 + 4];
                    auto one_sided = [&](float b0, float b1, float b2, float b3) {
                        const float first = sub(fmaf(4.0f, b1, mul(-3.0f, b0)), b2);
                        const float second = sub(fmaf(4.0f, b2, fmaf(-5.0f, b1, mul(2.0f, b0))), b3);
                        return fmaf(first, d2, mul(second, d1));
                    };
                    w1 = add(w1, one_sided(bx, s > 0 ? ZP(F_BX) : ZM(F_BX), far(S_BX, 2 * s), far(S_BX, 3 * s)));
                    w2 = add(w2, one_sided(by, s > 0 ? ZP(F_BY) : ZM(F_BY), far(S_BY, 2 * s), far(S_BY, 3 * s)));
                }
                const float jz = fmaf(cx, dBYx, mul(ncy, dBXy));
                const float jy = fmaf(cz, dBXz, mul(ncx, dBZx));
                const float jx = fmaf(cy, dBZy, mul(ncz, dBYz));
                const float ob = sc[K_OB];
                fu = fmaf(ob, fmaf(bz, jy, mul(nby, jz)), fu);
                fv = fmaf(ob, fmaf(bx, jz, mul(nbz, jx)), fv);
                fw = fmaf(ob, fmaf(by, jx, mul(nbx, jy)), fw);
                qr = fmaf(sc[K_OHM], fmaf(jx, jx, fmaf(jy, jy, mul(jz, jz))), qr);
            }
            const float ft = sub(mul(ri0, qr), nadv);

            // ---- FP64 RK3 register (3dmhdsub.h:168-192).  Z carries the full FP64
            // state across steps (written by substage 3 and by BCON), so substage 1
            // starts from it instead of from the FP32 copy: step_block_ZETA0 without
            // the FP32 rounding.  The last substage (and a halted record) stores U'
            // itself into Z.  widen_scaled gives F 2^-896 exactly; 2^896 sits in gdt
            // and zdt.  Infinite or not-a-number right-hand sides show up in F * 0.
            const float fl[8] = {fu, fv, fw, ft, fr, w1, w2, w3};
            float bad = 0.0f;
#pragma unroll
            for (int f = 0; f < NRAW; f++) bad = fmaf(fl[f], 0.0f, bad);
            double ftd = 0.0;  // with lShr the temperature's right-hand side is the FP64 FT
            if constexpr (SW::lShr) {
                ftd = widen_f32(ft) + a.FT[i];
                if (!halted) a.FT[i] = ftd;
            }
            // periodic images of a boundary cell
            const int ix = (x == 1) ? g.nx - 2 : (x == g.nx - 2 ? 2 - g.nx : 0);
            const int iy = (y == 1) ? (g.ny - 2) * (int)g.sy : (y == g.ny - 2 ? (2 - g.ny) * (int)g.sy : 0);
            auto update = [&](auto next_register, auto any) {
                float uf[NRAW];
                double un[NRAW];
                bool ordinary = true;
#pragma unroll
                for (int f = 0; f < NRAW; f++) {
                    double fd;
                    if (SW::lShr && f == S_TT) fd = ftd;
                    else fd = any ? widen_f32(fl[f]) * 0x1p-896 : widen_scaled(fl[f]);
                    un[f] = (any && halted) ? zf[f] : fma(rk[f == S_TT ? R_GT : R_G], fd, zf[f]);
                    a.Z.p[f][i] = next_register ? fma(rk[f == S_TT ? R_ZT : R_Z], fd, un[f]) : un[f];
                    if (f == S_TT) un[f] -= t0z;
                    if (f == S_RO) un[f] -= r0z;
                    ordinary = ordinary && narrow_ordinary(un[f]);
                    uf[f] = narrow_fast(un[f]);
                }
                if (!ordinary) {
#pragma unroll
                    for (int f = 0; f < NRAW; f++) uf[f] = narrow_f64(un[f]);
                }
#pragma unroll
                for (int f = 0; f < NRAW; f++) a.Uo.p[f][i] = uf[f];
                if (ix | iy) {
#pragma unroll
                    for (int f = 0; f < NRAW; f++) {
                        float* u1 = a.Uo.p[f] + i;
                        if (ix) u1[ix] = uf[f];
                        if (iy) u1[iy] = uf[f];
                        if (ix && iy) u1[ix + iy] = uf[f];
                    }
                }
            };
            // (the split keeps the last substage's unused register update off the
            // FP64 pipe; the general form serves a halted record and non-finite F)
            if (halted || bad != 0.0f) {
                if (a.substage < 2 && !halted) update(std::true_type{}, std::true_type{});
                else update(std::false_type{}, std::true_type{});
            } else if (a.substage < 2) {
                update(std::true_type{}, std::false_type{});
            } else {
                update(std::false_type{}, std::false_type{});
            }
        }
        if (z + 1 < ze) {
            // plane z + 2 into the slot of plane z - 1, of which every thread reads
            // its own points only; then Q1 and Q2 of plane z + 1
            asm volatile("cp.async.wait_all;" ::: "memory");
            const float* zr2 = row(z + 2);
            float dro2, ri2, w2, hw2 = 0.0f, t0, t1;
            w2 = put_point(zr2, stage, pc, Pm, true, dro2, ri2);
            if (hkind >= 0) hw2 = put_point(zr2, stage, hk, Pm, false, t0, t1);
            if (z + 3 <= ze) copy_plane(stage, z + 3);
            put_q(Pp, z + 1, ux1, vy1, w2, P0[F_W * kPlane + pc], hw2, P0[F_W * kPlane + hk]);
            q3m = q3c;
            q3c = q3p;
            dro0 = dro1;
            ri0 = ri1;
            dro1 = dro2;
            ri1 = ri2;
            float* tp = Pm;
            Pm = P0;
            P0 = Pp;
            Pp = tp;
        }
    }
    // BCON, as in the FP64 kernel
    if (active) {
        if ((a.walls & 1) && zb == 1) bcon32_cell<SW>(g, c, a.Uo, a.Z, a.bgR, a.bgT, a.timt, 0, x, y);
        if ((a.walls & 2) && ze == g.nz - 1) bcon32_cell<SW>(g, c, a.Uo, a.Z, a.bgR, a.bgT, a.timt, 1, x, y);
    }
}

}  // namespace fp32
}  // namespace mhd
