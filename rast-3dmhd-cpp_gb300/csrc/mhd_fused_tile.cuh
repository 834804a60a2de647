// mhd_fused_tile.cuh -- the fused FP64 RK3 substage for one tile of columns.
//
// A CTA owns a TX x TY tile of (x, y) columns and marches down a range of z
// planes.  Three z planes of the tile plus a one-cell halo live in a
// shared-memory ring; a plane's raw fields arrive by cp.async one plane ahead
// and its derived quantities (1/rho, the velocities u = RU/rho, v, w and the
// diagonal momentum fluxes p + RU u, p + RV v, p + RW w with p = rho T) are
// computed once per point.  One thread per column then evaluates the whole
// right-hand side of fluxes() (3dmhdsub.h:194-696) for cell (z, y, x), applies
// the RK update of step_block_GAM (3dmhdsub.h:181-192), forms the next
// substage's register Z' = U' + zeta*dt*F (step_block_ZETA, 3dmhdsub.h:168-179)
// and writes U' together with its periodic ghost images (communicate(),
// 3dmhdmpi.h:11-143, as dual stores).  The wall conditions BCON
// (3dmhdsub.h:720-873) follow in the same thread where its z range reaches
// three planes into the grid, else in a separate small kernel.
//
// GB300's FP64 unit takes 16 cycles of an SM for a warp's DFMA with three
// register operands, but 19 for a DADD, a DMUL or a DFMA with a constant-bank
// operand, whatever the number of active lanes (measured with one CTA per SM:
// 2.00 against 1.68 lanes per clock).  The kernel is bound by that unit, so
//   * every sum is fma(a, 1, b) and every product fma(a, b, -0), with the 1
//     and the -0 read from memory so that they stay register operands; both
//     are exactly a + b and a * b;
//   * scalars and per-z coefficients come through shared memory instead of
//     the constant bank;
//   * points of the halo are packed into as few warps as they fill.
// and the right-hand side is grouped for the fewest FP64 instructions:
//   * advection and diffusion along one axis share their operands:
//       -D(q RU) + s D2 q = q[+] (s+ - c RU[+]) + q[-] (s- + c RU[-]) - S q,
//     where the two coefficients (formed once per axis) serve every momentum
//     component without a C43 on that axis, and in the induction equation
//     (with u instead of RU) all three components of B;
//   * the diagonal momentum flux is differenced together with the pressure,
//     before any product, as the two nearly cancel against gravity;
//   * the viscous mixed derivatives are differences of sums of 1-D
//     differences, Q1 = D_y v + D_z w (at x +- 1), Q2 = D_x u + D_z w (at
//     y +- 1) and Q3 = D_x u + D_y v (at z +- 1, carried along the column),
//     formed once per point;
//   * uniform x and y grids (UXY) divide the equations by the x metric factor
//     kappa, which the RK coefficients put back: x derivatives are then plain
//     differences, and with equal x and y spacings (ISO) y derivatives too;
//   * 1/rho is the hardware estimate (relative error e below 2^-20) times
//     1 + e + e^2, three instructions for a remainder of order e^3.
// Measured against the version before it (the same terms per cell with each
// neighbour's products formed anew, plain sums and products, about 200 FP64
// instructions per cell): a step at 512x512x256 (lMag, lRot, lShr) 68.9 ->
// 55.4 ms, a batch of 24 instances 10.3 -> 8.3 ms per step, at 32x32x32 181 ->
// 138 us (with the split and the overlapped launches of mhd_fused.cu 53.8 ms and
// 72 us).  At 256x256x128 the FP64 unit is 94 % busy with lMag, lRot and lShr (167
// instructions per cell and substage), 90 % with lMag alone (184).
// Results agree with the reference to rounding (1e-12 of each field's
// max-norm after a step, checked against the oracle).
//
// Wall planes: the values the reference overwrites in BCON (RU, RV, RW, TT,
// BZ and, with lShr, the right-hand side FT) are finite but not the
// reference's before BCON runs; RO, BX, BY and everything on interior planes
// follow the reference.  The z ghost planes are never written (the reference
// only flips RO there between rho and 1/rho; those values reach no result).
#pragma once

#include "mhd_common.cuh"

namespace mhd {
namespace fused {

template <int TX, int TY>
struct Tile {
    static constexpr int kTX = TX;
    static constexpr int kTY = TY;
    static constexpr int kThreads = TX * TY;
    static constexpr int kPX = TX + 2;
    static constexpr int kPY = TY + 2;
    static constexpr int kPlane = kPX * kPY;
    static constexpr int kHalo = kPlane - kThreads;
    static_assert(kHalo <= kThreads, "one halo point per thread at most");
};

// quantities of a ring plane, with halo; Q_PX, Q_PY are the diagonal momentum
// fluxes P + RU u, P + RV v (P = rho T), which both neighbours difference
enum Q { Q_RU = 0, Q_RV, Q_TT, Q_U, Q_V, Q_W, Q_PX, Q_PY, Q_BX, Q_BY, Q_BZ, Q_N };
// quantities kept for the thread's own column only: RW and P + RW w
enum O { O_RW = 0, O_PZ, O_N };

template <class SW>
constexpr int nq() {
    return SW::lMag ? Q_N : Q_BX;
}
template <class SW>
constexpr int nraw() {
    return SW::lMag ? 8 : 5;
}

constexpr int kZRing = 4;  // per-z coefficient rows in flight (z, z + 1 in use, z + 2 arriving)

// shared memory, in doubles: ring [3][nq][plane], Q1 and Q2 [2][2][plane], raw
// staging [nraw][plane], own columns [3][O_N][threads], coefficient rows, scalars
template <class SW, class T>
constexpr size_t ring_doubles() {
    return (size_t)(3 * nq<SW>() + 4 + nraw<SW>()) * T::kPlane + (size_t)3 * O_N * T::kThreads + kZRing * ZR_N + SC_N;
}
template <class SW, class T>
constexpr size_t ring_bytes() {
    return ring_doubles<SW, T>() * sizeof(double);
}

// 1/x by Chebyshev's third-order iteration: r is the hardware estimate, e = 1 - x r, and
// 1/x = r / (1 - e) = r (1 + e + e^2) + O(e^3); within 2^-53 + 2^-59 of the value (a rounded
// quotient's error is 2^-53)
__device__ __forceinline__ double recip(double x, double one) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double e = fma(-x, r, one);
    e = fma(e, e, e);
    return fma(r, e, r);
}

// Store v at (z, y, x) and at every periodic ghost image of that cell.
__device__ __forceinline__ void store_with_images(double* F, const Grid& g, int z, int y, int x, double v) {
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

// BCON (3dmhdsub.h:720-873) for one wall cell of U' plus its periodic ghost images.
template <class SW>
__device__ __forceinline__ void bcon_cell(const Grid& g, const Consts& c, const Fields8& U, double timt, int wall, int x,
                                          int y) {
    const long long sz = g.sz;
    const double RRT = 1.0, RRB = -1.0, RPP = 0.0;
    const int z = wall == 0 ? 1 : g.nz - 2;
    const int s = wall == 0 ? 1 : -1;
    const long long i = (long long)z * sz + (long long)y * g.sy + x;
    const long long i1 = i + s * sz, i2 = i + 2 * s * sz;
    const double *RU = U.p[S_RU], *RV = U.p[S_RV], *TT = U.p[S_TT], *RO = U.p[S_RO];
    double ru, rv, tt;
    if constexpr (SW::lShr) {
        ru = 0.0;
        rv = (wall == 0 ? RRT : RRB) * cos(RPP * timt) * RO[i];
    } else {
        ru = RO[i] * (c.C43 * RU[i1] / RO[i1] - c.C13 * RU[i2] / RO[i2]);
        rv = RO[i] * (c.C43 * RV[i1] / RO[i1] - c.C13 * RV[i2] / RO[i2]);
    }
    if (wall == 0) {
        if (c.pl_mode == 1) {
            // cooling spot on the top wall (3dmhdsub.h:750-766)
            tt = 1.0f - (1.0f - c.pl_tpr) * c.plx[x] / c.pl_hh * c.ply[y] / c.pl_hh;
        } else if (c.pl_mode == 2) {
            const double DZ = 1.0f / (double)(g.nPz - 1) / c.dzzdz[z];
            tt = c.C43 * TT[i1] - c.C13 * TT[i2] -
                 c.C23 * DZ * (c.THETA - (c.THETA - c.pl_tpr) * c.plx[x] / c.pl_hh * c.ply[y] / c.pl_hh);
        } else if (c.iTCon == 1) {
            const double DZ = 1.0f / (float)(g.nPz - 1) / c.dzzdz[z];
            tt = c.lrem ? c.C43 * TT[i1] - c.C13 * TT[i2] + c.DZTU : c.C43 * TT[i1] - c.C13 * TT[i2] - c.C23 * DZ * c.THETA;
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
            tt = c.C43 * TT[i1] - c.C13 * TT[i2] + c.DZTB;
        } else {
            const double DZ = 1.0f / (float)(g.nPz - 1) / c.dzzdz[z];
            tt = c.C43 * TT[i1] - c.C13 * TT[i2] - c.C23 * DZ * c.THETA / c.RKAPA[z];
        }
    }
    store_with_images(U.p[S_RU], g, z, y, x, ru);
    store_with_images(U.p[S_RV], g, z, y, x, rv);
    store_with_images(U.p[S_RW], g, z, y, x, 0.0);
    store_with_images(U.p[S_TT], g, z, y, x, tt);
    if constexpr (SW::lMag) {
        if (c.iBCon == 0) store_with_images(U.p[S_BZ], g, z, y, x, 0.0);
    }
}

// One tile (bx, by) of one instance, z planes [zb, ze) of the interior.
// EXTRA: the instantiation with the optional temperature terms (the iTCon 2
// plume heat sink, lRem); the others carry no code for them.  ISO (with UXY):
// cx1 = cy1.
template <class SW, class T, bool UXY, bool EXTRA = false, bool ISO = false>
__device__ __forceinline__ void substage_tile(const FusedArgs& a, int bx, int by, int zb, int ze, double* smem) {
    constexpr int NQ = nq<SW>(), NRAW = nraw<SW>();
    constexpr int kTX = T::kTX, kPX = T::kPX, kPlane = T::kPlane, kTY = T::kTY, kThreads = T::kThreads;
    constexpr int kOwn = O_N * kThreads, kRing = NQ * kPlane;
    const Grid& g = a.g;
    const Consts& c = a.c;
    const Coefs& K = a.k;
    double* ring = smem;
    double* qbuf = ring + 3 * kRing;           // [parity][Q1, Q2][plane]
    double* stage = qbuf + 4 * kPlane;         // [nraw][plane]
    double* own = stage + NRAW * kPlane;       // [slot][O_N][thread]
    double* zrow = own + 3 * kOwn;             // [kZRing][ZR_N]
    double* sc = zrow + kZRing * ZR_N;         // [SC_N]
    const double* zt = K.zt[UXY ? 1 : 0];
    const int tid = threadIdx.x;
    const int x0 = 1 + bx * kTX, y0 = 1 + by * kTY;
    const int tx = tid % kTX, ty = tid / kTX;
    const int x = x0 + tx, y = y0 + ty;
    const bool active = (x <= g.nx - 2) && (y <= g.ny - 2);
    const int zl = 1, zr = g.nz - 1;

    // this thread's points of a plane: its own column, and one halo point of
    // the rows below and above the tile (in x), then of the columns left and
    // right, then of the corners
    const int pc = (ty + 1) * kPX + (tx + 1);
    const bool own_in = x < g.nx && y < g.ny;
    int hk = 0, hkind = -1;  // halo point, 0: y halo (needs Q2), 1: x halo (Q1), 2: corner
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
    const int hgx = x0 - 1 + hk % kPX, hgy = y0 - 1 + hk / kPX;
    if (hgx >= g.nx || hgy >= g.ny) hkind = -1;
    const long long ocol = (long long)y * g.sy + x, hcol = (long long)hgy * g.sy + hgx;
    const double* U0 = a.U.p[0];
    const long long fs = a.fs;  // distance of the fields, in elements

    // raw fields of point k (column offset col) of plane z into an [nraw][plane] area
    auto copy_point = [&](double* to, int k, long long col, int z) {
        const double* src = U0 + (long long)z * g.sz + col;
#pragma unroll
        for (int f = 0; f < NRAW; f++) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(to + f * kPlane + k);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
            src += fs;
        }
    };
    // every thread copies the points it later derives itself, so its own wait
    // is the only one the derivation needs
    auto copy_plane = [&](double* to, int z) {
        if (own_in) copy_point(to, pc, ocol, z);
        if (hkind >= 0) copy_point(to, hk, hcol, z);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // ring slots of planes z - 1, z, z + 1
    double *Pm = ring + (size_t)((zb - 1) % 3) * kRing, *P0 = ring + (size_t)(zb % 3) * kRing,
           *Pp = ring + (size_t)((zb + 1) % 3) * kRing;
    double *Om = own + (size_t)((zb - 1) % 3) * kOwn, *O0 = own + (size_t)(zb % 3) * kOwn,
           *Op = own + (size_t)((zb + 1) % 3) * kOwn;
    // the scalars and the first two coefficient rows (no kernel writes them); then
    // the first three planes, each into its own slot, where it is derived
    if (tid < SC_N) sc[tid] = K.sc[UXY ? 1 : 0][tid];
    for (int k = tid; k < 2 * ZR_N; k += kThreads)
        zrow[((zb + k / ZR_N) & (kZRing - 1)) * ZR_N + k % ZR_N] = zt[(size_t)(zb + k / ZR_N) * ZR_N + k % ZR_N];
    wait_previous();
    copy_plane(Pm, zb - 1);
    copy_plane(P0, zb);
    copy_plane(Pp, zb + 1);

    __syncthreads();
    const double one = sc[SC_ONE], nzero = sc[SC_NZ];
    auto add = [&](double p, double q) { return fma(p, one, q); };
    auto sub = [&](double p, double q) { return fma(-q, one, p); };
    auto mul = [&](double p, double q) { return fma(p, q, nzero); };
    // derivatives of raw x / y differences in units of kappa
    const int xc = own_in ? x : 1, yc = own_in ? y : 1;  // (ghost columns form Q1, Q2 too)
    const double gcx = UXY ? 1.0 : K.cx1[xc];
    const double gcy = ISO ? 1.0 : UXY ? sc[SC_CY] : K.cy1[yc];
    auto SX = [&](double d) { return UXY ? d : mul(gcx, d); };
    auto SY = [&](double d) { return ISO ? d : mul(gcy, d); };
    auto AX = [&](double d, double q) { return UXY ? add(d, q) : fma(gcx, d, q); };  // q + D_x
    auto AY = [&](double d, double q) { return ISO ? add(d, q) : fma(gcy, d, q); };
    // RK coefficients, kappa included: from the host, or from the device
    // time-step record; a halted record (dt below 1e-8) turns the substage
    // into a copy of U.  With lShr the temperature equation keeps true units.
    const bool halted = a.dtp && a.dtp[3] != 0.0;
    {
        const double gdt = a.dtp ? a.gam * a.dtp[0] : a.gdt;
        const double zdt = a.dtp ? a.zet * a.dtp[0] : a.zdt;
        if (tid == 0) {
            sc[SC_G] = gdt * sc[SC_KAPPA];
            sc[SC_Z] = zdt * sc[SC_KAPPA];
            sc[SC_GT] = SW::lShr ? gdt : gdt * sc[SC_KAPPA];
            sc[SC_ZT] = SW::lShr ? zdt : zdt * sc[SC_KAPPA];
        }
    }

    double ro0 = 1.0, ri0 = 1.0, ro1 = 1.0, ri1 = 1.0, ro2 = 1.0, ri2 = 1.0;  // rho, 1/rho of planes z, z + 1, z + 2

    // ring quantities of a copied point (the copy may lie in P itself: all of
    // it is read first); returns rho, 1/rho and w, and leaves RW and P + RW w
    // of the own column in ow
    auto derive_point = [&](const double* from, int k, double* P, double* ow, double& ro, double& ri, double& ww) {
        double r[NRAW];
#pragma unroll
        for (int f = 0; f < NRAW; f++) r[f] = from[f * kPlane + k];
        ro = r[S_RO];
        ri = recip(ro, one);
        const double uu = mul(r[S_RU], ri), vv = mul(r[S_RV], ri), p = mul(ro, r[S_TT]);
        ww = mul(r[S_RW], ri);
        P[Q_RU * kPlane + k] = r[S_RU];
        P[Q_RV * kPlane + k] = r[S_RV];
        P[Q_TT * kPlane + k] = r[S_TT];
        P[Q_U * kPlane + k] = uu;
        P[Q_V * kPlane + k] = vv;
        P[Q_W * kPlane + k] = ww;
        P[Q_PX * kPlane + k] = fma(r[S_RU], uu, p);
        P[Q_PY * kPlane + k] = fma(r[S_RV], vv, p);
        if (ow) {
            ow[O_RW * kThreads + tid] = r[S_RW];
            ow[O_PZ * kThreads + tid] = fma(r[S_RW], ww, p);
        }
        if constexpr (SW::lMag) {
            P[Q_BX * kPlane + k] = r[S_BX];
            P[Q_BY * kPlane + k] = r[S_BY];
            P[Q_BZ * kPlane + k] = r[S_BZ];
        }
    };
    double dux = 0.0, dvy = 0.0, wzc = 0.0;  // the own column's raw D_x u and D_y v, and D_z w, of plane z
    double q3m = 0.0, q3c = 0.0, q3p = 0.0;  // Q3 of planes z - 1, z, z + 1
    // the own column's D_x u and D_y v of a ring plane, and their sum Q3
    auto own_q3 = [&](const double* P, double& du, double& dv) {
        du = sub(P[Q_U * kPlane + pc + 1], P[Q_U * kPlane + pc - 1]);
        dv = sub(P[Q_V * kPlane + pc + kPX], P[Q_V * kPlane + pc - kPX]);
        return AX(du, SY(dv));
    };
    // Q1 = D_y v + D_z w and Q2 = D_x u + D_z w of plane z (ring plane P) at this
    // thread's points, from w of planes z + 1 (wp, hwp) and z - 1 (wm, hwm) there;
    // leaves dux, dvy, wzc of plane z
    auto put_q = [&](const double* P, int z, double du, double dv, double wp, double wm, double hwp, double hwm) {
        double* q1 = qbuf + (z & 1) * 2 * kPlane;
        double* q2 = q1 + kPlane;
        const double cz = zrow[(z & (kZRing - 1)) * ZR_N + ZR_CZ];
        if (own_in) {
            dux = du;
            dvy = dv;
            wzc = mul(cz, sub(wp, wm));
            q1[pc] = AY(dv, wzc);
            q2[pc] = AX(du, wzc);
        }
        if (hkind == 0) {
            const double d = sub(P[Q_U * kPlane + hk + 1], P[Q_U * kPlane + hk - 1]);
            const double s = UXY ? d : mul(K.cx1[hgx], d);
            q2[hk] = fma(cz, sub(hwp, hwm), s);
        } else if (hkind == 1) {
            const double d = sub(P[Q_V * kPlane + hk + kPX], P[Q_V * kPlane + hk - kPX]);
            const double s = ISO ? d : mul(UXY ? gcy : K.cy1[hgy], d);
            q1[hk] = fma(cz, sub(hwp, hwm), s);
        }
    };

    {
        asm volatile("cp.async.wait_all;" ::: "memory");
        double wm = 0.0, wp = 0.0, hwm = 0.0, hwp = 0.0, t0, t1, t2;
        if (own_in) {
            derive_point(Pm, pc, Pm, Om, t0, t1, wm);
            derive_point(P0, pc, P0, O0, ro0, ri0, t2);
            derive_point(Pp, pc, Pp, Op, ro1, ri1, wp);
        }
        if (hkind >= 0) {
            derive_point(Pm, hk, Pm, nullptr, t0, t1, hwm);
            derive_point(P0, hk, P0, nullptr, t0, t1, t2);
            derive_point(Pp, hk, Pp, nullptr, t0, t1, hwp);
        }
        __syncthreads();
        if (zb + 2 <= ze) copy_plane(stage, zb + 2);
        double du = 0.0, dv = 0.0;
        if (own_in) {
            // (inactive columns inside the grid are neighbours too)
            q3m = own_q3(Pm, du, dv);
            q3c = own_q3(P0, du, dv);
        }
        put_q(P0, zb, du, dv, wp, wm, hwp, hwm);
    }

    for (int z = zb; z < ze; z++) {
        __syncthreads();
        const double* R = zrow + (z & (kZRing - 1)) * ZR_N;
        // row z + 2 lands before the next plane's barrier
        if (tid < ZR_N && z + 2 <= ze) zrow[((z + 2) & (kZRing - 1)) * ZR_N + tid] = zt[(size_t)(z + 2) * ZR_N + tid];
        double dux1 = 0.0, dvy1 = 0.0;
        if (own_in) q3p = own_q3(Pp, dux1, dvy1);
        if (active) {
            auto C0 = [&](int q) { return P0[q * kPlane + pc]; };
            auto XP = [&](int q) { return P0[q * kPlane + pc + 1]; };
            auto XM = [&](int q) { return P0[q * kPlane + pc - 1]; };
            auto YP = [&](int q) { return P0[q * kPlane + pc + kPX]; };
            auto YM = [&](int q) { return P0[q * kPlane + pc - kPX]; };
            auto ZP = [&](int q) { return Pp[q * kPlane + pc]; };
            auto ZM = [&](int q) { return Pm[q * kPlane + pc]; };
            const double cz = R[ZR_CZ];
            const long long i = (long long)z * g.sz + ocol;
            // the RK register (read by substages 2 and 3) and FT of this column's
            // next plane into L2, so the next iteration's epilogue does not wait
            // on DRAM for them
            if (z + 1 < ze) {
                const long long inx = i + g.sz;
                if (a.substage != 0) {
#pragma unroll
                    for (int f = 0; f < NRAW; f++)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.Z.p[0] + f * fs + inx));
                }
                if constexpr (SW::lShr) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.FT + inx));
            }
            // uniform grids: second-derivative coefficients of both neighbours in x and y, scale
            // k = 0 ORE, 1 ORE*C43, 2 ORM
            auto sx = [&](int k) { return sc[SC_SX0 + k]; };
            auto sy = [&](int k) { return sc[SC_SY0 + k]; };
            // other grids: acc + b (p - 2 c + m) + a (p - m) along an axis.  Merged into
            // factors b + a and b - a the first-derivative part would carry an error of
            // eps b (stretched x and y, RE = RM = 2, 100 steps at 24x21x20: 1.7 times the
            // error of BX and BY against 80-bit arithmetic).
            auto d2 = [&](double b, double a_, double p, double m, double c0, double acc) {
                return fma(a_, sub(p, m), fma(b, fma(-2.0, c0, add(p, m)), acc));
            };
            auto lapx = [&](int q, int k, double acc) { return d2(K.xt[2 * k][xc], K.xt[2 * k + 1][xc], XP(q), XM(q), C0(q), acc); };
            auto lapy = [&](int q, int k, double acc) { return d2(K.yt[2 * k][yc], K.yt[2 * k + 1][yc], YP(q), YM(q), C0(q), acc); };
            auto lapz = [&](int q, int k, double acc) { return d2(R[ZR_SZ0 + 2 * k], R[ZR_SZ0 + 2 * k + 1], ZP(q), ZM(q), C0(q), acc); };

            const double rwp = Op[O_RW * kThreads + tid], rwm = Om[O_RW * kThreads + tid];
            const double u = C0(Q_U), v = C0(Q_V), w = C0(Q_W), tt = C0(Q_TT);

            // ---- continuity (3dmhdsub.h:204-227), one-sided dRW/dz on the walls
            const double rup = XP(Q_RU), rum = XM(Q_RU), rvp = YP(Q_RV), rvm = YM(Q_RV);
            double rwz = sub(rwp, rwm);
            if (z == zl) rwz = 4.0 * rwp - U0[S_RW * fs + i + 2 * g.sz];
            if (z == zr - 1) rwz = U0[S_RW * fs + i - 2 * g.sz] - 4.0 * rwm;
            const double fr = fma(-cz, rwz, AY(sub(rvm, rvp), SX(sub(rum, rup))));

            // ---- momentum: pressure and gravity (3dmhdsub.h:266-272), advection
            // (3dmhdsub.h:279-289), viscous Laplacians (3dmhdsub.h:462-472)
            double fu = SX(sub(XM(Q_PX), XP(Q_PX)));
            double fv = SY(sub(YM(Q_PY), YP(Q_PY)));
            double fw = fma(cz, sub(Om[O_PZ * kThreads + tid], Op[O_PZ * kThreads + tid]), mul(sc[SC_GRAV], ro0));
            if constexpr (UXY) {
                {
                    const double ap = sub(sx(0), rup), am = add(sx(0), rum);
                    fu = fma(sx(1), XP(Q_U), fma(sx(1), XM(Q_U), fu));
                    fv = fma(ap, XP(Q_V), fma(am, XM(Q_V), fv));
                    fw = fma(ap, XP(Q_W), fma(am, XM(Q_W), fw));
                }
                {
                    const double ap = ISO ? sub(sy(0), rvp) : fma(-gcy, rvp, sy(0));
                    const double am = ISO ? add(sy(0), rvm) : fma(gcy, rvm, sy(0));
                    fu = fma(ap, YP(Q_U), fma(am, YM(Q_U), fu));
                    fv = fma(sy(1), YP(Q_V), fma(sy(1), YM(Q_V), fv));
                    fw = fma(ap, YP(Q_W), fma(am, YM(Q_W), fw));
                }
                {
                    const double ap = fma(-cz, rwp, R[ZR_SZ0]), am = fma(cz, rwm, R[ZR_SZ0 + 1]);
                    fu = fma(ap, ZP(Q_U), fma(am, ZM(Q_U), fu));
                    fv = fma(ap, ZP(Q_V), fma(am, ZM(Q_V), fv));
                    fw = fma(R[ZR_SZ0 + 2], ZP(Q_W), fma(R[ZR_SZ0 + 3], ZM(Q_W), fw));
                }
                fu = fma(-R[ZR_SU], u, fu);
                fv = fma(-R[ZR_SV], v, fv);
                fw = fma(-R[ZR_SW], w, fw);
            } else {
                fu = fma(-gcy, fma(rvp, YP(Q_U), mul(-rvm, YM(Q_U))), fu);
                fu = fma(-cz, fma(rwp, ZP(Q_U), mul(-rwm, ZM(Q_U))), fu);
                fv = fma(-gcx, fma(rup, XP(Q_V), mul(-rum, XM(Q_V))), fv);
                fv = fma(-cz, fma(rwp, ZP(Q_V), mul(-rwm, ZM(Q_V))), fv);
                fw = fma(-gcx, fma(rup, XP(Q_W), mul(-rum, XM(Q_W))), fw);
                fw = fma(-gcy, fma(rvp, YP(Q_W), mul(-rvm, YM(Q_W))), fw);
                fu = lapz(Q_U, 0, lapy(Q_U, 0, lapx(Q_U, 1, fu)));
                fv = lapz(Q_V, 0, lapy(Q_V, 1, lapx(Q_V, 0, fv)));
                fw = lapz(Q_W, 1, lapy(Q_W, 0, lapx(Q_W, 0, fw)));
            }

            // ---- viscous cross terms (3dmhdsub.h:486-487,517-518,531-532)
            {
                const double* q1 = qbuf + (z & 1) * 2 * kPlane + pc;
                const double* q2 = q1 + kPlane;
                const double kqx = UXY ? sc[SC_KQX] : sc[SC_KQX] * gcx, kqy = UXY ? sc[SC_KQY] : sc[SC_KQY] * gcy;
                fu = fma(kqx, sub(q1[1], q1[-1]), fu);
                fv = fma(kqy, sub(q2[kPX], q2[-kPX]), fv);
                fw = fma(R[ZR_KQZ], sub(q3p, q3m), fw);
            }

            // ---- temperature: advection (3dmhdsub.h:293-296), conduction (:315-319)
            double ft;
            double qr;  // the temperature terms proportional to 1/rho, applied once at the end
            const double czw = mul(cz, w);
            double dTz = 0.0;
            if constexpr (!SW::lShr || !UXY) dTz = sub(ZP(Q_TT), ZM(Q_TT));
            if constexpr (!SW::lShr) {
                const double dTx = sub(XP(Q_TT), XM(Q_TT)), dTy = sub(YP(Q_TT), YM(Q_TT));
                ft = UXY ? mul(-u, dTx) : mul(-gcx * u, dTx);
                ft = ISO ? fma(-v, dTy, ft) : fma(-gcy * v, dTy, ft);
                ft = fma(-czw, dTz, ft);
            } else {
                ft = a.FT[i];  // the reference never re-initialises FT with lShr
            }
            {
                double lapT = 0.0;
                if constexpr (!UXY) {
                    lapT = d2(R[ZR_TZP], R[ZR_TZM], ZP(Q_TT), ZM(Q_TT), tt, lapy(Q_TT, 3, lapx(Q_TT, 3, 0.0)));
                } else if (EXTRA && c.lrem && !SW::lShr) {
                    lapT = mul(sc[SC_TX], XP(Q_TT));
                    lapT = fma(sc[SC_TX], XM(Q_TT), lapT);
                    lapT = fma(sc[SC_TY], YP(Q_TT), lapT);
                    lapT = fma(sc[SC_TY], YM(Q_TT), lapT);
                    lapT = fma(R[ZR_TZP], ZP(Q_TT), fma(R[ZR_TZM], ZM(Q_TT), lapT));
                    lapT = fma(-R[ZR_STL], tt, lapT);
                }
                if (EXTRA && c.lrem && !SW::lShr) {
                    // lRem: conduction of T - TTM(z) plus HRAD (3dmhdsub.h:297-313),
                    // as lap T + (HRAD - d2 TTM/dz2), the latter precomputed per z
                    qr = sc[SC_TMPC] * (lapT + c.lrem_g[z]);
                } else if constexpr (UXY) {
                    // kapz lap T + dkapz dT/dz with kapz folded into the per-z coefficients
                    qr = mul(R[ZR_KX], XP(Q_TT));
                    qr = fma(R[ZR_KX], XM(Q_TT), qr);
                    qr = fma(R[ZR_KY], YP(Q_TT), qr);
                    qr = fma(R[ZR_KY], YM(Q_TT), qr);
                    qr = fma(R[ZR_KZP], ZP(Q_TT), qr);
                    qr = fma(R[ZR_KZM], ZM(Q_TT), qr);
                    qr = fma(-R[ZR_ST], tt, qr);
                } else {
                    qr = fma(R[ZR_KZP], lapT, R[ZR_KZM] * dTz);  // kapz, dkapz cz1
                }
            }
            // internal plume heat sink (iTCon 2, 3dmhdsub.h:443-459)
            if constexpr (EXTRA) {
                if (c.pl_mode == 3) qr = fma(-c.pl_s * sc[SC_ST], c.plx[x] * c.ply[y] * c.plz[z], qr);
            }

            // velocity gradients in units of kappa (heating and induction); the z
            // gradients of u and v stay raw
            double ux = 0, uy = 0, dUz = 0, vx = 0, vy = 0, dVz = 0, wx = 0, wy = 0;
            if constexpr (!SW::lShr || SW::lMag) {
                ux = SX(dux);
                vx = SX(sub(XP(Q_V), XM(Q_V)));
                wx = SX(sub(XP(Q_W), XM(Q_W)));
                uy = SY(sub(YP(Q_U), YM(Q_U)));
                vy = SY(dvy);
                wy = SY(sub(YP(Q_W), YM(Q_W)));
                dUz = sub(ZP(Q_U), ZM(Q_U));
                dVz = sub(ZP(Q_V), ZM(Q_V));
            }
            // ---- viscous heating and pdV work (3dmhdsub.h:477-538, not with lShr):
            // ux^2 + vy^2 + wz^2 - ux vy - (ux + vy) wz = div^2 - 3 (ux vy + (ux + vy) wz)
            if constexpr (!SW::lShr) {
                const double div = add(q3c, wzc);
                const double s1 = add(uy, vx), s2 = fma(cz, dUz, wx), s3 = fma(cz, dVz, wy);
                double phi = fma(s1, s1, fma(s2, s2, mul(s3, s3)));
                phi = fma(sc[SC_C43], mul(div, div), phi);
                phi = fma(-sc[SC_C43X3], fma(wzc, q3c, mul(ux, vy)), phi);
                qr = fma(sc[SC_HQ], phi, qr);
                ft = fma(mul(sc[SC_MOCV], tt), div, ft);
            }

            // ---- Coriolis (3dmhdsub.h:540-545)
            if constexpr (SW::lRot) {
                const double omz = sc[SC_OMZ], omx = sc[SC_OMX], rv = C0(Q_RV);
                fu = fma(omz, rv, fu);
                fv = fma(-omz, C0(Q_RU), fv);
                fv = fma(omx, O0[O_RW * kThreads + tid], fv);
                fw = fma(-omx, rv, fw);
            }

            // ---- induction, Lorentz force, Ohmic heating (3dmhdsub.h:547-695)
            double w1 = 0, w2 = 0, w3 = 0;
            if constexpr (SW::lMag) {
                const double bx = C0(Q_BX), by = C0(Q_BY), bz = C0(Q_BZ);
                const bool wall = (z == zl || z == zr - 1);
                // stretching; one-sided dw/dz on the walls (3dmhdsub.h:572-584)
                double wzm = wzc;
                if (wall) {
                    const long long j = z == zl ? i + 2 * g.sz : i - 2 * g.sz;
                    const double w2nd = U0[S_RW * fs + j] / U0[S_RO * fs + j];
                    wzm = z == zl ? (4.0 * ZP(Q_W) - w2nd) * cz : (w2nd - 4.0 * ZM(Q_W)) * cz;
                }
                const double bzc = mul(cz, bz);
                w1 = fma(by, uy, fma(bzc, dUz, mul(-bx, add(vy, wzm))));
                w2 = fma(bx, vx, fma(bzc, dVz, mul(-by, add(ux, wzm))));
                w3 = fma(bx, wx, fma(by, wy, mul(-bz, q3c)));
                // advection and resistive Laplacians
                if constexpr (UXY) {
                    {
                        const double ap = sub(sx(2), u);
                        const double am = add(sx(2), u);
                        w1 = fma(ap, XP(Q_BX), fma(am, XM(Q_BX), w1));
                        w2 = fma(ap, XP(Q_BY), fma(am, XM(Q_BY), w2));
                        w3 = fma(ap, XP(Q_BZ), fma(am, XM(Q_BZ), w3));
                    }
                    {
                        const double ap = ISO ? sub(sy(2), v) : fma(-gcy, v, sy(2));
                        const double am = ISO ? add(sy(2), v) : fma(gcy, v, sy(2));
                        w1 = fma(ap, YP(Q_BX), fma(am, YM(Q_BX), w1));
                        w2 = fma(ap, YP(Q_BY), fma(am, YM(Q_BY), w2));
                        w3 = fma(ap, YP(Q_BZ), fma(am, YM(Q_BZ), w3));
                    }
                    const double ap = sub(R[ZR_SZ0 + 4], czw), am = add(R[ZR_SZ0 + 5], czw);
                    w3 = fma(ap, ZP(Q_BZ), fma(am, ZM(Q_BZ), w3));
                    w3 = fma(-R[ZR_SB], bz, w3);
                    if (!wall) {
                        const double S = R[ZR_SB];
                        w1 = fma(ap, ZP(Q_BX), fma(am, ZM(Q_BX), fma(-S, bx, w1)));
                        w2 = fma(ap, ZP(Q_BY), fma(am, ZM(Q_BY), fma(-S, by, w2)));
                    }
                } else {
                    const double cxu = mul(gcx, u), cyv = mul(gcy, v);
                    auto advect = [&](int q, double acc) {
                        acc = fma(-czw, sub(ZP(q), ZM(q)), acc);
                        return fma(-cxu, sub(XP(q), XM(q)), fma(-cyv, sub(YP(q), YM(q)), acc));
                    };
                    w1 = lapy(Q_BX, 2, lapx(Q_BX, 2, advect(Q_BX, w1)));
                    w2 = lapy(Q_BY, 2, lapx(Q_BY, 2, advect(Q_BY, w2)));
                    w3 = lapz(Q_BZ, 2, lapy(Q_BZ, 2, lapx(Q_BZ, 2, advect(Q_BZ, w3))));
                    if (!wall) {
                        w1 = lapz(Q_BX, 2, w1);
                        w2 = lapz(Q_BY, 2, w2);
                    }
                }
                if (wall) {
                    // d2B/dz2 with the one-sided wall stencils (3dmhdsub.h:640-654,673-687)
                    const double S = R[ZR_SBW];
                    const int s = (z == zl) ? 1 : -1;
                    const long long j2 = i + 2 * s * g.sz, j3 = i + 3 * s * g.sz;
                    const double a2 = R[ZR_WD2], b2 = R[ZR_WD1];
                    const double X1 = (s > 0) ? ZP(Q_BX) : ZM(Q_BX), X2 = U0[S_BX * fs + j2], X3 = U0[S_BX * fs + j3];
                    const double Y1 = (s > 0) ? ZP(Q_BY) : ZM(Q_BY), Y2 = U0[S_BY * fs + j2], Y3 = U0[S_BY * fs + j3];
                    const double sg = (double)s;
                    if constexpr (UXY) {
                        w1 = fma(-czw, ZP(Q_BX) - ZM(Q_BX), fma(-S, bx, w1));
                        w2 = fma(-czw, ZP(Q_BY) - ZM(Q_BY), fma(-S, by, w2));
                    }
                    w1 += sg * (-3.0 * bx + 4.0 * X1 - X2) * a2 + (2.0 * bx - 5.0 * X1 + 4.0 * X2 - X3) * b2;
                    w2 += sg * (-3.0 * by + 4.0 * Y1 - Y2) * a2 + (2.0 * by - 5.0 * Y1 + 4.0 * Y2 - Y3) * b2;
                }
                // current density j' = OBETA j (in units of kappa): the Lorentz force is
                // B x j' and the Ohmic heating proportional to |j'|^2
                const double ob = sc[SC_OB], ocz = R[ZR_OCZ];
                const double obx = UXY ? ob : ob * gcx, oby = ISO ? ob : ob * gcy;
                const double dBYx = sub(XP(Q_BY), XM(Q_BY)), dBXy = sub(YP(Q_BX), YM(Q_BX));
                const double dBZx = sub(XP(Q_BZ), XM(Q_BZ)), dBXz = sub(ZP(Q_BX), ZM(Q_BX));
                const double dBZy = sub(YP(Q_BZ), YM(Q_BZ)), dBYz = sub(ZP(Q_BY), ZM(Q_BY));
                const double jz = ISO ? mul(ob, sub(dBYx, dBXy)) : fma(obx, dBYx, mul(-oby, dBXy));
                const double jy = fma(ocz, dBXz, mul(-obx, dBZx));
                const double jx = fma(oby, dBZy, mul(-ocz, dBYz));
                fu = fma(bz, jy, fma(-by, jz, fu));
                fv = fma(bx, jz, fma(-bz, jx, fv));
                fw = fma(by, jx, fma(-bx, jy, fw));
                qr = fma(sc[SC_OHM], fma(jx, jx, fma(jy, jy, mul(jz, jz))), qr);
            }

            ft = fma(ri0, qr, ft);

            // ---- RK3 substage update and the next register (3dmhdsub.h:168-192); the
            // register is read before anything is written, as the stores may alias
            // the loads as far as the compiler knows
            const double fl[8] = {fu, fv, fw, ft, fr, w1, w2, w3};
            double zf[NRAW];
#pragma unroll
            for (int f = 0; f < NRAW; f++) {
                constexpr int ring_of[8] = {Q_RU, Q_RV, 0, Q_TT, 0, Q_BX, Q_BY, Q_BZ};
                if (a.substage == 0 || halted) zf[f] = f == S_RW ? O0[O_RW * kThreads + tid] : f == S_RO ? ro0 : C0(ring_of[f]);
                else zf[f] = a.Z.p[0][f * fs + i];
            }
#pragma unroll
            for (int f = 0; f < NRAW; f++) {
                const double un = halted ? zf[f] : fma(sc[f == S_TT ? SC_GT : SC_G], fl[f], zf[f]);
                store_with_images(a.Uo.p[0] + f * fs, g, z, y, x, un);
                if (a.substage < 2) a.Z.p[0][f * fs + i] = halted ? un : fma(sc[f == S_TT ? SC_ZT : SC_Z], fl[f], un);
            }
            if constexpr (SW::lShr) {
                if (!halted) a.FT[i] = ft;
            }
        }
        if (z + 1 < ze) {
            // plane z + 2 into the slot of plane z - 1, of which every thread reads
            // its own points only; then Q1 and Q2 of plane z + 1
            asm volatile("cp.async.wait_all;" ::: "memory");
            double w2 = 0.0, hw2 = 0.0, hr, hi;
            if (own_in) derive_point(stage, pc, Pm, Om, ro2, ri2, w2);
            if (hkind >= 0) derive_point(stage, hk, Pm, nullptr, hr, hi, hw2);
            if (z + 3 <= ze) copy_plane(stage, z + 3);
            put_q(Pp, z + 1, dux1, dvy1, w2, P0[Q_W * kPlane + pc], hw2, P0[Q_W * kPlane + hk]);
            q3m = q3c;
            q3c = q3p;
            ro0 = ro1;
            ri0 = ri1;
            ro1 = ro2;
            ri1 = ri2;
            double* t = Pm;
            Pm = P0;
            P0 = Pp;
            Pp = t;
            t = Om;
            Om = O0;
            O0 = Op;
            Op = t;
        }
    }
    // BCON of a wall reads the new values of its column two planes in, all
    // written by this thread when the z range holds them
    if (active) {
        if ((a.walls & 1) && zb == 1) bcon_cell<SW>(g, c, a.Uo, a.timt, 0, x, y);
        if ((a.walls & 2) && ze == g.nz - 1) bcon_cell<SW>(g, c, a.Uo, a.timt, 1, x, y);
    }
}

}  // namespace fused
}  // namespace mhd
