// mhd_split.h -- how a substage launch is cut into blocks of (tile, z range): plain
// C++, which the tests compile on its own.
#pragma once

#include <algorithm>

#ifdef __CUDACC__
#define MHD_SPLIT_HD __host__ __device__ __forceinline__
#else
#define MHD_SPLIT_HD inline
#endif

namespace mhd {

// planes next to a wall that BCON involves
constexpr int kWallPlanes = 3;

// Blocks of a substage launch, (tile, z range) each, of planes [lo, lo + planes).
// Every tile in `ranges` ranges, the tiles of a range one after another; or
// (ranges = 0) up to four classes of equal length, numbered in order: block j of a
// class is tile tile0 + j % tiles, planes [lo + z0 + len * (j / tiles), + len).
struct ZSplit {
    int lo, planes, nbx, tiles, ranges;
    int first, last;  // planes of the shortest range that begins at lo, and that ends the planes
    struct Class {
        int blocks, tile0, tiles, z0, len;
    } cls[4];
};

// Class of block j of a split into unequal numbers of ranges; j becomes its number in the class.
MHD_SPLIT_HD ZSplit::Class block_class(const ZSplit& s, int& j) {
    ZSplit::Class k = s.cls[0];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int c = 1; c < 4; c++) {
        if (j < k.blocks) continue;
        j -= k.blocks;
        k = s.cls[c];
    }
    return k;
}

// First plane of z range k of n over `planes` planes.
inline int chunk_begin(int planes, int k, int n) { return (int)((long long)planes * k / n); }

// Split of `planes` planes from lo on, of `tiles` tiles in rows of nbx, into n blocks:
// where n is no multiple of the tiles, the first n % tiles of them have one range
// more than the others, a tile's longer ranges come first, and the blocks are numbered
// by falling length.
inline ZSplit make_split(int lo, int planes, int nbx, int tiles, long long n) {
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
inline int range_length(const ZSplit& s, long long block) {
    int j = (int)block;
    return block_class(s, j).len;
}

// Whether the z ranges next to the walls hold the planes of BCON.
inline int split_walls(int nz, const ZSplit& s) {
    return (s.lo == 1 && s.first >= kWallPlanes ? 1 : 0) |
           (s.lo + s.planes == nz - 1 && s.last >= kWallPlanes ? 2 : 0);
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
// 2 % of the fastest on those 19 grids, and within 1.1 % without lMag, with lShr and
// with all three switches, whose planes cost 0.6 to 0.95 of the unit (nine grids of
// 32^3 to 200x150x100, 1 .. 32 ranges and the full wave).  Against at most eight ranges of four
// planes, us per step, launches not overlapped: 32x32x32 138 -> 87 (32 ranges of
// one plane), 97x45x61 (no field) 344 -> 272, 128x128x64 1146 -> 1094 (BCON inside
// the launch included).
inline long long choose_blocks(int nz, bool mixed, int resident, int nbx, long long tiles, int sms, int lo, int planes) {
    long long best = tiles;
    double best_cost = 1e300;
    const int need = (lo == 1 ? 1 : 0) | (lo + planes == nz - 1 ? 2 : 0);
    const long long wave = (long long)resident * sms;
    // A slab of a host-to-host step runs beside the slabs of other substages,
    // which fill its last wave: where a plane has a wave of tiles, about two waves
    // of long ranges.  ms per step with the model below and so: 256x256x128 (512
    // tiles) 8.79, 8.40; 240x248x64, 256x240x64 and 512x256x64 equal; 320x200x100
    // (500) 7.20, 7.35; 320x320x100 (800) 10.68, 10.78.  From half a wave on it would
    // lose: 200x150x100 (247) 3.55, 3.79; 224x232x128 (406) 6.72, 6.97.
    if (planes < nz - 2 && tiles >= wave)
        return tiles * std::max(1LL, std::min<long long>(planes, (2 * wave + tiles / 2) / tiles));
    for (int c = 1; c <= planes; c++) {
        const long long n = tiles * c;
        const double most = (planes + c - 1) / c, avg = (double)planes / c;
        double cost = n <= sms       ? 1.5 + 1.24 * most
                      : n <= 2 * sms ? 1.5 + 2.1 * most
                      : n <= wave    ? 1.5 + 2.95 * most
                                     : 1.0 + (double)((n + wave - 1) / wave) * (1.4 + 2.95 * avg);
        if (split_walls(nz, make_split(lo, planes, nbx, (int)tiles, n)) != need) cost += 0.6;
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
    if (resident == 3 && mixed && wave >= tiles && wave <= tiles * planes && wave % tiles != 0) {
        const ZSplit s = make_split(lo, planes, nbx, (int)tiles, wave);
        const int l1 = range_length(s, 0), l2 = range_length(s, sms), l3 = range_length(s, 2LL * sms);
        double cost = 1.7 + 2.95 * l3 + 2.1 * (l2 - l3) + 1.24 * (l1 - l2);
        if (split_walls(nz, s) != need) cost += 1.3;
        if (1.02 * cost < best_cost) best = wave;
    }
    return best;
}

// ---- FP32-storage substage -------------------------------------------------
constexpr int kTX32 = 32;       // columns of a tile
constexpr int kResident32 = 4;  // CTAs per SM

inline int split32_walls(int planes, int chunks) {
    return (chunk_begin(planes, 1, chunks) >= kWallPlanes ? 1 : 0) |
           (planes - chunk_begin(planes, chunks - 1, chunks) >= kWallPlanes ? 2 : 0);
}

// Microseconds (less a constant) per launch of n CTAs: tiles of ty rows, c z ranges.
// While all are resident, the planes of a CTA (0.4 more around a range) follow one
// another, L each, and share their SM's issue slots with the other CTAs, q each;
// with more CTAs than that, in waves that overlap in part, b per plane.  Last, a
// separate BCON launch where a range at a wall is too short for it.  Fitted to
// launches with lMag on 16 grids of 32^3 .. 512x384x96 cells, 1 .. 64 ranges and
// both tiles: on those grids the split that it chooses is within 1 % of the fastest.
inline double cost32(int ty, long long n, int sms, int planes, int c) {
    const double L = 2.1, q = ty == 4 ? 0.47 : 0.65, b = ty == 4 ? 4.27 : 4.73;
    const double start = ty == 4 ? 0.0 : 1.7, more = ty == 4 ? 6.4 : 7.0, f = ty == 4 ? 0.85 : 0.63;
    const long long wave = (long long)kResident32 * sms, per_sm = (n + sms - 1) / sms;
    const double most = (planes + c - 1) / c + 0.4, avg = (double)planes / c + 0.4;
    const double waves = f * (double)n / wave + (1.0 - f) * (double)((n + wave - 1) / wave);
    const double t = start + (n <= wave ? L * most + q * per_sm * avg : more + b * waves * avg);
    return split32_walls(planes, c) == 3 ? t : t + 3.1;
}

// Rows per tile and number of z ranges for one instance of nx x ny interior columns.
struct Split32 {
    int ty, chunks;
};
inline Split32 split32(int nx, int ny, int planes, int sms) {
    Split32 best{5, 1};
    double best_cost = 1e300;
    for (int ty = 4; ty <= 5; ty++) {
        const long long tiles = (long long)((nx + kTX32 - 1) / kTX32) * ((ny + ty - 1) / ty);
        for (int c = 1; c <= planes; c++) {
            const double cost = cost32(ty, tiles * c, sms, planes, c);
            if (cost < best_cost - 1e-9) {
                best_cost = cost;
                best = {ty, c};
            }
        }
    }
    return best;
}

}  // namespace mhd
