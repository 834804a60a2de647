// mhd_selftest.cu -- on-device checks of the integer-pipe conversions of
// mhd_convert.cuh against the hardware conversions, and of the substages'
// reciprocals against 1 / x.
#include "mhd_context.h"
#include "mhd_convert.cuh"
#include "mhd_fp32_tile.cuh"
#include "mhd_fused_tile.cuh"

namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ bool same_f32(float a, float b) {
    return (a != a && b != b) || __float_as_uint(a) == __float_as_uint(b);
}
__device__ __forceinline__ bool same_f64(double a, double b) {
    return (a != a && b != b) || __double_as_longlong(a) == __double_as_longlong(b);
}

// Test patterns: random bits; doubles near the float range edges and on
// rounding ties; random floats (all exponents, subnormals included).
__global__ void k_selftest(long long n, unsigned long long seed, unsigned long long* bad) {
    unsigned long long nb = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const unsigned long long h = mix64(seed ^ mix64((unsigned long long)t));
        double d;
        switch (t & 3) {
            case 0: d = __longlong_as_double((long long)h); break;
            case 1: {  // exponents around the float range, low bits forming ties
                const unsigned long long e = 1023 - 160 + (h >> 56) % 330;
                unsigned long long m = h & 0xfffffffffffffull;
                if ((h >> 40) & 1) m = (m & ~0x1fffffffull) | 0x10000000ull;  // exact tie
                d = __longlong_as_double((long long)((e << 52) | m | (h & 0x8000000000000000ull)));
                break;
            }
            case 2: d = 1.0 + (double)(h >> 11) * 0x1p-53; break;
            default: {
                const float f = __uint_as_float((unsigned)(h >> 32));
                if (!same_f64(mhd::widen_f32(f), (double)f)) nb++;
                d = __longlong_as_double((long long)h) * 0x1p-900;
            }
        }
        if (!same_f32(mhd::narrow_f64(d), __double2float_rn(d))) nb++;
        const float f = __double2float_rn(d);
        if (!same_f64(mhd::widen_f32(f), (double)f)) nb++;
        // the substage's forms: f 2^-896 for finite f, and the rounding of ordinary values
        if (isfinite(f) && !same_f64(mhd::widen_scaled(f) * 0x1p896, (double)f)) nb++;
        if (mhd::narrow_ordinary(d) && !same_f32(mhd::narrow_fast(d), f)) nb++;
    }
    if (nb) atomicAdd(bad, nb);
}

// recip32 on every float (bad[0]): within 2^-24 + 2^-43 of the value where it takes the
// Newton step; elsewhere zeros, infinities and NaN of the quotient exactly and the
// other results within one unit in the last place of it.  recip on n patterns with
// exponents -1020 .. 1020 (bad[1]): within 2^-53 + 2^-59, for an estimate good to 2^-20
// the bound of its rounding and the terms that its series leaves out.  1 - x r is exact
// in both tests (a product of two floats fits a double; the fused multiply-add's
// result fits where r is that close).
__global__ void k_selftest_recip(long long n, unsigned long long seed, double one, unsigned long long* bad) {
    unsigned long long b32 = 0, b64 = 0;
    const long long stride = (long long)gridDim.x * blockDim.x, t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long t = t0; t < (1LL << 32); t += stride) {
        const float x = __uint_as_float((unsigned)t), r = mhd::fp32::recip32(x), q = 1.0f / x;
        const float ax = fabsf(x);
        if (ax >= 0x1p-126f && ax <= 0x1p126f) {
            if (!(fabs(fma(-(double)x, (double)r, 1.0)) <= 0x1p-24 + 0x1p-43)) b32++;
        } else if (q != q || isinf(q) || q == 0.0f) {
            if (!same_f32(r, q)) b32++;
        } else {
            const int d = __float_as_int(r) - __float_as_int(q);
            if (d < -1 || d > 1) b32++;
        }
    }
    for (long long t = t0; t < n; t += stride) {
        const unsigned long long h = mix64(seed ^ mix64((unsigned long long)t));
        const unsigned long long e = 3 + (h >> 52) % 2041;
        const double x = __longlong_as_double((long long)((mix64(h) & 0x800fffffffffffffull) | e << 52));
        if (!(fabs(fma(-x, mhd::fused::recip(x, one), 1.0)) <= 0x1p-53 + 0x1p-59)) b64++;
    }
    if (b32) atomicAdd(bad, b32);
    if (b64) atomicAdd(bad + 1, b64);
}

}  // namespace

extern "C" int mhd_selftest_recip(long long n, unsigned long long seed, long long* bad32, long long* bad64) {
    if (n < 0 || !bad32 || !bad64) return MHD_ERR_INVALID;
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 2 * sizeof(unsigned long long)) != cudaSuccess) return MHD_ERR_NOMEM;
    cudaMemset(d, 0, 2 * sizeof(unsigned long long));
    k_selftest_recip<<<152 * 8, 256>>>(n, seed, 1.0, d);
    unsigned long long h[2] = {0, 0};
    const cudaError_t e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return MHD_ERR_CUDA;
    *bad32 = (long long)h[0];
    *bad64 = (long long)h[1];
    return MHD_OK;
}

extern "C" int mhd_selftest_convert(long long n, unsigned long long seed, long long* mismatches) {
    if (n < 0 || !mismatches) return MHD_ERR_INVALID;
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, sizeof(unsigned long long)) != cudaSuccess) return MHD_ERR_NOMEM;
    cudaMemset(d, 0, sizeof(unsigned long long));
    k_selftest<<<152 * 8, 256>>>(n, seed, d);
    unsigned long long h = 0;
    cudaError_t e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return MHD_ERR_CUDA;
    *mismatches = (long long)h;
    return MHD_OK;
}
