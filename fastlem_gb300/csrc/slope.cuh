// slope.cuh -- single-precision slope estimates for the steepest-descent receivers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fl {

// ---- float pairs: an elevation as hi + lo ------------------------------------------
//
// hi is the elevation cut to 24 significant bits, lo the remaining 29 rounded to 24, so
// |e - (hi + lo)| <= 2^-48 |e|.  A difference of two elevations then costs three f32
// additions instead of 64-bit integer work on both operands at every adjacency slot (about
// 20 instructions a slot instead of 60).  hi is NaN for values whose pair could leave the
// normal f32 range (zero is exact); rows that meet one are scanned in f64.
__device__ __forceinline__ float2 float_pair(double e) {
    const uint64_t b = (uint64_t)__double_as_longlong(e);
    const uint32_t top = (uint32_t)(b >> 32), ex = (top >> 20) & 0x7ffu, sign = top & 0x80000000u;
    if (ex - 950u > 170u)
        return make_float2((b << 1) == 0 ? 0.0f : __uint_as_float(0x7fc00000u), 0.0f);
    const float hi = __uint_as_float(sign | ((ex - 896u) << 23) | ((uint32_t)(b >> 29) & 0x7fffffu));
    const float lo = __uint2float_rn((uint32_t)b & 0x1fffffffu) *
                     __uint_as_float(sign | ((ex - 948u) << 23));
    return make_float2(hi, lo);
}

// The steepest of a row's slots by estimate.  With d = e_i - e_j, its estimate
// (hi_i - hi_j) + (lo_i - lo_j) is within 2^-23 |d| + 2^-45.4 |e_i| of it (two roundings of
// 2^-24; the pairs' errors and the rounding of lo_i - lo_j), so beyond 2^-24 |e_i| it has
// d's sign and a relative error below 2^-21.  The slope estimate adds the slot's 1/len and
// a product (2^-24 each): below 2^-20, as receivers.cu's comparison margin of 2^-17 needs.
// Differences below that threshold, NaN, slopes out of range and near-ties are left to the
// f64 scan.
struct PairScan {
    float hi, lo, thr, best = 0.0f, second = 0.0f;
    uint32_t slot = 0xffffffffu;
    bool exact = false;
    __device__ __forceinline__ explicit PairScan(float2 e)
        : hi(e.x), lo(e.y), thr(fabsf(e.x) * 5.9604644775390625e-08f) {}
    __device__ __forceinline__ void consider(uint32_t s, float2 ej, float ilen) {
        const float d = (hi - ej.x) + (lo - ej.y);
        const float f = d * ilen;
        exact |= !(fabsf(d) > thr);
        if (d > thr) {
            exact |= !(f > 1e-30f && f < 1e30f);
            second = fmaxf(second, fminf(best, f));
            if (f > best) {
                best = f;
                slot = s;
            }
        }
    }
    __device__ __forceinline__ bool decided() const {
        return !exact && !(second > best * (1.0f - 7.62939453125e-06f));
    }
};

// ---- estimates from the bit patterns of two doubles (the bounds are in receivers.cu) --
constexpr uint64_t kMant = (1ull << 52) - 1;
// Float estimate of (a - b) for non-negative finite doubles with bits A > B.
// Returns false when the result falls outside the normal f32 range.
__device__ __forceinline__ bool diff_estimate(uint64_t A, uint64_t B, float& out) {
    int ea = (int)(A >> 52), eb = (int)(B >> 52);
    uint64_t ma = (A & kMant) | (ea ? (1ull << 52) : 0);
    uint64_t mb = (B & kMant) | (eb ? (1ull << 52) : 0);
    ea = ea ? ea : 1;
    eb = eb ? eb : 1;
    int sh = ea - eb;
    uint64_t D;
    int E;
    if (sh <= 11) {
        D = (ma << sh) - mb;
        E = eb;
    } else {
        D = ma - (sh < 64 ? (mb >> sh) : 0);
        E = ea;
    }
    if (D == 0) return false;
    int lz = __clzll((long long)D);
    uint64_t top = D << lz;                      // leading one at bit 63
    int e2 = (63 - lz) + E - 1075;               // d = 1.xxx * 2^e2
    int fe = e2 + 127;
    if (fe <= 0 || fe >= 255) return false;
    uint32_t fb = ((uint32_t)fe << 23) | (uint32_t)((top >> 40) & 0x7fffffu);
    out = __uint_as_float(fb);
    return true;
}

// f32 estimate of a - b for non-negative finite doubles with bits A > B.  Sharing
// the exponent field e in [949, 1149], A - B is the difference in units of 2^(e-1075)
// (below 2^52) and the scaled result is a normal f32 number.  The 52-bit difference is
// converted as two 32-bit halves (a 64-bit integer conversion issues on the f64 pipe):
// the high half is exact, the low half truncated and the fused sum rounded, within
// 2^-23 relative.
__device__ __forceinline__ bool slope_diff(uint64_t A, uint64_t B, float& out) {
    const uint32_t e = (uint32_t)(A >> 52);
    if (e == (uint32_t)(B >> 52) && e - 949u <= 200u) {
        const uint64_t D = A - B;
        const float d = fmaf(__uint2float_rz((uint32_t)(D >> 32)), 4294967296.0f,
                             __uint2float_rz((uint32_t)D));
        out = d * __uint_as_float((e - 948u) << 23);
        return true;
    }
    return diff_estimate(A, B, out);
}

}  // namespace fl
