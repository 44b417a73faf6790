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

}  // namespace fl
