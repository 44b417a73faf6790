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
// d's sign and a relative error below 2^-21.4 + 2^-23 < 2^-20.9.  The slope estimate adds the
// slot's 1/len and a product (2^-24 each): below 2^-20.6, well within receivers.cu's comparison
// margin of 2^-17.
// Rows with a difference below that threshold (or NaN) are scanned from the doubles' bits
// (steepest_bits); slopes out of range and near-ties are left to the f64 scan.
struct PairScan {
    float hi, lo, thr, best = 0.0f, second = 0.0f;
    uint32_t slot = 0xffffffffu;
    bool exact = false, close = false;
    __device__ __forceinline__ explicit PairScan(float2 e)
        : hi(e.x), lo(e.y), thr(fabsf(e.x) * 5.9604644775390625e-08f) {}
    __device__ __forceinline__ void consider(uint32_t s, float2 ej, float ilen) {
        const float d = (hi - ej.x) + (lo - ej.y);
        const float f = d * ilen;
        close |= !(fabsf(d) > thr);
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
        return !exact && !close && !(second > best * (1.0f - 7.62939453125e-06f));
    }
};

// ---- estimates from the doubles' bits ----------------------------------------------

// a - b in f32 for non-negative finite doubles with bits A > B, within 2^-23 relative; false
// when it is outside the normal f32 range.  Sharing a binary exponent, as neighbours on a
// large base elevation do, the bits' difference is the exact one in units of the last place;
// otherwise it is formed in 64-bit integers, exactly for exponents up to 11 apart and with
// the smaller operand cut to the larger one's last place beyond, and then cut to 24 bits.
// (32-bit conversions, as a 64-bit one issues on the f64 pipe.)
__device__ __forceinline__ bool bits_diff(uint64_t A, uint64_t B, float& out) {
    constexpr uint64_t mant = (1ull << 52) - 1;
    const uint32_t xa = (uint32_t)(A >> 52), xb = (uint32_t)(B >> 52);
    if (xa == xb && xa - 949u <= 200u) {
        const uint64_t D = A - B;
        const float d = fmaf(__uint2float_rz((uint32_t)(D >> 32)), 4294967296.0f, __uint2float_rz((uint32_t)D));
        out = d * __uint_as_float((xa - 948u) << 23);
        return true;
    }
    const uint64_t ma = (A & mant) | (xa ? mant + 1 : 0), mb = (B & mant) | (xb ? mant + 1 : 0);
    const int ea = xa ? (int)xa : 1, eb = xb ? (int)xb : 1, sh = ea - eb;
    const uint64_t D = sh <= 11 ? (ma << sh) - mb : ma - (sh < 64 ? mb >> sh : 0);
    if (D == 0) return false;
    const int lz = __clzll((long long)D);
    const int fe = (63 - lz) + (sh <= 11 ? eb : ea) - 1075 + 127;
    if (fe <= 0 || fe >= 255) return false;
    out = __uint_as_float(((uint32_t)fe << 23) | ((uint32_t)((D << lz) >> 40) & 0x7fffffu));
    return true;
}

// The steepest slot of site i's row [s0, s1) by those estimates (0xffffffff: no neighbour is
// lower), or kUndecided: negative or non-finite elevations, slopes out of range, near-ties.
// On a base elevation of 10^7 every row of a terrain comes here: at 1M sites the pairs and the
// scan take 65 us an iteration, 264 with those rows in f64, 51 on no base elevation.
constexpr uint32_t kUndecided = 0xfffffffeu;
[[maybe_unused]] static __device__ __noinline__ uint32_t steepest_bits(const uint32_t* col, const float* ilen, const double* elev,
                                               uint32_t i, uint32_t s0, uint32_t s1) {
    const uint64_t EI = (uint64_t)__double_as_longlong(elev[i]);
    if ((EI >> 52) >= 0x7ff) return kUndecided;
    float best = 0.0f, second = 0.0f;
    uint32_t slot = 0xffffffffu;
    bool sure = true;
#pragma unroll 1
    for (uint32_t b = s0; b < s1; b += 4) {                // four neighbours in flight
        uint64_t e[4];
        float f[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t s = min(b + k, s1 - 1);
            e[k] = (uint64_t)__double_as_longlong(elev[__ldg(&col[s])]);
            f[k] = __ldg(&ilen[s]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (b + k >= s1) break;
            if ((e[k] >> 52) >= 0x7ff) {
                sure = false;
            } else if (EI > e[k]) {                        // lower: the bits are monotone
                float d = 0.0f;
                sure &= bits_diff(EI, e[k], d);
                d *= f[k];
                sure &= d > 1e-30f && d < 1e30f;
                second = fmaxf(second, fminf(best, d));
                if (d > best) {
                    best = d;
                    slot = b + k;
                }
            }
        }
    }
    return sure && !(second > best * (1.0f - 7.62939453125e-06f)) ? slot : kUndecided;
}

}  // namespace fl
