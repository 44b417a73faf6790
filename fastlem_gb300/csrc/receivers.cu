// receivers.cu -- steepest-descent receivers (src/lem/stream_tree.rs:109-137).
//
// For site i (not an outlet) the reference takes, over its adjacency row in order,
// every neighbour j with e_i > e_j, the slope s_j = (e_i - e_j) / len_j in f64, and
// keeps the first j whose slope is strictly larger than the best so far (starting
// from 0.0).  The result must be bit-exact, but GB300 issues f64 at 1/64 of the f32
// rate and a correctly rounded f64 divide costs ~9 f64 operations, which made the
// straightforward scan FP64-bound.  Here every candidate's slope is first estimated in f32
// from the elevations' float pairs (slope.cuh), made in a pass before: three additions and a product with the slot's 1/len, within 2^-20 of the
// slope.  If the largest estimate exceeds every other by more than a factor
// (1 - 2^-17)^-1, its exact slope is strictly the largest, so it is the reference's
// receiver.  A row with a difference below 2^-24 of the elevation is estimated from the
// doubles' bits instead, and what is left (near-ties, non-finite or out-of-range values) is
// rescanned exactly as the reference does.
// The scan is bound by instruction issue and the gathers' latency.  Estimates from the two
// doubles' bit patterns (64-bit subtraction, exponent checks and two conversions a slot)
// took 710 us at 16M sites and 57 us at 1M; the scan now takes 515 us and 43 us, the pairs'
// own pass 51 us and 7 us.

#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "kernels.h"
#include "slope.cuh"

namespace fl {
namespace {

constexpr int kRowFast = 12;   // rows up to this length gather their elevations at once

// Site i's receiver and receiver distance.  s0 / s1 bound its row; dmax is the
// largest row length (up to kRowFast) among the warp's sites on the short-row path,
// so the unrolled gathers stop where the warp's rows do.
__device__ __forceinline__ void scan_site(uint32_t i, uint32_t s0, uint32_t s1, uint32_t dmax,
                                          const uint32_t* __restrict__ col,
                                          const double* __restrict__ len,
                                          const float* __restrict__ ilen,
                                          const double* __restrict__ elev,
                                          const float2* __restrict__ pair,
                                          uint32_t* __restrict__ next, double* __restrict__ rlen,
                                          bool* lake, bool* went_exact) {
    PairScan sc(pair[i]);
    const uint32_t deg = s1 - s0;
    if (deg <= (uint32_t)kRowFast) {
        // short rows: all neighbour elevations in flight at once
        uint32_t jj[kRowFast];
        float2 ej[kRowFast];
#pragma unroll
        for (int k = 0; k < kRowFast; ++k) {
            if ((uint32_t)k >= dmax) break;
            if ((uint32_t)k < deg) jj[k] = col[s0 + k];
        }
#pragma unroll
        for (int k = 0; k < kRowFast; ++k) {
            if ((uint32_t)k >= dmax) break;
            if ((uint32_t)k < deg) ej[k] = pair[jj[k]];
        }
#pragma unroll
        for (int k = 0; k < kRowFast; ++k) {
            if ((uint32_t)k >= dmax) break;
            if ((uint32_t)k < deg) sc.consider(s0 + k, ej[k], ilen[s0 + k]);
        }
    } else {
        for (uint32_t s = s0; s < s1; ++s) sc.consider(s, pair[col[s]], ilen[s]);
    }
    uint32_t best_slot = sc.slot;
    bool exact = !sc.decided();
    if (sc.close && !sc.exact) {
        best_slot = steepest_bits(col, ilen, elev, i, s0, s1);
        exact = best_slot == kUndecided;
    }
    if (exact) {
        *went_exact = true;
        const double ei = elev[i];
        double steepest = 0.0;
        best_slot = kNone;
        for (uint32_t s = s0; s < s1; ++s) {
            uint32_t j = col[s];
            double ej = elev[j];
            if (ei > ej) {
                double slope = __ddiv_rn(__dsub_rn(ei, ej), len[s]);
                if (slope > steepest) {
                    steepest = slope;
                    best_slot = s;
                }
            }
        }
    }
    if (best_slot == kNone) {
        next[i] = i;
        rlen[i] = 1.0;
        *lake = true;
        return;
    }
    // A duplicate of the receiver later in the row has the same slope and never wins
    // (strictly larger only; in the estimate it is a near-tie), so best_slot is the
    // receiver's first entry, the one has_edge reports.
    next[i] = col[best_slot];
    rlen[i] = len[best_slot];
}


__global__ void k_receivers(uint32_t n, const uint32_t* __restrict__ row,
                            const uint32_t* __restrict__ col, const double* __restrict__ len,
                            const float* __restrict__ ilen, const double* __restrict__ elev,
                            const float2* __restrict__ pair, const uint8_t* __restrict__ outlet, uint32_t* __restrict__ next,
                            double* __restrict__ rlen, int* __restrict__ flags,
                            const uint32_t* __restrict__ tid, const uint32_t* __restrict__ titer) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool lake = false, went_exact = false, scan = false;
    uint32_t s0 = 0, s1 = 0;
    // a converged packed terrain keeps its routed receivers
    if (i < n && !(tid && titer[tid[i]])) {
        if (outlet[i]) {
            next[i] = i;
            rlen[i] = 1.0;
        } else {
            s0 = row[i];
            s1 = row[i + 1];
            scan = true;
        }
    }
    const uint32_t deg = s1 - s0;
    const uint32_t dmax = __reduce_max_sync(0xffffffffu, deg <= (uint32_t)kRowFast ? deg : 0u);
    if (scan) scan_site(i, s0, s1, dmax, col, len, ilen, elev, pair, next, rlen, &lake, &went_exact);
    block_flag(flags, kHasLake, lake);
    if (__syncthreads_or(went_exact) && threadIdx.x == 0) atomicAdd(&flags[kExact], 1);
}

// 1/len per slot in f32 for the slope estimates, NaN where that is not a normal f32
// number (the row then takes the exact scan).
__global__ void k_inv_len(uint64_t nnz, const double* __restrict__ len, float* __restrict__ ilen) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < nnz;
         s += (uint64_t)gridDim.x * blockDim.x) {
        const float f = __double2float_rn(__ddiv_rn(1.0, len[s]));
        ilen[s] = (f >= FLT_MIN && f <= FLT_MAX) ? f : __int_as_float(0x7fc00000);
    }
}

}  // namespace

void launch_receivers(cudaStream_t st, uint32_t n, const uint32_t* row, const uint32_t* col,
                      const double* len, const float* ilen, const double* elev,
                      const float2* pair, const uint8_t* outlet, uint32_t* next, double* rlen, int* flags,
                      const uint32_t* tid, const uint32_t* titer) {
    k_receivers<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(
        n, row, col, len, ilen, elev, pair, outlet, next, rlen, flags, tid && titer ? tid : nullptr, titer);
}

void launch_inv_len(cudaStream_t st, uint64_t nnz, const double* len, float* ilen) {
    if (nnz == 0) return;
    const uint64_t blocks = std::min<uint64_t>((nnz + kThreads - 1) / kThreads, 152ull * 64);
    k_inv_len<<<(unsigned)blocks, kThreads, 0, st>>>(nnz, len, ilen);
}

}  // namespace fl
