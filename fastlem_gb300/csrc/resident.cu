// resident.cu -- solves of many iterations a kernel launch, for terrains whose working state
// fits the SMs' shared memory (src/lem/generator.rs:140-210, every iteration, bit-exact).
//
// The stage-by-stage pass (receivers.cu, solver.cu, basin.cu) spends an iteration of a
// small or middling terrain on launches and grid barriers: about 28 dependent launches and
// 60 barriers, 280 us at 1,000 sites and 450 us at 65,000, while the longest river is only
// 22 and 159 sites long.  Here a terrain is cut into contiguous ranges of its (Hilbert)
// memory order, one per block, one block per SM, and the block keeps its range's areas,
// response times, donor lists and pending counts in shared memory for the whole solve.
// What is left on an iteration's critical path is the longest river's chain of additions.
// An iteration takes 29 us at 1,000 sites, 60 us at 10,000 and 120 us at 65,000 (with slope
// limits 94 us at 10,000, 420 before): about 0.3 us a river site and direction.
//
//   receivers   every site's steepest neighbour, from the elevations' float pairs
//   barrier     (all receivers known; lakes, if any, are re-routed here)
//   link        per site its donors in reverse row order (the reference's addition order)
//   up          a lane starts at a leaf and walks down the river: it counts itself off its
//               receiver's donors, and the last donor to arrive adds the receiver's donors
//               and goes on; no lane waits for another.  The value of a donor in another
//               block is published in L2; a polling lane fetches it and walks on from there.
//   w           1 / (k sqrt(A)) * len where A or len changed, packed on dense warps
//   down        every lane waits for its site's receiver's response time in shared memory;
//               polling lanes wait for receivers in other blocks
//   elevation   from the site's and its basin outlet's response time; with slope limits
//               the limited elevations then go the same way down once more
//   barrier     (all elevations written; did any change?)
// A step of a lone walk costs its instructions at about six cycles each and two f64
// additions (64 cycles each, 104 with the way in and out of the f64 pipe): 300 to 400
// cycles at best, against some 1,000 for an earlier form with 64-bit pointers, separate
// list and flag words and a finished list for every block (39, 102 and 222 us an iteration).
//
// Values published across blocks use two slots per site, by the iteration's parity: a slot
// is set back to the pending marker one iteration later, when its readers have passed a
// barrier, so the publishing store is itself the flag (a time travels with its basin's root
// as one 16-byte value) and an iteration needs two barriers.  That a value has arrived says
// nothing about any other address -- the stores and loads are relaxed, and values go on
// through third blocks -- so whoever needs a root's time and elevation polls the root's own
// slots; in practice they are there at the first look.  Every wait is bounded.
//
// One launch takes many terrains (packed models): blocks take (terrain, part) slots in
// order, largest terrains first, and a terrain starts when its last part is taken.  Only
// the newest terrain can be partly taken, so the blocks that wait for its other parts wait
// for terrains that are running.  A launch ends by the clock (kResidentShareNs), and what a
// terrain cannot finish here -- long rivers, too many far donors -- the staged pass takes over
// (resident_solve in solver.cu).

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "slope.cuh"

namespace fl {
namespace {

constexpr uint32_t kEdges = kResidentEdges;     // donors in other blocks: one polling lane each
// A block's threads; its last warps poll for other blocks' values, the others walk.
constexpr uint32_t kT = 1024, kPollLanes = 128, kW = kT - kPollLanes;
constexpr uint64_t kPendingBits = 0x7ff4000000000000ull;   // a signalling NaN: never a result
constexpr uint64_t kQuietNan = 0x7ff8000000000000ull;
constexpr uint32_t kNoOutlet = 0x80000000u;     // root id bit: the root is not an outlet

__device__ __forceinline__ uint64_t ld_relaxed64(const double* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(double* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double from_bits(uint64_t b) { return __longlong_as_double((long long)b); }
// NaN payloads are not published (integer test: an f64 comparison takes 109 cycles)
__device__ __forceinline__ uint64_t published(double x) {
    const uint64_t b = bits(x);
    return (b << 1) > 0xffe0000000000000ull ? kQuietNan : b;
}
// 16 bytes as one access
__device__ __forceinline__ void ld_relaxed128(const void* p, uint64_t& lo, uint64_t& hi) {
    asm volatile("{.reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t;}" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_relaxed128(void* p, uint64_t lo, uint64_t hi) {
    asm volatile("{.reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t;}" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
// Exchange slots of site g (by iteration parity): area; response time with the basin's root,
// as one 16-byte value; limited elevation, or a root's elevation.
__device__ __forceinline__ double* area_slot(const ResidentArgs& a, uint32_t g, uint32_t par) { return a.xarea + 2ull * g + par; }
__device__ __forceinline__ double* time_slot(const ResidentArgs& a, uint32_t g, uint32_t par) { return a.xtime + 4ull * g + 2 * par; }
__device__ __forceinline__ double* elev_slot(const ResidentArgs& a, uint32_t g, uint32_t par) { return a.xelev + 2ull * g + par; }

__device__ __forceinline__ void raise(ResidentCtrl* c, int code) { atomicCAS(&c->error, 0, code); }

// What a block needs at hand about its terrain.
struct Group {
    unsigned long long* bar;   // four rotating barrier words
    ResidentCtrl* ctrl;
    uint32_t parts, part;
    uint32_t k;                // barriers passed
    bool ok;
    bool stop;                 // part 0 asked for the end of the launch at the last barrier
};

// Barrier over the terrain's blocks; returns whether any thread of any block set pred.  With
// part 0's ask every block finds gr.stop set.
// gr.ok turns false (for all threads) when the wait ran out or a block raised an error: that
// block does not arrive, and the others see the error while they wait.
__device__ __noinline__ bool group_barrier(Group& gr, bool pred, bool ask = false) {
    __shared__ int s_any, s_ok, s_stop;
    const int mine = __syncthreads_or(pred);
    if (gr.parts == 1) {
        gr.stop = __syncthreads_or(ask);
        return mine != 0;
    }
    if (threadIdx.x == 0) {
        unsigned long long* w = &gr.bar[gr.k & 3];
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(1ull | ((unsigned long long)(mine ? 1 : 0) << 32) | ((unsigned long long)ask << 48)) : "memory");
        uint32_t spins = 0;
        unsigned long long v;
        s_ok = 1;
        while ((uint32_t)(v = ld_acquire64(w)) < gr.parts) {
            if (++spins > kSpinLimit || ((spins & 63) == 0 && ld_acquire(&gr.ctrl->error) != 0)) {
                raise(gr.ctrl, kErrBarrier);
                s_ok = 0;
                break;
            }
        }
        s_any = (int)(v >> 32) & 0xffff;
        s_stop = (int)(v >> 48);
        // every block has arrived here, so has read the word of two barriers back; it is used
        // again two barriers on, which no block reaches before this one's next arrival
        if (gr.part == 0) atomicExch(&gr.bar[(gr.k + 2) & 3], 0ull);
    }
    __syncthreads();
    const bool any = s_any != 0;
    gr.ok = s_ok != 0;
    gr.stop = s_stop != 0;
    ++gr.k;
    __syncthreads();
    return any;
}

// When the block's waits of the iteration are to be given up (global_ns; shared).
__device__ __forceinline__ unsigned long long& wait_until() {
    __shared__ unsigned long long ns;
    return ns;
}
constexpr unsigned long long kNoTime = ~0ull;
// When the launch's share of time is over (shared).
__device__ __forceinline__ unsigned long long& share_end() {
    __shared__ unsigned long long ns;
    return ns;
}

__device__ __forceinline__ bool give_up(Group& gr, uint32_t& spins) {
    if (++spins > kSpinLimit) {
        raise(gr.ctrl, kErrWait);
        return true;
    }
    if ((spins & 255) != 0) return false;
    const unsigned long long until = wait_until();
    if (until != kNoTime && global_ns() > until) raise(gr.ctrl, kErrLate);
    return ld_acquire(&gr.ctrl->error) != 0;
}

// The reference's scan of site g's row: its slot, or kNone.
__device__ __noinline__ uint32_t steepest_exact(const uint32_t* row, const uint32_t* col, const double* len,
                                                const double* elev, uint32_t g) {
    const double ei = elev[g];
    double top = 0.0;
    uint32_t slot = kNone;
#pragma unroll 1
    for (uint32_t s = __ldg(&row[g]), e = __ldg(&row[g + 1]); s < e; ++s) {
        const double ej = elev[__ldg(&col[s])];
        if (ei > ej) {
            const double m = __ddiv_rn(__dsub_rn(ei, ej), __ldg(&len[s]));
            if (m > top) {
                top = m;
                slot = s;
            }
        }
    }
    return slot;
}

// The steepest-descent receiver of site g from the elevations' float pairs (slope.cuh):
// its slot, or kNone.
__device__ __forceinline__ uint32_t steepest(const ResidentArgs& a, uint32_t g) {
    const uint32_t s0 = __ldg(&a.row[g]), s1 = __ldg(&a.row[g + 1]);
    const float2 own = a.pair[g];
    PairScan sc(own);
#pragma unroll 1
    for (uint32_t b = s0; b < s1; b += 4) {
        float2 e[4];
        float f[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t s = min(b + k, s1 - 1);
            e[k] = a.pair[__ldg(&a.col[s])];
            f[k] = __ldg(&a.ilen[s]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (b + k < s1) sc.consider(b + k, e[k], f[k]);
    }
    if (sc.decided()) return sc.slot;
    if (sc.close && !sc.exact) {
        const uint32_t slot = steepest_bits(a.col, a.ilen, a.elev, g, s0, s1);
        if (slot != kUndecided) return slot;
    }
    return steepest_exact(a.row, a.col, a.len, a.elev, g);
}

__device__ __forceinline__ double edge_or_one(const ResidentArgs& a, uint32_t i, uint32_t j) {
    const uint32_t s0 = __ldg(&a.row[i]), e = __ldg(&a.row[i + 1]);
#pragma unroll 1
    for (uint32_t s = s0; s < e; s += 4) {               // four columns in flight
        uint32_t c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = __ldg(&a.col[min(s + k, e - 1)]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (s + k < e && c[k] == j) return __ldg(&a.len[s + k]);
    }
    return 1.0;
}

// Lake re-routing (stream_tree.rs:139-243) of the terrain's receivers: labels by pointer
// jumping, the first processed entry of every lake, path reversal (as solver.cu's kernels).
__device__ __noinline__ void reroute_lakes(const ResidentArgs& a, Group& gr, uint32_t lo, uint32_t S) {
#pragma unroll 1
    for (uint32_t v = threadIdx.x; v < S; v += blockDim.x) {
        a.lab[lo + v] = __ldcg(&a.next[lo + v]);
        a.best[lo + v] = kNoKey;
    }
    group_barrier(gr, false);
    uint32_t *cur = a.lab, *out = a.lab2;
    for (uint32_t round = 0; gr.ok; ++round) {
        bool moved = false;
#pragma unroll 1
        for (uint32_t v = threadIdx.x; v < S; v += blockDim.x) {
            const uint32_t l = __ldcg(&cur[lo + v]);
            const uint32_t ll = __ldcg(&cur[l]);
            out[lo + v] = ll;
            moved |= ll != l;
        }
        const bool more = group_barrier(gr, moved);
        uint32_t* t = cur;
        cur = out;
        out = t;
        if (!more) break;
        if (round >= 64) {                               // a receiver cycle
            raise(gr.ctrl, kErrForest);
            gr.ok = false;
        }
    }
    if (!gr.ok) return;
#pragma unroll 1
    for (uint32_t v = threadIdx.x; v < S; v += blockDim.x) {
        const uint32_t g = lo + v, r = __ldg(&a.rank[g]);
        if (r == kNone) continue;
        const uint32_t own = __ldcg(&cur[g]);
        const uint32_t s0 = __ldg(&a.row[g]), s1 = __ldg(&a.row[g + 1]);
        for (uint32_t s = s0; s < s1; ++s) {
            const uint32_t L = __ldcg(&cur[__ldg(&a.col[s])]);
            if (__ldg(&a.outlet[L]) || L == own) continue;
            const unsigned long long key = ((unsigned long long)r << 32) | (s - s0);
            if (key < __ldcg(&a.best[L])) atomicMin(&a.best[L], key);
        }
    }
    group_barrier(gr, false);
    if (!gr.ok) return;
    bool cyclic = false;
#pragma unroll 1
    for (uint32_t v = threadIdx.x; v < S; v += blockDim.x) {
        const unsigned long long key = __ldcg(&a.best[lo + v]);
        if (key == kNoKey) continue;
        uint32_t nk = __ldg(&a.sor[key >> 32]);
        uint32_t k = __ldg(&a.col[__ldg(&a.row[nk]) + (uint32_t)key]);
        for (uint32_t steps = 0;; ++steps) {
            if (steps > a.n) {
                raise(gr.ctrl, kErrForest);
                cyclic = true;
                break;
            }
            const uint32_t nx = __ldcg(&a.next[k]);
            a.next[k] = nk;
            a.rlen[k] = edge_or_one(a, k, nk);
            if (nx == k) break;
            nk = k;
            k = nx;
        }
    }
    if (__syncthreads_or(cyclic)) gr.ok = false;
    else group_barrier(gr, false);
}

// ---- shared memory, by 32-bit address (accesses keep their order) ----
__device__ __forceinline__ uint64_t lds64(uint32_t p) {
    uint64_t v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ldsd(uint32_t p) { return from_bits(lds64(p)); }
__device__ __forceinline__ uint32_t lds32(uint32_t p) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t p) {
    uint16_t v;
    asm volatile("ld.shared.b16 %0, [%1];" : "=h"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void sts64(uint32_t p, uint64_t v) {
    asm volatile("st.shared.b64 [%0], %1;" ::"r"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void stsd(uint32_t p, double v) { sts64(p, bits(v)); }
__device__ __forceinline__ void sts32(uint32_t p, uint32_t v) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t p, uint32_t v) {
    asm volatile("st.shared.b16 [%0], %1;" ::"r"(p), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ uint32_t atom_add(uint32_t p, uint32_t x) {
    uint32_t v;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(v) : "r"(p), "r"(x) : "memory");
    return v;
}
// ... that orders this thread's accesses before and after it for the block
__device__ __forceinline__ uint32_t atom_add_ordered(uint32_t p, uint32_t x) {
    uint32_t v;
    asm volatile("atom.acq_rel.cta.shared.add.u32 %0, [%1], %2;" : "=r"(v) : "r"(p), "r"(x) : "memory");
    return v;
}
// 16 bytes as one access
__device__ __forceinline__ void sts128(uint32_t p, uint64_t lo, uint64_t hi) {
    asm volatile("{.reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.cta.shared.b128 [%0], t;}" ::"r"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ void lds128(uint32_t p, uint64_t& lo, uint64_t& hi) {
    asm volatile("{.reg .b128 t; ld.relaxed.cta.shared.b128 t, [%2]; mov.b128 {%0, %1}, t;}" : "=l"(lo), "=l"(hi) : "r"(p) : "memory");
}

// Shared memory of a block for up to `cap` sites (resident_smem): 24 bytes a site (32 with
// slope limits), so that packed models keep as many terrains in flight as possible.  A site
// is a 16-byte record and a word; donors and receivers are 16-bit record numbers.  On a lone
// walk every instruction costs about six cycles: one access brings a record, and one atomic
// the count, the kind and the receiver.
enum Field : uint32_t {
    fVal = 0,      // f64: area, then w, response time, (free, then limited) elevation
    fDon = 8,      // u16 x 4: donors in addition order (way up)
    fRoot = 8,     // u32: the basin's root (way down)
    fState = 12    // u32: 0, 1 with the response time, 2 with the limited elevation
};
// word: donors still to arrive, kind bits, the receiver's record number
constexpr uint32_t kCount = 0xffu;
constexpr uint32_t kRoot = 0x100u;       // its own receiver
constexpr uint32_t kFar = 0x200u;        // its receiver is in another block
constexpr uint32_t kFarDonor = 0x400u;   // it has a donor in another block
constexpr uint32_t kLong = 0x800u;       // more than four donors
constexpr uint32_t kMany = 0x1000u;      // three or four donors
constexpr uint32_t kPlain = 0xffffu & ~kFarDonor;   // these bits are 1: last of one or two
                                                    // donors, receiver in the block
constexpr int kParentShift = 16;
struct Block {
    uint32_t at;        // records: sites, then far donors (their areas), then the -0.0 that
                        // stands for "no donor" (x + -0.0 is x whatever x is)
    uint32_t cap, none; // none: that record's number
    uint32_t lim, words, far_id, far_to, out, order, list;
    __device__ __forceinline__ uint32_t rec(uint32_t v) const { return at + v * 16; }
    __device__ __forceinline__ uint32_t word(uint32_t v) const { return words + v * 4; }
};
template <bool kSlope>
__device__ __forceinline__ Block carve(uint32_t cap) {
    extern __shared__ __align__(128) unsigned char sm[];
    Block b;
    b.at = ((uint32_t)__cvta_generic_to_shared(sm) + 15u) & ~15u;
    b.cap = cap;
    b.none = cap + kEdges;
    b.lim = b.rec(b.none + 1);                   // f64 [cap] with slope limits: tan * len
    b.words = b.lim + (kSlope ? 8 * cap : 0);    // u32 [cap]
    b.far_id = b.words + 4 * cap;                // u32 [kEdges] a far donor's site
    b.far_to = b.far_id + 4 * kEdges;            // u16 [kEdges] the record it drains to
    b.out = b.far_to + 2 * kEdges;               // u16 [kEdges] records with a far receiver
    b.order = b.out + 2 * kEdges;                // u16 [cap] sites in order of finishing, leaves first
    b.list = b.order + 2 * cap;                  // u16 [cap]
    return b;
}

// The pollers' loop over this lane's entries of a far list of n: src(e) is where entry e's
// value (kPair: and its root, 16 bytes) is published, ready(e, value, root) takes it, walk()
// does what that started.
template <bool kPair, class Src, class Ready, class Walk>
__device__ __forceinline__ bool poll_far(Group& gr, uint32_t n, Src src, Ready ready, Walk walk) {
    constexpr uint32_t kMine = kEdges / kPollLanes;
    const uint32_t me = (threadIdx.x & 31u) * (kPollLanes / 32) + (threadIdx.x - kW) / 32;   // over the warps
    const uint32_t rounds = (n + kPollLanes - 1) / kPollLanes;
    bool lost = false;
    // all of a lane's entries at once: none waits for another
    if (n) {
        uint32_t left = 0, spins = 0;
        const double* at[kMine];
#pragma unroll
        for (uint32_t q = 0; q < kMine; ++q) {
            const uint32_t e = me + q * kPollLanes;
            at[q] = nullptr;
            if (e < n) {
                left |= 1u << q;
                at[q] = src(e);
            }
        }
        while (__any_sync(0xffffffffu, left != 0)) {
            uint64_t b[kMine], r[kMine];
#pragma unroll
            for (uint32_t q = 0; q < kMine; ++q) {
                b[q] = kPendingBits;
                r[q] = 0;
                if ((left >> q) & 1u) {
                    if (kPair) ld_relaxed128(at[q], b[q], r[q]);
                    else b[q] = ld_relaxed64(at[q]);
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < kMine; ++q)
                if (q < rounds && __any_sync(0xffffffffu, b[q] != kPendingBits)) {
                    if (b[q] != kPendingBits) {
                        left &= ~(1u << q);
                        ready(me + q * kPollLanes, b[q], r[q]);
                    }
                    walk();
                }
            if (left && give_up(gr, spins)) {
                left = 0;
                lost = true;
            }
        }
    }
    return lost;
}

// Appends of the lanes with pred set, one atomic per warp (all lanes call it).
__device__ __forceinline__ uint32_t warp_slots(uint32_t* counter, bool pred) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    const int lane = threadIdx.x & 31;
    uint32_t at = 0;
    if (lane == 0 && m) at = atomicAdd(counter, (uint32_t)__popc(m));
    return __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// x plus the areas of all donors of site v, in reverse row order: for sites with more donors
// than a record holds.
template <bool kSlope>
__device__ __noinline__ double add_long(const ResidentArgs& a, uint32_t lo, uint32_t S, uint32_t nfar,
                                        uint32_t v, double x) {
    const Block bk = carve<kSlope>(a.cap);
    const uint32_t g = lo + v, s0 = __ldg(&a.row[g]);
#pragma unroll 1
    for (uint32_t s = __ldg(&a.row[g + 1]); s-- > s0;) {
        const uint32_t j = __ldg(&a.col[s]), d = j - lo;
        if (d < S) {
            const uint32_t w = lds32(bk.word(d));
            if (!(w & (kRoot | kFar)) && (w >> kParentShift) == v) x = __dadd_rn(x, ldsd(bk.rec(d)));
        } else {
#pragma unroll 1
            for (uint32_t e = 0; e < nfar; ++e)
                if (lds32(bk.far_id + 4 * e) == j && lds16(bk.far_to + 2 * e) == v)
                    x = __dadd_rn(x, ldsd(bk.rec(bk.cap + e)));
        }
    }
    return x;
}

// The limited elevation of site g where the product cannot stand in for the quotient.
__device__ __noinline__ double limit_exact(const double* tanms, const double* rlen, uint32_t g, double own,
                                           double x, double d) {
    const double tn = tanms[g], dist = rlen[g];
    return !isnan(tn) && __ddiv_rn(d, dist) > tn ? __dadd_rn(x, __dmul_rn(tn, dist)) : own;
}

// The way down over the block's sites, each in the hands of one lane that waits for its
// receiver's value: kTimes response times (a record's value is w before), else limited
// elevations (the free elevation before).  Roots are settled already.  In a block of more
// sites than walking lanes a warp takes 32 sites at a time, last finished first: a receiver
// finishes after its donors, and so does the list entry, so of all unsettled sites (of all
// blocks) the one that finished last has its receiver's value and a lane.
template <bool kSlope, bool kTimes>
__device__ __forceinline__ bool settle_down(const ResidentArgs& a, Group& gr, const Block& bk, uint32_t lo,
                                            uint32_t S, uint32_t par, uint32_t nout) {
    constexpr uint32_t kReady = kTimes ? 1 : 2;
    bool lost = false;
    // site v (its word w, its own value) gets its value from its receiver's value x and root
    auto settle = [&](uint32_t v, uint32_t w, double x, double own, uint32_t root) {
        if (kTimes) {
            x = __dadd_rn(x, own);                       // never -0.0: the root's is not
        } else {
            // e <= e_receiver + tan * len.  The reference compares (e - e_receiver) / len
            // with tan; a difference more than 8 ulps from the rounded product is on the
            // same side of it as the rounded quotient is of tan.
            const double rise = ldsd(bk.lim + 8 * v), d = __dsub_rn(own, x), most = __dadd_rn(x, rise);
            const int64_t gap = (int64_t)(bits(d) - bits(rise));
            if ((bits(rise) >> 63) == 0 && (bits(d) << 1) < 0xffe0000000000000ull && (gap > 8 || gap < -8))
                x = (int64_t)bits(d) > (int64_t)bits(rise) ? most : own;
            else                                         // no limit, or divide
                x = (root & kNoOutlet) ? own : limit_exact(a.tanms, a.rlen, lo + v, own, x, d);
        }
        sts128(bk.rec(v), bits(x), (uint64_t)kReady << 32 | root);
        if (w & kFarDonor) {
            if (kTimes) st_relaxed128(time_slot(a, lo + v, par), published(x), root);
            else st_relaxed64(elev_slot(a, lo + v, par), published(x));
        }
    };
    if (threadIdx.x < kW) {
        uint32_t spins = 0;
#pragma unroll 1
        for (uint32_t i = threadIdx.x; i < ((S + 31u) & ~31u) && !lost; i += kW) {
            const bool mine = i < S;
            const uint32_t v = S <= kW ? i : mine ? lds16(bk.order + 2 * (S - 1 - i)) : 0u;
            uint32_t w = kRoot;
            double own = 0.0;
            if (mine) {
                w = lds32(bk.word(v));
                own = ldsd(bk.rec(v));
            }
            const uint32_t p = bk.rec(w >> kParentShift);
            bool todo = !(w & (kRoot | kFar));
            while (__any_sync(0xffffffffu, todo)) {
                if (todo) {
                    uint64_t x, rs;
                    lds128(p, x, rs);
                    if ((uint32_t)(rs >> 32) == kReady) {
                        settle(v, w, from_bits(x), own, (uint32_t)rs);
                        todo = false;
                    } else if (give_up(gr, spins)) {
                        todo = false;
                        lost = true;
                    }
                }
            }
            lost = __any_sync(0xffffffffu, lost);
        }
    } else {
        lost = poll_far<kTimes>(
            gr, nout,
            [&](uint32_t j) -> const double* {
                const uint32_t p = __ldcg(&a.next[lo + lds16(bk.out + 2 * j)]);
                return kTimes ? time_slot(a, p, par) : elev_slot(a, p, par);
            },
            [&](uint32_t j, uint64_t b, uint64_t root) {
                const uint32_t v = lds16(bk.out + 2 * j);
                settle(v, lds32(bk.word(v)), from_bits(b), ldsd(bk.rec(v)),
                       kTimes ? (uint32_t)root : lds32(bk.rec(v) + fRoot));
            },
            []() {});
    }
    return __syncthreads_or(lost) == 0;
}

// One terrain's iterations up to its fixed point, its limit or the end of the launch's share.
template <bool kSlope>
__device__ void solve_terrain(const ResidentArgs& a, const ResidentTerrain& tr, Group& gr) {
    __shared__ uint32_t s_fin, s_far, s_out, s_list;
    __shared__ unsigned long long s_since;    // part 0: when the iteration started
    const uint32_t tid = threadIdx.x;
    const uint32_t each = tr.n / tr.parts, rest = tr.n % tr.parts;
    const uint32_t lo = tr.lo + gr.part * each + min(gr.part, rest);
    const uint32_t S = each + (gr.part < rest ? 1u : 0u);
    const Block bk = carve<kSlope>(a.cap);
    ResidentCtrl* ctrl = gr.ctrl;

    uint32_t it = ctrl->iters;
    bool valid = it > 0;                      // w, wa, wl hold the previous iteration's
#pragma unroll 1
    for (uint32_t v = tid; v < S; v += kT) {
        const uint32_t g = lo + v;
        for (uint32_t par = 0; par < 2; ++par) {
            st_relaxed64(area_slot(a, g, par), kPendingBits);
            st_relaxed128(time_slot(a, g, par), kPendingBits, 0);
            st_relaxed64(elev_slot(a, g, par), kPendingBits);
        }
        sts32(bk.word(v), 0);
    }
    if (tid == 0) stsd(bk.rec(bk.none), -0.0);
    group_barrier(gr, false);

    const bool keeps_time = gr.part == 0 && tid == 0;
    uint32_t slow = keeps_time ? ctrl->slow : 0;   // the time rule's points
    if (keeps_time) s_since = global_ns();
    while (gr.ok) {
        const uint32_t par = it & 1u;
        // ---- receivers
        bool lake = false;
        if (tid == 0) s_fin = s_far = s_out = s_list = 0;
        auto note = [&](uint32_t v, uint32_t p) {
            const uint32_t g = lo + v;
            sts32(bk.word(v), p == g ? kRoot : p - lo < S ? (p - lo) << kParentShift : kFar);
        };
#pragma unroll 1
        for (uint32_t v = tid; v < S; v += kT) {
            const uint32_t g = lo + v;
            // last iteration's published values have been read: their slots are free
            const uint32_t was = lds32(bk.word(v));
            if (was & kFar) st_relaxed64(area_slot(a, g, par ^ 1u), kPendingBits);
            if (was & (kFarDonor | kRoot)) {
                st_relaxed128(time_slot(a, g, par ^ 1u), kPendingBits, 0);
                if (kSlope || (was & kRoot)) st_relaxed64(elev_slot(a, g, par ^ 1u), kPendingBits);
            }
            uint32_t slot = kNone;
            if (!__ldg(&a.outlet[g])) {
                slot = steepest(a, g);
                lake |= slot == kNone;
            }
            const uint32_t p = slot == kNone ? g : __ldg(&a.col[slot]);
            a.next[g] = p;
            a.rlen[g] = slot == kNone ? 1.0 : __ldg(&a.len[slot]);
            note(v, p);
            stsd(bk.rec(v), __ldg(&a.area[g]));
        }
        const bool lakes = group_barrier(gr, lake);
        if (!gr.ok) break;
        if (lakes) {
            if (!a.rank_ready) {              // the same verdict in every block
                if (gr.part == 0 && tid == 0) ctrl->need_rank = 1;
                break;
            }
            reroute_lakes(a, gr, lo, S);
            if (!gr.ok) break;
#pragma unroll 1
            for (uint32_t v = tid; v < S; v += kT) note(v, __ldcg(&a.next[lo + v]));
            __syncthreads();
        }
        // ---- link
#pragma unroll 1
        for (uint32_t base = 0; base < S; base += kT) {
            const uint32_t v = base + tid;
            bool leaf = false, out = false;
            if (v < S) {
                const uint32_t g = lo + v;
                const uint32_t s0 = __ldg(&a.row[g]), s1 = __ldg(&a.row[g + 1]);
                uint32_t cnt = 0, kind = 0;
                uint64_t dn = (uint64_t)bk.none * 0x0001000100010001ull;
#pragma unroll 1
                for (uint32_t hi = s1; hi > s0; hi = hi > s0 + 4 ? hi - 4 : s0) {
                    uint32_t j[4];
                    bool don[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) j[k] = __ldg(&a.col[max(hi, s0 + 1 + k) - 1 - k]);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t d = j[k] - lo;
                        don[k] = false;
                        if (hi >= s0 + 1 + k) {
                            if (d < S) {
                                const uint32_t w = lds32(bk.word(d));
                                don[k] = !(w & (kRoot | kFar)) && (w >> kParentShift) == v;
                            } else {
                                don[k] = __ldcg(&a.next[j[k]]) == g;
                            }
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (don[k]) {
                            uint32_t d = j[k] - lo;
                            if (d >= S) {
                                kind |= kFarDonor;
                                const uint32_t e = atomicAdd(&s_far, 1u);
                                if (e < kEdges) {              // else reported below
                                    sts32(bk.far_id + 4 * e, j[k]);
                                    sts16(bk.far_to + 2 * e, v);
                                }
                                d = bk.cap + e;
                            }
                            if (cnt < 4) dn = (dn & ~(0xffffull << (16 * cnt))) | ((uint64_t)(d & 0xffffu) << (16 * cnt));
                            ++cnt;
                        }
                }
                if (cnt > 2) kind |= cnt > 4 ? kLong : kMany;
                const uint32_t w = lds32(bk.word(v)) | kind | cnt;
                sts32(bk.word(v), w);
                sts64(bk.rec(v) + fDon, dn);
                leaf = cnt == 0;
                out = (w & kFar) != 0;
            }
            const uint32_t at = warp_slots(&s_fin, leaf);
            if (leaf) sts16(bk.order + 2 * at, v);
            if (__any_sync(0xffffffffu, out)) {
                const uint32_t ot = warp_slots(&s_out, out);
                if (out && ot < kEdges) sts16(bk.out + 2 * ot, v);
            }
        }
        // the first iteration's rivers are as long as any: past the time for which the rule
        // ends a solve at once, it is dropped on the way (all its waits are behind this point)
        if (tid == 0) wait_until() = a.slow_ns && it == 0 ? global_ns() + 2 * a.slow_ns : kNoTime;
        __syncthreads();
        const uint32_t nleaf = s_fin, nfar = s_far, nout = s_out;
        __syncthreads();                      // ... before the walks count on
        if (nfar > kEdges || nout > kEdges) { // the other blocks see it at their next wait
            if (tid == 0) raise(ctrl, kErrCapacity);
            gr.ok = false;
            break;
        }
        // ---- up: p is the receiver of a site that has just become final (have); count it
        // off and go on if it was the last
        const bool many = S > kW;             // settle_down needs the order
        const uint32_t fin = (uint32_t)__cvta_generic_to_shared(&s_fin);
        bool have = false, lost = false;
        uint32_t p = 0;
        auto leave = [&](uint32_t v, uint32_t w) {        // v is final, w its word
            have = !(w & (kRoot | kFar));
            p = w >> kParentShift;
            if (w & kFar) st_relaxed64(area_slot(a, lo + v, par), published(ldsd(bk.rec(v))));
        };
        auto step = [&]() {
            uint64_t xb, dd;
            const uint32_t w = atom_add_ordered(bk.word(p), ~0u);
            const uint32_t r = bk.rec(p);
            lds128(r, xb, dd);
            double x = from_bits(xb);
            uint32_t at = 0;
            if (many && (w & kCount) == 1u) at = atom_add(fin, 1u);
            if ((w & kPlain) == 1u) {
                const double y0 = ldsd(bk.rec((uint32_t)dd & 0xffffu)), y1 = ldsd(bk.rec((uint32_t)dd >> 16));
                x = __dadd_rn(__dadd_rn(x, y0), y1);
                stsd(r, x);
                if (many) sts16(bk.order + 2 * at, p);
                p = w >> kParentShift;
            } else if ((w & kCount) == 1u) {
                if (w & kLong) {
                    x = add_long<kSlope>(a, lo, S, nfar, p, x);
                } else {
                    const double y0 = ldsd(bk.rec((uint32_t)dd & 0xffffu)), y1 = ldsd(bk.rec((uint32_t)dd >> 16)),
                                 y2 = ldsd(bk.rec((uint32_t)(dd >> 32) & 0xffffu)),
                                 y3 = ldsd(bk.rec((uint32_t)(dd >> 48)));
                    x = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(x, y0), y1), y2), y3);
                }
                stsd(r, x);
                if (many) sts16(bk.order + 2 * at, p);
                leave(p, w);
            } else {
                have = false;
            }
        };
        if (tid < kW) {
#pragma unroll 1
            for (uint32_t i = tid;;) {
                if (!have && i < nleaf) {
                    const uint32_t v = lds16(bk.order + 2 * i);
                    leave(v, lds32(bk.word(v)));
                    i += kW;
                }
                if (!__any_sync(0xffffffffu, have || i < nleaf)) break;
                if (have) step();
            }
        } else {
            lost = poll_far<false>(
                gr, nfar, [&](uint32_t e) -> const double* { return area_slot(a, lds32(bk.far_id + 4 * e), par); },
                [&](uint32_t e, uint64_t b, uint64_t) {
                    sts64(bk.rec(bk.cap + e), b);
                    p = lds16(bk.far_to + 2 * e);
                    have = true;
                },
                [&]() {
                    while (__any_sync(0xffffffffu, have))
                        if (have) step();
                });
        }
        if (__syncthreads_or(lost)) {
            gr.ok = false;
            break;
        }
        // ---- w, where an operand changed since the previous iteration
        bool cyclic = false;
#pragma unroll 1
        for (uint32_t base = 0; base < S; base += kT) {
            const uint32_t u = base + tid;
            bool need = false;
            if (u < S) {
                const uint32_t g = lo + u;
                need = !valid || lds64(bk.rec(u)) != bits(__ldcg(&a.wa[g])) ||
                       bits(__ldcg(&a.rlen[g])) != bits(__ldcg(&a.wl[g]));
                cyclic |= (lds32(bk.word(u)) & kCount) != 0;    // never reached: not a forest
            }
            const uint32_t at = warp_slots(&s_list, need);
            if (need) sts16(bk.list + 2 * at, u);
        }
        if (__syncthreads_or(cyclic)) {
            if (tid == 0) raise(ctrl, kErrForest);
            gr.ok = false;
            break;
        }
        const uint32_t nlist = s_list;
#pragma unroll 1
        for (uint32_t i = tid; i < nlist; i += kT) {
            const uint32_t u = lds16(bk.list + 2 * i), g = lo + u;
            const double A = ldsd(bk.rec(u)), l = __ldcg(&a.rlen[g]);
            const double cel = __dmul_rn(__ldg(&a.k[g]), __dsqrt_rn(A));
            a.w[g] = __dmul_rn(__ddiv_rn(1.0, cel), l);
            a.wa[g] = A;
            a.wl[g] = l;
        }
        valid = true;
        __syncthreads();
        // ---- down: the roots, then response times
        bool changed = false;
#pragma unroll 1
        for (uint32_t u = tid; u < S; u += kT) {
            const uint32_t g = lo + u, r = bk.rec(u), w = lds32(bk.word(u));
            const double wv = __ldcg(&a.w[g]);
            if (!(w & kRoot)) {
                sts128(r, bits(wv), 0);
                continue;
            }
            const double t = plus_zero(plus_zero(wv));
            const bool out = __ldg(&a.outlet[g]) != 0;
            double ne = __ldcg(&a.elev[g]);
            if (out) {
                const double old_e = ne, dt = __dsub_rn(t, t);
                ne = __dadd_rn(old_e, __dmul_rn(__ldg(&a.u[g]), dt > 0.0 ? dt : 0.0));
                if (kSlope) {
                    const double tn = __ldg(&a.tanms[g]), dist = __ldcg(&a.rlen[g]);
                    if (!isnan(tn) && __ddiv_rn(__dsub_rn(ne, old_e), dist) > tn)
                        ne = __dadd_rn(old_e, __dmul_rn(tn, dist));
                }
                changed |= ne != old_e;
                a.elev[g] = ne;
                a.pair[g] = float_pair(ne);
            }
            const uint32_t root = out ? g : g | kNoOutlet;
            sts128(r, bits(t), (uint64_t)1 << 32 | root);
            // for its donors in other blocks and for its basin's sites, wherever they are (an
            // elevation is the result of an addition, so never the pending marker)
            st_relaxed128(time_slot(a, g, par), published(t), root);
            st_relaxed64(elev_slot(a, g, par), bits(ne));
        }
        __syncthreads();
        if (!settle_down<kSlope, true>(a, gr, bk, lo, S, par, nout)) {
            gr.ok = false;
            break;
        }
        // ---- elevations
        uint32_t spins = 0;
#pragma unroll 1
        for (uint32_t u = tid; u < S; u += kT) {
            const uint32_t g = lo + u, rec = bk.rec(u), r = lds32(rec + fRoot);
            const bool is_root = (r & ~kNoOutlet) == g;
            double ne = 0.0;
            if (!(r & kNoOutlet) && !is_root) {
                uint64_t tb, eb, root;
                while (true) {
                    ld_relaxed128(time_slot(a, r, par), tb, root);
                    eb = ld_relaxed64(elev_slot(a, r, par));
                    if (tb != kPendingBits && eb != kPendingBits) break;
                    if (give_up(gr, spins)) {
                        lost = true;
                        break;
                    }
                }
                if (lost) break;
                const double to = from_bits(tb), eo = from_bits(eb);
                const double dt = __dsub_rn(ldsd(rec), to);
                ne = __dadd_rn(eo, __dmul_rn(__ldg(&a.u[g]), dt > 0.0 ? dt : 0.0));
                if (!kSlope) {
                    changed |= ne != __ldcg(&a.elev[g]);
                    a.elev[g] = ne;
                    a.pair[g] = float_pair(ne);
                }
            } else if (kSlope) {
                ne = __ldcg(&a.elev[g]);
            }
            if (kSlope) {
                // tan * len, or a negative number where there is no limit or the product
                // cannot stand in for the quotient
                const double tn = __ldg(&a.tanms[g]), dist = __ldcg(&a.rlen[g]), rise = __dmul_rn(tn, dist);
                stsd(bk.lim + 8 * u, tn > 1e-200 && dist > 0.0 && rise > 1e-200 && rise < 1e200 && !(r & kNoOutlet) ? rise : -1.0);
                sts128(rec, bits(ne), (uint64_t)(is_root ? 2 : 1) << 32 | r);
            }
        }
        if (__syncthreads_or(lost)) {
            gr.ok = false;
            break;
        }
        if (kSlope) {
            if (!settle_down<kSlope, false>(a, gr, bk, lo, S, par, nout)) {
                gr.ok = false;
                break;
            }
#pragma unroll 1
            for (uint32_t u = tid; u < S; u += kT) {
                const uint32_t r = lds32(bk.rec(u) + fRoot), g = lo + u;
                if ((r & kNoOutlet) || r == g) continue;
                const double ne = ldsd(bk.rec(u));
                changed |= ne != __ldcg(&a.elev[g]);
                a.elev[g] = ne;
                a.pair[g] = float_pair(ne);
            }
        }
        ++it;
        bool ask = false;
        if (keeps_time) {
            const unsigned long long now = global_ns(), took = now - s_since;
            if (a.slow_ns) slow = took <= a.slow_ns ? 0 : slow + (took > 2 * a.slow_ns ? kSlowPoints : 1);
            ask = slow >= kSlowPoints || now > share_end();
            s_since = now;
        }
        const bool more = group_barrier(gr, changed, ask);
        if (!gr.ok) break;
        if (!more || it >= a.limit) {
            if (keeps_time) ctrl->done = 1;
            break;
        }
        if (gr.stop) {                        // long rivers: the staged pass goes on
            if (keeps_time) ctrl->left = slow >= kSlowPoints;
            break;
        }
    }
    if (keeps_time) {
        ctrl->iters = it;
        ctrl->slow = slow;
    }
}

template <bool kSlope>
__global__ void __launch_bounds__(kT, 1) k_resident(const __grid_constant__ ResidentArgs a) {
    __shared__ uint32_t s_slot;
    __shared__ bool s_go;
    if (threadIdx.x == 0) {
        const unsigned long long now = global_ns(), first = atomicCAS(a.started, 0ull, now);
        share_end() = (first ? first : now) + a.share_ns;
    }
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_slot = atomicAdd(a.ticket, 1u);
        __syncthreads();
        const uint32_t slot = s_slot;
        if (slot >= a.slots) return;
        const uint32_t t = a.slot_terrain[slot];
        const ResidentTerrain tr = a.terrains[t];
        unsigned long long* const words = a.bars + (unsigned long long)kResidentWords * t;
        Group gr{words, a.ctrl + t, tr.parts, slot - tr.slot0, 0, true, false};
        if (gr.ctrl->done) continue;          // settled in an earlier launch
        // its first block decides for all of them whether there is time to start
        if (threadIdx.x == 0) {
            const unsigned long long mine = global_ns() > share_end() ? 2 : 1, first = atomicCAS(&words[4], 0ull, mine);
            s_go = (first ? first : mine) == 1;
        }
        __syncthreads();
        if (!s_go) continue;
        solve_terrain<kSlope>(a, tr, gr);
    }
}

// What a row tells of its site's donors: bad[0] unless every edge of the graph appears exactly
// once in either end's row, no site is its own neighbour and no row is longer than the donor
// count can hold (the resident solve's graphs); bad[1] unless every site is named exactly once
// in each short row (kTileRow) of a site that it names (the tiles', which leave longer rows to
// the rounds).  Rows longer than kResidentMaxRow are taken by their block together.
__global__ void __launch_bounds__(kThreads) k_check_rows(uint32_t n, const uint32_t* __restrict__ row,
                                                         const uint32_t* __restrict__ col, int* __restrict__ bad) {
    __shared__ uint32_t s_long[kThreads], s_count;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool odd = false, unlike = false;
    // how often site v's row [r0, r1) names u
    auto times = [&](uint32_t r0, uint32_t r1, uint32_t u) {
        uint32_t c = 0;
        for (uint32_t q = r0; q < r1; ++q) c += col[q] == u;
        return c;
    };
    if (i < n) {
        const uint32_t s0 = row[i], s1 = row[i + 1];
        const bool is_long = s1 - s0 > kResidentMaxRow;
        odd = is_long;
        if (is_long) s_long[atomicAdd(&s_count, 1u)] = i;
        for (uint32_t s = s0; s < s1 && !is_long && !unlike; ++s) {
            const uint32_t j = col[s], r0 = row[j], r1 = row[j + 1];
            if (j == i) unlike = true;
            if (r1 - r0 > kResidentMaxRow) odd = true;
            else if (times(r0, r1, i) != 1) {
                odd = true;
                unlike |= r1 - r0 <= kTileRow;
            }
            if (!odd) odd = times(s + 1, s1, j) != 0;
        }
    }
    __syncthreads();
    for (uint32_t l = 0; l < s_count; ++l) {
        const uint32_t v = s_long[l];
        for (uint32_t s = row[v] + threadIdx.x; s < row[v + 1] && !unlike; s += blockDim.x) {
            const uint32_t j = col[s], r0 = row[j], r1 = row[j + 1];
            unlike |= r1 - r0 <= kTileRow && times(r0, r1, v) != 1;
        }
    }
    if (__syncthreads_or(odd || unlike) && threadIdx.x == 0) bad[0] = 1;
    if (__syncthreads_or(unlike) && threadIdx.x == 0) bad[1] = 1;
}

}  // namespace

size_t resident_smem(uint32_t cap, bool slope) {
    return (size_t)cap * (24 + (slope ? 8 : 0)) + (size_t)kEdges * 24 + 32;
}

uint32_t resident_cap(bool slope) {
    return (uint32_t)((kResidentSmem - kEdges * 24 - 32) / (24 + (slope ? 8 : 0))) & ~7u;
}

uint32_t resident_blocks() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (uint32_t)std::max(1, sms);
}

cudaError_t launch_resident(const ResidentArgs& a, bool slope, uint32_t blocks, cudaStream_t st) {
    const void* kern = slope ? (const void*)k_resident<true> : (const void*)k_resident<false>;
    const size_t sm = resident_smem(a.cap, slope);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResidentSmem);
    if (e != cudaSuccess) return e;
    void* argv[] = {(void*)&a};
    return cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(kT), argv, sm, st);
}

void launch_check_rows(cudaStream_t st, uint32_t n, const uint32_t* row, const uint32_t* col, int* bad) {
    k_check_rows<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(n, row, col, bad);
}

}  // namespace fl
