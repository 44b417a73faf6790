// resident.cu -- whole solves in one kernel launch, for terrains whose working state fits
// the SMs' shared memory (src/lem/generator.rs:140-210, every iteration, bit-exact).
//
// The stage-by-stage pass (receivers.cu, solver.cu, basin.cu) spends an iteration of a
// small or middling terrain on launches and grid barriers: about 28 dependent launches and
// 60 barriers, 280 us at 1,000 sites and 450 us at 65,000, while the longest river is only
// 22 and 159 sites long.  Here a terrain is cut into contiguous ranges of its (Hilbert)
// memory order, one per block, one block per SM, and the block keeps its range's areas,
// response times, donor lists and pending counts in shared memory for the whole solve.
// What is left on an iteration's critical path is the longest river's chain of additions.
// An iteration takes 39 us at 1,000 sites, 102 us at 10,000 and 222 us at 65,000 (with
// slope limits 174 us at 10,000, 420 before): 0.3 to 0.6 us a river site and direction, a
// chain of dependent instructions at some six cycles each.
//
//   receivers   every site's steepest neighbour; elevations are read through L2
//   barrier     (all receivers known; lakes, if any, are re-routed here)
//   link        per site the list of its donors in reverse row order (the reference's
//               addition order): first donor, next sibling, number of donors
//   up          a thread starts at a leaf and walks down the river: it counts itself off
//               its receiver's donors, and the last donor to arrive adds the receiver's
//               list and goes on; no thread ever waits for another.  A donor in another
//               block is an extra list entry whose value that block publishes in L2;
//               one lane per such entry polls for it.  Finished sites are listed in order.
//   w           1 / (k sqrt(A)) * len where A or len changed, packed on dense warps
//   down        the finished list backwards (a receiver finishes after its donors, so it
//               is listed after them): each lane waits for its site's receiver's response
//               time, in shared memory or, across blocks, in L2
//   elevation   from the site's and its basin outlet's response time; with slope limits
//               the limited elevations run down the same list once more
//   barrier     (all elevations written; did any change?)
// Values published across blocks use two slots per site, by the iteration's parity: a slot
// is set back to the pending marker one iteration later, when its readers have passed a
// barrier, so the publishing store is itself the flag and an iteration needs two barriers.
//
// Every wait is bounded.  Waiting lanes never block a site that an earlier one in the
// order needs: a block's list is in order of finishing, and across blocks a receiver
// finishes after its donors, so of all unfinished sites the one that finished last in the
// upward pass always has its receiver's value and a thread.
//
// One launch takes many terrains (packed models): blocks take (terrain, part) slots in
// order, largest terrains first, and a terrain starts when its last part is taken.  Only
// the newest terrain can be partly taken, so the blocks that wait for its other parts wait
// for terrains that are running.

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "slope.cuh"

namespace fl {
namespace {

constexpr uint32_t kT = kResidentThreads;
constexpr uint32_t kEdges = kResidentEdges;     // donors in other blocks: one polling lane each
// Warps that walk up from the leaves (the rest, or all when all walk, poll for far donors)
// and that walk down, in blocks of up to kFewSites sites: with a site or two per thread the
// walks are few and long, and the f64 lanes (16 cycles an instruction however few of its
// lanes are active) and the polls of idle warps hold them up.
constexpr uint32_t kFewSites = 2048, kFewWarps = 16;
constexpr uint32_t kEnd = 0xffffu;              // end of a donor list
constexpr uint64_t kPendingBits = 0x7ff4000000000000ull;   // a signalling NaN: never a result
constexpr uint64_t kQuietNan = 0x7ff8000000000000ull;
constexpr uint32_t kNoOutlet = 0x80000000u;     // root id bit: the root is not an outlet

// per-site word: donors still to arrive, kind bits, the receiver's index in the block
constexpr uint32_t kCount = 0xffu;
constexpr uint32_t kRoot = 0x100u;              // its own receiver
constexpr uint32_t kFar = 0x200u;               // its receiver is in another block
constexpr uint32_t kFarDonor = 0x400u;          // it has a donor in another block
constexpr int kParentShift = 16;

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
// Ordering fences without the sequential consistency of __threadfence.
__device__ __forceinline__ void fence_block() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ uint64_t bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double from_bits(uint64_t b) { return __longlong_as_double((long long)b); }
__device__ __forceinline__ uint64_t published(double x) { return isnan(x) ? kQuietNan : bits(x); }
// plus_zero without an f64 comparison (64 cycles on the river's critical path)
__device__ __forceinline__ double plus_zero_bits(double x) {
    const uint64_t b = bits(x);
    return from_bits((b << 1) == 0 ? 0 : b);
}

// Exchange slots of site g (by iteration parity): area, response time, limited elevation.
__device__ __forceinline__ double* area_slot(const ResidentArgs& a, uint32_t g, uint32_t par) { return a.xch + 4ull * g + par; }
__device__ __forceinline__ double* time_slot(const ResidentArgs& a, uint32_t g, uint32_t par) { return a.xch + 4ull * g + 2 + par; }
__device__ __forceinline__ double* elev_slot(const ResidentArgs& a, uint32_t g, uint32_t par) { return a.xch2 + 4ull * g + par; }
// A root's response time, and the root of a site whose time other blocks read.
__device__ __forceinline__ double* root_time(const ResidentArgs& a, uint32_t g) { return a.xch2 + 4ull * g + 2; }

__device__ __forceinline__ void raise(ResidentCtrl* c, int code) { atomicCAS(&c->error, 0, code); }

// What a block needs at hand about its terrain.
struct Group {
    unsigned long long* bar;   // four rotating barrier words
    ResidentCtrl* ctrl;
    uint32_t parts, part;
    uint32_t k;                // barriers passed
    bool ok;
};

// Barrier over the terrain's blocks; returns whether any thread of any block set pred.
// gr.ok turns false when the wait ran out or an error was raised (for all threads).
__device__ __noinline__ bool group_barrier(Group& gr, bool pred) {
    __shared__ int s_any, s_ok;
    const int mine = __syncthreads_or(pred);
    if (gr.parts == 1) {
        if (threadIdx.x == 0) s_ok = ld_acquire(&gr.ctrl->error) == 0;
        __syncthreads();
        gr.ok = s_ok != 0;
        __syncthreads();
        return mine != 0;
    }
    if (threadIdx.x == 0) {
        unsigned long long* w = &gr.bar[gr.k & 3];
        fence_gpu();
        // every block has read the word two barriers back: clear it for its next use
        if (gr.part == 0) atomicExch(&gr.bar[(gr.k + 2) & 3], 0ull);
        fence_gpu();
        atomicAdd(w, 1ull | ((unsigned long long)(mine ? 1 : 0) << 32));
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
        s_any = (int)(v >> 32);
        if (ld_acquire(&gr.ctrl->error) != 0) s_ok = 0;
        fence_gpu();
    }
    __syncthreads();
    const bool any = s_any != 0;
    gr.ok = s_ok != 0;
    ++gr.k;
    __syncthreads();
    return any;
}

__device__ __forceinline__ bool give_up(Group& gr, uint32_t& spins) {
    if (++spins > kSpinLimit) {
        raise(gr.ctrl, kErrWait);
        return true;
    }
    return (spins & 255) == 0 && ld_acquire(&gr.ctrl->error) != 0;
}

// The reference's scan of site g's row: its slot, or kNone.
__device__ __noinline__ uint32_t steepest_exact(const uint32_t* row, const uint32_t* col, const double* len,
                                                const double* elev, uint32_t g) {
    const double ei = elev[g];
    double top = 0.0;
    uint32_t slot = kNone;
#pragma unroll 1
    for (uint32_t s = row[g], e = row[g + 1]; s < e; ++s) {
        const double ej = elev[col[s]];
        if (ei > ej) {
            const double m = __ddiv_rn(__dsub_rn(ei, ej), len[s]);
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
    const uint32_t s0 = a.row[g], s1 = a.row[g + 1];
    const float2 own = a.pair[g];
    PairScan sc(own);
#pragma unroll 1
    for (uint32_t b = s0; b < s1; b += 4) {
        float2 e[4];
        float f[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t s = min(b + k, s1 - 1);
            e[k] = a.pair[a.col[s]];
            f[k] = a.ilen[s];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (b + k < s1) sc.consider(b + k, e[k], f[k]);
    }
    return sc.decided() ? sc.slot : steepest_exact(a.row, a.col, a.len, a.elev, g);
}

__device__ __forceinline__ double edge_or_one(const ResidentArgs& a, uint32_t i, uint32_t j) {
    for (uint32_t s = a.row[i], e = a.row[i + 1]; s < e; ++s)
        if (a.col[s] == j) return a.len[s];
    return 1.0;
}

// Lake re-routing (stream_tree.rs:139-243) of the terrain's receivers: labels by pointer
// jumping, the first processed entry of every lake, path reversal (as solver.cu's kernels).
__device__ __noinline__ void reroute_lakes(const ResidentArgs& a, Group& gr, uint32_t lo, uint32_t S) {
#pragma unroll 1
    for (uint32_t v = threadIdx.x; v < S; v += kT) {
        a.lab[lo + v] = __ldcg(&a.next[lo + v]);
        a.best[lo + v] = kNoKey;
    }
    group_barrier(gr, false);
    uint32_t *cur = a.lab, *out = a.lab2;
    for (uint32_t round = 0; gr.ok; ++round) {
        bool moved = false;
#pragma unroll 1
        for (uint32_t v = threadIdx.x; v < S; v += kT) {
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
    for (uint32_t v = threadIdx.x; v < S; v += kT) {
        const uint32_t g = lo + v, r = a.rank[g];
        if (r == kNone) continue;
        const uint32_t own = __ldcg(&cur[g]);
        const uint32_t s0 = a.row[g], s1 = a.row[g + 1];
        for (uint32_t s = s0; s < s1; ++s) {
            const uint32_t L = __ldcg(&cur[a.col[s]]);
            if (a.outlet[L] || L == own) continue;
            const unsigned long long key = ((unsigned long long)r << 32) | (s - s0);
            if (key < __ldcg(&a.best[L])) atomicMin(&a.best[L], key);
        }
    }
    group_barrier(gr, false);
    if (!gr.ok) return;
#pragma unroll 1
    for (uint32_t v = threadIdx.x; v < S; v += kT) {
        const unsigned long long key = __ldcg(&a.best[lo + v]);
        if (key == kNoKey) continue;
        uint32_t nk = a.sor[key >> 32];
        uint32_t k = a.col[a.row[nk] + (uint32_t)key];
        for (uint32_t steps = 0;; ++steps) {
            if (steps > a.n) {
                raise(gr.ctrl, kErrForest);
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
    group_barrier(gr, false);
}

// Shared memory of a block for up to `cap` sites (resident_smem): values, per-site words,
// donor lists (first donor, next sibling), the finished list and the far donors.
struct Block {
    double* val;        // [cap + kEdges] area, then response time, then limited elevation
    uint32_t* word;     // [cap]
    uint32_t* far_id;   // [kEdges] a far donor's site
    uint16_t* first;    // [cap] first donor in addition order; with sib, later the roots
    uint16_t* sib;      // [cap + kEdges]
    uint16_t* order;    // [cap] finished sites in order
    uint16_t* far_to;   // [kEdges] the site it drains to
};

__device__ __forceinline__ Block carve(unsigned char* sm, uint32_t cap) {
    Block b;
    b.val = reinterpret_cast<double*>(sm);
    b.word = reinterpret_cast<uint32_t*>(b.val + cap + kEdges);
    b.far_id = b.word + cap;
    b.first = reinterpret_cast<uint16_t*>(b.far_id + kEdges);
    b.sib = b.first + cap;
    b.order = b.sib + cap + kEdges;
    b.far_to = b.order + cap;
    return b;
}

// One terrain's iterations up to its fixed point, its limit or the launch's share.
template <bool kSlope>
__device__ void solve_terrain(const ResidentArgs& a, const ResidentTerrain& tr, Group& gr,
                              unsigned char* smem) {
    __shared__ uint32_t s_fin, s_far, s_list;
    const uint32_t tid = threadIdx.x;
    const uint32_t each = tr.n / tr.parts, rest = tr.n % tr.parts;
    const uint32_t lo = tr.lo + gr.part * each + min(gr.part, rest);
    const uint32_t S = each + (gr.part < rest ? 1u : 0u);
    const Block bk = carve(smem, a.cap);
    volatile uint64_t* vval = reinterpret_cast<volatile uint64_t*>(bk.val);
    volatile uint32_t* vword = bk.word;
    uint32_t* root = reinterpret_cast<uint32_t*>(bk.first);   // over first and sib
    ResidentCtrl* ctrl = gr.ctrl;
    const uint32_t walkers = S > kFewSites ? kT : kFewWarps * 32;

    uint32_t it = ctrl->iters;
    const uint32_t stop = (uint32_t)min((uint64_t)it + a.chunk, (uint64_t)a.limit);
    bool valid = it > 0;                      // w, wa, wl hold the previous iteration's
#pragma unroll 1
    for (uint32_t v = tid; v < S; v += kT) {
        const uint32_t g = lo + v;
        for (uint32_t par = 0; par < 2; ++par) {
            st_relaxed64(area_slot(a, g, par), kPendingBits);
            st_relaxed64(time_slot(a, g, par), kPendingBits);
            if (kSlope) st_relaxed64(elev_slot(a, g, par), kPendingBits);
        }
        bk.word[v] = 0;
    }
    group_barrier(gr, false);

    while (gr.ok && it < stop) {
        const uint32_t par = it & 1u;
        // ---- receivers
        bool lake = false;
#pragma unroll 1
        for (uint32_t v = tid; v < S; v += kT) {
            const uint32_t g = lo + v;
            // last iteration's published values have been read: their slots are free
            const uint32_t was = bk.word[v];
            if (was & kFar) st_relaxed64(area_slot(a, g, par ^ 1u), kPendingBits);
            if (was & kFarDonor) {
                st_relaxed64(time_slot(a, g, par ^ 1u), kPendingBits);
                if (kSlope) st_relaxed64(elev_slot(a, g, par ^ 1u), kPendingBits);
            }
            uint32_t slot = kNone;
            if (!a.outlet[g]) {
                slot = steepest(a, g);
                lake |= slot == kNone;
            }
            const uint32_t p = slot == kNone ? g : a.col[slot];
            a.next[g] = p;
            a.rlen[g] = slot == kNone ? 1.0 : a.len[slot];
            bk.word[v] = p == g ? kRoot : p - lo < S ? (p - lo) << kParentShift : kFar;
            bk.val[v] = a.area[g];
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
            for (uint32_t v = tid; v < S; v += kT) {
                const uint32_t g = lo + v, p = __ldcg(&a.next[g]);
                bk.word[v] = p == g ? kRoot : p - lo < S ? (p - lo) << kParentShift : kFar;
            }
        }
        // ---- link
        if (tid == 0) s_fin = s_far = 0;
        __syncthreads();
#pragma unroll 1
        for (uint32_t base = 0; base < S; base += kT) {
            const uint32_t v = base + tid;
            bool leaf = false;
            if (v < S) {
                const uint32_t g = lo + v;
                const uint32_t s0 = a.row[g], s1 = a.row[g + 1];
                uint32_t cnt = 0, prev = kEnd, far = 0;
                for (uint32_t hi = s1; hi > s0; hi = hi > s0 + 8 ? hi - 8 : s0) {
                    uint32_t j[8];
                    uint32_t don = 0, faro = 0;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (hi >= s0 + 1 + k) j[k] = a.col[hi - 1 - k];
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (hi >= s0 + 1 + k) {
                            const uint32_t d = j[k] - lo;
                            if (d < S) {
                                const uint32_t w = vword[d];
                                if (!(w & (kRoot | kFar)) && (w >> kParentShift) == v) don |= 1u << k;
                            } else if (__ldcg(&a.next[j[k]]) == g) {
                                faro |= 1u << k;
                            }
                        }
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (((don | faro) >> k) & 1u) {
                            uint32_t code = j[k] - lo;
                            if ((faro >> k) & 1u) {
                                const uint32_t e = atomicAdd(&s_far, 1u);
                                far = kFarDonor;
                                if (e >= kEdges) continue;        // reported below
                                bk.far_id[e] = j[k];
                                bk.far_to[e] = (uint16_t)v;
                                code = a.cap + e;
                            }
                            if (prev == kEnd) bk.first[v] = (uint16_t)code;
                            else bk.sib[prev] = (uint16_t)code;
                            prev = code;
                            ++cnt;
                        }
                }
                if (prev != kEnd) bk.sib[prev] = (uint16_t)kEnd;
                vword[v] = vword[v] | cnt | far;
                leaf = cnt == 0;
            }
            const unsigned m = __ballot_sync(0xffffffffu, leaf);
            uint32_t at = 0;
            if ((tid & 31) == 0 && m) at = atomicAdd(&s_fin, (uint32_t)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (leaf) bk.order[at + __popc(m & ((1u << (tid & 31)) - 1u))] = (uint16_t)v;
        }
        __syncthreads();
        const uint32_t nleaf = s_fin, nfar = s_far;
        __syncthreads();
        if (nfar > kEdges) {                  // the other blocks see it at their next wait
            if (tid == 0) raise(ctrl, kErrCapacity);
            gr.ok = false;
            break;
        }
        // ---- up: site v is final (have); count it off its receiver and go on if last
        bool have = false;
        uint32_t v = 0;
        auto arrive = [&](uint32_t p) {
            fence_block();
            const uint32_t old = atomicSub(&bk.word[p], 1u);
            have = (old & kCount) == 1u;
            if (have) {
                fence_block();
                double x = from_bits(vval[p]);
                uint32_t d = bk.first[p];
                for (uint32_t q = 0; q < kResidentMaxRow && d != kEnd; ++q) {
                    const double y = from_bits(vval[d]);
                    d = bk.sib[d];
                    x = __dadd_rn(x, y);
                }
                vval[p] = bits(x);
                bk.order[atomicAdd(&s_fin, 1u)] = (uint16_t)p;
                v = p;
            }
        };
        auto step = [&]() {
            const uint32_t w = vword[v];
            if (w & (kRoot | kFar)) {
                if (w & kFar) st_relaxed64(area_slot(a, lo + v, par), published(from_bits(vval[v])));
                have = false;
            } else {
                arrive(w >> kParentShift);
            }
        };
        bool lost_up = false;
        if (tid < walkers) {
#pragma unroll 1
        for (uint32_t i = tid;;) {
            if (!have && i < nleaf) {
                v = bk.order[i];
                i += walkers;
                have = true;
            }
            if (!__any_sync(0xffffffffu, have)) break;
            if (have) step();
        }
        }
        const uint32_t poll0 = walkers == kT ? 0 : walkers;
        if (tid >= poll0) {
            // far donors spread over the warps; a warp with a walk under way does not poll
            const uint32_t e = (tid & 31u) * ((kT - poll0) / 32) + ((tid - poll0) >> 5);
            bool wait = e < nfar, lost = false;
            const double* src = wait ? area_slot(a, bk.far_id[e], par) : nullptr;
            uint32_t spins = 0;
            while (__any_sync(0xffffffffu, wait)) {
                if (wait) {
                    const uint64_t b = ld_relaxed64(src);
                    if (b != kPendingBits) {
                        vval[a.cap + e] = b;
                        wait = false;
                        arrive(bk.far_to[e]);
                    } else if (give_up(gr, spins)) {
                        wait = false;
                        lost = true;
                    }
                }
                while (__any_sync(0xffffffffu, have))
                    if (have) step();
            }
            lost_up = lost;
        }
        if (__syncthreads_or(lost_up)) {
            gr.ok = false;
            break;
        }
        if (s_fin != S) {                     // a receiver cycle: never in a forest
            if (tid == 0) raise(ctrl, kErrForest);
            gr.ok = false;
            break;
        }
        // ---- w, where an operand changed since the previous iteration
        if (tid == 0) s_list = 0;
        __syncthreads();
        uint16_t* list = bk.first;
#pragma unroll 1
        for (uint32_t base = 0; base < S; base += kT) {
            const uint32_t u = base + tid;
            bool need = false;
            if (u < S) {
                const uint32_t g = lo + u;
                need = !valid || bits(bk.val[u]) != bits(__ldcg(&a.wa[g])) ||
                       bits(__ldcg(&a.rlen[g])) != bits(__ldcg(&a.wl[g]));
            }
            const unsigned m = __ballot_sync(0xffffffffu, need);
            uint32_t at = 0;
            if ((tid & 31) == 0 && m) at = atomicAdd(&s_list, (uint32_t)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (need) list[at + __popc(m & ((1u << (tid & 31)) - 1u))] = (uint16_t)u;
        }
        __syncthreads();
        const uint32_t nlist = s_list;
#pragma unroll 1
        for (uint32_t i = tid; i < nlist; i += kT) {
            const uint32_t u = list[i], g = lo + u;
            const double A = bk.val[u], l = __ldcg(&a.rlen[g]);
            const double cel = __dmul_rn(a.k[g], __dsqrt_rn(A));
            a.w[g] = __dmul_rn(__ddiv_rn(1.0, cel), l);
            a.wa[g] = A;
            a.wl[g] = l;
        }
        valid = true;
        __syncthreads();
#pragma unroll 1
        for (uint32_t u = tid; u < S; u += kT) vval[u] = kPendingBits;
        __syncthreads();
        // ---- down: response times
        bool changed = false, lost = false;
        if (tid < walkers)
#pragma unroll 1
        for (uint32_t base = 0; base < S; base += walkers) {
            const uint32_t i = base + tid;
            bool todo = i < S, far = false;
            uint32_t p = 0, w = 0;
            double wv = 0.0;
            const double* src = nullptr;
            auto publish = [&](double t, uint32_t r) {
                root[v] = r;
                fence_block();
                vval[v] = bits(t);
                if (w & kFarDonor) {
                    a.root[lo + v] = r;
                    fence_gpu();
                    st_relaxed64(time_slot(a, lo + v, par), published(t));
                }
                todo = false;
            };
            auto settle = [&](uint64_t tb, uint32_t r) {
                publish(plus_zero_bits(__dadd_rn(from_bits(tb), wv)), r);
            };
            if (todo) {
                v = bk.order[S - 1 - i];
                w = vword[v];
                wv = __ldcg(&a.w[lo + v]);
                if (w & kRoot) {
                    const uint32_t g = lo + v;
                    const double t = plus_zero(plus_zero(wv)), old_e = __ldcg(&a.elev[g]);
                    const bool out = a.outlet[g] != 0;
                    if (out) {
                        const double dt = __dsub_rn(t, t);
                        double ne = __dadd_rn(old_e, __dmul_rn(a.u[g], dt > 0.0 ? dt : 0.0));
                        if (kSlope) {
                            const double tn = a.tanms[g], dist = __ldcg(&a.rlen[g]);
                            if (!isnan(tn)) {
                                const double m = __ddiv_rn(__dsub_rn(ne, old_e), dist);
                                if (m > tn) ne = __dadd_rn(old_e, __dmul_rn(tn, dist));
                            }
                        }
                        changed |= ne != old_e;
                        a.elev[g] = ne;
                        a.pair[g] = float_pair(ne);
                    }
                    *root_time(a, g) = t;     // read after the value published here
                    publish(t, out ? g : g | kNoOutlet);
                } else if (w & kFar) {
                    far = true;
                    src = time_slot(a, __ldcg(&a.next[lo + v]), par);
                } else {
                    p = w >> kParentShift;
                }
            }
            uint32_t spins = 0;
            while (__any_sync(0xffffffffu, todo)) {
                uint64_t fb = kPendingBits;
                if (todo && far) fb = ld_relaxed64(src);      // in flight over the local polls
#pragma unroll 1
                for (int k = 0; k < 4; ++k)
                    if (todo && !far) {
                        const uint64_t tb = vval[p];
                        if (tb != kPendingBits) {
                            fence_block();
                            settle(tb, reinterpret_cast<volatile uint32_t*>(root)[p]);
                        }
                    }
                if (todo && far && fb != kPendingBits) {
                    fence_gpu();
                    settle(fb, __ldcg(&a.root[__ldcg(&a.next[lo + v])]));
                }
                if (todo && give_up(gr, spins)) {
                    todo = false;
                    lost = true;
                }
            }
            if (__any_sync(0xffffffffu, lost)) break;
        }
        if (__syncthreads_or(lost)) {
            gr.ok = false;
            break;
        }
        // ---- elevations
#pragma unroll 1
        for (uint32_t u = tid; u < S; u += kT) {
            const uint32_t r = root[u], g = lo + u;
            if (!(r & kNoOutlet) && r != g) {
                const double to = __ldcg(root_time(a, r)), eo = __ldcg(&a.elev[r]);
                const double dt = __dsub_rn(from_bits(vval[u]), to);
                const double ne = __dadd_rn(eo, __dmul_rn(a.u[g], dt > 0.0 ? dt : 0.0));
                if (kSlope) {
                    a.ef[g] = ne;
                } else {
                    changed |= ne != __ldcg(&a.elev[g]);
                    a.elev[g] = ne;
                    a.pair[g] = float_pair(ne);
                }
            }
            if (kSlope) vval[u] = kPendingBits;
        }
        if (kSlope) {
            // the limit e_v <= e_receiver + tan * len, down the same list.  The reference
            // compares (e_v - e_r) / len with tan; unless the difference is within 2^-50 of
            // tan * len, the comparison with the (positive) product decides it.
            __syncthreads();
            if (tid < walkers)
#pragma unroll 1
            for (uint32_t base = 0; base < S; base += walkers) {
                const uint32_t i = base + tid;
                bool todo = i < S, far = false;
                uint32_t p = 0, w = 0;
                double ne = 0.0, rise = 0.0, above = 0.0, below = 0.0, tn = 0.0, dist = 1.0;
                const double* src = nullptr;
                auto store = [&](double e) {
                    vval[v] = published(e);
                    if (w & kFarDonor) st_relaxed64(elev_slot(a, lo + v, par), published(e));
                    todo = false;
                };
                auto limit = [&](uint64_t eb) {
                    const double ep = from_bits(eb), d = __dsub_rn(ne, ep);
                    bool over;
                    if (d > above) over = true;
                    else if (d < below) over = false;
                    else over = __ddiv_rn(d, dist) > tn;
                    if (over) ne = __dadd_rn(ep, rise);
                    store(ne);
                };
                double old_e = 0.0;
                bool moves = false;
                if (todo) {
                    v = bk.order[S - 1 - i];
                    const uint32_t g = lo + v;
                    w = vword[v];
                    const uint32_t r = root[v];
                    if (r & kNoOutlet) {
                        todo = false;
                    } else if (w & kRoot) {
                        store(__ldcg(&a.elev[g]));
                    } else {
                        moves = true;
                        ne = __ldcg(&a.ef[g]);
                        tn = a.tanms[g];
                        dist = __ldcg(&a.rlen[g]);
                        old_e = __ldcg(&a.elev[g]);
                        if (isnan(tn)) {
                            store(ne);
                        } else {
                            rise = __dmul_rn(tn, dist);
                            const double gap = __dmul_rn(rise, 0x1p-50);
                            above = __dadd_rn(rise, gap);
                            below = __dsub_rn(rise, gap);
                            if (!(tn > 1e-200 && dist > 0.0 && rise > 1e-200 && rise < 1e200)) {
                                // the product cannot stand in for the quotient: divide
                                above = from_bits(0x7ff0000000000000ull);
                                below = -above;
                            }
                            if (w & kFar) {
                                far = true;
                                src = elev_slot(a, __ldcg(&a.next[g]), par);
                            } else {
                                p = w >> kParentShift;
                            }
                        }
                    }
                }
                uint32_t spins = 0;
                while (__any_sync(0xffffffffu, todo)) {
                    uint64_t fb = kPendingBits;
                    if (todo && far) fb = ld_relaxed64(src);
#pragma unroll 1
                    for (int k = 0; k < 4; ++k)
                        if (todo && !far) {
                            const uint64_t eb = vval[p];
                            if (eb != kPendingBits) limit(eb);
                        }
                    if (todo && far && fb != kPendingBits) limit(fb);
                    if (todo && give_up(gr, spins)) {
                        todo = false;
                        lost = true;
                    }
                }
                if (__any_sync(0xffffffffu, lost)) break;
                if (moves) {
                    changed |= ne != old_e;
                    a.elev[lo + v] = ne;
                    a.pair[lo + v] = float_pair(ne);
                }
            }
            if (__syncthreads_or(lost)) {
                gr.ok = false;
                break;
            }
        }
        ++it;
        const bool more = group_barrier(gr, changed);
        if (!gr.ok) break;
        if (!more || it >= a.limit) {
            if (gr.part == 0 && tid == 0) ctrl->done = 1;
            break;
        }
    }
    if (gr.part == 0 && tid == 0) ctrl->iters = it;
}

template <bool kSlope>
__global__ void __launch_bounds__(kT, 1) k_resident(const __grid_constant__ ResidentArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_slot;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_slot = atomicAdd(a.ticket, 1u);
        __syncthreads();
        const uint32_t slot = s_slot;
        if (slot >= a.slots) return;
        const uint32_t t = a.slot_terrain[slot];
        const ResidentTerrain tr = a.terrains[t];
        Group gr{a.bars + 4ull * t, a.ctrl + t, tr.parts, slot - tr.slot0, 0, true};
        if (gr.ctrl->done) continue;          // settled in an earlier launch
        solve_terrain<kSlope>(a, tr, gr, smem);
    }
}

// Whether every edge of the graph appears exactly once in either end's row, no site is its
// own neighbour and no row is longer than the donor count can hold.
__global__ void k_check_simple(uint32_t n, const uint32_t* __restrict__ row,
                               const uint32_t* __restrict__ col, int* __restrict__ bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool b = false;
    if (i < n) {
        const uint32_t s0 = row[i], s1 = row[i + 1];
        b = s1 - s0 > kResidentMaxRow;
        for (uint32_t s = s0; s < s1 && !b; ++s) {
            const uint32_t j = col[s];
            b = j == i;
            for (uint32_t q = s + 1; q < s1; ++q) b |= col[q] == j;
            uint32_t back = 0;
            const uint32_t r0 = row[j], r1 = row[j + 1];
            if (r1 - r0 > kResidentMaxRow) b = true;
            for (uint32_t q = r0; q < r1 && !b; ++q) back += col[q] == i;
            b |= back != 1;
        }
    }
    if (__syncthreads_or(b) && threadIdx.x == 0) *bad = 1;
}

}  // namespace

size_t resident_smem(uint32_t cap) { return (size_t)cap * 18 + (size_t)kEdges * 16; }

uint32_t resident_cap() { return (uint32_t)((kResidentSmem - kEdges * 16) / 18) & ~7u; }

uint32_t resident_blocks() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (uint32_t)std::max(1, sms);
}

cudaError_t launch_resident(const ResidentArgs& a, bool slope, uint32_t blocks, cudaStream_t st) {
    const void* kern = slope ? (const void*)k_resident<true> : (const void*)k_resident<false>;
    const size_t sm = resident_smem(a.cap);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kResidentSmem);
    if (e != cudaSuccess) return e;
    void* argv[] = {(void*)&a};
    return cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(kT), argv, sm, st);
}

void launch_check_simple(cudaStream_t st, uint32_t n, const uint32_t* row, const uint32_t* col,
                         int* bad) {
    k_check_simple<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(n, row, col, bad);
}

}  // namespace fl
