// The reduction: lock-free pivot claiming with group-parallel sorted-set XOR merges.
//
// Reference counterparts:
//   spectral-sequence block loop       include/specseq.h:592-704 (GPU_Compute)
//   pivot claim + addition queue       include/kernel.h:583-633 (BlockScan, BlockGenAddition)
//   column addition, warp phase        include/kernel.h:691-743, 814-936 (ProcColumnPair)
//   column addition, block phase       include/kernel.h:744-792, 939-1065 (ProcColumnPair_121Block)
//   CPU tail stage                     include/specseq.h:705-1046 (no counterpart here:
//                                      every column is finished on the device)
//
// Two tiers, as in the reference's two phases.  Light tier: warps reduce the
// columns whose entries fit in a warp's shared-memory buffers (level-1
// capacity), four tiny ones at a time.  Heavy tier: a column that outgrows them
// is handed to a second kernel in which a whole CTA reduces it with buffers of
// the level-2 capacity, and beyond that in exact-size arena buffers.  Both tiers
// add in rounds (below) and share the column routine, written once over a
// "group" (warp or CTA).
//
// Pivot table.  pivot[row] holds the owning column and the arena slot of the
// owner's version (pv_pack), so the owner's entries are one dependent load
// away.  A column whose lowest row L has no owner, or an owner with a larger
// index, publishes its current entries (fresh arena slot, then its
// descriptor) and claims L with a 64-bit compare-and-swap.  Published column
// versions are never modified afterwards, so a reader holding an older entry
// still adds a valid earlier column with the same lowest row.  Displacing a
// larger owner hands that owner to the displacing group, which reduces it
// next (no other group can reach it), so there is no work queue to wait on and
// no spin-wait at all.  Every addition adds an earlier column with the same
// lowest row, so the result is a left-to-right reduction and the pairs equal
// those of any sequential one.  Claiming a row also clears the row's own
// column (twist clearing).
//
// The boundary matrix's edges, columns of two entries at most, are reduced by a walk of
// their own (sspp_edges.cu) when no longer column of dimension 1 is among them.
//
// Additions.  A column in shared memory takes its additions in rounds: the
// owners of all its top rows at once (round_adds).  What a round cannot take
// (an addend of more than kRoundAddend entries, a sum that does not fit, a column
// in the arena) goes one addition at a time: the addend is staged into shared
// memory with 16-byte vector loads (header and entries in one pass when it fits);
// the next lowest row is known before the merge - it is the largest index at
// which the tops of the two lists stop agreeing - so the pivot entry of that row
// is requested before the merge starts and arrives while it runs.  The merge
// computes each element's output slot from its rank in the other list minus twice
// the cancelled pairs before it (one ballot/prefix per round for both lists): no
// atomics, no scratch in global memory.
#include <algorithm>
#include <climits>
#include <mutex>

#include "sspp_kernels.cuh"
#include "sspp_launch.h"

namespace sspp {

struct ReduceArgs {
    int32_t ncols;
    const int32_t* active;  // light tier: the step's columns
    int32_t cap;          // shared-memory capacity per buffer (ints), multiple of 32
    int32_t* arena;
    int64_t arena_cap;
    unsigned long long* arena_top;
    uint64_t* desc;
    int32_t* low;
    uint64_t* pivot;
    uint8_t* state;
    uint8_t* cleared;
    int* ctr;             // per step: [0] chunk counter, [1] [2] heavy pool range, [3] heavy pull counter,
                          // [4] warp-tier blocks finished
    int32_t listed;       // how many
    int* ctr_next;        // the next step's counters (its pool range starts where this step's ends), or null
    int32_t* heavy;       // heavy pool (columns handed to the CTA tier, appended in step order)
    int* pool_tail;
    int* heavy_done;      // pool columns finished by the CTA tier
    int* gate_host;       // mapped host mirror of heavy_done, or null
    int64_t pool_cap;
    int* err;
    long long* counters;
    int32_t light_chain;  // warp tier: additions per column before handing it to the CTA tier (0 = no limit)
    const int4* app;      // inline short apparent columns by row (Device::app)
};

// Where one reduction of a column stops: the band's lowest row (a column whose
// low drops below it parks), and the counter of the work it came from, so that
// a long chain in the warp tier moves to the CTA tier once that work is fully
// handed out (drain_ctr >= drain_total).
struct Band {
    int32_t minrow;
    const int* drain_ctr;
    int32_t drain_total;
};

constexpr int kMaxMergesPerColumn = 1 << 24;

// A pivot entry read early, before it is known whether it is needed: relaxed,
// so a fence (acquire) must come before the owner's slot is read through it.
__device__ __forceinline__ uint64_t ld_relaxed_u64(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint64_t ld_acquire_u64(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_u64(uint64_t* p, uint64_t v) {
    asm volatile("st.release.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// ------------------------------------------------------------------ groups
struct WarpG {
    static constexpr int kSize = 32;
    __device__ __forceinline__ int rank() const { return threadIdx.x & 31; }
    __device__ __forceinline__ bool leader() const { return (threadIdx.x & 31) == 0; }
    __device__ __forceinline__ void sync() const { __syncwarp(); }
    // __syncwarp orders the leader's preceding memory accesses (an acquire in
    // particular) before the other lanes' following ones
    __device__ __forceinline__ int bcast(int v) const {
        __syncwarp();
        return __shfl_sync(kFull, v, 0);
    }
    __device__ __forceinline__ unsigned long long bcast64(unsigned long long v) const {
        __syncwarp();
        return __shfl_sync(kFull, v, 0);
    }
    __device__ __forceinline__ unsigned long long bcast64_last(unsigned long long v) const {
        __syncwarp();
        return __shfl_sync(kFull, v, 31);
    }
    // exclusive counts of fa and fb over lower ranks, and their group totals
    __device__ __forceinline__ void prefix2(bool fa, bool fb, int& pa, int& pb, int& ta, int& tb) const {
        const unsigned lt = lanemask_lt();
        unsigned ma = __ballot_sync(kFull, fa), mb = __ballot_sync(kFull, fb);
        pa = __popc(ma & lt);
        pb = __popc(mb & lt);
        ta = __popc(ma);
        tb = __popc(mb);
    }
    __device__ __forceinline__ int sum(int v) const { return warp_sum(v); }
    __device__ __forceinline__ int min_all(int v) const { return __reduce_min_sync(kFull, v); }
    // exclusive prefix of v over lower ranks; tot = group total
    __device__ __forceinline__ int prefix_int(int v, int& tot) const {
        int inc = warp_inclusive_scan(v);
        tot = __shfl_sync(kFull, inc, 31);
        return inc - v;
    }
};

template <int T>
struct BlockG {
    static constexpr int kSize = T;
    static constexpr int kWarps = T / 32;
    int* sm;                  // 2 * (kWarps + 2) ints: two scan buffers, used alternately
    unsigned long long* sb;   // two 8-byte broadcast slots, used alternately
    mutable int slot = 0;
    mutable int sbuf = 0;
    // alternating buffers: buffer b is rewritten only two collectives later,
    // after every thread has passed the barrier of the collective in between
    __device__ __forceinline__ int* scan_buf() const {
        int* b = sm + sbuf * (kWarps + 2);
        sbuf ^= 1;
        return b;
    }
    __device__ __forceinline__ int rank() const { return threadIdx.x; }
    __device__ __forceinline__ bool leader() const { return threadIdx.x == 0; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    // one barrier: consecutive broadcasts alternate slots, and a slot is only
    // rewritten after every thread has passed the following broadcast's barrier
    __device__ __forceinline__ unsigned long long bcast64(unsigned long long v) const {
        unsigned long long* p = sb + slot;
        slot ^= 1;
        if (threadIdx.x == 0) *p = v;
        __syncthreads();
        return *p;
    }
    __device__ __forceinline__ int bcast(int v) const { return int(bcast64((unsigned long long)(unsigned)v)); }
    __device__ __forceinline__ unsigned long long bcast64_last(unsigned long long v) const {
        unsigned long long* p = sb + slot;
        slot ^= 1;
        if (threadIdx.x == T - 1) *p = v;
        __syncthreads();
        return *p;
    }
    __device__ __forceinline__ void prefix2(bool fa, bool fb, int& pa, int& pb, int& ta, int& tb) const {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const unsigned lt = lanemask_lt();
        int* b = scan_buf();
        unsigned ma = __ballot_sync(kFull, fa), mb = __ballot_sync(kFull, fb);
        if (lane == 0) b[wid] = __popc(ma) | (__popc(mb) << 16);
        __syncthreads();
        if (wid == 0) {
            int c = lane < kWarps ? b[lane] : 0;
            int inc = warp_inclusive_scan(c);
            if (lane < kWarps) b[lane] = inc - c;
            if (lane == kWarps - 1) b[kWarps] = inc;
        }
        __syncthreads();
        const int base = b[wid], tot = b[kWarps];
        pa = (base & 0xffff) + __popc(ma & lt);
        pb = (base >> 16) + __popc(mb & lt);
        ta = tot & 0xffff;
        tb = tot >> 16;
    }
    __device__ __forceinline__ int prefix_int(int v, int& tot) const {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        int* b = scan_buf();
        int inc = warp_inclusive_scan(v);
        if (lane == 31) b[wid] = inc;
        __syncthreads();
        if (wid == 0) {
            int c = lane < kWarps ? b[lane] : 0;
            int ci = warp_inclusive_scan(c);
            if (lane < kWarps) b[lane] = ci - c;
            if (lane == kWarps - 1) b[kWarps] = ci;
        }
        __syncthreads();
        tot = b[kWarps];
        return b[wid] + inc - v;
    }
    __device__ __forceinline__ int min_all(int v) const {
        int* b = scan_buf();
        v = __reduce_min_sync(kFull, v);
        if ((threadIdx.x & 31) == 0) b[threadIdx.x >> 5] = v;
        __syncthreads();
        int m = b[0];
#pragma unroll
        for (int k = 1; k < kWarps; k++) m = min(m, b[k]);
        return m;
    }
    __device__ __forceinline__ int sum(int v) const {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        int* b = scan_buf();
        int w = warp_sum(v);
        if (lane == 0) b[wid] = w;
        __syncthreads();
        if (wid == 0) {
            int c = lane < kWarps ? b[lane] : 0;
            c = warp_sum(c);
            if (lane == 0) b[kWarps] = c;
        }
        __syncthreads();
        return b[kWarps];
    }
};

// --------------------------------------------------------------- list ops
// List loads: shared-memory lists with ld.shared, arena lists through L2
// (ld.global.cg: arena slots written by other SMs must not be served from a
// stale L1 line).  The space of each list is a template parameter, so no load
// carries a runtime branch or generic addressing.
__device__ __forceinline__ int lds(const int32_t* p) {
    int v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(unsigned(__cvta_generic_to_shared(p))));
    return v;
}
template <bool GL>
__device__ __forceinline__ int ld(const int32_t* p) {
    if constexpr (GL) return __ldcg(p);
    else return lds(p);
}
__device__ __forceinline__ int ldv(const int32_t* p, bool global) { return global ? __ldcg(p) : lds(p); }

// A store the host sees without synchronising (mapped pinned memory); stores
// of different CTAs may land out of order, so the host reads a lower bound.
__device__ __forceinline__ void st_relaxed_sys(int* p, int v) {
    asm volatile("st.relaxed.sys.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// calls F<ga, gb>(...) with the spaces known at compile time
#define SSPP_DISPATCH2(ga, gb, CALL) \
    ((ga) ? ((gb) ? CALL(true, true) : CALL(true, false)) : ((gb) ? CALL(false, true) : CALL(false, false)))

// first index k in [0, n) with a[k] >= x
template <bool GL>
__device__ __forceinline__ int lower_bound_t(const int32_t* a, int n, int x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (ld<GL>(a + mid) < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// number of indices common to sorted lists a and b (b is searched)
template <class G, bool GA, bool GB>
__device__ int count_common_t(const G& g, const int32_t* a, int na, const int32_t* b, int nb) {
    int e = 0;
    for (int i = g.rank(); i < na; i += G::kSize) {
        int x = ld<GA>(a + i);
        int r = lower_bound_t<GB>(b, nb, x);
        e += (r < nb && ld<GB>(b + r) == x);
    }
    return g.sum(e);
}

template <class G>
__device__ int count_common(const G& g, const int32_t* a, int na, bool ga, const int32_t* b, int nb, bool gb) {
    if (na > nb) {  // search the shorter list's elements in the longer one
        const int32_t* t = a; a = b; b = t;
        int tn = na; na = nb; nb = tn;
        bool tg = ga; ga = gb; gb = tg;
    }
#define SSPP_CC(A_, B_) count_common_t<G, A_, B_>(g, a, na, b, nb)
    return SSPP_DISPATCH2(ga, gb, SSPP_CC);
#undef SSPP_CC
}

// out = a xor b (as index sets) in one pass over both lists.  Element a[i]
// survives unless it is in b; it lands at i + rank_b(a[i]) - 2 * (cancelled
// a's before i), symmetrically for b.  Writes stay below out_cap.  Returns the
// output length and pads it to a multiple of four with INT_MAX.
// Two lower-bound searches in lockstep (x in b, y in a): two independent load
// chains per step.  Equality comes from the probe that last moved `hi` (the
// final position was probed then), so no extra dependent load is needed.
template <bool GA, bool GB>
__device__ __forceinline__ void rank2(const int32_t* a, int na, const int32_t* b, int nb, int x, bool vx, int y, bool vy,
                                      int& rx, bool& ex, int& ry, bool& ey) {
    int lo1 = 0, hi1 = vx ? nb : 0, lo2 = 0, hi2 = vy ? na : 0;
    int h1 = INT_MIN, h2 = INT_MIN;
    while (lo1 < hi1 || lo2 < hi2) {
        const bool s1 = lo1 < hi1, s2 = lo2 < hi2;
        const int m1 = (lo1 + hi1) >> 1, m2 = (lo2 + hi2) >> 1;
        const int v1 = s1 ? ld<GB>(b + m1) : 0;
        const int v2 = s2 ? ld<GA>(a + m2) : 0;
        if (s1) {
            if (v1 < x) lo1 = m1 + 1;
            else { hi1 = m1; h1 = v1; }
        }
        if (s2) {
            if (v2 < y) lo2 = m2 + 1;
            else { hi2 = m2; h2 = v2; }
        }
    }
    rx = lo1;
    ex = vx && lo1 < nb && h1 == x;
    ry = lo2;
    ey = vy && lo2 < na && h2 == y;
}

template <class G, bool GA, bool GB>
__device__ int xor_merge(const G& g, const int32_t* a, int na, const int32_t* b, int nb, int32_t* out, int out_cap,
                         int* err) {
    int carry_a = 0, carry_b = 0;
    const int n = na > nb ? na : nb;
    for (int base = 0; base < n; base += G::kSize) {
        const int i = base + g.rank();
        const bool va = i < na, vb = i < nb;
        const int x = va ? ld<GA>(a + i) : 0;
        const int y = vb ? ld<GB>(b + i) : 0;
        int ra, rb;
        bool ea, eb;
        rank2<GA, GB>(a, na, b, nb, x, va, y, vb, ra, ea, rb, eb);
        int pa, pb, ta, tb;
        g.prefix2(ea, eb, pa, pb, ta, tb);
        if (va && !ea) {
            int pos = i + ra - 2 * (carry_a + pa);
            if (pos >= 0 && pos < out_cap) out[pos] = x;
            else atomicOr(err, ERRB_BAD_INPUT);  // inputs were not strictly increasing
        }
        if (vb && !eb) {
            int pos = i + rb - 2 * (carry_b + pb);
            if (pos >= 0 && pos < out_cap) out[pos] = y;
            else atomicOr(err, ERRB_BAD_INPUT);
        }
        carry_a += ta;
        carry_b += tb;
    }
    const int out_len = na + nb - 2 * carry_a;
    const int padn = int(pad4(out_len) - out_len);
    if (g.rank() < padn && out_len + g.rank() < out_cap) out[out_len + g.rank()] = INT_MAX;
    g.sync();
    return out_len;
}

// Merge-path form of the same merge.  M = merge(a, b), a first on ties, so
// every equal pair is adjacent in M as (a[i], b[j]).  Thread t owns positions
// [tK, tK + K) of M per round: one binary search finds its split (i, j), a
// short walk emits the elements of its positions that have no equal partner
// (a pair cut by a slice boundary is dropped on both sides), and a group
// prefix sum of the per-thread counts places them.  The walk runs twice
// (count, then write) so nothing is held in registers.
template <int K, bool GA, bool GB>
__device__ __forceinline__ int path_walk(const int32_t* a, int na, const int32_t* b, int nb, int d0, int total,
                                         int32_t* out, int out_off, int out_cap, bool emit, int* err) {
    int lo = d0 - nb > 0 ? d0 - nb : 0, hi = d0 < na ? d0 : na;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (ld<GA>(a + mid - 1) <= ld<GB>(b + d0 - mid)) lo = mid;
        else hi = mid - 1;
    }
    int i = lo, j = d0 - lo, pos = d0, cnt = 0;
    const int end = d0 + K < total ? d0 + K : total;
    // b[j] partners the element just before this slice (a[i-1])
    if (pos < end && i > 0 && j < nb && ld<GA>(a + i - 1) == ld<GB>(b + j)) { j++; pos++; }
    while (pos < end) {
        const int x = i < na ? ld<GA>(a + i) : INT_MAX;
        const int y = j < nb ? ld<GB>(b + j) : INT_MAX;
        if (i < na && (j >= nb || x <= y)) {
            if (j < nb && x == y) {  // equal pair: drop both (the partner may open the next slice)
                i++;
                pos++;
                if (pos < end) { j++; pos++; }
                continue;
            }
            if (emit) {
                if (out_off + cnt < out_cap) out[out_off + cnt] = x;
                else atomicOr(err, ERRB_BAD_INPUT);
            }
            cnt++;
            i++;
        } else {
            if (emit) {
                if (out_off + cnt < out_cap) out[out_off + cnt] = y;
                else atomicOr(err, ERRB_BAD_INPUT);
            }
            cnt++;
            j++;
        }
        pos++;
    }
    return cnt;
}

template <class G, int K, bool GA, bool GB>
__device__ int xor_merge_path(const G& g, const int32_t* a, int na, const int32_t* b, int nb, int32_t* out,
                              int out_cap, int* err) {
    const int total = na + nb;
    int written = 0;
    for (int base = 0; base < total; base += G::kSize * K) {
        const int d0 = base + g.rank() * K;
        int cnt = d0 < total ? path_walk<K, GA, GB>(a, na, b, nb, d0, total, out, 0, out_cap, false, err) : 0;
        int tot;
        const int off = g.prefix_int(cnt, tot);
        if (cnt) path_walk<K, GA, GB>(a, na, b, nb, d0, total, out, written + off, out_cap, true, err);
        written += tot;
    }
    const int padn = int(pad4(written) - written);
    if (g.rank() < padn && written + g.rank() < out_cap) out[written + g.rank()] = INT_MAX;
    g.sync();
    return written;
}

template <class G>
struct PathK;
template <>
struct PathK<WarpG> {
    static constexpr int K = 4;
};
template <int T>
struct PathK<BlockG<T>> {
    static constexpr int K = 8;
};

// Rank form while both lists fit in two rounds of the group (one binary
// search per element, all independent); merge-path beyond that, where the
// per-element searches would take many rounds.
template <class G, bool GA, bool GB>
__device__ __forceinline__ int merge_t(const G& g, const int32_t* a, int na, const int32_t* b, int nb, int32_t* out,
                                       int out_cap, int* err) {
    if ((na > nb ? na : nb) <= 2 * G::kSize) return xor_merge<G, GA, GB>(g, a, na, b, nb, out, out_cap, err);
    return xor_merge_path<G, PathK<G>::K, GA, GB>(g, a, na, b, nb, out, out_cap, err);
}

template <class G>
__device__ int merge(const G& g, const int32_t* a, int na, bool ga, const int32_t* b, int nb, bool gb, int32_t* out,
                     int out_cap, int* err) {
#define SSPP_MG(A_, B_) merge_t<G, A_, B_>(g, a, na, b, nb, out, out_cap, err)
    return SSPP_DISPATCH2(ga, gb, SSPP_MG);
#undef SSPP_MG
}

// largest index of a xor b below their common top a[na-1] == b[nb-1]; -1 if none
__device__ __forceinline__ int next_low(const int32_t* a, int na, bool ga, const int32_t* b, int nb, bool gb) {
    int i = na - 2, j = nb - 2;
    while (i >= 0 && j >= 0) {
        int x = ldv(a + i, ga), y = ldv(b + j, gb);
        if (x != y) return x > y ? x : y;
        i--;
        j--;
    }
    if (i >= 0) return ldv(a + i, ga);
    if (j >= 0) return ldv(b + j, gb);
    return -1;
}

// global -> shared copy of int4 units [k0, k1) of a slot
template <class G>
__device__ __forceinline__ void copy4(const G& g, int32_t* dst, const int32_t* src, int k0, int k1) {
    const int4* s4 = reinterpret_cast<const int4*>(src);
    int4* d4 = reinterpret_cast<int4*>(dst);
    for (int k = k0 + g.rank(); k < k1; k += G::kSize) d4[k] = __ldcg(s4 + k);
}

template <class G>
__device__ __forceinline__ void store4(const G& g, int32_t* dst, const int32_t* src, int n4) {
    const int4* s4 = reinterpret_cast<const int4*>(src);
    int4* d4 = reinterpret_cast<int4*>(dst);
    for (int k = g.rank(); k < n4; k += G::kSize) d4[k] = s4[k];
}

// Bump allocation of `ints` (multiple of 4) in the arena; -1 when exhausted.
template <class G>
__device__ __forceinline__ int64_t alloc(const G& g, const ReduceArgs& A, int64_t ints) {
    unsigned long long off = 0;
    if (g.leader()) {
        off = atomicAdd(A.arena_top, (unsigned long long)ints);
        if (int64_t(off) + ints > A.arena_cap) {
            atomicOr(A.err, ERRB_CAPACITY);
            off = ~0ull;
        }
    }
    off = g.bcast64(off);
    return off == ~0ull ? -1 : int64_t(off);
}

// Working column of one group.
struct Work {
    int32_t* buf;      // current entries (shared memory, or the data part of an arena slot)
    int len;
    bool global;       // buf lives in the arena
    bool gpriv;        // buf is a private arena buffer (never published, reusable)
    int64_t gslot;     // arena slot of buf when global
    int64_t gcap;      // ints of that slot
    int64_t slot;      // arena slot of the published version
    bool dirty;        // differs from the published version
};

// Makes the working column the published version of `col`; false when the
// arena is exhausted.
template <class G>
__device__ bool publish(const G& g, const ReduceArgs& A, int col, Work& w) {
    int64_t so;
    if (w.global) {
        so = w.gslot;
        w.gpriv = false;  // published versions are immutable
    } else {
        so = alloc(g, A, slot_ints(w.len));
        if (so < 0) return false;
        store4(g, A.arena + so + kHdr, w.buf, int(pad4(w.len)) >> 2);
        if (g.leader()) cnt_add(&A.counters[CNT_PUBLISHED], (long long)slot_ints(w.len));
    }
    if (g.leader()) *reinterpret_cast<int4*>(A.arena + so) = make_int4(w.len, col, 0, 0);
    g.sync();
    if (g.leader()) {
        __threadfence();
        A.desc[col] = pack_desc(uint64_t(so), uint32_t(w.len));
    }
    w.slot = so;
    w.dirty = false;
    return true;
}

enum Outcome { OUT_OWNER, OUT_ZERO, OUT_PARKED, OUT_DEFERRED, OUT_FAIL };

// additions between two looks at a column's cleared flag
constexpr int kClearCheck = 64;

// Rounds of additions.  Every row of the working column that an earlier
// column owns may take that owner's addition, not only the lowest one: an entry
// above the final lowest row has to go anyway, and adding an earlier column is
// a left-to-right operation whichever entry it cancels.  So one round takes the
// column's top rows, one per thread (at most G::kSize of them), and adds the
// owners of all rows that have one at once:
//   - each thread reads its row's inline apparent column and pivot entry
//     together, then a published owner's header and entries: one chain of
//     dependent loads per round instead of one per addition;
//   - the addends' other entries, and the rows that take no addition (no
//     owner, a later one, or one longer than kRoundAddend entries), are
//     gathered in shared memory and sorted (64 per warp in registers, then
//     ranked across the warps' runs);
//   - entries that occur an even number of times cancel, and the rest is merged
//     into what is left of the column by ranks, as a symmetric difference.
// A round ends the loop when the lowest row itself takes no addition (it must
// be claimed, or its owner goes through the general path) or the column is
// empty or below the band.
// Bound: latency (about a dozen barriers and two or three dependent loads per
// round); the point is the number of rounds.  On the 64^3 lower-star grid the
// longest chain of 3,725 single additions takes 123 rounds of 32 rows with 3,807
// additions, 40 rounds of 128 with 4,339.
constexpr int kRoundAddend = 32;  // longest published addend taken in a round

// two values per lane, element 2 * lane + {0, 1} of 64: ascending bitonic sort
__device__ __forceinline__ void warp_sort64(int& x0, int& x1) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 64; k <<= 1) {
        const bool up = ((2 * lane) & k) == 0;
#pragma unroll
        for (int j = k >> 1; j > 1; j >>= 1) {
            const int y0 = __shfl_xor_sync(kFull, x0, j >> 1), y1 = __shfl_xor_sync(kFull, x1, j >> 1);
            const bool keep_min = (((2 * lane) & j) == 0) == up;
            x0 = keep_min ? min(x0, y0) : max(x0, y0);
            x1 = keep_min ? min(x1, y1) : max(x1, y1);
        }
        const int lo = min(x0, x1), hi = max(x0, x1);
        x0 = up ? lo : hi;
        x1 = up ? hi : lo;
    }
}

// one value per lane, ascending
__device__ __forceinline__ void warp_sort32(int& x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int y = __shfl_xor_sync(kFull, x, j);
            x = (((lane & j) == 0) == ((lane & k) == 0)) ? min(x, y) : max(x, y);
        }
    }
}

// Shared memory of a group's rounds besides its column buffers: the sorted
// entries and, per entry, the counts of kept and cancelled entries before it.
template <class G>
struct RoundMem {
    static constexpr int kEntries = 2 * G::kSize;  // entries of one round
    int32_t s[kEntries];
    int32_t pre[kEntries + 1];  // kept before | cancelled before << 15 | cancels << 30
};

// Returns the number of rounds done, or -1 after a failed self-check; *stop is
// set when the column was cleared meanwhile.  The column moves between w.buf and
// `other`; sp holds the gathered entries.
template <class G>
__device__ int round_adds(const G& g, const ReduceArgs& A, int32_t minrow, int col, Work& w, int32_t* other,
                          int32_t* sp, RoundMem<G>& R, int& L, uint64_t& e, long long& adds, long long& add_ints,
                          bool* cleared) {
    constexpr int kS = G::kSize, kWarps = kS / 32, kM = RoundMem<G>::kEntries;
    const int rank = g.rank(), lane = threadIdx.x & 31, wid = kWarps > 1 ? rank >> 5 : 0;
    const int mlimit = min(kM, A.cap);
    int32_t* a = w.buf;
    int32_t* out = other;
    int n = w.len, Lc = L, rounds = 0, n_inline = 0, n_slot = 0;
    bool fail = false;
    uint64_t ev = kNoOwner;
    while (n > 0 && Lc >= minrow) {
        // ---- the top rows and their owners
        const int idx = n - 1 - rank;
        const int r = idx >= 0 ? lds(a + idx) : -1;
        const bool valid = r >= 0 && r >= minrow && r < A.ncols;
        int4 q = make_int4(-1, 0, 0, 0);
        ev = kNoOwner;
        unsigned clr = 0;
        if (valid) {
            q = __ldg(A.app + r);
            ev = ld_acquire_u64(A.pivot + r);
        }
        if (rank == 0) clr = ld_acquire_u8(A.cleared + col);
        const bool inl = q.x >= 0;
        bool own = inl;
        int cnt = inl ? q.x : 0;
        const int32_t* src = nullptr;
        if (!inl && pv_col(ev) < col && pv_slot(ev) + 2 * kHdr <= uint64_t(A.arena_cap)) {
            src = A.arena + pv_slot(ev);
            const int4 h = __ldcg(reinterpret_cast<const int4*>(src));
            q = __ldcg(reinterpret_cast<const int4*>(src) + 1);  // the first entries (a slot without any is not an owner's)
            if (h.x >= 1 && h.x <= kRoundAddend && h.y == pv_col(ev) &&
                int64_t(pv_slot(ev)) + slot_ints(h.x) <= A.arena_cap) {
                own = true;
                cnt = h.x - 1;
            }
        } else if (inl) {
            q = make_int4(q.y, q.z, q.w, 0);
        }
        // ---- how many rows this round takes: what they leave must fit the buffers
        const int c = idx >= 0 ? (own ? cnt : 1) : 0;
        int tot;
        const int pre = g.prefix_int(c, tot);
        const bool ok = idx >= 0 && pre + c <= mlimit && idx + pre + c <= A.cap && (rank > 0 || own);
        const int K = g.min_all(clr ? -1 : (ok ? kS : rank));
        if (K <= 0) {
            *cleared = K < 0;
            break;
        }
        // ---- gather
        if (rank < K) {
            if (!own) {
                sp[pre] = r;
            } else {
                if (cnt > 0) sp[pre] = q.x;
                if (cnt > 1) sp[pre + 1] = q.y;
                if (cnt > 2) sp[pre + 2] = q.z;
                if (cnt > 3) {
                    sp[pre + 3] = q.w;
                    for (int k = 4; k < cnt; k++) sp[pre + k] = __ldcg(src + kHdr + k);
                }
                n_inline += inl;
                n_slot += !inl;
            }
            if (rank == K - 1) R.pre[kM] = pre + c;  // entries of the rows taken
        }
        g.sync();
        const int m = lds(R.pre + kM);
        const int nc = n - K;
        if (kWarps == 1 && nc == 0 && m <= 32) {
            // a warp's short column, all of it taken: one entry per lane, sorted and
            // cancelled in registers
            int x = lane < m ? lds(sp + lane) : INT_MAX;
            warp_sort32(x);
            const int up = __shfl_up_sync(kFull, x, 1);
            const unsigned in = m == 32 ? kFull : (1u << m) - 1;
            const unsigned head = __ballot_sync(kFull, lane < m && (lane == 0 || x != up));
            // a run goes on to the next head (or the end); odd runs keep one entry
            const unsigned later = lane == 31 ? 0u : head & (kFull << (lane + 1));
            const int end = later ? __ffs(later) - 1 : __popc(in);
            const unsigned keep = __ballot_sync(kFull, ((head >> lane) & 1) && ((end - lane) & 1));
            const int nn = __popc(keep), at = __popc(keep & lanemask_lt());
            if ((keep >> lane) & 1) out[at] = x;
            if (lane < int(pad4(nn) - nn)) out[nn + lane] = INT_MAX;
            const int nl = keep ? __shfl_sync(kFull, x, 31 - __clz(keep)) : -1;
            __syncwarp();
            add_ints += n + m + nn;
            n = nn;
            int32_t* t = a;
            a = out;
            out = t;
            rounds++;
            if (nl >= Lc) {
                if (g.leader()) atomicOr(A.err, ERRB_CHECK);
                fail = true;
                break;
            }
            Lc = nl;
            continue;
        }
        // ---- sort
        const int i0 = 2 * rank;
        int x0 = INT_MAX, x1 = INT_MAX;
        if (kWarps == 1 || 64 * wid < m) {
            if (i0 < m) x0 = lds(sp + i0);
            if (i0 + 1 < m) x1 = lds(sp + i0 + 1);
            warp_sort64(x0, x1);
            if (kWarps == 1) {
                R.s[i0] = x0;
                R.s[i0 + 1] = x1;
            }
        }
        if constexpr (kWarps > 1) {
            const int runs = (m + 63) >> 6;
            if (runs == 1) {
                if (wid == 0) {
                    R.s[i0] = x0;
                    R.s[i0 + 1] = x1;
                }
            } else {
                __syncthreads();  // every gathered entry is in registers
                if (wid < runs) {
                    if (i0 < mlimit) sp[i0] = x0;
                    if (i0 + 1 < mlimit) sp[i0 + 1] = x1;
                }
                __syncthreads();
                if (wid < runs) {
                    // ranks over the other runs (equal entries of earlier runs come first); the last
                    // run's padding stays behind every entry
                    int p0 = 2 * lane, p1 = 2 * lane + 1;
                    for (int k = 0; k < runs; k++) {
                        if (k == wid) continue;
                        const int len = min(64, m - 64 * k);
                        const int bump = k < wid ? 1 : 0;
                        if (x0 != INT_MAX) p0 += lower_bound_t<false>(sp + 64 * k, len, x0 + bump);
                        if (x1 != INT_MAX) p1 += lower_bound_t<false>(sp + 64 * k, len, x1 + bump);
                    }
                    if (x0 != INT_MAX) R.s[p0] = x0;
                    if (x1 != INT_MAX) R.s[p1] = x1;
                }
            }
        }
        g.sync();
        // ---- parity of each entry, and whether the rest of the column holds it
        int kept0 = 0, canc0 = 0, kept1 = 0, canc1 = 0, rc0 = 0, rc1 = 0;
        auto look = [&](int i, int& x, int& rc, int& kept, int& canc) {
            if (i >= m) return;
            x = lds(R.s + i);
            if (i > 0 && lds(R.s + i - 1) == x) return;
            int j = i + 1;
            while (j < m && lds(R.s + j) == x) j++;
            if (((j - i) & 1) == 0) return;
            rc = lower_bound_t<false>(a, nc, x);
            canc = rc < nc && lds(a + rc) == x;
            kept = !canc;
        };
        look(i0, x0, rc0, kept0, canc0);
        look(i0 + 1, x1, rc1, kept1, canc1);
        int tp;
        const int pp = g.prefix_int((kept0 + kept1) | ((canc0 + canc1) << 15), tp);
        const int pp1 = pp + (kept0 | (canc0 << 15));
        if (i0 < m) R.pre[i0] = pp | (canc0 << 30);
        if (i0 + 1 < m) R.pre[i0 + 1] = pp1 | (canc1 << 30);
        const int kept_all = tp & 0x7fff, canc_all = tp >> 15;
        // self-check on every store: positions stay inside the buffer (sorted lists never leave it)
        auto put = [&](int pos, int x) {
            if (unsigned(pos) < unsigned(A.cap)) out[pos] = x;
            else atomicOr(A.err, ERRB_CHECK);
        };
        if (kept0) put(rc0 - (pp >> 15) + (pp & 0x7fff), x0);
        if (kept1) put(rc1 - (pp1 >> 15) + (pp1 & 0x7fff), x1);
        g.sync();
        // ---- the rest of the column, shifted by the entries kept and cancelled below each
        const int s0 = m > 0 ? lds(R.s) : INT_MAX;
        for (int j = rank; j < nc; j += kS) {
            const int y = lds(a + j);
            if (y < s0) {
                out[j] = y;
                continue;
            }
            const int p = lower_bound_t<false>(R.s, m, y);
            if (p == m) {
                put(j - canc_all + kept_all, y);
            } else {
                const int v = lds(R.pre + p);
                if (!(v >> 30) || lds(R.s + p) != y) put(j - ((v >> 15) & 0x7fff) + (v & 0x7fff), y);
            }
        }
        const int nn = nc - canc_all + kept_all;
        if (rank < int(pad4(nn) - nn)) out[nn + rank] = INT_MAX;
        g.sync();
        add_ints += n + m + nn;
        n = nn;
        int32_t* t = a;
        a = out;
        out = t;
        rounds++;
        const int nl = n > 0 ? lds(a + n - 1) : -1;
        if (nl >= Lc) {  // self-check: the lowest row only moves down
            if (g.leader()) atomicOr(A.err, ERRB_CHECK);
            fail = true;
            break;
        }
        Lc = nl;
    }
    if (fail) return -1;
    e = g.bcast64(ev);  // the entry of the row the rounds stopped at
    if (rounds > 0) {
        w.buf = a;
        w.len = n;
        w.dirty = true;
        L = Lc;
        const int ni = g.sum(n_inline), ns = g.sum(n_slot);
        adds += ni + ns;
        if (g.leader() && kWarps > 1) {
            cnt_add(&A.counters[CNT_FAST_INLINE], ni);
            cnt_add(&A.counters[CNT_FAST_SLOT], ns);
        }
    }
    return rounds;
}

// Reduces column `col` until it owns its lowest row, becomes zero, or its
// lowest row drops below the band.  With `defer`, a column whose entries (or
// whose next addend or sum) exceed the shared capacity is published and
// returned as OUT_DEFERRED for the heavy tier; without it such columns continue
// in arena buffers.  *displaced receives the owner this column displaced (-1
// if none).  sp holds kHdr + cap ints (staged addend with its header).
template <class G>
__device__ Outcome reduce_column(const G& g, const ReduceArgs& A, const Band& band, int col, int32_t* sw0,
                                 int32_t* sw1, int32_t* sp, RoundMem<G>& rm, bool defer, int* displaced) {
    const int32_t minrow = band.minrow;
    *displaced = -1;
    uint64_t d = 0;
    if (g.leader()) d = ld_cg_u64(A.desc + col);
    d = g.bcast64(d);
    Work w;
    w.len = int(desc_len(d));
    w.slot = int64_t(desc_off(d));
    w.dirty = false;
    if (w.slot + slot_ints(w.len) > A.arena_cap) {  // self-check: descriptor inside the arena
        if (g.leader()) atomicOr(A.err, ERRB_CHECK);
        return OUT_FAIL;
    }
    if (w.len <= A.cap) {
        copy4(g, sw0, A.arena + w.slot + kHdr, 0, int(pad4(w.len)) >> 2);
        g.sync();
        w.buf = sw0;
        w.global = false;
        w.gslot = 0;
    } else if (defer) {
        return OUT_DEFERRED;
    } else {
        w.buf = A.arena + w.slot + kHdr;
        w.global = true;
        w.gslot = w.slot;
    }
    w.gpriv = false;
    w.gcap = 0;
    // a private arena buffer freed by the last merge, reused by the next one
    // that does not fit in shared memory (chains of long sums then need two
    // buffers, not one per addition)
    int64_t spare = -1, spare_cap = 0;
    long long adds = 0, add_ints = 0;
    Outcome res = OUT_FAIL;
    int L = w.len ? ldv(w.buf + w.len - 1, w.global) : -1;
    uint64_t e = kNoOwner;
    if (L >= A.ncols) {  // self-check: row index in range
        if (g.leader()) atomicOr(A.err, ERRB_CHECK);
        return OUT_FAIL;
    }
    // inline apparent column of row r (every thread loads it: one transaction per warp)
    auto app_of = [&](int r) { return (r >= 0 && r >= minrow) ? __ldg(A.app + r) : make_int4(-1, 0, 0, 0); };
    if (w.global && L >= minrow) {
        if (g.leader()) e = ld_acquire_u64(A.pivot + L);
        e = g.bcast64(e);
    }
    // speculative first staging round: header + as many entries as one pass of the group reads
    const int first4 = min(G::kSize, (kHdr + A.cap) >> 2);
    int next_check = 0;
    for (int iter = 0;; iter++) {
        bool clr = false;
        if (!w.global) {  // rounds of additions; they end with the entry of the row they stop at
            const int done = round_adds(g, A, minrow, col, w, w.buf == sw0 ? sw1 : sw0, sp, rm, L, e, adds, add_ints,
                                        &clr);
            if (done < 0) break;
            iter += done;
        } else if (iter >= next_check) {
            next_check = iter + kClearCheck;
            int c = 0;
            if (g.leader()) c = int(ld_acquire_u8(A.cleared + col));
            clr = g.bcast(c) != 0;
        }
        // Cleared meanwhile: a column of the next higher dimension claimed this
        // column's row, so the column is positive and zero once reduced (and a row
        // never loses its owner, so it stays cleared).  It owns no row now (a claim
        // ends the reduction), so it stops here as zero.
        if (clr) {
            if (g.leader()) {
                A.desc[col] = pack_desc(0, 0);
                A.low[col] = -1;
            }
            res = OUT_ZERO;
            break;
        }
        if (w.len == 0) {
            if (g.leader()) {
                A.desc[col] = pack_desc(0, 0);
                A.low[col] = -1;
            }
            res = OUT_ZERO;
            break;
        }
        if (iter > kMaxMergesPerColumn) {
            if (g.leader()) atomicOr(A.err, ERRB_TIMEOUT);
            break;
        }
        if (L < minrow) {
            if (w.dirty && !publish(g, A, col, w)) break;
            if (g.leader()) A.low[col] = L;
            res = OUT_PARKED;
            break;
        }
        const int p = pv_col(e);
        if (p > col) {  // no owner, or a larger one: claim the row
            if (w.dirty && !publish(g, A, col, w)) break;
            uint64_t old = 0;
            if (g.leader()) {
                // the column's final state goes out before the claim: a group
                // that later displaces it writes its own state after this one
                const uint8_t was = A.state[col];
                A.low[col] = L;
                A.state[col] = ST_OWNER;
                __threadfence();
                old = atomicCAS(reinterpret_cast<unsigned long long*>(A.pivot + L), (unsigned long long)e,
                                (unsigned long long)pv_pack(col, uint64_t(w.slot)));
                if (old != e) A.state[col] = was;  // not claimed: still in progress here
            }
            old = g.bcast64(old);
            if (old == e) {
                if (g.leader()) {
                    if (e == kNoOwner) A.cleared[L] = 1;  // twist clearing of the positive row column
                    else cnt_add(&A.counters[CNT_DISPLACED], 1ll);
                }
                *displaced = (e == kNoOwner) ? -1 : p;
                res = OUT_OWNER;
                break;
            }
            e = old;  // someone else changed the owner; look again
            continue;
        }
        // long chains of the warp tier: once the step's window is handed out they
        // only hold up the step's tail, and the CTA tier continues them on a side
        // stream while the next step runs (iter counts rounds here)
        if (defer && band.drain_ctr && A.light_chain > 0 && iter >= A.light_chain) {
            int drained = 0;
            if (g.leader()) drained = __ldcg(band.drain_ctr) >= band.drain_total;
            if (g.bcast(drained)) {
                if (w.dirty && !publish(g, A, col, w)) break;
                res = OUT_DEFERRED;
                break;
            }
        }
        // add the owner's version (p < col, same lowest row): stage header + entries
        if (pv_slot(e) + kHdr > uint64_t(A.arena_cap)) {  // self-check: entry inside the arena
            if (g.leader()) atomicOr(A.err, ERRB_CHECK);
            break;
        }
        const int32_t* src = A.arena + pv_slot(e);
        const int4 apc = app_of(L);
        int plen;
        if (apc.x >= 0) {  // apparent owner: its entries are inline, no arena read
            plen = apc.x + 1;
            if (g.leader()) {
                sp[kHdr] = apc.y;
                sp[kHdr + 1] = apc.z;
                sp[kHdr + 2] = apc.w;
                sp[kHdr + 3] = INT_MAX;
                sp[kHdr + apc.x] = L;
            }
            g.sync();
        } else {
            copy4(g, sp, src, 0, first4);
            g.sync();
            plen = sp[0];
            if (plen < 1 || plen > int(kMaxColLen) || sp[1] != p ||
                int64_t(pv_slot(e)) + slot_ints(plen) > A.arena_cap) {  // self-check: header of the owner's version
                if (g.leader()) atomicOr(A.err, ERRB_CHECK);
                break;
            }
        }
        const int32_t* pb;
        bool pg;
        if (apc.x >= 0) {
            pb = sp + kHdr;
            pg = false;
        } else if (plen <= A.cap) {
            const int n4 = (kHdr + int(pad4(plen))) >> 2;
            if (n4 > first4) {
                copy4(g, sp, src, first4, n4);
                g.sync();
            }
            pb = sp + kHdr;
            pg = false;
        } else if (defer) {
            if (w.dirty && !publish(g, A, col, w)) break;
            res = OUT_DEFERRED;
            break;
        } else {
            pb = src + kHdr;
            pg = true;
        }
        if (g.leader() && (plen == 0 || ldv(pb + plen - 1, pg) != L)) atomicOr(A.err, ERRB_BAD_INPUT);
        // the next lowest row is known before the merge: request its pivot entry now
        const int L2 = next_low(w.buf, w.len, w.global, pb, plen, pg);
        if (L2 >= A.ncols) {  // self-check: row index in range
            if (g.leader()) atomicOr(A.err, ERRB_CHECK);
            break;
        }
        // the group's last thread takes the entry: in short merges it holds no
        // element, so its acquire load completes while the others merge
        uint64_t pref = kNoOwner;
        if (g.rank() == G::kSize - 1 && L2 >= minrow && L2 >= 0) pref = ld_acquire_u64(A.pivot + L2);
        int out_len;
        const int bound = w.len + plen - 2;
        if (bound <= A.cap) {
            int32_t* dst = (w.global || w.buf == sw1) ? sw0 : sw1;
            out_len = merge(g, w.buf, w.len, w.global, pb, plen, pg, dst, A.cap, A.err);
            if (w.global && w.gpriv) {
                spare = w.gslot;
                spare_cap = w.gcap;
            }
            w.buf = dst;
            w.global = false;
        } else {
            const int common = count_common(g, w.buf, w.len, w.global, pb, plen, pg);
            out_len = w.len + plen - 2 * common;
            if (out_len > int(kMaxColLen)) {
                if (g.leader()) atomicOr(A.err, ERRB_LEN);
                break;
            }
            if (out_len <= A.cap) {
                int32_t* dst = (w.global || w.buf == sw1) ? sw0 : sw1;
                merge(g, w.buf, w.len, w.global, pb, plen, pg, dst, A.cap, A.err);
                if (w.global && w.gpriv) {
                    spare = w.gslot;
                    spare_cap = w.gcap;
                }
                w.buf = dst;
                w.global = false;
            } else if (defer) {
                if (w.dirty && !publish(g, A, col, w)) break;
                res = OUT_DEFERRED;
                break;
            } else {
                const int64_t need = slot_ints(out_len);
                int64_t so, cap_so;
                if (spare >= 0 && spare_cap >= need) {
                    so = spare;
                    cap_so = spare_cap;
                    spare = -1;
                } else {
                    cap_so = (need + (need >> 1) + 3) & ~int64_t(3);  // slack for a growing sum
                    so = alloc(g, A, cap_so);
                    if (so < 0) break;
                    if (g.leader()) cnt_add(&A.counters[CNT_PUBLISHED], (long long)cap_so);
                }
                merge(g, w.buf, w.len, w.global, pb, plen, pg, A.arena + so + kHdr, int(pad4(out_len)), A.err);
                if (w.global && w.gpriv) {
                    spare = w.gslot;
                    spare_cap = w.gcap;
                }
                w.buf = A.arena + so + kHdr;
                w.global = true;
                w.gpriv = true;
                w.gslot = so;
                w.gcap = cap_so;
            }
        }
        adds++;
        add_ints += w.len + plen + out_len;
        w.len = out_len;
        w.dirty = true;
        L = L2;
        e = g.bcast64_last(pref);
    }
    if (g.leader() && adds) {
        cnt_add(&A.counters[CNT_ADDITIONS], adds);
        cnt_add(&A.counters[CNT_ADD_INTS], add_ints);
        if (!defer) cnt_add(&A.counters[CNT_HEAVY_ADDS], adds);
    }
    return res;
}

// Final state of a column after reduce_column; returns false on failure.
template <class G>
__device__ __forceinline__ bool settle(const G& g, const ReduceArgs& A, int col, Outcome o) {
    if (g.leader()) {
        switch (o) {
            case OUT_OWNER: break;  // written before the claim
            case OUT_ZERO: A.state[col] = ST_ZERO; break;
            case OUT_DEFERRED: {
                A.state[col] = ST_HEAVY;
                int i = atomicAdd(A.pool_tail, 1);
                if (i < A.pool_cap) A.heavy[i] = col;
                else atomicOr(A.err, ERRB_CAPACITY);  // pool full: the run is repeated with a larger one
                break;
            }
            default: __threadfence(); st_release_u8(A.state + col, ST_ACTIVE); break;  // parked / failed
        }
    }
    g.sync();
    return o != OUT_FAIL;
}

// The last warp-tier block of a step to finish marks the step's slice of the
// CTA-tier pool: it ends at the pool tail, where the next step's slice starts
// (every deferral of the step is appended before its block finishes).
__device__ void light_block_done(const ReduceArgs& A) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(A.ctr + 4, 1) == int(gridDim.x) - 1) {
            __threadfence();
            const int t = ld_acquire(A.pool_tail);
            A.ctr[2] = t;
            if (A.ctr_next) A.ctr_next[1] = t;
        }
    }
}

// Light tier.  Most columns a step lists are tiny: at 64^3, 99% of them hold at
// most 8 entries throughout and need one round of additions (two to four
// addends) before they claim a row.  A warp therefore reduces four columns at a
// time, eight lanes each with one entry per lane (largest first), in lockstep:
// every pass of the loop refills idle groups, reads all groups' rows' inline
// columns and pivot entries together, sorts what the addends leave (at most 16
// entries a group) in registers, and publishes and claims for the groups that
// reached a row to claim.  The dependent loads and the instructions of a pass
// are shared by four columns.  A column that outgrows its group (more than 8
// entries, more than 16 gathered, or a long addend) is published and finished
// by the whole warp (reduce_column).
constexpr int kGroup = 8;            // lanes and entries of a tiny column
constexpr int kGroupGather = 16;     // entries a tiny column's round may gather

// two values per lane over 8 lanes, element 2 * (lane & 7) + {0, 1}: descending bitonic sort of 16
__device__ __forceinline__ void group_sort16(int& x0, int& x1) {
    const int gl = threadIdx.x & (kGroup - 1);
#pragma unroll
    for (int k = 2; k <= 16; k <<= 1) {
        const bool down = ((2 * gl) & k) == 0;
#pragma unroll
        for (int j = k >> 1; j > 1; j >>= 1) {
            const int y0 = __shfl_xor_sync(kFull, x0, j >> 1), y1 = __shfl_xor_sync(kFull, x1, j >> 1);
            const bool keep_max = (((2 * gl) & j) == 0) == down;
            x0 = keep_max ? max(x0, y0) : min(x0, y0);
            x1 = keep_max ? max(x1, y1) : min(x1, y1);
        }
        const int lo = min(x0, x1), hi = max(x0, x1);
        x0 = down ? hi : lo;
        x1 = down ? lo : hi;
    }
}

// bit i of an 8-bit mask to bit 2i
__device__ __forceinline__ unsigned spread8(unsigned b) {
    b = (b | (b << 4)) & 0x0f0fu;
    b = (b | (b << 2)) & 0x3333u;
    return (b | (b << 1)) & 0x5555u;
}

// At least 6 blocks per SM (80 registers, 20 bytes spilled).  64^3, one block per
// dimension: 8 / 7 / 6 / 5 blocks 1,228 / 1,192 / 1,223 / 1,250 us of reduction; small
// inputs prefer few blocks (1,200-point cloud 396 / 375 / 360 / 356 us).
constexpr int kLightMinBlocks = 6;
__global__ void __launch_bounds__(128, kLightMinBlocks) k_reduce_light(ReduceArgs A) {
    extern __shared__ __align__(16) int32_t smem[];
    __shared__ RoundMem<WarpG> s_rm[4];
    RoundMem<WarpG>& rm = s_rm[threadIdx.x >> 5];
    WarpG g;
    const int lane = g.rank(), gl = lane & (kGroup - 1), lead = lane & ~(kGroup - 1);
    int32_t* sw0 = smem + size_t(threadIdx.x >> 5) * (3 * A.cap + kHdr);
    int32_t* gbuf = rm.s + 2 * lead;  // 16 entries per group
    const int count = A.listed;
    const int warps = gridDim.x * (blockDim.x >> 5);
    // list entries a warp takes at a time: enough to keep its groups busy, few enough to share a short list
    const int chunk = max(4, min(32, count / (2 * warps)));
    const Band band{INT32_MIN, A.ctr, count};  // the whole dimension is one block
    long long n_adds = 0, n_ints = 0, n_pub = 0;
    int n_disp = 0;
    // the chunk: lane i holds its i-th column and descriptor; avail marks the lanes not handed out yet
    int ck_col = -1;
    uint64_t ck_desc = 0;
    unsigned avail = 0;
    bool more = true, stop = false;
    // the group's column: entries v (descending, -1 beyond n), the arena slot of its published version
    int col = -1, n = 0, v = -1;
    int64_t slot = 0;
    bool dirty = false, displaced = false;
    while (!stop) {
        // ---- refill
        unsigned idle = __ballot_sync(kFull, col < 0 && gl == 0);
        if (idle && !avail && more) {
            int base = 0;
            if (lane == 0) base = atomicAdd(A.ctr, chunk);
            base = __shfl_sync(kFull, base, 0);
            more = base < count;
            bool run = false;
            if (lane < chunk && base + lane < count) {
                ck_col = A.active[base + lane];
                ck_desc = ld_cg_u64(A.desc + ck_col);
                run = ld_acquire_u8(A.state + ck_col) == ST_ACTIVE && !ld_acquire_u8(A.cleared + ck_col);
            }
            avail = __ballot_sync(kFull, run);
            if (!avail && more) continue;
        }
        if (idle == 0x01010101u && !avail) break;
        bool fresh = displaced;
        int src = -1;
#pragma unroll
        for (int q = 0; q < 32; q += kGroup) {
            if (((idle >> q) & 1) && avail) {
                const int s = __ffs(avail) - 1;
                avail &= avail - 1;
                if (lead == q) src = s;
            }
        }
        uint64_t d = __shfl_sync(kFull, (unsigned long long)ck_desc, src & 31);
        const int c2 = __shfl_sync(kFull, ck_col, src & 31);
        if (src >= 0) {
            col = c2;
            fresh = true;
        } else if (displaced) {
            d = ld_cg_u64(A.desc + col);
        }
        displaced = false;
        bool bad = false, ovf = false;
        if (fresh) {
            n = int(desc_len(d));
            slot = int64_t(desc_off(d));
            dirty = false;
            v = -1;
            bad = slot + slot_ints(n) > A.arena_cap;  // self-check: descriptor inside the arena
            ovf = n > kGroup;
            if (!bad && !ovf && gl < n) v = __ldcg(A.arena + slot + kHdr + n - 1 - gl);
        }
        int L = __shfl_sync(kFull, v, lead);
        bad = bad || L >= A.ncols;  // self-check: row index in range
        if (__any_sync(kFull, bad)) {
            if (bad && gl == 0) atomicOr(A.err, ERRB_CHECK);
            stop = true;
            break;
        }
        // ---- rows' owners
        const bool act = col >= 0 && !ovf && n > 0;
        int4 q4 = make_int4(-1, 0, 0, 0);
        uint64_t ev = kNoOwner;
        unsigned clr = 0;
        if (act && gl < n) {
            q4 = __ldg(A.app + v);
            ev = ld_acquire_u64(A.pivot + v);
            if (gl == 0) clr = ld_acquire_u8(A.cleared + col);
        }
        bool own = q4.x >= 0;
        int cnt = own ? q4.x : 1;  // a row without an addend stays
        const int32_t* as = nullptr;
        if (!own && pv_col(ev) < col && pv_slot(ev) + 2 * kHdr <= uint64_t(A.arena_cap)) {
            as = A.arena + pv_slot(ev);
            const int4 h = __ldcg(reinterpret_cast<const int4*>(as));
            q4 = __ldcg(reinterpret_cast<const int4*>(as) + 1);
            if (h.x >= 1 && h.x <= kGroupGather && h.y == pv_col(ev) &&
                int64_t(pv_slot(ev)) + slot_ints(h.x) <= A.arena_cap) {
                own = true;
                cnt = h.x - 1;
            }
        } else if (own) {
            q4 = make_int4(q4.y, q4.z, q4.w, 0);
        }
        if (!act || gl >= n) cnt = 0;
        int pre = cnt;
#pragma unroll
        for (int o = 1; o < kGroup; o <<= 1) {
            const int t = __shfl_up_sync(kFull, pre, o, kGroup);
            if (gl >= o) pre += t;
        }
        const int m = __shfl_sync(kFull, pre, lead + kGroup - 1);
        pre -= cnt;
        const bool low_own = __shfl_sync(kFull, own ? 1 : 0, lead) != 0;
        const uint64_t e = __shfl_sync(kFull, (unsigned long long)ev, lead);
        const bool cleared = __shfl_sync(kFull, clr, lead) != 0;
        const bool claim = act && !cleared && !low_own && pv_col(e) > col;
        const bool round = act && !cleared && low_own && m <= kGroupGather;
        ovf = ovf || (act && !cleared && !claim && !round);
        // ---- one round for the groups whose lowest row has an owner
        if (__any_sync(kFull, round)) {
            const unsigned owned = __ballot_sync(kFull, round && own && gl < n);
            if (round && gl < n) {
                if (!own) {
                    gbuf[pre] = v;
                } else {
                    if (cnt > 0) gbuf[pre] = q4.x;
                    if (cnt > 1) gbuf[pre + 1] = q4.y;
                    if (cnt > 2) gbuf[pre + 2] = q4.z;
                    if (cnt > 3) {
                        gbuf[pre + 3] = q4.w;
                        for (int k = 4; k < cnt; k++) gbuf[pre + k] = __ldcg(as + kHdr + k);
                    }
                }
            }
            __syncwarp();
            int x0 = round && 2 * gl < m ? lds(gbuf + 2 * gl) : -1;
            int x1 = round && 2 * gl + 1 < m ? lds(gbuf + 2 * gl + 1) : -1;
            group_sort16(x0, x1);
            // runs of equal entries: odd ones keep one entry
            const int mr = round ? m : 0;
            const int up = __shfl_up_sync(kFull, x1, 1);
            const bool h0 = 2 * gl < mr && (gl == 0 || x0 != up), h1 = 2 * gl + 1 < mr && x1 != x0;
            const unsigned heads = spread8((__ballot_sync(kFull, h0) >> lead) & 0xffu) |
                                   (spread8((__ballot_sync(kFull, h1) >> lead) & 0xffu) << 1) | (1u << mr);
            const bool k0 = h0 && (__ffs(heads >> (2 * gl + 1)) & 1), k1 = h1 && (__ffs(heads >> (2 * gl + 2)) & 1);
            const unsigned b0 = (__ballot_sync(kFull, k0) >> lead) & 0xffu, b1 = (__ballot_sync(kFull, k1) >> lead) & 0xffu;
            const int nn = __popc(b0) + __popc(b1);
            const unsigned lt = (1u << gl) - 1;
            const int p0 = __popc(b0 & lt) + __popc(b1 & lt), p1 = p0 + (k0 ? 1 : 0);
            __syncwarp();  // every gathered entry has been read
            if (round && nn <= kGroup) {
                if (k0) gbuf[p0] = x0;
                if (k1) gbuf[p1] = x1;
            }
            __syncwarp();
            if (round) {
                if (nn <= kGroup) {
                    if (gl == 0) {
                        n_adds += __popc((owned >> lead) & 0xffu);
                        n_ints += n + m + nn;
                    }
                    n = nn;
                    v = gl < nn ? lds(gbuf + gl) : -1;
                    dirty = true;
                } else {
                    ovf = true;
                }
            }
            const int nl = __shfl_sync(kFull, v, lead);
            bad = round && !ovf && nl >= L;  // self-check: the lowest row only moves down
            if (__any_sync(kFull, bad)) {
                if (bad && gl == 0) atomicOr(A.err, ERRB_CHECK);
                stop = true;
                break;
            }
            L = nl;
        }
        // ---- what the group's column has come to
        const bool zero = col >= 0 && !ovf && (n == 0 || cleared);
        const bool pub = dirty && (claim || ovf);
        if (__any_sync(kFull, pub)) {  // one allocation for all groups
            const int want = pub && gl == 0 ? int(slot_ints(n)) : 0;
            const int inc = warp_inclusive_scan(want);
            const int tot = __shfl_sync(kFull, inc, 31);
            unsigned long long off = 0;
            if (lane == 0) {
                off = atomicAdd(A.arena_top, (unsigned long long)tot);
                if (int64_t(off) + tot > A.arena_cap) {
                    atomicOr(A.err, ERRB_CAPACITY);
                    off = ~0ull;
                }
                n_pub += tot;
            }
            off = __shfl_sync(kFull, off, 0);
            if (off == ~0ull) {
                stop = true;
                break;
            }
            const int64_t so = int64_t(off) + __shfl_sync(kFull, inc - want, lead);
            if (pub) {
                slot = so;
                dirty = false;
                if (gl < n) A.arena[so + kHdr + n - 1 - gl] = v;
                else if (gl < int(pad4(n))) A.arena[so + kHdr + gl] = INT_MAX;
                if (gl == 0) {
                    *reinterpret_cast<int4*>(A.arena + so) = make_int4(n, col, 0, 0);
                    A.desc[col] = pack_desc(uint64_t(so), uint32_t(n));
                }
            }
            __syncwarp();
        }
        int next = -1;  // leader: the owner the claim displaced; col when the claim failed
        if (gl == 0 && (claim || zero)) {
            if (claim) {
                // the column's final state goes out before the claim: a group
                // that later displaces it writes its own state after this one
                A.low[col] = L;
                A.state[col] = ST_OWNER;
                __threadfence();
                const uint64_t old = atomicCAS(reinterpret_cast<unsigned long long*>(A.pivot + L), (unsigned long long)e,
                                               (unsigned long long)pv_pack(col, uint64_t(slot)));
                if (old != e) {
                    A.state[col] = ST_ACTIVE;
                    next = col;  // someone else changed the owner; look again
                } else if (e == kNoOwner) {
                    A.cleared[L] = 1;  // twist clearing of the positive row column
                } else {
                    n_disp++;
                    next = pv_col(e);
                }
            } else {
                A.desc[col] = pack_desc(0, 0);
                A.low[col] = -1;
                A.state[col] = ST_ZERO;
            }
        }
        next = __shfl_sync(kFull, next, lead);
        if (claim) {
            if (next != col) {
                col = next;  // idle, or the displaced owner
                displaced = next >= 0;
            }
        } else if (zero) {
            col = -1;
        }
        // ---- columns that outgrew their groups, one after another by the whole warp
        unsigned big = __ballot_sync(kFull, ovf && gl == 0);
        while (big && !stop) {
            const int q = __ffs(big) - 1;
            big &= big - 1;
            int c = __shfl_sync(kFull, col, q);
            while (c >= 0) {  // the column, then any owner it displaced
                int nx = -1;
                const Outcome o = reduce_column(g, A, band, c, sw0, sw0 + A.cap, sw0 + 2 * A.cap, rm, true, &nx);
                if (!settle(g, A, c, o)) {
                    stop = true;
                    break;
                }
                c = nx;
            }
            if (lead == q) col = -1;
        }
        if (ovf) n = 0;
    }
    n_adds = warp_sum(n_adds);
    n_ints = warp_sum(n_ints);
    n_disp = warp_sum(n_disp);
    if (lane == 0) {
        if (n_adds) cnt_add(&A.counters[CNT_ADDITIONS], n_adds);
        if (n_ints) cnt_add(&A.counters[CNT_ADD_INTS], n_ints);
        if (n_pub) cnt_add(&A.counters[CNT_PUBLISHED], n_pub);
        if (n_disp) cnt_add(&A.counters[CNT_DISPLACED], (long long)n_disp);
    }
    light_block_done(A);
}

// Heavy tier: one CTA per deferred column, buffers of the level-2 capacity.
// Like the reference's block phase (include/kernel.h:966-1060) it does not
// stop at the band: a column handed over is reduced until it owns its lowest
// row or becomes zero.
template <int T>
__global__ void __launch_bounds__(T, 1) k_reduce_heavy(ReduceArgs A) {
    extern __shared__ __align__(16) int32_t smem[];
    __shared__ int gsm[2 * (T / 32 + 2)];
    __shared__ unsigned long long gsb[2];
    __shared__ RoundMem<BlockG<T>> rm;
    BlockG<T> g;
    g.sm = gsm;
    g.sb = gsb;
    int32_t* sw0 = smem;
    int32_t* sw1 = sw0 + A.cap;
    int32_t* sp = sw1 + A.cap;
    const int hb = __ldcg(A.ctr + 1), he = __ldcg(A.ctr + 2);
    const Band band{INT32_MIN, nullptr, 0};
    while (true) {
        int k = 0;
        if (g.leader()) k = hb + atomicAdd(A.ctr + 3, 1);
        k = g.bcast(k);
        if (k >= he) break;
        int col = __ldcg(A.heavy + k);
        while (col >= 0) {
            int next = -1;
            Outcome o = reduce_column(g, A, band, col, sw0, sw1, sp, rm, false, &next);
            if (!settle(g, A, col, o)) return;
            col = next;
        }
        if (g.leader() && A.heavy_done) {  // progress for the host's dimension gate
            const int v = atomicAdd(A.heavy_done, 1) + 1;
            if (A.gate_host) st_relaxed_sys(A.gate_host, v);
        }
    }
}

// ------------------------------------------------------------- work queue
// One persistent, cooperative launch drains the (complex, block) items of a
// whole schedule: every spectral-sequence block of every complex of a batch
// (one complex when not batched), in each complex's own block order, with
// each complex's own dimension gate.  The host loop it replaces issues, per
// block, a warp-tier launch and a CTA-tier launch and synchronises at every
// dimension (the reference: include/specseq.h:616-661, three launches and a
// host synchronisation per block).
//
// Blocks [0, heavy_ctas) reduce the columns the warp tier defers, taken from a
// pool in order; the other blocks run independent warps over the open items.
// An item opens when its predecessor of the same complex has finished; the
// first item of a complex's next dimension opens once at most gate_left of the
// complex's CTA-tier columns are left (none for its last item, after which the
// complex is finished).  An item's entries are the columns its predecessors
// parked (their lowest row below the band; kept with that row, so a later
// block looks at a parked column without loading it) followed by the columns
// its block adds to the window; a warp takes `chunk` of them at a time.
// Columns of different complexes never share rows, so the items of different
// complexes run concurrently.  All blocks are resident (cooperative launch),
// so a block may poll for work that another block produces; every poll is
// bounded by spin_limit, after which the launch sets ERRB_TIMEOUT and leaves.

__device__ __forceinline__ int ld_acq(const int* p) { return ld_acquire(p); }
__device__ __forceinline__ void st_rel(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void queue_fail(const ReduceArgs& A, const QueueArgs& Q, int bits) {
    atomicOr(A.err, bits);
    st_rel(Q.abort, 1);
}

// Opens complex c's next item once its CTA-tier columns allow (c waits at a
// gate, its current item ci finished); any lane may call it.
__device__ void queue_try_gate(const QueueArgs& Q, int c, int ci) {
    const bool last = ci + 1 >= Q.item_end[c];
    if (ld_acq(Q.hpend + c) > (last ? 0 : Q.gate_left)) return;
    if (atomicCAS(Q.gate + c, 1, 0) != 1) return;
    if (last) {
        st_rel(Q.cur + c, -1);
        __threadfence();
        atomicAdd(Q.finished, 1);
    } else {
        st_rel(Q.cur + c, ci + 1);
    }
}

// Item `it` of complex c has finished: the next item opens, or, after the
// last block of a dimension, the complex waits at its gate.
__device__ __forceinline__ void queue_finish_item(const QueueArgs& Q, int c, int it, int flags) {
    __threadfence();
    if (flags & QF_LAST_OF_DIM) st_rel(Q.gate + c, 1);
    else st_rel(Q.cur + c, it + 1);
}

// Final state of a warp-tier column taken from the queue (settle's rules;
// deferred columns go to the pool, parked ones to the next item's list).
__device__ bool settle_q(const ReduceArgs& A, const QueueArgs& Q, int cc, int col, Outcome o, int it, int2* lout,
                         int32_t lcap) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) {
        switch (o) {
            case OUT_OWNER: break;
            case OUT_ZERO: A.state[col] = ST_ZERO; break;
            case OUT_DEFERRED: {
                A.state[col] = ST_HEAVY;
                atomicAdd(Q.hpend + cc, 1);
                const int i = atomicAdd(Q.pool_tail, 1);
                if (i < Q.pool_cap) {
                    Q.pool_c[i] = cc;
                    __threadfence();
                    st_rel(Q.pool + i, col);
                } else {
                    queue_fail(A, Q, ERRB_CAPACITY);  // the run is repeated with a larger pool
                }
                break;
            }
            case OUT_PARKED: {
                const int low = A.low[col];
                __threadfence();
                st_release_u8(A.state + col, ST_ACTIVE);
                const int j = atomicAdd(Q.lin + it + 1, 1);
                if (j < lcap) lout[j] = make_int2(col, low);
                else queue_fail(A, Q, ERRB_CAPACITY);
                break;
            }
            default:
                __threadfence();
                st_release_u8(A.state + col, ST_ACTIVE);
                queue_fail(A, Q, ERRB_CHECK);
                ok = false;
                break;
        }
    }
    __syncwarp();
    return __shfl_sync(kFull, ok ? 1 : 0, 0) != 0;
}

__device__ void queue_light(const ReduceArgs& A, const QueueArgs& Q, int32_t* sw0, int32_t* sw1, int32_t* sp,
                            RoundMem<WarpG>& rm, int warps_per_block) {
    WarpG g;
    const int lane = g.rank();
    const int wl = (blockIdx.x - Q.heavy_ctas) * warps_per_block + (threadIdx.x >> 5);
    int start = Q.ncplx > 0 ? wl % Q.ncplx : 0;
    long long idle = 0;
    while (true) {
        int stop = 0;
        if (lane == 0) stop = ld_acq(Q.abort) || ld_acq(Q.finished) >= Q.ncplx;
        if (__shfl_sync(kFull, stop, 0)) break;
        // an open item with entries left: the lanes look at 32 complexes at a time
        int it = -1, cc = -1;
        for (int base = 0; base < Q.ncplx && it < 0; base += 32) {
            int myit = -1, c = -1;
            if (base + lane < Q.ncplx) {
                c = (start + base + lane) % Q.ncplx;
                const int ci = ld_acq(Q.cur + c);
                if (ci >= 0) {
                    if (ld_acq(Q.gate + c)) {
                        queue_try_gate(Q, c, ci);
                    } else {
                        const QItem& I = Q.items[ci];
                        const int total = ld_acq(Q.lin + ci) + (I.nend - I.nbeg);
                        if (total == 0) {  // nothing to do: whoever sees it first finishes it
                            if (atomicCAS(Q.taken + ci, 0, 1) == 0) queue_finish_item(Q, c, ci, I.flags);
                        } else if (__ldcg(Q.taken + ci) < total) {
                            myit = ci;
                        }
                    }
                }
            }
            const unsigned m = __ballot_sync(kFull, myit >= 0);
            if (m) {
                const int src = __ffs(m) - 1;
                it = __shfl_sync(kFull, myit, src);
                cc = __shfl_sync(kFull, c, src);
            }
        }
        if (it < 0) {
            if (++idle > Q.spin_limit) {
                if (lane == 0) queue_fail(A, Q, ERRB_TIMEOUT);
                break;
            }
            __nanosleep(256);
            continue;
        }
        idle = 0;
        start = cc;
        const QItem I = Q.items[it];
        const int nl = ld_acq(Q.lin + it);
        const int total = nl + (I.nend - I.nbeg);
        int base = 0;
        if (lane == 0) base = atomicAdd(Q.taken + it, Q.chunk);
        base = __shfl_sync(kFull, base, 0);
        if (base >= total) continue;
        const int cnt = min(Q.chunk, total - base);
        const int32_t lcap = Q.list_cap[cc];
        const int2* lin_list = Q.lists + Q.list_off[cc] + ((I.flags & QF_HALF) ? lcap : 0);
        int2* lout = Q.lists + Q.list_off[cc] + ((I.flags & QF_HALF) ? 0 : lcap);
        int col = -1, lowc = 0;
        bool run = false, park = false;
        if (lane < cnt) {
            const int e = base + lane;
            if (e < nl) {
                const int2 v = lin_list[e];
                col = v.x;
                lowc = v.y;
            } else {
                col = A.active[I.nbeg + (e - nl)];
                lowc = __ldcg(A.low + col);
            }
            if (col < 0 || col >= A.ncols) {  // self-check: a list or active entry in range
                queue_fail(A, Q, ERRB_CHECK);
                col = -1;
            } else {
                const bool act = ld_acquire_u8(A.state + col) == ST_ACTIVE && !ld_acquire_u8(A.cleared + col);
                run = act && lowc >= I.minrow;
                park = act && lowc < I.minrow;
            }
        }
        // still below the band: on to the next item's list as they are
        const unsigned pm = __ballot_sync(kFull, park);
        if (pm) {
            int pb = 0;
            if (lane == 0) pb = atomicAdd(Q.lin + it + 1, __popc(pm));
            pb = __shfl_sync(kFull, pb, 0);
            if (park) {
                const int j = pb + __popc(pm & lanemask_lt());
                if (j < lcap) lout[j] = make_int2(col, lowc);
                else queue_fail(A, Q, ERRB_CAPACITY);
            }
        }
        const Band band{I.minrow, Q.taken + it, total};
        unsigned m = __ballot_sync(kFull, run);
        bool failed = false;
        while (m && !failed) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            int c2 = __shfl_sync(kFull, col, src);
            while (c2 >= 0) {  // the column, then any owner it displaced
                int next = -1;
                const Outcome o = reduce_column(g, A, band, c2, sw0, sw1, sp, rm, true, &next);
                if (!settle_q(A, Q, cc, c2, o, it, lout, lcap)) {
                    failed = true;
                    break;
                }
                c2 = next;
            }
        }
        if (failed) break;
        // the chunk is finished; the warp finishing the item opens the next one
        int fin = 0;
        if (lane == 0) {
            __threadfence();
            fin = atomicAdd(Q.done + it, cnt) + cnt == total;
            if (fin) queue_finish_item(Q, cc, it, I.flags);
        }
        __syncwarp();
    }
}

template <int T>
__device__ void queue_heavy(const ReduceArgs& A, const QueueArgs& Q, const BlockG<T>& g, int32_t* sw0, int32_t* sw1,
                            int32_t* sp, RoundMem<BlockG<T>>& rm) {
    const Band band{INT32_MIN, nullptr, 0};
    long long idle = 0;
    while (true) {
        unsigned long long pk = 0;  // bit 63: stop; else (complex << 32) | column, or all ones for none
        if (g.leader()) {
            if (ld_acq(Q.abort) || ld_acq(Q.finished) >= Q.ncplx) {
                pk = 1ull << 63;
            } else {
                pk = ~0ull >> 1;
                const int h = ld_acq(Q.pool_head);
                if (h < Q.pool_cap) {
                    const int v = ld_acq(Q.pool + h);
                    if (v >= 0 && atomicCAS(Q.pool_head, h, h + 1) == h)
                        pk = (uint64_t(uint32_t(Q.pool_c[h])) << 32) | uint32_t(v);
                }
            }
        }
        pk = g.bcast64(pk);
        if (pk >> 63) break;
        if (pk == (~0ull >> 1)) {
            if (++idle > Q.spin_limit) {
                if (g.leader()) queue_fail(A, Q, ERRB_TIMEOUT);
                break;
            }
            if (g.leader()) __nanosleep(512);
            continue;
        }
        idle = 0;
        const int cc = int(pk >> 32);
        int col = int(uint32_t(pk));
        while (col >= 0) {
            int next = -1;
            const Outcome o = reduce_column(g, A, band, col, sw0, sw1, sp, rm, false, &next);
            if (!settle(g, A, col, o)) {
                if (g.leader()) queue_fail(A, Q, ERRB_CHECK);
                return;
            }
            col = next;
        }
        if (g.leader()) {
            __threadfence();
            atomicSub(Q.hpend + cc, 1);
        }
    }
}

// Al: warp-tier arguments (cap = level-1 capacity), Ah: CTA tier (level 2).
template <int T>
__global__ void __launch_bounds__(T, 1) k_reduce_queue(ReduceArgs Al, ReduceArgs Ah, QueueArgs Q) {
    extern __shared__ __align__(16) int32_t smem[];
    __shared__ int gsm[2 * (T / 32 + 2)];
    __shared__ unsigned long long gsb[2];
    __shared__ union {
        RoundMem<BlockG<T>> cta;
        RoundMem<WarpG> warp[T / 32];
    } rm;
    if (int(blockIdx.x) < Q.heavy_ctas) {
        BlockG<T> g;
        g.sm = gsm;
        g.sb = gsb;
        queue_heavy<T>(Ah, Q, g, smem, smem + Ah.cap, smem + 2 * Ah.cap, rm.cta);
    } else {
        int32_t* sw0 = smem + size_t(threadIdx.x >> 5) * (3 * Al.cap + kHdr);
        queue_light(Al, Q, sw0, sw0 + Al.cap, sw0 + 2 * Al.cap, rm.warp[threadIdx.x >> 5], T / 32);
    }
}

// ------------------------------------------------------- fill-in account
// What a reduction that takes its columns in order, one addition of the lowest row's
// owner at a time, would read: the allocation-free call's one-block kernel takes new room
// for as much, and what it has no room for is refused.  With the pairs known (the pivots
// of the finished reduction) every step of a column is: its lowest row's owner is an
// earlier column, whose reduced form is added, or the column itself.  So the columns are
// gone through side by side, a warp each, handed out in order; a warp waits for an owner
// that is not ready yet, which an earlier ticket's warp is at work on.  Columns that own
// their row from the start (apparent pairs) take no addition and are not listed.
//
// Bound by the longest chain of additions of columns that wait for one another (26 for
// a 700-point Rips complex's 4,544 additions, 905 of 15,146 for a 20^3 grid), 1 us each
// for short columns and 4 for some hundred entries: the call takes 289 us instead of 250
// and 4.5 ms instead of 0.7 (the one-block kernel 9.5 and 128 ms).  Columns of more than
// kFillCap entries, and anything else out of the ordinary, set the error word: the
// one-block kernel finds out by itself then.
constexpr int kFillCap = 960;  // ints of each of a warp's three lists (45 KB a block)
constexpr int kFillPolls = 1 << 20;

struct FillArgs {
    int32_t listed;
    const int32_t* active;
    int32_t* arena;
    int64_t arena_cap;
    const int64_t* off;       // the columns' slots, unless all are short
    const uint64_t* pivot;
    const int32_t* leftmost;
    const int4* app;
    uint64_t* ready;          // [n] slot + 1 of a listed column's reduced form
    int64_t room;
    Ctl* ctl;
};

__global__ void __launch_bounds__(128) k_fill_account(const __grid_constant__ FillArgs A) {
    __shared__ __align__(16) int32_t s_list[4][3][kFillCap];
    WarpG g;
    const int lane = g.rank();
    int32_t(*list)[kFillCap] = s_list[threadIdx.x >> 5];
    int* err = &A.ctl->err;
    const bool all_short = A.ctl->max_len <= kShortLen;
    auto slot_of = [&](int32_t c) { return all_short ? int64_t(kShortSlot) * c : A.off[c]; };
    // a column's entries from its slot into dst, the first 124 with its header (there are
    // guard ints behind the arena); -1 when it is too long
    auto fetch = [&](int64_t slot, int32_t* dst) {
        const int4 q = __ldcg(reinterpret_cast<const int4*>(A.arena + slot) + lane);
        const int len = __shfl_sync(kFull, q.x, 0), n4 = int(pad4(len)) >> 2;
        if (len > kFillCap) return -1;
        if (lane > 0 && lane <= n4) reinterpret_cast<int4*>(dst)[lane - 1] = q;
        if (n4 > 31) copy4(g, dst, A.arena + slot + kHdr, 31, n4);
        __syncwarp();
        return len;
    };
    for (;;) {
        int t = 0;
        if (lane == 0) t = ld_acquire(err) ? A.listed : atomicAdd(&A.ctl->fill_next, 1);
        t = g.bcast(t);
        if (t >= A.listed) return;
        const int32_t col = A.active[t];
        if (A.pivot[col] != kNoOwner) continue;  // a birth: cleared before its turn
        int64_t slot = slot_of(col);
        int32_t *w = list[0], *o = list[1];
        int n = fetch(slot, w);
        bool ok = n >= 0, added = false;
        long long cost = 0;
        while (ok && n > 0) {
            const int32_t L = lds(w + n - 1);
            const uint64_t e = A.pivot[L];
            const int4 q = A.app[L];  // its owner's other entries, if apparent and short
            const int32_t lm = A.leftmost[L];
            const int32_t p = pv_col(e);
            if (e != kNoOwner && p == col) break;
            ok = e != kNoOwner && p < col;
            if (!ok) break;
            int pn;
            if (q.x >= 0) {
                pn = q.x + 1;
                if (lane < pn) list[2][lane] = lane == q.x ? L : lane == 0 ? q.y : lane == 1 ? q.z : q.w;
                __syncwarp();
            } else {
                // apparent: the leftmost column of its lowest row, never changed
                pn = lm == p ? fetch(slot_of(p), list[2]) : 0;
                if (pn == 0 || (pn > 0 && lds(list[2] + pn - 1) != L)) {  // listed: reduced, once it is there
                    unsigned long long r = 0;
                    if (lane == 0)
                        for (int polls = 0;
                             (r = ld_acquire_u64(A.ready + p)) == 0 && polls < kFillPolls && !ld_acquire(err); polls++)
                            __nanosleep(64);
                    r = g.bcast64(r);
                    ok = r != 0;
                    if (!ok) break;
                    __syncwarp();
                    pn = fetch(int64_t(r) - 1, list[2]);
                }
            }
            ok = pn > 0 && n + pn - 2 <= kFillCap && lds(list[2] + pn - 1) == L;
            if (!ok) break;
            cost += n + pn;
            n = merge(g, w, n, false, list[2], pn, false, o, kFillCap, err);
            int32_t* x = w;
            w = o;
            o = x;
            added = true;
            ok = n == 0 || lds(w + n - 1) < L;  // (the lowest row moves down with every addition)
        }
        if (ok && added && n > 0) {
            const int64_t ints = slot_ints(n);
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(&A.ctl->arena_top, (unsigned long long)ints);
            slot = int64_t(g.bcast64(at));
            ok = slot + ints <= A.arena_cap;
            if (ok) {
                store4(g, A.arena + slot + kHdr, w, int(pad4(n)) >> 2);
                if (lane == 0) *reinterpret_cast<int4*>(A.arena + slot) = make_int4(n, col, 0, 0);
            }
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) {
            if (ok && cost) ok = int64_t(atomicAdd(&A.ctl->fill, (unsigned long long)cost)) + cost <= A.room;
            if (!ok) atomicOr(err, ERRB_CAPACITY);
            else if (n > 0) st_release_u64(A.ready + col, uint64_t(slot) + 1);
        }
        __syncwarp();
    }
}

void fill_account_launch(const Device& D, int32_t listed, int64_t room, uint64_t* ready, int sms, cudaStream_t s) {
    if (listed <= 0) return;
    const FillArgs A{listed,  D.active,   D.arena, D.arena_cap, D.scratch64,
                     D.pivot, D.leftmost, D.app,   ready,       room,        D.ctl};
    const int grid = int(std::min<int64_t>((int64_t(listed) + 3) / 4, int64_t(sms) * 4));
    k_fill_account<<<grid, 128, 0, s>>>(A);
}

// per complex and dimension: active columns, min first row over non-empty
// columns and max low + 1 over active columns (the quantities ColumnShrink
// computes for the whole matrix, include/specseq.h:374-398)
__global__ void k_queue_info(int64_t n, int32_t k, const int64_t* cstart, const int32_t* perm, const int32_t* rdim,
                             const int32_t* arena, const uint64_t* desc, const int32_t* low, const uint8_t* state,
                             int32_t* act_cnt, int32_t* min_row, int32_t* max_row) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const uint64_t d = desc[i];
        const uint32_t len = desc_len(d);
        if (!len) continue;
        const int64_t x = perm[i];
        int32_t a = 0, b = k;  // largest a with cstart[a] <= x
        while (b - a > 1) {
            const int32_t mid = (a + b) >> 1;
            if (cstart[mid] <= x) a = mid;
            else b = mid;
        }
        const int dm = rdim[i];
        const int64_t slot = int64_t(a) * kNumDims + dm;
        atomicMin(min_row + slot, arena[desc_off(d) + kHdr]);
        if (state[i] == ST_ACTIVE) {
            atomicAdd(act_cnt + slot, 1);
            atomicMax(max_row + slot, low[i] + 1);
        }
    }
}

int queue_complex_info(const Device& D, int32_t k, const int64_t* d_cstart, int32_t* act_cnt, int32_t* min_row,
                       int32_t* max_row, cudaStream_t s) {
    const int64_t m = int64_t(k) * kNumDims;
    cudaMemsetAsync(act_cnt, 0, sizeof(int32_t) * m, s);
    fill_i32(min_row, INT32_MAX, m, s);
    fill_i32(max_row, -1, m, s);
    if (D.n == 0) return 0;
    int64_t g = (D.n + 255) / 256;
    if (g > 65536) g = 65536;
    k_queue_info<<<unsigned(g), 256, 0, s>>>(D.n, k, d_cstart, D.perm, D.dim, D.arena, D.desc, D.low, D.state, act_cnt,
                                             min_row, max_row);
    return 3;
}

int light_smem_bytes(int cap) { return 4 * (3 * cap + kHdr) * 4; }
int heavy_smem_bytes(int cap) { return (3 * cap + kHdr) * 4; }

// Passes (rounds and single additions) of a warp-tier column after which, once
// its step's window is fully handed out, it moves to the CTA tier: a step's light
// launch lasts as long as its longest chain, while CTA-tier launches overlap
// later steps on side streams.  Handing chains over while the window still has
// work would only move parallel work onto the (fewer) CTAs.
constexpr int32_t kLightChain = 8;

static ReduceArgs make_args(const Device& D, const int32_t* active, int cap, int* ctr) {
    ReduceArgs A;
    A.ncols = int32_t(D.n);
    A.active = active;
    A.cap = cap;
    A.arena = D.arena;
    A.arena_cap = D.arena_cap;
    A.arena_top = D.arena_top;
    A.desc = D.desc;
    A.low = D.low;
    A.pivot = D.pivot;
    A.state = D.state;
    A.cleared = D.cleared;
    A.ctr = ctr;
    A.ctr_next = nullptr;
    A.listed = 0;
    A.heavy = D.heavy;
    A.pool_tail = D.pool_tail;
    A.heavy_done = D.heavy_done;
    A.gate_host = D.gate_host;
    A.pool_cap = D.pool_cap;
    A.err = D.err;
    A.counters = D.counters;
    A.light_chain = kLightChain;
    A.app = D.app;
    return A;
}

void reduce_light_launch(const Device& D, int32_t beg, int32_t end, int cap, int* ctr, int* ctr_next, int grid,
                         cudaStream_t s) {
    ReduceArgs A = make_args(D, D.active + beg, cap, ctr);
    A.listed = end - beg;
    A.ctr_next = ctr_next;
    k_reduce_light<<<grid, 128, light_smem_bytes(cap), s>>>(A);
}

void reduce_heavy_launch(const Device& D, int cap, int threads, int* ctr, int grid, cudaStream_t s) {
    ReduceArgs A = make_args(D, nullptr, cap, ctr);
    if (threads == 256) k_reduce_heavy<256><<<grid, 256, heavy_smem_bytes(cap), s>>>(A);
    else k_reduce_heavy<128><<<grid, 128, heavy_smem_bytes(cap), s>>>(A);
}

// The dynamic shared-memory limit is a property of the kernel (per device),
// shared by every context of the process: contexts with different capacities
// (the server's workers, each autotuned) only ever raise it, under a lock, so
// that no launch finds it lowered below its own request.
static cudaError_t raise_smem_limit(const void* fn, int slot, int bytes) {
    static std::mutex mu;
    static int limit[64][5] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> l(mu);
    int& cur = limit[dev & 63][slot];
    if (bytes <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

static int queue_smem_bytes(int cap1, int cap2, int threads) {
    const int light = (threads / 32) * (3 * cap1 + kHdr) * 4;
    const int heavy = (3 * cap2 + kHdr) * 4;
    return light > heavy ? light : heavy;
}

cudaError_t queue_configure(int cap1, int cap2, int threads, int* blocks_per_sm) {
    const int smem = queue_smem_bytes(cap1, cap2, threads);
    *blocks_per_sm = 0;
    cudaError_t e;
    if (threads == 256) {
        e = raise_smem_limit(reinterpret_cast<const void*>(k_reduce_queue<256>), 3, smem);
        if (e != cudaSuccess) return e;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_reduce_queue<256>, 256, smem);
    }
    e = raise_smem_limit(reinterpret_cast<const void*>(k_reduce_queue<128>), 4, smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_reduce_queue<128>, 128, smem);
}

cudaError_t reduce_queue_launch(const Device& D, int cap1, int cap2, int threads, const QueueArgs& Q, int grid,
                                cudaStream_t s) {
    ReduceArgs Al = make_args(D, D.active, cap1, nullptr);
    ReduceArgs Ah = make_args(D, nullptr, cap2, nullptr);
    Al.gate_host = Ah.gate_host = nullptr;
    Al.heavy_done = Ah.heavy_done = nullptr;
    QueueArgs q = Q;
    void* args[] = {&Al, &Ah, &q};
    const int smem = queue_smem_bytes(cap1, cap2, threads);
    if (threads == 256)
        return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_reduce_queue<256>), grid, 256, args, smem, s);
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_reduce_queue<128>), grid, 128, args, smem, s);
}

cudaError_t reduce_configure(int cap1, int cap2, int heavy_threads, int* light_blocks_per_sm,
                             int* heavy_blocks_per_sm) {
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k_reduce_light), 0, light_smem_bytes(cap1));
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(light_blocks_per_sm, k_reduce_light, 128, light_smem_bytes(cap1));
    if (e != cudaSuccess) return e;
    if (heavy_threads == 256) {
        e = raise_smem_limit(reinterpret_cast<const void*>(k_reduce_heavy<256>), 1, heavy_smem_bytes(cap2));
        if (e != cudaSuccess) return e;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(heavy_blocks_per_sm, k_reduce_heavy<256>, 256,
                                                             heavy_smem_bytes(cap2));
    }
    e = raise_smem_limit(reinterpret_cast<const void*>(k_reduce_heavy<128>), 2, heavy_smem_bytes(cap2));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(heavy_blocks_per_sm, k_reduce_heavy<128>, 128,
                                                         heavy_smem_bytes(cap2));
}

}  // namespace sspp
