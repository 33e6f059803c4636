// Dimension 1 of the boundary matrix: edge columns, which hold two vertices at most
// and stay that short, so their reduction is a walk in a forest instead of sorted
// merges.  A row's pivot entry {column c, other entry p} is the whole reduced column
// {p, v}: adding it to a column that holds v replaces v by p.  Smirnov and Morozov
// ("Triplet Merge Trees", 2017) build merge trees from such triples, in parallel and
// in any order of the edges; the pivots here are theirs, column for column.
//
// While the forest is worked on, the vertices' pivot entries hold p + 1 where the
// arena slot stands otherwise (0: the column has no other entry).  A thread takes an
// edge: both of its entries move up the forest while their owner is an earlier
// column; two equal entries cancel (the column is zero); else it claims the larger
// one's row, from a later owner too, whose column it then carries on with.  An entry
// {c, p} whose p has an earlier owner than c is shortened on the way by p's column,
// an addition from the left like any other.  An entry is one word that is swapped
// whole, so no ordering with other memory is needed until the finish writes the new
// owners' columns to their own slots (nobody refers to an edge that owned no row).
//
// Nothing here depends on the higher dimensions, so the launch runs beside them on a
// stream of its own; an edge that one of their claims would have cleared is positive
// and comes out zero.  (In a matrix that is no chain complex it may not: the pairs'
// scan finds such an edge and the run is repeated with the edges last.)
//
// Bound by the chain of reads up the forest, one trip to L2 a step where the general
// tiers take a pass of reading, sorting and claiming.  400-point Rips input: 57 us at
// the end of the reduction before, beside the triangles now (reduction 155 -> 95 us);
// 1,200-point cloud 280 -> 212, 100,000-vertex graph after an edge collapse 160 -> 110,
// 20,000-point Rips input, edges alone, then the dual: 1,010 -> 962.
#include <algorithm>
#include <climits>

#include "sspp_kernels.cuh"
#include "sspp_launch.h"

namespace sspp {

namespace {
constexpr int kMaxHops = 1 << 24;

struct EdgeArgs {
    uint64_t* pivot;
    const int32_t* active;
    int32_t listed, rows;  // edges to reduce; vertices (the reordered rows [0, rows))
    int32_t* arena;
    int64_t arena_cap;
    uint64_t* desc;
    int32_t* low;
    uint8_t* state;
    uint8_t* cleared;
    const int4* app;
    long long* counters;
    int* err;
};

__device__ __forceinline__ uint64_t ld_word(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t tree_entry(int32_t col, int32_t other) {
    return (uint64_t(uint32_t(other + 1)) << 31) | uint64_t(uint32_t(col));
}
__device__ __forceinline__ int32_t tree_other(uint64_t e) { return int32_t(e >> 31) - 1; }

// the two entries of column `col` (first -1: one entry); false when it is not such a column
__device__ __forceinline__ bool edge_entries(const EdgeArgs& A, int32_t col, int& n, int32_t& lo, int32_t& hi) {
    const uint64_t d = ld_cg_u64(A.desc + col);
    const int64_t slot = int64_t(desc_off(d));
    n = int(desc_len(d));
    if (n > 2 || slot + 2 * kHdr > A.arena_cap) return false;
    const int2 e = __ldcg(reinterpret_cast<const int2*>(A.arena + slot + kHdr));
    lo = n == 2 ? e.x : -1;
    hi = n == 2 ? e.y : n == 1 ? e.x : -1;
    return hi < A.rows && lo < hi + (n == 0);
}

__device__ __forceinline__ void open_rows(const EdgeArgs& A, int first, int step) {
    for (int v = first; v < A.rows; v += step) {
        const uint64_t e = A.pivot[v];
        if (e == kNoOwner) continue;
        const int32_t c = pv_col(e);
        int4 q = __ldg(A.app + v);
        bool ok = true;
        if (q.x < 0) {  // an owner from an earlier run over the same columns
            int n = 0;
            ok = edge_entries(A, c, n, q.y, q.z) && n > 0;
            q.x = n - 1;
        }
        if (!ok || q.x > 1) {  // self-check: an edge column
            atomicOr(A.err, ERRB_CHECK);
            q.x = 0;
        }
        A.pivot[v] = tree_entry(c, q.x == 1 ? q.y : -1);
    }
}

// Moves x to its owner's other entry when the owner is an earlier column than c;
// `from` and `at` are the row left last and the entry it was left by.
__device__ __forceinline__ bool hop(const EdgeArgs& A, uint64_t e, int32_t c, int32_t& x, int32_t& from, uint64_t& at) {
    if (x < 0 || pv_col(e) >= c) return false;
    const int32_t p = tree_other(e);
    if (from >= 0 && pv_col(e) < pv_col(at))
        atomicCAS(reinterpret_cast<unsigned long long*>(A.pivot + from), (unsigned long long)at,
                  (unsigned long long)tree_entry(pv_col(at), p));
    from = x;
    at = e;
    x = p;
    return true;
}

__device__ __forceinline__ void unite(const EdgeArgs& A, int first, int step) {
    long long adds = 0, disp = 0;
    for (int i = first; i < A.listed; i += step) {
        int32_t c = A.active[i], a, b;
        if (A.state[c] != ST_ACTIVE || A.cleared[c]) continue;
        int n = 0;
        if (!edge_entries(A, c, n, b, a)) {
            atomicOr(A.err, ERRB_CHECK);
            continue;
        }
        int32_t fa = -1, fb = -1;  // rows left last
        uint64_t ea = 0, eb = 0;
        for (int it = 0;; it++) {
            if (a == b) {  // (both -1: nothing left)
                A.desc[c] = pack_desc(0, 0);
                A.low[c] = -1;
                A.state[c] = ST_ZERO;
                break;
            }
            if (it > kMaxHops) {
                atomicOr(A.err, ERRB_TIMEOUT);
                break;
            }
            if (a < b) {
                const int32_t t = a, ft = fa;
                const uint64_t et = ea;
                a = b, fa = fb, ea = eb;
                b = t, fb = ft, eb = et;
            }
            const uint64_t wa = ld_word(A.pivot + a), wb = b >= 0 ? ld_word(A.pivot + b) : kNoOwner;
            const bool ha = hop(A, wa, c, a, fa, ea), hb = hop(A, wb, c, b, fb, eb);
            if (ha || hb) {
                adds += int(ha) + int(hb);
                continue;
            }
            const uint64_t old = atomicCAS(reinterpret_cast<unsigned long long*>(A.pivot + a), (unsigned long long)wa,
                                           (unsigned long long)tree_entry(c, b));
            if (old != wa) continue;  // its owner changed: look again
            if (wa == kNoOwner) break;
            // the later owner's column goes on without a: the two columns' sum
            disp++;
            adds++;
            c = pv_col(wa);
            a = tree_other(wa);
            fa = fb = -1;
        }
    }
    adds = warp_sum(adds);
    disp = warp_sum(disp);
    if (lane_id() == 0) {
        if (adds) {
            cnt_add(&A.counters[CNT_ADDITIONS], adds);
            cnt_add(&A.counters[CNT_ADD_INTS], 6 * adds);
        }
        if (disp) cnt_add(&A.counters[CNT_DISPLACED], disp);
    }
}

__device__ __forceinline__ void close_rows(const EdgeArgs& A, int first, int step) {
    for (int v = first; v < A.rows; v += step) {
        const uint64_t e = ld_word(A.pivot + v);
        if (e == kNoOwner) continue;
        const int32_t c = pv_col(e), p = tree_other(e);
        const uint64_t slot = desc_off(A.desc[c]);
        A.pivot[v] = pv_pack(c, slot);
        if (A.state[c] == ST_OWNER) continue;  // from the init passes: its column stands as it is
        if (int64_t(slot) + 2 * kHdr > A.arena_cap) {  // self-check: descriptor inside the arena
            atomicOr(A.err, ERRB_CHECK);
            continue;
        }
        const int n = p >= 0 ? 2 : 1;
        *reinterpret_cast<int4*>(A.arena + slot) = make_int4(n, c, 0, 0);
        *reinterpret_cast<int4*>(A.arena + slot + kHdr) =
            n == 2 ? make_int4(p, v, INT_MAX, INT_MAX) : make_int4(v, INT_MAX, INT_MAX, INT_MAX);
        A.desc[c] = pack_desc(slot, uint32_t(n));
        A.low[c] = v;
        A.state[c] = ST_OWNER;
        A.cleared[v] = 1;
    }
}

// phases [from, to] of open, unite, close; more than one needs a grid of one block
template <int T>
__global__ void __launch_bounds__(T) k_edges(const __grid_constant__ EdgeArgs A, int from, int to) {
    const int first = blockIdx.x * T + threadIdx.x, step = gridDim.x * T;
    for (int p = from; p <= to; p++) {
        if (p == 0) open_rows(A, first, step);
        else if (p == 1) unite(A, first, step);
        else close_rows(A, first, step);
        __syncthreads();
    }
}
}  // namespace

// Up to 8192 vertices and edges together one block does all three phases: two launches
// fewer (2,000-point Rips input: 77 against 82 us of reduction; with 20,000 vertices one
// block takes 1,306 us where three launches take 966).
constexpr int64_t kOneBlock = 8192;

int reduce_edges(Device& D, int32_t beg, int32_t end, int32_t rows, cudaStream_t s) {
    EdgeArgs A{D.pivot,  D.active + beg, end - beg, rows,  D.arena,    D.arena_cap, D.desc,
               D.low, D.state,        D.cleared, D.app, D.counters, D.err};
    if (int64_t(rows) + (end - beg) <= kOneBlock) {
        k_edges<1024><<<1, 1024, 0, s>>>(A, 0, 2);
        return 1;
    }
    const unsigned gr = unsigned(std::min<int64_t>((int64_t(rows) + 127) / 128, 4096));
    const unsigned ge = unsigned(std::min<int64_t>((int64_t(end - beg) + 127) / 128, 4096));
    k_edges<128><<<gr, 128, 0, s>>>(A, 0, 0);
    k_edges<128><<<ge, 128, 0, s>>>(A, 1, 1);
    k_edges<128><<<gr, 128, 0, s>>>(A, 2, 2);
    return 3;
}

}  // namespace sspp
