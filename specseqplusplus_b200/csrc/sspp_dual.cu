// Dualization: the anti-transpose of the cleared and compressed matrix, built
// in the arena behind the primal columns, with the pivot table, the column
// states, the dimensions and the per-dimension ranges carried over.
//
// Reference counterparts:
//   count / offsets / scatter     include/kernel.h:521-560 (countNonZeros,
//                                 computeOffsets, dualizeMatrixKernel)
//   per-column sort               include/specseq.h:329-332 (one thrust::sort
//                                 per column, launched from a host loop)
//   pivot and flag remap          include/kernel.h:562-580 (dualizeAuxArray)
//   dimension reversal            include/specseq.h:347-349
//   pairs mapped back             include/specseq.h:1188
// Primal row r of primal column j becomes dual row n-1-j of dual column n-1-r.
// An apparent pair (low l, column c) of the primal matrix becomes the dual
// pair (low n-1-c, column n-1-l).  Here every step is a device pass: the
// per-column sort is one lane per column (up to 8 entries) or one warp (registers
// up to 32 entries, shared memory up to 1024), and the rare longer columns are
// sorted by one CTA with shared-memory chunk sorts and merge-path merges in global
// memory.
//
// Mode 2 (no counterpart in the reference) dualizes after the boundary
// matrix's edge columns have been reduced: the 0-dimensional pairs are known,
// the dual columns of vertices are left alone, and the dual columns of the
// edges those pairs kill are cleared.  The dual columns of dimension >= 1 only
// hold cofaces of dimension >= 2, whose columns that reduction never touched.
// On lower-star grids the dual columns of vertices carry addition chains of
// tens of thousands of steps; mode 2 avoids them while keeping the short dual
// chains of dimensions >= 1 on Rips complexes.
#include <climits>

#include "sspp_launch.h"
#include "sspp_scan.cuh"

namespace sspp {

namespace {

constexpr int kWarpSortCap = 1024;  // ints of shared memory per warp
constexpr int kSortWarps = 8;
constexpr int kLongThreads = 1024;
constexpr int kLongChunk = 8192;    // ints sorted in shared memory by the CTA

unsigned grid_of(int64_t n, int threads, int64_t maxg) {
    int64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > maxg) g = maxg;
    return unsigned(g);
}

__device__ __forceinline__ int next_pow2(int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

// Whether primal column j is left out of the dual: in mode 2 the edges, whose rows
// are the vertices alone.  `info` is the dual's once the slots have their offsets.
__device__ __forceinline__ bool left_out(int64_t j, int64_t n, int skip_edges, const DimInfo* info, bool flipped) {
    if (!skip_edges) return false;
    const int64_t b = info->col_begin[1], e = info->col_end[1];
    return flipped ? j >= n - e && j < n - b : j >= b && j < e;
}

__global__ void k_dual_count(int64_t n, const int32_t* arena, const uint64_t* desc, int skip_edges,
                             const DimInfo* info, int32_t* cnt) {
    for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < n; j += int64_t(gridDim.x) * blockDim.x) {
        if (left_out(j, n, skip_edges, info, false)) continue;
        const uint64_t d = desc[j];
        const int32_t* c = arena + desc_off(d) + kHdr;
        const uint32_t len = desc_len(d);
        for (uint32_t k = 0; k < len; k++) atomicAdd(&cnt[n - 1 - c[k]], 1);
    }
}

// The end of the scan that gives every dual column its slot.  misc[0] = dual region
// base (ints into the arena, -1 when it does not fit), misc[1] = dual region size,
// misc[2] = number of long columns.  The dimensions' ranges are mirrored and their
// row bounds and active counts emptied.
struct DualReserve {
    int64_t n;
    unsigned long long* top;
    int64_t arena_cap;
    int64_t* misc;
    DimInfo* info;
    int* err;
    __device__ void operator()(int64_t total) const {
        const int64_t base = int64_t(*top);
        for (int d = 0; d < kNumDims; d++) {
            const int32_t b = info->col_begin[d], e = info->col_end[d];
            info->col_begin[d] = int32_t(n - e);
            info->col_end[d] = int32_t(n - b);
            info->min_row[d] = INT_MAX;
            info->max_row[d] = -1;
            info->act_end[d] = 0;
        }
        misc[2] = 0;
        if (base + total > arena_cap) {
            misc[0] = -1;
            atomicOr(err, ERRB_CAPACITY);
            return;
        }
        misc[0] = base;
        misc[1] = total;
        *top = (unsigned long long)(base + total);
    }
};

// scatter: filled[] counts up as the entries land (unsorted)
__global__ void k_dual_fill(int64_t n, const uint64_t* desc, int skip_edges, const DimInfo* info, const int64_t* off,
                            const int64_t* misc, int32_t* filled, int32_t* arena) {
    const int64_t base = misc[0];
    if (base < 0) return;
    for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < n; j += int64_t(gridDim.x) * blockDim.x) {
        if (left_out(j, n, skip_edges, info, true)) continue;
        const uint64_t d = desc[j];
        const int32_t* col = arena + desc_off(d) + kHdr;
        const uint32_t len = desc_len(d);
        for (uint32_t k = 0; k < len; k++) {
            const int64_t c = n - 1 - col[k];
            arena[base + off[c] + kHdr + atomicAdd(&filled[c], 1)] = int32_t(n - 1 - j);
        }
    }
}

// ascending; INT32_MAX padding ends up last
__device__ __forceinline__ void order2(int32_t& a, int32_t& b) {
    const int32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}
__device__ __forceinline__ void sort4(int4& q) {
    order2(q.x, q.y);
    order2(q.z, q.w);
    order2(q.x, q.z);
    order2(q.y, q.w);
    order2(q.y, q.z);
}

// What the dual's column c takes over from the primal column at the mirrored index.
struct Mirror {
    uint64_t owner;  // its pivot entry as a row
    int32_t low, dim;
    uint8_t state;
};

struct DualCols {
    int64_t n;
    const int64_t* off;
    const int32_t* cnt;
    int64_t* misc;
    int32_t* arena;
    int32_t* longlist;
    uint64_t* desc;
    int32_t* low;
    int32_t* dim;
    uint64_t* pivot;
    uint8_t* state;
    uint8_t* cleared;
    int4* app;
    DimInfo* info;
    int* err;
    int h0_done;
};

__device__ __forceinline__ void read_mirror(const DualCols& D, int64_t j, Mirror& m) {
    m = Mirror{kNoOwner, -1, 0, ST_ZERO};
    if (j < 0) return;
    m.owner = D.pivot[j];
    m.low = D.low[j];
    m.dim = D.dim[j];
    m.state = D.state[j];
}

// Column c's slot and what its lane reads of it, all before either of the lane's columns
// is worked on.
struct Slot {
    int64_t o, low_off;  // ints into the arena; the slot offset of the dual column that owns row c
    int len;
    int4 a, b;  // the first 8 entries of a column of at most 8
};

__device__ __forceinline__ void read_place(const DualCols& D, int64_t base, int64_t c, Slot& t) {
    t.o = t.low_off = 0;
    t.len = 0;
    t.a = t.b = make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX);
    if (c < 0) return;
    t.o = base + D.off[c];
    t.len = D.cnt[c];
}

__device__ __forceinline__ void read_entries(const DualCols& D, const Mirror& m, Slot& t) {
    if (t.len >= 1 && t.len <= 8) t.a = *reinterpret_cast<const int4*>(D.arena + t.o + kHdr);
    if (t.len >= 5 && t.len <= 8) t.b = *reinterpret_cast<const int4*>(D.arena + t.o + kHdr + 4);
    if (m.state == ST_OWNER) t.low_off = D.off[D.n - 1 - m.low];
}

// Dual column c of this lane (-1: none; the warp calls together): its entries sorted,
// its header and padding, and everything else the reduction keeps of it.
__device__ __forceinline__ void finish_columns(const DualCols& D, int64_t base, int64_t c, const Mirror& m,
                                               const Slot& t, int32_t* s, int* smin, int* smax, int* sact) {
    const int lane = threadIdx.x & 31;
    const int len = t.len;
    const int64_t o = t.o;
    int32_t first = INT_MAX, last = -1;
    int4 a = t.a;
    if (c >= 0) {
        *reinterpret_cast<int4*>(D.arena + o) = make_int4(len, int32_t(c), 0, 0);
        if (len >= 1 && len <= 8) {
            int4* d4 = reinterpret_cast<int4*>(D.arena + o + kHdr);
            if (len < 4) a.w = INT_MAX;
            if (len < 3) a.z = INT_MAX;
            if (len < 2) a.y = INT_MAX;
            sort4(a);
            if (len <= 4) {
                last = len == 1 ? a.x : len == 2 ? a.y : len == 3 ? a.z : a.w;
            } else {
                int4 b = t.b;
                if (len < 8) b.w = INT_MAX;
                if (len < 7) b.z = INT_MAX;
                if (len < 6) b.y = INT_MAX;
                sort4(b);
                // bitonic merge of the ascending halves
                order2(a.x, b.w);
                order2(a.y, b.z);
                order2(a.z, b.y);
                order2(a.w, b.x);
                sort4(a);
                sort4(b);
                last = len == 5 ? b.x : len == 6 ? b.y : len == 7 ? b.z : b.w;
                d4[1] = b;
            }
            d4[0] = a;
            first = a.x;
        }
    }
    // four columns of 9 to 32 entries at a time: their loads are under way together
    for (unsigned mid = __ballot_sync(0xffffffffu, len > 8 && len <= 32); mid;) {
        int q[4], ql[4];
        int32_t *data[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            q[u] = mid ? __ffs(mid) - 1 : -1;
            mid &= mid - 1;
            ql[u] = __shfl_sync(0xffffffffu, len, q[u] & 31);
            data[u] = D.arena + __shfl_sync(0xffffffffu, o, q[u] & 31) + kHdr;
            v[u] = q[u] >= 0 && lane < ql[u] ? data[u][lane] : INT_MAX;
        }
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int32_t x = __shfl_xor_sync(0xffffffffu, v[u], j);
                    v[u] = keep_min ? min(v[u], x) : max(v[u], x);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int32_t bottom = __shfl_sync(0xffffffffu, v[u], 0), top = __shfl_sync(0xffffffffu, v[u], ql[u] - 1);
            if (q[u] >= 0 && lane < int(pad4(ql[u]))) data[u][lane] = v[u];
            if (lane == q[u]) {
                first = bottom;
                last = top;
            }
        }
    }
    for (unsigned big = __ballot_sync(0xffffffffu, len > 32); big; big &= big - 1) {
        const int q = __ffs(big) - 1;
        const int ql = __shfl_sync(0xffffffffu, len, q);
        int32_t* data = D.arena + __shfl_sync(0xffffffffu, o, q) + kHdr;
        int32_t bottom, top;
        if (ql <= kWarpSortCap) {
            const int p = next_pow2(ql);
            for (int i = lane; i < p; i += 32) s[i] = i < ql ? data[i] : INT_MAX;
            __syncwarp();
            for (int k = 2; k <= p; k <<= 1) {
                for (int j = k >> 1; j > 0; j >>= 1) {
                    for (int i = lane; i < p; i += 32) {
                        const int ixj = i ^ j;
                        if (ixj > i) {
                            const int32_t x = s[i], y = s[ixj];
                            if ((x > y) == ((i & k) == 0)) {
                                s[i] = y;
                                s[ixj] = x;
                            }
                        }
                    }
                    __syncwarp();
                }
            }
            for (int i = lane; i < int(pad4(ql)); i += 32) data[i] = i < ql ? s[i] : INT_MAX;
            bottom = s[0];
            top = s[ql - 1];
            __syncwarp();
        } else {
            int32_t x = -1, y = INT_MAX;
            for (int i = lane; i < ql; i += 32) {
                x = max(x, data[i]);
                y = min(y, data[i]);
            }
            for (int i = ql + lane; i < int(pad4(ql)); i += 32) data[i] = INT_MAX;
            top = __reduce_max_sync(0xffffffffu, x);
            bottom = __reduce_min_sync(0xffffffffu, y);
            if (lane == q) {
                const int64_t at = atomicAdd(reinterpret_cast<unsigned long long*>(&D.misc[2]), 1ull);
                D.longlist[at] = int32_t(c);
            }
        }
        if (lane == q) {
            first = bottom;
            last = top;
        }
    }
    if (c < 0) return;
    const bool vertex = D.h0_done && m.dim == 0, owns = m.owner != kNoOwner, negative = m.state == ST_OWNER;
    D.desc[c] = pack_desc(uint64_t(o), uint32_t(len));
    D.low[c] = last;
    D.dim[c] = m.dim;
    D.cleared[c] = negative;
    const uint8_t st = m.state == ST_DROPPED ? ST_DROPPED
                       : owns                ? (vertex ? ST_ZERO : ST_OWNER)
                       : negative            ? ST_CLEARED
                       : len && !vertex      ? ST_ACTIVE
                                             : ST_ZERO;
    D.state[c] = st;
    // as a row: owned by the dual column of the primal column's lowest row, whose
    // lane writes the inline copy
    uint64_t e = kNoOwner;
    if (negative) {
        const int64_t dc = D.n - 1 - m.low;
        e = pv_pack(int32_t(dc), uint64_t(base + t.low_off));
    } else {
        D.app[c] = make_int4(-1, INT_MAX, INT_MAX, INT_MAX);
    }
    D.pivot[c] = e;
    if (owns) {
        const int64_t dr = D.n - 1 - pv_col(m.owner);
        const bool inl = !vertex && len <= 4;
        if (!vertex && last != dr) atomicOr(D.err, ERRB_CHECK);  // self-check: the dual owner's lowest row
        else
            D.app[dr] = make_int4(inl ? len - 1 : -1, inl && len > 1 ? a.x : INT_MAX, inl && len > 2 ? a.y : INT_MAX,
                                  inl && len > 3 ? a.z : INT_MAX);
    }
    if (len) {
        atomicMin(&smin[m.dim], first);
        if (st == ST_ACTIVE) {
            atomicMax(&smax[m.dim], last + 1);
            atomicAdd(&sact[m.dim], 1);
        }
    }
}

// Finishes the dual columns: sorted entries, descriptors, lows, states, dimensions,
// clearing, the pivot table with its inline copies, and the dimensions' row bounds.
// h0_done: the 0-dimensional pairs came from the boundary matrix, so the dual columns
// of vertices are never reduced.  Dual column c and dual row c come from primal row
// and column n-1-c, so a lane takes a column and the mirrored one, reads what both
// were and then writes both in place.  A warp takes 32 of each: columns of up to 8
// entries (nearly all) are sorted by their own lanes in registers, those of up to 32 by
// the whole warp, four at a time, longer ones one after another in shared memory (up to
// kWarpSortCap; the rest goes to the long list, unsorted, but with its low known).
// Bound by the latency of its dependent reads (25% of the memory's bandwidth, 21% of
// L2's): 20,000 points (2.67 M columns) 143 us with both columns' reads in turn and one
// longer column at a time, 100 like this (and 230 where sorting, remapping the pivots,
// inline columns and row bounds took nine launches); 64 requests 576 -> 446.
__global__ void __launch_bounds__(kSortWarps * 32) k_dual_finish(const __grid_constant__ DualCols D) {
    __shared__ int32_t sm[kSortWarps][kWarpSortCap];
    __shared__ int smin[kNumDims], smax[kNumDims], sact[kNumDims];
    const int64_t base = D.misc[0];
    if (base < 0) return;
    if (threadIdx.x < kNumDims) {
        smin[threadIdx.x] = INT_MAX;
        smax[threadIdx.x] = -1;
        sact[threadIdx.x] = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t half = (D.n + 1) / 2;
    for (int64_t c0 = (int64_t(blockIdx.x) * kSortWarps + w) * 32; c0 < half;
         c0 += int64_t(gridDim.x) * kSortWarps * 32) {
        const int64_t c = c0 + lane < half ? c0 + lane : -1;
        const int64_t j = c < 0 ? -1 : D.n - 1 - c;
        Mirror mc, mj;
        read_mirror(D, j, mc);
        read_mirror(D, c, mj);
        Slot tc, tj;
        const int64_t j2 = j == c ? -1 : j;
        read_place(D, base, c, tc);
        read_place(D, base, j2, tj);
        read_entries(D, mc, tc);
        read_entries(D, mj, tj);
        finish_columns(D, base, c, mc, tc, sm[w], smin, smax, sact);
        finish_columns(D, base, j2, mj, tj, sm[w], smin, smax, sact);
    }
    __syncthreads();
    if (threadIdx.x < kNumDims) {
        if (smin[threadIdx.x] != INT_MAX) atomicMin(&D.info->min_row[threadIdx.x], smin[threadIdx.x]);
        if (smax[threadIdx.x] >= 0) atomicMax(&D.info->max_row[threadIdx.x], smax[threadIdx.x]);
        if (sact[threadIdx.x]) atomicAdd(&D.info->act_end[threadIdx.x], sact[threadIdx.x]);
    }
}

// number of entries taken from a among the first `diag` outputs of merge(a, b)
__device__ __forceinline__ int64_t merge_split(const int32_t* a, int64_t na, const int32_t* b, int64_t nb,
                                               int64_t diag) {
    int64_t lo = diag > nb ? diag - nb : 0, hi = diag < na ? diag : na;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a[mid] <= b[diag - 1 - mid]) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// One CTA sorts the long columns one after the other: bitonic sorts of
// kLongChunk-int chunks in shared memory, then rounds of pairwise merges
// between the column and `tmp` (at least as long as the longest column).
__global__ void __launch_bounds__(kLongThreads) k_dual_sort_long(const int64_t* off, const int64_t* misc,
                                                                 int32_t* arena, const int32_t* longlist,
                                                                 int32_t* tmp) {
    __shared__ int32_t s[kLongChunk];
    const int64_t base = misc[0];
    if (base < 0) return;
    const int64_t nlong = misc[2];
    const int t = threadIdx.x;
    for (int64_t q = 0; q < nlong; q++) {
        int32_t* hdr = arena + base + off[longlist[q]];
        const int64_t len = hdr[0];
        int32_t* data = hdr + kHdr;
        for (int64_t ch = 0; ch < len; ch += kLongChunk) {
            const int m = int(len - ch < kLongChunk ? len - ch : kLongChunk);
            const int p = next_pow2(m);
            for (int i = t; i < p; i += kLongThreads) s[i] = i < m ? data[ch + i] : INT_MAX;
            __syncthreads();
            for (int k = 2; k <= p; k <<= 1) {
                for (int j = k >> 1; j > 0; j >>= 1) {
                    for (int i = t; i < p; i += kLongThreads) {
                        const int ixj = i ^ j;
                        if (ixj > i) {
                            const int32_t a = s[i], b = s[ixj];
                            if ((a > b) == ((i & k) == 0)) {
                                s[i] = b;
                                s[ixj] = a;
                            }
                        }
                    }
                    __syncthreads();
                }
            }
            for (int i = t; i < m; i += kLongThreads) data[ch + i] = s[i];
            __syncthreads();
        }
        int32_t* src = data;
        int32_t* dst = tmp;
        for (int64_t w = kLongChunk; w < len; w <<= 1) {
            for (int64_t a0 = 0; a0 < len; a0 += 2 * w) {
                const int64_t na = (a0 + w < len ? w : len - a0);
                const int64_t nb = (a0 + 2 * w < len ? w : (len - a0 - na > 0 ? len - a0 - na : 0));
                const int32_t* A = src + a0;
                const int32_t* B = A + na;
                const int64_t tot = na + nb;
                const int64_t per = (tot + kLongThreads - 1) / kLongThreads;
                const int64_t o0 = int64_t(t) * per < tot ? int64_t(t) * per : tot;
                const int64_t o1 = o0 + per < tot ? o0 + per : tot;
                int64_t ia = merge_split(A, na, B, nb, o0);
                int64_t ib = o0 - ia;
                for (int64_t o = o0; o < o1; o++) {
                    if (ia < na && (ib >= nb || A[ia] <= B[ib])) dst[a0 + o] = A[ia++];
                    else dst[a0 + o] = B[ib++];
                }
            }
            __syncthreads();
            int32_t* x = src;
            src = dst;
            dst = x;
        }
        if (src != data)
            for (int64_t i = t; i < len; i += kLongThreads) data[i] = src[i];
        __syncthreads();
    }
}

// [2 n], in the pairs' death list, which is free until they are extracted
int32_t* dual_lengths(const Device& D) { return reinterpret_cast<int32_t*>(D.death_of); }

}  // namespace

int dualize_begin(Device& D, int mode, cudaStream_t s) {
    const int64_t n = D.n;
    const unsigned g = grid_of(n, 256, 65536);
    // the columns' lengths, and as many counters for the fill (the scan between the two
    // reads the lengths, so they have to stay)
    int32_t* cnt = dual_lengths(D);
    int32_t* filled = cnt + n;
    int64_t* off = D.scratch64;
    const int skip = mode == 2;
    cudaMemsetAsync(cnt, 0, 2 * sizeof(int32_t) * n, s);
    k_dual_count<<<g, 256, 0, s>>>(n, D.arena, D.desc, skip, D.diminfo, cnt);
    scan([=] __device__(int64_t c) -> int64_t { return slot_ints(cnt[c]); },
         [=] __device__(int64_t c, int64_t pre, int64_t) { off[c] = pre; }, n, D.blk, s, DualReserve{n, D.arena_top, D.arena_cap, D.misc, D.diminfo, D.err});
    k_dual_fill<<<g, 256, 0, s>>>(n, D.desc, skip, D.diminfo, off, D.misc, filled, D.arena);
    return 3;
}

int dualize_end(Device& D, int mode, cudaStream_t s) {
    const int64_t n = D.n;
    // the row bounds go to the DimInfo through a few atomics per block: few blocks
    k_dual_finish<<<grid_of((n + 1) / 2, kSortWarps * 32, 2048), kSortWarps * 32, 0, s>>>(
        DualCols{n, D.scratch64, dual_lengths(D), D.misc, D.arena, D.active, D.desc, D.low, D.dim, D.pivot, D.state, D.cleared,
                 D.app, D.diminfo, D.err, mode == 2});
    // the pairs buffer (4n ints) is free until the pairs are extracted
    k_dual_sort_long<<<1, kLongThreads, 0, s>>>(D.scratch64, D.misc, D.arena, D.active,
                                                reinterpret_cast<int32_t*>(D.pairs));
    return 2;
}

}  // namespace sspp
