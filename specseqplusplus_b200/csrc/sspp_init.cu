// Dimension reorder, init passes, active lists and pair extraction.
//
// Reference counterparts:
//   dimension-stable reorder           include/specseq.h:439-483 (Formatted)
//   lowest one / leftmost column       include/kernel.h:444-457 (initleft_kernel)
//   apparent pivots, youngest-facet
//   clearing, negative columns         include/kernel.h:459-481 (initlookup_kernel)
//   clearing                           include/kernel.h:483-493 (clearing_kernel)
//   row compression                    include/kernel.h:495-520 (compress_kernel)
//   active list and per-dim bounds     include/specseq.h:365-409 (ColumnShrink)
//   pairs in input indices, sorted     include/specseq.h:1182-1193
// Here the reorder, the padded column layout and the compaction are device
// passes (the reference does them on the host), the active list is a device
// stream compaction, and pairs come out sorted by construction (each simplex is
// the birth of at most one pair, so compaction in birth order sorts them).
#include <climits>

#include "sspp_launch.h"
#include "sspp_scan.cuh"

namespace sspp {

template <typename T>
__global__ void k_fill(T* p, T v, int64_t n) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) p[i] = v;
}

static unsigned grid_for(int64_t n, int threads) {
    int64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > (int64_t(1) << 30)) g = int64_t(1) << 30;
    return unsigned(g);
}

void fill_i32(int32_t* p, int32_t v, int64_t n, cudaStream_t s) {
    if (n > 0) k_fill<int32_t><<<grid_for(n, 256) > 4096 ? 4096 : grid_for(n, 256), 256, 0, s>>>(p, v, n);
}
void fill_i64(int64_t* p, int64_t v, int64_t n, cudaStream_t s) {
    if (n > 0) k_fill<int64_t><<<grid_for(n, 256) > 4096 ? 4096 : grid_for(n, 256), 256, 0, s>>>(p, v, n);
}

// Input validation before any index is used: dimensions in range and col_ptr
// non-decreasing from 0 to nnz (device-resident inputs are only checked here).
// The same pass counts the columns of each dimension, per tile for the reorder
// (dimcnt) and in total for the host (dimtot, zeroed before), and finds the
// longest column, and whether an edge has more than two faces.  It also starts the init passes' state of every column, in
// order: no leftmost column yet, no pivot owner, not cleared, not negative.  A warp
// takes 32 * kPartRounds consecutive columns (20.3 M columns: 101 us, where a ballot
// per dimension and round instead of packed counts took 115).
constexpr int kPartThreads = 256;
constexpr int kPartRounds = 4;  // 2, 4 and 8 measured alike on large inputs, 8 slower on small ones
constexpr int kPartTile = kPartThreads * kPartRounds;
static_assert(kNumDims <= 8 && 32 * kPartRounds < 256, "a warp's counts are packed in 8 bits a dimension");

int64_t part_tiles(int64_t n) { return (n + kPartTile - 1) / kPartTile; }

__global__ void __launch_bounds__(kPartThreads) k_validate(const int32_t* dims, const int64_t* colptr, int64_t n,
                                                           int64_t nnz, int32_t* dimcnt, Ctl* ctl, int32_t* leftmost,
                                                           uint64_t* pivot, uint8_t* cleared, uint8_t* negative) {
    __shared__ int s_cnt[kNumDims];
    __shared__ int s_len, s_bad, s_wide;
    if (threadIdx.x < kNumDims) s_cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_len = s_bad = s_wide = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t j0 = int64_t(blockIdx.x) * kPartTile + (threadIdx.x >> 5) * (32 * kPartRounds) + lane;
    unsigned long long mine = 0;  // columns of each dimension, 8 bits each (a warp's are at most 128)
    int longest = 0;
    bool bad = false, wide = false;
#pragma unroll
    for (int k = 0; k < kPartRounds; k++) {
        const int64_t j = j0 + 32 * k;
        int d = -1;
        if (j < n) {
            d = dims[j];
            const int64_t a = colptr[j], b = colptr[j + 1], len = b - a;
            if (d < 0 || d > kMaxDim || len < 0 || len > kMaxColLen || (j == 0 && a != 0) || (j == n - 1 && b != nnz))
                bad = true;
            else
                longest = max(longest, int(len));
            if (d >= 0 && d <= kMaxDim) mine += 1ull << (8 * d);
            wide = wide || (d == 1 && len > 2);
            leftmost[j] = INT_MAX;
            pivot[j] = kNoOwner;
            cleared[j] = 0;
            negative[j] = 0;
        }
    }
    mine = warp_sum(mine);
    if (lane < kNumDims && (mine >> (8 * lane)) & 255) atomicAdd(&s_cnt[lane], int((mine >> (8 * lane)) & 255));
    longest = __reduce_max_sync(kFull, longest);
    if (lane == 0 && longest) atomicMax(&s_len, longest);
    if (bad) s_bad = 1;
    if (wide) s_wide = 1;
    __syncthreads();
    if (threadIdx.x < kNumDims) {
        const int c = s_cnt[threadIdx.x];
        dimcnt[int64_t(blockIdx.x) * kNumDims + threadIdx.x] = c;
        if (c) atomicAdd(&ctl->dimtot[threadIdx.x], (unsigned long long)c);
    }
    if (threadIdx.x == 0) {
        if (s_len > 0) atomicMax(&ctl->max_len, s_len);
        if (s_bad) atomicOr(&ctl->err, ERRB_BAD_INPUT);
        if (s_wide) ctl->wide_edges = 1;
    }
}

int validate(Device& D, cudaStream_t s) {
    if (D.n <= 0) return 0;
    k_validate<<<unsigned(part_tiles(D.n)), kPartThreads, 0, s>>>(D.in_dims, D.in_colptr, D.n, D.nnz, D.dimcnt, D.ctl,
                                                              D.leftmost, D.pivot, D.cleared, D.negative);
    return 1;
}

// Batch of k complexes copied side by side: complex i's face indices are
// shifted by its first column cstart[i], and its col_ptr entries (without the
// leading 0) by its first entry estart[i].
__device__ __forceinline__ int32_t batch_member(const int64_t* start, int32_t k, int64_t x) {
    int32_t a = 0, b = k;  // largest a with start[a] <= x
    while (b - a > 1) {
        const int32_t m = (a + b) >> 1;
        if (start[m] <= x) a = m;
        else b = m;
    }
    return a;
}

__global__ void k_batch_rebase(int64_t n, int64_t nnz, int32_t k, const int64_t* cstart, const int64_t* estart,
                               int64_t* colptr, int32_t* rows, int* bad) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < nnz; t += stride) {
        const int32_t i = batch_member(estart, k, t);
        const int32_t r = rows[t];
        if (r < 0 || r >= cstart[i + 1] - cstart[i]) *bad = 1;  // a face outside its own complex
        rows[t] = r + int32_t(cstart[i]);
    }
    for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < n; j += stride)
        colptr[j + 1] += estart[batch_member(cstart, k, j)];
}

int batch_rebase(int64_t n, int64_t nnz, int32_t k, const int64_t* d_cstart, const int64_t* d_estart,
                 int64_t* colptr, int32_t* rows, int* d_bad, cudaStream_t s) {
    const int64_t m = n > nnz ? n : nnz;
    if (m == 0 || k <= 1) return 0;
    k_batch_rebase<<<grid_for(m, 256) > 16384 ? 16384 : grid_for(m, 256), 256, 0, s>>>(n, nnz, k, d_cstart, d_estart,
                                                                                       colptr, rows, d_bad);
    return 1;
}

// Per-complex result slices of a batch: the sorted pairs (by birth) and the
// ascending essentials of complex i start at the first entry >= cstart[i].
__global__ void k_batch_bounds(int32_t k, const int64_t* cstart, int64_t npairs, const int64_t* pairs, int64_t ness,
                               const int64_t* ess, int64_t* pstart, int64_t* estart) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= k; i += gridDim.x * blockDim.x) {
        const int64_t x = cstart[i];
        int64_t lo = 0, hi = npairs;
        while (lo < hi) {
            const int64_t m = (lo + hi) >> 1;
            if (pairs[2 * m] < x) lo = m + 1;
            else hi = m;
        }
        pstart[i] = lo;
        lo = 0;
        hi = ness;
        while (lo < hi) {
            const int64_t m = (lo + hi) >> 1;
            if (ess[m] < x) lo = m + 1;
            else hi = m;
        }
        estart[i] = lo;
    }
}

// pairs and essentials in their own complex's indices
__global__ void k_batch_localize(int64_t npairs, int64_t ness, int32_t k, const int64_t* cstart, const int64_t* pairs,
                                 const int64_t* ess, int64_t* lpairs, int64_t* less) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < npairs; t += stride) {
        const int64_t b = pairs[2 * t], o = cstart[batch_member(cstart, k, b)];
        lpairs[2 * t] = b - o;
        lpairs[2 * t + 1] = pairs[2 * t + 1] - o;
    }
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < ness; t += stride)
        less[t] = ess[t] - cstart[batch_member(cstart, k, ess[t])];
}

int batch_bounds(int32_t k, const int64_t* d_cstart, int64_t npairs, const int64_t* pairs, int64_t ness,
                 const int64_t* ess, int64_t* d_pstart, int64_t* d_estart, cudaStream_t s) {
    k_batch_bounds<<<grid_for(int64_t(k) + 1, 128), 128, 0, s>>>(k, d_cstart, npairs, pairs, ness, ess, d_pstart,
                                                                 d_estart);
    return 1;
}

int batch_localize(int64_t npairs, int64_t ness, int32_t k, const int64_t* d_cstart, const int64_t* pairs,
                   const int64_t* ess, int64_t* lpairs, int64_t* less, cudaStream_t s) {
    const int64_t m = npairs > ness ? npairs : ness;
    if (m == 0) return 0;
    k_batch_localize<<<grid_for(m, 256) > 16384 ? 16384 : grid_for(m, 256), 256, 0, s>>>(npairs, ness, k, d_cstart,
                                                                                         pairs, ess, lpairs, less);
    return 1;
}

// ------------------------------------------------------------------ reorder
// The passes below run before the host has read the validation's verdict: each
// leaves at once when the error word is set, so no unchecked index is used.

// Per-dimension totals -> dimension ranges of the reordered columns; also empties
// the active segments (act_end counts first) and the row bounds that later passes
// fill.
__device__ void dim_ranges(const int64_t* total, DimInfo* info) {
    int64_t at = 0;
    for (int d = 0; d < kNumDims; d++) {
        info->col_begin[d] = int32_t(at);
        at += total[d];
        info->col_end[d] = int32_t(at);
        info->act_begin[d] = info->act_end[d] = 0;
        info->min_row[d] = INT_MAX;
        info->max_row[d] = -1;
    }
}

// First reordered index of each tile's columns of each dimension (dimcnt, in
// place), and the ranges.  One block; thread (chunk, dimension) takes a chunk of
// consecutive tiles.  Inputs of up to kInlineTiles tiles skip it: their tiles add
// up the counts themselves.
constexpr int kInlineTiles = 256;
__global__ void __launch_bounds__(1024) k_dim_offsets(int32_t* dimcnt, int64_t nb, Ctl* ctl) {
    if (ctl->err) return;
    __shared__ int64_t s_sum[128][kNumDims];
    __shared__ int64_t s_total[kNumDims];
    const int d = threadIdx.x & 7, c = threadIdx.x >> 3;
    const int64_t per = (nb + 127) / 128, b0 = c * per, b1 = b0 + per < nb ? b0 + per : nb;
    int64_t sum = 0;
    for (int64_t b = b0; b < b1; b++) sum += dimcnt[b * kNumDims + d];
    s_sum[c][d] = sum;
    __syncthreads();
    if (threadIdx.x < kNumDims) {
        int64_t run = 0;
        for (int k = 0; k < 128; k++) {
            const int64_t v = s_sum[k][threadIdx.x];
            s_sum[k][threadIdx.x] = run;
            run += v;
        }
        s_total[threadIdx.x] = run;
    }
    __syncthreads();
    if (threadIdx.x == 0) dim_ranges(s_total, &ctl->info);
    int64_t run = s_sum[c][d];
    for (int q = 0; q < d; q++) run += s_total[q];
    for (int64_t b = b0; b < b1; b++) {
        const int32_t v = dimcnt[b * kNumDims + d];
        dimcnt[b * kNumDims + d] = int32_t(run);
        run += v;
    }
}

// Stable rank of each column inside its dimension -> reordered index.  Unless
// every column is short, also records its length for the slot scan that follows.
__global__ void __launch_bounds__(kPartThreads) k_dim_assign(const int32_t* dims, const int64_t* colptr, int64_t n,
                                                             int64_t nb, const int32_t* dimcnt, Ctl* ctl,
                                                             int32_t* newidx, int32_t* perm, int32_t* rdim,
                                                             int32_t* rlen) {
    if (ctl->err) return;
    constexpr int kWarps = kPartThreads / 32;
    __shared__ int s_warp[kWarps][kNumDims];
    __shared__ int64_t s_base[kNumDims], s_total[kNumDims];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t tile = blockIdx.x;
    const bool all_short = ctl->max_len <= kShortLen;
    if (tile == 0 && threadIdx.x == 0 && all_short) ctl->arena_top = (unsigned long long)(kShortSlot * n);
    const int64_t j0 = tile * kPartTile + wid * (32 * kPartRounds) + lane;
    int d[kPartRounds], r[kPartRounds];
#pragma unroll
    for (int k = 0; k < kPartRounds; k++) d[k] = j0 + 32 * k < n ? dims[j0 + 32 * k] : -1;
    if (nb <= kInlineTiles) {  // warp q: dimension q
        int64_t before = 0, total = 0;
        for (int64_t b = lane; b < nb; b += 32) {
            const int64_t v = dimcnt[b * kNumDims + wid];
            total += v;
            if (b < tile) before += v;
        }
        before = warp_sum(before);
        total = warp_sum(total);
        if (lane == 0) {
            s_base[wid] = before;
            s_total[wid] = total;
        }
    } else if (threadIdx.x < kNumDims) {
        s_base[threadIdx.x] = dimcnt[tile * kNumDims + threadIdx.x];
    }
    // rank within the warp's columns, and the warp's counts, of the dimensions there are
    // (20.3 M columns in four dimensions: 100 us, 143 with ballots for all eight)
    unsigned present = 0;
#pragma unroll
    for (int q = 0; q < kNumDims; q++) present |= unsigned(ctl->dimtot[q] != 0) << q;
    int run[kNumDims] = {};
#pragma unroll
    for (int k = 0; k < kPartRounds; k++) {
        r[k] = 0;
#pragma unroll
        for (int q = 0; q < kNumDims; q++) {
            if (!((present >> q) & 1)) continue;
            const unsigned m = __ballot_sync(kFull, d[k] == q);
            if (d[k] == q) r[k] = run[q] + __popc(m & lanemask_lt());
            run[q] += __popc(m);
        }
    }
#pragma unroll
    for (int q = 0; q < kNumDims; q++)
        if (lane == q) s_warp[wid][q] = run[q];
    __syncthreads();
    if (nb <= kInlineTiles) {
        if (tile == 0 && threadIdx.x == 0) dim_ranges(s_total, &ctl->info);
        if (threadIdx.x < kNumDims) {
            int64_t at = s_base[threadIdx.x];
            for (int q = 0; q < threadIdx.x; q++) at += s_total[q];
            s_base[threadIdx.x] = at;
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kPartRounds; k++) {
        if (d[k] < 0) continue;
        const int64_t j = j0 + 32 * k;
        int64_t at = s_base[d[k]] + r[k];
        for (int w = 0; w < wid; w++) at += s_warp[w][d[k]];
        const int32_t idx = int32_t(at);
        newidx[j] = idx;
        perm[idx] = int32_t(j);
        rdim[idx] = d[k];
        if (!all_short) rlen[idx] = int32_t(colptr[j + 1] - colptr[j]);
    }
}

// Copies input column j into the padded arena slot of its reordered index
// i = newidx[j] with rows remapped to reordered indices; validates range,
// strict order and face dimension (a face of a dimension-d column must land in
// the reordered range of dimension d-1).  Threads walk the input columns, so
// col_ptr and the faces are read in order and each slot is written whole.
// With `lows` it also does the first init pass (include/kernel.h:444-457):
// the column's lowest row, and each row's leftmost column by atomicMin (the
// stable reorder keeps a column's rows ascending), read first: the columns of a
// row come roughly in order, so most find an earlier one there.  Short columns
// go through registers and are stored as two 16-byte halves of their slot; their
// descriptors are left to the compression unless write_desc asks for them (they are
// read before it, or also when it does not run).
// A column is a chain of four dependent trips to memory with little to do in between: at
// 64^3 neither memory (29% of its bandwidth) nor L2 (43%) was busy.  The reads of a
// trip go out together, of K columns on large inputs (K = 2: 32 registers, 4 bytes spilled).
template <int K>
__global__ void __launch_bounds__(256) k_scatter_cols(int64_t n, const int64_t* colptr, const int32_t* rows, const int32_t* dims,
                               const int32_t* newidx, const int64_t* off, Ctl* ctl, int32_t* arena,
                               uint64_t* desc, int32_t* low, int32_t* leftmost, bool lows, bool write_desc) {
    if (ctl->err & ~ERRB_FACES) return;
    __shared__ int32_t s_beg[kNumDims], s_end[kNumDims];
    if (threadIdx.x < kNumDims) {
        s_beg[threadIdx.x] = ctl->info.col_begin[threadIdx.x];
        s_end[threadIdx.x] = ctl->info.col_end[threadIdx.x];
    }
    __syncthreads();
    const bool all_short = ctl->max_len <= kShortLen;
    for (int64_t j0 = blockIdx.x * int64_t(256 * K) + threadIdx.x; j0 < n; j0 += int64_t(gridDim.x) * (256 * K)) {
        if (all_short) {
            int len[K], i[K], dj[K];
            int64_t b[K];
            int32_t x[K][kShortLen];
            unsigned bad = 0;
#pragma unroll
            for (int q = 0; q < K; q++) {
                const int64_t j = j0 + 256 * q;
                len[q] = 0;
                i[q] = -1;
                dj[q] = 0;
                b[q] = 0;
                if (j < n) {
                    b[q] = colptr[j];
                    len[q] = int(colptr[j + 1] - b[q]);
                    i[q] = newidx[j];
                    dj[q] = dims[j];
                }
            }
#pragma unroll
            for (int q = 0; q < K; q++)
#pragma unroll
                for (int k = 0; k < kShortLen; k++) x[q][k] = k < len[q] ? rows[b[q] + k] : INT_MAX;
#pragma unroll
            for (int q = 0; q < K; q++)
#pragma unroll
                for (int k = 0; k < kShortLen; k++)
                    if (k < len[q] && (x[q][k] < 0 || x[q][k] >= n || (k > 0 && x[q][k] <= x[q][k - 1]))) bad |= 1u << q;
#pragma unroll
            for (int q = 0; q < K; q++)
#pragma unroll
                for (int k = 0; k < kShortLen; k++)
                    if (k < len[q] && !((bad >> q) & 1)) x[q][k] = newidx[x[q][k]];
#pragma unroll
            for (int q = 0; q < K; q++) {
                if (i[q] < 0) continue;
                const int32_t fb = dj[q] > 0 ? s_beg[dj[q] - 1] : 0, fe = dj[q] > 0 ? s_end[dj[q] - 1] : 0;
                int32_t last = -1;
#pragma unroll
                for (int k = 0; k < kShortLen; k++)
                    if (k < len[q]) {
                        if (x[q][k] < fb || x[q][k] >= fe) bad |= 1u << q;
                        last = x[q][k];
                    }
                const bool wrong = (bad >> q) & 1;
                const int64_t o = int64_t(kShortSlot) * i[q];
                const int32_t m = wrong ? 0 : len[q];
                *reinterpret_cast<int4*>(arena + o) = make_int4(m, i[q], 0, 0);
                *reinterpret_cast<int4*>(arena + o + kHdr) = wrong ? make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX)
                                                                   : make_int4(x[q][0], x[q][1], x[q][2], x[q][3]);
                if (write_desc) desc[i[q]] = pack_desc(uint64_t(o), uint32_t(m));
                if (lows) low[i[q]] = m == 0 ? -1 : last;
                len[q] = m;
            }
            if (bad) atomicOr(&ctl->err, ERRB_FACES);
            if (lows) {
                unsigned first = 0;  // rows whose leftmost column may be this one
#pragma unroll
                for (int q = 0; q < K; q++)
#pragma unroll
                    for (int k = 0; k < kShortLen; k++)
                        if (k < len[q] && __ldcg(leftmost + x[q][k]) > i[q]) first |= 1u << (q * kShortLen + k);
#pragma unroll
                for (int q = 0; q < K; q++)
#pragma unroll
                    for (int k = 0; k < kShortLen; k++)
                        if ((first >> (q * kShortLen + k)) & 1) atomicMin(&leftmost[x[q][k]], i[q]);
            }
            continue;
        }
        for (int q = 0; q < K; q++) {
            const int64_t j = j0 + 256 * q;
            if (j >= n) break;
            const int64_t b = colptr[j], len = colptr[j + 1] - b;
            const int32_t i = newidx[j];
            const int64_t o = off[i];
            const int dj = dims[j];
            const int32_t fb = dj > 0 ? s_beg[dj - 1] : 0, fe = dj > 0 ? s_end[dj - 1] : 0;
            bool bad = false;
            int32_t last = -1, prev = -1;
            int32_t* data = arena + o + kHdr;
            for (int64_t k = 0; k < len && !bad; k++) {
                const int32_t r = rows[b + k];
                if (r < 0 || r >= n || r <= prev) { bad = true; break; }
                const int32_t x = newidx[r];
                if (x < fb || x >= fe) { bad = true; break; }
                prev = r;
                data[k] = x;
                last = x;
            }
            const int64_t m = bad ? 0 : len;
            for (int64_t k = m; k < pad4(m); k++) data[k] = INT_MAX;
            *reinterpret_cast<int4*>(arena + o) = make_int4(int32_t(m), i, 0, 0);
            desc[i] = pack_desc(uint64_t(o), uint32_t(m));
            if (lows && !bad)
                for (int64_t k = 0; k < len; k++)
                    if (__ldcg(leftmost + data[k]) > i) atomicMin(&leftmost[data[k]], i);
            if (bad) atomicOr(&ctl->err, ERRB_FACES);
            if (lows) low[i] = bad || len == 0 ? -1 : last;
        }
    }
}

// Columns per thread of two passes over all columns, from 2^17 columns up (below, one
// each: apparent pairs of 55,000 columns 3.6 us with 1, 4.5 with 4; of 250,000 8.6 and
// 4.9).  20.3 M columns (93^3):
// apparent pairs 430 / 290 / 190 / 233 us with 1 / 2 / 4 / 8, the scatter 438 / 419 / 517
// with 1 / 2 / 4 (530 when each read of a leftmost column was followed by its atomic);
// 2.67 M (20,000 points) 70 / 46 / 36 / 41 and 73 / 73 / 85.
constexpr int64_t kManyCols = int64_t(1) << 17;
constexpr int kScatterCols = 2, kApparentCols = 4;
unsigned cols_grid(int64_t n, int k, int64_t most) {
    return unsigned(std::min<int64_t>((n + 256 * k - 1) / (256 * k), most));
}

int reorder(Device& D, bool lows, bool write_desc, cudaStream_t s) {
    const int64_t n = D.n, nb = part_tiles(n);
    int launches = 3;
    if (nb > kInlineTiles) {
        k_dim_offsets<<<1, 1024, 0, s>>>(D.dimcnt, nb, D.ctl);
        launches++;
    }
    // the active list is built later: until then its buffer holds the reordered lengths
    int32_t* rlen = D.active;
    k_dim_assign<<<unsigned(nb), kPartThreads, 0, s>>>(D.in_dims, D.in_colptr, n, nb, D.dimcnt, D.ctl, D.newidx, D.perm,
                                                       D.dim, rlen);
    // padded column offsets in reordered order, unless every column is short (in a
    // refused input they may be sums of old lengths; nobody reads them)
    int64_t* off = D.scratch64;
    Ctl* ctl = D.ctl;
    bool zeroed;
    int64_t* blk = scan_region(D, 0, &zeroed);
    scan([=] __device__(int64_t i) -> int64_t { return slot_ints(max(rlen[i], 0)); },
         [=] __device__(int64_t i, int64_t pre, int64_t) { off[i] = pre; }, n, blk, s,
         [=] __device__(int64_t total) { ctl->arena_top = (unsigned long long)total; }, zeroed, &ctl->max_len, kShortLen);
    const auto scatter = n < kManyCols ? k_scatter_cols<1> : k_scatter_cols<kScatterCols>;
    scatter<<<cols_grid(n, n < kManyCols ? 1 : kScatterCols, 65536), 256, 0, s>>>(
        n, D.in_colptr, D.in_rows, D.in_dims, D.newidx, off, D.ctl, D.arena, D.desc, D.low, D.leftmost, lows, write_desc);
    return launches;
}

// ------------------------------------------------------------- init passes
// lowest row and leftmost columns when the reorder did not compute them (an
// edge collapse emptied columns in between); leftmost starts at INT_MAX
__global__ void k_init_low(int64_t n, const int32_t* arena, const uint64_t* desc, int32_t* low, int32_t* leftmost) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        uint64_t d = desc[i];
        const int32_t* c = arena + desc_off(d) + kHdr;
        uint32_t len = desc_len(d);
        low[i] = len ? c[len - 1] : -1;
        for (uint32_t k = 0; k < len; k++) atomicMin(&leftmost[c[k]], int32_t(i));
    }
}

// A column's slot, length and entries (short columns: both halves of the slot in
// two 16-byte loads, no descriptor).
struct ColRef {
    int64_t slot;
    int len;
    int4 q;  // the entries of a short column
    __device__ __forceinline__ int32_t at(const int32_t* arena, int k, bool all_short) const {
        return all_short ? (k == 0 ? q.x : k == 1 ? q.y : k == 2 ? q.z : q.w) : arena[slot + kHdr + k];
    }
};
__device__ __forceinline__ ColRef col_ref(int64_t i, const int32_t* arena, const uint64_t* desc, bool all_short) {
    ColRef c;
    if (all_short) {
        c.slot = int64_t(kShortSlot) * i;
        c.len = arena[c.slot];
        c.q = *reinterpret_cast<const int4*>(arena + c.slot + kHdr);
    } else {
        const uint64_t d = desc[i];
        c.slot = int64_t(desc_off(d));
        c.len = int(desc_len(d));
        c.q = make_int4(0, 0, 0, 0);
    }
    return c;
}

// Three dependent trips a column; bound by their latency (at 64^3 21% of the memory's
// bandwidth, 14% of L2's), so a thread takes K columns at once on large inputs.
template <int K>
__global__ void __launch_bounds__(256) k_init_apparent(int64_t n, const int32_t* arena, const uint64_t* desc,
                                                       const int32_t* low, const int32_t* leftmost, uint64_t* pivot,
                                                       uint8_t* cleared, uint8_t* negative, Ctl* ctl) {
    if (ctl->err) return;
    const bool all_short = ctl->max_len <= kShortLen;
    long long app = 0;
    for (int64_t i0 = blockIdx.x * int64_t(256 * K) + threadIdx.x; i0 < n; i0 += int64_t(gridDim.x) * (256 * K)) {
        int32_t l[K], lm[K];
        int4 e[K];
        int len[K];
#pragma unroll
        for (int q = 0; q < K; q++) l[q] = i0 + 256 * q < n ? low[i0 + 256 * q] : -1;
#pragma unroll
        for (int q = 0; q < K; q++) lm[q] = l[q] >= 0 ? leftmost[l[q]] : -1;
        // the entries of the columns that are not their lowest row's leftmost one
#pragma unroll
        for (int q = 0; q < K; q++) {
            len[q] = 0;
            e[q] = make_int4(0, 0, 0, 0);
            if (all_short && l[q] >= 0 && lm[q] != int32_t(i0 + 256 * q)) {
                const ColRef c = col_ref(i0 + 256 * q, arena, desc, true);
                len[q] = c.len;
                e[q] = c.q;
            }
        }
        unsigned neg = 0;
#pragma unroll
        for (int q = 0; q < K; q++) {  // the lowest entry's is known; the others' at once
            const int32_t i = int32_t(i0 + 256 * q);
            const int32_t x = len[q] > 1 ? leftmost[e[q].x] : -1, y = len[q] > 2 ? leftmost[e[q].y] : -1,
                          z = len[q] > 3 ? leftmost[e[q].z] : -1;
            if (x == i || y == i || z == i) neg |= 1u << q;
        }
#pragma unroll
        for (int q = 0; q < K; q++) {
            const int64_t i = i0 + 256 * q;
            if (l[q] < 0) continue;
            cleared[l[q]] = 1;  // the youngest facet of any simplex is positive
            bool is_neg = (neg >> q) & 1;
            if (lm[q] == int32_t(i)) {  // no earlier column can ever reach row l
                pivot[l[q]] = pv_pack(int32_t(i), all_short ? uint64_t(kShortSlot) * uint64_t(i) : desc_off(desc[i]));
                is_neg = true;  // its other entries need not be looked at
                app++;
            } else if (!all_short) {
                const ColRef c = col_ref(i, arena, desc, false);
                for (int k = 0; k < c.len && !is_neg; k++) is_neg = leftmost[c.at(arena, k, false)] == int32_t(i);
            }
            if (is_neg) negative[i] = 1;
        }
    }
    app = warp_sum(app);
    if ((threadIdx.x & 31) == 0 && app) cnt_add(&ctl->counters[CNT_APPARENT], app);
}

// Clears positive columns and removes negative rows in place.  With `app` it
// also writes the inline apparent columns (Device::app): a column that owns its
// lowest row l by an apparent pair writes app[l]; a row without an owner
// writes its own entry (each row's entry has exactly one writer).  With
// `rinfo` (non-null: the reordered dimensions) it also gathers the per-
// dimension row bounds of the schedule (min first row over non-empty columns,
// max lowest row + 1 over active ones; ColumnShrink, include/specseq.h:374-398)
// into info, whose bounds must start at INT_MAX / -1.
__global__ void k_init_compress(int64_t n, int32_t* arena, uint64_t* desc, int32_t* low, const uint64_t* pivot,
                                const uint8_t* cleared, const uint8_t* negative, uint8_t* state,
                                const uint8_t* dropped, bool keep_rows, int4* app, const int32_t* rinfo, Ctl* ctl) {
    DimInfo* info = &ctl->info;
    long long* counters = ctl->counters;
    const bool all_short = ctl->max_len <= kShortLen;
    __shared__ int smin[kNumDims], smax[kNumDims], sact[kNumDims];
    __shared__ int s_err;  // one look per block: other blocks may set the error word meanwhile
    if (threadIdx.x == 0) s_err = ctl->err;
    if (threadIdx.x < kNumDims) {
        smin[threadIdx.x] = INT_MAX;
        smax[threadIdx.x] = -1;
        sact[threadIdx.x] = 0;
    }
    __syncthreads();
    if (s_err) return;
    long long ncl = 0, nact = 0;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        if (app && pivot[i] == kNoOwner) app[i] = make_int4(-1, INT_MAX, INT_MAX, INT_MAX);
        const bool drop = dropped && dropped[i];
        if (drop || cleared[i]) {
            const int64_t slot = all_short ? int64_t(kShortSlot) * i : int64_t(desc_off(desc[i]));
            const int32_t l = low[i];
            if (!drop && l >= 0 && pv_col(pivot[l]) == int32_t(i)) atomicOr(&ctl->err, ERRB_FACES);  // positive and negative
            desc[i] = pack_desc(uint64_t(slot), 0);  // its slot is not read any more
            low[i] = -1;
            state[i] = drop ? ST_DROPPED : ST_CLEARED;
            ncl += !drop;
            continue;
        }
        ColRef c = col_ref(i, arena, desc, all_short);
        int m = 0;
        int32_t l = -1, first = INT_MAX;
        int4 v = make_int4(-1, INT_MAX, INT_MAX, INT_MAX);  // the inline column, should it own its row
        if (all_short) {
            int32_t y[kShortLen] = {INT_MAX, INT_MAX, INT_MAX, INT_MAX};
#pragma unroll
            for (int k = 0; k < kShortLen; k++) {
                const int32_t r = k == 0 ? c.q.x : k == 1 ? c.q.y : k == 2 ? c.q.z : c.q.w;
                if (k < c.len && (keep_rows || !negative[r])) {
                    if (m == 0) y[0] = r;
                    else if (m == 1) y[1] = r;
                    else if (m == 2) y[2] = r;
                    else y[3] = r;
                    m++;
                    l = r;
                }
            }
            first = y[0];
            if (m != c.len) {
                arena[c.slot] = m;
                *reinterpret_cast<int4*>(arena + c.slot + kHdr) = make_int4(y[0], y[1], y[2], y[3]);
            }
            v = make_int4(m - 1, m > 1 ? y[0] : INT_MAX, m > 2 ? y[1] : INT_MAX, m > 3 ? y[2] : INT_MAX);
        } else {
            int32_t* col = arena + c.slot + kHdr;
            if (keep_rows) {
                m = c.len;
            } else {
                for (int k = 0; k < c.len; k++) {
                    const int32_t r = col[k];
                    if (!negative[r]) col[m++] = r;
                }
            }
            for (int k = m; k < c.len; k++) col[k] = INT_MAX;
            arena[c.slot] = m;
            if (m) {
                l = col[m - 1];
                first = col[0];
                if (m <= 4) v = make_int4(m - 1, m > 1 ? col[0] : INT_MAX, m > 2 ? col[1] : INT_MAX, m > 3 ? col[2] : INT_MAX);
            }
        }
        desc[i] = pack_desc(uint64_t(c.slot), uint32_t(m));
        low[i] = l;
        const uint8_t st = (m == 0) ? ST_ZERO : (pv_col(pivot[l]) == int32_t(i) ? ST_OWNER : ST_ACTIVE);
        state[i] = st;
        if (rinfo && m > 0) {
            const int dm = rinfo[i];
            atomicMin(&smin[dm], first);
            if (st == ST_ACTIVE) {
                atomicMax(&smax[dm], l + 1);
                atomicAdd(&sact[dm], 1);
            }
        }
        if (app && st == ST_OWNER) app[l] = v;
        nact += (st == ST_ACTIVE);
    }
    ncl = warp_sum(ncl);
    nact = warp_sum(nact);
    if ((threadIdx.x & 31) == 0) {
        if (ncl) cnt_add(&counters[CNT_CLEARED], ncl);
        if (nact) cnt_add(&counters[CNT_ACTIVE], nact);
    }
    if (rinfo) {
        __syncthreads();
        if (threadIdx.x < kNumDims) {
            if (smin[threadIdx.x] != INT_MAX) atomicMin(&info->min_row[threadIdx.x], smin[threadIdx.x]);
            if (smax[threadIdx.x] >= 0) atomicMax(&info->max_row[threadIdx.x], smax[threadIdx.x]);
            if (sact[threadIdx.x]) atomicAdd(&info->act_end[threadIdx.x], sact[threadIdx.x]);
        }
    }
}

int init_passes(Device& D, bool lows_done, cudaStream_t s) {
    const int64_t n = D.n;
    const unsigned g = grid_for(n, 256) > 65536 ? 65536 : grid_for(n, 256);
    if (!lows_done) k_init_low<<<g, 256, 0, s>>>(n, D.arena, D.desc, D.low, D.leftmost);
    const auto apparent = n < kManyCols ? k_init_apparent<1> : k_init_apparent<kApparentCols>;
    apparent<<<cols_grid(n, n < kManyCols ? 1 : kApparentCols, 65536), 256, 0, s>>>(n, D.arena, D.desc, D.low, D.leftmost, D.pivot, D.cleared, D.negative, D.ctl);
    return lows_done ? 1 : 2;
}

int init_compress(Device& D, const uint8_t* dropped, bool keep_rows, bool final, cudaStream_t s) {
    const int64_t n = D.n;
    // the row bounds go to the DimInfo through a few atomics per block: few blocks
    const unsigned g = grid_for(n, 256) > 4096 ? 4096 : grid_for(n, 256);
    k_init_compress<<<g, 256, 0, s>>>(n, D.arena, D.desc, D.low, D.pivot, D.cleared, D.negative, D.state, dropped,
                                      keep_rows, final ? D.app : nullptr, final ? D.dim : nullptr, D.ctl);
    return 1;
}

// Active list in reordered order (dimension segments are contiguous).  act_end
// holds each dimension's count of active columns, gathered with the row bounds;
// the scan's end turns the counts into segments.
int active_list(Device& D, cudaStream_t s) {
    const int64_t n = D.n;
    int32_t* act = D.active;
    DimInfo* info = D.diminfo;
    bool zeroed;
    int64_t* blk = scan_region(D, 1, &zeroed);
    scan(ScanBytes{D.state, ST_ACTIVE}, [=] __device__(int64_t i, int64_t pre) { act[pre] = int32_t(i); },
         n, blk, s,
         [=] __device__(int64_t) {
             int32_t at = 0;
             // reordered columns ascend with the dimension, or descend (dual)
             const bool down = info->col_begin[0] > info->col_begin[kNumDims - 1];
             for (int k = 0; k < kNumDims; k++) {
                 const int d = down ? kNumDims - 1 - k : k;
                 const int32_t c = info->act_end[d];
                 info->act_begin[d] = at;
                 info->act_end[d] = at += c;
             }
         },
         zeroed);
    return 1;
}

// ------------------------------------------------------------------- pairs
// Primal: input simplex j (reordered i) is a birth when row i has an owner, whose
// simplex is its death; it is a death when column i owns a row; neither, and not
// dropped by an edge collapse: essential.  (A column that owns a row is marked as an
// owner in every chain complex; in other matrices its marks may have gone with its lowest
// row, when that row is negative.  The counts show it, every column being one of a
// birth, a death, essential and dropped, and the pairs are then taken by the marks.)  One
// scan in input order writes both lists (births ascending, so the pairs come out sorted): it reads the maps and
// the pivot table in two nearly sequential streams per dimension, and only the
// deaths' input indices at random.  64^3: 81 us; a scatter by birth and two scans over
// its marks took 250.
struct PairsOut {
    int64_t n;
    const int32_t* newidx;
    const int32_t* perm;
    const uint64_t* pivot;
    const uint8_t* state;
    int64_t* pairs;
    int64_t* ess;
    long long* counters;
    int* err;
    int32_t edge_begin, edge_end;  // the edges, if reduced beside the dimensions above them
};
constexpr int64_t kBirths = (int64_t(1) << kScanClassShift) - 1;  // class 1: births, class 2: essentials

struct PairsValue {
    PairsOut o;
    __device__ ScanClass operator()(int64_t j) const {
        const int32_t i = o.newidx[j];
        const uint64_t e = o.pivot[i];
        const uint8_t st = o.state[i];
        return {uint8_t(e != kNoOwner ? 1 : (st == ST_OWNER || st == ST_DROPPED ? 0 : 2))};
    }
};
// kWide: a pair is one 16-byte store (the context's buffer); otherwise two stores of 8
// bytes, for a caller's buffer that only int64_t's alignment holds for.
template <bool kWide>
struct PairsSink {
    PairsOut o;
    __device__ void operator()(int64_t j, const int64_t (&pre)[kScanBatch], const uint8_t (&cls)[kScanBatch]) const {
        int32_t c[kScanBatch], death[kScanBatch];
        bool twice = false;
#pragma unroll
        for (int u = 0; u < kScanBatch; u++) c[u] = cls[u] == 1 ? o.newidx[j + 32 * u] : -1;
#pragma unroll
        for (int u = 0; u < kScanBatch; u++)
            if (c[u] >= 0) c[u] = pv_col(o.pivot[c[u]]);
#pragma unroll
        for (int u = 0; u < kScanBatch; u++) death[u] = c[u] >= 0 ? o.perm[c[u]] : -1;
        // an edge that owns a row may not be one itself (looked for here, at the vertices: in
        // the value above it cost 30 us at 64^3)
#pragma unroll
        for (int u = 0; u < kScanBatch; u++)
            if (c[u] >= o.edge_begin && c[u] < o.edge_end) twice = twice || o.pivot[c[u]] != kNoOwner;
#pragma unroll
        for (int u = 0; u < kScanBatch; u++) {
            if (cls[u] == 1) {
                int64_t* p = o.pairs + 2 * (pre[u] & kBirths);
                if constexpr (kWide) {
                    *reinterpret_cast<longlong2*>(p) = make_longlong2(j + 32 * u, death[u]);
                } else {
                    p[0] = j + 32 * u;
                    p[1] = death[u];
                }
            } else if (cls[u] == 2) {
                o.ess[pre[u] >> kScanClassShift] = j + 32 * u;
            }
        }
        if (twice) atomicOr(o.err, ERRB_ORDER);
    }
};
struct PairsDone {
    PairsOut o;
    __device__ void operator()(int64_t total) const {
        o.counters[CNT_NPAIRS] = total & kBirths;
        o.counters[CNT_NESS] = total >> kScanClassShift;
    }
};

// By marks.  Dual: the dual row r' owned by dual column c' maps back to the primal pair
// (n-1-c', n-1-r') of the dualized matrix's own numbering, and perm maps those
// to input indices; scattered by birth first, since a column that owns a row from
// the boundary matrix's pass (mode 2) is not marked as one.
__global__ void k_pairs_scatter(int64_t n, const uint64_t* pivot, const int32_t* perm, bool dual, int64_t* death_of,
                                uint8_t* paired) {
    for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < n; r += int64_t(gridDim.x) * blockDim.x) {
        const uint64_t e = pivot[r];
        if (e == kNoOwner) continue;
        const int64_t c = pv_col(e), birth = perm[dual ? n - 1 - c : r], death = perm[dual ? n - 1 - r : c];
        death_of[birth] = death;
        paired[birth] = 1;
        paired[death] = 1;
    }
}

__global__ void k_mark_dropped(int64_t n, const uint8_t* dropped, const int32_t* perm, uint8_t* paired) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        if (dropped[i]) paired[perm[i]] = 1;
}

// Small results go to pinned host memory with the control block, in the launch that
// would otherwise be the control block's copy: the calls that hand them out then only
// copy host memory, where each cost 20 us of copying and waiting (pairs and essentials
// of 6,700 columns 43 -> 10 us, of 55,000 columns 69 -> 21 us; results of several 100,000
// columns leave the host's caches on the way and gain nothing).
__global__ void __launch_bounds__(256) k_push_results(const Ctl* ctl, const int64_t* pairs, const int64_t* ess, Ctl* h_ctl,
                                                      int64_t* h_pairs, int64_t max_pairs, int64_t* h_ess,
                                                      int64_t max_ess) {
    const int64_t first = blockIdx.x * int64_t(256) + threadIdx.x, step = gridDim.x * int64_t(256);
    constexpr int kWords = int(offsetof(Ctl, step) / sizeof(int));
    for (int64_t i = first; i < kWords; i += step)
        reinterpret_cast<int*>(h_ctl)[i] = reinterpret_cast<const int*>(ctl)[i];
    const int64_t np = min(int64_t(ctl->counters[CNT_NPAIRS]), max_pairs);
    const int64_t ne = min(int64_t(ctl->counters[CNT_NESS]), max_ess);
    for (int64_t i = first; i < np; i += step)
        reinterpret_cast<longlong2*>(h_pairs)[i] = reinterpret_cast<const longlong2*>(pairs)[i];
    for (int64_t i = first; i < ne; i += step) h_ess[i] = ess[i];
}

int push_results(const Device& D, Ctl* h_ctl, int64_t* h_pairs, int64_t max_pairs, int64_t* h_ess, int64_t max_ess,
                 cudaStream_t s) {
    const unsigned g = unsigned(std::min<int64_t>(std::max<int64_t>((D.n + 255) / 256, 1), 64));
    k_push_results<<<g, 256, 0, s>>>(D.ctl, D.pairs, D.ess, h_ctl, h_pairs, max_pairs, h_ess, max_ess);
    return 1;
}

int extract_pairs(Device& D, int dual, const uint8_t* dropped, cudaStream_t s, bool marks, const int* unless) {
    const int64_t n = D.n;
    const PairsOut o{n, D.newidx, D.perm, D.pivot, D.state, D.pairs, D.ess, D.counters, D.err,
                     D.edge_begin, D.edge_end};
    bool zeroed;
    int64_t* blk = scan_region(D, 2, &zeroed);
    if (!dual && !marks) {
        if (reinterpret_cast<uintptr_t>(D.pairs) % sizeof(longlong2) == 0)
            scan(PairsValue{o}, PairsSink<true>{o}, n, blk, s, PairsDone{o}, zeroed, nullptr, 0, unless);
        else
            scan(PairsValue{o}, PairsSink<false>{o}, n, blk, s, PairsDone{o}, zeroed, nullptr, 0, unless);
        return 1;
    }
    // (the context's own buffer)
    longlong2* pairs = reinterpret_cast<longlong2*>(D.pairs);
    const unsigned g = grid_for(n, 256) > 65536 ? 65536 : grid_for(n, 256);
    fill_i64(D.death_of, -1, n, s);
    cudaMemsetAsync(D.negative, 0, n, s);  // reused as the "paired or dropped" mark
    k_pairs_scatter<<<g, 256, 0, s>>>(n, D.pivot, D.perm, dual != 0, D.death_of, D.negative);
    if (dropped) k_mark_dropped<<<g, 256, 0, s>>>(n, dropped, D.perm, D.negative);
    const int64_t* death_of = D.death_of;
    const uint8_t* paired = D.negative;
    int64_t* ess = D.ess;
    scan([=] __device__(int64_t j) -> ScanClass { return {uint8_t(death_of[j] >= 0 ? 1 : (paired[j] ? 0 : 2))}; },
         [=] __device__(int64_t j, const int64_t (&pre)[kScanBatch], const uint8_t (&cls)[kScanBatch]) {
             int64_t death[kScanBatch];
#pragma unroll
             for (int u = 0; u < kScanBatch; u++) death[u] = cls[u] == 1 ? death_of[j + 32 * u] : -1;
#pragma unroll
             for (int u = 0; u < kScanBatch; u++) {
                 if (cls[u] == 1) pairs[pre[u] & kBirths] = make_longlong2(j + 32 * u, death[u]);
                 else if (cls[u] == 2) ess[pre[u] >> kScanClassShift] = j + 32 * u;
             }
         },
         n, blk, s, PairsDone{o}, zeroed);
    return 3 + (dropped ? 1 : 0);
}

}  // namespace sspp
