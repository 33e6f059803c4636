// One-pass exclusive scan over an index space: value(i) -> count (int64_t, or
// ScanClass for a selection), sink(i, exclusive prefix, value), and at the end
// done(total).  Used for column offsets and stream compaction.
//
// value(i) must not read anything that a sink or done writes: a tile whose
// predecessors do not answer (kScanPolls) takes their values itself, when other
// tiles' sinks may have run already.
//
// Tiles of 4096 items (1024 in mid-sized scans) per 256-thread block.  A warp takes 512
// (128) consecutive items, 32 at a time, so that values are read and prefixes written coalesced.  Tiles
// publish their sums and read their predecessors' (decoupled look-back: Merrill and
// Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016; 256 tiles
// at a time: with a warp's 32 the prefix needed 50 hops over 1,605 tiles, and the
// pair lists took 217 us instead of 92), so every value is read once.  The three
// passes it replaces (sums, sums of sums, prefixes with 16 consecutive items per
// thread) took 18 + 3 + 46 us over 6.57 M lengths where this takes 41, and 5-9 us and
// three launches over a few thousand items, where this is one launch of 5 us (from
// 4,097 items on with a clearing of the tile states before it).
#pragma once
#include <type_traits>

#include "sspp_kernels.cuh"

namespace sspp {

constexpr int kScanThreads = 256;
// Items per lane.  A few items each put a scan of some ten thousand items on more SMs and
// shorten each lane's chain; on large inputs they mean more tiles to look back over.
// (Pairs of 6,700 columns 8 -> 4 us, of 55,000 9.5 -> 4.8, of 210,000 14 -> 11; whole
// requests 2-6% below 2^18 columns.)
constexpr int kScanItems = 16, kScanFewItems = 4;
constexpr int64_t kScanOneTile = kScanThreads * kScanItems;  // a single tile needs no look-back
constexpr int64_t kScanFewMax = int64_t(1) << 18;

// A tile's published state: flag in the top two bits (0 nothing, 1 the tile's own
// sum, 2 the sum up to and including it), the sum below.
constexpr unsigned long long kScanSum = 1ull << 62, kScanPrefix = 2ull << 62, kScanValue = kScanSum - 1;
#ifndef SSPP_SCAN_POLLS
#define SSPP_SCAN_POLLS (1 << 22)
#endif
constexpr int kScanPolls = SSPP_SCAN_POLLS;

__device__ __forceinline__ unsigned long long scan_load(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void scan_store(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The values of a lane (items lane + 32 k of its warp's, which start at `begin`) and their exclusive prefixes within the warp.
template <class T, int kItems>
struct ScanLane {  // numbers
    T v[kItems], ex[kItems];
    template <class F>
    __device__ __forceinline__ int64_t load(const F& value, int64_t begin, int64_t n) {
        const int64_t first = begin + (threadIdx.x & 31);
#pragma unroll
        for (int k = 0; k < kItems; k++) v[k] = first + 32 * k < n ? value(first + 32 * k) : T(0);
        T run = 0;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            const T inc = warp_inclusive_scan(v[k]);
            ex[k] = run + inc - v[k];
            run += __shfl_sync(kFull, inc, 31);
        }
        return int64_t(run);
    }
    template <class G>
    __device__ __forceinline__ void store(const G& sink, int64_t begin, int64_t n, int64_t base) const {
        const int64_t first = begin + (threadIdx.x & 31);
#pragma unroll
        for (int k = 0; k < kItems; k++)
            if (first + 32 * k < n) sink(first + 32 * k, base + int64_t(ex[k]), v[k]);
    }
    template <class F>
    static __device__ __forceinline__ int64_t number(const F& value, int64_t i, int64_t n) {
        return int64_t(value(i));
    }
};

// A selection: class 1 and class 2 of the items are counted side by side, in the
// low kScanClassShift bits of the prefix and above them (0: neither).  Ballots
// count them, so nothing but two masks is kept per 32 items.
constexpr int kScanClassShift = 31;
struct ScanClass {
    uint8_t c;
};
// Its sink takes kScanBatch items of a lane at a time (j, j + 32, ...: prefixes and
// classes, 0 also beyond the end), so that what it reads for them is under way together
// (pairs, a chain of three reads: 6,700 columns 12 us one item at a time, 8 by four, 8.5 by
// eight; 6.57 M 97 / 81 / 102; 20.3 M 270 / 248 / 300, eight costing warps).
constexpr int kScanBatch = 4;
template <int kItems>
struct ScanLane<ScanClass, kItems> {
    unsigned one[kItems], two[kItems];
    static __device__ __forceinline__ int64_t pack(int a, int b) { return int64_t(a) | (int64_t(b) << kScanClassShift); }
    template <class F>
    __device__ __forceinline__ int64_t load(const F& value, int64_t begin, int64_t n) {
        const int64_t first = begin + (threadIdx.x & 31);
        uint8_t c[kItems];
#pragma unroll
        for (int k = 0; k < kItems; k++) c[k] = first + 32 * k < n ? value(first + 32 * k).c : 0;
        int a = 0, b = 0;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            one[k] = __ballot_sync(kFull, c[k] == 1);
            two[k] = __ballot_sync(kFull, c[k] == 2);
            a += __popc(one[k]);
            b += __popc(two[k]);
        }
        return pack(a, b);
    }
    template <class G>
    __device__ __forceinline__ void store(const G& sink, int64_t begin, int64_t n, int64_t base) const {
        const unsigned lt = lanemask_lt();
        const int lane = threadIdx.x & 31;
        const int64_t first = begin + lane;
#pragma unroll
        for (int k0 = 0; k0 < kItems; k0 += kScanBatch) {
            int64_t pre[kScanBatch];
            uint8_t c[kScanBatch];
#pragma unroll
            for (int u = 0; u < kScanBatch; u++) {
                const unsigned a = one[k0 + u], b = two[k0 + u];
                c[u] = uint8_t(((a >> lane) & 1) | (((b >> lane) & 1) << 1));
                pre[u] = base + pack(__popc(a & lt), __popc(b & lt));
                base += pack(__popc(a), __popc(b));
            }
            sink(first + 32 * k0, pre, c);
        }
    }
    template <class F>
    static __device__ __forceinline__ int64_t number(const F& value, int64_t i, int64_t n) {
        const ScanClass x = value(i);
        return pack(x.c == 1, x.c == 2);
    }
};

// Selection by a byte array (16-byte aligned): items whose byte equals `want`.  A
// lane takes 16 consecutive items with one load; the sink sees selected items only.
struct ScanBytes {
    const uint8_t* p;
    uint8_t want;
    __device__ __forceinline__ ScanBytes operator()(int64_t) const { return *this; }
};
template <int kItems>
struct ScanLane<ScanBytes, kItems> {
    static_assert(kItems == 16, "one 16-byte load per lane");
    unsigned sel;  // bit k: item 16 * lane + k
    int pre;
    template <class F>
    __device__ __forceinline__ int64_t load(const F& value, int64_t begin, int64_t n) {
        const int64_t first = begin + 16 * (threadIdx.x & 31);
        sel = 0;
        if (first + 16 <= n) {
            const uint4 q = *reinterpret_cast<const uint4*>(value.p + first);
            const unsigned w[4] = {q.x, q.y, q.z, q.w}, all = value.want * 0x01010101u;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned eq = __vcmpeq4(w[k], all) & 0x08040201u;  // one bit of each equal byte
                sel |= ((eq | eq >> 8 | eq >> 16 | eq >> 24) & 15u) << (4 * k);
            }
        } else {
            for (int k = 0; k < 16; k++)
                if (first + k < n && value.p[first + k] == value.want) sel |= 1u << k;
        }
        const int cnt = __popc(sel), inc = warp_inclusive_scan(cnt);
        pre = inc - cnt;
        return __shfl_sync(kFull, inc, 31);
    }
    template <class G>
    __device__ __forceinline__ void store(const G& sink, int64_t begin, int64_t, int64_t base) const {
        const int64_t first = begin + 16 * (threadIdx.x & 31);
        base += pre;
        for (unsigned m = sel; m; m &= m - 1) sink(first + __ffs(m) - 1, base++);
    }
    template <class F>
    static __device__ __forceinline__ int64_t number(const F& value, int64_t i, int64_t n) {
        return value.p[i] == value.want;
    }
};

template <int kItems, class F, class G, class H>
__global__ void __launch_bounds__(kScanThreads) k_scan(F value, G sink, H done, int64_t n, int64_t nb, int64_t* blk,
                                                       const int* skip_upto, int skip_limit, const int* unless) {
    if (skip_upto && *skip_upto <= skip_limit) return;
    if (unless && *unless) return;
    using Lane = ScanLane<decltype(value(int64_t(0))), kItems>;
    constexpr int kTile = kScanThreads * kItems;
    constexpr int kWarps = kScanThreads / 32;
    __shared__ int64_t s_warp[kWarps];
    __shared__ int64_t s_look[kWarps];
    __shared__ int s_seen[kWarps];
    unsigned long long* state = reinterpret_cast<unsigned long long*>(blk);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t tile = blockIdx.x;
    const int64_t begin = tile * kTile + int64_t(wid) * (32 * kItems);
    Lane items;
    const int64_t run = items.load(value, begin, n);
    if (lane == 0) s_warp[wid] = run;
    __syncthreads();
    int64_t mine = 0, sum = 0;  // sums of the warps before this one, and of the tile
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        if (w < wid) mine += s_warp[w];
        sum += s_warp[w];
    }
    // look back, a tile per thread, to the nearest prefix
    int64_t base = 0;
    if (tile > 0) {
        if (threadIdx.x == 0) scan_store(state + tile, kScanSum | (unsigned long long)sum);
        int64_t t = tile - 1;
        for (int polls = 0;;) {
            const int64_t j = t - threadIdx.x;
            const unsigned long long x = j >= 0 ? scan_load(state + j) : kScanPrefix;
            const unsigned pm = __ballot_sync(kFull, (x >> 62) == 2), zm = __ballot_sync(kFull, (x >> 62) == 0);
            const unsigned upto = pm ? (pm & (0u - pm)) * 2 - 1 : kFull;  // lanes up to the first prefix
            const int64_t part = warp_sum((upto >> lane) & 1 ? int64_t(x & kScanValue) : int64_t(0));
            __syncthreads();  // the previous poll's results have been read
            if (lane == 0) {
                s_look[wid] = part;
                s_seen[wid] = (zm & upto) ? 0 : (pm ? 2 : 1);
            }
            __syncthreads();
            int64_t add = 0;
            int seen = 1;
            for (int w = 0; w < kWarps && seen == 1; w++) {
                seen = s_seen[w];
                add += s_look[w];
            }
            if (seen == 0) {
                if (++polls < kScanPolls) continue;
                // the predecessors do not answer: add their values up here
                base = 0;
                for (int64_t i = threadIdx.x; i < tile * kTile; i += kScanThreads) base += Lane::number(value, i, n);
                base = warp_sum(base);
                __syncthreads();
                if (lane == 0) s_look[wid] = base;
                __syncthreads();
                base = 0;
                for (int w = 0; w < kWarps; w++) base += s_look[w];
                break;
            }
            base += add;
            if (seen == 2) break;
            t -= kScanThreads;
        }
    }
    if (threadIdx.x == 0) {
        scan_store(state + tile, kScanPrefix | (unsigned long long)(base + sum));
        if (tile == nb - 1) {
            blk[nb] = base + sum;
            done(base + sum);
        }
    }
    items.store(sink, begin, n, base + mine);
}

struct ScanNoop {
    __device__ void operator()(int64_t) const {}
};

// Tiles of a scan of numbers or classes over n items, and of any scan over up to n items
// at most.
inline bool scan_few(int64_t n) { return n > kScanOneTile && n <= kScanFewMax; }
inline int64_t scan_blocks(int64_t n) {
    const int64_t tile = kScanThreads * (scan_few(n) ? kScanFewItems : kScanItems);
    return (n + tile - 1) / tile;
}
inline int64_t scan_most_blocks(int64_t n) {
    return (n + kScanOneTile - 1) / kScanOneTile + kScanFewMax / (kScanThreads * kScanFewItems);
}

// Scratch (blk) must hold scan_blocks(n) + 1 entries (a selection by bytes: as many as
// fewer); the total is left after the last tile's.  zeroed: the entries are zero already.
// A launch whose *skip_upto turns out to be at most skip_limit, or whose *unless is set,
// does nothing (neither may change while it runs).
template <class F, class G, class H = ScanNoop>
void scan(F value, G sink, int64_t n, int64_t* blk, cudaStream_t s, H done = H(), bool zeroed = false,
          const int* skip_upto = nullptr, int skip_limit = 0, const int* unless = nullptr) {
    constexpr bool bytes = std::is_same<F, ScanBytes>::value;
    const int64_t nb = bytes ? (n + kScanOneTile - 1) / kScanOneTile : scan_blocks(n);
    if (nb == 0) {
        cudaMemsetAsync(blk, 0, sizeof(int64_t), s);
        return;
    }
    if (nb > 1 && !zeroed) cudaMemsetAsync(blk, 0, sizeof(int64_t) * size_t(nb), s);
    if (!bytes && scan_few(n))
        k_scan<bytes ? kScanItems : kScanFewItems>
            <<<unsigned(nb), kScanThreads, 0, s>>>(value, sink, done, n, nb, blk, skip_upto, skip_limit, unless);
    else
        k_scan<kScanItems>
            <<<unsigned(nb), kScanThreads, 0, s>>>(value, sink, done, n, nb, blk, skip_upto, skip_limit, unless);
}

// Tile states of one of a Device's regions, zero unless a scan used them since
// the init passes' clearing (then *zeroed is false and the scan clears them).
inline int64_t* scan_region(Device& D, int q, bool* zeroed) {
    *zeroed = (D.blk_zero >> q) & 1;
    D.blk_zero &= ~(1u << q);
    return D.blk + q * D.blk_stride;
}

}  // namespace sspp
