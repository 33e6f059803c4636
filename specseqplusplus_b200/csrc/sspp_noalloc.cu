// Allocation-free reduction: sspp_reduce_noalloc (declared in include/sspp.h).
//
// Some callers cannot let a library allocate device memory.  A serving process
// that reserves all of its GPU memory up front for its own request pool has no
// room for, and no wish for, allocations it does not control; a pipeline that
// keeps several streams busy cannot afford cudaMalloc / cudaFree, which
// synchronise the whole device and stall every stream while they run.  The
// context API (sspp_create / sspp_reduce) allocates its buffers on first use,
// so such callers get this one entry point instead.
//
// Everything it needs lives in g_scratch below, a file-scope device array of
// kScratchInts ints (64 MiB) that every GPU which loads this library holds
// until the process exits.  The caller passes the boundary matrix and the
// output buffers, all in device memory; nothing else is allocated.  Limits:
// at most kMaxCols columns, and 3 * ncols + nnz + fill-in must fit in the
// array (the host rejects inputs that leave less than kFillReserve ints for
// fill-in; a reduction whose fill-in still overflows returns SSPP_ERR_CAPACITY and
// writes neither pairs nor their number).
//
// The array's device address is looked up with cudaGetSymbolAddress the
// first time the entry point runs on a device (with that device current) and
// cached per device, so the first call on each device should be made before
// any stream capture begins.  Every call then copies the kernel's status word
// back to the host and synchronises the stream, so it returns only once the
// reduction has finished.  Every call reuses the same array and leaves its
// contents behind; the kernel clears what must start empty (the pivot table,
// the arena cursor, the error word) itself.  Two calls that overlap on the
// GPU - on two streams, or from two threads - share the array and corrupt each
// other: serialise them.
//
// Validation happens in the kernel before any reduction: col_ptr must start
// at 0, end at nnz and never decrease (every column's range inside [0, nnz]),
// dimensions must lie in 0..7, and each column's faces must be ascending, in
// range and one dimension lower; anything else is SSPP_ERR_BAD_INPUT.
//
// Two ways.  For more than kFewCols columns, and while the engine's arrays (about 71
// bytes per column and the padded column arena) fit in the scratch array, its own
// passes run there on the caller's stream (reduce_in_scratch): the same reorder,
// apparent pairs and reduction kernels as the context API's, one block per dimension.
// Otherwise,
// and whenever that run does not end cleanly (malformed input, arena or fill-in
// limit, or a matrix that is not a chain complex where the two could differ),
// k_reduce_noalloc decides: the standard twist (clearing) reduction, dimensions
// from high to low, run by one thread block: columns one after another, each
// addition a block-wide merge of two sorted index lists.
//
// The pairs are the same for every well-formed matrix, chain complex or not: the
// negative-row compression, the only pass that needs the boundary of a boundary
// to be zero, is left out here, and a run in which a column is both a birth and a
// death (possible only without that property, where the twist's clearing would
// have come first) goes to k_reduce_noalloc.
//
// The fill-in limit is that of k_reduce_noalloc, which takes new room for every single
// addition.  The passes need far less (250 columns of 4,096 rows over rows owned by
// short columns overflow it after four of them), and how much depends on the order in
// which their blocks run, so their own additions say nothing about it: once the pairs
// are known, k_fill_account adds up what k_reduce_noalloc's would take.  More than
// its room is refused at once; where the account cannot tell, k_reduce_noalloc runs.
//
// Measured (B200, device-resident input): 700 points (7,678 columns) 9.5 ms by one
// block, 0.29 ms by the engine's passes, of which the account is 0.04.
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "sspp_kernels.cuh"
#include "sspp_launch.h"
#include "sspp_scan.cuh"

namespace {

#ifndef SSPP_SCRATCH_INTS
#define SSPP_SCRATCH_INTS (int64_t(16) << 20)
#endif
constexpr int64_t kScratchInts = SSPP_SCRATCH_INTS;  // 64 MiB
constexpr int64_t kMaxCols = int64_t(1) << 20;
constexpr int64_t kFillReserve = kScratchInts / 4;   // ints kept free for fill-in
constexpr int kCtl = 16;                            // control words at the start of the array
constexpr int kMaxDevices = 64;
constexpr int kThreads = 256;

// control words
enum { C_ERR = 0, C_TOP_LO = 1, C_TOP_HI = 2, C_NPAIRS_LO = 3, C_NPAIRS_HI = 4, C_MAXDIM = 5 };
enum { E_BAD_INPUT = 1, E_CAPACITY = 2 };

static __device__ __align__(256) int32_t g_scratch[kScratchInts];

void* g_scratch_addr[kMaxDevices] = {};
std::mutex g_setup_mu;

// block-wide exclusive prefix of v; tot = block total (two barriers)
__device__ int block_prefix(int v, int& tot, int* sm) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) sm[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int c = lane < kThreads / 32 ? sm[lane] : 0;
        int ci = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, ci, o);
            if (lane >= o) ci += t;
        }
        if (lane < kThreads / 32) sm[lane] = ci - c;
        if (lane == kThreads / 32 - 1) sm[kThreads / 32] = ci;
    }
    __syncthreads();
    tot = sm[kThreads / 32];
    int r = sm[wid] + inc - v;
    __syncthreads();
    return r;
}

__device__ int lower_bound_g(const int32_t* a, int n, int x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// out = a xor b; returns the output length
__device__ int block_xor(const int32_t* a, int na, const int32_t* b, int nb, int32_t* out, int* sm) {
    int ca = 0, cb = 0;
    const int n = na > nb ? na : nb;
    for (int base = 0; base < n; base += kThreads) {
        const int i = base + threadIdx.x;
        const bool va = i < na, vb = i < nb;
        const int x = va ? a[i] : 0, y = vb ? b[i] : 0;
        const int ra = va ? lower_bound_g(b, nb, x) : 0;
        const int rb = vb ? lower_bound_g(a, na, y) : 0;
        const bool ea = va && ra < nb && b[ra] == x;
        const bool eb = vb && rb < na && a[rb] == y;
        int ta, tb;
        const int pa = block_prefix(ea ? 1 : 0, ta, sm);
        const int pb = block_prefix(eb ? 1 : 0, tb, sm);
        if (va && !ea) out[i + ra - 2 * (ca + pa)] = x;
        if (vb && !eb) out[i + rb - 2 * (cb + pb)] = y;
        ca += ta;
        cb += tb;
    }
    __syncthreads();
    return na + nb - 2 * ca;
}

// Scratch layout (ints): [0, kCtl) control, pivot[n] (owner column of each
// row, -1 = none), off[n] and len[n] (current version of each column), then
// the arena: the input columns, followed by column versions created by
// additions.
__global__ void __launch_bounds__(kThreads) k_reduce_noalloc(int32_t* S, int64_t n, int64_t nnz, const int32_t* dims,
                                                            const int64_t* col_ptr, const int32_t* rows,
                                                            int64_t* pairs, int64_t* npairs) {
    __shared__ int sm[kThreads / 32 + 1];
    __shared__ int s_flag;
    int32_t* ctl = S;
    int32_t* pivot = S + kCtl;
    int32_t* off = pivot + n;
    int32_t* len = off + n;
    int32_t* arena = len + n;
    const int64_t arena_cap = kScratchInts - (kCtl + 3 * n);
    // what must start empty: error word, cursor, pivot table
    if (threadIdx.x == 0) {
        ctl[C_ERR] = 0;
        ctl[C_MAXDIM] = 0;
        s_flag = 0;
    }
    __syncthreads();
    if (col_ptr[0] != 0 || col_ptr[n] != nnz) {
        if (threadIdx.x == 0) ctl[C_ERR] = E_BAD_INPUT;
        return;
    }
    int maxd = 0;
    for (int64_t j = threadIdx.x; j < n; j += kThreads) {
        pivot[j] = -1;
        const int64_t b = col_ptr[j], e = col_ptr[j + 1];
        const int d = dims[j];
        // every column's range must lie inside [0, nnz] before any entry is
        // read or copied (the copy runs in the same pass as the checks)
        bool bad = b < 0 || e < b || e > nnz || d < 0 || d > sspp::kMaxDim;
        for (int64_t k = b; k < e && !bad; k++) {
            const int32_t r = rows[k];
            if (r < 0 || r >= n || (k > b && r <= rows[k - 1]) || dims[r] != d - 1) bad = true;
            else arena[k] = r;
        }
        if (bad) atomicOr(&s_flag, E_BAD_INPUT);
        off[j] = int32_t(b);
        len[j] = bad ? 0 : int32_t(e - b);
        maxd = d > maxd ? d : maxd;
    }
    atomicMax(&ctl[C_MAXDIM], maxd);
    __syncthreads();
    if (s_flag) {
        if (threadIdx.x == 0) ctl[C_ERR] = s_flag;
        return;
    }
    const int top_dim = ctl[C_MAXDIM];
    int64_t top = nnz;  // arena cursor (same value in every thread)
    for (int d = top_dim; d >= 1; d--) {
        for (int64_t j = 0; j < n; j++) {
            if (dims[j] != d || len[j] == 0) continue;  // other dimension, zero or cleared
            int32_t* w = arena + off[j];
            int wl = len[j];
            bool failed = false;
            while (wl > 0) {
                const int L = w[wl - 1];
                const int p = pivot[L];
                if (p < 0) break;
                const int32_t* pb = arena + off[p];
                const int pl = len[p];
                if (top + wl + pl > arena_cap) { failed = true; break; }
                int32_t* o = arena + top;
                const int ol = block_xor(w, wl, pb, pl, o, sm);
                top += wl + pl;
                w = o;
                wl = ol;
            }
            if (failed) {
                if (threadIdx.x == 0) ctl[C_ERR] = E_CAPACITY;
                return;
            }
            if (threadIdx.x == 0) {
                off[j] = int32_t(w - arena);
                len[j] = wl;
                if (wl > 0) {
                    const int L = w[wl - 1];
                    pivot[L] = int32_t(j);
                    len[L] = 0;  // twist: the column of the lowest row is positive
                }
            }
            __syncthreads();
        }
    }
    // pairs in birth order: row r owned by column c is the pair (r, c)
    int64_t written = 0;
    for (int64_t base = 0; base < n; base += kThreads) {
        const int64_t r = base + threadIdx.x;
        const int c = r < n ? pivot[r] : -1;
        int tot;
        const int pre = block_prefix(c >= 0 ? 1 : 0, tot, sm);
        if (c >= 0) {
            pairs[2 * (written + pre)] = r;
            pairs[2 * (written + pre) + 1] = c;
        }
        written += tot;
    }
    if (threadIdx.x == 0) {
        *npairs = written;
        ctl[C_TOP_LO] = int32_t(top & 0xffffffff);
        ctl[C_TOP_HI] = int32_t(top >> 32);
    }
}

// ---------------------------------------------------------------------------
// the engine's passes in the scratch array

using namespace sspp;

constexpr int kCap1 = 64;          // warp-tier column capacity (ints), as the context API's bound
constexpr int kCap2 = 8192;        // CTA-tier column capacity
// Up to here k_reduce_noalloc is done before the passes' launches and two waits are:
// 51 / 92 / 134 / 201 columns 54 / 92 / 115 / 154 us against 90 / 145 / 155 / 173,
// 226 / 293 / 410 columns 197 / 153 / 337 against 192 / 148 / 221.
constexpr int64_t kFewCols = 224;
constexpr int64_t kGuard = 8192;   // ints after the arena: staging reads a first pass beyond a slot

// Engine arrays carved out of the scratch array; false when they leave too
// little for the arena.  Buffers whose lifetimes do not meet share memory: the
// pairs pass's essentials lie in the column descriptors.
bool carve(int32_t* scratch, int64_t n, int64_t nnz, Device& D) {
    char* p = reinterpret_cast<char*>(scratch);
    char* const end = p + sizeof(int32_t) * kScratchInts;
    auto take = [&](auto*& out, int64_t count) {
        using T = std::remove_reference_t<decltype(*out)>;
        out = reinterpret_cast<T*>(p);
        p += (sizeof(T) * size_t(count) + 255) & ~size_t(255);
    };
    // cleared together: the control block and the scans' tile states
    take(D.ctl, 1);
    D.blk_stride = scan_most_blocks(n) + 2;
    take(D.blk, 3 * D.blk_stride);
    take(D.dim, n);
    take(D.perm, n);
    take(D.newidx, n);
    take(D.scratch64, n + 1);
    take(D.desc, n + 1);
    take(D.low, n);
    take(D.pivot, n);
    take(D.state, n);
    take(D.cleared, n);
    take(D.negative, n);
    take(D.leftmost, n);
    take(D.active, n);
    take(D.app, n);
    take(D.dimcnt, (part_tiles(n) + 1) * kNumDims);
    D.pool_cap = n;
    take(D.heavy, D.pool_cap);
    D.arena = reinterpret_cast<int32_t*>(p);
    D.arena_cap = p < end ? ((end - p) / int64_t(sizeof(int32_t)) - kGuard) & ~int64_t(3) : 0;
    D.n = n;
    D.nnz = nnz;
    D.diminfo = &D.ctl->info;
    D.counters = D.ctl->counters;
    D.arena_top = &D.ctl->arena_top;
    D.err = &D.ctl->err;
    D.pool_tail = &D.ctl->pool_tail;
    D.heavy_done = &D.ctl->heavy_done;
    D.ess = reinterpret_cast<int64_t*>(D.desc);
    // the input's slots, and as much again for the reduction's column versions
    return D.arena_cap >= 2 * (nnz + (kHdr + 3) * n + 4);
}

// A column that owns a row and whose own row is owned (see the header).
__global__ void k_check_complex(int64_t n, const uint64_t* pivot, const uint8_t* state, int* err) {
    for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < n; r += int64_t(gridDim.x) * blockDim.x)
        if (pivot[r] != kNoOwner && state[r] == ST_OWNER) atomicOr(err, ERRB_CHECK);
}

// *npairs is written by a run that ends cleanly only.
__global__ void k_store_npairs(const Ctl* st, int64_t* npairs) {
    if (st->err == 0) *npairs = st->counters[CNT_NPAIRS];
}

// The device's multiprocessors and the reduction kernels' blocks per
// multiprocessor, once per device.
struct Launch {
    int sms = 0, light = 0, heavy = 0;
};

cudaError_t launch_shape(int dev, Launch* out) {
    static Launch known[kMaxDevices];
    std::lock_guard<std::mutex> lock(g_setup_mu);
    Launch& l = known[dev];
    if (l.sms == 0) {
        Launch f;
        cudaError_t e = reduce_configure(kCap1, kCap2, 256, &f.light, &f.heavy);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&f.sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        if (f.light < 1 || f.heavy < 1) return cudaErrorInvalidConfiguration;
        l = f;
    }
    *out = l;
    return cudaSuccess;
}

// How a run of the engine's passes ended: the pairs are in place, or their fill-in is
// refused, or k_reduce_noalloc has to run.
enum class Ended { Done, Refused, Unknown };

// Runs the engine's passes in the scratch array.
cudaError_t reduce_in_scratch(int32_t* scratch, int dev, int64_t n, int64_t nnz, const int32_t* d_dims,
                              const int64_t* d_col_ptr, const int32_t* d_rows, int64_t* d_pairs, int64_t* d_npairs,
                              cudaStream_t s, Ended* ended) {
    *ended = Ended::Unknown;
    Device D;
    if (n <= kFewCols || !carve(scratch, n, nnz, D)) return cudaSuccess;
    Launch shape;
    cudaError_t e = launch_shape(dev, &shape);
    if (e != cudaSuccess) return e;
    D.in_dims = const_cast<int32_t*>(d_dims);
    D.in_colptr = const_cast<int64_t*>(d_col_ptr);
    D.in_rows = const_cast<int32_t*>(d_rows);
    D.pairs = d_pairs;
    Ctl h;
    cudaMemsetAsync(D.ctl, 0, size_t(reinterpret_cast<char*>(D.blk + 3 * D.blk_stride) - reinterpret_cast<char*>(D.ctl)), s);
    D.blk_zero = 7;
    validate(D, s);  // the passes leave when it finds a fault
    reorder(D, true, false, s);
    init_passes(D, true, s);
    init_compress(D, nullptr, true, true, s);
    active_list(D, s);
    cudaMemcpyAsync(&h, D.ctl, offsetof(Ctl, step), cudaMemcpyDeviceToHost, s);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    if (h.err) return cudaSuccess;
    int* ctr = D.ctl->step;  // cleared with the control block, one step per dimension
    for (int d = kMaxDim; d >= 1; d--) {
        const int64_t b = h.info.act_begin[d], end = h.info.act_end[d], window = end - b;
        if (window <= 0) continue;
        const int grid = int(std::min<int64_t>((window + 3) / 4, int64_t(shape.sms) * shape.light));
        reduce_light_launch(D, int32_t(b), int32_t(end), kCap1, ctr, d > 1 ? ctr + kStepCtr : nullptr, grid, s);
        reduce_heavy_launch(D, kCap2, 256, ctr,
                            int(std::min<int64_t>(int64_t(shape.sms) * std::min(shape.heavy, 2), window)), s);
        ctr += kStepCtr;
    }
    k_check_complex<<<unsigned(std::min<int64_t>((n + 255) / 256, 4096)), 256, 0, s>>>(n, D.pivot, D.state, D.err);
    // (the descriptors are not needed any more, and the essentials come later)
    uint64_t* ready = D.desc;
    cudaMemsetAsync(ready, 0, sizeof(uint64_t) * size_t(n), s);
    const int64_t room = kScratchInts - (kCtl + 3 * n) - nnz;  // k_reduce_noalloc's room for fill-in
    fill_account_launch(D, h.info.act_end[kMaxDim], room, ready, shape.sms, s);
    extract_pairs(D, 0, nullptr, s, false, D.err);  // nothing goes to the caller unless all is well
    k_store_npairs<<<1, 1, 0, s>>>(D.ctl, d_npairs);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    cudaMemcpyAsync(&h, D.ctl, offsetof(Ctl, step), cudaMemcpyDeviceToHost, s);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    if (h.err == 0) *ended = Ended::Done;
    else if (int64_t(h.fill) > room) *ended = Ended::Refused;
    return cudaSuccess;
}

int32_t fail(char* msg, int32_t cap, int32_t code, const char* text) {
    if (msg && cap > 0) {
        std::strncpy(msg, text, size_t(cap) - 1);
        msg[cap - 1] = '\0';
    }
    return code;
}

}  // namespace

extern "C" int32_t sspp_reduce_noalloc(int64_t ncols, int64_t nnz, const int32_t* d_dims, const int64_t* d_col_ptr,
                                       const int32_t* d_rows, int64_t* d_pairs, int64_t* d_npairs, void* stream,
                                       char* err_msg, int32_t err_cap) {
    if (ncols < 0 || nnz < 0 || !d_col_ptr || !d_npairs || (ncols > 0 && (!d_dims || !d_pairs)) || (nnz > 0 && !d_rows))
        return fail(err_msg, err_cap, SSPP_ERR_BAD_INPUT, "null pointer or negative size");
    if (ncols > kMaxCols)
        return fail(err_msg, err_cap, SSPP_ERR_BAD_INPUT, "too many columns for the allocation-free path (max 1048576)");
    if (kCtl + 3 * ncols + nnz + kFillReserve > kScratchInts)
        return fail(err_msg, err_cap, SSPP_ERR_BAD_INPUT,
                    "matrix too large for the allocation-free path: 3 * ncols + nnz must stay below 12582896");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return fail(err_msg, err_cap, SSPP_ERR_CUDA, "no current CUDA device");
    void* addr = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_setup_mu);
        if (!g_scratch_addr[dev]) {
            // once per device, with that device current
            cudaError_t e = cudaGetSymbolAddress(&g_scratch_addr[dev], g_scratch);
            if (e != cudaSuccess) {
                g_scratch_addr[dev] = nullptr;
                return fail(err_msg, err_cap, SSPP_ERR_CUDA, cudaGetErrorString(e));
            }
        }
        addr = g_scratch_addr[dev];
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Ended ended;
    cudaError_t e = reduce_in_scratch(static_cast<int32_t*>(addr), dev, ncols, nnz, d_dims, d_col_ptr, d_rows, d_pairs,
                                      d_npairs, s, &ended);
    if (e != cudaSuccess) return fail(err_msg, err_cap, SSPP_ERR_CUDA, cudaGetErrorString(e));
    const char* const kFillIn = "fill-in exceeded the 64 MiB allocation-free scratch array";
    if (ended == Ended::Done) return fail(err_msg, err_cap, SSPP_OK, "");
    if (ended == Ended::Refused) return fail(err_msg, err_cap, SSPP_ERR_CAPACITY, kFillIn);
    k_reduce_noalloc<<<1, kThreads, 0, s>>>(static_cast<int32_t*>(addr), ncols, nnz, d_dims, d_col_ptr, d_rows,
                                            d_pairs, d_npairs);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(err_msg, err_cap, SSPP_ERR_CUDA, cudaGetErrorString(e));
    int32_t err = 0;
    e = cudaMemcpyAsync(&err, addr, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(err_msg, err_cap, SSPP_ERR_CUDA, cudaGetErrorString(e));
    if (err & E_BAD_INPUT)
        return fail(err_msg, err_cap, SSPP_ERR_BAD_INPUT,
                    "malformed boundary matrix (col_ptr, face order, range or dimension)");
    if (err & E_CAPACITY)
        return fail(err_msg, err_cap, SSPP_ERR_CAPACITY, kFillIn);
    return fail(err_msg, err_cap, SSPP_OK, "");
}
