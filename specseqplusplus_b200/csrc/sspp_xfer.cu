// Staged host <-> device transfers (see sspp_xfer.h).
#include "sspp_xfer.h"

#include <algorithm>
#include <cstring>

namespace sspp {

namespace {
constexpr size_t kHalfBytes = size_t(32) << 20;    // each half of the pinned buffer
constexpr size_t kDirectBytes = size_t(1) << 20;   // up to this, plain copies or one kernel's
constexpr size_t kDirectPieces = 8;                // more pieces than this are staged and move as one
constexpr size_t kMinTaskBytes = size_t(1) << 20;  // smallest share of one host thread

// Host-to-device copies of a few to a hundred megabytes go in chunks of 4 MB:
// the copy engine starts after the first one, and the staging memory stays in the
// caches.  A single chunk waits for the whole fill (20 MB: 2.2-2.6 ms; in 4 MB
// chunks 0.65 ms, in 2 MB 0.75 ms, in 8 MB 0.9-1.5 ms); larger copies have many
// chunks either way and lose to the per-chunk wake-ups (310 MB: 8.5-8.9 ms in 32 MB
// chunks, 10.2 ms in 4 MB).  Shares of 256 KB there; up to one chunk the wake-ups
// cost more than they bring (2.4 MB: 0.18 ms in shares of 1 MB, 0.32 ms in finer
// ones).
constexpr size_t kSmallChunk = size_t(4) << 20;
constexpr size_t kManyChunks = size_t(128) << 20;

// Up to 1 MB from pageable memory: a plain copy of each array costs the host 15-25 us
// and a wait, whatever its size.  The arrays are put into pinned memory one after
// another instead (each at a 16-byte boundary) and one kernel, which needs no waiting
// for, fetches them all over the link.  A 400-point Rips
// input's 210 KB in three arrays: the load takes 69 us with plain copies, 19 us like this.
struct Fetch {
    const uint8_t* src[kDirectPieces];
    uint8_t* dst[kDirectPieces];
    unsigned bytes[kDirectPieces];  // multiples of 4
    int n;
};

__global__ void __launch_bounds__(256) k_fetch(const __grid_constant__ Fetch f) {
    const unsigned first = blockIdx.x * 256 + threadIdx.x, step = gridDim.x * 256;
    for (int p = 0; p < f.n; p++) {
        const unsigned words = f.bytes[p] / 4;
        unsigned done = 0;
        if (reinterpret_cast<uintptr_t>(f.dst[p]) % 16 == 0) {
            const int4* s = reinterpret_cast<const int4*>(f.src[p]);
            int4* d = reinterpret_cast<int4*>(f.dst[p]);
            for (unsigned i = first; i < words / 4; i += step) d[i] = s[i];
            done = words & ~3u;
        }
        const int* s = reinterpret_cast<const int*>(f.src[p]);
        int* d = reinterpret_cast<int*>(f.dst[p]);
        for (unsigned i = done + first; i < words; i += step) d[i] = s[i];
    }
}
}  // namespace

HostPool::HostPool(int threads) {
    for (int i = 1; i < threads; i++) workers_.emplace_back([this] { loop(); });
}

HostPool::~HostPool() {
    {
        std::lock_guard<std::mutex> l(mu_);
        stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : workers_) t.join();
}

void HostPool::loop() {
    uint64_t seen = 0;
    for (;;) {
        std::unique_lock<std::mutex> l(mu_);
        cv_.wait(l, [&] { return stop_ || gen_ != seen; });
        if (stop_) return;
        seen = gen_;
        while (next_ < tasks_) {
            const int i = next_++;
            const std::function<void(int)>* f = fn_;
            l.unlock();
            (*f)(i);
            l.lock();
            if (--pending_ == 0) done_cv_.notify_all();
        }
    }
}

void HostPool::run(int tasks, const std::function<void(int)>& fn) {
    if (tasks <= 0) return;
    if (tasks == 1 || workers_.empty()) {
        for (int i = 0; i < tasks; i++) fn(i);
        return;
    }
    std::unique_lock<std::mutex> l(mu_);
    fn_ = &fn;
    tasks_ = tasks;
    next_ = 0;
    pending_ = tasks;
    gen_++;
    cv_.notify_all();
    while (next_ < tasks_) {
        const int i = next_++;
        l.unlock();
        fn(i);
        l.lock();
        --pending_;
    }
    done_cv_.wait(l, [&] { return pending_ == 0; });
    fn_ = nullptr;
}

Xfer::~Xfer() {
    if (small_) {
        if (small_used_) cudaEventSynchronize(small_ev_);
        cudaFreeHost(small_);
    }
    if (small_ev_) cudaEventDestroy(small_ev_);
    if (stage_) {
        for (int h = 0; h < 2; h++)
            if (used_[h]) cudaEventSynchronize(ev_[h]);
        cudaFreeHost(stage_);
    }
    for (auto e : ev_)
        if (e) cudaEventDestroy(e);
    delete pool_;
}

HostPool& Xfer::pool() {
    if (!pool_) {
        const unsigned hw = std::max(1u, std::min(std::thread::hardware_concurrency(), 16u));
        pool_ = new HostPool(threads_ > 0 ? std::min(threads_, int(hw)) : int(hw));
    }
    return *pool_;
}

cudaError_t Xfer::ensure() {
    if (stage_) return cudaSuccess;
    cudaError_t e = cudaMallocHost(&stage_, 2 * kHalfBytes);
    if (e != cudaSuccess) {
        stage_ = nullptr;
        return e;
    }
    half_ = kHalfBytes;
    for (int h = 0; h < 2; h++) {
        e = cudaEventCreateWithFlags(&ev_[h], cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void Xfer::parallel_copy(const std::vector<Piece>& pieces, const std::vector<Seg>& segs, size_t fill,
                         uint8_t* stage, bool to_stage, size_t least) {
    const int tasks = int(std::max<size_t>(1, std::min<size_t>(size_t(pool().size()), fill / least)));
    pool().run(tasks, [&](int t) {
        const size_t lo = fill * size_t(t) / size_t(tasks), hi = fill * size_t(t + 1) / size_t(tasks);
        for (const Seg& g : segs) {
            const size_t a = std::max(lo, g.so), b = std::min(hi, g.so + g.len);
            if (a >= b) continue;
            const Piece& p = pieces[g.piece];
            if (to_stage)
                std::memcpy(stage + a, static_cast<const uint8_t*>(p.src) + g.off + (a - g.so), b - a);
            else
                std::memcpy(static_cast<uint8_t*>(p.dst) + g.off + (a - g.so), stage + a, b - a);
        }
    });
}

// next chunk of at most `cap` bytes of the piece stream starting at (pi, po)
static size_t next_chunk(const std::vector<Piece>& pieces, size_t& pi, size_t& po, size_t cap,
                         std::vector<size_t>& out) {
    size_t fill = 0;
    while (pi < pieces.size() && fill < cap) {
        const size_t take = std::min(cap - fill, pieces[pi].bytes - po);
        if (take) {
            out.push_back(pi);
            out.push_back(po);
            out.push_back(take);
            out.push_back(fill);
        }
        fill += take;
        po += take;
        if (po == pieces[pi].bytes) {
            pi++;
            po = 0;
        }
    }
    return fill;
}

// host memory the copy engines can read directly (cudaMallocHost / registered)
static bool pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();  // unregistered pageable memory on some drivers
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// memory the host itself reads and writes, pinned or not
bool host_memory(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered || a.type == cudaMemoryTypeHost;
}

static bool all_pinned(const std::vector<Piece>& pieces, bool src) {
    for (const Piece& p : pieces)
        if (p.bytes && !pinned(src ? p.src : p.dst)) return false;
    return true;
}

cudaError_t Xfer::reserve_small() {
    if (small_) return cudaSuccess;
    cudaError_t e = cudaEventCreateWithFlags(&small_ev_, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
    e = cudaMallocHost(&small_, kDirectBytes + 16 * kDirectPieces);
    if (e != cudaSuccess) small_ = nullptr;
    return e;
}

// at most kDirectPieces pieces of at most kDirectBytes together, in whole words
cudaError_t Xfer::fetch_small(const std::vector<Piece>& pieces, cudaStream_t s) {
    cudaError_t e;
    if (small_used_ && (e = cudaEventSynchronize(small_ev_)) != cudaSuccess) return e;
    Fetch f{};
    size_t at = 0, most = 0;
    for (const Piece& p : pieces) {
        if (!p.bytes) continue;
        std::memcpy(small_ + at, p.src, p.bytes);
        f.src[f.n] = small_ + at;
        f.dst[f.n] = static_cast<uint8_t*>(p.dst);
        f.bytes[f.n++] = unsigned(p.bytes);
        at += (p.bytes + 15) & ~size_t(15);
        most = std::max(most, p.bytes);
    }
    k_fetch<<<unsigned(std::min<size_t>((most + 4095) / 4096, 256)), 256, 0, s>>>(f);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaEventRecord(small_ev_, s)) != cudaSuccess) return e;
    small_used_ = true;
    return cudaSuccess;
}

// The staged segments from `stage` to their places: one DMA per run that is contiguous
// on the device.
cudaError_t Xfer::send(const std::vector<Piece>& pieces, const std::vector<Seg>& segs, const uint8_t* stage,
                       cudaStream_t s) {
    for (size_t k = 0; k < segs.size();) {
        uint8_t* d0 = static_cast<uint8_t*>(pieces[segs[k].piece].dst) + segs[k].off;
        size_t len = segs[k].len, k2 = k + 1;
        const int grp = pieces[segs[k].piece].group;
        while (k2 < segs.size() && grp >= 0 && pieces[segs[k2].piece].group == grp &&
               static_cast<uint8_t*>(pieces[segs[k2].piece].dst) + segs[k2].off == d0 + len)
            len += segs[k2++].len;
        const cudaError_t e = cudaMemcpyAsync(d0, stage + segs[k].so, len, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
        k = k2;
    }
    return cudaSuccess;
}

// Many small pieces (a batch of small matrices), through the buffer of small copies: the
// large one, 64 MB of pinned memory, would cost a context's first batch 50 ms.
cudaError_t Xfer::send_small(const std::vector<Piece>& pieces, cudaStream_t s) {
    cudaError_t e;
    if (small_used_ && (e = cudaEventSynchronize(small_ev_)) != cudaSuccess) return e;
    std::vector<Seg> segs;
    size_t at = 0;
    for (size_t i = 0; i < pieces.size(); i++) {
        const Piece& p = pieces[i];
        if (!p.bytes) continue;
        std::memcpy(small_ + at, p.src, p.bytes);
        segs.push_back({i, 0, p.bytes, at});
        at += p.bytes;
    }
    if ((e = send(pieces, segs, small_, s)) != cudaSuccess) return e;
    if ((e = cudaEventRecord(small_ev_, s)) != cudaSuccess) return e;
    small_used_ = true;
    return cudaSuccess;
}

cudaError_t Xfer::h2d(const std::vector<Piece>& pieces, cudaStream_t s) {
    size_t total = 0;
    for (const Piece& p : pieces) total += p.bytes;
    if (total == 0) return cudaSuccess;
    cudaError_t e;
    if (small_ && total <= kDirectBytes && pieces.size() <= kDirectPieces && !all_pinned(pieces, true)) {
        bool ok = true;
        for (const Piece& p : pieces)
            ok = ok && (!p.bytes || ((reinterpret_cast<uintptr_t>(p.dst) | p.bytes) % 4 == 0 && host_memory(p.src)));
        if (ok) return fetch_small(pieces, s);
    }
    // small: plain copies, unless many; pinned sources: straight to the copy engine
    if ((total <= kDirectBytes && pieces.size() <= kDirectPieces) || all_pinned(pieces, true)) {
        for (const Piece& p : pieces)
            if (p.bytes && (e = cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyHostToDevice, s)) != cudaSuccess)
                return e;
        return cudaStreamSynchronize(s);  // pageable sources may be reused by the caller
    }
    if (small_ && total <= kDirectBytes) return send_small(pieces, s);
    if ((e = ensure()) != cudaSuccess) return e;
    const bool small = total > kSmallChunk && total <= kManyChunks;
    const size_t chunk = small ? kSmallChunk : half_;
    size_t pi = 0, po = 0;
    int h = 0;
    std::vector<size_t> raw;
    std::vector<Seg> segs;
    for (;;) {
        raw.clear();
        const size_t fill = next_chunk(pieces, pi, po, chunk, raw);
        if (fill == 0) break;
        segs.clear();
        for (size_t i = 0; i < raw.size(); i += 4) segs.push_back({raw[i], raw[i + 1], raw[i + 2], raw[i + 3]});
        if (used_[h] && (e = cudaEventSynchronize(ev_[h])) != cudaSuccess) return e;
        uint8_t* st = stage_ + size_t(h) * half_;
        parallel_copy(pieces, segs, fill, st, true, small ? kMinTaskBytes / 4 : kMinTaskBytes);
        if ((e = send(pieces, segs, st, s)) != cudaSuccess) return e;
        if ((e = cudaEventRecord(ev_[h], s)) != cudaSuccess) return e;
        used_[h] = true;
        h ^= 1;
    }
    return cudaSuccess;
}

cudaError_t Xfer::d2h(const std::vector<Piece>& pieces, cudaStream_t s) {
    size_t total = 0;
    for (const Piece& p : pieces) total += p.bytes;
    if (total == 0) return cudaSuccess;
    cudaError_t e;
    if (total <= kDirectBytes || all_pinned(pieces, false)) {
        for (const Piece& p : pieces)
            if (p.bytes && (e = cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
                return e;
        return cudaStreamSynchronize(s);
    }
    if ((e = ensure()) != cudaSuccess) return e;
    size_t pi = 0, po = 0;
    int h = 0;
    std::vector<size_t> raw;
    std::vector<Seg> cur, prev;
    size_t prev_fill = 0;
    int prev_h = -1;
    for (;;) {
        raw.clear();
        const size_t fill = next_chunk(pieces, pi, po, half_, raw);
        if (fill > 0) {
            cur.clear();
            for (size_t i = 0; i < raw.size(); i += 4) cur.push_back({raw[i], raw[i + 1], raw[i + 2], raw[i + 3]});
            if (used_[h] && (e = cudaEventSynchronize(ev_[h])) != cudaSuccess) return e;
            uint8_t* st = stage_ + size_t(h) * half_;
            for (size_t k = 0; k < cur.size();) {  // one DMA per run contiguous on the device
                const uint8_t* s0 = static_cast<const uint8_t*>(pieces[cur[k].piece].src) + cur[k].off;
                size_t len = cur[k].len, k2 = k + 1;
                const int grp = pieces[cur[k].piece].group;
                while (k2 < cur.size() && grp >= 0 && pieces[cur[k2].piece].group == grp &&
                       static_cast<const uint8_t*>(pieces[cur[k2].piece].src) + cur[k2].off == s0 + len)
                    len += cur[k2++].len;
                if ((e = cudaMemcpyAsync(st + cur[k].so, s0, len, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
                    return e;
                k = k2;
            }
            if ((e = cudaEventRecord(ev_[h], s)) != cudaSuccess) return e;
            used_[h] = true;
        }
        if (prev_h >= 0) {  // the previous chunk's bytes go out while this chunk's DMA runs
            if ((e = cudaEventSynchronize(ev_[prev_h])) != cudaSuccess) return e;
            parallel_copy(pieces, prev, prev_fill, stage_ + size_t(prev_h) * half_, false, kMinTaskBytes);
        }
        if (fill == 0) break;
        prev.swap(cur);
        prev_fill = fill;
        prev_h = h;
        h ^= 1;
    }
    return cudaSuccess;
}

}  // namespace sspp
