// Filtered flag complexes built on the device, written as boundary matrices.
//
// The reference takes its complexes from external tools (Dionysus / CGAL
// writers, phat-highclear/addons/rips.cpp and alpha_3.cpp) through PHAT files
// (src/main.cu:90-167).  Here the complex is built where it is reduced, so a
// request ships a point cloud or a scalar field (a few MB) instead of its
// boundary matrix (tens of MB for a 64^3 grid).
//
// Both builders produce a flag complex: the Rips complex is the clique complex
// of the graph of pairs at distance <= radius, and the Freudenthal (Kuhn)
// triangulation of a grid is the clique complex of its edge graph (vertices
// joined when their offset is a non-zero 0/1 vector; a clique is a chain in
// the componentwise order, which is a Kuhn simplex).  A simplex's value is the
// largest of its edges' values (Rips: float32 length; lower-star: the larger
// vertex value), vertices have value 0 (Rips) or the field value (lower-star).
//
// Several point clouds are built as one: their points lie one after another, so
// the graph is block-diagonal and every stage below runs once for all of them;
// only the cell grids (one per cloud) and the sort key (the cloud above the
// value) know the clouds.  64 clouds of 200-5,000 points (11.5 M columns): 34 ms one
// after another, where each build's 7 synchronisations and a few thousand threads
// left the GPU idle, 2.7 ms as one.
//
// Layout.  Vertices 0..V-1.  Edges are the concatenated upper adjacency lists
// (vertex i's neighbours j > i, ascending), so edge ids are in lexicographic
// order.  Triangles (i,j,k) are numbered edge (i,j) by edge, third vertex k
// ascending, found by merging the lists of i (after j) and j; tetrahedra
// (i,j,k,l) triangle by triangle, merging the triangles of edge (i,j) after k
// with the list of k.  Every list comes out in lexicographic order by
// construction, and every facet's id is known from the merge positions (one
// binary search in a short triangle segment for two of a tetrahedron's
// facets).  The global column order (value, dimension, tuple) is one stable
// radix sort of the 32-bit value keys over the concatenation (vertices, edges,
// triangles, tetrahedra), which is already in (dimension, tuple) order.
//
// Floating point is reproduced exactly: distances are summed in coordinate
// order with round-to-nearest and no contraction (__fadd_rn / __fmul_rn,
// __fsqrt_rn), maxima are of bitwise-canonical values (-0 is stored as +0 and
// NaN is rejected), so the matrix equals the host builder's bit for bit.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_segmented_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <initializer_list>
#include <vector>

#include "sspp_build.h"
#include "sspp_scan.cuh"

namespace sspp {
namespace {

constexpr int kT = 256;

unsigned grid_for(int64_t n, int64_t cap = 1 << 16) {
    int64_t g = (n + kT - 1) / kT;
    return unsigned(std::max<int64_t>(1, std::min(g, cap)));
}

#define GRID_STRIDE(i, n) \
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < (n); i += int64_t(gridDim.x) * blockDim.x)

__device__ __forceinline__ uint32_t fkey(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fval(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
// max with the host's std::max semantics; on canonical values any order gives the same bits
__device__ __forceinline__ float vmax(float a, float b) { return (a < b) ? b : a; }

template <class T>
cudaError_t take(BuildScratch& S, int slot, int64_t count, cudaStream_t s, T** out) {
    const size_t want = std::max<size_t>(sizeof(T) * size_t(std::max<int64_t>(count, 1)), 256);
    if (S.cap[slot] < want) {
        if (S.p[slot]) cudaFreeAsync(S.p[slot], s);
        S.p[slot] = nullptr;
        S.cap[slot] = 0;
        const size_t grown = want + want / 4;
        cudaError_t e = cudaMallocAsync(&S.p[slot], grown, s);
        if (e != cudaSuccess) {
            S.p[slot] = nullptr;
            return e;
        }
        S.cap[slot] = grown;
    }
    *out = static_cast<T*>(S.p[slot]);
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// vertex values: canonical copy (NaN rejected, -0 stored as +0)

__global__ void k_canon(const float* in, float* out, int64_t n, int* flag) {
    GRID_STRIDE(i, n) {
        float v = in[i];
        if (v != v) atomicOr(flag, 1);
        out[i] = (v == 0.0f) ? 0.0f : v;
    }
}

// ---------------------------------------------------------------------------
// Freudenthal grid: upper adjacency

struct Grid {
    int64_t gx, gy, gz;
};

__device__ __forceinline__ int ls_degree(Grid g, int64_t v) {
    const int64_t x = v % g.gx, y = (v / g.gx) % g.gy, z = v / (g.gx * g.gy);
    const int bits = int(x + 1 < g.gx) + int(y + 1 < g.gy) + int(z + 1 < g.gz);
    return (1 << bits) - 1;
}

struct GridDegree {
    Grid g;
    __device__ int64_t operator()(int64_t v) const { return ls_degree(g, v); }
};

__global__ void k_ls_fill(Grid g, const float* val, const int64_t* up_off, int32_t* up_v, float* up_w,
                          int32_t* e_src) {
    const int64_t nv = g.gx * g.gy * g.gz;
    GRID_STRIDE(v, nv) {
        const int64_t x = v % g.gx, y = (v / g.gx) % g.gy, z = v / (g.gx * g.gy);
        int32_t nb[7];
        int m = 0;
        for (int a = 1; a < 8; a++) {
            const int64_t x1 = x + (a & 1), y1 = y + ((a >> 1) & 1), z1 = z + ((a >> 2) & 1);
            if (x1 >= g.gx || y1 >= g.gy || z1 >= g.gz) continue;
            const int32_t u = int32_t((z1 * g.gy + y1) * g.gx + x1);
            int q = m++;
            while (q > 0 && nb[q - 1] > u) {  // ascending (the offsets already grow with the mask)
                nb[q] = nb[q - 1];
                q--;
            }
            nb[q] = u;
        }
        const int64_t o = up_off[v];
        const float fv = val[v];
        for (int q = 0; q < m; q++) {
            up_v[o + q] = nb[q];
            up_w[o + q] = vmax(fv, val[nb[q]]);
            e_src[o + q] = int32_t(v);
        }
    }
}

// ---------------------------------------------------------------------------
// Rips: cell grids, points by cell, neighbour search

// A cloud on the device: what the host knows, then its cell grid.  A grid has at
// most 4 * npts + kCellSlack cells (larger cells than the radius asks for when the
// radius is tiny), numbered from cell0 with x fastest.
struct CloudD {
    int64_t p0, f0, cell0;  // first point, first float of its coordinates, first cell
    int32_t npts, D, maxdim;
    float radius;
    double lo[3];
    double side;
    int32_t n[3];
    // Radii below kTinyRadius: squares of such distances underflow, so points much further
    // apart than the radius may have a distance that is not.  Edges are those between
    // points of neighbouring cells of this grid, the host builder's.
    double fine_side;
    int32_t fine_n[3];
    // while the bounding box is found (k_cloud_grid)
    uint32_t key_lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, key_hi[3] = {0, 0, 0};
    int32_t bad = 0, arrived = 0;
};
constexpr int kCellSlack = 64;
constexpr float kTinyRadius = 1e-19f;
constexpr int kBoxPoints = 2048, kBoxBlocks = 512;  // points a block at least, blocks a cloud at most
__host__ __device__ inline int box_blocks(int64_t npts) {
    const int64_t b = (npts + kBoxPoints - 1) / kBoxPoints;
    return int(b < 1 ? 1 : b > kBoxBlocks ? kBoxBlocks : b);
}

__device__ __forceinline__ int32_t cell_coord(double lo, double side, int32_t n, float x) {
    const double t = floor((double(x) - lo) / side);
    const int32_t k = int32_t(t);
    return k < 0 ? 0 : (k >= n ? n - 1 : k);
}
__device__ __forceinline__ int32_t cell_coord(const CloudD& c, int d, float x) {
    return cell_coord(c.lo[d], c.side, c.n[d], x);
}
__device__ __forceinline__ bool fine_neighbours(const CloudD& c, int d, float x, float y) {
    return abs(cell_coord(c.lo[d], c.fine_side, c.fine_n[d], x) - cell_coord(c.lo[d], c.fine_side, c.fine_n[d], y)) <= 1;
}

// Cloud blockIdx.x's bounding box (also rejects non-finite coordinates), by box_blocks of
// its size, and, by the last of them, its cell grid.  Cells of side > radius: a margin
// of 2^-10 covers the rounding of the float distance and of the cell coordinate; at most
// ~1000 per axis.  (One block whatever the size made loads of 300,000 and 1 M points
// 1,146 and 4,307 us where they take 780 and 1,930 now.)
__global__ void __launch_bounds__(kT) k_cloud_grid(const float* p, CloudD* clouds, int* flag) {
    __shared__ uint32_t s_lo[3], s_hi[3];
    __shared__ int s_bad;
    CloudD& c = clouds[blockIdx.x];
    const int blocks = box_blocks(c.npts);
    if (int(blockIdx.y) >= blocks) return;
    if (c.maxdim == 0) {  // points alone: nobody is looked for, and any coordinate will do
        if (blockIdx.y == 0 && threadIdx.x == 0) {
            for (int d = 0; d < 3; d++) {
                c.lo[d] = 0.0;
                c.n[d] = 1;
            }
            c.side = 1.0;
        }
        return;
    }
    if (threadIdx.x < 3) {
        s_lo[threadIdx.x] = 0xFFFFFFFFu;
        s_hi[threadIdx.x] = 0;
    }
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    const int D = c.D;
    uint32_t lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi[3] = {0, 0, 0};
    bool bad = false;
    for (int i = blockIdx.y * kT + threadIdx.x; i < c.npts; i += blocks * kT) {
        for (int d = 0; d < D; d++) {
            const float x = p[c.f0 + int64_t(i) * D + d];
            if (!isfinite(x)) bad = true;
            const uint32_t k = fkey(x);
            lo[d] = min(lo[d], k);
            hi[d] = max(hi[d], k);
        }
    }
    for (int d = 0; d < D; d++) {
        lo[d] = __reduce_min_sync(0xFFFFFFFFu, lo[d]);
        hi[d] = __reduce_max_sync(0xFFFFFFFFu, hi[d]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&s_lo[d], lo[d]);
            atomicMax(&s_hi[d], hi[d]);
        }
    }
    if (bad) s_bad = 1;
    __syncthreads();
    if (threadIdx.x < 3 && blocks > 1) {
        atomicMin(&c.key_lo[threadIdx.x], s_lo[threadIdx.x]);
        atomicMax(&c.key_hi[threadIdx.x], s_hi[threadIdx.x]);
        if (threadIdx.x == 0 && s_bad) atomicOr(&c.bad, 1);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x) return;
    if (blocks > 1) {
        __threadfence();
        if (atomicAdd(&c.arrived, 1) != blocks - 1) return;
        __threadfence();
        for (int d = 0; d < 3; d++) {
            s_lo[d] = __ldcg(&c.key_lo[d]);
            s_hi[d] = __ldcg(&c.key_hi[d]);
        }
        s_bad = __ldcg(&c.bad);
    }
    if (s_bad) atomicOr(flag, 1);
    double ext[3] = {0, 0, 0}, ext_max = 0.0;
    for (int d = 0; d < 3; d++) c.lo[d] = 0.0;
    if (c.npts > 0 && !s_bad) {
        for (int d = 0; d < D; d++) {
            c.lo[d] = double(fval(s_lo[d]));
            ext[d] = double(fval(s_hi[d])) - c.lo[d];
            ext_max = fmax(ext_max, ext[d]);
        }
    }
    double side = fmax(fmax(double(c.radius) * (1.0 + 1.0 / 1024.0), ext_max / 1000.0), 1e-30);
    c.fine_side = side;
    for (int d = 0; d < 3; d++) c.fine_n[d] = d < D ? int32_t(fmin(1001.0, floor(ext[d] / side) + 1.0)) : 1;
    for (;; side *= 1.25) {
        int64_t total = 1;
        for (int d = 0; d < 3; d++) {
            c.n[d] = d < D ? int32_t(fmin(1001.0, floor(ext[d] / side) + 1.0)) : 1;
            total *= c.n[d];
        }
        if (total <= 4 * int64_t(c.npts) + kCellSlack) break;  // reached: one cell once side > ext_max
    }
    c.side = side;
}

// the cloud of point i
__device__ __forceinline__ int cloud_of(const CloudD* clouds, int k, int64_t i) {
    int a = 0, b = k;  // largest a with p0 <= i (an empty cloud shares its p0 with the next one)
    while (b - a > 1) {
        const int m = (a + b) >> 1;
        if (clouds[m].p0 <= i) a = m;
        else b = m;
    }
    return a;
}

// each point's cell and its place in it
__global__ void k_cells(const float* p, int64_t n, const CloudD* clouds, int k, int32_t* count, uint32_t* pcell,
                        int32_t* pslot) {
    GRID_STRIDE(i, n) {
        const CloudD& c = clouds[cloud_of(clouds, k, i)];
        const float* x = p + c.f0 + (i - c.p0) * c.D;
        int64_t id = 0;
        for (int d = c.D - 1; d >= 0; d--) id = id * c.n[d] + cell_coord(c, d, x[d]);
        id += c.cell0;
        pcell[i] = uint32_t(id);
        pslot[i] = atomicAdd(count + id, 1);
    }
}

// points in cell order: coordinates (0 beyond D) and the point's index
__global__ void k_sort_points(const float* p, int64_t n, const CloudD* clouds, int k, const int64_t* start,
                              const uint32_t* pcell, const int32_t* pslot, float4* spt) {
    GRID_STRIDE(i, n) {
        const CloudD& c = clouds[cloud_of(clouds, k, i)];
        const float* x = p + c.f0 + (i - c.p0) * c.D;
        spt[start[pcell[i]] + pslot[i]] = make_float4(x[0], c.D > 1 ? x[1] : 0.0f, c.D > 2 ? x[2] : 0.0f,
                                                      __int_as_float(int32_t(i)));
    }
}

// One warp per point, points in cell order (neighbouring warps read the same
// cells).  The up to nine rows of three cells around a point are ranges of the
// sorted points: lanes 0-8 read their bounds together, then all lanes test the
// candidates.  FILL = false counts the point's upper neighbours into count[i]
// and the largest count into *most; FILL = true writes them from up_off[i]:
// ascending (sorted by the warp, up to kNbrSort of them) or, with `raw`, as
// found.  One thread per point, searching the sorted cells, took 111 us for the
// two passes over 5,000 points in the plane, a warp with direct cell starts 16 us.
constexpr int kNbrWarps = 8;
constexpr int kNbrSort = 256;

template <bool FILL>
__global__ void __launch_bounds__(kNbrWarps * 32) k_nbrs(int64_t n, const CloudD* clouds, int k, const int64_t* start,
                                                         const float4* spt, const int64_t* up_off, int32_t* count, int32_t* up_v,
                                                         float* up_w, int32_t* e_src, bool raw, int* most) {
    __shared__ uint64_t s_buf[FILL ? kNbrWarps : 1][kNbrSort];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t* buf = s_buf[FILL ? w : 0];
    int top = 0;
    for (int64_t m = int64_t(blockIdx.x) * kNbrWarps + w; m < n; m += int64_t(gridDim.x) * kNbrWarps) {
        const float4 pi = spt[m];
        const int32_t i = __float_as_int(pi.w);
        const CloudD& c = clouds[cloud_of(clouds, k, i)];
        const int D = c.D;
        const float radius = c.radius;
        int64_t b = 0, e = 0;
        if (lane < 9 && c.maxdim > 0) {  // row lane: y offset lane % 3 - 1, z offset lane / 3 - 1
            const int cx = cell_coord(c, 0, pi.x);
            const int y = D > 1 ? cell_coord(c, 1, pi.y) + lane % 3 - 1 : lane % 3;
            const int z = D > 2 ? cell_coord(c, 2, pi.z) + lane / 3 - 1 : lane / 3;
            if (y >= 0 && y < c.n[1] && z >= 0 && z < c.n[2]) {
                const int64_t row = c.cell0 + (int64_t(z) * c.n[1] + y) * c.n[0];
                b = start[row + max(cx - 1, 0)];
                e = start[row + min(cx + 1, c.n[0] - 1) + 1];
            }
        }
        int cnt = 0;
        const int64_t base = FILL ? up_off[i] : 0;
        for (unsigned rows = __ballot_sync(0xFFFFFFFFu, e > b); rows; rows &= rows - 1) {
            const int r = __ffs(rows) - 1;
            const int64_t rb = __shfl_sync(0xFFFFFFFFu, b, r), re = __shfl_sync(0xFFFFFFFFu, e, r);
            for (int64_t q0 = rb; q0 < re; q0 += 32) {
                bool hit = false;
                int32_t j = 0;
                float dist = 0.0f;
                if (q0 + lane < re) {
                    const float4 pj = spt[q0 + lane];
                    j = __float_as_int(pj.w);
                    if (j > i) {
                        float t = __fsub_rn(pi.x, pj.x);
                        float s = __fadd_rn(0.0f, __fmul_rn(t, t));
                        if (D > 1) {
                            t = __fsub_rn(pi.y, pj.y);
                            s = __fadd_rn(s, __fmul_rn(t, t));
                        }
                        if (D > 2) {
                            t = __fsub_rn(pi.z, pj.z);
                            s = __fadd_rn(s, __fmul_rn(t, t));
                        }
                        dist = __fsqrt_rn(s);
                        hit = dist <= radius;
                        if (hit && radius < kTinyRadius)
                            hit = fine_neighbours(c, 0, pi.x, pj.x) && (D < 2 || fine_neighbours(c, 1, pi.y, pj.y)) &&
                                  (D < 3 || fine_neighbours(c, 2, pi.z, pj.z));
                    }
                }
                const unsigned hm = __ballot_sync(0xFFFFFFFFu, hit);
                if (FILL && hit) {
                    const int at = cnt + __popc(hm & ((1u << lane) - 1));
                    if (raw) {
                        up_v[base + at] = j;
                        up_w[base + at] = dist;
                    } else if (at < kNbrSort) {
                        buf[at] = (uint64_t(uint32_t(j)) << 32) | __float_as_uint(dist);
                    }
                }
                cnt += __popc(hm);
            }
        }
        if (!FILL) {
            if (lane == 0) count[i] = cnt;
            top = max(top, cnt);
            continue;
        }
        for (int q = lane; q < cnt; q += 32) e_src[base + q] = i;
        if (raw) continue;
        __syncwarp();
        if (cnt <= 32) {
            uint64_t x = lane < cnt ? buf[lane] : ~0ull;
#pragma unroll
            for (int a = 2; a <= 32; a <<= 1) {
#pragma unroll
                for (int h = a >> 1; h > 0; h >>= 1) {
                    const uint64_t y = __shfl_xor_sync(0xFFFFFFFFu, x, h);
                    const bool keep_min = ((lane & h) == 0) == ((lane & a) == 0);
                    x = (y < x) == keep_min ? y : x;
                }
            }
            if (lane < cnt) {
                up_v[base + lane] = int32_t(x >> 32);
                up_w[base + lane] = __uint_as_float(uint32_t(x));
            }
        } else {
            int p2 = 64;
            while (p2 < cnt) p2 <<= 1;
            for (int q = cnt + lane; q < p2; q += 32) buf[q] = ~0ull;
            __syncwarp();
            for (int a = 2; a <= p2; a <<= 1) {
                for (int h = a >> 1; h > 0; h >>= 1) {
                    for (int q = lane; q < p2; q += 32) {
                        const int l = q ^ h;
                        if (l > q) {
                            const uint64_t x = buf[q], y = buf[l];
                            if ((x > y) == ((q & a) == 0)) {
                                buf[q] = y;
                                buf[l] = x;
                            }
                        }
                    }
                    __syncwarp();
                }
            }
            for (int q = lane; q < cnt; q += 32) {
                up_v[base + q] = int32_t(buf[q] >> 32);
                up_w[base + q] = __uint_as_float(uint32_t(buf[q]));
            }
        }
        __syncwarp();  // the warp's buffer is rewritten for its next point
    }
    if (!FILL && lane == 0 && top > 0) atomicMax(most, top);
}

// ---------------------------------------------------------------------------
// cliques

// The clouds of a build whose maximal dimensions differ (null: all the same).
struct DimLimit {
    const CloudD* clouds;
    int k;
    __device__ __forceinline__ bool below(int32_t vertex, int dim) const {
        return clouds && clouds[cloud_of(clouds, k, vertex)].maxdim < dim;
    }
};

// triangles (i, j, k), k > j, over edge e = (i, j)
template <bool FILL>
__global__ void k_tri(int64_t E, const int64_t* up_off, const int32_t* up_v, const float* up_w, const int32_t* e_src,
                      DimLimit lim, const int64_t* tri_off, int32_t* count, int32_t* tri_k, int4* tri_f, float* tri_w) {
    GRID_STRIDE(e, E) {
        const int32_t i = e_src[e], j = up_v[e];
        int64_t a = e + 1, b = up_off[j];
        const int64_t ae = lim.below(i, 2) ? a : up_off[i + 1], be = up_off[j + 1];
        int32_t cnt = 0;
        const int64_t base = FILL ? tri_off[e] : 0;
        const float we = FILL ? up_w[e] : 0.0f;
        while (a < ae && b < be) {
            const int32_t va = up_v[a], vb = up_v[b];
            if (va < vb) {
                a++;
            } else if (va > vb) {
                b++;
            } else {
                if (FILL) {
                    const int64_t t = base + cnt;
                    tri_k[t] = va;
                    tri_f[t] = make_int4(int32_t(e), int32_t(a), int32_t(b), 0);
                    tri_w[t] = vmax(vmax(we, up_w[a]), up_w[b]);
                }
                cnt++;
                a++;
                b++;
            }
        }
        if (!FILL) count[e] = cnt;
    }
}

// the triangle of edge e whose third vertex is l (it exists: every clique's faces do)
__device__ __forceinline__ int32_t tri_of(const int64_t* tri_off, const int32_t* tri_k, int32_t e, int32_t l) {
    int64_t lo = tri_off[e], hi = tri_off[e + 1];
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (tri_k[mid] < l) lo = mid + 1;
        else hi = mid;
    }
    return int32_t(lo);
}

// tetrahedra (i, j, k, l), l > k, over triangle t = (i, j, k)
template <bool FILL>
__global__ void k_tet(int64_t T, const int64_t* up_off, const int32_t* up_v, const float* up_w, const int64_t* tri_off,
                      const int32_t* tri_k, const int4* tri_f, const float* tri_w, const int32_t* e_src, DimLimit lim,
                      const int64_t* tet_off, int32_t* count, int4* tet_f, float* tet_w) {
    GRID_STRIDE(t, T) {
        const int4 f = tri_f[t];
        const int32_t k = tri_k[t];
        int64_t a = t + 1, b = up_off[k];
        const int64_t ae = lim.clouds && lim.below(e_src[f.x], 3) ? a : tri_off[f.x + 1], be = up_off[k + 1];
        int32_t cnt = 0;
        const int64_t base = FILL ? tet_off[t] : 0;
        const float wt = FILL ? tri_w[t] : 0.0f;
        while (a < ae && b < be) {
            const int32_t va = tri_k[a], vb = up_v[b];
            if (va < vb) {
                a++;
            } else if (va > vb) {
                b++;
            } else {
                if (FILL) {
                    const int64_t q = base + cnt;
                    tet_f[q] = make_int4(int32_t(t), int32_t(a), tri_of(tri_off, tri_k, f.y, va),
                                         tri_of(tri_off, tri_k, f.z, va));
                    tet_w[q] = vmax(vmax(wt, tri_w[a]), up_w[b]);
                }
                cnt++;
                a++;
                b++;
            }
        }
        if (!FILL) count[t] = cnt;
    }
}

// ---------------------------------------------------------------------------
// global order and the matrix

struct Sizes {
    int64_t V, E, T, Q;
};

__device__ __forceinline__ int dim_of(const Sizes& z, int64_t c) {
    return c < z.V ? 0 : (c < z.V + z.E ? 1 : (c < z.V + z.E + z.T ? 2 : 3));
}

// The sort key of a column: its value, and above it the cloud's number when
// there are several (K = uint64_t).
template <class K>
__global__ void k_keys(Sizes z, const float* vval, const float* up_w, const float* tri_w, const float* tet_w,
                       const int64_t* cut, int k, K* key, int32_t* idx) {
    const int64_t N = z.V + z.E + z.T + z.Q;
    GRID_STRIDE(c, N) {
        float v;
        int64_t x = c;
        int d = 0;
        if (c < z.V) {
            v = vval ? vval[c] : 0.0f;
        } else if (c < z.V + z.E) {
            v = up_w[x = c - z.V];
            d = 1;
        } else if (c < z.V + z.E + z.T) {
            v = tri_w[x = c - z.V - z.E];
            d = 2;
        } else {
            v = tet_w[x = c - z.V - z.E - z.T];
            d = 3;
        }
        K key_c = fkey(v);
        if constexpr (sizeof(K) == 8) {  // the cloud: the simplices of one dimension lie cloud after cloud
            const int64_t* first = cut + int64_t(d) * (k + 1);
            int a = 0, b = k;
            while (b - a > 1) {
                const int m = (a + b) >> 1;
                if (first[m] <= x) a = m;
                else b = m;
            }
            key_c |= K(a) << 32;
        }
        key[c] = key_c;
        idx[c] = int32_t(c);
    }
}

// Each cloud's first vertex, edge, triangle and tetrahedron (cut, four rows of
// k + 1) and its first column in the sorted order (starts).
__global__ void k_cuts(const CloudD* clouds, int k, Sizes z, const int64_t* up_off, const int64_t* tri_off,
                       const int64_t* tet_off, int64_t* cut, int64_t* starts) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= k; c += gridDim.x * blockDim.x) {
        const int64_t v = c < k ? clouds[c].p0 : z.V;
        const int64_t e = z.E ? up_off[v] : 0;
        const int64_t t = tri_off ? tri_off[e] : 0;
        const int64_t q = tet_off ? tet_off[t] : 0;
        cut[c] = v;
        cut[k + 1 + c] = e;
        cut[2 * (k + 1) + c] = t;
        cut[3 * (k + 1) + c] = q;
        starts[c] = v + e + t + q;
    }
}

template <class K>
__global__ void k_place(int64_t N, Sizes z, const K* key, const int32_t* perm, int32_t* rank, int32_t* dims,
                        float* values) {
    GRID_STRIDE(g, N) {
        const int32_t c = perm[g];
        rank[c] = int32_t(g);
        dims[g] = dim_of(z, c);
        values[g] = fval(uint32_t(key[g]));
    }
}

struct ColLen {
    const int32_t* dims;
    __device__ int64_t operator()(int64_t g) const { return dims[g] == 0 ? 0 : dims[g] + 1; }
};

// Exclusive prefix from `first` into off[i]; the total into off[n].
struct OffSink {
    int64_t* off;
    int64_t n;
    int64_t first = 0;
    __device__ void operator()(int64_t i, int64_t pre, int64_t v) const {
        off[i] = first + pre;
        if (i == n - 1) off[n] = first + pre + v;
    }
};

struct ReadI32 {
    const int32_t* a;
    __device__ int64_t operator()(int64_t i) const { return a[i]; }
};

__global__ void k_rows(int64_t N, Sizes z, const int32_t* perm, const int32_t* rank, const int32_t* e_src,
                       const int32_t* up_v, const int4* tri_f, const int4* tet_f, const int64_t* col_ptr, int64_t ent0,
                       int32_t col0, int32_t* rows) {
    GRID_STRIDE(g, N) {
        const int64_t c = perm[g];
        int32_t r[4];
        int k;
        if (c < z.V) {
            continue;
        } else if (c < z.V + z.E) {
            const int64_t e = c - z.V;
            r[0] = rank[e_src[e]];
            r[1] = rank[up_v[e]];
            k = 2;
        } else if (c < z.V + z.E + z.T) {
            const int4 f = tri_f[c - z.V - z.E];
            r[0] = rank[z.V + f.x];
            r[1] = rank[z.V + f.y];
            r[2] = rank[z.V + f.z];
            k = 3;
        } else {
            const int4 f = tet_f[c - z.V - z.E - z.T];
            const int64_t o = z.V + z.E;
            r[0] = rank[o + f.x];
            r[1] = rank[o + f.y];
            r[2] = rank[o + f.z];
            r[3] = rank[o + f.w];
            k = 4;
        }
        for (int a = 1; a < k; a++) {
            const int32_t x = r[a];
            int b = a;
            while (b > 0 && r[b - 1] > x) {
                r[b] = r[b - 1];
                b--;
            }
            r[b] = x;
        }
        const int64_t o = col_ptr[g] - ent0;
        for (int a = 0; a < k; a++) rows[o + a] = r[a] + col0;
    }
}

#define BK(call)                                                       \
    do {                                                               \
        cudaError_t e_ = (call);                                       \
        if (e_ != cudaSuccess) {                                       \
            *err = std::string(#call) + ": " + cudaGetErrorString(e_); \
            return BUILD_CUDA;                                         \
        }                                                              \
    } while (0)

int fail(std::string* err, const std::string& msg) {
    *err = msg;
    return BUILD_BAD_INPUT;
}

// Reads up to 8 int64 values from device memory (one synchronisation).
int read_back(BuildScratch& S, std::initializer_list<const int64_t*> src, int64_t* dst, cudaStream_t s,
              std::string* err) {
    int q = 0;
    for (const int64_t* p : src) BK(cudaMemcpyAsync(S.h_misc + q++, p, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    BK(cudaStreamSynchronize(s));
    std::memcpy(dst, S.h_misc, sizeof(int64_t) * size_t(q));
    return 0;
}

// Counts of n items, until scan_counts has read them (the ranks come later).
int take_counts(BuildScratch& S, int64_t n, cudaStream_t s, int32_t** count, std::string* err) {
    BK(take(S, BuildScratch::RANK, n, s, count));
    return 0;
}

// off[0..n) = exclusive scan of count[0..n), off[n] = total.
int scan_counts(BuildScratch& S, const int32_t* count, int64_t* off, int64_t n, cudaStream_t s, std::string* err) {
    if (n == 0) {
        BK(cudaMemsetAsync(off, 0, sizeof(int64_t), s));
        return 0;
    }
    int64_t* blk;
    BK(take(S, BuildScratch::BLK, scan_most_blocks(n) + 2, s, &blk));
    scan(ReadI32{count}, OffSink{off, n}, n, blk, s);
    BK(cudaGetLastError());
    return 0;
}

constexpr int64_t kMaxCols = int64_t(1) << 31;

// Several clouds are built as one up to this many columns (about 80 bytes of
// scratch each); beyond it the caller takes fewer at a time.
#ifndef SSPP_MAX_JOINT_COLS
#define SSPP_MAX_JOINT_COLS (int64_t(1) << 26)
#endif
constexpr int64_t kMaxJointCols = SSPP_MAX_JOINT_COLS;

// The clouds of a build (one, or a grid: k = 1 and no table).
struct Clouds {
    const CloudD* d = nullptr;
    int k = 1;
    bool mixed = false;         // their maximal dimensions differ
    int64_t* starts = nullptr;  // host, k + 1
};

template <class K>
int sort_columns(BuildScratch& S, const Sizes& z, const float* vval, const float* up_w, const float* tri_w,
                 const float* tet_w, const int64_t* cut, int k, int end_bit, cudaStream_t s, int32_t* dims,
                 float* values, int32_t* rank, const int32_t** perm, std::string* err) {
    const int64_t N = z.V + z.E + z.T + z.Q;
    K *key_a, *key_b;
    int32_t *idx_a, *idx_b;
    BK(take(S, BuildScratch::KEY_A, N, s, &key_a));
    BK(take(S, BuildScratch::KEY_B, N, s, &key_b));
    BK(take(S, BuildScratch::IDX_A, N, s, &idx_a));
    BK(take(S, BuildScratch::IDX_B, N, s, &idx_b));
    k_keys<K><<<grid_for(N), kT, 0, s>>>(z, vval, up_w, tri_w, tet_w, cut, k, key_a, idx_a);
    cub::DoubleBuffer<K> dk(key_a, key_b);
    cub::DoubleBuffer<int32_t> dv(idx_a, idx_b);
    size_t tmp_bytes = 0;
    BK(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, dk, dv, int(N), 0, end_bit, s));
    char* tmp;
    BK(take(S, BuildScratch::TMP, int64_t(tmp_bytes), s, &tmp));
    BK(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, dk, dv, int(N), 0, end_bit, s));
    *perm = dv.Current();
    k_place<K><<<grid_for(N), kT, 0, s>>>(N, z, dk.Current(), *perm, rank, dims, values);
    return 0;
}

// Cliques of the graph in S (UP_OFF / UP_V / UP_W / E_SRC over nv vertices, E
// edges), the global order and the matrix.
int build_flag(BuildScratch& S, int64_t nv, int64_t E, const float* vval, int maxdim, const Clouds& cl, cudaStream_t s,
               const Sink& sink, Built* out, std::string* err) {
    const int64_t* up_off = static_cast<const int64_t*>(S.p[BuildScratch::UP_OFF]);
    const int32_t* up_v = static_cast<const int32_t*>(S.p[BuildScratch::UP_V]);
    const float* up_w = static_cast<const float*>(S.p[BuildScratch::UP_W]);
    const int32_t* e_src = static_cast<const int32_t*>(S.p[BuildScratch::E_SRC]);
    Sizes z{nv, E, 0, 0};
    auto check_size = [&](int64_t cols) {
        if (cl.k > 1 && cols > kMaxJointCols) return int(BUILD_SPLIT);
        return cols >= kMaxCols ? fail(err, "complex too large (columns >= 2^31)") : 0;
    };
    if (int rc = check_size(z.V + z.E)) return rc;
    const DimLimit lim{cl.mixed ? cl.d : nullptr, cl.k};
    int64_t *tri_off = nullptr, *tet_off = nullptr;
    int32_t* tri_k = nullptr;
    int4* tri_f = nullptr;
    float* tri_w = nullptr;
    int4* tet_f = nullptr;
    float* tet_w = nullptr;
    int32_t* count = nullptr;
    if (maxdim >= 2 && z.E > 0) {
        BK(take(S, BuildScratch::TRI_OFF, z.E + 1, s, &tri_off));
        if (take_counts(S, z.E, s, &count, err)) return BUILD_CUDA;
        k_tri<false><<<grid_for(z.E), kT, 0, s>>>(z.E, up_off, up_v, up_w, e_src, lim, nullptr, count, nullptr, nullptr,
                                                  nullptr);
        if (scan_counts(S, count, tri_off, z.E, s, err)) return BUILD_CUDA;
        if (read_back(S, {tri_off + z.E}, &z.T, s, err)) return BUILD_CUDA;
        if (int rc = check_size(z.V + z.E + z.T)) return rc;
        BK(take(S, BuildScratch::TRI_K, z.T, s, &tri_k));
        BK(take(S, BuildScratch::TRI_F, z.T, s, &tri_f));
        BK(take(S, BuildScratch::TRI_W, z.T, s, &tri_w));
        k_tri<true><<<grid_for(z.E), kT, 0, s>>>(z.E, up_off, up_v, up_w, e_src, lim, tri_off, nullptr, tri_k, tri_f,
                                                 tri_w);
        if (maxdim >= 3 && z.T > 0) {
            BK(take(S, BuildScratch::TET_OFF, z.T + 1, s, &tet_off));
            if (take_counts(S, z.T, s, &count, err)) return BUILD_CUDA;
            k_tet<false><<<grid_for(z.T), kT, 0, s>>>(z.T, up_off, up_v, up_w, tri_off, tri_k, tri_f, tri_w, e_src, lim,
                                                      nullptr, count, nullptr, nullptr);
            if (scan_counts(S, count, tet_off, z.T, s, err)) return BUILD_CUDA;
            if (read_back(S, {tet_off + z.T}, &z.Q, s, err)) return BUILD_CUDA;
            if (int rc = check_size(z.V + z.E + z.T + z.Q)) return rc;
            BK(take(S, BuildScratch::TET_F, z.Q, s, &tet_f));
            BK(take(S, BuildScratch::TET_W, z.Q, s, &tet_w));
            k_tet<true><<<grid_for(z.T), kT, 0, s>>>(z.T, up_off, up_v, up_w, tri_off, tri_k, tri_f, tri_w, e_src, lim,
                                                     tet_off, nullptr, tet_f, tet_w);
        }
    }
    const int64_t N = z.V + z.E + z.T + z.Q;
    const int64_t nnz = 2 * z.E + 3 * z.T + 4 * z.Q;
    int64_t* cut = nullptr;
    if (cl.k > 1) {
        BK(take(S, BuildScratch::STARTS, 5 * (int64_t(cl.k) + 1), s, &cut));
        int64_t* d_starts = cut + 4 * (int64_t(cl.k) + 1);
        k_cuts<<<grid_for(cl.k + 1), kT, 0, s>>>(cl.d, cl.k, z, up_off, tri_off, tet_off, cut, d_starts);
        BK(cudaMemcpyAsync(cl.starts, d_starts, sizeof(int64_t) * (size_t(cl.k) + 1), cudaMemcpyDeviceToHost, s));
    } else if (cl.starts) {
        cl.starts[0] = 0;
        cl.starts[1] = N;
    }
    Built b;
    BK(sink.reserve(N, nnz, &b));
    if (N > 0) {
        int32_t* rank;
        const int32_t* perm = nullptr;
        BK(take(S, BuildScratch::RANK, N, s, &rank));
        int end_bit = 32;
        while (cl.k > (int64_t(1) << (end_bit - 32))) end_bit++;
        const int rc = cl.k > 1 ? sort_columns<uint64_t>(S, z, vval, up_w, tri_w, tet_w, cut, cl.k, end_bit, s, b.dims,
                                                         b.values, rank, &perm, err)
                                : sort_columns<uint32_t>(S, z, vval, up_w, tri_w, tet_w, nullptr, 1, 32, s, b.dims,
                                                         b.values, rank, &perm, err);
        if (rc) return rc;
        int64_t* blk;
        BK(take(S, BuildScratch::BLK, scan_most_blocks(N) + 2, s, &blk));
        scan(ColLen{b.dims}, OffSink{b.col_ptr, N, sink.ent0}, N, blk, s);
        if (nnz > 0)
            k_rows<<<grid_for(N), kT, 0, s>>>(N, z, perm, rank, e_src, up_v, tri_f, tet_f, b.col_ptr, sink.ent0,
                                              int32_t(sink.col0), b.rows);
    } else if (sink.ent0 == 0) {
        BK(cudaMemsetAsync(b.col_ptr, 0, sizeof(int64_t), s));
    }
    BK(cudaGetLastError());
    b.ncols = N;
    b.nnz = nnz;
    *out = b;
    return 0;
}

}  // namespace

Sink scratch_sink(BuildScratch& S, cudaStream_t s) {
    Sink k;
    k.reserve = [&S, s](int64_t ncols, int64_t nnz, Built* b) -> cudaError_t {
        cudaError_t e = take(S, BuildScratch::DIMS, ncols + 1, s, &b->dims);
        if (e == cudaSuccess) e = take(S, BuildScratch::COLPTR, ncols + 1, s, &b->col_ptr);
        if (e == cudaSuccess) e = take(S, BuildScratch::ROWS, nnz, s, &b->rows);
        if (e == cudaSuccess) e = take(S, BuildScratch::VALUES, ncols, s, &b->values);
        return e;
    };
    return k;
}

int build_lowerstar(BuildScratch& S, const float* d_values, int64_t gx, int64_t gy, int64_t gz, int maxdim,
                    cudaStream_t s, const Sink& sink, Built* out, std::string* err) {
    if (gx < 1 || gy < 1 || gz < 1 || maxdim < 0 || maxdim > 3) return fail(err, "bad grid size or maxdim");
    if (gx > kMaxCols || gy > kMaxCols || gz > kMaxCols || gx * gy > kMaxCols || gx * gy * gz >= kMaxCols / 8)
        return fail(err, "grid too large (vertices >= 2^28)");
    const int64_t nv = gx * gy * gz;
    if (!S.h_misc) BK(cudaMallocHost(&S.h_misc, 8 * sizeof(int64_t)));
    int* flag;
    float* vval;
    int64_t* up_off;
    BK(take(S, BuildScratch::MISC, 8, s, &flag));
    BK(cudaMemsetAsync(flag, 0, sizeof(int64_t), s));
    BK(take(S, BuildScratch::VVAL, nv, s, &vval));
    k_canon<<<grid_for(nv), kT, 0, s>>>(d_values, vval, nv, flag);
    BK(take(S, BuildScratch::UP_OFF, nv + 1, s, &up_off));
    int64_t* blk;
    BK(take(S, BuildScratch::BLK, scan_most_blocks(nv) + 2, s, &blk));
    const Grid g{gx, gy, gz};
    scan(GridDegree{g}, OffSink{up_off, nv}, nv, blk, s);
    int64_t got[2];
    if (read_back(S, {up_off + nv, reinterpret_cast<int64_t*>(flag)}, got, s, err)) return BUILD_CUDA;
    if (got[1]) return fail(err, "NaN vertex value");
    // the upper adjacency holds every edge; a matrix of vertices alone leaves them out
    const int64_t E = got[0];
    int32_t *up_v, *e_src;
    float* up_w;
    BK(take(S, BuildScratch::UP_V, E, s, &up_v));
    BK(take(S, BuildScratch::UP_W, E, s, &up_w));
    BK(take(S, BuildScratch::E_SRC, E, s, &e_src));
    k_ls_fill<<<grid_for(nv), kT, 0, s>>>(g, vval, up_off, up_v, up_w, e_src);
    BK(cudaGetLastError());
    return build_flag(S, nv, maxdim >= 1 ? E : 0, vval, maxdim, Clouds{}, s, sink, out, err);
}

int build_clouds(BuildScratch& S, const float* d_points, const Cloud* clouds, int k, cudaStream_t s, const Sink& sink,
                 int64_t* starts, Built* out, std::string* err) {
    std::vector<CloudD> h;
    h.reserve(size_t(k));
    int64_t n = 0, f = 0, most = 0;
    int maxdim = 0;
    bool mixed = false;
    for (int c = 0; c < k; c++) {
        const Cloud& q = clouds[c];
        if (q.npts < 0 || q.space_dim < 1 || q.space_dim > 3 || q.maxdim < 0 || q.maxdim > 3 || !(q.radius >= 0.0f) ||
            !std::isfinite(q.radius))
            return fail(err, "bad point count, space dimension, radius or maxdim");
        if (q.npts >= kMaxCols / 8) return fail(err, "too many points (>= 2^28)");
        if (k > 1 && n + q.npts >= kMaxCols / 8) return BUILD_SPLIT;
        CloudD d{};
        d.p0 = n;
        d.f0 = f;
        d.cell0 = 4 * n + int64_t(kCellSlack) * c;
        d.npts = int32_t(q.npts);
        d.D = q.space_dim;
        d.maxdim = q.maxdim;
        d.radius = q.radius;
        h.push_back(d);
        n += q.npts;
        most = std::max(most, q.npts);
        f += q.npts * q.space_dim;
        mixed = mixed || (c > 0 && q.maxdim != clouds[0].maxdim);
        maxdim = std::max(maxdim, int(q.maxdim));
    }
    if (!S.h_misc) BK(cudaMallocHost(&S.h_misc, 8 * sizeof(int64_t)));
    Clouds cl;
    cl.k = k;
    cl.mixed = mixed;
    cl.starts = starts;
    if (maxdim == 0 && k == 1) {  // points alone: no graph (and any coordinate will do)
        return build_flag(S, n, 0, nullptr, 0, cl, s, sink, out, err);
    }
    const int64_t cells = 4 * n + int64_t(kCellSlack) * k;
    int* flag;      // [0] non-finite coordinate, [2] largest upper degree
    CloudD* dc;
    int64_t *up_off, *start;
    uint32_t* pcell;
    int32_t *pslot, *count;
    float4* spt;
    BK(take(S, BuildScratch::MISC, 8, s, &flag));
    BK(take(S, BuildScratch::CLOUDS, k, s, &dc));
    BK(take(S, BuildScratch::UP_OFF, n + 1, s, &up_off));
    BK(take(S, BuildScratch::CELL, cells + 1, s, &start));
    BK(take(S, BuildScratch::PCELL, n, s, &pcell));
    BK(take(S, BuildScratch::PSLOT, n, s, &pslot));
    BK(take(S, BuildScratch::SPT, n, s, &spt));
    BK(take(S, BuildScratch::RANK, cells, s, &count));  // counts per cell; the ranks come later
    BK(cudaMemsetAsync(flag, 0, 4 * sizeof(int), s));
    BK(cudaMemcpyAsync(dc, h.data(), sizeof(CloudD) * h.size(), cudaMemcpyHostToDevice, s));
    BK(cudaMemsetAsync(count, 0, sizeof(int32_t) * size_t(cells), s));
    k_cloud_grid<<<dim3(unsigned(k), unsigned(box_blocks(most))), kT, 0, s>>>(d_points, dc, flag);
    int64_t got[3] = {0, 0, 0};
    const unsigned ng = unsigned(std::max<int64_t>(1, std::min<int64_t>((n + kNbrWarps - 1) / kNbrWarps, 1 << 16)));
    if (n > 0) {
        k_cells<<<grid_for(n), kT, 0, s>>>(d_points, n, dc, k, count, pcell, pslot);
        int64_t* blk;
        BK(take(S, BuildScratch::BLK, scan_most_blocks(std::max(cells, n)) + 2, s, &blk));
        scan(ReadI32{count}, OffSink{start, cells}, cells, blk, s);
        k_sort_points<<<grid_for(n), kT, 0, s>>>(d_points, n, dc, k, start, pcell, pslot, spt);
        // (there are at least four cells per point: the cells' counts have been scanned)
        k_nbrs<false><<<ng, kNbrWarps * 32, 0, s>>>(n, dc, k, start, spt, nullptr, count, nullptr, nullptr, nullptr,
                                                    false, flag + 2);
    }
    if (scan_counts(S, count, up_off, n, s, err)) return BUILD_CUDA;
    if (read_back(S, {up_off + n, reinterpret_cast<int64_t*>(flag), reinterpret_cast<int64_t*>(flag + 2)}, got, s, err))
        return BUILD_CUDA;
    if (got[1]) return fail(err, "non-finite point coordinate");
    const int64_t E = got[0];
    if (k > 1 && n + E > kMaxJointCols) return BUILD_SPLIT;
    if (n + E >= kMaxCols) return fail(err, "complex too large (columns >= 2^31)");
    int32_t *up_v, *e_src;
    float* up_w;
    BK(take(S, BuildScratch::UP_V, E, s, &up_v));
    BK(take(S, BuildScratch::UP_W, E, s, &up_w));
    BK(take(S, BuildScratch::E_SRC, E, s, &e_src));
    if (E > 0) {
        // each vertex's upper neighbours ascending: sorted by the warp that finds
        // them, or, where a vertex has more than fit its buffer, all by a segmented sort
        const bool raw = got[2] > kNbrSort;
        int32_t* v = up_v;
        float* w = up_w;
        if (raw) {
            BK(take(S, BuildScratch::UP_V2, E, s, &v));
            BK(take(S, BuildScratch::UP_W2, E, s, &w));
        }
        k_nbrs<true><<<ng, kNbrWarps * 32, 0, s>>>(n, dc, k, start, spt, up_off, nullptr, v, w, e_src, raw,
                                                   nullptr);
        if (raw) {
            size_t sb = 0;
            BK(cub::DeviceSegmentedSort::StableSortPairs(nullptr, sb, v, up_v, w, up_w, int(E), int(n), up_off,
                                                         up_off + 1, s));
            char* tmp;
            BK(take(S, BuildScratch::TMP, int64_t(sb), s, &tmp));
            BK(cub::DeviceSegmentedSort::StableSortPairs(tmp, sb, v, up_v, w, up_w, int(E), int(n), up_off, up_off + 1,
                                                         s));
        }
    }
    BK(cudaGetLastError());
    cl.d = dc;
    return build_flag(S, n, E, nullptr, maxdim, cl, s, sink, out, err);
}

cudaError_t build_stage(BuildScratch& S, size_t bytes, cudaStream_t s, void** out) {
    char* p;
    cudaError_t e = take(S, BuildScratch::IN, int64_t(bytes), s, &p);
    *out = p;
    return e;
}

void build_free(BuildScratch& S) {
    for (int q = 0; q < BuildScratch::NUM; q++) {
        if (S.p[q]) cudaFree(S.p[q]);
        S.p[q] = nullptr;
        S.cap[q] = 0;
    }
    if (S.h_misc) cudaFreeHost(S.h_misc);
    S.h_misc = nullptr;
}

}  // namespace sspp
