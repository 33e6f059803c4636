// Device builders of filtered flag complexes (Vietoris-Rips of a point cloud,
// lower-star filtration of the Freudenthal triangulation of a 3-D grid) that
// write the boundary matrix straight into device memory, in the column order
// of the reference's input files: (filtration value, dimension, lexicographic
// vertex tuple).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <string>

namespace sspp {

// Stream-ordered device buffers, grown on demand and reused across builds.
struct BuildScratch {
    enum {
        UP_OFF, UP_V, UP_W, UP_V2, UP_W2, E_SRC,      // upper adjacency (edges in lexicographic order)
        TRI_OFF, TRI_K, TRI_F, TRI_W,                 // triangles: third vertex, facet edges, value
        TET_OFF, TET_F, TET_W,                        // tetrahedra: facet triangles, value
        VVAL, IN, CLOUDS, STARTS,                     // vertex values, copied input, clouds and their starts
        CELL, PCELL, PSLOT, SPT,                      // Rips cells: starts, points' cells and places, sorted points
        KEY_A, KEY_B, IDX_A, IDX_B, RANK,             // global order
        DIMS, COLPTR, ROWS, VALUES,                   // the boundary matrix
        BLK, MISC, TMP, NUM
    };
    void* p[NUM] = {};
    size_t cap[NUM] = {};
    int64_t* h_misc = nullptr;  // pinned, 8 entries
};

struct Built {
    int64_t ncols = 0, nnz = 0;
    int32_t* dims = nullptr;
    int64_t* col_ptr = nullptr;
    int32_t* rows = nullptr;
    float* values = nullptr;
};

// One point cloud of a build.
struct Cloud {
    int64_t npts;
    int32_t space_dim;  // 1..3
    int32_t maxdim;     // 0..3
    float radius;
};

// Where the matrix goes: called once its size is known; fills dims (ncols),
// col_ptr (ncols + 1), rows (nnz) and values (ncols).  Column indices in rows
// start at col0 and col_ptr at ent0, so that a matrix can be written behind
// another one (col_ptr[0] is then the earlier one's last entry).
struct Sink {
    std::function<cudaError_t(int64_t ncols, int64_t nnz, Built* out)> reserve;
    int64_t col0 = 0, ent0 = 0;
};

// Status of a build besides 0: bad input (non-finite coordinate, size limit), a
// CUDA error, or several clouds that together need more scratch than one build
// takes (the caller builds them in smaller groups); a message in *err.
enum { BUILD_BAD_INPUT = -1, BUILD_CUDA = -2, BUILD_SPLIT = -3 };

// The Vietoris-Rips complexes of k clouds, one after another in one matrix
// (block-diagonal, each in its own column order), all stages run once for all of
// them.  points: device array, cloud after cloud, each npts x space_dim row-major.
// starts (host, k + 1): each cloud's first column, relative to col0.
int build_clouds(BuildScratch& S, const float* d_points, const Cloud* clouds, int k, cudaStream_t s, const Sink& sink,
                 int64_t* starts, Built* out, std::string* err);

// values: device array gx*gy*gz, x fastest.  All simplices of the Freudenthal
// triangulation up to maxdim (<= 3).
int build_lowerstar(BuildScratch& S, const float* d_values, int64_t gx, int64_t gy, int64_t gz, int maxdim,
                    cudaStream_t s, const Sink& sink, Built* out, std::string* err);

// A sink that writes to the scratch's own buffers.
Sink scratch_sink(BuildScratch& S, cudaStream_t s);

// Device buffer of at least `bytes` for a copy of the caller's input (the IN slot).
cudaError_t build_stage(BuildScratch& S, size_t bytes, cudaStream_t s, void** out);

void build_free(BuildScratch& S);

}  // namespace sspp
