// Host-side launchers of the engine's device passes.
#pragma once
#include <cuda_runtime.h>

#include "sspp_internal.h"

namespace sspp {

void fill_i32(int32_t* p, int32_t v, int64_t n, cudaStream_t s);
void fill_i64(int64_t* p, int64_t v, int64_t n, cudaStream_t s);

// input (filtration order) -> dimension-sorted padded arena layout; writes
// D.newidx, D.perm, D.dim, D.desc, D.diminfo->col_begin/col_end and
// D.arena_top (the arena ints used).
// Each launcher returns the number of kernels it launched.
int64_t part_tiles(int64_t n);            // tiles of the validation and the reorder (D.dimcnt: kNumDims each)
int validate(Device& D, cudaStream_t s);  // sets ERRB_BAD_INPUT; the passes after it leave when it is set
// k complexes copied side by side (cstart/estart: k+1 column / entry starts on
// the device): shifts each one's face indices and col_ptr entries; *d_bad = 1
// when a face index lies outside its own complex
int batch_rebase(int64_t n, int64_t nnz, int32_t k, const int64_t* d_cstart, const int64_t* d_estart,
                 int64_t* colptr, int32_t* rows, int* d_bad, cudaStream_t s);
// lows: also the lowest rows and leftmost columns (the first init pass)
// write_desc: also the descriptors of short columns, which init_compress writes
// otherwise (needed when anything reads them before it)
int reorder(Device& D, bool lows, bool write_desc, cudaStream_t s);

// per-complex slice starts (k+1 each) of the sorted pairs and essentials
int batch_bounds(int32_t k, const int64_t* d_cstart, int64_t npairs, const int64_t* pairs, int64_t ness,
                 const int64_t* ess, int64_t* d_pstart, int64_t* d_estart, cudaStream_t s);
// pairs / essentials with each complex's first column subtracted
int batch_localize(int64_t npairs, int64_t ness, int32_t k, const int64_t* d_cstart, const int64_t* pairs,
                   const int64_t* ess, int64_t* lpairs, int64_t* less, cudaStream_t s);

// lows_done: the reorder computed the lowest rows and leftmost columns
int init_passes(Device& D, bool lows_done, cudaStream_t s);
// keep_rows: leave negative rows in the columns (whole reduced columns, for
// representative cycles); otherwise they are removed.
// final (no dualization follows at once): also the inline apparent columns, the
// per-dimension row bounds and the counts of active columns
int init_compress(Device& D, const uint8_t* dropped, bool keep_rows, bool final, cudaStream_t s);
// (the row bounds and the counts of active columns were gathered with the states)
int active_list(Device& D, cudaStream_t s);
// anti-transpose of the compressed matrix behind the primal columns in the
// arena; remaps pivots, states, dims, inline columns, row bounds and the
// per-dimension column ranges.
// mode 1: the whole matrix; mode 2: after the edge columns were reduced (the
// 0-dimensional pairs are final, the vertices' dual columns are skipped).  The
// first part reads no edge column in mode 2, so their reduction may still run.
int dualize_begin(Device& D, int mode, cudaStream_t s);
int dualize_end(Device& D, int mode, cudaStream_t s);
// the control block up to its step counters and, as far as they fit, the pairs and
// essentials into host memory that the device can write
int push_results(const Device& D, Ctl* h_ctl, int64_t* h_pairs, int64_t max_pairs, int64_t* h_ess, int64_t max_ess,
                 cudaStream_t s);
// dimension 1 of the boundary matrix (active list entries [beg, end), no column of
// more than two entries) over the vertices, the reordered rows [0, rows)
int reduce_edges(Device& D, int32_t beg, int32_t end, int32_t rows, cudaStream_t s);
// marks (always for a dual): by marking both columns of every pair, instead of by the
// columns' states.  unless (neither dual nor marks): a device word; when it is set, nothing
// is written
int extract_pairs(Device& D, int dual, const uint8_t* dropped, cudaStream_t s, bool marks = false,
                  const int* unless = nullptr);

// Device work queue of (complex, block) items (one persistent launch per
// schedule; see k_reduce_queue).  An item is one spectral-sequence block of
// one complex in one dimension: the slice of the active list it adds to the
// window and the band's lowest row.
struct QItem {
    int32_t cplx;
    int32_t nbeg, nend;  // active-list entries that enter the window with this block
    int32_t minrow;      // the band's lowest row (INT32_MIN: the dimension's completion sweep)
    int32_t flags;       // QF_* below
    int32_t pad[3];
};
enum : int32_t {
    QF_LAST_OF_DIM = 1,  // the complex's next item (if any) is of its next dimension
    QF_HALF = 2,         // this item reads the parked columns from the second half of its complex's list
};

struct QueueArgs {
    const QItem* items;
    int32_t nitems, ncplx;
    int* taken;            // [nitems] entries handed out
    int* done;             // [nitems] entries finished
    int* lin;              // [nitems + 1] parked columns each item starts with (written by its predecessor)
    int* cur;              // [ncplx] current item of each complex; -1 once the complex is finished
    int* gate;             // [ncplx] 1: the complex's block sequence waits for its CTA-tier columns
    int* hpend;            // [ncplx] CTA-tier columns of the complex not finished yet
    const int32_t* item_end;   // [ncplx] one past the complex's last item
    const int64_t* list_off;   // [ncplx] the complex's parked-column list (two halves)
    const int32_t* list_cap;   // [ncplx] entries per half
    int2* lists;           // (column, lowest row)
    int32_t* pool;         // deferred columns for the CTA tier (-1 until written)
    int32_t* pool_c;       // their complexes
    int32_t pool_cap;
    int* pool_head;        // next slot the CTA tier takes
    int* pool_tail;        // next slot written
    int* finished;         // complexes finished
    int* abort;            // set on any failure: every block leaves
    int32_t heavy_ctas;    // blocks [0, heavy_ctas) reduce CTA-tier columns; the others run warps
    int32_t gate_left;     // a complex's next dimension starts once at most this many of its CTA-tier columns are left
    int32_t chunk;         // entries a warp takes at a time
    int32_t cap1;          // warp buffers (ints)
    long long spin_limit;  // idle polls before a block gives up (SSPP_ERR_TIMEOUT)
};

// per complex: active columns and band bounds of each dimension, from the
// state after the init passes (out: [k][kNumDims] each)
int queue_complex_info(const Device& D, int32_t k, const int64_t* d_cstart, int32_t* act_cnt, int32_t* min_row,
                       int32_t* max_row, cudaStream_t s);
// blocks per SM of the queue kernel with these capacities (0: it does not fit)
cudaError_t queue_configure(int cap1, int cap2, int threads, int* blocks_per_sm);
// cooperative launch of the queue kernel on `grid` blocks
cudaError_t reduce_queue_launch(const Device& D, int cap1, int cap2, int threads, const QueueArgs& Q, int grid,
                                cudaStream_t s);

cudaError_t reduce_configure(int cap1, int cap2, int heavy_threads, int* light_blocks_per_sm,
                             int* heavy_blocks_per_sm);
// One dimension's light tier: warps reduce the columns active[beg, end) that are
// still active.  ctr: the step's counters; the launch's last block also marks the
// step's CTA-tier pool slice (ctr[2], and ctr_next[1] of the next step when given).
void reduce_light_launch(const Device& D, int32_t beg, int32_t end, int cap, int* ctr, int* ctr_next, int grid,
                         cudaStream_t s);
// After a reduction with whole columns and no error: the ints that the additions of a
// column-after-column reduction read, `listed` active columns, added up into ctl->fill;
// sets ERRB_CAPACITY when they exceed `room`, or when it cannot tell.  ready: [n], zeroed.
void fill_account_launch(const Device& D, int32_t listed, int64_t room, uint64_t* ready, int sms, cudaStream_t s);
void reduce_heavy_launch(const Device& D, int cap, int threads, int* ctr, int grid, cudaStream_t s);

}  // namespace sspp
