// Internal declarations shared by the translation units of libdist_gnn_b200.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <mutex>
#include "dist_gnn_b200.h"

#define DG_CUDA(expr)                                        \
    do {                                                     \
        cudaError_t _e = (expr);                             \
        if (_e != cudaSuccess) return (int)_e;               \
    } while (0)

// Rows longer than the threshold are cut into chunks, one lane group each.  A group walks its entries a few dependent gathers
// at a time, so the longest row or chunk bounds a kernel's duration from below, and a small block has too few rows to hide it:
// 64 entries below 1 M, 128 beyond (F = 256, 150,001 nodes: 199 us against 221 with 64; 2.4 M nodes, F = 48: 2.28 ms against 2.52
// with 256), and 256 where rows are long on average (dense graph, F = 256: 5.6 ms against 6.3 with 128).
static inline int32_t dg_default_chunk(int64_t nnz, int32_t m) { return nnz < (1 << 20) ? 64 : nnz < 128 * (int64_t)m ? 128 : 256; }

// What dg_spmm_csr_static holds against its capacity are chunks of this many entries wherever the plan's own lengths are defaults.
#define DG_STATIC_CHUNK 256

// Nothing throws across the C ABI: entries that use the host's allocator, or call something that does, are function-try-blocks that
// end in this, with the code of the exception under way.
int dg_exception() noexcept;

#define DG_FINISH_TILES 16        // column tiles of one launch: arrival counts are kept per split row and tile

// One chunk of a split (heavy) row: entries [e0, e0 + len) of row `row`; its partial sum lands in scratch row `slot`.
struct dg_chunk {
    int64_t e0;
    int32_t len;
    int32_t row;
    int32_t slot;
    int32_t slot0, nchunks;       // the row's partial sums are scratch rows [slot0, slot0 + nchunks)
    int32_t heavy;                // which split row it is
};

// One row whose entries span more than one task of the streaming kernel: its partial sums sit in carry slots
// 2*t_first+1 (the piece that starts the row) and 2*t (t_first < t <= t_last, pieces that continue it).
struct dg_split_row {
    int32_t row;
    int32_t t_first;
    int32_t t_last;
    int32_t pad;
};

#define DG_DEFAULT_TASK_NNZ 1024

#define DG_STATUS_WORDS 4
#define DG_TILE_WORDS 2           // from here: whether the product under way may use its tiles (dg_tiles.h)
#define DG_LARGEST_ELEMENT 0
#define DG_GATHER_ALL 1

struct dg_tiles;      // dg_tiles.h

struct dg_plan {
    int device;
    int32_t m, k;
    int64_t nnz;
    int32_t heavy_threshold, chunk;
    int64_t* rowptr;          // device, m + 1
    const int32_t* col;       // device, borrowed
    dg_chunk* chunks;         // device, n_chunks
    int* arrived;             // device, n_heavy * DG_FINISH_TILES, zero between products
    int32_t n_chunks, n_heavy;
    int64_t heavy_nnz, max_row_nnz, touched_columns;
    int64_t static_chunks;    // chunks that count against the static entry's capacity
    float* scratch;           // device, grown on demand by dg_spmm_prepare
    int64_t scratch_floats;
    bool no_padded_copy;      // there was no memory for one
    // streaming kernel: the entry list cut into tasks of task_nnz entries, one warp each (0 until that family is first used)
    int32_t task_nnz, n_tasks, n_split;
    int32_t* task_first_row;  // device, n_tasks: the row that holds entry t * task_nnz
    dg_split_row* split;      // device, n_split rows that span tasks, ascending
    dg_tiles* tiles;          // tensor-core part of the split rows, or null
    int* status;              // device words: [0] set non-zero by a kernel that gave up on a bounded wait, [1] the last check
                              // (by number) that found other ids than the plan's, then the tiles' (DG_TILE_WORDS)
    int checks;               // checks issued so far
    std::mutex issue;         // held while a checked product is issued (dg_spmm_csr_checked)
};

int dg_stream_selected();     // non-zero while dg_select_kernel(2) is in force
int dg_spmm_stream_eligible(const dg_plan* plan, const float* B, int64_t ldb, const float* C, int64_t ldc, int32_t F);
int dg_spmm_stream_launch(const dg_plan* plan, const float* val, const float* B, int64_t ldb, float* C, int64_t ldc,
                          int32_t F, float alpha, float beta, uint32_t flags, const float* row_scale, const float* bias,
                          float* scratch, cudaStream_t stream, int* launches);

// Launches the product with an explicit scratch area (at least n_chunks x F floats; room for a padded copy of an odd-width
// operand behind it is used where it is there); shared by the plan-owned and the fixed-scratch entry points.
// `check` != 0: C stays as it is if that check has failed (row kernels only).  `split` false: no row is split, no scratch used.
int dg_spmm_launch(const dg_plan* plan, const float* val, const float* B, int64_t ldb, float* C, int64_t ldc,
                   int32_t F, float alpha, float beta, uint32_t flags, const float* row_scale, const float* bias,
                   float* scratch, int64_t scratch_floats, cudaStream_t stream, int check = 0);
int dg_spmm_launch_rows(const dg_plan* plan, const float* val, const float* B, int64_t ldb, float* C, int64_t ldc,
                        int32_t F, float alpha, float beta, uint32_t flags, const float* row_scale, const float* bias,
                        float* scratch, int64_t scratch_floats, cudaStream_t stream, int check = 0, bool split = true);
int dg_plan_build_lean(const int32_t* row, const int32_t* col, int64_t nnz, int32_t m, int32_t k, void* stream, dg_plan** out);
int dg_plan_ensure_tasks(dg_plan* plan, cudaStream_t stream);
// Device memory of plans (dg_pool.cu), on the current device.  A block may be freed once the device is done with it.
int dg_pool_alloc(void** out, size_t bytes);
int dg_device_alloc(void** out, size_t bytes);      // not from the pool, freed with cudaFree
void dg_pool_free(void* ptr, bool building = false) noexcept;      // building: a temporary of plan construction
int* dg_status_word();        // the current device's, or null
int dg_spmm_prepare(const dg_plan* plan, int32_t F, cudaStream_t stream);
int dg_check_spmm_args(const dg_plan* plan, const float* val, const float* B, int64_t ldb, const float* C, int64_t ldc,
                       int32_t F, uint32_t flags, const float* row_scale, const float* bias);
