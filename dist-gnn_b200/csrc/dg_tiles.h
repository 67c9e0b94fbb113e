// Dense tiles of a sparse block (dg_tiles.cu): the part of a plan's entries that the tensor cores multiply.
//
// A dense tile multiplies its zeros too, and values and operand are cut into bf16 pieces.  Both are right for numbers of a size
// whose products neither overflow nor vanish; an infinity, a NaN or a number beyond kTileBound would reach rows that have no entry
// there, or turn an infinity into NaN, and numbers that are all below kTileLeast lose bits.  So values like that get no tiles,
// and an operand like that has its whole product gathered: k_tile_columns, which reads every element the tiles use, leaves the
// largest in the plan's word DG_LARGEST_ELEMENT; where that does not fit, k_tile_mma sets DG_GATHER_ALL, which k_tile_columns
// cleared, and does nothing else; k_spmm reads DG_GATHER_ALL and clears the other.  Each word is written by one kernel of the
// three and read by a later one, so that captured graphs can be replayed.
//
// The tiles hold copies of the values.  k_tile_mma compares the values of every product with what they were then, and sets
// DG_GATHER_ALL where they differ: a product never uses others than those in front of it.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "dg_internal.h"

struct dg_slab {            // one non-empty 128 x 32 tile
    int32_t col_tile;       // which 32 of the frequent columns
    int32_t first, count;   // its entries: records [first, first + count)
};
struct dg_segment {         // consecutive slabs of one row tile that one CTA multiplies into one partial result
    int32_t slab0, slab1, slot, pad;
};

struct dg_tiles {
    const float* val;             // where the values lay that the records were made from: products with others do not use the tiles
    void* value_sums;             // what they were: sums, a record per checking warp
    float least_operand;          // an operand without any element of this size is too small for the tiles
    int64_t entries;              // entries in tiles
    int32_t n_slabs, n_segments, n_columns, col_tiles, ctas;
    uint2* records;               // [entries] three bf16 pieces of the value and the position in the tile
    dg_slab* slabs;
    dg_segment* segments;
    int32_t* cta_segment;         // [ctas + 1] first segment of every CTA
    int32_t* columns;             // [n_columns] ids of the frequent columns
    int2* parts;                  // per split row: {slot * 128 + row in the tile, number of partial results}
    // what is left of the split rows
    int32_t* rest_col;
    float* rest_val;
    dg_chunk* rest_chunks;
    int32_t n_rest_chunks;
    int* status;                  // the device's word of kernels that gave up (dg_status_word)
};

// Scratch floats that a product of width F takes for the tiles (0: the tiles are not used at this width).
int64_t dg_tiles_scratch_floats(const dg_plan* plan, int32_t F);
// Launches the tensor-core part: partial results of the tiled rows land at `area`, 16-byte pieces of 128 rows side by side.
int dg_tiles_launch(const dg_plan* plan, const float* B, int64_t ldb, int32_t F, float* area, cudaStream_t stream, int* launches, int wait_limit);
void dg_tiles_free(dg_tiles* t);      // the device is done with it
