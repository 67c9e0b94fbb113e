// What the one-off passes over a matrix share (dg_plan.cu, dg_tiles.cu).
#pragma once
#include <algorithm>
#include <vector>
#include "dg_internal.h"

constexpr int kBands = 4096;          // column bands that chunks are ordered by

__device__ __forceinline__ int band_of(int32_t column, int32_t k) { return (int)((int64_t)column * kBands / k); }

// Blocks of the pool that go back to it at the end of the scope; the stream that used them is waited for first.
struct PoolScope {
    cudaStream_t stream;
    std::vector<void*> blocks;
    bool idle = false;                // the stream has been synchronised since the last use
    explicit PoolScope(cudaStream_t s) : stream(s) {}
    PoolScope(const PoolScope&) = delete;
    ~PoolScope()
    {
        if (!idle && !blocks.empty()) cudaStreamSynchronize(stream);
        for (void* p : blocks) dg_pool_free(p, true);
    }
    template <class X> int alloc(X** out, size_t count)
    {
        *out = nullptr;
        blocks.push_back(nullptr);    // first, so that no block is lost where the list cannot grow
        void* p = nullptr;
        const int rc = dg_pool_alloc(&p, std::max<size_t>(count, 1) * sizeof(X));
        if (rc == DG_OK) blocks.back() = p;
        else blocks.pop_back();
        *out = (X*)p;
        return rc;
    }
};
