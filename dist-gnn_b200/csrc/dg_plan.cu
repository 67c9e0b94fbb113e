// Plan construction: row-sorted COO -> CSR row offsets, index validation, split-row chunk table, column census.
//
// Replaces the per-call descriptor set-up of the reference's cuSPARSE wrapper (light_dist_gnn/spmm_cpp/spmm.cpp:19-24)
// and the coo2csr conversion of its CUDA-10 variant (spmm_original.cpp:140-146) by a one-off device pass.
//
// Everything is built on the device and the host waits once, for a handful of counts.  What bounds it is one pass over the
// ids (16 bytes an entry from a loader's int64 block, 8 from int32 arrays); tables are allocated at their upper bounds
// out of the pool.  Built in steps with the tables sorted on the host it took two copies each way and five waits: plan and
// first product of a 300,007-row block with 15.3 M entries 8.3 ms (30 ms when the allocator was slow), now 0.8 ms.
#include <algorithm>
#include <new>
#include <vector>
#include "dg_build.h"
#include "dg_tiles.h"

namespace {

constexpr int T = 256;
constexpr int kEntriesPerThread = 2;         // 15.3 M entries: 74 us; with 4 82, with 8 130, with 1 93 (waiting for the columns' bitmap)

struct PlanCounts {
    unsigned long long max_row, heavy_nnz, touched, static_chunks;
    int32_t n_heavy, n_chunks;
    int bad;
    int pad;
};

// One pass over the ids: checks every entry, fills the row offsets of the rows that start between an entry and the one
// before it, narrows 64-bit column ids to `col32`, and marks the columns in a bitmap (null: no census).  Entry nnz stands for
// the end of the matrix.
template <class Id>
__global__ void __launch_bounds__(T) k_ingest(const Id* __restrict__ row, const Id* __restrict__ col, int64_t nnz, int32_t m, int32_t k,
                                              int32_t* __restrict__ col32, int64_t* __restrict__ rowptr, uint32_t* __restrict__ bitmap,
                                              PlanCounts* __restrict__ counts)
{
    const int64_t base = (int64_t)blockIdx.x * (T * kEntriesPerThread) + threadIdx.x;
    const int lane = threadIdx.x & 31;
    Id cur[kEntriesPerThread], c[kEntriesPerThread], prev0[kEntriesPerThread];
#pragma unroll
    for (int i = 0; i < kEntriesPerThread; ++i) {
        const int64_t e = base + (int64_t)i * T;
        cur[i] = e < nnz ? __ldcs(row + e) : (Id)m;
        c[i] = e < nnz ? __ldcs(col + e) : (Id)0;
        prev0[i] = lane == 0 && e > 0 && e <= nnz ? row[e - 1] : (Id)-1;
    }
    bool bad = false;
#pragma unroll
    for (int i = 0; i < kEntriesPerThread; ++i) {
        const int64_t e = base + (int64_t)i * T;
        const Id before = __shfl_up_sync(0xffffffffu, cur[i], 1);
        const Id prev = lane == 0 ? prev0[i] : before;
        if (e > nnz) continue;
        bool ok = prev >= -1 && prev < m && cur[i] >= 0 && cur[i] <= m && prev <= cur[i];
        if (e < nnz) ok = ok && cur[i] < m && c[i] >= 0 && c[i] < k;
        if (!ok) {
            bad = true;
            continue;
        }
        for (int32_t r = (int32_t)prev + 1; r <= (int32_t)cur[i]; ++r) rowptr[r] = e;
        if (e < nnz) {
            const int32_t cc = (int32_t)c[i];
            if (col32) col32[e] = cc;
            if (bitmap) {
                const uint32_t bit = 1u << (cc & 31);
                if (!(bitmap[cc >> 5] & bit)) atomicOr(&bitmap[cc >> 5], bit);
            }
        }
    }
    if (bad) atomicExch(&counts->bad, 1);
}

__device__ __forceinline__ int2 block_scan(int2 v, int2* warp_sums)      // inclusive; warp_sums: T / 32 + 1 entries, last = total
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int2 s = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, s.x, off), y = __shfl_up_sync(0xffffffffu, s.y, off);
        if (lane >= off) { s.x += x; s.y += y; }
    }
    if (lane == 31) warp_sums[warp] = s;
    __syncthreads();
    int2 add = make_int2(0, 0), all = make_int2(0, 0);
    const int warps = blockDim.x >> 5;
    for (int w = 0; w < warps; ++w) {
        const int2 x = warp_sums[w];
        if (w < warp) { add.x += x.x; add.y += x.y; }
        all.x += x.x; all.y += x.y;
    }
    if (threadIdx.x == 0) warp_sums[warps] = all;
    __syncthreads();
    return make_int2(s.x + add.x, s.y + add.y);
}

__device__ __forceinline__ int2 split_of(const int64_t* rowptr, int32_t i, int32_t m, int32_t threshold, int32_t chunk, int64_t* e0, int64_t* e1)
{
    if (i >= m) return make_int2(0, 0);
    *e0 = rowptr[i];
    *e1 = rowptr[i + 1];
    return *e1 - *e0 > threshold ? make_int2(1, (int)((*e1 - *e0 + chunk - 1) / chunk)) : make_int2(0, 0);
}

// Per 256 rows: how many are split, and into how many chunks; over all, how many chunks the static entry counts.
__global__ void __launch_bounds__(T) k_row_census(const int64_t* __restrict__ rowptr, int32_t m, int32_t threshold, int32_t chunk, int32_t static_threshold,
                                                  int32_t static_chunk, int2* __restrict__ block_sums, PlanCounts* __restrict__ counts)
{
    if (counts->bad) return;
    __shared__ int2 sums[T / 32 + 1];
    __shared__ unsigned long long longest, split, pieces;          // one global atomic a block, not one a warp
    if (threadIdx.x == 0) longest = split = pieces = 0;
    int64_t e0 = 0, e1 = 0;
    const int2 s = split_of(rowptr, blockIdx.x * T + threadIdx.x, m, threshold, chunk, &e0, &e1);
    block_scan(s, sums);
    unsigned long long deg = (unsigned long long)(e1 - e0), heavy = s.x ? deg : 0;
    uint32_t part = e1 - e0 > static_threshold ? ((uint32_t)(e1 - e0) + (uint32_t)static_chunk - 1) / (uint32_t)static_chunk : 0;
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, deg, off);
        deg = o > deg ? o : deg;
        heavy += __shfl_xor_sync(0xffffffffu, heavy, off);
    }
    part = __reduce_add_sync(0xffffffffu, part);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&longest, deg);
        if (heavy) atomicAdd(&split, heavy);
        if (part) atomicAdd(&pieces, (unsigned long long)part);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    block_sums[blockIdx.x] = sums[T / 32];
    if (longest) atomicMax(&counts->max_row, longest);
    if (split) atomicAdd(&counts->heavy_nnz, split);
    if (pieces) atomicAdd(&counts->static_chunks, pieces);
}

// One CTA: exclusive sums over the blocks' counts in place, and over the columns' bitmap.
__global__ void __launch_bounds__(1024) k_scan_blocks(int2* __restrict__ block_sums, int32_t blocks, PlanCounts* __restrict__ counts)
{
    if (counts->bad) return;
    __shared__ int2 sums[33];
    int2 carry = make_int2(0, 0);
    for (int32_t b0 = 0; b0 < blocks; b0 += 1024) {
        const int32_t b = b0 + threadIdx.x;
        const int2 v = b < blocks ? block_sums[b] : make_int2(0, 0);
        const int2 s = block_scan(v, sums);
        if (b < blocks) block_sums[b] = make_int2(carry.x + s.x - v.x, carry.y + s.y - v.y);
        carry.x += sums[32].x;
        carry.y += sums[32].y;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        counts->n_heavy = carry.x;
        counts->n_chunks = carry.y;
    }
}

__global__ void k_count_bits(const uint32_t* __restrict__ bitmap, int64_t words, PlanCounts* __restrict__ counts)
{
    unsigned long long local = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += stride) local += __popc(bitmap[w]);
    for (int off = 16; off > 0; off >>= 1) local += __shfl_xor_sync(0xffffffffu, local, off);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(&counts->touched, local);
}

// The chunks of every split row, in row order, and how many start in each column band.  The CTA's threads share its rows'
// chunks out evenly (a row of 100,000 entries has hundreds).
__global__ void __launch_bounds__(T) k_emit_chunks(const int64_t* __restrict__ rowptr, int32_t m, int32_t k, int32_t threshold, int32_t chunk,
                                                   const int2* __restrict__ block_first, const int32_t* __restrict__ col,
                                                   dg_chunk* __restrict__ chunks, int32_t* __restrict__ bands, const PlanCounts* __restrict__ counts)
{
    if (counts->bad) return;
    __shared__ int2 sums[T / 32 + 1];
    __shared__ int64_t first[T], last[T];
    __shared__ int2 upto[T];                                      // split rows and chunks up to and with this row
    int64_t e0 = 0, e1 = 0;
    const int2 s = split_of(rowptr, blockIdx.x * T + threadIdx.x, m, threshold, chunk, &e0, &e1);
    const int2 incl = block_scan(s, sums);
    first[threadIdx.x] = e0;
    last[threadIdx.x] = e1;
    upto[threadIdx.x] = incl;
    __syncthreads();
    const int2 before = block_first[blockIdx.x];
    for (int c = threadIdx.x; c < sums[T / 32].y; c += T) {
        int lo = 0, hi = T - 1;                                   // the row of chunk c: the first with upto.y > c
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (upto[mid].y > c) hi = mid; else lo = mid + 1;
        }
        const int row_first = lo > 0 ? upto[lo - 1].y : 0, n = upto[lo].y - row_first;
        const int64_t e = first[lo] + (int64_t)(c - row_first) * chunk, left = last[lo] - e;
        chunks[before.y + c] = dg_chunk{e, (int32_t)(left < chunk ? left : chunk), (int32_t)(blockIdx.x * T + lo), before.y + c,
                                        before.y + row_first, n, before.x + upto[lo].x - 1};
        atomicAdd(&bands[band_of(col[e], k)], 1);
    }
}

// One CTA: exclusive sums over the bands.
__global__ void __launch_bounds__(1024) k_scan_bands(int32_t* __restrict__ bands, const PlanCounts* __restrict__ counts)
{
    if (counts->bad || counts->n_chunks == 0) return;
    __shared__ int2 sums[33];
    int v[kBands / 1024], local = 0;
    for (int i = 0; i < kBands / 1024; ++i) local += v[i] = bands[threadIdx.x * (kBands / 1024) + i];
    int at = block_scan(make_int2(local, 0), sums).x - local;
    for (int i = 0; i < kBands / 1024; ++i) {
        bands[threadIdx.x * (kBands / 1024) + i] = at;
        at += v[i];
    }
}

// Visiting order of the chunks.  A chunk's scratch row is fixed, so the list may be walked in any order without changing a
// bit of the result.  Chunks are handed to lane groups in list order, CTAs in launch order; ordered by the column band their
// window starts in (the entries of a row are in ascending column order), the warps that run at the same time gather
// from the same band of B's rows instead of from all of B, which is what lets the L2 hold the band's popular rows (2.4 M
// nodes, F = 256: 11.8 -> 9.6 ms per product; F = 100: 6.1 -> 4.9 ms).
__global__ void k_order_chunks(const dg_chunk* __restrict__ in, dg_chunk* __restrict__ out, int32_t* __restrict__ bands,
                               const int32_t* __restrict__ col, int32_t k, const PlanCounts* __restrict__ counts)
{
    if (counts->bad) return;
    const int32_t n = counts->n_chunks;
    for (int32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const dg_chunk ch = in[c];
        out[atomicAdd(&bands[band_of(col[ch.e0], k)], 1)] = ch;
    }
}

// Thread t: the row that holds entry t * task_nnz, i.e. the smallest r with rowptr[r + 1] > t * task_nnz.
__global__ void k_task_first_row(const int64_t* __restrict__ rowptr, int32_t m, int64_t task_nnz, int32_t n_tasks,
                                 int32_t* __restrict__ first_row)
{
    const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tasks) return;
    const int64_t e = (int64_t)t * task_nnz;
    int32_t lo = 0, hi = m;            // answer in [0, m): entry e exists, so some row ends beyond it
    while (lo < hi) {
        const int32_t mid = lo + (hi - lo) / 2;
        if (rowptr[mid + 1] > e) hi = mid; else lo = mid + 1;
    }
    first_row[t] = lo;
}

// Rows whose entries fall into more than one task.
__global__ void k_split_census(const int64_t* __restrict__ rowptr, int32_t m, int64_t task_nnz,
                               dg_split_row* __restrict__ out, int32_t capacity, int32_t* __restrict__ count)
{
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int64_t e0 = rowptr[i], e1 = rowptr[i + 1];
    if (e1 <= e0) return;
    const int64_t t0 = e0 / task_nnz, t1 = (e1 - 1) / task_nnz;
    if (t0 == t1) return;
    const int32_t slot = atomicAdd(count, 1);
    if (slot < capacity) out[slot] = dg_split_row{i, (int32_t)t0, (int32_t)t1, 0};
}

int build_tasks(dg_plan* p, int32_t task_nnz, cudaStream_t stream)
{
    dg_pool_free(p->task_first_row);
    dg_pool_free(p->split);
    p->task_first_row = nullptr;
    p->split = nullptr;
    p->task_nnz = task_nnz;
    p->n_tasks = (int32_t)((p->nnz + task_nnz - 1) / task_nnz);
    p->n_split = 0;
    if (p->n_tasks == 0) return DG_OK;
    int rc = dg_pool_alloc((void**)&p->task_first_row, (size_t)p->n_tasks * sizeof(int32_t));
    if (rc) return rc;
    k_task_first_row<<<(p->n_tasks + T - 1) / T, T, 0, stream>>>(p->rowptr, p->m, task_nnz, p->n_tasks, p->task_first_row);
    PoolScope tmp(stream);
    dg_split_row* d_rows = nullptr;
    int32_t* d_count = nullptr;
    const int32_t capacity = p->n_tasks;      // a row can only be cut at one of the n_tasks - 1 task boundaries
    if ((rc = tmp.alloc(&d_rows, (size_t)capacity)) || (rc = tmp.alloc(&d_count, 1))) return rc;
    DG_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int32_t), stream));
    k_split_census<<<(p->m + T - 1) / T, T, 0, stream>>>(p->rowptr, p->m, task_nnz, d_rows, capacity, d_count);
    int32_t h_count = 0;
    DG_CUDA(cudaMemcpyAsync(&h_count, d_count, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));
    DG_CUDA(cudaGetLastError());
    if (h_count > capacity) return DG_ERR_STATE;
    if (h_count > 0) {
        std::vector<dg_split_row> rows((size_t)h_count);
        DG_CUDA(cudaMemcpy(rows.data(), d_rows, rows.size() * sizeof(dg_split_row), cudaMemcpyDeviceToHost));
        std::sort(rows.begin(), rows.end(), [](const dg_split_row& a, const dg_split_row& b) { return a.row < b.row; });
        if ((rc = dg_pool_alloc((void**)&p->split, rows.size() * sizeof(dg_split_row)))) return rc;
        DG_CUDA(cudaMemcpy(p->split, rows.data(), rows.size() * sizeof(dg_split_row), cudaMemcpyHostToDevice));
        p->n_split = h_count;
    }
    return DG_OK;
}

}  // namespace

// Task tables of the streaming kernel, built when that family is first used on a plan.
int dg_plan_ensure_tasks(dg_plan* p, cudaStream_t stream)
{
    return p->task_nnz > 0 ? DG_OK : build_tasks(p, DG_DEFAULT_TASK_NNZ, stream);
}

extern "C" int dg_plan_set_task_size(dg_plan* p, int32_t task_nnz, void* stream)
try {
    if (!p) return DG_ERR_NULL;
    if (task_nnz <= 0) task_nnz = DG_DEFAULT_TASK_NNZ;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != p->device) return DG_ERR_STATE;
    DG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));     // earlier products may still read the old tables
    return build_tasks(p, task_nnz, (cudaStream_t)stream);
} catch (...) {
    return dg_exception();
}

extern "C" int dg_plan_device_status(const dg_plan* p, int* host_status, void* stream)
{
    if (!p || !host_status) return DG_ERR_NULL;
    DG_CUDA(cudaMemcpyAsync(host_status, p->status, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    DG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return DG_OK;
}

namespace {

// lean: a plan that will serve one product and be destroyed (dg_spmm_coo): the distinct-column census (statistics only) is
// left out; touched_columns then reads k.
template <class Id>
int plan_build(const Id* row, const Id* col, int64_t nnz, int32_t m, int32_t k, int32_t heavy_threshold, int32_t chunk, bool lean,
               int32_t* col32, void* stream_, dg_plan** out)
{
    if (!out) return DG_ERR_NULL;
    *out = nullptr;
    if (nnz < 0 || m < 0 || k < 0) return DG_ERR_DIMS;
    if (nnz > 0 && (!row || !col || (sizeof(Id) == 8 && !col32))) return DG_ERR_NULL;
    if (nnz > 0 && (m == 0 || k == 0)) return DG_ERR_DIMS;
    const int32_t static_threshold = heavy_threshold > 0 ? heavy_threshold : DG_STATIC_CHUNK, static_chunk = chunk > 0 ? chunk : DG_STATIC_CHUNK;
    if (heavy_threshold <= 0) heavy_threshold = dg_default_chunk(nnz, m);
    if (chunk <= 0) chunk = dg_default_chunk(nnz, m);
    cudaStream_t stream = (cudaStream_t)stream_;

    dg_plan* p = new (std::nothrow) dg_plan();
    if (!p) return (int)cudaErrorMemoryAllocation;
    p->m = m; p->k = k; p->nnz = nnz;
    p->col = sizeof(Id) == 8 ? col32 : reinterpret_cast<const int32_t*>(col);
    p->heavy_threshold = heavy_threshold; p->chunk = chunk;
    int rc = DG_OK;
    struct Owner {                        // until the plan is handed out
        dg_plan* plan;
        ~Owner() { dg_plan_destroy(plan); }
    } owner{p};
    if ((rc = (int)cudaGetDevice(&p->device)) != 0) return rc;

    // upper bounds: a split row holds more than heavy_threshold entries, and its last chunk may be a short one
    const int64_t max_heavy = std::min<int64_t>(nnz / ((int64_t)heavy_threshold + 1), m), max_chunks = nnz / chunk + max_heavy;
    if (max_chunks > INT32_MAX) return DG_ERR_UNSUPPORTED;
    const int64_t words = lean ? 0 : ((int64_t)k + 31) / 32;
    const int32_t row_blocks = (int32_t)(((int64_t)m + T - 1) / T);
    PoolScope tmp(stream);
    uint8_t* zeroed = nullptr;            // counts, column bands, column bitmap: cleared by one memset
    int2* block_sums = nullptr;
    dg_chunk* in_row_order = nullptr;
    const size_t zero_bytes = sizeof(PlanCounts) + kBands * sizeof(int32_t) + (size_t)words * sizeof(uint32_t);
    if ((rc = dg_pool_alloc((void**)&p->rowptr, ((size_t)m + 1) * sizeof(int64_t))) || (rc = dg_pool_alloc((void**)&p->status, DG_STATUS_WORDS * sizeof(int))) ||
        (rc = tmp.alloc(&zeroed, zero_bytes)) || (rc = tmp.alloc(&block_sums, (size_t)row_blocks)))
        return rc;
    if (max_chunks > 0 && ((rc = dg_pool_alloc((void**)&p->chunks, (size_t)max_chunks * sizeof(dg_chunk))) ||
                           (rc = dg_pool_alloc((void**)&p->arrived, (size_t)max_heavy * DG_FINISH_TILES * sizeof(int))) ||
                           (rc = tmp.alloc(&in_row_order, (size_t)max_chunks))))
        return rc;
    PlanCounts* counts = reinterpret_cast<PlanCounts*>(zeroed);
    int32_t* bands = reinterpret_cast<int32_t*>(counts + 1);
    uint32_t* bitmap = words ? reinterpret_cast<uint32_t*>(bands + kBands) : nullptr;
    cudaMemsetAsync(zeroed, 0, zero_bytes, stream);
    cudaMemsetAsync(p->status, 0, DG_STATUS_WORDS * sizeof(int), stream);
    if (max_chunks > 0) cudaMemsetAsync(p->arrived, 0, (size_t)max_heavy * DG_FINISH_TILES * sizeof(int), stream);

    const int64_t per_block = (int64_t)T * kEntriesPerThread;
    k_ingest<Id><<<(unsigned)((nnz + 1 + per_block - 1) / per_block), T, 0, stream>>>(row, col, nnz, m, k, sizeof(Id) == 8 ? col32 : nullptr, p->rowptr,
                                                                                     bitmap, counts);
    if (row_blocks > 0) {
        k_row_census<<<row_blocks, T, 0, stream>>>(p->rowptr, m, heavy_threshold, chunk, static_threshold, static_chunk, block_sums, counts);
        if (max_chunks > 0) {
            k_scan_blocks<<<1, 1024, 0, stream>>>(block_sums, row_blocks, counts);
            k_emit_chunks<<<row_blocks, T, 0, stream>>>(p->rowptr, m, k, heavy_threshold, chunk, block_sums, p->col, in_row_order, bands, counts);
            k_scan_bands<<<1, 1024, 0, stream>>>(bands, counts);
            k_order_chunks<<<(unsigned)std::min<int64_t>((max_chunks + T - 1) / T, 148 * 8), T, 0, stream>>>(in_row_order, p->chunks, bands, p->col, k, counts);
        }
    }
    if (words > 0) k_count_bits<<<(unsigned)std::min<int64_t>((words + T - 1) / T, 148 * 8), T, 0, stream>>>(bitmap, words, counts);
    PlanCounts h{};
    if ((rc = (int)cudaMemcpyAsync(&h, counts, sizeof(h), cudaMemcpyDeviceToHost, stream)) || (rc = (int)cudaStreamSynchronize(stream)) ||
        (rc = (int)cudaGetLastError()))
        return rc;
    tmp.idle = true;
    if (h.bad) return DG_ERR_INDEX;
    if (h.n_heavy > max_heavy || h.n_chunks > max_chunks) return DG_ERR_STATE;      // cannot happen
    p->max_row_nnz = (int64_t)h.max_row;
    p->heavy_nnz = (int64_t)h.heavy_nnz;
    p->touched_columns = lean ? (int64_t)k : (int64_t)h.touched;
    p->n_heavy = h.n_heavy;
    p->n_chunks = h.n_chunks;
    p->static_chunks = (int64_t)h.static_chunks;
    *out = p;
    owner.plan = nullptr;
    return DG_OK;
}

}  // namespace

int dg_plan_build_lean(const int32_t* row, const int32_t* col, int64_t nnz, int32_t m, int32_t k, void* stream, dg_plan** out)
{
    return plan_build<int32_t>(row, col, nnz, m, k, 0, 0, true, nullptr, stream, out);
}

extern "C" int dg_plan_create_ex(const int32_t* row, const int32_t* col, int64_t nnz, int32_t m, int32_t k,
                                 int32_t heavy_threshold, int32_t chunk, void* stream, dg_plan** out)
try {
    return plan_build<int32_t>(row, col, nnz, m, k, heavy_threshold, chunk, false, nullptr, stream, out);
} catch (...) {
    return dg_exception();
}

extern "C" int dg_plan_create_i64(const int64_t* row, const int64_t* col, int64_t nnz, int32_t m, int32_t k, int32_t heavy_threshold,
                                  int32_t chunk, int32_t* col32, void* stream, dg_plan** out)
try {
    return plan_build<int64_t>(row, col, nnz, m, k, heavy_threshold, chunk, false, col32, stream, out);
} catch (...) {
    return dg_exception();
}

extern "C" int dg_plan_create(const int32_t* row, const int32_t* col, int64_t nnz, int32_t m, int32_t k, void* stream,
                              dg_plan** out)
{
    return dg_plan_create_ex(row, col, nnz, m, k, 0, 0, stream, out);
}

extern "C" int dg_plan_destroy(dg_plan* p)
{
    if (!p) return DG_OK;
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != p->device) cudaSetDevice(p->device);
    cudaDeviceSynchronize();              // products on any stream are done with the blocks before the pool may hand them out
    for (void* b : {(void*)p->rowptr, (void*)p->chunks, (void*)p->arrived, (void*)p->scratch, (void*)p->task_first_row, (void*)p->split, (void*)p->status})
        dg_pool_free(b);
    dg_tiles_free(p->tiles);
    if (prev != p->device && prev >= 0) cudaSetDevice(prev);
    delete p;
    return DG_OK;
}

extern "C" int dg_plan_get_stats(const dg_plan* p, dg_plan_stats* o)
{
    if (!p || !o) return DG_ERR_NULL;
    o->nnz = p->nnz; o->m = p->m; o->k = p->k;
    o->heavy_threshold = p->heavy_threshold; o->chunk = p->chunk;
    o->heavy_rows = p->n_heavy; o->heavy_chunks = p->n_chunks;
    o->heavy_nnz = p->heavy_nnz; o->max_row_nnz = p->max_row_nnz; o->touched_columns = p->touched_columns;
    return DG_OK;
}

extern "C" int dg_plan_copy_rowptr(const dg_plan* p, int64_t* host_rowptr, void* stream)
{
    if (!p || !host_rowptr) return DG_ERR_NULL;
    DG_CUDA(cudaMemcpyAsync(host_rowptr, p->rowptr, ((size_t)p->m + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost,
                            (cudaStream_t)stream));
    DG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return DG_OK;
}

// ---- are these the ids a plan was built from? -------------------------------------------------------------------------
namespace {

__global__ void __launch_bounds__(T) k_ids_equal(const int32_t* __restrict__ row_a, const int32_t* __restrict__ row_b,
                                                 const int32_t* __restrict__ col_a, const int32_t* __restrict__ col_b, int64_t nnz,
                                                 volatile int* differ, volatile int* failed_check, int check)
{
    bool same = true;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += stride)
        same = same && (__ldcs(row_a + e) == __ldcs(row_b + e)) & (__ldcs(col_a + e) == __ldcs(col_b + e));
    if (!same) {
        *differ = 1;
        *failed_check = check;
    }
}

// What a host thread keeps for its checks, as long as it lives.  The verdict is a word of pinned host memory that only a
// difference writes: the call waits for the kernel and reads it, no copy back.
struct Verdict {
    int* word = nullptr;
    cudaEvent_t done[64] = {};
    ~Verdict()
    {
        if (word) cudaFreeHost(word);
        for (cudaEvent_t e : done)
            if (e) cudaEventDestroy(e);
    }
};

}  // namespace

// The product is issued behind the check without waiting for its verdict, and writes nothing if that is negative: the host's
// wait runs beside the product instead of in front of it (306,129-row block, F = 256: 214 -> 207 us a call; 5,000-row block: 40 -> 36).
extern "C" int dg_spmm_csr_checked(const dg_plan* plan, const int32_t* plan_row, const int32_t* plan_col, const int32_t* row, const int32_t* col,
                                   const float* val, const float* B, int64_t ldb, float* C, int64_t ldc, int32_t F, float alpha, float beta,
                                   int* host_equal, void* stream_)
try {
    int rc = dg_check_spmm_args(plan, val, B, ldb, C, ldc, F, 0u, nullptr, nullptr);
    if (rc) return rc;
    if (!host_equal || (plan->nnz > 0 && (!plan_row || !plan_col || !row || !col))) return DG_ERR_NULL;
    cudaStream_t stream = (cudaStream_t)stream_;
    // The scratch grows, and a check and the product behind it are issued, under one lock: the word that the product reads holds one
    // check's number, and another thread's check between the two could take its place.
    dg_plan* p = const_cast<dg_plan*>(plan);
    std::unique_lock<std::mutex> lock(p->issue);
    if ((rc = dg_spmm_prepare(plan, F, stream))) return rc;
    *host_equal = 1;
    auto product = [&](int check) {
        return dg_spmm_launch(plan, val, B, ldb, C, ldc, F, alpha, beta, 0u, nullptr, nullptr, plan->scratch, plan->scratch_floats, stream, check);
    };
    if (plan->nnz == 0) return product(0);
    static thread_local Verdict verdict;
    cudaEvent_t& done = verdict.done[plan->device & 63];
    if (!verdict.word) DG_CUDA(cudaHostAlloc((void**)&verdict.word, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
    if (!done) DG_CUDA(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
    *verdict.word = 0;
    int* differ = nullptr;
    DG_CUDA(cudaHostGetDevicePointer((void**)&differ, verdict.word, 0));
    p->checks = p->checks == INT32_MAX ? 1 : p->checks + 1;
    const int64_t blocks = (plan->nnz + T - 1) / T;
    k_ids_equal<<<(unsigned)std::min<int64_t>(blocks, 148 * 8), T, 0, stream>>>(plan_row, row, plan_col, col, plan->nnz, differ, plan->status + 1, p->checks);
    DG_CUDA(cudaGetLastError());
    DG_CUDA(cudaEventRecord(done, stream));
    const bool rows = !dg_spmm_stream_eligible(plan, B, ldb, C, ldc, F);
    rc = rows ? product(p->checks) : DG_OK;
    lock.unlock();
    DG_CUDA(cudaEventSynchronize(done));
    *host_equal = *(volatile int*)verdict.word == 0;
    if (rc == DG_OK && !rows && *host_equal) {
        lock.lock();
        rc = product(0);
    }
    return rc;
} catch (...) {
    return dg_exception();
}
