// CSR row block x dense fp32 operand for sm_100a:  C = epilogue(alpha * A * B + beta * C).
//
// Replaces cusparseSpMM(COO_ALG4) as called by the reference (light_dist_gnn/spmm_cpp/spmm.cpp:26-28).
//
// The product is a gather: every stored entry (i, j, a) pulls the F-float row j of B and adds a * B[j,:] into
// row i of C.  HBM / L2 bandwidth bounds it.  Scheduling (k_spmm):
//   * light rows (<= heavy_threshold entries): a group of 4 to 32 lanes per row, out of CTA-local windows sorted by length;
//   * heavy rows: cut into chunks of `chunk` entries at plan time; one lane group per chunk leaves a partial sum in
//     scratch, and the last one to arrive adds the partials in chunk order and applies the epilogue.  No float
//     atomics anywhere: the result is bit-reproducible.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <vector>
#include "dg_internal.h"
#include "dg_tiles.h"
#include "dg_umma.h"

namespace {

// ---- instrumentation: event pairs around products while a profile is open -------------------------------------------
struct ProfileState {
    std::mutex mu;
    bool open = false;
    std::vector<cudaEvent_t> events;     // pairs; reused between profiles
    size_t used = 0;
    double alg_bytes = 0, gather_bytes = 0, flops = 0;
    int64_t products = 0;
};
ProfileState g_profile;
std::atomic<int64_t> g_kernel_launches{0};

cudaEvent_t profile_event(cudaStream_t stream)   // caller holds the mutex
{
    if (g_profile.used == g_profile.events.size()) {
        cudaEvent_t e;
        if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
        g_profile.events.push_back(e);
    }
    cudaEvent_t e = g_profile.events[g_profile.used++];
    cudaEventRecord(e, stream);
    return e;
}

struct SpmmArgs {
    const int64_t* rowptr;
    const int32_t* col;
    const float* val;
    const float* B;
    float* C;
    const float* row_scale;
    const float* bias;
    const dg_chunk* chunks;
    const int32_t* chunk_col;   // entries of the chunks: the matrix's own, or what the tiles leave of the split rows
    const float* chunk_val;
    const int2* parts;          // kTiled: partial results of the tiles per split row (dg_tiles.h)
    const float4* part_area;
    int64_t part_ld4;           // 16-byte pieces of a partial row
    int* tile_words;            // kTiled, kWhole: dg_plan::status + DG_TILE_WORDS
    int* arrived;               // [n_heavy x DG_FINISH_TILES] partial sums of a split row that are in place; zero between products
    float* scratch;
    int64_t ldb, ldc, lds;      // lds: row stride of the partial sums
    int32_t m, F;
    int32_t heavy_threshold;
    int32_t n_chunks;
    int32_t rows_per_cta;
    int32_t vec_first, vec_end; // the vectors of a row this launch covers
    float alpha, beta;
    uint32_t flags;
    int check;                  // non-zero: nothing is written if *failed_check says that this check failed
    const int* failed_check;
};

// VEC floats side by side, aligned to as many (8: 32 bytes).  A gathered row comes by way of the L1, which holds the most frequent ones.
template <int VEC> __device__ __forceinline__ void load_vec(const float* p, float (&out)[VEC])
{
    if constexpr (VEC == 8) {
        asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(out[0]), "=f"(out[1]), "=f"(out[2]), "=f"(out[3]), "=f"(out[4]), "=f"(out[5]), "=f"(out[6]), "=f"(out[7]) : "l"(p));
    } else if constexpr (VEC == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p));
        out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    } else if constexpr (VEC == 2) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(p));
        out[0] = v.x; out[1] = v.y;
    } else {
        out[0] = __ldg(p);
    }
}
// Pieces of at most 16 bytes, by the given access.
template <int VEC, class Use> __device__ __forceinline__ void each_piece(Use use)
{
    if constexpr (VEC == 8) {
        use(0);
        use(4);
    } else {
        use(0);
    }
}
template <int VEC> struct Piece { using type = float4; };
template <> struct Piece<2> { using type = float2; };
template <> struct Piece<1> { using type = float; };
template <int VEC> using piece_t = typename Piece<VEC>::type;
__device__ __forceinline__ void set_scaled(float* acc, float scale, float4 v) { acc[0] = scale * v.x; acc[1] = scale * v.y; acc[2] = scale * v.z; acc[3] = scale * v.w; }
__device__ __forceinline__ void set_scaled(float* acc, float scale, float2 v) { acc[0] = scale * v.x; acc[1] = scale * v.y; }
__device__ __forceinline__ void set_scaled(float* acc, float scale, float v) { acc[0] = scale * v; }
__device__ __forceinline__ void add(float* acc, float4 v) { acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w; }
__device__ __forceinline__ void add(float* acc, float2 v) { acc[0] += v.x; acc[1] += v.y; }
__device__ __forceinline__ void add(float* acc, float v) { acc[0] += v; }
__device__ __forceinline__ void pack(float4& v, const float* acc) { v = make_float4(acc[0], acc[1], acc[2], acc[3]); }
__device__ __forceinline__ void pack(float2& v, const float* acc) { v = make_float2(acc[0], acc[1]); }
__device__ __forceinline__ void pack(float& v, const float* acc) { v = acc[0]; }

// What is left to do with a sum before it is stored: alpha * sum + beta * C (alpha == 1 has beta * C in the sum already), row
// scale, bias, ReLU.
__device__ __forceinline__ float finish(const SpmmArgs& a, float sum, const float* c, int32_t row, int32_t colidx)
{
    float out = sum;
    if (a.alpha != 1.f) {
        out *= a.alpha;
        if (a.beta != 0.f) out = fmaf(a.beta, *c, out);
    }
    if (a.flags & DG_EPI_ROW_SCALE) out *= __ldg(a.row_scale + row);
    if (a.flags & DG_EPI_BIAS) out += __ldg(a.bias + colidx);
    if (a.flags & DG_EPI_RELU) out = fmaxf(out, 0.f);
    return out;
}

// ---- the product -------------------------------------------------------------------------------------------------------
// A warp is G = 32 / LPR groups of LPR lanes, and every group works on an item of its own: a row, or a chunk of a split
// row.  Lane gl of a group owns the TPL vectors (VEC floats each) gl, gl + LPR, ... of the column tile blockIdx.y, so a
// gathered row of B is read with coalesced loads of up to 256 bits; the group reads LPR (col, val) pairs at a time, the next
// LPR while it works on these, and hands them out by shuffle, U gathers in flight before the first FMA.  A row is summed
// in entry order by one group, whatever LPR is.
//
// The first `chunk_ctas` CTAs take the chunks of the split rows, NG = 256 / LPR at a time; each group leaves its partial
// sum in scratch and adds one to its row's count, and the group that finds the count complete adds the row's partial sums in
// chunk order and writes the row (no second launch, no float atomics, the same bits every time).
//
// The other CTAs own `rows_per_cta` <= 256 consecutive rows each.  They read the window's row offsets with one coalesced
// load (a warp that fetches its own row's offsets waits a memory latency per row), sort the rows by length class in shared
// memory and hand them out longest first, G at a time, so that the rows a warp works on together are about equally long and
// the last rows of a CTA are short ones.  The first entries of the next G rows are requested before the current ones are
// gathered.
//
// What bounds it: the gathers.  Wide rows that the L2 holds come at 18 TB/s, 64 bytes a clock and SM (dense graph, F = 256: 41 GB in
// 2.27 ms with the L2 at 79 % of its throughput, issue slots at 36 %); larger graphs are held
// up by the L2 and by what misses it (1 M nodes, 49 M entries: L2 65 %, DRAM 49 %, hit rate 63 %); narrow rows by the L1's data pipe, issue
// and latency (300 k nodes, F = 100: 11 TB/s, L1 data pipe 75 %, issue 61 %, L2 50 %; 1 M nodes, F = 64: 10 TB/s, 56, 53, 43 %); small graphs and
// short rows by latency, which the offsets in shared memory, the look-ahead and U hide.  Against separate kernels with a warp per
// row (B200, us per product):
//   10,000 nodes, 210 k entries, F = 64: 74 -> 17      150,001 nodes, 2.6 M entries, F = 256: 263 -> 204; F = 48: 156 -> 79
//   1 M nodes, 17 M entries, F = 64: 748 -> 400, F = 16: 582 -> 194        306 k-row stage block, 1.9 M entries, F = 256: 281 -> 182
//   2,449,029 nodes, 126 M entries, F = 256: 10,000 -> 8,640, F = 100: 5,760 -> 4,350, F = 48: 3,620 -> 2,230
// MODE kTiled: a product with tiles, whose partial results the split rows take in; kWhole: its second launch.  That does nothing
// unless the tiles could not be used (dg_tiles.h): then the first one has left the split rows alone, and a few CTAs per SM gather
// them whole (as last CTAs of the first launch: 4 % faster at F = 100, 1 to 3 % slower at F = 256 and 48, by its registers).  kPlain is
// compiled without any of this: with the branches in it eight stage blocks (F = 256) took 1 % longer.
// PADDED: the operand is the padded copy of a matrix whose rows are not 16-byte multiples; C is then written float by float.
enum { kPlain, kTiled, kWhole };
template <int VEC, int LPR, int TPL, int U, int MINB, bool PADDED, int MODE>
__global__ void __launch_bounds__(256, MINB) k_spmm(const SpmmArgs a, const int chunk_ctas)
{
    constexpr int G = 32 / LPR, NG = 256 / LPR;
    static_assert(U <= LPR, "a batch of U gathers comes from one set of LPR entries");
    const int gl = threadIdx.x % LPR, grp = (threadIdx.x & 31) / LPR;
    const int vec0 = a.vec_first + blockIdx.y * (LPR * TPL) + gl;
    bool on[TPL];
#pragma unroll
    for (int t = 0; t < TPL; ++t) on[t] = vec0 + t * LPR < a.vec_end;
    const float* bl = a.B + (int64_t)vec0 * VEC;
    const int64_t ldb = a.ldb;
    float acc[TPL][VEC];
    const int failed = a.check ? __ldcg(a.failed_check) : 0;      // under way while the first offsets and entries are

    // acc += sum over this group's `len` entries; `e` is this lane's first entry, c / v hold it already
    auto gather = [&](const int32_t* col, const float* val, int64_t e, int len, int c, float v) {
        const int longest = G == 1 ? len : __reduce_max_sync(0xffffffffu, len);
#pragma unroll 1
        for (int base = 0; base < longest; base += LPR) {
            int c_next = 0;
            float v_next = 0.f;
            if (base + LPR + gl < len) {
                c_next = __ldcs(col + e + base + LPR);            // streamed once: keep it from displacing rows of B in cache
                v_next = __ldcs(val + e + base + LPR);
            }
            const int cnt = LPR % U ? min(LPR, len - base) : len - base, steps = min(LPR, longest - base);
#pragma unroll 1
            for (int k = 0; k < steps; k += U) {
                float x[U][TPL][VEC], w[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = __shfl_sync(0xffffffffu, c, k + u, LPR);
                    w[u] = __shfl_sync(0xffffffffu, v, k + u, LPR);          // 0 beyond the last entry
                    if (LPR % U && k + u >= LPR) w[u] = 0.f;                 // the next set's
                    const float* row = bl + j * ldb;
#pragma unroll
                    for (int t = 0; t < TPL; ++t) {
                        if (k + u < cnt && on[t]) {
                            load_vec<VEC>(row + t * LPR * VEC, x[u][t]);
                        } else {
#pragma unroll
                            for (int q = 0; q < VEC; ++q) x[u][t][q] = 0.f;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int t = 0; t < TPL; ++t)
#pragma unroll
                        for (int q = 0; q < VEC; ++q) acc[t][q] = fmaf(w[u], x[u][t][q], acc[t][q]);
            }
            c = c_next;
            v = v_next;
        }
    };
    // acc = beta * C[row] where the product starts from it (alpha == 1: no registers for the old row beside the sum, and its
    // latency runs under the first gathers'), else 0
    auto begin_row = [&](int32_t row, bool add) {
        const float* cp = a.C + (int64_t)row * a.ldc + (int64_t)vec0 * VEC;
#pragma unroll
        for (int t = 0; t < TPL; ++t) {
#pragma unroll
            for (int q = 0; q < VEC; ++q) acc[t][q] = 0.f;
            if (!add || !on[t]) continue;
            const float* p = cp + t * LPR * VEC;
            if constexpr (PADDED) {
#pragma unroll
                for (int q = 0; q < VEC; ++q)
                    if ((vec0 + t * LPR) * VEC + q < a.F) acc[t][q] = a.beta * __ldcs(p + q);
            } else {
                each_piece<VEC>([&](int at) { set_scaled(acc[t] + at, a.beta, __ldcs(reinterpret_cast<const piece_t<VEC>*>(p + at))); });
            }
        }
    };
    const bool add_first = a.beta != 0.f && a.alpha == 1.f;
    auto store_row = [&](int32_t row) {
        float* cp = a.C + (int64_t)row * a.ldc + (int64_t)vec0 * VEC;
#pragma unroll
        for (int t = 0; t < TPL; ++t) {
            if (!on[t]) continue;
            const int c0 = (vec0 + t * LPR) * VEC;
            float* p = cp + t * LPR * VEC;
            if (a.alpha != 1.f || a.flags) {
#pragma unroll
                for (int q = 0; q < VEC; ++q)
                    if (!PADDED || c0 + q < a.F) acc[t][q] = finish(a, acc[t][q], p + q, row, c0 + q);
            }
            if constexpr (PADDED) {
#pragma unroll
                for (int q = 0; q < VEC; ++q)
                    if (c0 + q < a.F) __stcs(p + q, acc[t][q]);
            } else {
                each_piece<VEC>([&](int at) {
                    piece_t<VEC> v;
                    pack(v, acc[t] + at);
                    __stcs(reinterpret_cast<piece_t<VEC>*>(p + at), v);
                });
            }
        }
    };

    // NG chunks of split rows, from chunk id0 on
    auto run_chunks = [&](int id0) {
        const int id = id0 + threadIdx.x / LPR;
        const bool valid = id < a.n_chunks;
        dg_chunk ch{};
        if (valid) ch = a.chunks[id];
        int c = 0;
        float v = 0.f;
        if (gl < ch.len) {
            c = __ldcs(a.chunk_col + ch.e0 + gl);
            v = __ldcs(a.chunk_val + ch.e0 + gl);
        }
        if (a.check && failed == a.check) return;
        begin_row(0, false);
        gather(a.chunk_col, a.chunk_val, ch.e0 + gl, ch.len, c, v);
        if (valid) {
            float* sp = a.scratch + (int64_t)ch.slot * a.lds + (int64_t)vec0 * VEC;
#pragma unroll
            for (int t = 0; t < TPL; ++t) {
                if (!on[t]) continue;
                float* p = sp + t * LPR * VEC;
                each_piece<VEC>([&](int at) {
                    piece_t<VEC> v;
                    pack(v, acc[t] + at);
                    __stcg(reinterpret_cast<piece_t<VEC>*>(p + at), v);
                });
            }
        }
        __threadfence();                                          // the partial sum is in place before the count says so
        __syncwarp();
        int before = -1;
        if (valid && gl == 0) before = atomicAdd(a.arrived + (int64_t)ch.heavy * DG_FINISH_TILES + blockIdx.y, 1);
        before = __shfl_sync(0xffffffffu, before, 0, LPR);
        if (!valid || before != ch.nchunks - 1) return;
        __threadfence();
        if (gl == 0) a.arrived[(int64_t)ch.heavy * DG_FINISH_TILES + blockIdx.y] = 0;
        begin_row(ch.row, add_first);
        const float* sp = a.scratch + (int64_t)ch.slot0 * a.lds + (int64_t)vec0 * VEC;
#pragma unroll
        for (int t = 0; t < TPL; ++t) {
            if (!on[t]) continue;
            const float* p = sp + t * LPR * VEC;
#pragma unroll 4
            for (int s = 0; s < ch.nchunks; ++s) {
                const float* ps = p + s * a.lds;
                each_piece<VEC>([&](int at) { add(acc[t] + at, __ldcg(reinterpret_cast<const piece_t<VEC>*>(ps + at))); });
            }
        }
        if constexpr (MODE == kTiled) {
            const int2 part = a.parts[ch.heavy];
            const float4* p = a.part_area + ((int64_t)(part.x >> 7) * a.part_ld4 + vec0 * (VEC / 4)) * 128 + (part.x & 127);
            for (int s = 0; s < part.y; ++s, p += a.part_ld4 * 128)
#pragma unroll
                for (int t = 0; t < TPL; ++t) {
                    if (!on[t]) continue;
                    each_piece<VEC>([&](int at) { add(acc[t] + at, __ldcg(p + (t * LPR * (VEC / 4) + at / 4) * 128)); });
                }
        }
        store_row(ch.row);
    };
    if constexpr (MODE == kTiled) {
        if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) a.tile_words[DG_LARGEST_ELEMENT] = 0;      // for the next product
        if ((int)blockIdx.x < chunk_ctas && __ldcg(a.tile_words + DG_GATHER_ALL) != 0) return;
    }
    if constexpr (MODE == kWhole) {
        if (__ldcg(a.tile_words + DG_GATHER_ALL) == 0) return;
        for (int id0 = blockIdx.x * NG; id0 < a.n_chunks; id0 += chunk_ctas * NG) run_chunks(id0);
        return;
    }
    if ((int)blockIdx.x < chunk_ctas) {
        run_chunks(blockIdx.x * NG);
        return;
    }

    constexpr int kClasses = 24;
    __shared__ int64_t first[257];                                // row offsets of the window
    __shared__ uint8_t order[256];                                // its light rows, longest class first
    __shared__ int count[kClasses], start[kClasses + 1], next;
    const int32_t row0 = ((int)blockIdx.x - chunk_ctas) * a.rows_per_cta;
    const int nrows = min(a.rows_per_cta, a.m - row0);
    // An empty row of a product that is added to C stays as it is, neither read nor written: three fifths of the rows of a stage block
    // on power-law graphs (eight 306,129-row blocks into one result, F = 256: 1,819 -> 1,459 us).
    const bool keeps = add_first && a.beta == 1.f && !a.flags;
    if (threadIdx.x < kClasses) count[threadIdx.x] = 0;
    if (threadIdx.x == 0) next = 0;
    for (int i = threadIdx.x; i <= nrows; i += 256) first[i] = __ldg(a.rowptr + row0 + i);
    __syncthreads();
    int cls = -1, place = 0;
    if ((int)threadIdx.x < nrows) {
        const int64_t len = first[threadIdx.x + 1] - first[threadIdx.x];
        if (len <= a.heavy_threshold && (len > 0 || !keeps)) {
            const int s = ((int)len + LPR - 1) / LPR;             // batches of LPR entries: classes 0, 1, 2, 3, 4-5, 6-7, 8-11, ...
            const int rank = s < 4 ? s : 2 * (31 - __clz(s)) + ((s >> (30 - __clz(s))) & 1);
            cls = kClasses - 1 - min(rank, kClasses - 1);
            place = atomicAdd(&count[cls], 1);
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int n = threadIdx.x < kClasses ? count[threadIdx.x] : 0, sum = n;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, sum, off);
            if ((int)threadIdx.x >= off) sum += o;
        }
        if (threadIdx.x <= kClasses) start[threadIdx.x] = sum - n;
    }
    __syncthreads();
    if (cls >= 0) order[start[cls] + place] = (uint8_t)threadIdx.x;
    __syncthreads();
    if (a.check && failed == a.check) return;
    const int total = start[kClasses];

    int r = -1, c = 0;
    float v = 0.f;
    auto take = [&] {                                             // the next G rows, one per group, and their first entries
        int b = 0;
        if ((threadIdx.x & 31) == 0) b = atomicAdd(&next, G);
        b = __shfl_sync(0xffffffffu, b, 0);
        r = -1; c = 0; v = 0.f;
        if (b + grp < total) {
            r = order[b + grp];
            const int64_t e = first[r] + gl;
            if (e < first[r + 1]) {
                c = __ldcs(a.col + e);
                v = __ldcs(a.val + e);
            }
        }
        return b < total;
    };
    bool more = take();
    while (more) {
        const int cur = r, cur_c = c;
        const float cur_v = v;
        more = take();
        const bool valid = cur >= 0;
        begin_row(row0 + cur, add_first && valid);
        const int64_t e = valid ? first[cur] : 0;
        gather(a.col, a.val, e + gl, valid ? (int)(first[cur + 1] - e) : 0, cur_c, cur_v);
        if (valid) store_row(row0 + cur);
    }
}

template <int VEC, int LPR, int TPL, int U, int MINB, bool PADDED, bool TILES = VEC >= 4>
int launch(const SpmmArgs& args, const SpmmArgs* whole, cudaStream_t stream)
{
    constexpr int NG = 256 / LPR, tile = LPR * TPL;
    SpmmArgs a = args;
    const int chunk_ctas = (a.n_chunks + NG - 1) / NG;
    const int64_t row_ctas = ((int64_t)a.m + a.rows_per_cta - 1) / a.rows_per_cta;
    for (; a.vec_first < a.vec_end; a.vec_first += tile * DG_FINISH_TILES) {
        const dim3 grid((unsigned)(chunk_ctas + row_ctas), (unsigned)std::min((a.vec_end - a.vec_first + tile - 1) / tile, DG_FINISH_TILES));
        if (!whole) k_spmm<VEC, LPR, TPL, U, MINB, PADDED, kPlain><<<grid, 256, 0, stream>>>(a, chunk_ctas);
        g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
        if constexpr (TILES) {
            if (!whole) continue;
            k_spmm<VEC, LPR, TPL, U, MINB, PADDED, kTiled><<<grid, 256, 0, stream>>>(a, chunk_ctas);
            SpmmArgs w = *whole;
            w.vec_first = a.vec_first;
            w.vec_end = a.vec_end;
            const int ctas = std::min((w.n_chunks + NG - 1) / NG, 148 * 4);
            k_spmm<VEC, LPR, TPL, U, MINB, PADDED, kWhole><<<dim3((unsigned)ctas, grid.y), 256, 0, stream>>>(w, ctas);
            g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
        }
    }
    return (int)cudaGetLastError();
}

// Lanes per item and gathers in flight by the number of vectors in a row and the size of the matrix.  Whole tiles of 64
// float4 first; what is left behind them takes launches of its own, 32 vectors and then up to 32 more, unless it fills most
// of a tile (115 M entries, F = 604: 18.4 -> 16.6 ms).
// Large matrices (from 4 M entries) run best with half the lanes and twice the vectors each: two (or four) rows are in flight
// per warp, a gather is several independent loads, and index traffic and shuffles are shared by more of them; small ones
// have too few rows for that and want a row spread over more lanes.  us per product, this form against twice the lanes:
//   F = 256: 1 M nodes / 17 M entries 1,545 -> 1,296, 2.4 M / 126 M 9,850 -> 8,640; 10,000 nodes / 210 k entries 27 -> 41 (not taken)
//   F = 100: 936 -> 717, 5,540 -> 4,350, 150 k nodes / 2.6 M entries 131 -> 115; F = 48: 470 -> 389, 2,750 -> 2,250
// Where rows are whole, aligned 32-byte pieces (`octets`) the wide form reads those: half the load instructions, with 24 warps
// instead of 32 (F = 256: 2.4 M / 126 M with tiles 7,810 -> 7,550, 1 M / 17 M 1,291 -> 1,274, 300 k / 15 M 876 -> 855; F = 512: 2,860 -> 2,800).
// Small matrices, wide rows: three gathers in flight (with four, 72 bytes of spills: eight 306 k-row stage blocks 1,459 -> 1,409,
// 150 k / 2.6 M F = 256 204 -> 197, F = 200 197 -> 190).
// 65 to 96 floats, from 4 M entries: 8 lanes of three vectors, of which at most 7 idle (16 x 2: up to 15).  1 M / 17 M F = 96 675 -> 618, F = 68
// 655 -> 583, 600 k / 21 M 676 -> 622, 2.4 M / 126 M 4,190 -> 3,920, 300 k / 15 M 471 -> 447, 2.4 M / 42 M 1,727 -> 1,727 (F = 68 1,668 -> 1,631); 150 k / 2.6 M
// 111 -> 119 (not taken).  Not taken either beside tiles in windows of 64 rows, which leave too few rows for four groups a warp (200 k / 10 M F = 96
// 308 -> 325, F = 68 297 -> 306; windows of 128: 300 k / 12 M F = 96 388 -> 387, F = 68 377 -> 364), nor for short rows out of DRAM, read as they
// are: fewer than eight entries a row and an operand of four times the L2 (2.4 M / 16 M F = 96 1,009 -> 1,108, 4 M / 20 M 1,475 -> 1,615;
// 2.4 M / 22 M 1,189 -> 1,094, 1.5 M / 7.5 M 540 -> 516, padded F = 65 2.4 M / 12 M 1,081 -> 1,033).
// 33 to 48 floats, from 4 M entries, or from 1 M with 64 k rows or more where the operand is read as it is, without tiles: 4 lanes of
// three, eight rows a warp, as long as the L2 holds the operand, or three eighths of it where rows straddle sectors.  F = 48: 200 k rows / 10 M
// 223 -> 184, 250 k / 8 M 199 -> 170, 30 k / 8 M 161 -> 149, 250 k / 1.4 M 78 -> 70, 80 k / 1.2 M 53 -> 52, 600 k / 21 M (115 MB) 394 -> 393;
// padded from 41: 200 k / 10 M 232 -> 214, 30 k / 8 M 168 -> 165.  Not taken: 30 k / 3 M 70 -> 72, 30 k / 1.1 M 35 -> 46 (too few rows for so many
// groups); padded 80 k / 1.2 M 62 -> 66; F = 44 300 k / 15 M (53 MB) 320 -> 324; 1.5 M / 62 M (288 MB) 1,125 -> 1,190; with tiles 306 k / 16 M 303 -> 310.
constexpr int64_t kL2Bytes = (int64_t)126 << 20;
template <int VEC, bool PADDED>
int launch_vec(SpmmArgs a, const SpmmArgs* whole, int64_t nnz, int32_t k, bool octets, cudaStream_t stream)
{
    const bool large = nnz >= (int64_t)4 << 20, small = nnz < (int64_t)1 << 20;
    const int end = a.vec_end, wide = end % 64 > 48 ? end : end / 64 * 64;
    int rc = DG_OK;
    if (wide > 0) {
        a.vec_end = wide;
        if constexpr (VEC == 4 && !PADDED) {
            if (large && octets) {
                SpmmArgs o = a;
                o.vec_end = wide / 2;
                rc = launch<8, 16, 2, 2, 3, PADDED>(o, whole, stream);
                a.vec_first = wide;
            }
        }
        if (a.vec_first == 0) rc = large ? launch<VEC, 16, 4, 2, 4, PADDED>(a, whole, stream) : launch<VEC, 32, 2, VEC == 4 ? 3 : 4, 4, PADDED>(a, whole, stream);
        a.vec_first = wide;
    }
    while (rc == DG_OK && a.vec_first < end) {
        a.vec_end = std::min(end, a.vec_first + 32);
        const int nvec = a.vec_end - a.vec_first;
        bool thirds = false;
        if constexpr (VEC == 4) {
            const bool many = large || (!small && !PADDED && a.m >= 1 << 16);
            if (nvec > 8 && nvec <= 12 && many && !whole && k * a.ldb * 4 <= (a.ldb % 8 ? kL2Bytes * 3 / 8 : kL2Bytes)) {
                rc = launch<VEC, 4, 3, 4, 4, PADDED, false>(a, nullptr, stream);
                thirds = true;
            } else if (nvec > 16 && nvec <= 24 && large && !(whole && a.rows_per_cta < 128) &&
                       (PADDED || nnz >= 8 * (int64_t)a.m || k * a.ldb <= kL2Bytes)) {
                rc = launch<VEC, 8, 3, 4, 3, PADDED>(a, whole, stream);
                thirds = true;
            }
        }
        if (thirds) {}
        else if (nvec <= 4) rc = launch<VEC, 4, 1, 4, 5, PADDED>(a, whole, stream);
        else if (nvec <= 8) rc = launch<VEC, 8, 1, 8, 4, PADDED>(a, whole, stream);
        else if (nvec <= 16) rc = large ? launch<VEC, 8, 2, 8, 3, PADDED>(a, whole, stream) : launch<VEC, 16, 1, 4, 5, PADDED>(a, whole, stream);
        else rc = small ? launch<VEC, 32, 1, 4, 5, PADDED>(a, whole, stream) : launch<VEC, 16, 2, 4, 4, PADDED>(a, whole, stream);
        a.vec_first = a.vec_end;
    }
    return rc;
}

bool aligned(const void* p, size_t bytes) { return (reinterpret_cast<uintptr_t>(p) % bytes) == 0; }

// Floats of scratch behind the partial sums for a padded copy of the operand, 0 where none is made.  The copy costs a pass
// over B and pays where its rows are gathered several times: 200,003 nodes, 10.2 M entries, F = 41: 336 -> 235 us.
int64_t pad_floats(const dg_plan* plan, int32_t F)
{
    return !plan->no_padded_copy && F % 4 && F > 4 && plan->nnz >= 4 * (int64_t)plan->k ? (int64_t)plan->k * ((F + 3) / 4 * 4) : 0;
}

// Floats of scratch behind those for the tensor-core part, 0 where it is not used: the tiles hold these very values.
int64_t tile_floats(const dg_plan* plan, const float* val, int32_t F)
{
    return plan->tiles && (!val || plan->tiles->val == val) ? dg_tiles_scratch_floats(plan, F) : 0;
}

int64_t partial_floats(const dg_plan* plan, int32_t F) { return (int64_t)plan->n_chunks * ((F + 3) / 4 * 4); }

}  // namespace

int dg_check_spmm_args(const dg_plan* plan, const float* val, const float* B, int64_t ldb, const float* C, int64_t ldc,
                       int32_t F, uint32_t flags, const float* row_scale, const float* bias)
{
    if (!plan) return DG_ERR_NULL;
    if (F < 0 || ldb < F || ldc < F) return DG_ERR_DIMS;
    if (flags & ~(DG_EPI_ROW_SCALE | DG_EPI_BIAS | DG_EPI_RELU)) return DG_ERR_UNSUPPORTED;
    if (plan->m > 0 && F > 0 && !C) return DG_ERR_NULL;
    if (plan->nnz > 0 && F > 0 && (!val || !B)) return DG_ERR_NULL;
    if ((flags & DG_EPI_ROW_SCALE) && !row_scale) return DG_ERR_NULL;
    if ((flags & DG_EPI_BIAS) && !bias) return DG_ERR_NULL;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != plan->device) return DG_ERR_STATE;
    return DG_OK;
}

int dg_spmm_launch_rows(const dg_plan* plan, const float* val, const float* B, int64_t ldb, float* C, int64_t ldc,
                        int32_t F, float alpha, float beta, uint32_t flags, const float* row_scale, const float* bias,
                        float* scratch, int64_t scratch_floats, cudaStream_t stream, int check, bool split)
{
    if (plan->m == 0 || F == 0) return DG_OK;
    SpmmArgs a{};
    a.check = check; a.failed_check = plan->status + 1;
    a.rowptr = plan->rowptr; a.col = plan->col; a.val = val; a.B = B; a.C = C;
    a.row_scale = row_scale; a.bias = bias; a.chunks = plan->chunks; a.arrived = plan->arrived; a.scratch = scratch;
    a.chunk_col = plan->col; a.chunk_val = val;
    a.ldb = ldb; a.ldc = ldc; a.lds = F; a.m = plan->m; a.F = F;
    a.heavy_threshold = split ? plan->heavy_threshold : INT32_MAX; a.n_chunks = split ? plan->n_chunks : 0;
    // Rows per CTA: as wide a window as still makes 2,000 of them, 13 for each of the B200's 148 SMs (wider windows sort better and
    // share their offsets; 64 rows are best at 150 k rows, 128 at 300 k, 256 from 1 M).
    a.rows_per_cta = 32;
    while (a.rows_per_cta < 256 && (int64_t)a.rows_per_cta * 2 * 2000 <= plan->m) a.rows_per_cta *= 2;
    a.alpha = alpha; a.beta = beta; a.flags = flags;
    // widest vector the shapes and addresses allow (B may be NULL only when there is nothing to gather)
    int vec = 1;
    if (F % 4 == 0 && ldb % 4 == 0 && ldc % 4 == 0 && aligned(B, 16) && aligned(C, 16)) vec = 4;
    else if (F % 2 == 0 && ldb % 2 == 0 && ldc % 2 == 0 && aligned(B, 8) && aligned(C, 8)) vec = 2;
    const int64_t copy = pad_floats(plan, F), sums = partial_floats(plan, F), tiled = tile_floats(plan, val, F);
    const bool padded = vec < 4 && copy > 0 && sums + copy <= scratch_floats && aligned(scratch, 16);
    SpmmArgs whole;
    const bool tiles = tiled > 0 && (vec == 4 || padded) && sums + copy + tiled <= scratch_floats && aligned(scratch, 16);
    if (tiles) {
        float* area = scratch + sums + copy;
        int launches = 0;
        const int rc = dg_tiles_launch(plan, B, ldb, F, area, stream, &launches, dg::kWaitLimit);
        if (rc) return rc;
        g_kernel_launches.fetch_add(launches, std::memory_order_relaxed);
        const dg_tiles* t = plan->tiles;
        a.tile_words = plan->status + DG_TILE_WORDS;
        a.chunks = t->rest_chunks; a.n_chunks = t->n_rest_chunks; a.chunk_col = t->rest_col; a.chunk_val = t->rest_val;
        a.parts = t->parts; a.part_area = reinterpret_cast<const float4*>(area); a.part_ld4 = (F + 3) / 4;
    }
    if (padded) {
        float* wide = scratch + sums;
        const int64_t ld = (F + 3) / 4 * 4;
        const int rc = dg_pad_rows(B, ldb, plan->k, F, wide, ld, stream);
        if (rc) return rc;
        g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
        a.B = wide; a.ldb = ld; a.lds = ld;
    }
    a.vec_end = padded ? (int32_t)(a.ldb / 4) : F / vec;
    if (tiles) {                                                  // the same product without them
        whole = a;
        whole.chunks = plan->chunks; whole.n_chunks = plan->n_chunks; whole.chunk_col = plan->col; whole.chunk_val = val;
        whole.parts = nullptr;
    }
    const SpmmArgs* w = tiles ? &whole : nullptr;
    if (padded) return launch_vec<4, true>(a, w, plan->nnz, plan->k, false, stream);
    switch (vec) {
        case 4: return launch_vec<4, false>(a, w, plan->nnz, plan->k, F % 8 == 0 && ldb % 8 == 0 && aligned(B, 32), stream);
        case 2: return launch_vec<2, false>(a, w, plan->nnz, plan->k, false, stream);
        default: return launch_vec<1, false>(a, w, plan->nnz, plan->k, false, stream);
    }
}

// Picks the kernel family (streaming when the operands allow it, row kernels otherwise) and brackets the product with
// profile events while a profile is open.
int dg_spmm_launch(const dg_plan* plan, const float* val, const float* B, int64_t ldb, float* C, int64_t ldc,
                   int32_t F, float alpha, float beta, uint32_t flags, const float* row_scale, const float* bias,
                   float* scratch, int64_t scratch_floats, cudaStream_t stream, int check)
{
    if (plan->m == 0 || F == 0) return DG_OK;
    bool profiled = false;
    {
        std::lock_guard<std::mutex> lock(g_profile.mu);
        if (g_profile.open) {
            profiled = profile_event(stream) != nullptr;
            const double rw = 4.0 * F * plan->m * (beta != 0.f ? 2.0 : 1.0), csr = 8.0 * plan->nnz + 4.0 * (plan->m + 1.0);
            g_profile.alg_bytes += csr + 4.0 * F * plan->touched_columns + rw;
            g_profile.gather_bytes += csr + 4.0 * F * plan->nnz + rw;
            g_profile.flops += 2.0 * plan->nnz * F;
            g_profile.products += 1;
        }
    }
    int rc;
    if (dg_spmm_stream_eligible(plan, B, ldb, C, ldc, F)) {
        int launches = 0;
        rc = dg_spmm_stream_launch(plan, val, B, ldb, C, ldc, F, alpha, beta, flags, row_scale, bias, scratch, stream, &launches);
        g_kernel_launches.fetch_add(launches, std::memory_order_relaxed);
    } else {
        rc = dg_spmm_launch_rows(plan, val, B, ldb, C, ldc, F, alpha, beta, flags, row_scale, bias, scratch, scratch_floats, stream, check);
    }
    if (profiled) {
        std::lock_guard<std::mutex> lock(g_profile.mu);
        profile_event(stream);
    }
    return rc;
}

extern "C" int dg_profile_begin(void)
try {
    std::lock_guard<std::mutex> lock(g_profile.mu);
    g_profile.open = true;
    g_profile.used = 0;
    g_profile.alg_bytes = g_profile.gather_bytes = g_profile.flops = 0;
    g_profile.products = 0;
    g_kernel_launches.store(0);
    return DG_OK;
} catch (...) {
    return dg_exception();
}

extern "C" int dg_profile_end(dg_profile* out)
try {
    if (!out) return DG_ERR_NULL;
    std::lock_guard<std::mutex> lock(g_profile.mu);
    g_profile.open = false;
    DG_CUDA(cudaDeviceSynchronize());
    double ms = 0;
    for (size_t i = 0; i + 1 < g_profile.used; i += 2) {
        float t = 0.f;
        DG_CUDA(cudaEventElapsedTime(&t, g_profile.events[i], g_profile.events[i + 1]));
        ms += t;
    }
    *out = dg_profile{ms, g_profile.alg_bytes, g_profile.gather_bytes, g_profile.flops, g_profile.products,
                      g_kernel_launches.load()};
    g_profile.used = 0;
    return DG_OK;
} catch (...) {
    return dg_exception();
}

// Grows the plan's scratch to what a product of width F may need (either kernel family); allocates and synchronises
// `stream` only when it has to grow.  The stage loops call it for every plan before they enqueue anything, so that an
// allocation failure cannot leave a loop half issued.  Only the partial sums of the split rows are indispensable: a plan that cannot have
// more goes on without its tiles, and then without padded copies, for good (asking again would stall every product).
int dg_spmm_prepare(const dg_plan* plan, int32_t F, cudaStream_t stream)
{
    if (!plan) return DG_ERR_NULL;
    dg_plan* p = const_cast<dg_plan*>(plan);
    if (dg_stream_selected()) {
        const int rc = dg_plan_ensure_tasks(p, stream);
        if (rc) return rc;
    }
    for (;;) {
        const int64_t rows = partial_floats(plan, F) + pad_floats(plan, F) + tile_floats(plan, nullptr, F), tasks = dg_stream_selected() ? 2 * (int64_t)plan->n_tasks * F : 0;
        const int64_t need = rows > tasks ? rows : tasks;
        if (need <= p->scratch_floats) return DG_OK;
        DG_CUDA(cudaStreamSynchronize(stream));
        dg_pool_free(p->scratch);
        p->scratch = nullptr;
        p->scratch_floats = 0;
        const int rc = dg_pool_alloc((void**)&p->scratch, (size_t)need * sizeof(float));
        if (rc == DG_OK) p->scratch_floats = need;
        if (rc != (int)cudaErrorMemoryAllocation) return rc;
        if (tile_floats(plan, nullptr, F) > 0) {
            dg_tiles_free(p->tiles);
            p->tiles = nullptr;
        } else if (pad_floats(plan, F) > 0) {
            p->no_padded_copy = true;
        } else {
            return rc;
        }
    }
}

extern "C" int dg_spmm_csr(const dg_plan* plan, const float* val, const float* B, int64_t ldb, float* C, int64_t ldc,
                           int32_t F, float alpha, float beta, uint32_t flags, const float* row_scale,
                           const float* bias, void* stream)
try {
    int rc = dg_check_spmm_args(plan, val, B, ldb, C, ldc, F, flags, row_scale, bias);
    if (rc) return rc;
    if ((rc = dg_spmm_prepare(plan, F, (cudaStream_t)stream))) return rc;      // first use at this width may grow the scratch
    return dg_spmm_launch(plan, val, B, ldb, C, ldc, F, alpha, beta, flags, row_scale, bias, plan->scratch, plan->scratch_floats,
                          (cudaStream_t)stream);
} catch (...) {
    return dg_exception();
}

extern "C" int dg_spmm_coo(const int32_t* row, const int32_t* col, const float* val, int64_t nnz, int32_t m, int32_t k,
                           const float* B, float* C, int32_t F, float alpha, float beta, void* stream)
try {
    dg_plan* plan = nullptr;
    int rc = dg_plan_build_lean(row, col, nnz, m, k, stream, &plan);
    if (rc) return rc;
    rc = dg_spmm_csr(plan, val, B, F, C, F, F, alpha, beta, 0u, nullptr, nullptr, stream);
    if (rc == DG_OK) rc = (int)cudaStreamSynchronize((cudaStream_t)stream);   // the plan's buffers die below
    dg_plan_destroy(plan);
    return rc;
} catch (...) {
    return dg_exception();
}

extern "C" const char* dg_strerror(int code)
{
    switch (code) {
        case DG_OK: return "ok";
        case DG_ERR_NULL: return "a required pointer is NULL";
        case DG_ERR_DIMS: return "negative or inconsistent sizes";
        case DG_ERR_INDEX: return "sparse indices are not row-sorted or fall outside the matrix";
        case DG_ERR_UNSUPPORTED: return "unsupported request";
        case DG_ERR_STATE: return "object used in the wrong state or on the wrong device";
        case DG_ERR_SCRATCH: return "request exceeds the fixed scratch capacity";
        default: break;
    }
    if (code >= DG_NCCL_ERROR_BASE) return "NCCL error (code - 10000 is the ncclResult_t)";
    if (code > 0) return cudaGetErrorString((cudaError_t)code);
    return "unknown error";
}

extern "C" int dg_version(void) { return 100; }
