// Dense tiles: the hub x hub corner of a power-law block on the tensor cores.
//
// A gather moves 4 F bytes from the L2 to an SM for every entry, 64 bytes a clock at best, which is what bounds k_spmm on large
// blocks (16 clocks an entry at F = 256).  Sorted by length and by frequency, the split rows and the frequent columns of a
// power-law graph meet in tiles that are 5 to 90 % full: one row of B serves several rows of such a tile, and multiplying
// the whole 128 x 32 tile, zeros included, costs the SM as much as gathering some 160 of its entries.  So tiles
// with more than that (kTileMin) are multiplied as dense matrices and the rest of the split rows is gathered as before.
//
// fp32 in and out: every value and every element of B is cut into three bf16 pieces (8 + 8 + 8 bits, which is all of an fp32
// number), and six tcgen05.mma kind::f16 passes add the products of pieces down to 2^-16, dropping 2^-24 and below:
// high x high into one fp32 accumulator, the five small ones into another.  The tensor cores truncate when they add into
// an accumulator, so after kFlushSlabs tiles (512 columns, 32 additions) both are added, rounded to nearest, into the partial
// result and restarted.  Measured against float64 on the dense graph: 1.8e-7 relative; the gather alone is at the same level.
//
// Per product: k_tile_columns gathers the frequent columns' rows of B, splits and transposes them into the layout
// the tensor cores read (K-major, no swizzle, 8 x 16-byte core matrices); k_tile_mma runs one CTA per SM over its share of
// the tiles: a warp fetches the 32-column slab of B with one bulk copy, two groups of four warps clear the A tile and
// scatter its records into it in turn, one thread issues the MMAs, and the groups drain the accumulators.  Partial results of a
// row tile that several CTAs share are added by k_spmm where it finishes the row.
// Measured (B200): 232,965 nodes / 115 M entries, 64 % of the entries in 91,000 tiles: F = 256 6.18 -> 3.3 ms, F = 604
// 16.6 -> 8.9 ms; 306,128 nodes / 15.8 M entries, F = 256: 1.03 -> 0.84 ms.  The tensor pipe is busy for 55 to 59 % of k_tile_mma's
// time, the rest is waiting for a tile to be filled after an accumulator was drained.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <new>
#include <utility>
#include "dg_build.h"
#include "dg_tiles.h"
#include "dg_umma.h"

namespace {

using namespace dg;

constexpr int kTileRows = 128, kTileCols = 32;
constexpr int kTileElems = kTileRows * kTileCols;
constexpr int kTileMin = 160;             // entries from which a tile is worth multiplying
constexpr int kMaxColumns = 1 << 16;      // frequent columns considered, at most
constexpr float kTileBound = 9.2233720e18f;     // 2^63: a product of two smaller numbers is finite, with a factor of 4 to spare for sums
// The small pieces of numbers far below this fall under the smallest bf16 and the products under the smallest fp32: an operand, or a
// product of value and operand, that is nowhere larger loses bits (error against float64, whole operand at 2^-110 1.2e-7, at 2^-115
// 9e-7, at 2^-120 2.8e-5; gathered 1.5e-7).  Small elements beside larger ones do no harm.
constexpr float kTileLeast = 7.8886091e-31f;    // 2^-100
// `largest`: bits of the largest magnitude, ordered as the numbers are with infinities and NaN above them
__device__ __forceinline__ bool unfit_operand(int largest, float least)
{
    return largest >= __float_as_int(kTileBound) || (largest > 0 && largest < __float_as_int(least));
}
constexpr int kFlushSlabs = 16;
constexpr int kTileStages = 3;
constexpr int kValueWarps = 4;            // of every CTA, to see whether the values are still those of the tiles
constexpr int kScatterThreads = 256, kGroupThreads = 128, kTileThreads = kScatterThreads + 64 + 32 * kValueWarps;
constexpr int kAhead = 8;                 // records a thread holds for its group's next tile
constexpr int T = 256;

// Where element (r, c) of a tile lies: core matrices of 8 rows x 8 columns (128 bytes), rows of cores first.
__host__ __device__ __forceinline__ int tile_element(int r, int c) { return (c >> 3) * (kTileRows * 8) + (r >> 3) * 64 + (r & 7) * 8 + (c & 7); }

__device__ __forceinline__ uint32_t bf16_bits(float x)
{
    uint32_t r;
    asm("{\n\t.reg .b16 h;\n\tcvt.rn.bf16.f32 h, %1;\n\tcvt.u32.u16 %0, h;\n\t}" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void split3(float x, uint32_t& h, uint32_t& m, uint32_t& l)
{
    h = bf16_bits(x);
    const float rest = x - __uint_as_float(h << 16);
    m = bf16_bits(rest);
    l = bf16_bits(rest - __uint_as_float(m << 16));
}
// Shared-memory matrix descriptor, K-major without swizzle: `lbo` bytes between core matrices along K, `sbo` along M / N.
__device__ __forceinline__ uint64_t umma_desc_plain(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// What a warp remembers of its share of the values, in fours: the sum modulo 2^64 of products of pairs, every value shifted by a key
// that depends on its place, and the plain sum modulo 2^32.  One changed value always shows (in the second sum where its partner
// is zero), several do but for one chance in some 2^32 a share.  Nine instructions for four values: hashing every one by itself
// cost the MMAs beside it twice as much.
struct ValueSum {
    unsigned long long pairs;
    uint32_t plain, pad;
};
__device__ __forceinline__ void add_values(ValueSum& sum, uint4 x, uint32_t at)
{
    const uint32_t key = at * 0x9E3779B1u, a = x.x + key, b = x.y + key + 0x85EBCA6Bu, c = x.z + key + 0xC2B2AE35u, d = x.w + key + 0x27D4EB2Fu;
    sum.pairs += (unsigned long long)a * b;
    sum.pairs += (unsigned long long)c * d;
    sum.plain += a + b + c + d;
}
__device__ __forceinline__ ValueSum value_sum(const float* __restrict__ val, int64_t nnz, int share, int shares)
{
    const int lane = threadIdx.x & 31;
    const int64_t fours = (nnz + 3) / 4, per = (fours + shares - 1) / shares, end = min(fours, (share + 1) * per);
    int64_t i = min(fours, share * per);
    ValueSum sum{};
    if ((reinterpret_cast<uintptr_t>(val) & 15) == 0) {
        constexpr int kInFlight = 8;
        for (; i + 32 * kInFlight <= min(end, nnz / 4); i += 32 * kInFlight) {
            uint4 x[kInFlight];
#pragma unroll
            for (int j = 0; j < kInFlight; ++j) x[j] = __ldcs(reinterpret_cast<const uint4*>(val) + i + j * 32 + lane);
#pragma unroll
            for (int j = 0; j < kInFlight; ++j) add_values(sum, x[j], (uint32_t)i + j * 32 + lane);
        }
    }
    for (i += lane; i < end; i += 32) {
        uint32_t x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = 4 * i + j < nnz ? __float_as_uint(__ldcs(val + 4 * i + j)) : 0u;
        add_values(sum, make_uint4(x[0], x[1], x[2], x[3]), (uint32_t)i);
    }
    for (int off = 16; off > 0; off >>= 1) {
        sum.pairs += __shfl_xor_sync(0xffffffffu, sum.pairs, off);
        sum.plain += __shfl_xor_sync(0xffffffffu, sum.plain, off);
    }
    return sum;
}
__global__ void __launch_bounds__(32 * kValueWarps) k_value_sums(const float* __restrict__ val, int64_t nnz, ValueSum* __restrict__ sums)
{
    const int share = blockIdx.x * kValueWarps + (threadIdx.x >> 5);
    const ValueSum sum = value_sum(val, nnz, share, gridDim.x * kValueWarps);
    if ((threadIdx.x & 31) == 0) sums[share] = sum;
}

// Slab images of B: [panel][column tile][piece][k octet][n][8] bf16.  One thread makes one 16-byte octet of all three pieces.
__global__ void __launch_bounds__(T) k_tile_columns(const float* __restrict__ B, int64_t ldb, const int32_t* __restrict__ columns, int32_t n_columns,
                                                    int32_t col_tiles, int32_t F, int32_t n_pad, uint16_t* __restrict__ out, int* __restrict__ words)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) words[DG_GATHER_ALL] = 0;
    __shared__ int block_largest;
    if (threadIdx.x == 0) block_largest = 0;
    int largest = 0;
    uint16_t* image = out + ((int64_t)blockIdx.y * col_tiles + blockIdx.x) * 3 * n_pad * kTileCols;
    for (int i = threadIdx.x; i < n_pad * (kTileCols / 8); i += T) {
        const int n = i % n_pad, octet = i / n_pad, f = blockIdx.y * n_pad + n;
        uint32_t h[8], m[8], l[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = blockIdx.x * kTileCols + octet * 8 + j;
            const float x = k < n_columns && f < F ? __ldg(B + (int64_t)__ldg(columns + k) * ldb + f) : 0.f;
            largest = max(largest, __float_as_int(fabsf(x)));
            split3(x, h[j], m[j], l[j]);
        }
        uint4* at = reinterpret_cast<uint4*>(image) + octet * n_pad + n;
        const int piece = n_pad * (kTileCols / 8);
        at[0] = make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
        at[piece] = make_uint4(m[0] | m[1] << 16, m[2] | m[3] << 16, m[4] | m[5] << 16, m[6] | m[7] << 16);
        at[2 * piece] = make_uint4(l[0] | l[1] << 16, l[2] | l[3] << 16, l[4] | l[5] << 16, l[6] | l[7] << 16);
    }
    largest = __reduce_max_sync(0xffffffffu, largest);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) atomicMax(&block_largest, largest);
    __syncthreads();
    if (threadIdx.x == 0 && block_largest > __ldcg(words + DG_LARGEST_ELEMENT)) atomicMax(words + DG_LARGEST_ELEMENT, block_largest);
}

struct TileArgs {
    const dg_slab* slabs;
    const dg_segment* segments;
    const int32_t* cta_segment;
    const uint2* records;
    const uint16_t* images;
    float4* partial;                      // [slot][ld4][128]
    int32_t ld4, F4, n_pad, col_tiles;    // 16-byte pieces of a partial row; of those, how many are wanted
    int *status, *device_status;          // the plan's word and the device's
    float least;                          // an operand without any element of this size is too small
    int* words;                           // dg_plan::status + DG_TILE_WORDS
    int wait_limit;                       // polls of a wait
    const float* val;                     // the matrix's values, nnz of them, and what the tiles remember of them
    const ValueSum* value_sums;
    int64_t nnz;
};

// blockIdx.x: the CTA's share of the tiles, blockIdx.y: panel of n_pad columns.  Warps 0-3 and 4-7: the two scatter groups
// (group g fills tiles g, g + 2, ... and drains the 16-column pieces g, g + 2, ... of the accumulators), 8: copies, 9: MMA issue, the
// others see whether the values are still those of the tiles (beside the MMAs, which leave DRAM alone: 504 MB, F = 256 548 -> 579 us,
// F = 48 321 -> 338; the pass alone would be 77 us.  Half as many warps: 30 to 60 us longer where the tiles are few).
//
// A group drains a finished run of tiles two or three tiles after its end, so that the tiles of the next run are being
// filled meanwhile.  Why nothing deadlocks: filling tile t waits for the MMAs of tile t - 3 (its stage), those of t - 3 wait
// only for drains of runs that end before t - 3, and both groups drain such a run by the time they have filled tile t - 1
// (group of t - 2: runs up to t - 4 after filling it, the other likewise).  No phase bit is ambiguous: a group that waits
// for tile t - 3 has already waited for t - 5, so the phase before the awaited one (t - 6) is complete.
__global__ void __launch_bounds__(kTileThreads, 1) k_tile_mma(const TileArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 127u) & ~127u;
    unsigned char* gbase = smem_raw + (base - raw);
    const int n = a.n_pad;
    const uint32_t b_piece = (uint32_t)n * kTileCols * 2, b_bytes = 3 * b_piece;
    constexpr uint32_t a_piece = kTileElems * 2, a_bytes = 3 * a_piece;
    const uint32_t stage_bytes = a_bytes + b_bytes, bars = base + kTileStages * stage_bytes;
    const uint32_t full_b = bars, ready_a = bars + 8 * kTileStages, empty = bars + 16 * kTileStages, acc_full = bars + 24 * kTileStages,
                   acc_empty = acc_full + 8, done = acc_full + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + kTileStages * stage_bytes + 24 * kTileStages + 24);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kTileStages; ++s) {
            mbar_init(full_b + 8 * s, 1);
            mbar_init(ready_a + 8 * s, 4);
            mbar_init(empty + 8 * s, 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 8);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot, acc_small = tmem + 256;
    bool ok = true;

    const bool unfit = unfit_operand(__ldcg(a.words + DG_LARGEST_ELEMENT), a.least);   // the whole product will be gathered: no tiles for anybody
    if (unfit && threadIdx.x == 0) a.words[DG_GATHER_ALL] = 1;
    const int seg0 = a.cta_segment[blockIdx.x], seg1 = unfit ? seg0 : a.cta_segment[blockIdx.x + 1];
    const int slab0 = seg0 < seg1 ? a.segments[seg0].slab0 : 0, total = seg0 < seg1 ? a.segments[seg1 - 1].slab1 - slab0 : 0;
    const dg_slab* slabs = a.slabs + slab0;

    if (warp == 8) {                                              // copies of B's slabs
        const uint16_t* images = a.images + (int64_t)blockIdx.y * a.col_tiles * 3 * n * kTileCols;
        int next = lane < total ? __ldg(&slabs[lane].col_tile) : 0, cur = 0;
        int t = 0;
        for (; t < total; ++t) {
            const int s = t % kTileStages, u = t / kTileStages;
            if ((t & 31) == 0) {
                cur = next;
                next = t + 32 + lane < total ? __ldg(&slabs[t + 32 + lane].col_tile) : 0;
            }
            const int tile = __shfl_sync(0xffffffffu, cur, t & 31);
            if (u > 0) ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * s, (u - 1) & 1, a.wait_limit));
            if (!ok) break;
            if (lane == 0) {
                mbar_expect_tx(full_b + 8 * s, b_bytes);
                bulk_load(base + s * stage_bytes + a_bytes, images + (int64_t)tile * 3 * n * kTileCols, b_bytes, full_b + 8 * s);
            }
            __syncwarp();
        }
        await_loads(full_b, t, kTileStages);
    } else if (warp == 9) {
        if (lane == 0) {                                          // MMA issue
            // fp32 accumulator, bf16 A and B, both K-major, 128 x n
            const uint32_t idesc = 1u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(n >> 3) << 17 | (uint32_t)(kTileRows >> 4) << 24;
            int t = 0, run = 0;
            for (int seg = seg0; seg < seg1 && ok; ++seg) {
                const int count = a.segments[seg].slab1 - a.segments[seg].slab0;
                for (int i = 0; i < count && ok; ++i, ++t) {
                    const int s = t % kTileStages, u = t / kTileStages, in_run = i % kFlushSlabs;
                    if (in_run == 0 && run > 0) ok = mbar_wait(acc_empty, (run - 1) & 1, a.wait_limit);
                    ok = ok && mbar_wait(full_b + 8 * s, u & 1, a.wait_limit) && mbar_wait(ready_a + 8 * s, u & 1, a.wait_limit);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t A = base + s * stage_bytes, Bs = A + a_bytes;
#pragma unroll
                    for (int k = 0; k < kTileCols / 16; ++k) {    // 16 columns = two octets per MMA
                        const uint32_t ao = k * 2 * kTileRows * 16, bo = k * 2 * n * 16;
                        const uint64_t ah = umma_desc_plain(A + ao, kTileRows * 16, 128), am = umma_desc_plain(A + a_piece + ao, kTileRows * 16, 128),
                                       al = umma_desc_plain(A + 2 * a_piece + ao, kTileRows * 16, 128);
                        const uint64_t bh = umma_desc_plain(Bs + bo, n * 16, 128), bm = umma_desc_plain(Bs + b_piece + bo, n * 16, 128),
                                       bl = umma_desc_plain(Bs + 2 * b_piece + bo, n * 16, 128);
                        const uint32_t add = in_run > 0 || k > 0 ? 1u : 0u;
                        umma_bf16(tmem, ah, bh, idesc, add);
                        umma_bf16(acc_small, ah, bm, idesc, add);
                        umma_bf16(acc_small, am, bh, idesc, 1u);
                        umma_bf16(acc_small, am, bm, idesc, 1u);
                        umma_bf16(acc_small, ah, bl, idesc, 1u);
                        umma_bf16(acc_small, al, bh, idesc, 1u);
                    }
                    umma_commit(empty + 8 * s);
                    if (in_run == kFlushSlabs - 1 || i == count - 1) {
                        umma_commit(acc_full);
                        ++run;
                    }
                }
            }
            await_mmas(done);
        }
    } else if (warp > 9) {
        const int share = blockIdx.x * kValueWarps + warp - 10;
        if (blockIdx.y == 0 && !unfit) {
            const ValueSum sum = value_sum(a.val, a.nnz, share, gridDim.x * kValueWarps), then = a.value_sums[share];
            if (lane == 0 && (sum.pairs != then.pairs || sum.plain != then.plain)) a.words[DG_GATHER_ALL] = 1;
        }
    } else {
        const int group = warp >> 2, q = warp & 3, tid = threadIdx.x & (kGroupThreads - 1);
        int run = 0, seg = seg0, seg_begin = 0, seg_end = seg0 < seg1 ? a.segments[seg0].slab1 - slab0 : 0;
        // Adds the accumulators into the partial result of the segment.  Only this thread ever touches these 16-byte pieces, in
        // program order, so the sum order is fixed; the reduction is sent to L2 and not waited for.
        auto drain = [&](bool first, bool last) {
            ok = __all_sync(0xffffffffu, mbar_wait(acc_full, run & 1, a.wait_limit));      // tcgen05.ld is warp-collective
            ++run;
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int piece0 = blockIdx.y * (n / 4);
            float4* p = a.partial + ((int64_t)a.segments[seg].slot * a.ld4 + piece0) * kTileRows + q * 32 + lane;
            for (int c0 = group * 16; c0 < n; c0 += 32) {
                uint32_t big[16], small[16];
                tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, big);
                tmem_ld16(acc_small + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, small);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (piece0 + c0 / 4 + j >= a.F4) break;
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = __uint_as_float(big[4 * j + e]) + __uint_as_float(small[4 * j + e]);
                    float4* at = p + (int64_t)(c0 / 4 + j) * kTileRows;
                    if (first) __stcg(at, make_float4(v[0], v[1], v[2], v[3]));
                    else asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(at), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty);
            if (last) {
                ++seg;
                seg_begin = seg_end;
                if (seg < seg1) seg_end = a.segments[seg].slab1 - slab0;
            }
        };
        auto drain_if_end = [&](int t) {                          // called for every tile of the CTA once, in order
            if (t < 0 || t >= total || !ok) return;
            const int i = t - seg_begin;
            const bool last = t == seg_end - 1;
            if (last || i % kFlushSlabs == kFlushSlabs - 1) drain(i < kFlushSlabs, last);
        };
        uint2 rec[kAhead];
        int count = 0, first = 0;
        int2 meta = make_int2(0, 0), meta_next = lane < total ? make_int2(__ldg(&slabs[lane].first), __ldg(&slabs[lane].count)) : make_int2(0, 0);
        auto fetch = [&](int t) {                                 // this group's next tile: its first records
            if ((t & 31) < 2) {
                meta = meta_next;
                const int b = (t & ~31) + 32 + lane;
                meta_next = b < total ? make_int2(__ldg(&slabs[b].first), __ldg(&slabs[b].count)) : make_int2(0, 0);
            }
            first = __shfl_sync(0xffffffffu, meta.x, t & 31);
            count = __shfl_sync(0xffffffffu, meta.y, t & 31);
            if (t >= total) count = 0;
#pragma unroll
            for (int e = 0; e < kAhead; ++e)
                if (tid + e * kGroupThreads < count) rec[e] = __ldcs(a.records + first + tid + e * kGroupThreads);
        };
        fetch(group);
        int filled = -1;                                          // the last tile this group filled
        for (int t = group; t < total; t += 2) {                  // no way out of this loop: its barrier wants all four warps
            const int s = t % kTileStages, u = t / kTileStages;
            if (ok && u > 0) ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * s, (u - 1) & 1, a.wait_limit));
            unsigned char* A = gbase + s * stage_bytes;
            if (ok) {
#pragma unroll
                for (int z = 0; z < (int)a_bytes / 16 / kGroupThreads; ++z) reinterpret_cast<uint4*>(A)[tid + z * kGroupThreads] = make_uint4(0, 0, 0, 0);
            }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kGroupThreads) : "memory");
            if (!ok) continue;
            uint16_t* A16 = reinterpret_cast<uint16_t*>(A);
            auto put = [&](uint2 v) {
                const uint32_t pos = v.y >> 16;
                A16[pos] = (uint16_t)v.x;
                A16[kTileElems + pos] = (uint16_t)(v.x >> 16);
                A16[2 * kTileElems + pos] = (uint16_t)v.y;
            };
#pragma unroll
            for (int e = 0; e < kAhead; ++e)
                if (tid + e * kGroupThreads < count) put(rec[e]);
            for (int j0 = tid + kAhead * kGroupThreads; j0 < count; j0 += kAhead * kGroupThreads) {
                uint2 more[kAhead];
#pragma unroll
                for (int e = 0; e < kAhead; ++e)
                    if (j0 + e * kGroupThreads < count) more[e] = __ldcs(a.records + first + j0 + e * kGroupThreads);
#pragma unroll
                for (int e = 0; e < kAhead; ++e)
                    if (j0 + e * kGroupThreads < count) put(more[e]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(ready_a + 8 * s);
            filled = t;
            fetch(t + 2);
            drain_if_end(t - 3);
            drain_if_end(t - 2);
        }
        for (int t = filled >= 0 ? filled - 1 : 0; t < total; ++t) drain_if_end(t);
    }
    if (!ok) {
        atomicExch(a.status, 1);
        atomicExch(a.device_status, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

int panels_of(int32_t F) { return (F + 255) / 256; }
int panel_width(int32_t F) { const int p = panels_of(F); return ((F + p - 1) / p + 15) / 16 * 16; }

}  // namespace

// ---- finding the tiles -----------------------------------------------------------------------------------------------------
// One-off, on the device; the host waits three times, for how many columns are frequent, how many tiles are dense enough and how
// many segments and chunks came of it.  Four passes over the entries of the split rows, one chunk per warp, and a few over the
// lists of rows, columns and tiles in between; what bounds it are the atomics on the counts of hub columns and tiles.  With the
// lists sorted and the tiles chosen on the host, the table of all tiles crossing PCIe twice: 15.8 M entries 7.1 -> 0.9 ms,
// 40.6 M 12 -> 1.9, 115 M (dense) 17 -> 5.2, 126 M 24 -> 8.0, 260 M 57 -> 15: about what one product of 256 columns takes.
namespace {

struct SplitRow { int32_t row, len; };
struct Keyed { int32_t key, id; };

struct Found {                            // what the host waits for
    int32_t columns, least, max_weight;   // frequent columns: how many, from which weight on, the largest
    int32_t slabs, entries, segments, rest_chunks, rest;
    int32_t largest;                      // bits of the largest magnitude among the tiled values
    int32_t unordered;                    // some row's columns do not strictly ascend
    long long cost;                       // of all slabs, in half clocks
};

__global__ void k_split_rows(const dg_chunk* __restrict__ chunks, int32_t n_chunks, const int64_t* __restrict__ rowptr, SplitRow* __restrict__ rows,
                             Keyed* __restrict__ by_length)
{
    const int32_t c = blockIdx.x * T + threadIdx.x;
    if (c >= n_chunks || chunks[c].slot != chunks[c].slot0) return;
    const int32_t r = chunks[c].row, h = chunks[c].heavy, len = (int32_t)min((int64_t)INT32_MAX, rowptr[r + 1] - rowptr[r]);
    rows[h] = SplitRow{r, len};
    by_length[h] = Keyed{len, h};
}

// How many entries of split rows every column holds, and whether a row's columns ascend: an entry that comes twice has one place in a
// tile, so tiles are for rows whose columns strictly ascend, as coalescing leaves them.
__global__ void __launch_bounds__(T) k_column_weights(const dg_chunk* __restrict__ chunks, int32_t n_chunks, const int32_t* __restrict__ col,
                                                      int32_t* __restrict__ weight, Found* __restrict__ found)
{
    const int32_t c = blockIdx.x * (T / 32) + (threadIdx.x >> 5);
    if (c >= n_chunks) return;
    const dg_chunk ch = chunks[c];
    bool ascend = true;
    for (int i = threadIdx.x & 31; i < ch.len; i += 32) {
        const int32_t cc = col[ch.e0 + i];
        if (i > 0 || ch.slot != ch.slot0) ascend = ascend && col[ch.e0 + i - 1] < cc;      // the row's first entry has none before it
        atomicAdd(&weight[cc], 1);
    }
    if (!ascend) found->unordered = 1;
}

constexpr int kWeightBins = 4096;
__global__ void __launch_bounds__(T) k_weight_histogram(const int32_t* __restrict__ weight, int32_t k, int32_t* __restrict__ bins, Found* __restrict__ found)
{
    __shared__ int32_t local[kWeightBins];
    for (int i = threadIdx.x; i < kWeightBins; i += T) local[i] = 0;
    __syncthreads();
    int32_t most = 0;
    for (int32_t i = blockIdx.x * T + threadIdx.x; i < k; i += gridDim.x * T) {
        const int32_t w = weight[i];
        most = max(most, w);
        atomicAdd(&local[min(w, kWeightBins - 1)], 1);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0) atomicMax(&found->max_weight, most);
    __syncthreads();
    for (int i = threadIdx.x; i < kWeightBins; i += T)
        if (local[i]) atomicAdd(&bins[i], local[i]);
}

// Columns of at least that weight in the order of their ids.  PASS 0: how many of every T; 1: the columns.
template <int PASS>
__global__ void __launch_bounds__(T) k_frequent_columns(const int32_t* __restrict__ weight, int32_t k, int32_t least, int32_t* __restrict__ first,
                                                        Keyed* __restrict__ out)
{
    const int32_t i = blockIdx.x * T + threadIdx.x;
    const bool is = i < k && weight[i] >= least;
    if constexpr (PASS == 0) {
        const int n = __syncthreads_count(is);
        if (threadIdx.x == 0) first[blockIdx.x] = n;
    } else {
        __shared__ int warp_count[T / 32];
        const unsigned mine = __ballot_sync(0xffffffffu, is);
        if ((threadIdx.x & 31) == 0) warp_count[threadIdx.x >> 5] = __popc(mine);
        __syncthreads();
        int at = first[blockIdx.x];
        for (int w = 0; w < (int)threadIdx.x >> 5; ++w) at += warp_count[w];
        if (is) out[at + __popc(mine & ((1u << (threadIdx.x & 31)) - 1))] = Keyed{weight[i], i};
    }
}

// One digit of a stable sort, largest keys first.  A CTA takes kSortBlock elements, a warp an eighth of them in strips of 32, in
// order; equal digits of a strip find one another by __match_any_sync.  PASS 0: how many of every digit, [digit][CTA]; 1: to their places.
constexpr int kSortBlock = 2048;
template <int PASS>
__global__ void __launch_bounds__(T) k_sort_digit(const Keyed* __restrict__ in, Keyed* __restrict__ out, int32_t n, int shift, int32_t* __restrict__ first)
{
    constexpr int kWarps = T / 32, kStrips = kSortBlock / T;
    __shared__ int count[kWarps][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kWarps * 256; i += T) (&count[0][0])[i] = 0;
    __syncthreads();
    const int32_t begin = blockIdx.x * kSortBlock + warp * (kSortBlock / kWarps) + lane;
    Keyed x[kStrips];
    int place[kStrips];                   // among the warp's elements with this digit
#pragma unroll
    for (int s = 0; s < kStrips; ++s) {
        const int32_t i = begin + s * 32;
        const bool valid = i < n;
        if (valid) x[s] = in[i];
        const int digit = valid ? 255 - (x[s].key >> shift & 255) : 256;
        const unsigned same = __match_any_sync(0xffffffffu, digit);
        int before = 0;
        if (valid) before = count[warp][digit];
        __syncwarp();
        place[s] = before + __popc(same & ((1u << lane) - 1));
        if (valid && lane == __ffs(same) - 1) count[warp][digit] = before + __popc(same);
        __syncwarp();
    }
    __syncthreads();
    for (int d = threadIdx.x; d < 256; d += T) {
        int sum = PASS == 0 ? 0 : first[(int64_t)d * gridDim.x + blockIdx.x];
        for (int w = 0; w < kWarps; ++w) {
            const int c = count[w][d];
            count[w][d] = sum;
            sum += c;
        }
        if (PASS == 0) first[(int64_t)d * gridDim.x + blockIdx.x] = sum;
    }
    if (PASS == 0) return;
    __syncthreads();
#pragma unroll
    for (int s = 0; s < kStrips; ++s)
        if (begin + s * 32 < n) out[count[warp][255 - (x[s].key >> shift & 255)] + place[s]] = x[s];
}

// rank[id] = place in the sorted list; the ids themselves, where wanted.
__global__ void k_ranks(const Keyed* __restrict__ sorted, int32_t n, int32_t* __restrict__ rank, int32_t* __restrict__ ids)
{
    const int32_t i = blockIdx.x * T + threadIdx.x;
    if (i >= n) return;
    rank[sorted[i].id] = i;
    if (ids) ids[i] = sorted[i].id;
}

// MODE 0: how many entries every tile would hold.  MODE 1: how many entries of every chunk lie outside the chosen tiles.
// MODE 2: the entries themselves, into their tiles' records (in any order: a record says where it belongs) and, in order,
// into what is left of the rows.
template <int MODE>
__global__ void __launch_bounds__(T) k_tile_entries(const dg_chunk* __restrict__ chunks, int32_t n_chunks, const int32_t* __restrict__ col,
                                                    const float* __restrict__ val, const int32_t* __restrict__ row_rank,
                                                    const int32_t* __restrict__ col_rank, int32_t col_tiles, int32_t* __restrict__ tile,
                                                    int32_t* __restrict__ cursor, int32_t* __restrict__ rest, uint2* __restrict__ records,
                                                    int32_t* __restrict__ rest_col, float* __restrict__ rest_val, int* __restrict__ largest)
{
    const int32_t c = blockIdx.x * (T / 32) + (threadIdx.x >> 5);
    if (c >= n_chunks) return;
    const int lane = threadIdx.x & 31;
    const dg_chunk ch = chunks[c];
    const int32_t rr = row_rank[ch.heavy];
    int32_t* row_tile = tile + (int64_t)(rr / kTileRows) * col_tiles;
    int32_t left = MODE == 2 ? rest[ch.slot] : 0;
    int biggest = 0;
    for (int base = 0; base < ch.len; base += 32) {
        const bool valid = base + lane < ch.len;
        int32_t cc = 0, cr = -1;
        if (valid) {
            cc = __ldcs(col + ch.e0 + base + lane);
            cr = __ldg(col_rank + cc);
        }
        if constexpr (MODE == 0) {
            if (cr >= 0) atomicAdd(row_tile + cr / kTileCols, 1);
        } else {
            const int32_t slab = cr >= 0 ? __ldg(row_tile + cr / kTileCols) : -1;
            const unsigned out = __ballot_sync(0xffffffffu, valid && slab < 0);
            if constexpr (MODE == 2) {
                if (valid) {
                    const float v = __ldcs(val + ch.e0 + base + lane);
                    if (slab >= 0) {
                        uint32_t h, m, l;
                        split3(v, h, m, l);
                        biggest = max(biggest, __float_as_int(fabsf(v)));       // ordered as the numbers are, a NaN above them
                        records[atomicAdd(cursor + slab, 1)] =
                            make_uint2(h | m << 16, l | (uint32_t)tile_element(rr % kTileRows, cr % kTileCols) << 16);
                    } else {
                        const int32_t at = left + __popc(out & ((1u << lane) - 1));
                        rest_col[at] = cc;
                        rest_val[at] = v;
                    }
                }
            }
            left += __popc(out);
        }
    }
    if (MODE == 1 && lane == 0) rest[ch.slot] = left;
    if (MODE == 2) {
        biggest = __reduce_max_sync(0xffffffffu, biggest);
        if (lane == 0 && biggest > *(volatile int*)largest) atomicMax(largest, biggest);
    }
}

// The tiles with at least kTileMin entries, in order of row tile and column tile, and what multiplying one costs: 2,400 clocks and
// 1.5 for every record beyond 1,024 (counted in half clocks).
struct Chosen { int32_t slabs, entries; long long cost; };
__device__ __forceinline__ Chosen operator+(const Chosen& a, const Chosen& b) { return Chosen{a.slabs + b.slabs, a.entries + b.entries, a.cost + b.cost}; }
__device__ __forceinline__ Chosen chosen(int32_t count)
{
    return count < kTileMin ? Chosen{0, 0, 0} : Chosen{1, count, 4800 + 3 * (long long)max(0, count - 1024)};
}
__device__ __forceinline__ Chosen shift_up(const Chosen& v, int off)
{
    return Chosen{__shfl_up_sync(0xffffffffu, v.slabs, off), __shfl_up_sync(0xffffffffu, v.entries, off), __shfl_up_sync(0xffffffffu, v.cost, off)};
}
__device__ __forceinline__ Chosen block_before(const Chosen& v, Chosen* warp_sum, Chosen* all)      // sum over the threads before this one
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Chosen s = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const Chosen o = shift_up(s, off);
        if (lane >= off) s = s + o;
    }
    if (lane == 31) warp_sum[warp] = s;
    Chosen before = shift_up(s, 1);
    if (lane == 0) before = Chosen{0, 0, 0};
    __syncthreads();
    Chosen total{0, 0, 0};
    for (int w = 0; w < (int)blockDim.x >> 5; ++w) {
        if (w < warp) before = before + warp_sum[w];
        total = total + warp_sum[w];
    }
    __syncthreads();
    *all = total;
    return before;
}

// One CTA: from which weight on a column is frequent.  The most frequent columns, at most kMaxColumns, and none so rare that a
// tile could not reach kTileMin with its like.
__global__ void __launch_bounds__(1024) k_least_weight(const int32_t* __restrict__ bins, Found* __restrict__ found)
{
    __shared__ Chosen warp_sum[32];
    __shared__ int32_t least;
    if (threadIdx.x == 0) least = kWeightBins;
    constexpr int kEach = kWeightBins / 1024;
    Chosen mine{0, 0, 0}, all;
    int32_t n[kEach];
#pragma unroll
    for (int j = 0; j < kEach; ++j) mine.cost += n[j] = bins[kWeightBins - 1 - ((int)threadIdx.x * kEach + j)];
    long long columns = block_before(mine, warp_sum, &all).cost, kept = 0;
    int32_t at = kWeightBins;
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
        const int32_t w = kWeightBins - 1 - (threadIdx.x * kEach + j);
        columns += n[j];
        if (w > kTileMin / kTileCols && columns <= kMaxColumns) at = w, kept = columns;
    }
    if (at < kWeightBins) atomicMin(&least, at);
    __syncthreads();
    if (at < kWeightBins && at == least) {
        found->least = at;
        found->columns = (int32_t)kept;
    }
}

constexpr int kChooseBlock = T * 4;
// PASS 0: sums of every kChooseBlock tiles.  1: the slabs, the table (which slab a tile is, or -1), and which CTA multiplies a slab: equal
// shares of the cost, in order.
template <int PASS>
__global__ void __launch_bounds__(T) k_choose_tiles(int32_t* __restrict__ tile, int64_t tiles, int32_t col_tiles, int32_t ctas, Chosen* __restrict__ sums,
                                                    dg_slab* __restrict__ slabs, int32_t* __restrict__ cursor, int2* __restrict__ place,
                                                    const Found* __restrict__ found)
{
    __shared__ Chosen warp_sum[T / 32];
    const int64_t i0 = (int64_t)blockIdx.x * kChooseBlock + threadIdx.x * 4;
    int32_t count[4];
    Chosen mine{0, 0, 0}, all;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        count[j] = i0 + j < tiles ? tile[i0 + j] : 0;
        mine = mine + chosen(count[j]);
    }
    Chosen at = block_before(mine, warp_sum, &all);
    if constexpr (PASS == 0) {
        if (threadIdx.x == 0) sums[blockIdx.x] = all;
    } else {
        at = at + sums[blockIdx.x];
        const long long cost = found->cost;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i0 + j >= tiles) break;
            const Chosen c = chosen(count[j]);
            tile[i0 + j] = c.slabs ? at.slabs : -1;
            if (c.slabs) {
                slabs[at.slabs] = dg_slab{(int32_t)((i0 + j) % col_tiles), at.entries, count[j]};
                cursor[at.slabs] = at.entries;
                place[at.slabs] = make_int2((int32_t)((i0 + j) / col_tiles), (int32_t)min((long long)ctas - 1, at.cost * ctas / cost));
            }
            at = at + c;
        }
    }
}

// One CTA: exclusive sums over the blocks' sums, in place.
__global__ void __launch_bounds__(1024) k_sum_chosen(Chosen* __restrict__ sums, int32_t blocks, Found* __restrict__ found)
{
    __shared__ Chosen warp_sum[32];
    Chosen carry{0, 0, 0}, all;
    for (int32_t b0 = 0; b0 < blocks; b0 += 1024) {
        const int32_t b = b0 + threadIdx.x;
        const Chosen before = block_before(b < blocks ? sums[b] : Chosen{0, 0, 0}, warp_sum, &all);
        if (b < blocks) sums[b] = carry + before;
        carry = carry + all;
    }
    if (threadIdx.x == 0) {
        found->slabs = carry.slabs;
        found->entries = carry.entries;
        found->cost = carry.cost;
    }
}

// One CTA: consecutive slabs of one row tile and one CTA are a segment.  `place`: row tile and CTA of every slab.
__global__ void __launch_bounds__(1024) k_segments(const int2* __restrict__ place, int32_t slabs, int32_t ctas, dg_segment* __restrict__ segments,
                                                   int32_t* __restrict__ cta_segment, int2* __restrict__ tile_parts, Found* __restrict__ found)
{
    __shared__ Chosen warp_sum[32];
    int32_t carry = 0;
    for (int32_t s0 = 0; s0 < slabs; s0 += 4 * 1024) {
        const int32_t b = s0 + threadIdx.x * 4;
        int2 at[4], before = b > 0 && b <= slabs ? place[b - 1] : make_int2(-1, -1);
        Chosen mine{0, 0, 0}, all;
        for (int j = 0; j < 4; ++j) {
            at[j] = b + j < slabs ? place[b + j] : make_int2(-1, -1);
            const int2 p = j ? at[j - 1] : before;
            if (b + j < slabs && (p.x != at[j].x || p.y != at[j].y)) ++mine.slabs;
        }
        int32_t g = carry + block_before(mine, warp_sum, &all).slabs;
        for (int j = 0; j < 4 && b + j < slabs; ++j) {
            const int2 p = j ? at[j - 1] : before;
            if (p.x != at[j].x || p.y != at[j].y) {
                segments[g].slab0 = b + j;
                segments[g].slot = g;
                segments[g].pad = 0;
                if (g > 0) segments[g - 1].slab1 = b + j;
                for (int c = p.y + 1; c <= at[j].y; ++c) cta_segment[c] = g;
                if (p.x != at[j].x) tile_parts[at[j].x].x = g;
                atomicAdd(&tile_parts[at[j].x].y, 1);
                ++g;
            }
            if (b + j == slabs - 1) {
                segments[g - 1].slab1 = slabs;
                for (int c = at[j].y + 1; c <= ctas; ++c) cta_segment[c] = g;
                found->segments = g;
            }
        }
        carry += all.slabs;
    }
}

__global__ void k_row_parts(const int32_t* __restrict__ row_rank, int32_t n_rows, const int2* __restrict__ tile_parts, int2* __restrict__ parts)
{
    const int32_t h = blockIdx.x * T + threadIdx.x;
    if (h >= n_rows) return;
    const int32_t r = row_rank[h];
    const int2 of = tile_parts[r / kTileRows];
    parts[h] = make_int2(of.x * kTileRows + r % kTileRows, of.y);
}

// Exclusive sums in place, one CTA; the total goes behind the last element.
__global__ void __launch_bounds__(1024) k_exclusive_sums(int32_t* __restrict__ v, int32_t n)
{
    __shared__ int32_t warp_sum[32];
    int32_t carry = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int32_t b = 0; b < n; b += 1024 * 4) {
        int32_t x[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t i = b + threadIdx.x * 4 + j;
            x[j] = i < n ? v[i] : 0;
            sum += x[j];
        }
        int32_t s = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int32_t o = __shfl_up_sync(0xffffffffu, s, off);
            if (lane >= off) s += o;
        }
        if (lane == 31) warp_sum[warp] = s;
        __syncthreads();
        int32_t before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) before += warp_sum[w];
            all += warp_sum[w];
        }
        int32_t at = carry + before + s - sum;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t i = b + threadIdx.x * 4 + j;
            if (i < n) v[i] = at;
            at += x[j];
        }
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) v[n] = carry;
}

// Chunks of what is left of every split row, at least one (it may be empty: whoever works on a row's last chunk writes the row).
// PASS 0: how many per row; 1: how many start in each column band; 2: the chunks, by band.
template <int PASS>
__global__ void k_rest_chunks(const SplitRow* __restrict__ rows, int32_t n_rows, const int32_t* __restrict__ first_slot, const int32_t* __restrict__ rest,
                              int32_t chunk, const int32_t* __restrict__ rest_col, int32_t k, int32_t* __restrict__ chunk_first,
                              int32_t* __restrict__ bands, dg_chunk* __restrict__ out)
{
    const int32_t h = blockIdx.x * T + threadIdx.x;
    if (h >= n_rows) return;
    const int32_t begin = rest[first_slot[h]], len = rest[first_slot[h + 1]] - begin, n = len > 0 ? (len + chunk - 1) / chunk : 1;
    if constexpr (PASS == 0) {
        chunk_first[h] = n;
    } else {
        for (int32_t j = 0; j < n; ++j) {
            const int32_t e = begin + j * chunk, count = min(chunk, len - j * chunk), band = count > 0 ? band_of(rest_col[e], k) : 0;
            const int32_t at = atomicAdd(&bands[band], 1);
            if constexpr (PASS == 2) out[at] = dg_chunk{e, count, rows[h].row, chunk_first[h] + j, chunk_first[h], n, h};
        }
    }
}

__global__ void k_first_slots(const dg_chunk* __restrict__ chunks, int32_t n_chunks, int32_t n_rows, int32_t* __restrict__ first_slot)
{
    const int32_t c = blockIdx.x * T + threadIdx.x;
    if (c == 0) first_slot[n_rows] = n_chunks;
    if (c < n_chunks && chunks[c].slot == chunks[c].slot0) first_slot[chunks[c].heavy] = chunks[c].slot0;
}

unsigned grid_of(int64_t n, int per_block) { return (unsigned)((n + per_block - 1) / per_block); }

// `list` sorted by key, largest first, equal keys in the order they have; the result is where the pointer says.
int sort_keyed(Keyed** list, Keyed** spare, int32_t n, int32_t max_key, int32_t* first, cudaStream_t stream)
{
    const int32_t blocks = (int32_t)grid_of(n, kSortBlock);
    for (int shift = 0; shift < 32 && (max_key >> shift) > 0; shift += 8) {
        k_sort_digit<0><<<blocks, T, 0, stream>>>(*list, nullptr, n, shift, first);
        k_exclusive_sums<<<1, 1024, 0, stream>>>(first, 256 * blocks);
        k_sort_digit<1><<<blocks, T, 0, stream>>>(*list, *spare, n, shift, first);
        std::swap(*list, *spare);
    }
    return (int)cudaGetLastError();
}

// Fills `t`; returns DG_OK with t->entries == 0 where tiles would not pay.
int build_tiles(const dg_plan* p, const float* val, cudaStream_t stream, dg_tiles* t)
{
    if (p->n_heavy < kTileRows || p->nnz >= ((int64_t)1 << 31)) return DG_OK;
    PoolScope tmp(stream);
    int rc, dev = 0, ctas = 0;
    DG_CUDA(cudaGetDevice(&dev));
    DG_CUDA(cudaDeviceGetAttribute(&ctas, cudaDevAttrMultiProcessorCount, dev));
    SplitRow* rows = nullptr;
    Keyed *by_length = nullptr, *frequent = nullptr, *spare = nullptr;
    int32_t *first_slot = nullptr, *weight = nullptr, *bins = nullptr, *col_rank = nullptr, *row_rank = nullptr, *first = nullptr;
    Found* found = nullptr;
    const int32_t longest_list = std::max(p->n_heavy, kMaxColumns), column_blocks = (int32_t)grid_of(p->k, T);
    const size_t sums = std::max<size_t>((size_t)256 * grid_of(longest_list, kSortBlock), column_blocks) + 1;
    if ((rc = tmp.alloc(&rows, p->n_heavy)) || (rc = tmp.alloc(&by_length, p->n_heavy)) || (rc = tmp.alloc(&spare, longest_list)) ||
        (rc = tmp.alloc(&first, sums)) || (rc = tmp.alloc(&first_slot, (size_t)p->n_heavy + 1)) || (rc = tmp.alloc(&weight, p->k)) ||
        (rc = tmp.alloc(&bins, kWeightBins)) || (rc = tmp.alloc(&col_rank, p->k)) || (rc = tmp.alloc(&row_rank, p->n_heavy)) ||
        (rc = tmp.alloc(&frequent, kMaxColumns)) || (rc = tmp.alloc(&found, 1)))
        return rc;
    DG_CUDA(cudaMemsetAsync(weight, 0, (size_t)p->k * sizeof(int32_t), stream));
    DG_CUDA(cudaMemsetAsync(bins, 0, kWeightBins * sizeof(int32_t), stream));
    DG_CUDA(cudaMemsetAsync(found, 0, sizeof(Found), stream));
    DG_CUDA(cudaMemsetAsync(col_rank, 0xff, (size_t)p->k * sizeof(int32_t), stream));
    k_split_rows<<<grid_of(p->n_chunks, T), T, 0, stream>>>(p->chunks, p->n_chunks, p->rowptr, rows, by_length);
    k_first_slots<<<grid_of(p->n_chunks, T), T, 0, stream>>>(p->chunks, p->n_chunks, p->n_heavy, first_slot);
    k_column_weights<<<grid_of(p->n_chunks, T / 32), T, 0, stream>>>(p->chunks, p->n_chunks, p->col, weight, found);
    k_weight_histogram<<<148, T, 0, stream>>>(weight, p->k, bins, found);
    k_least_weight<<<1, 1024, 0, stream>>>(bins, found);
    Found h{};
    auto read = [&] {
        const cudaError_t e = cudaMemcpyAsync(&h, found, sizeof(h), cudaMemcpyDeviceToHost, stream);
        return (int)(e != cudaSuccess ? e : cudaStreamSynchronize(stream));
    };
    if ((rc = read())) return rc;
    if (h.columns < kTileCols || h.unordered) return DG_OK;

    // columns by weight, rows by length
    t->n_columns = h.columns;
    t->col_tiles = (int32_t)grid_of(h.columns, kTileCols);
    const int32_t row_tiles = (int32_t)grid_of(p->n_heavy, kTileRows);
    const int64_t tiles = (int64_t)row_tiles * t->col_tiles;
    if (tiles > (int64_t)1 << 26) return DG_OK;
    const int32_t choose_blocks = (int32_t)grid_of(tiles, kChooseBlock);
    int32_t *tile = nullptr, *rest = nullptr;
    Chosen* chosen_sums = nullptr;
    if ((rc = dg_pool_alloc((void**)&t->columns, (size_t)h.columns * sizeof(int32_t))) || (rc = tmp.alloc(&tile, (size_t)tiles)) ||
        (rc = tmp.alloc(&rest, (size_t)p->n_chunks + 1)) || (rc = tmp.alloc(&chosen_sums, (size_t)choose_blocks)))
        return rc;
    k_frequent_columns<0><<<column_blocks, T, 0, stream>>>(weight, p->k, h.least, first, nullptr);
    k_exclusive_sums<<<1, 1024, 0, stream>>>(first, column_blocks);
    k_frequent_columns<1><<<column_blocks, T, 0, stream>>>(weight, p->k, h.least, first, frequent);
    Keyed* other = spare;                               // the sorted columns are read before the rows are sorted
    if ((rc = sort_keyed(&frequent, &other, h.columns, h.max_weight, first, stream))) return rc;
    k_ranks<<<grid_of(h.columns, T), T, 0, stream>>>(frequent, h.columns, col_rank, t->columns);
    if ((rc = sort_keyed(&by_length, &spare, p->n_heavy, (int32_t)std::min<int64_t>(INT32_MAX, p->max_row_nnz), first, stream))) return rc;
    k_ranks<<<grid_of(p->n_heavy, T), T, 0, stream>>>(by_length, p->n_heavy, row_rank, nullptr);

    // how full the tiles are, and which of them are worth it
    DG_CUDA(cudaMemsetAsync(tile, 0, (size_t)tiles * sizeof(int32_t), stream));
    const unsigned warps = grid_of(p->n_chunks, T / 32);
    k_tile_entries<0><<<warps, T, 0, stream>>>(p->chunks, p->n_chunks, p->col, val, row_rank, col_rank, t->col_tiles, tile, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
    k_choose_tiles<0><<<choose_blocks, T, 0, stream>>>(tile, tiles, t->col_tiles, ctas, chosen_sums, nullptr, nullptr, nullptr, found);
    k_sum_chosen<<<1, 1024, 0, stream>>>(chosen_sums, choose_blocks, found);
    if ((rc = read())) return rc;
    if (h.slabs == 0 || h.entries < p->nnz / 8) return DG_OK;      // the columns' images and another launch cost more than that saves

    // the slabs, equal shares of the work for every CTA, cut again where the row tile changes
    t->n_slabs = h.slabs;
    t->ctas = ctas;
    const int64_t left = p->heavy_nnz - h.entries, max_segments = std::min<int64_t>(h.slabs, (int64_t)row_tiles + ctas),
                  max_rest_chunks = std::min<int64_t>(p->n_chunks, p->n_heavy + left / p->chunk);
    int32_t *cursor = nullptr, *chunk_first = nullptr, *bands = nullptr;
    int2 *place = nullptr, *tile_parts = nullptr;
    if ((rc = tmp.alloc(&cursor, (size_t)h.slabs)) || (rc = tmp.alloc(&place, (size_t)h.slabs)) || (rc = tmp.alloc(&tile_parts, (size_t)row_tiles)) ||
        (rc = tmp.alloc(&chunk_first, (size_t)p->n_heavy + 1)) || (rc = tmp.alloc(&bands, kBands + 1)) ||
        (rc = dg_pool_alloc((void**)&t->slabs, (size_t)h.slabs * sizeof(dg_slab))) ||
        (rc = dg_pool_alloc((void**)&t->segments, (size_t)max_segments * sizeof(dg_segment))) ||
        (rc = dg_pool_alloc((void**)&t->cta_segment, ((size_t)ctas + 1) * sizeof(int32_t))) ||
        (rc = dg_pool_alloc((void**)&t->parts, (size_t)p->n_heavy * sizeof(int2))) ||
        (rc = dg_pool_alloc((void**)&t->records, (size_t)h.entries * sizeof(uint2))) ||
        (rc = dg_pool_alloc((void**)&t->rest_col, (size_t)std::max<int64_t>(left, 1) * sizeof(int32_t))) ||
        (rc = dg_pool_alloc((void**)&t->rest_val, (size_t)std::max<int64_t>(left, 1) * sizeof(float))) ||
        (rc = dg_pool_alloc((void**)&t->rest_chunks, (size_t)max_rest_chunks * sizeof(dg_chunk))) ||
        (rc = dg_pool_alloc(&t->value_sums, (size_t)ctas * kValueWarps * sizeof(ValueSum))))
        return rc;
    DG_CUDA(cudaMemsetAsync(tile_parts, 0, (size_t)row_tiles * sizeof(int2), stream));
    DG_CUDA(cudaMemsetAsync(bands, 0, kBands * sizeof(int32_t), stream));
    k_choose_tiles<1><<<choose_blocks, T, 0, stream>>>(tile, tiles, t->col_tiles, ctas, chosen_sums, t->slabs, cursor, place, found);
    k_segments<<<1, 1024, 0, stream>>>(place, h.slabs, ctas, t->segments, t->cta_segment, tile_parts, found);
    k_row_parts<<<grid_of(p->n_heavy, T), T, 0, stream>>>(row_rank, p->n_heavy, tile_parts, t->parts);

    // the entries into the slabs' records and into what is left of the rows, with its chunks in the order of the column band they start in
    k_tile_entries<1><<<warps, T, 0, stream>>>(p->chunks, p->n_chunks, p->col, val, row_rank, col_rank, t->col_tiles, tile, nullptr, rest, nullptr, nullptr, nullptr, nullptr);
    k_exclusive_sums<<<1, 1024, 0, stream>>>(rest, p->n_chunks);
    k_tile_entries<2><<<warps, T, 0, stream>>>(p->chunks, p->n_chunks, p->col, val, row_rank, col_rank, t->col_tiles, tile, cursor, rest, t->records, t->rest_col,
                                               t->rest_val, &found->largest);
    const unsigned row_blocks = grid_of(p->n_heavy, T);
    k_rest_chunks<0><<<row_blocks, T, 0, stream>>>(rows, p->n_heavy, first_slot, rest, p->chunk, t->rest_col, p->k, chunk_first, bands, nullptr);
    k_exclusive_sums<<<1, 1024, 0, stream>>>(chunk_first, p->n_heavy);
    k_rest_chunks<1><<<row_blocks, T, 0, stream>>>(rows, p->n_heavy, first_slot, rest, p->chunk, t->rest_col, p->k, chunk_first, bands, nullptr);
    k_exclusive_sums<<<1, 1024, 0, stream>>>(bands, kBands);
    k_rest_chunks<2><<<row_blocks, T, 0, stream>>>(rows, p->n_heavy, first_slot, rest, p->chunk, t->rest_col, p->k, chunk_first, bands, t->rest_chunks);
    k_value_sums<<<ctas, 32 * kValueWarps, 0, stream>>>(val, p->nnz, static_cast<ValueSum*>(t->value_sums));
    DG_CUDA(cudaMemcpyAsync(&found->rest_chunks, chunk_first + p->n_heavy, sizeof(int32_t), cudaMemcpyDeviceToDevice, stream));
    DG_CUDA(cudaMemcpyAsync(&found->rest, rest + p->n_chunks, sizeof(int32_t), cudaMemcpyDeviceToDevice, stream));
    if ((rc = read())) return rc;
    tmp.idle = true;
    DG_CUDA(cudaGetLastError());
    if (h.rest != left || h.rest_chunks > max_rest_chunks || h.segments > max_segments) return DG_ERR_STATE;     // cannot happen
    float largest;
    memcpy(&largest, &h.largest, sizeof(float));
    if (!(largest < kTileBound) || largest < kTileLeast) return DG_OK;
    t->least_operand = largest < 1.f ? kTileLeast / largest : kTileLeast;
    t->val = val;
    t->n_segments = h.segments;
    t->n_rest_chunks = h.rest_chunks;
    t->entries = h.entries;
    return DG_OK;
}

}  // namespace

void dg_tiles_free(dg_tiles* t)
{
    if (!t) return;
    for (void* b : {(void*)t->records, (void*)t->slabs, (void*)t->segments, (void*)t->cta_segment, (void*)t->columns, (void*)t->parts, (void*)t->rest_col,
                    (void*)t->rest_val, (void*)t->rest_chunks, t->value_sums})
        dg_pool_free(b);
    delete t;
}

extern "C" int dg_plan_add_tiles(dg_plan* p, const float* val, void* stream)
try {
    if (!p || (p->nnz > 0 && !val)) return DG_ERR_NULL;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != p->device) return DG_ERR_STATE;
    const int dropped = dg_plan_drop_tiles(p, stream);
    if (dropped) return dropped;
    struct Owner {                        // until the plan has them
        dg_tiles* tiles;
        cudaStream_t stream;
        ~Owner()
        {
            if (tiles) cudaStreamSynchronize(stream);
            dg_tiles_free(tiles);
        }
    } owner{new (std::nothrow) dg_tiles(), (cudaStream_t)stream};
    dg_tiles* t = owner.tiles;
    if (!t) return (int)cudaErrorMemoryAllocation;
    t->status = dg_status_word();
    const int rc = t->status ? build_tiles(p, val, (cudaStream_t)stream, t) : DG_ERR_STATE;
    if (rc != DG_OK || t->entries == 0) return rc;
    p->tiles = t;
    owner.tiles = nullptr;
    return DG_OK;
} catch (...) {
    return dg_exception();
}

extern "C" int dg_plan_drop_tiles(dg_plan* p, void* stream)
try {
    if (!p) return DG_ERR_NULL;
    if (!p->tiles) return DG_OK;
    DG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    dg_tiles_free(p->tiles);
    p->tiles = nullptr;
    return DG_OK;
} catch (...) {
    return dg_exception();
}

// The give-up path on purpose: the tensor-core part of a product, with waits of no polls at all.
extern "C" int dg_tiles_wait_selftest(const dg_plan* p, const float* B, int64_t ldb, int32_t F, void* stream)
try {
    if (!p || !B) return DG_ERR_NULL;
    if (F < 1 || ldb < F) return DG_ERR_DIMS;
    int rc = dg_spmm_prepare(p, F, (cudaStream_t)stream);
    if (rc) return rc;
    const int64_t need = dg_tiles_scratch_floats(p, F);
    if (need == 0 || need > p->scratch_floats) return DG_ERR_STATE;
    int launches = 0;
    return dg_tiles_launch(p, B, ldb, F, p->scratch, (cudaStream_t)stream, &launches, 0);
} catch (...) {
    return dg_exception();
}

extern "C" int64_t dg_plan_tiled_entries(const dg_plan* p) { return p && p->tiles ? p->tiles->entries : 0; }

// Narrow operands are gathered: a tile costs at least its six passes over A whatever the width is.
int64_t dg_tiles_scratch_floats(const dg_plan* p, int32_t F)
{
    const dg_tiles* t = p->tiles;
    if (!t || F < 32) return 0;
    const int64_t F4 = (F + 3) / 4 * 4;
    return (int64_t)t->n_segments * kTileRows * F4 + (int64_t)panels_of(F) * t->col_tiles * 3 * panel_width(F) * kTileCols / 2;
}

int dg_tiles_launch(const dg_plan* p, const float* B, int64_t ldb, int32_t F, float* area, cudaStream_t stream, int* launches, int wait_limit)
{
    const dg_tiles* t = p->tiles;
    const int32_t F4 = (F + 3) / 4, panels = panels_of(F), n_pad = panel_width(F);
    uint16_t* images = reinterpret_cast<uint16_t*>(area + (int64_t)t->n_segments * kTileRows * F4 * 4);
    k_tile_columns<<<dim3((unsigned)t->col_tiles, (unsigned)panels), T, 0, stream>>>(B, ldb, t->columns, t->n_columns, t->col_tiles, F, n_pad, images, p->status + DG_TILE_WORDS);
    const TileArgs a{t->slabs, t->segments, t->cta_segment, t->records, images, reinterpret_cast<float4*>(area), F4, F4, n_pad, t->col_tiles, p->status, t->status, t->least_operand, p->status + DG_TILE_WORDS, wait_limit, t->val, static_cast<const ValueSum*>(t->value_sums), p->nnz};
    const size_t smem = kTileStages * (3 * kTileElems * 2 + (size_t)3 * n_pad * kTileCols * 2) + 24 * kTileStages + 32 + 128;
    static std::atomic<bool> allowed[64];
    if (p->device < 0 || p->device >= 64) return DG_ERR_STATE;
    if (!allowed[p->device].load(std::memory_order_relaxed)) {
        DG_CUDA(cudaFuncSetAttribute(k_tile_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        allowed[p->device].store(true, std::memory_order_relaxed);
    }
    k_tile_mma<<<dim3((unsigned)t->ctas, (unsigned)panels), kTileThreads, smem, stream>>>(a);
    *launches += 2;
    return (int)cudaGetLastError();
}
