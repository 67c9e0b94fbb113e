// Dense tiles: the hub x hub corner of a power-law block on the tensor cores.
//
// A gather moves 4 F bytes through an SM's 64-byte-a-clock port for every entry, which is what bounds k_spmm on large blocks
// (16 clocks an entry at F = 256).  Sorted by length and by frequency, the split rows and the frequent columns of a
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
// 16.6 -> 8.9 ms; 306,128 nodes / 15.8 M entries, F = 256: 1.03 -> 0.84 ms.  The MMAs themselves are half of k_tile_mma's time, the
// rest is waiting for a tile to be filled after an accumulator was drained.
#include <algorithm>
#include <atomic>
#include <new>
#include <vector>
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
// One-off, on the device except for sorting the row and column lists (at most some 100,000 keys each) and choosing the tiles.
// Four passes over the entries of the split rows, one chunk per warp; about 10 ms for 107 M entries.
namespace {

struct SplitRow { int32_t row, len; };

__global__ void k_split_rows(const dg_chunk* __restrict__ chunks, int32_t n_chunks, const int64_t* __restrict__ rowptr, SplitRow* __restrict__ rows)
{
    const int32_t c = blockIdx.x * T + threadIdx.x;
    if (c >= n_chunks || chunks[c].slot != chunks[c].slot0) return;
    const int32_t r = chunks[c].row;
    rows[chunks[c].heavy] = SplitRow{r, (int32_t)min((int64_t)INT32_MAX, rowptr[r + 1] - rowptr[r])};
}

// How many entries of split rows every column holds.
__global__ void __launch_bounds__(T) k_column_weights(const dg_chunk* __restrict__ chunks, int32_t n_chunks, const int32_t* __restrict__ col,
                                                      int32_t* __restrict__ weight)
{
    const int32_t c = blockIdx.x * (T / 32) + (threadIdx.x >> 5);
    if (c >= n_chunks) return;
    const dg_chunk ch = chunks[c];
    for (int i = threadIdx.x & 31; i < ch.len; i += 32) atomicAdd(&weight[col[ch.e0 + i]], 1);
}

constexpr int kWeightBins = 4096;
__global__ void __launch_bounds__(T) k_weight_histogram(const int32_t* __restrict__ weight, int32_t k, int32_t* __restrict__ bins)
{
    __shared__ int32_t local[kWeightBins];
    for (int i = threadIdx.x; i < kWeightBins; i += T) local[i] = 0;
    __syncthreads();
    for (int32_t i = blockIdx.x * T + threadIdx.x; i < k; i += gridDim.x * T) atomicAdd(&local[min(weight[i], kWeightBins - 1)], 1);
    __syncthreads();
    for (int i = threadIdx.x; i < kWeightBins; i += T)
        if (local[i]) atomicAdd(&bins[i], local[i]);
}

__global__ void k_frequent_columns(const int32_t* __restrict__ weight, int32_t k, int32_t least, int2* __restrict__ out, int32_t capacity, int32_t* __restrict__ count)
{
    const int32_t i = blockIdx.x * T + threadIdx.x;
    if (i >= k || weight[i] < least) return;
    const int32_t at = atomicAdd(count, 1);
    if (at < capacity) out[at] = make_int2(i, weight[i]);
}

__global__ void k_column_ranks(const int32_t* __restrict__ columns, int32_t n, int32_t* __restrict__ rank)
{
    const int32_t i = blockIdx.x * T + threadIdx.x;
    if (i < n) rank[columns[i]] = i;
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

template <class X> int upload(X** device, const std::vector<X>& host, cudaStream_t stream)
{
    const int rc = dg_pool_alloc((void**)device, std::max<size_t>(host.size(), 1) * sizeof(X));
    if (rc) return rc;
    return host.empty() ? DG_OK : (int)cudaMemcpyAsync(*device, host.data(), host.size() * sizeof(X), cudaMemcpyHostToDevice, stream);
}

// Fills `t`; returns DG_OK with t->entries == 0 where tiles would not pay.
int build_tiles(const dg_plan* p, const float* val, cudaStream_t stream, dg_tiles* t)
{
    if (p->n_heavy < kTileRows || p->nnz >= ((int64_t)1 << 31)) return DG_OK;
    PoolScope tmp(stream);
    int rc;
    SplitRow* d_rows = nullptr;
    int32_t *first_slot = nullptr, *weight = nullptr, *bins = nullptr, *col_rank = nullptr, *row_rank = nullptr;
    int2* frequent = nullptr;
    const size_t bins_n = kWeightBins + 2;
    if ((rc = tmp.alloc(&d_rows, p->n_heavy)) || (rc = tmp.alloc(&first_slot, (size_t)p->n_heavy + 1)) || (rc = tmp.alloc(&weight, p->k)) ||
        (rc = tmp.alloc(&bins, bins_n)) || (rc = tmp.alloc(&col_rank, p->k)) || (rc = tmp.alloc(&row_rank, p->n_heavy)) ||
        (rc = tmp.alloc(&frequent, kMaxColumns)))
        return rc;
    DG_CUDA(cudaMemsetAsync(weight, 0, (size_t)p->k * sizeof(int32_t), stream));
    DG_CUDA(cudaMemsetAsync(bins, 0, bins_n * sizeof(int32_t), stream));
    DG_CUDA(cudaMemsetAsync(col_rank, 0xff, (size_t)p->k * sizeof(int32_t), stream));
    k_split_rows<<<grid_of(p->n_chunks, T), T, 0, stream>>>(p->chunks, p->n_chunks, p->rowptr, d_rows);
    k_first_slots<<<grid_of(p->n_chunks, T), T, 0, stream>>>(p->chunks, p->n_chunks, p->n_heavy, first_slot);
    k_column_weights<<<grid_of(p->n_chunks, T / 32), T, 0, stream>>>(p->chunks, p->n_chunks, p->col, weight);
    k_weight_histogram<<<148, T, 0, stream>>>(weight, p->k, bins);
    std::vector<int32_t> h_bins(kWeightBins);
    std::vector<SplitRow> h_rows((size_t)p->n_heavy);
    DG_CUDA(cudaMemcpyAsync(h_bins.data(), bins, kWeightBins * sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaMemcpyAsync(h_rows.data(), d_rows, h_rows.size() * sizeof(SplitRow), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));

    // the most frequent columns, at most kMaxColumns, and none so rare that a tile could not reach kTileMin with its like
    int32_t least = kWeightBins - 1;
    int64_t columns = h_bins[kWeightBins - 1];
    while (least > 1 + kTileMin / kTileCols && columns + h_bins[least - 1] <= kMaxColumns) columns += h_bins[--least];
    if (columns < kTileCols || columns > kMaxColumns) return DG_OK;
    int32_t *d_count = bins + kWeightBins, *largest = d_count + 1;
    k_frequent_columns<<<grid_of(p->k, T), T, 0, stream>>>(weight, p->k, least, frequent, kMaxColumns, d_count);
    std::vector<int2> h_frequent((size_t)columns);
    DG_CUDA(cudaMemcpyAsync(h_frequent.data(), frequent, h_frequent.size() * sizeof(int2), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));
    std::sort(h_frequent.begin(), h_frequent.end(), [](const int2& a, const int2& b) { return a.y != b.y ? a.y > b.y : a.x < b.x; });
    std::vector<int32_t> h_columns(h_frequent.size());
    for (size_t i = 0; i < h_columns.size(); ++i) h_columns[i] = h_frequent[i].x;
    t->n_columns = (int32_t)columns;
    t->col_tiles = (int32_t)((columns + kTileCols - 1) / kTileCols);
    // longest rows first
    std::vector<int32_t> by_length(h_rows.size()), h_rank(h_rows.size());
    for (size_t i = 0; i < by_length.size(); ++i) by_length[i] = (int32_t)i;
    std::stable_sort(by_length.begin(), by_length.end(), [&](int32_t a, int32_t b) { return h_rows[a].len > h_rows[b].len; });
    for (size_t i = 0; i < by_length.size(); ++i) h_rank[by_length[i]] = (int32_t)i;

    const int32_t row_tiles = (p->n_heavy + kTileRows - 1) / kTileRows;
    const int64_t tiles = (int64_t)row_tiles * t->col_tiles;
    if (tiles > (int64_t)1 << 26) return DG_OK;
    int32_t *tile = nullptr, *rest = nullptr;
    if ((rc = upload(&t->columns, h_columns, stream)) || (rc = tmp.alloc(&tile, (size_t)tiles)) || (rc = tmp.alloc(&rest, (size_t)p->n_chunks + 1))) return rc;
    DG_CUDA(cudaMemcpyAsync(row_rank, h_rank.data(), h_rank.size() * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
    k_column_ranks<<<grid_of(columns, T), T, 0, stream>>>(t->columns, t->n_columns, col_rank);
    DG_CUDA(cudaMemsetAsync(tile, 0, (size_t)tiles * sizeof(int32_t), stream));
    const unsigned warps = grid_of(p->n_chunks, T / 32);
    k_tile_entries<0><<<warps, T, 0, stream>>>(p->chunks, p->n_chunks, p->col, val, row_rank, col_rank, t->col_tiles, tile, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
    std::vector<int32_t> h_tile((size_t)tiles);
    DG_CUDA(cudaMemcpyAsync(h_tile.data(), tile, h_tile.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));

    std::vector<dg_slab> slabs;
    std::vector<int32_t> h_cursor, slab_row_tile;
    int64_t entries = 0;
    double cost = 0;
    auto slab_cost = [](int32_t count) { return 2400.0 + 1.5 * std::max(0, count - 1024); };      // clocks, as measured
    for (int64_t i = 0; i < tiles; ++i) {
        const int32_t count = h_tile[i];
        h_tile[i] = -1;
        if (count < kTileMin) continue;
        h_tile[i] = (int32_t)slabs.size();
        slab_row_tile.push_back((int32_t)(i / t->col_tiles));
        h_cursor.push_back((int32_t)entries);
        slabs.push_back(dg_slab{(int32_t)(i % t->col_tiles), (int32_t)entries, count});
        entries += count;
        cost += slab_cost(count);
    }
    if (slabs.empty() || entries < p->nnz / 8) return DG_OK;       // the columns' images and another launch cost more than that saves

    // equal shares of the work for every CTA, cut again where the row tile changes
    int dev = 0, ctas = 0;
    DG_CUDA(cudaGetDevice(&dev));
    DG_CUDA(cudaDeviceGetAttribute(&ctas, cudaDevAttrMultiProcessorCount, dev));
    std::vector<dg_segment> segments;
    std::vector<int32_t> cta_segment(1, 0), tile_slot(row_tiles, 0), tile_parts(row_tiles, 0);
    double done = 0;
    for (size_t s = 0; s < slabs.size(); ++s) {
        const bool new_cta = (int)cta_segment.size() < ctas && done >= cost * (double)cta_segment.size() / ctas && s > 0;
        const bool new_row = s == 0 || slab_row_tile[s] != slab_row_tile[s - 1];
        if (new_cta) cta_segment.push_back((int32_t)segments.size());
        if (new_cta || new_row) {
            if (!segments.empty()) segments.back().slab1 = (int32_t)s;
            const int32_t rt = slab_row_tile[s], slot = (int32_t)segments.size();
            if (new_row) tile_slot[rt] = slot;
            ++tile_parts[rt];
            segments.push_back(dg_segment{(int32_t)s, (int32_t)slabs.size(), slot, 0});
        }
        done += slab_cost(slabs[s].count);
    }
    t->ctas = (int32_t)cta_segment.size();
    cta_segment.push_back((int32_t)segments.size());
    std::vector<int2> parts(h_rows.size());
    for (size_t h = 0; h < parts.size(); ++h) {
        const int32_t rt = h_rank[h] / kTileRows;
        parts[h] = make_int2(tile_slot[rt] * kTileRows + h_rank[h] % kTileRows, tile_parts[rt]);
    }

    int32_t* cursor = nullptr;
    if ((rc = tmp.alloc(&cursor, slabs.size()))) return rc;
    DG_CUDA(cudaMemcpyAsync(tile, h_tile.data(), h_tile.size() * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
    DG_CUDA(cudaMemcpyAsync(cursor, h_cursor.data(), h_cursor.size() * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
    k_tile_entries<1><<<warps, T, 0, stream>>>(p->chunks, p->n_chunks, p->col, val, row_rank, col_rank, t->col_tiles, tile, nullptr, rest, nullptr, nullptr, nullptr, nullptr);
    k_exclusive_sums<<<1, 1024, 0, stream>>>(rest, p->n_chunks);
    int32_t h_rest = 0;
    DG_CUDA(cudaMemcpyAsync(&h_rest, rest + p->n_chunks, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));
    if (h_rest != p->heavy_nnz - entries) return DG_ERR_STATE;     // cannot happen
    if ((rc = dg_pool_alloc((void**)&t->records, (size_t)entries * sizeof(uint2))) ||
        (rc = dg_pool_alloc((void**)&t->rest_col, std::max<size_t>(h_rest, 1) * sizeof(int32_t))) ||
        (rc = dg_pool_alloc((void**)&t->rest_val, std::max<size_t>(h_rest, 1) * sizeof(float))) || (rc = upload(&t->slabs, slabs, stream)) ||
        (rc = upload(&t->segments, segments, stream)) || (rc = upload(&t->cta_segment, cta_segment, stream)) || (rc = upload(&t->parts, parts, stream)))
        return rc;
    k_tile_entries<2><<<warps, T, 0, stream>>>(p->chunks, p->n_chunks, p->col, val, row_rank, col_rank, t->col_tiles, tile, cursor, rest, t->records, t->rest_col,
                                               t->rest_val, largest);
    // chunks of the rest, in the order of the column band they start in
    int32_t *chunk_first = nullptr, *bands = nullptr;
    if ((rc = tmp.alloc(&chunk_first, (size_t)p->n_heavy + 1)) || (rc = tmp.alloc(&bands, kBands + 1))) return rc;
    DG_CUDA(cudaMemsetAsync(bands, 0, kBands * sizeof(int32_t), stream));
    const unsigned row_blocks = grid_of(p->n_heavy, T);
    k_rest_chunks<0><<<row_blocks, T, 0, stream>>>(d_rows, p->n_heavy, first_slot, rest, p->chunk, t->rest_col, p->k, chunk_first, bands, nullptr);
    k_exclusive_sums<<<1, 1024, 0, stream>>>(chunk_first, p->n_heavy);
    k_rest_chunks<1><<<row_blocks, T, 0, stream>>>(d_rows, p->n_heavy, first_slot, rest, p->chunk, t->rest_col, p->k, chunk_first, bands, nullptr);
    k_exclusive_sums<<<1, 1024, 0, stream>>>(bands, kBands);
    DG_CUDA(cudaMemcpyAsync(&t->n_rest_chunks, chunk_first + p->n_heavy, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));
    if ((rc = dg_pool_alloc((void**)&t->rest_chunks, (size_t)t->n_rest_chunks * sizeof(dg_chunk)))) return rc;
    k_rest_chunks<2><<<row_blocks, T, 0, stream>>>(d_rows, p->n_heavy, first_slot, rest, p->chunk, t->rest_col, p->k, chunk_first, bands, t->rest_chunks);
    if ((rc = dg_pool_alloc(&t->value_sums, (size_t)t->ctas * kValueWarps * sizeof(ValueSum)))) return rc;
    k_value_sums<<<t->ctas, 32 * kValueWarps, 0, stream>>>(val, p->nnz, static_cast<ValueSum*>(t->value_sums));
    float h_largest = 0.f;
    DG_CUDA(cudaMemcpyAsync(&h_largest, largest, sizeof(float), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));
    DG_CUDA(cudaGetLastError());
    if (!(h_largest < kTileBound) || h_largest < kTileLeast) return DG_OK;
    t->least_operand = h_largest < 1.f ? kTileLeast / h_largest : kTileLeast;
    t->val = val;
    t->n_slabs = (int32_t)slabs.size();
    t->n_segments = (int32_t)segments.size();
    t->entries = entries;
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
