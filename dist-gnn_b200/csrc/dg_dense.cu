// Dense transform of the GCN layer on the 5th-generation tensor cores:  C[M x N] = act(A[M x K] * Bt[N x K]^T), fp32 in
// and out, for the tall-skinny shapes either side of the SpMM (Z*W and AG*W^T: light_dist_gnn/models/gcn.py:41, :49;
// M = rows of the rank's block, K and N <= 256).
//
// fp32 accuracy from TF32 tensor cores: every operand is cut into a TF32-exact head (sign, exponent, top 10 mantissa
// bits) and its residual tail, and the accumulator (fp32, in tensor memory) receives
//     A_head*B_head + A_head*B_tail + A_tail*B_head
// (the dropped tail*tail term is 2^-22 relative).  The small matrix Bt is split once on the host side of the call
// (dg_dense_split); A is split inside the kernel, in shared memory, on its way from TMA to the MMA.  The tensor cores
// ignore the low 13 bits of a TF32 operand (verified: identical bits with and without a masked copy), so the tile as
// loaded serves as head and only the tail is written.
//
// k_dense_nt: one CTA per 128-row tile.  Warp 0 drives TMA (128B-swizzled boxes of 32 K-columns: A rows, Bt head, Bt tail)
// through a 2-stage ring; warps 2-5 split A and later drain the accumulator (tcgen05.ld) to global memory with the
// optional ReLU / ReLU-backward mask; one thread of warp 1 issues the tcgen05.mma instructions (kind::tf32, 128 x N x 8,
// operands described by shared-memory matrix descriptors, accumulator in TMEM columns) and commits them to the mbarriers
// that recycle the stages.  k_dense_nt_pair: a CTA pair on every TPC walks over tiles of 256 rows with two accumulators and separate
// epilogue warps (wider results; by_pairs).  k_dense_tn (further down): the weight gradient X^T * G,
// both operands MN-major, split-K over the CTAs with periodic accumulator flushes.
// Every mbarrier wait is bounded; a role that gives up sets the status word and the CTA still frees its TMEM.
#include <cuda.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include "dg_internal.h"
#include "dg_umma.h"

namespace {

using namespace dg;

constexpr int BM = 128;             // rows per CTA tile (UMMA M)
constexpr int BK = 32;              // fp32 K-columns per stage = one 128-byte swizzle row
constexpr int STAGES = 2;
constexpr int kThreads = 192;

struct DenseArgs {
    float* C;
    int64_t ldc;
    int64_t M;
    int32_t N, K, n_pad;            // n_pad = N rounded up to 16 (UMMA N)
    uint32_t relu;
    const float* mask;              // optional [M x N]: the result is zeroed where mask <= 0 (ReLU backward), else nullptr
    int64_t ldm;
    int* status;
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// Shared-memory matrix descriptor of a K-major tile stored as 128-byte rows with the 128B swizzle: 8-row groups are
// 1024 bytes apart (stride byte offset), the leading byte offset is unused for this layout, descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);            // start address, 16-byte units
    d |= (uint64_t)1 << 16;                                   // leading byte offset (ignored with swizzle), 16-byte units
    d |= (uint64_t)(1024 >> 4) << 32;                         // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                                   // descriptor version for sm_100
    d |= (uint64_t)2 << 61;                                   // layout type: SWIZZLE_128B
    return d;
}
// The same for rows of 64 bytes with the 64B swizzle: 8-row groups are 512 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t smem_addr)
{
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
// Instruction descriptor for kind::tf32: fp32 accumulator, TF32 A and B, both K-major, shape 128 x n_pad.
__device__ __forceinline__ uint32_t umma_idesc_tf32(int n_pad)
{
    uint32_t d = 0;
    d |= 1u << 4;                                             // accumulator format: F32
    d |= 2u << 7;                                             // A format: TF32
    d |= 2u << 10;                                            // B format: TF32
    d |= (uint32_t)(n_pad >> 3) << 17;                        // N / 8
    d |= (uint32_t)(BM >> 4) << 24;                           // M / 16
    return d;
}
__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
}  // namespace

namespace {

// Epilogue of one warp: 32 rows of the accumulator (tensor-memory address `acc`, this warp's lane quarter included) to
// rows row0.. of C, with the optional ReLU and ReLU-backward mask.  A lane holds one row, so stores straight from the
// registers touch 32 cache lines an instruction (and so do the mask's loads); the piece goes through `stage` in shared memory
// (32 rows of 36 floats, conflict-free both ways) and leaves as whole 128-byte row pieces, four rows an instruction.
constexpr int kStagePitch = 36, kStageBytes = 32 * kStagePitch * 4;
__device__ __forceinline__ void store_rows(const DenseArgs& a, uint32_t acc, float* stage, int64_t row0, int lane)
{
    const bool vec = a.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0 &&
                     (!a.mask || (a.ldm % 4 == 0 && (reinterpret_cast<uintptr_t>(a.mask) & 15) == 0));
    const int rows = (int)min((int64_t)32, a.M - row0);
    for (int c0 = 0; c0 < a.n_pad; c0 += 32) {
        const bool pieces = vec && c0 + 32 <= a.N;                // whole 128-byte pieces of every row
        const int r4 = lane >> 3, col4 = c0 + (lane & 7) * 4;
        float4 mk[8];
        if (pieces && a.mask) {                                   // requested before the accumulator read so that both are in flight
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i * 4 + r4 < rows) mk[i] = __ldg(reinterpret_cast<const float4*>(a.mask + (row0 + i * 4 + r4) * a.ldm + col4));
        }
        uint32_t r[32];
        tmem_ld16(acc + (uint32_t)c0, r);
        if (c0 + 16 < a.n_pad) tmem_ld16(acc + (uint32_t)c0 + 16, r + 16);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float4* mine = reinterpret_cast<float4*>(stage + lane * kStagePitch);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            mine[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
        __syncwarp();
        if (pieces) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (i * 4 + r4 >= rows) continue;
                float4 v = *reinterpret_cast<const float4*>(stage + (i * 4 + r4) * kStagePitch + (lane & 7) * 4);
                if (a.relu) v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
                if (a.mask) {
                    if (!(mk[i].x > 0.f)) v.x = 0.f;
                    if (!(mk[i].y > 0.f)) v.y = 0.f;
                    if (!(mk[i].z > 0.f)) v.z = 0.f;
                    if (!(mk[i].w > 0.f)) v.w = 0.f;
                }
                __stcs(reinterpret_cast<float4*>(a.C + (row0 + i * 4 + r4) * a.ldc + col4), v);
            }
        } else if (c0 + lane < a.N) {                             // odd strides and the last columns: a row's floats side by side
            const int c = c0 + lane;
            for (int i0 = 0; i0 < rows; i0 += 8) {                // eight rows' mask values in flight
                float mrow[8];
                if (a.mask) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (i0 + i < rows) mrow[i] = __ldg(a.mask + (row0 + i0 + i) * a.ldm + c);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i0 + i >= rows) break;
                    float v = stage[(i0 + i) * kStagePitch + lane];
                    if (a.relu) v = fmaxf(v, 0.f);
                    if (a.mask && !(mrow[i] > 0.f)) v = 0.f;
                    __stcs(a.C + (row0 + i0 + i) * a.ldc + c, v);
                }
            }
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kThreads, 1)
k_dense_nt(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBh,
           const __grid_constant__ CUtensorMap tmBt, const DenseArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;                 // swizzled tiles need 1024-byte alignment
    unsigned char* gbase = smem_raw + (base - raw);
    const int b_bytes = a.n_pad * 128;                            // one slab of Bt: n_pad rows x 128 bytes
    const int stage_bytes = 2 * BM * 128 + 2 * b_bytes;           // A head, A tail, Bt head, Bt tail
    const uint32_t bars = base + STAGES * stage_bytes;
    const uint32_t full0 = bars, ready0 = bars + 8 * STAGES, empty0 = bars + 16 * STAGES, acc_full = bars + 24 * STAGES, done = acc_full + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + STAGES * stage_bytes + 24 * STAGES + 16);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t m0 = (int64_t)blockIdx.x * BM;
    const int nslabs = (a.K + BK - 1) / BK;
    int tmem_cols = 32;
    while (tmem_cols < a.n_pad) tmem_cols <<= 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(ready0 + 8 * s, 128);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {                                              // one warp allocates the accumulator columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {                                          // TMA producer
            int i = 0;
            for (; i < nslabs && ok; ++i) {
                const int s = i % STAGES, u = i / STAGES;
                if (u > 0) ok = mbar_wait(empty0 + 8 * s, (u - 1) & 1);
                if (!ok) break;
                const uint32_t st = base + s * stage_bytes;
                mbar_expect_tx(full0 + 8 * s, BM * 128 + 2 * b_bytes);
                tma_load_2d(st, &tmA, i * BK, (int)m0, full0 + 8 * s);
                tma_load_2d(st + 2 * BM * 128, &tmBh, i * BK, 0, full0 + 8 * s);
                tma_load_2d(st + 2 * BM * 128 + b_bytes, &tmBt, i * BK, 0, full0 + 8 * s);
            }
            await_loads(full0, i, STAGES);
        }
    } else if (warp == 1) {
        if (lane == 0) {                                          // MMA issuer
            const uint32_t idesc = umma_idesc_tf32(a.n_pad);
            for (int i = 0; i < nslabs && ok; ++i) {
                const int s = i % STAGES, u = i / STAGES;
                ok = mbar_wait(ready0 + 8 * s, u & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t st = base + s * stage_bytes;
                const uint64_t a_head = umma_desc_sw128(st), a_tail = umma_desc_sw128(st + BM * 128);
                const uint64_t b_head = umma_desc_sw128(st + 2 * BM * 128), b_tail = umma_desc_sw128(st + 2 * BM * 128 + b_bytes);
#pragma unroll
                for (int k = 0; k < BK / 8; ++k) {               // 8 TF32 columns = 32 bytes per MMA: +2 in 16-byte units
                    umma_tf32(tmem, a_tail + 2 * k, b_head + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma_tf32(tmem, a_head + 2 * k, b_tail + 2 * k, idesc, 1u);
                    umma_tf32(tmem, a_head + 2 * k, b_head + 2 * k, idesc, 1u);
                }
                umma_commit(empty0 + 8 * s);                      // the stage is free once these MMAs have read it
            }
            if (ok) umma_commit(acc_full);
            await_mmas(done);
        }
    } else {
        const int t = threadIdx.x - 64;                           // 0..127: split A, then drain the accumulator
        for (int i = 0; i < nslabs && ok; ++i) {
            const int s = i % STAGES, u = i / STAGES;
            ok = mbar_wait(full0 + 8 * s, u & 1);
            if (!ok) break;
            float4* head = reinterpret_cast<float4*>(gbase + (size_t)s * stage_bytes);
            float4* tail = head + BM * 128 / 16;
#pragma unroll 4
            for (int j = t; j < BM * 128 / 16; j += 128) {
                const float4 x = head[j];
                float4 h;
                h.x = __uint_as_float(__float_as_uint(x.x) & 0xFFFFE000u); h.y = __uint_as_float(__float_as_uint(x.y) & 0xFFFFE000u);
                h.z = __uint_as_float(__float_as_uint(x.z) & 0xFFFFE000u); h.w = __uint_as_float(__float_as_uint(x.w) & 0xFFFFE000u);
                head[j] = h;
                tail[j] = make_float4(x.x - h.x, x.y - h.y, x.z - h.z, x.w - h.w);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(ready0 + 8 * s);
        }
        if (ok) ok = mbar_wait(acc_full, 0);
        ok = __all_sync(0xffffffffu, ok);                         // tcgen05.ld below is warp-collective: decide as a warp
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int q = warp & 3;                               // a warp may only read its own quarter of the TMEM lanes
            // every load has landed and every MMA has read its operands: the stages are free for the staging of the rows
            if (m0 + q * 32 < a.M)
                store_rows(a, tmem + ((uint32_t)(q * 32) << 16), reinterpret_cast<float*>(gbase + q * kStageBytes), m0 + q * 32, lane);
        }
    }
    if (!ok) atomicExch(a.status, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
}

// The same product by CTA pairs (cta_group::2), one pair on the two SMs of every TPC, that walk over tiles of 256 rows: a CTA holds
// 128 rows of A and half the rows of Bt, the tensor cores of both read both halves of Bt, and each CTA's tensor memory receives its 128
// rows of the result.  Two accumulators (columns 0 / 256) and separate warps for the operand split and the epilogue, so that tile t is
// read out and stored while tile t+1 is loaded, split and multiplied.
// Warps: 0 TMA, 1 MMA issue (even CTA) + tensor-memory allocation, 2-5 split A, 6-13 epilogue (lane quarter w % 4; two warps a quarter take
// its 32-column pieces in turn).
// The ring holds half slabs of 16 columns (64-byte rows, 64B swizzle), as many as fit (6 at 256 columns, 10 at most).
// Barriers: full (own CTA, TMA), ready (even CTA: the split warps of both), empty and acc_full (both CTAs, by commit), acc_empty (even CTA:
// the epilogue warps of both).
//
// What bounds it: at 256 x 256 the MMAs (tensor pipe 68 %, with the mask 64 and DRAM 60 %; a single CTA's shared memory was busy with fetching both operands' 12 KB for
// every MMA and refilling Bt's 512 KB for every 128 rows, which a pair halves), below some 100 columns of A DRAM and the epilogue.
// 2,449,029 rows (us, one CTA per SM with four epilogue warps -> pair): 256 -> 256 1,600 -> 1,535, with the mask 1,930 -> 1,720;
// 100 -> 256 1,100 -> 895; 47 -> 256 with the mask 1,600 -> 1,110; 602 -> 256 4,280 -> 3,540; 256 -> 128 1,540 -> 1,065 (one tile per
// CTA).  150,001 rows: 256 -> 256 102 -> 100, with the mask 126 -> 109; 100 -> 256 76 -> 61.
// The warp that issues the MMAs walks through its loop together and one lane issues (elect_one).  With one lane in the whole loop the issue
// itself was the limit: 125 clocks an MMA, 197 with the tail passes behind the head passes, whatever the width and however many stages.  ns per
// half slab, 3,000 rows: 96 columns 386 -> 320, 160 600 -> 293, 256 599 -> 446.  us, one CTA -> pair -> this: 150,001 rows 256 -> 160 76 -> 84 -> 68,
// 256 -> 192 82 -> 85 -> 74, 256 -> 256 98 -> 94 -> 90; 3,000 rows 256 -> 160 13.6 -> 15.0 -> 12.1; 2,449,029 rows (in turn, 20 ms between launches)
// 256 -> 256 1,492 -> 1,428, with the mask 1,678 -> 1,574, 602 -> 256 3,423 -> 3,238, 256 -> 128 1,017 -> 904.
constexpr int PK = 16, kMaxPairStages = 10, kSplitWarps = 4, kEpilogueWarps = 8;
constexpr int kThreadsPair = 32 * (2 + kSplitWarps + kEpilogueWarps);
constexpr int kPieceBytes = 32 * 32 * 4;                          // staging of an epilogue warp: 32 rows x 32 columns
constexpr int kPairBarBytes = 8 * (3 * kMaxPairStages + 5) + 8;

__device__ __forceinline__ void umma_tf32_pair(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

template <bool MASK>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreadsPair, 1)
k_dense_nt_pair(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBh,
                const __grid_constant__ CUtensorMap tmBt, const DenseArgs a, const int n_tiles, const int stages)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* gbase = smem_raw + (base - raw);
    constexpr int a_bytes = BM * PK * 4;
    const int half_n = a.n_pad / 2, b_bytes = half_n * PK * 4;
    const int stage_bytes = 2 * a_bytes + 2 * b_bytes;            // A head, A tail, Bt head, Bt tail
    const int staging = stages * stage_bytes;                     // the epilogue warps' row pieces
    const uint32_t bars = base + staging + kEpilogueWarps * kPieceBytes;
    const uint32_t full0 = bars, ready0 = bars + 8 * kMaxPairStages, empty0 = bars + 16 * kMaxPairStages;
    const uint32_t acc_full0 = bars + 24 * kMaxPairStages, acc_empty0 = acc_full0 + 16, done = acc_empty0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + staging + kEpilogueWarps * kPieceBytes + 24 * kMaxPairStages + 40);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int nhalves = (a.K + PK - 1) / PK;
    constexpr int kTmemCols = 512;                                // two accumulators of up to 256 columns

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(ready0 + 8 * s, 2 * kSplitWarps);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full0 + 8 * b, 1);
            mbar_init(acc_empty0 + 8 * b, 2 * kEpilogueWarps);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {                                          // TMA producer: one ring of stages across all tiles
            int it = 0, s = 0, phase = 1;
            for (int tile = pair; tile < n_tiles && ok; tile += pairs) {
                const int row0 = (int)((int64_t)tile * (2 * BM) + rank * BM);      // rows beyond the matrix arrive as zeros
                for (int i = 0; i < nhalves; ++i, ++it) {
                    if (it >= stages) ok = mbar_wait(empty0 + 8 * s, phase);
                    if (!ok) break;
                    const uint32_t st = base + s * stage_bytes;
                    mbar_expect_tx(full0 + 8 * s, a_bytes + 2 * b_bytes);
                    tma_load_2d(st, &tmA, i * PK, row0, full0 + 8 * s);
                    tma_load_2d(st + 2 * a_bytes, &tmBh, i * PK, rank * half_n, full0 + 8 * s);
                    tma_load_2d(st + 2 * a_bytes + b_bytes, &tmBt, i * PK, rank * half_n, full0 + 8 * s);
                    if (++s == stages) s = 0, phase ^= 1;
                }
            }
            await_loads(full0, it, stages);
        }
    } else if (warp == 1) {
        if (rank == 0) {                                          // MMA issuer: the warp waits and counts together, one lane issues
            const bool issuer = elect_one(), tails_last = a.n_pad > 128;
            // the issuing lane polls: all of them polling held the epilogue up (306,128 rows 32 -> 112 45.1 us, 46.7)
            auto wait = [&](uint32_t bar, int parity) { return __any_sync(0xffffffffu, issuer && mbar_wait(bar, parity)) != 0; };
            const uint32_t idesc = umma_idesc_tf32(a.n_pad) + ((uint32_t)(BM >> 4) << 24);      // 2 * BM rows
            const uint64_t desc0 = umma_desc_sw64(base);
            const uint32_t next_stage = (uint32_t)stage_bytes >> 4, tail = a_bytes >> 4, b_head = 2 * tail, b_tail = b_head + ((uint32_t)b_bytes >> 4);
            int s = 0, phase = 0, lt = 0;
            for (int tile = pair; tile < n_tiles && ok; tile += pairs, ++lt) {
                const int b = lt & 1, v = lt >> 1;
                if (lt >= 2) ok = wait(acc_empty0 + 8 * b, (v - 1) & 1);     // both epilogues have drained this accumulator
                const uint32_t acc = tmem + (uint32_t)(b * 256);
                for (int i = 0; i < nhalves && ok; i += 2) {
                    // The tensor cores read a TF32 operand from a 32-bit container and ignore its low 13 bits (verified: identical
                    // bits with a masked copy), so the tile as TMA delivered it is the head.  The order of the additions decides the last
                    // bits, and those the sign of a ReLU's input: over a slab of two halves, the tail passes come behind the head
                    // passes (wide results) or beside them (narrow ones), as in the kernels of one CTA.
                    const int s0 = s, halves = min(2, nhalves - i);
                    for (int h = 0; h < halves && ok; ++h) {
                        ok = wait(ready0 + 8 * s, phase);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint64_t d = desc0 + (uint32_t)s * next_stage;
                        if (issuer) {
#pragma unroll
                            for (int k = 0; k < PK / 8; ++k) {    // 8 TF32 columns = 32 bytes per MMA: +2 in 16-byte units
                                const uint32_t add = i > 0 || h > 0 || k > 0 ? 1u : 0u;
                                if (!tails_last) umma_tf32_pair(acc, d + tail + 2 * k, d + b_head + 2 * k, idesc, add);
                                umma_tf32_pair(acc, d + 2 * k, d + b_tail + 2 * k, idesc, tails_last ? add : 1u);
                                umma_tf32_pair(acc, d + 2 * k, d + b_head + 2 * k, idesc, 1u);
                            }
                            if (!tails_last) umma_commit_pair(empty0 + 8 * s);
                        }
                        __syncwarp();
                        if (++s == stages) s = 0, phase ^= 1;
                    }
                    for (int h = 0, t = s0; tails_last && h < halves && ok; ++h) {
                        const uint64_t d = desc0 + (uint32_t)t * next_stage;
                        if (issuer) {
#pragma unroll
                            for (int k = 0; k < PK / 8; ++k) umma_tf32_pair(acc, d + tail + 2 * k, d + b_head + 2 * k, idesc, 1u);
                            umma_commit_pair(empty0 + 8 * t);
                        }
                        __syncwarp();
                        if (++t == stages) t = 0;
                    }
                }
                if (ok && issuer) umma_commit_pair(acc_full0 + 8 * b);
                __syncwarp();
            }
            if (issuer) await_mmas_pair(done);
            __syncwarp();
        } else if (lane == 0) {
            mbar_wait(done, 0);
        }
    } else if (warp < 2 + kSplitWarps) {
        const int t = threadIdx.x - 64;                           // split the A half slab of every stage
        const uint32_t leader_ready0 = in_leader(ready0);
        int s = 0, phase = 0;
        for (int tile = pair; tile < n_tiles && ok; tile += pairs) {
            for (int i = 0; i < nhalves; ++i) {
                ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, phase));
                if (!ok) break;
                const float4* head = reinterpret_cast<const float4*>(gbase + (size_t)s * stage_bytes) + t;
                float4* tail = reinterpret_cast<float4*>(gbase + (size_t)s * stage_bytes + a_bytes) + t;
                float4 x[a_bytes / 16 / (32 * kSplitWarps)];
#pragma unroll
                for (int j = 0; j < a_bytes / 16 / (32 * kSplitWarps); ++j) x[j] = head[j * 32 * kSplitWarps];
#pragma unroll
                for (int j = 0; j < a_bytes / 16 / (32 * kSplitWarps); ++j) {
                    float4 h;
                    h.x = __uint_as_float(__float_as_uint(x[j].x) & 0xFFFFE000u); h.y = __uint_as_float(__float_as_uint(x[j].y) & 0xFFFFE000u);
                    h.z = __uint_as_float(__float_as_uint(x[j].z) & 0xFFFFE000u); h.w = __uint_as_float(__float_as_uint(x[j].w) & 0xFFFFE000u);
                    tail[j * 32 * kSplitWarps] = make_float4(x[j].x - h.x, x[j].y - h.y, x[j].z - h.z, x[j].w - h.w);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_ready0 + 8 * s);
                if (++s == stages) s = 0, phase ^= 1;
            }
        }
    } else {
        const int q = warp & 3, first = (warp - 2 - kSplitWarps) / 4 * 32;      // a warp may only read its own quarter of the TMEM lanes
        constexpr int step = kEpilogueWarps / 4 * 32;
        const uint32_t leader_acc_empty0 = in_leader(acc_empty0);
        float4* stage = reinterpret_cast<float4*>(gbase + staging + (warp - 2 - kSplitWarps) * kPieceBytes);
        const bool vec = a.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0 &&
                         (!MASK || (a.ldm % 4 == 0 && (reinterpret_cast<uintptr_t>(a.mask) & 15) == 0));
        const int r4 = lane >> 3, piece = lane & 7;
        int lt = 0;
        for (int tile = pair; tile < n_tiles; tile += pairs, ++lt) {
            const int b = lt & 1, v = lt >> 1;
            const int64_t row0 = (int64_t)tile * (2 * BM) + rank * BM + q * 32;
            const int rows = (int)max((int64_t)0, min((int64_t)32, a.M - row0));
            const uint32_t acc = tmem + (uint32_t)(b * 256) + ((uint32_t)(q * 32) << 16);
            for (int c0 = first; c0 < a.n_pad; c0 += step) {
                const bool whole = vec && c0 + 32 <= a.N;         // 128-byte pieces of every row, four rows an instruction
                [[maybe_unused]] float4 mk[8];
                if (MASK && whole) {                              // under way while the accumulator is waited for and read
                    const float* m = a.mask + (row0 + r4) * a.ldm + c0 + piece * 4;
#pragma unroll
                    for (int i = 0; i < 8; ++i, m += 4 * a.ldm)
                        if (i * 4 + r4 < rows) mk[i] = __ldg(reinterpret_cast<const float4*>(m));
                }
                if (c0 == first) {
                    ok = __all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * b, v & 1));     // tcgen05.ld is warp-collective
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                {
                    uint32_t r[32];
                    tmem_ld16(acc + (uint32_t)c0, r);
                    tmem_ld16(acc + (uint32_t)c0 + 16, r + 16);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c0 + step >= a.n_pad) {                   // the accumulator has been read: its next tile may start
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(leader_acc_empty0 + 8 * b);
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j)                   // a lane holds one row: through shared memory, conflict-free both ways
                        stage[lane * 8 + (j ^ (lane & 7))] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                }
                __syncwarp();
                if (whole) {
                    float4 x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = stage[(i * 4 + r4) * 8 + (piece ^ ((i * 4 + r4) & 7))];
                    float* c = a.C + (row0 + r4) * a.ldc + c0 + piece * 4;
#pragma unroll
                    for (int i = 0; i < 8; ++i, c += 4 * a.ldc) {
                        if (a.relu) x[i] = make_float4(fmaxf(x[i].x, 0.f), fmaxf(x[i].y, 0.f), fmaxf(x[i].z, 0.f), fmaxf(x[i].w, 0.f));
                        if (MASK) {
                            if (!(mk[i].x > 0.f)) x[i].x = 0.f;
                            if (!(mk[i].y > 0.f)) x[i].y = 0.f;
                            if (!(mk[i].z > 0.f)) x[i].z = 0.f;
                            if (!(mk[i].w > 0.f)) x[i].w = 0.f;
                        }
                        if (i * 4 + r4 < rows) __stcs(reinterpret_cast<float4*>(c), x[i]);
                    }
                } else if (c0 + lane < a.N) {                     // odd strides and the last columns: a row's floats side by side
                    const float* flat = reinterpret_cast<const float*>(stage);
                    for (int i0 = 0; i0 < rows; i0 += 8) {        // eight rows' mask values in flight
                        [[maybe_unused]] float mrow[8];
                        if (MASK) {
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (i0 + i < rows) mrow[i] = __ldg(a.mask + (row0 + i0 + i) * a.ldm + c0 + lane);
                        }
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            if (i0 + i >= rows) break;
                            float x = flat[((i0 + i) * 8 + ((lane >> 2) ^ ((i0 + i) & 7))) * 4 + (lane & 3)];
                            if (a.relu) x = fmaxf(x, 0.f);
                            if (MASK && !(mrow[i] > 0.f)) x = 0.f;
                            __stcs(a.C + (row0 + i0 + i) * a.ldc + c0 + lane, x);
                        }
                    }
                }
                __syncwarp();
            }
            if (!ok) break;
        }
    }
    if (!ok) atomicExch(a.status, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync();                                               // no CTA leaves while the other's MMAs read its operands or arrive at its barriers
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

__global__ void k_tf32_split(const float* __restrict__ src, float* __restrict__ head, float* __restrict__ tail, int64_t count)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float x = src[i];
    const float h = __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
    head[i] = h;
    tail[i] = x - h;
}

// Heads and tails of whole operands, transposed on the way where asked (32 x 32 tiles through shared memory, so that both
// sides are coalesced), rows zero-filled up to ldb.  One launch splits every weight of a network: the operands are a few
// hundred kilobytes, so a launch each costs more than the work.
constexpr int kSplitJobs = 16;
struct SplitJobs {
    dg_split_job job[kSplitJobs];
    int first_tile[kSplitJobs + 1];                               // running count of 32 x 32 tiles
    int count;
};

__global__ void __launch_bounds__(256) k_tf32_split_operands(const __grid_constant__ SplitJobs jobs)
{
    __shared__ float tile[32][33];
    int j = 0;
    while (j + 1 < jobs.count && (int)blockIdx.x >= jobs.first_tile[j + 1]) ++j;
    const dg_split_job& s = jobs.job[j];
    const int local = (int)blockIdx.x - jobs.first_tile[j], k_tiles = (int)((s.ldb + 31) / 32);
    const int k0 = local % k_tiles * 32, n0 = local / k_tiles * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int n = s.transposed ? n0 + tx : n0 + r, k = s.transposed ? k0 + r : k0 + tx;
        const float x = n < s.N && k < s.K ? s.w[s.transposed ? (int64_t)k * s.ldw + n : (int64_t)n * s.ldw + k] : 0.f;
        if (s.transposed) tile[tx][r] = x; else tile[r][tx] = x;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int n = n0 + r, k = k0 + tx;
        if (n >= s.N || k >= s.ldb) continue;
        const float x = tile[r][tx];
        const float h = __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
        s.head[(int64_t)n * s.ldb + k] = h;
        s.tail[(int64_t)n * s.ldb + k] = x - h;
    }
}

// Raises a kernel's dynamic shared-memory limit to the most a CTA can have, once per device instead of before every launch.
int allow_smem(const void* kernel, std::atomic<bool>* done)
{
    int dev = 0;
    DG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return DG_ERR_STATE;
    if (done[dev].load(std::memory_order_relaxed)) return DG_OK;
    DG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    done[dev].store(true, std::memory_order_relaxed);
    return DG_OK;
}

int sm_count()
{
    static std::atomic<int> count[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int n = count[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        count[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

}  // namespace

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled()
{
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// 2-D fp32 row-major matrix [rows x cols] with leading dimension ld, boxes of box_cols (32: 128B swizzle, 16: 64B swizzle) columns x box_rows rows,
// out-of-range elements read as zero.
int make_map(CUtensorMap* map, const float* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows, int box_cols = BK)
{
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return DG_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == BK ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? DG_OK : DG_ERR_UNSUPPORTED;
}

// Which of the two kernels multiplies; an element is the same sum in the same order in both.  n_pad: columns rounded up to 16.
// Up to 80 columns two one-tile CTAs fit an SM.  While all of them are resident at once, and for no more than one wave of those of up to 128
// columns, there is no next tile for a pair to overlap with, and its cluster barriers and remote arrivals are not won back
// unless the depth is large or ends in a half slab, which spares it padding.  us, one tile per CTA against pair:
//   10,000 rows 64 -> 96 6.0 and 6.5, 64 -> 80 6.6 and 7.1, 128 -> 80 8.2 and 8.6; 100 -> 128 9.0 and 8.0 (pair), 128 -> 96 7.8 and 7.6 (pair), 256 -> 80 11.5 and 10.9 (pair)
//   25,000 rows 64 -> 80 8.0 and 9.7, 256 -> 72 14.9 and 17.1; 64 -> 96 10.8 and 8.5 (pair: a second wave)
// With more rows the pair wins (150,001 rows 100 -> 72 40.6 and 31.7, 256 -> 80 58 and 53, 256 -> 128 96 and 59) but for shallow products up to 80
// columns with the mask, which wait for its rows and have more warps to do so as two CTAs (150,001 rows 64 -> 65 57 and 61, 100,000 rows
// 64 -> 80 26.8 and 30.7).  Up to 64 columns the line was drawn when a pair issued its MMAs more slowly (256 -> 47 860 and 895; now 830 and 701).
bool by_pairs(int64_t M, int n_pad, int K, bool masked, int sms)
{
    if (n_pad <= 64) return false;
    const int64_t tiles = (M + BM - 1) / BM;
    const bool half_slab = (K - 1) % BK < BK / 2;
    if (tiles <= sms) return n_pad > 128 || half_slab || K > (n_pad > 80 ? 96 : 128);
    return n_pad > 80 || (tiles > 2 * sms && (!masked || K > 64));
}

}  // namespace

extern "C" int dg_dense_split(const float* src, float* head, float* tail, int64_t count, void* stream)
{
    if (count < 0) return DG_ERR_DIMS;
    if (count == 0) return DG_OK;
    if (!src || !head || !tail) return DG_ERR_NULL;
    k_tf32_split<<<(unsigned)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(src, head, tail, count);
    return (int)cudaGetLastError();
}

extern "C" int dg_dense_split_operands(const dg_split_job* host_jobs, int32_t count, void* stream)
{
    if (count < 0) return DG_ERR_DIMS;
    if (count > 0 && !host_jobs) return DG_ERR_NULL;
    for (int32_t i = 0; i < count; ++i) {
        const dg_split_job& s = host_jobs[i];
        if (s.N < 0 || s.K < 0 || s.ldb < s.K || s.ldb >= ((int64_t)1 << 24) || s.ldw < (s.transposed ? s.N : s.K)) return DG_ERR_DIMS;
        if (s.N > 0 && s.K > 0 && (!s.w || !s.head || !s.tail)) return DG_ERR_NULL;
    }
    for (int32_t i0 = 0; i0 < count; i0 += kSplitJobs) {
        SplitJobs jobs{};
        int64_t tiles = 0;
        for (int32_t i = i0; i < count && i < i0 + kSplitJobs; ++i) {
            if (host_jobs[i].N == 0 || host_jobs[i].K == 0) continue;
            jobs.job[jobs.count] = host_jobs[i];
            jobs.first_tile[jobs.count++] = (int)tiles;
            tiles += (host_jobs[i].ldb + 31) / 32 * ((host_jobs[i].N + 31) / 32);
            if (tiles >= ((int64_t)1 << 31)) return DG_ERR_UNSUPPORTED;
            jobs.first_tile[jobs.count] = (int)tiles;
        }
        if (tiles > 0) k_tf32_split_operands<<<(unsigned)tiles, 256, 0, (cudaStream_t)stream>>>(jobs);
    }
    return (int)cudaGetLastError();
}

extern "C" int dg_dense_supported(int64_t M, int32_t N, int32_t K, int64_t lda, int64_t ldb, const void* A, const void* Bh, const void* Bt)
{
    if (M <= 0 || N <= 0 || K <= 0 || M >= ((int64_t)1 << 31)) return 0;
    if (lda % 4 || ldb % 4 || lda < K || ldb < K) return 0;                       // TMA strides are multiples of 16 bytes
    if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(Bh) | reinterpret_cast<uintptr_t>(Bt)) & 15) return 0;
    return encode_tiled() != nullptr;
}

extern "C" int dg_dense_nt(const float* A, int64_t lda, const float* Bt_head, const float* Bt_tail, int64_t ldb, float* C,
                           int64_t ldc, int64_t M, int32_t N, int32_t K, int32_t relu, void* stream)
{
    return dg_dense_nt_masked(A, lda, Bt_head, Bt_tail, ldb, C, ldc, M, N, K, relu, nullptr, 0, stream);
}

extern "C" int dg_dense_nt_masked(const float* A, int64_t lda, const float* Bt_head, const float* Bt_tail, int64_t ldb, float* C,
                                  int64_t ldc, int64_t M, int32_t N, int32_t K, int32_t relu, const float* mask, int64_t ldm,
                                  void* stream)
{
    if (!A || !Bt_head || !Bt_tail || !C) return DG_ERR_NULL;
    if (ldc < N || (mask && ldm < N)) return DG_ERR_DIMS;
    if (!dg_dense_supported(M, N, K, lda, ldb, A, Bt_head, Bt_tail)) return DG_ERR_UNSUPPORTED;
    if (N > 256) {      // a result wider than one accumulator: panels of 256 columns, A is streamed once per panel
        for (int32_t n0 = 0; n0 < N; n0 += 256) {
            const int rc = dg_dense_nt_masked(A, lda, Bt_head + (int64_t)n0 * ldb, Bt_tail + (int64_t)n0 * ldb, ldb, C + n0, ldc, M,
                                              N - n0 < 256 ? N - n0 : 256, K, relu, mask ? mask + n0 : nullptr, ldm, stream);
            if (rc) return rc;
        }
        return DG_OK;
    }
    DenseArgs a{};
    a.C = C; a.ldc = ldc; a.M = M; a.N = N; a.K = K; a.n_pad = (N + 15) / 16 * 16; a.relu = relu ? 1u : 0u;
    a.mask = mask; a.ldm = ldm;
    a.status = dg_status_word();
    if (!a.status) return DG_ERR_STATE;
    const int sms = sm_count();
    if (sms <= 0) return DG_ERR_STATE;
    const bool pair = by_pairs(M, a.n_pad, K, mask != nullptr, sms);
    CUtensorMap tmA, tmBh, tmBt;
    int rc;
    if (!pair) {
        const size_t smem = STAGES * (size_t)BK * 4 * (2 * BM + 2 * a.n_pad) + 24 * STAGES + 48 + 1024;
        if ((rc = make_map(&tmA, A, M, K, lda, BM)) || (rc = make_map(&tmBh, Bt_head, N, K, ldb, a.n_pad)) ||
            (rc = make_map(&tmBt, Bt_tail, N, K, ldb, a.n_pad)))
            return rc;
        static std::atomic<bool> granted[64];
        if ((rc = allow_smem((const void*)k_dense_nt, granted))) return rc;
        k_dense_nt<<<(unsigned)((M + BM - 1) / BM), kThreads, smem, (cudaStream_t)stream>>>(tmA, tmBh, tmBt, a);
        return (int)cudaGetLastError();
    }
    a.n_pad = (N + 31) / 32 * 32;                                 // both CTAs hold whole groups of 16 of its rows
    if ((rc = make_map(&tmA, A, M, K, lda, BM, PK)) || (rc = make_map(&tmBh, Bt_head, N, K, ldb, a.n_pad / 2, PK)) ||
        (rc = make_map(&tmBt, Bt_tail, N, K, ldb, a.n_pad / 2, PK)))
        return rc;
    const size_t stage = (size_t)PK * 4 * (2 * BM + a.n_pad), rest = kEpilogueWarps * kPieceBytes + kPairBarBytes + 1024;
    const int stages = (int)std::min<size_t>(kMaxPairStages, (227 * 1024 - rest) / stage);
    static std::atomic<bool> granted[64];
    static std::atomic<bool> granted_masked[64];
    if ((rc = mask ? allow_smem((const void*)k_dense_nt_pair<true>, granted_masked) : allow_smem((const void*)k_dense_nt_pair<false>, granted))) return rc;
    const int n_tiles = (int)((M + 2 * BM - 1) / (2 * BM));
    (mask ? k_dense_nt_pair<true> : k_dense_nt_pair<false>)<<<2u * (unsigned)std::min(n_tiles, sms / 2), kThreadsPair, stages * stage + rest, (cudaStream_t)stream>>>(
        tmA, tmBh, tmBt, a, n_tiles, stages);
    return (int)cudaGetLastError();
}

extern "C" int dg_dense_status(int* host_status, void* stream)
{
    if (!host_status) return DG_ERR_NULL;
    int* w = dg_status_word();
    if (!w) return DG_ERR_STATE;
    DG_CUDA(cudaMemcpyAsync(host_status, w, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    DG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return DG_OK;
}

extern "C" int dg_dense_status_reset(void* stream)
{
    int* w = dg_status_word();
    if (!w) return DG_ERR_STATE;
    DG_CUDA(cudaMemsetAsync(w, 0, sizeof(int), (cudaStream_t)stream));
    return DG_OK;
}

// Self-test of the give-up path every dense kernel shares: a CTA allocates tensor-memory columns as the kernels do, then
// waits - with a limit of a few thousand polls - on an mbarrier that nothing ever arrives at.  The wait runs out, the
// thread records it in `flag`, the CTA frees its tensor memory and the kernel returns normally.  Nothing traps or spins
// without bound; the context stays usable, which the caller can check by running a product afterwards.
namespace {
__global__ void __launch_bounds__(64, 1) k_dense_wait_selftest(int* flag, int limit)
{
    __shared__ __align__(8) unsigned long long bar_storage;
    __shared__ uint32_t tmem_slot;
    const uint32_t bar = smem_u32(&bar_storage);
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(32) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (threadIdx.x == 0 && !mbar_wait(bar, 0, limit)) atomicExch(flag, 1);      // nobody arrives: the wait must give up
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(32) : "memory");
}
}  // namespace

extern "C" int dg_dense_wait_selftest(int* host_gave_up, void* stream)
{
    if (!host_gave_up) return DG_ERR_NULL;
    int* flag = nullptr;
    DG_CUDA(cudaMalloc((void**)&flag, sizeof(int)));
    cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), (cudaStream_t)stream);
    if (e == cudaSuccess) {
        k_dense_wait_selftest<<<1, 64, 0, (cudaStream_t)stream>>>(flag, 4096);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(host_gave_up, flag, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    cudaFree(flag);
    return (int)e;
}

// ---- weight-gradient product  D[Km x Nn] = X[n x Km]^T * G[n x Nn]  (models/gcn.py:50) -------------------------------------
// The reduction runs over the n rows of the block, so both operands are read "MN-major": a TMA box of 32 columns x 16
// rows lands as 16 rows of 128 bytes in the 32-byte-atom variant of the 128B swizzle, which is the one layout the tensor
// cores accept for 32-bit MN-major operands (the plain 128B swizzle makes them read zeros); the boxes of one operand lie
// 2048 bytes apart (leading byte offset), 4-row groups 512 bytes.  The rows are cut into as many ranges as there are CTAs; a range is
// streamed through a ring, BOTH operands are split into TF32 head and tail in shared memory, the three
// passes are accumulated into fp32 accumulators in tensor memory, and the range's partial D goes to scratch; a second
// kernel adds the partials of all ranges in order (deterministic).
//
// One operand, P, lies along the 128 rows of an MMA, the other, Q, along its up to 256 columns.  As one lane alone issues them here, an MMA
// takes some 130 clocks for 128 rows however few columns it has, so P is the narrower operand (256 x 47: 47 columns padded to 128 rows, once
// over Q's 256, instead of twice over 48) and D comes out transposed where that is G.  Where both are wider than 128 the
// CTAs of a pair (cta_group::2) hold 128 columns of P and half of Q each, and take two ranges, one after the other.  An element of D is
// the same sum in the same order either way.
namespace {

constexpr int TN_ROWS = 16;                     // rows of X / G per stage (two MMA k-steps of 8)
constexpr int TN_BOX_BYTES = TN_ROWS * 128;     // one 32-column box
constexpr int TN_P_BYTES = 4 * TN_BOX_BYTES;    // the 128 columns of P that a CTA holds
constexpr int kTnSplitWarps = 8, kTnThreads = 32 * (2 + kTnSplitWarps + 4);
constexpr int kMaxTnStages = 8, kTnBarBytes = 8 * (3 * kMaxTnStages + 5) + 8;

struct DenseTnArgs {
    float4* partial;                            // [range][CTA of the pair][q_store / 4][p_store]: four columns of Q, rows side by side
    int64_t n;                                  // rows to reduce over
    int64_t rows_per_range;                     // multiple of TN_ROWS
    int32_t ranges;
    int32_t p_cols, q_cols;                     // columns of P and Q
    int32_t q_pad;                              // columns of the MMA: a multiple of 16, of 64 for a pair
    int32_t p_store, q_store;                   // rows and columns of a CTA's partial: multiples of 16
    int32_t flush_slabs;                        // slabs accumulated in tensor memory between two flushes
    int32_t stages;
    int32_t swapped;                            // P is G
    int* status;
};

// MN-major tile of 32-bit elements.  The tensor cores read such operands only in the "128B swizzle with 32-byte atoms"
// layout (32-byte chunks of a 128-byte row XOR-ed with the row index modulo 4), which TMA writes in its
// SWIZZLE_128B_ATOM_32B mode: 4-row groups are 512 bytes apart (stride byte offset), the 32-column boxes 2048 bytes
// (leading byte offset).
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(TN_BOX_BYTES >> 4) << 16;                 // leading byte offset: next 32 columns of M / N
    d |= (uint64_t)(512 >> 4) << 32;                          // stride byte offset: next 4 rows of K
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)1 << 61;                                   // layout type: SWIZZLE_128B_BASE32B
    return d;
}

// What bounds it: shared memory (MN-major 32-bit operands are read at half its rate) for wide operands, the MMAs' 130 clocks for narrow
// ones.  2,449,029 rows (us; four warps that split and flush in turn, two accumulators of one CTA -> this): 256 x 256 1,830 -> 1,660,
// 100 x 256 1,205 -> 940, 256 x 47 1,017 -> 787, 256 x 128 1,280 -> 970; 150,001 rows: 127 -> 120, 91 -> 73, 78 -> 66, 96 -> 71.
// Warps: 0 TMA, 1 MMA issue + tensor-memory allocation, 2-9 split, 10-13 flush.  Two accumulators (columns 0 / 256): while one is added to
// the partial result the other takes the next rows.
template <bool PAIR>
__device__ __forceinline__ void dense_tn(const CUtensorMap& tmP, const CUtensorMap& tmQ, const DenseTnArgs& a)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* gbase = smem_raw + (base - raw);
    const int rank = PAIR ? blockIdx.x & 1 : 0;
    const int range0 = PAIR ? blockIdx.x & ~1 : blockIdx.x, range1 = min(a.ranges, range0 + (PAIR ? 2 : 1));
    const int p0 = rank * 128, q0 = rank * (a.q_pad / 2);         // first columns of this CTA
    const int p_boxes = max(0, min(4, (a.p_cols - p0 + 31) / 32)), q_boxes = (PAIR ? a.q_pad / 2 : a.q_pad + 31) / 32;
    const int q_bytes = q_boxes * TN_BOX_BYTES;
    const int stage_bytes = 2 * TN_P_BYTES + 2 * q_bytes;         // P head, P tail, Q head, Q tail
    const uint32_t bars = base + a.stages * stage_bytes;
    const uint32_t full0 = bars, ready0 = bars + 8 * kMaxTnStages, empty0 = bars + 16 * kMaxTnStages, acc_full0 = bars + 24 * kMaxTnStages;
    const uint32_t acc_empty0 = acc_full0 + 16, done = acc_empty0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + a.stages * stage_bytes + 24 * kMaxTnStages + 40);
    const int T = a.flush_slabs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto slabs_of = [&](int range) { return (int)((max((int64_t)0, min(a.rows_per_range, a.n - range * a.rows_per_range)) + TN_ROWS - 1) / TN_ROWS); };
    constexpr int kTmemCols = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(ready0 + 8 * s, (PAIR ? 2 : 1) * kTnSplitWarps);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full0 + 8 * b, 1);
            mbar_init(acc_empty0 + 8 * b, (PAIR ? 2 : 1) * 4);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    auto sync_unit = [&] {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if constexpr (PAIR) cluster_sync();
        else __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    sync_unit();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;
    auto commit = [](uint32_t bar) {
        if constexpr (PAIR) umma_commit_pair(bar);
        else umma_commit(bar);
    };
    auto arrive = [](uint32_t bar) {                              // `bar`: of the CTA that issues the MMAs
        if constexpr (PAIR) mbar_arrive_cluster(bar);
        else mbar_arrive(bar);
    };
    uint32_t issuer_ready0 = ready0, issuer_acc_empty0 = acc_empty0;
    if constexpr (PAIR) {
        issuer_ready0 = in_leader(ready0);
        issuer_acc_empty0 = in_leader(acc_empty0);
    }

    if (warp == 0) {
        if (lane == 0) {                                          // TMA producer
            int it = 0, s = 0, phase = 1;
            for (int range = range0; range < range1; ++range) {
                const int nslabs = slabs_of(range);
                for (int i = 0; i < nslabs && ok; ++i, ++it) {
                    if (it >= a.stages) ok = mbar_wait(empty0 + 8 * s, phase);
                    if (!ok) break;
                    const uint32_t st = base + s * stage_bytes;
                    const int r0 = (int)(range * a.rows_per_range + (int64_t)i * TN_ROWS);
                    mbar_expect_tx(full0 + 8 * s, (p_boxes + q_boxes) * TN_BOX_BYTES);
                    for (int j = 0; j < p_boxes; ++j) tma_load_2d(st + j * TN_BOX_BYTES, &tmP, p0 + 32 * j, r0, full0 + 8 * s);
                    for (int j = 0; j < q_boxes; ++j) tma_load_2d(st + 2 * TN_P_BYTES + j * TN_BOX_BYTES, &tmQ, q0 + 32 * j, r0, full0 + 8 * s);
                    if (++s == a.stages) s = 0, phase ^= 1;
                }
            }
            await_loads(full0, it, a.stages);
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {                             // MMA issuer
            // A and B MN-major, 128 rows per CTA
            const uint32_t idesc = (umma_idesc_tf32(a.q_pad) + (PAIR ? (uint32_t)(BM >> 4) << 24 : 0u)) | (1u << 15) | (1u << 16);
            int s = 0, phase = 0, group = 0;
            for (int range = range0; range < range1; ++range) {
                const int nslabs = slabs_of(range);
                for (int i = 0; i < nslabs && ok; ++i) {
                    const int b = group & 1, in_group = i % T;    // the accumulators change, and restart, with every flush group
                    if (in_group == 0 && group >= 2) ok = mbar_wait(acc_empty0 + 8 * b, ((group >> 1) - 1) & 1);
                    ok = ok && mbar_wait(ready0 + 8 * s, phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t st = base + s * stage_bytes, acc = tmem + (uint32_t)(b * 256);
                    const uint64_t p_head = umma_desc_mn_sw128(st), p_tail = umma_desc_mn_sw128(st + TN_P_BYTES);
                    const uint64_t q_head = umma_desc_mn_sw128(st + 2 * TN_P_BYTES), q_tail = umma_desc_mn_sw128(st + 2 * TN_P_BYTES + q_bytes);
                    auto multiply = [&](uint64_t p, uint64_t q, uint32_t add) {
                        if constexpr (PAIR) umma_tf32_pair(acc, p, q, idesc, add);
                        else umma_tf32(acc, p, q, idesc, add);
                    };
#pragma unroll
                    for (int k = 0; k < TN_ROWS / 8; ++k) {       // one 8-row group (1024 bytes) per MMA; the tail of X comes first
                        const uint64_t adv = (uint64_t)(k * (1024 >> 4));
                        multiply((a.swapped ? p_head : p_tail) + adv, (a.swapped ? q_tail : q_head) + adv, (in_group > 0 || k > 0) ? 1u : 0u);
                        multiply((a.swapped ? p_tail : p_head) + adv, (a.swapped ? q_head : q_tail) + adv, 1u);
                        multiply(p_head + adv, q_head + adv, 1u);
                    }
                    commit(empty0 + 8 * s);
                    if (in_group == T - 1 || i == nslabs - 1) {
                        commit(acc_full0 + 8 * b);
                        ++group;
                    }
                    if (++s == a.stages) s = 0, phase ^= 1;
                }
            }
            if constexpr (PAIR) await_mmas_pair(done);
            else await_mmas(done);
        } else if (lane == 0) {
            mbar_wait(done, 0);
        }
    } else if (warp < 2 + kTnSplitWarps) {
        // The tile as loaded serves as head, its tail goes behind it.  Half the warps take the even boxes, half the odd ones.  Columns of P
        // that it does not have are neither loaded nor split: what lies there reaches rows of the accumulators, and of a pair's partial
        // results, that k_dense_tn_reduce leaves out.
        const int t = threadIdx.x - 64, half = t >> 7, boxes = p_boxes + q_boxes;
        int s = 0, phase = 0, slabs = 0;
        for (int range = range0; range < range1; ++range) slabs += slabs_of(range);
        for (int i = 0; i < slabs; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, phase));
            if (!ok) break;
            unsigned char* st = gbase + (size_t)s * stage_bytes + (t & 127) * 16;
            auto at = [&](int box) { return st + (box < p_boxes ? box * TN_BOX_BYTES : 2 * TN_P_BYTES + (box - p_boxes) * TN_BOX_BYTES); };
            for (int b0 = half; b0 < boxes; b0 += 8) {
                float4 x[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (b0 + 2 * j < boxes) x[j] = *reinterpret_cast<const float4*>(at(b0 + 2 * j));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int box = b0 + 2 * j;
                    if (box >= boxes) break;
                    float4 h;
                    h.x = __uint_as_float(__float_as_uint(x[j].x) & 0xFFFFE000u); h.y = __uint_as_float(__float_as_uint(x[j].y) & 0xFFFFE000u);
                    h.z = __uint_as_float(__float_as_uint(x[j].z) & 0xFFFFE000u); h.w = __uint_as_float(__float_as_uint(x[j].w) & 0xFFFFE000u);
                    *reinterpret_cast<float4*>(at(box) + (box < p_boxes ? TN_P_BYTES : q_bytes)) = make_float4(x[j].x - h.x, x[j].y - h.y, x[j].z - h.z, x[j].w - h.w);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive(issuer_ready0 + 8 * s);
            if (++s == a.stages) s = 0, phase ^= 1;
        }
    } else {
        // Flush: the tensor cores add into their accumulator with truncation, an error that grows with the length
        // of the chain, so after T slabs an accumulator is added - rounded to nearest - into this CTA's partial
        // result (which stays in L2) and restarts from zero.
        const int q = warp & 3, row = q * 32 + lane;              // a warp may only read its own quarter of the TMEM lanes
        const bool stored = row < a.p_store;
        int group = 0;
        for (int range = range0; range < range1 && ok; ++range) {
            float4* part = a.partial + (int64_t)((PAIR ? 2 : 1) * range + rank) * (a.q_store / 4) * a.p_store + row;
            const int groups = (slabs_of(range) + T - 1) / T;
            for (int g = 0; g < groups; ++g, ++group) {
                const int b = group & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * b, (group >> 1) & 1));        // tcgen05.ld is warp-collective
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int c0 = 0; c0 < a.q_store; c0 += 32) {      // two 16-column reads in flight per wait
                    const int two = c0 + 16 < a.q_store;          // warp-uniform
                    uint32_t r[32];
                    const uint32_t acc = tmem + (uint32_t)(b * 256) + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
                    tmem_ld16(acc, r);
                    if (two) tmem_ld16(acc + 16, r + 16);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float4* p = part + (int64_t)(c0 / 4) * a.p_store;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (!stored || (j >= 4 && !two)) break;
                        // Only this thread ever touches these 16 bytes, in program order, so the sum order is fixed; the
                        // reduction is sent to L2 and not waited for.
                        if (g == 0)
                            __stcg(p + j * a.p_store, make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                                  __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])));
                        else
                            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + j * a.p_store), "f"(__uint_as_float(r[4 * j])),
                                         "f"(__uint_as_float(r[4 * j + 1])), "f"(__uint_as_float(r[4 * j + 2])), "f"(__uint_as_float(r[4 * j + 3]))
                                         : "memory");
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive(issuer_acc_empty0 + 8 * b);
            }
            if (groups == 0 && stored)                            // a range without rows contributes zeros
                for (int j = 0; j < a.q_store / 4; ++j) __stcg(part + (int64_t)j * a.p_store, make_float4(0.f, 0.f, 0.f, 0.f));
        }
    }
    if (!ok) atomicExch(a.status, 1);
    sync_unit();                                                  // no CTA leaves while the other's MMAs read its operands or arrive at its barriers
    if (warp == 1) {
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}
__global__ void __launch_bounds__(kTnThreads, 1)
k_dense_tn(const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmQ, const DenseTnArgs a)
{
    dense_tn<false>(tmP, tmQ, a);
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kTnThreads, 1)
k_dense_tn_pair(const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmQ, const DenseTnArgs a)
{
    dense_tn<true>(tmP, tmQ, a);
}

// Adds the ranges' partials slot by slot, in order; slots of the padding are skipped.  A CTA takes 128 slots, eight warps fetch 40 ranges'
// at a time, 512 bytes each, and four add them (one thread a slot, loads and adds of its own, took 7.6 to 17 us: now 4.5 to 5.7, 256 x 256 7.1 to 8.6).
__global__ void __launch_bounds__(256) k_dense_tn_reduce(const float* __restrict__ partial, int ranges, int32_t slots, float* __restrict__ D, int64_t ldd,
                                                         int32_t p_cols, int32_t q_cols, int32_t p_store, int32_t q_store, int transposed)
{
    constexpr int kEach = 5, kChunk = 8 * kEach;
    __shared__ float4 part[2][kChunk][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float4* from = reinterpret_cast<const float4*>(partial) + blockIdx.x * 32 + lane;      // slots are a multiple of 256
    float sum = 0.f;
    for (int r0 = 0, b = 0; r0 < ranges; r0 += kChunk, b ^= 1) {
        const int n = min(kChunk, ranges - r0);
        float4 x[kEach];
#pragma unroll
        for (int j = 0; j < kEach; ++j)
            if (warp + 8 * j < n) x[j] = __ldcg(from + (int64_t)(r0 + warp + 8 * j) * (slots / 4));
#pragma unroll
        for (int j = 0; j < kEach; ++j)
            if (warp + 8 * j < n) part[b][warp + 8 * j][lane] = x[j];
        __syncthreads();                                          // whoever fills this buffer next has passed the next one of these
        if (threadIdx.x < 128)
#pragma unroll 8
            for (int r = 0; r < n; ++r) sum += reinterpret_cast<const float*>(part[b][r])[threadIdx.x];
    }
    if (threadIdx.x >= 128) return;
    const int i = blockIdx.x * 128 + threadIdx.x;
    const int half_slots = p_store * q_store, half = i / half_slots, in_half = i % half_slots, c4 = in_half / (4 * p_store), rest = in_half % (4 * p_store);
    const int p = half * 128 + rest / 4, q = c4 * 4 + rest % 4;
    if (p >= p_cols || q >= q_cols) return;
    D[transposed ? (int64_t)q * ldd + p : (int64_t)p * ldd + q] = sum;
}

int make_map_box(CUtensorMap* map, const float* ptr, int64_t rows, int64_t cols, int64_t ld, int box_cols, int box_rows)
{
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return DG_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? DG_OK : DG_ERR_UNSUPPORTED;
}

}  // namespace

extern "C" int dg_dense_tn_supported(int64_t n, int32_t Km, int32_t Nn, int64_t ldx, int64_t ldg, const void* X, const void* G)
{
    if (n <= 0 || Km <= 0 || Nn <= 0 || n >= ((int64_t)1 << 31)) return 0;
    if (ldx % 4 || ldg % 4 || ldx < Km || ldg < Nn) return 0;
    if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(G)) & 15) return 0;
    return encode_tiled() != nullptr;
}

extern "C" int dg_dense_tn(const float* X, int64_t ldx, const float* G, int64_t ldg, float* D, int64_t ldd, int64_t n,
                           int32_t Km, int32_t Nn, float* scratch, int64_t scratch_floats, int32_t max_ctas, void* stream)
{
    if (!X || !G || !D || !scratch) return DG_ERR_NULL;
    if (ldd < Nn || max_ctas < 1 || (reinterpret_cast<uintptr_t>(scratch) & 15)) return DG_ERR_DIMS;
    if (!dg_dense_tn_supported(n, Km, Nn, ldx, ldg, X, G)) return DG_ERR_UNSUPPORTED;
    if (Km > 256 || Nn > 256) {     // wider than two accumulators: 256 x 256 panels of D, one after the other on the stream
        for (int32_t m0 = 0; m0 < Km; m0 += 256)                  // (they share `scratch`; the operands are streamed once per panel)
            for (int32_t c0 = 0; c0 < Nn; c0 += 256) {
                const int rc = dg_dense_tn(X + m0, ldx, G + c0, ldg, D + (int64_t)m0 * ldd + c0, ldd, n, Km - m0 < 256 ? Km - m0 : 256,
                                           Nn - c0 < 256 ? Nn - c0 : 256, scratch, scratch_floats, max_ctas, stream);
                if (rc) return rc;
            }
        return DG_OK;
    }
    if (max_ctas == 1 && Km > 128 && Nn > 128) {      // no CTA to pair with: both halves of X, one after the other (the same sums in the same order)
        const int rc = dg_dense_tn(X, ldx, G, ldg, D, ldd, n, 128, Nn, scratch, scratch_floats, 1, stream);
        return rc ? rc : dg_dense_tn(X + 128, ldx, G, ldg, D + (int64_t)128 * ldd, ldd, n, Km - 128, Nn, scratch, scratch_floats, 1, stream);
    }
    const bool pair = std::min(Km, Nn) > 128, swapped = !pair && Nn < Km;
    if (pair) max_ctas &= ~1;                                     // whole pairs, and no more CTAs than allowed
    DenseTnArgs a{};
    a.n = n;
    a.p_cols = swapped ? Nn : Km;
    a.q_cols = swapped ? Km : Nn;
    a.q_store = (a.q_cols + 15) / 16 * 16;
    a.q_pad = pair ? (a.q_cols + 63) / 64 * 64 : a.q_store;       // a pair's halves are whole boxes
    a.p_store = pair ? 128 : (a.p_cols + 15) / 16 * 16;
    const int64_t slabs = (n + TN_ROWS - 1) / TN_ROWS;
    a.ranges = (int)std::min<int64_t>(max_ctas, slabs);
    a.rows_per_range = (slabs + a.ranges - 1) / a.ranges * TN_ROWS;
    a.swapped = swapped;
    const int64_t slots = (int64_t)(pair ? 2 : 1) * a.p_store * a.q_store;     // a range's partial, padding included
    if (a.ranges * slots > scratch_floats) return DG_ERR_SCRATCH;
    a.flush_slabs = 16;                                           // 256 rows = 96 tensor-core accumulations per chain
    a.partial = reinterpret_cast<float4*>(scratch);
    a.status = dg_status_word();
    if (!a.status) return DG_ERR_STATE;
    CUtensorMap tmX, tmG;
    int rc;
    if ((rc = make_map_box(&tmX, X, n, Km, ldx, 32, TN_ROWS)) || (rc = make_map_box(&tmG, G, n, Nn, ldg, 32, TN_ROWS))) return rc;
    const size_t stage = 2 * TN_P_BYTES + 2 * (((pair ? a.q_pad / 2 : a.q_pad) + 31) / 32) * TN_BOX_BYTES;
    a.stages = (int)std::min<size_t>(kMaxTnStages, (227 * 1024 - kTnBarBytes - 1024) / stage);
    const size_t smem = a.stages * stage + kTnBarBytes + 1024;
    const CUtensorMap &tmP = swapped ? tmG : tmX, &tmQ = swapped ? tmX : tmG;
    static std::atomic<bool> granted[64], granted_pair[64];
    if ((rc = pair ? allow_smem((const void*)k_dense_tn_pair, granted_pair) : allow_smem((const void*)k_dense_tn, granted))) return rc;
    (pair ? k_dense_tn_pair : k_dense_tn)<<<pair ? (a.ranges + 1) / 2 * 2 : a.ranges, kTnThreads, smem, (cudaStream_t)stream>>>(tmP, tmQ, a);
    k_dense_tn_reduce<<<(unsigned)(slots / 128), 256, 0, (cudaStream_t)stream>>>(scratch, a.ranges, (int32_t)slots, D, ldd, a.p_cols, a.q_cols, a.p_store, a.q_store, swapped);
    return (int)cudaGetLastError();
}
