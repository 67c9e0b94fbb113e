// Row-wise helpers either side of the distributed SpMM.
#include "dg_internal.h"

#define DG_ROWS_LOSS_PARTS (148 * 8)      // most CTAs of the loss, and the partial sums they leave

namespace {

// One 16-byte piece of a destination row per thread: 4 source floats (neighbouring threads read neighbouring floats), one
// aligned store.  Bound by memory: n * (cols + ld_dst) * 4 bytes.
__global__ void __launch_bounds__(256) k_pad_rows(const float* __restrict__ src, int64_t ld_src, int64_t n, int32_t cols,
                                                  float* __restrict__ dst, int32_t pieces)
{
    const int64_t total = n * pieces, stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int64_t row = i / pieces;
        const int c = (int)(i - row * pieces) * 4;
        const float* s = src + row * ld_src + c;
        float4 v;
        v.x = c < cols ? __ldcs(s) : 0.f;
        v.y = c + 1 < cols ? __ldcs(s + 1) : 0.f;
        v.z = c + 2 < cols ? __ldcs(s + 2) : 0.f;
        v.w = c + 3 < cols ? __ldcs(s + 3) : 0.f;
        reinterpret_cast<float4*>(dst)[i] = v;
    }
}

// ---- mean cross-entropy over the rows that carry a target --------------------------------------------------------------
// The step's loss reads the logits of the train rows once and its gradient reads them once more and writes n x C floats: 12 bytes per row
// and class.  As separate passes (row gather, log-softmax, a one-CTA loss reduction, its
// backward, the softmax backward, a scatter into zeros) it took 5.5 ms of a 66 ms step at 2,449,029 x 47.
// What bounds them is instructions, and the wait for a row: loss_form.
// A group of LPR lanes owns a row; lanes read neighbouring classes.  Sums are taken in a fixed order (rows of a thread in
// order, lanes and warps by a tree, CTAs in order), so the loss is bit-reproducible.
constexpr int kLossThreads = 256;

template <int LPR> __device__ __forceinline__ float group_max(float v)
{
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, v, off);
        v = o > v || o != o ? o : v;
    }
    return v;
}
template <int LPR> __device__ __forceinline__ float group_sum(float v)
{
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// The rows a group works on, one after the other, their first KEPT * LPR classes in registers.  AHEAD: a row's target is requested two rows
// ahead, its classes one row ahead.
template <int LPR, int KEPT, bool AHEAD> struct Rows {
    const float* x;
    const int32_t* target;
    int64_t ld, n, row, step;
    int32_t C, t, t_next;
    float v[AHEAD ? KEPT : 1];
    __device__ __forceinline__ int32_t target_of(int64_t r) const { return r < n ? __ldg(target + r) : -1; }
    __device__ __forceinline__ void fetch(float* to)
    {
        const int lane = threadIdx.x % LPR;
        const float* r = x + row * ld;
#pragma unroll
        for (int j = 0; j < KEPT; ++j) to[j] = t >= 0 && lane + j * LPR < C ? __ldg(r + lane + j * LPR) : __int_as_float(0xff800000);
    }
    __device__ __forceinline__ Rows(const float* x_, int64_t ld_, int64_t n_, int32_t C_, const int32_t* target_) : x(x_), target(target_), ld(ld_), n(n_), C(C_)
    {
        constexpr int RPB = kLossThreads / LPR;
        row = (int64_t)blockIdx.x * RPB + threadIdx.x / LPR;
        step = (int64_t)gridDim.x * RPB;
        if constexpr (AHEAD) {
            t = target_of(row);
            t_next = target_of(row + step);
            fetch(v);
        }
    }
    // Moves on: `e` and `of` receive the row it was at.
    __device__ __forceinline__ int64_t next(float* e, int32_t& of)
    {
        const int64_t was = row;
        if constexpr (AHEAD) {
            of = t;
#pragma unroll
            for (int j = 0; j < KEPT; ++j) e[j] = v[j];
            row += step;
            t = t_next;
            t_next = target_of(row + step);
            fetch(v);
        } else {
            of = t = target_of(row);
            fetch(e);
            row += step;
        }
        return was;
    }
};

template <int LPR, int KEPT, bool AHEAD>
__global__ void __launch_bounds__(kLossThreads) k_rows_ce_forward(const float* __restrict__ x, int64_t ld, int64_t n, int32_t C,
                                                                  const int32_t* __restrict__ target, float* __restrict__ lse,
                                                                  double* __restrict__ partial)
{
    constexpr int RPB = kLossThreads / LPR;
    const int lane = threadIdx.x % LPR;
    double loss = 0.0;
    Rows<LPR, KEPT, AHEAD> rows(x, ld, n, C, target);
    for (int64_t base = (int64_t)blockIdx.x * RPB; base < n; base += (int64_t)gridDim.x * RPB) {
        float e[KEPT ? KEPT : 1], mx = __int_as_float(0xff800000);
        int32_t t;
        const int64_t row = rows.next(e, t);
        const bool on = t >= 0;                                   // the same in every lane of a row's group
        const float* r = x + row * ld;
#pragma unroll
        for (int j = 0; j < KEPT; ++j) mx = e[j] > mx || e[j] != e[j] ? e[j] : mx;           // a NaN stays
        if (on)
            for (int c = lane + KEPT * LPR; c < C; c += LPR) {
                const float v = __ldg(r + c);
                mx = v > mx || v != v ? v : mx;
            }
        mx = group_max<LPR>(mx);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < KEPT; ++j)
            if (on && lane + j * LPR < C) sum += expf(e[j] - mx);
        if (on)
            for (int c = lane + KEPT * LPR; c < C; c += LPR) sum += expf(__ldg(r + c) - mx);
        sum = group_sum<LPR>(sum);
        if (on && lane == 0) {
            const float l = logf(sum);
            lse[row] = mx + l;
            loss += (double)(l - (__ldg(r + t) - mx));
        }
    }
    __shared__ double warp_sum[kLossThreads / 32];
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = loss;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kLossThreads / 32; ++w) s += warp_sum[w];
        partial[blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(kLossThreads) k_rows_ce_mean(const double* __restrict__ partial, int parts, double inv_count, float* __restrict__ loss)
{
    __shared__ double warp_sum[kLossThreads / 32];
    double s = 0.0;
    for (int i = threadIdx.x; i < parts; i += kLossThreads) s += partial[i];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        s = 0.0;
        for (int w = 0; w < kLossThreads / 32; ++w) s += warp_sum[w];
        *loss = (float)(s * inv_count);
    }
}

// grad[row, c] = (softmax(x[row])[c] - [c == target]) * upstream / count, zero for rows without a target and beyond C.
// The softmax is taken from the row's maximum and sum anew: against a stored logsumexp it would carry that number's rounding, which
// grows with the logits (error of the gradient against float64, 47 classes: around 0 1.6e-7, 100 1.3e-6, 10,000 1.6e-4; this way
// 5e-8 everywhere, as PyTorch's).  A lane's exponentials stay in registers up to
// KEPT classes a lane, so an exponential a class is all it takes, as with the logsumexp.
template <int LPR, int KEPT, bool AHEAD>
__global__ void __launch_bounds__(kLossThreads) k_rows_ce_backward(const float* __restrict__ x, int64_t ld, int64_t n, int32_t C,
                                                                   const int32_t* __restrict__ target, const float* __restrict__ upstream,
                                                                   float inv_count, float* __restrict__ grad, int64_t ldg)
{
    constexpr int RPB = kLossThreads / LPR;
    const int lane = threadIdx.x % LPR;
    const float scale = __ldg(upstream) * inv_count;
    Rows<LPR, KEPT, AHEAD> rows(x, ld, n, C, target);
    for (int64_t base = (int64_t)blockIdx.x * RPB; base < n; base += (int64_t)gridDim.x * RPB) {
        float e[KEPT ? KEPT : 1], mx = __int_as_float(0xff800000);
        int32_t t;
        const int64_t row = rows.next(e, t);
        const bool on = t >= 0;
        const float* r = x + row * ld;
#pragma unroll
        for (int j = 0; j < KEPT; ++j) mx = e[j] > mx || e[j] != e[j] ? e[j] : mx;           // a NaN stays
        if (on)
            for (int c = lane + KEPT * LPR; c < C; c += LPR) {
                const float v = __ldg(r + c);
                mx = v > mx || v != v ? v : mx;
            }
        mx = group_max<LPR>(mx);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < KEPT; ++j)
            if (on && lane + j * LPR < C) sum += e[j] = expf(e[j] - mx);
        if (on)
            for (int c = lane + KEPT * LPR; c < C; c += LPR) sum += expf(__ldg(r + c) - mx);
        const float inv = 1.f / group_sum<LPR>(sum);
        if (row >= n) continue;
        float* g = grad + row * ldg;
#pragma unroll
        for (int j = 0; j < KEPT; ++j) {
            const int c = lane + j * LPR;
            if (c < ldg) g[c] = on && c < C ? (e[j] * inv - (c == t ? 1.f : 0.f)) * scale : 0.f;
        }
        for (int c = lane + KEPT * LPR; c < ldg; c += LPR)
            g[c] = on && c < C ? (expf(__ldg(r + c) - mx) * inv - (c == t ? 1.f : 0.f)) * scale : 0.f;
    }
}

// The kernel that a loss takes: lanes a row, classes a lane keeps in registers, and whether the next row is requested ahead.
// Eight classes a lane share row, target, shuffles and logarithm among more rows of a warp than four do, as long as there are rows enough
// for so few lanes.  The look-ahead pays where the rows come from DRAM; out of the L2 its registers cost more than it hides.  Up to
// 16 classes four lanes keep one class or four: eight slots would be idle.  Beyond 128 classes the forward pass reads a row
// twice, out of the L1.  us, forward and gradient, four a lane -> eight -> eight and ahead (C > 128: none kept -> four -> eight):
//   2,449,029 x 47 (460 MB) 282 329 -> 191 265 -> 182 257; x 16 (157 MB) 81 92 (ahead 71 88) -> 93 121 -> 85 117; x 2 57 67 -> 71 93 -> 73 97
//   150,001 x 47 (28 MB) 19.6 20.6 -> 15.1 16.9 -> 15.8 18.3; x 10 7.8 6.6 -> 8.7 8.3 -> 9.6 9.2; 10,000 x 32 4.3 2.7 -> 4.4 3.3 -> 4.5 3.3
//   150,001 x 130 36 - -> 41 54 -> 41 59, x 200 42 - -> 48 72 -> 47 65
struct LossForm {
    int lanes, kept;
    bool ahead;
};
LossForm loss_form(int64_t n, int32_t C, int64_t ld, bool backward)
{
    if (C > 128) return {32, !backward ? 0 : C <= 160 ? 4 : 8, false};
    const bool ahead = n * ld * 4 > (int64_t)64 << 20;            // half of the L2: what else passes through it needs the rest
    if (C <= 4) return {4, 1, false};
    if (C <= 16) return {4, 4, ahead};
    const int few = C <= 32 ? 4 : C <= 64 ? 8 : 16;
    if (n * few < 1 << 16) return {2 * few, 4, false};
    return {few, 8, ahead};
}

// `use` is called with the form's lanes, classes and look-ahead as constants.
template <int N> using Int = std::integral_constant<int, N>;
template <bool BACKWARD, class Use> void with_form(const LossForm& f, Use use)
{
    auto either = [&](auto lanes, auto kept) {
        if (f.ahead) use(lanes, kept, std::true_type{});
        else use(lanes, kept, std::false_type{});
    };
    switch (f.lanes) {
        case 4: f.kept == 1 ? use(Int<4>{}, Int<1>{}, std::false_type{}) : f.kept == 4 ? either(Int<4>{}, Int<4>{}) : either(Int<4>{}, Int<8>{}); break;
        case 8: f.kept == 4 ? use(Int<8>{}, Int<4>{}, std::false_type{}) : either(Int<8>{}, Int<8>{}); break;
        case 16: f.kept == 4 ? use(Int<16>{}, Int<4>{}, std::false_type{}) : either(Int<16>{}, Int<8>{}); break;
        default:
            if constexpr (!BACKWARD) {
                f.kept == 4 ? use(Int<32>{}, Int<4>{}, std::false_type{}) : use(Int<32>{}, Int<0>{}, std::false_type{});
            } else {
                f.kept == 4 ? use(Int<32>{}, Int<4>{}, std::false_type{}) : use(Int<32>{}, Int<8>{}, std::false_type{});
            }
    }
}

unsigned loss_blocks(int64_t n, int lpr)
{
    const int64_t rows_per_block = kLossThreads / lpr, blocks = (n + rows_per_block - 1) / rows_per_block;
    return (unsigned)(blocks < DG_ROWS_LOSS_PARTS ? blocks : DG_ROWS_LOSS_PARTS);
}

}  // namespace

extern "C" int dg_rows_cross_entropy(const float* x, int64_t ld, int64_t n, int32_t C, const int32_t* target, int64_t count, float* lse,
                                     double* scratch, float* loss, void* stream)
{
    if (n <= 0 || C <= 0 || count <= 0 || ld < C) return DG_ERR_DIMS;
    if (!x || !target || !lse || !scratch || !loss) return DG_ERR_NULL;
    cudaStream_t s = (cudaStream_t)stream;
    const LossForm form = loss_form(n, C, ld, false);
    const unsigned blocks = loss_blocks(n, form.lanes);
    with_form<false>(form, [&](auto lanes, auto kept, auto ahead) {
        k_rows_ce_forward<lanes(), kept(), ahead()><<<blocks, kLossThreads, 0, s>>>(x, ld, n, C, target, lse, scratch);
    });
    k_rows_ce_mean<<<1, kLossThreads, 0, s>>>(scratch, (int)blocks, 1.0 / (double)count, loss);
    return (int)cudaGetLastError();
}

extern "C" int dg_rows_cross_entropy_grad(const float* x, int64_t ld, int64_t n, int32_t C, const int32_t* target, int64_t count,
                                          const float* lse, const float* upstream, float* grad, int64_t ldg, void* stream)
{
    if (n <= 0 || C <= 0 || count <= 0 || ld < C || ldg < C) return DG_ERR_DIMS;
    if (!x || !target || !lse || !upstream || !grad) return DG_ERR_NULL;
    cudaStream_t s = (cudaStream_t)stream;
    const LossForm form = loss_form(n, C, ld, true);
    const unsigned blocks = loss_blocks(n, form.lanes);
    const float inv = (float)(1.0 / (double)count);
    with_form<true>(form, [&](auto lanes, auto kept, auto ahead) {
        k_rows_ce_backward<lanes(), kept(), ahead()><<<blocks, kLossThreads, 0, s>>>(x, ld, n, C, target, upstream, inv, grad, ldg);
    });
    return (int)cudaGetLastError();
}

extern "C" int dg_pad_rows(const float* src, int64_t ld_src, int64_t n, int32_t cols, float* dst, int64_t ld_dst, void* stream)
{
    if (n < 0 || cols < 0 || ld_src < cols || ld_dst < cols || ld_dst % 4 || ld_dst >= ((int64_t)1 << 31)) return DG_ERR_DIMS;
    if (n == 0 || ld_dst == 0) return DG_OK;
    if (!src || !dst) return DG_ERR_NULL;
    if (reinterpret_cast<uintptr_t>(dst) & 15) return DG_ERR_DIMS;
    const int64_t total = n * (ld_dst / 4), blocks = (total + 255) / 256;
    k_pad_rows<<<(unsigned)(blocks < 148 * 32 ? blocks : 148 * 32), 256, 0, (cudaStream_t)stream>>>(src, ld_src, n, cols, dst, (int32_t)(ld_dst / 4));
    return (int)cudaGetLastError();
}

extern "C" int32_t dg_rows_loss_scratch(void) { return DG_ROWS_LOSS_PARTS; }
