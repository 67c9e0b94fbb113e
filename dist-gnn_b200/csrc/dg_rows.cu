// Row-wise helpers either side of the distributed SpMM.
#include "dg_internal.h"

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

}  // namespace

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
