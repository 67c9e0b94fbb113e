// dg_spmm_csr_static: the local product for callers that must not allocate device memory.
//
// Who needs it: a host program whose device memory is already fully reserved by its own pool (a cudaMalloc from a
// library would fail or fragment it), or a latency-critical loop that cannot afford the implicit device-wide
// synchronisation of cudaMalloc / cudaFree.  dg_spmm_csr grows a plan-owned scratch buffer with cudaMalloc the first
// time a plan is used at a wider F; this variant never allocates: the partial sums of split (heavy) rows go to a
// fixed array that is part of the library image, so every GPU that loads the library carries it until the process ends.
//
// Limit: DG_STATIC_SCRATCH_FLOATS floats (16 MiB).  A request counts F floats for every chunk of DG_STATIC_CHUNK entries of the
// rows longer than that (the plan's own lengths where its maker gave any); a larger one is refused with DG_ERR_SCRATCH before anything
// is launched.  The chunks that plans really have are two to four times as many where their length is a default, so a product within
// the limit may not fit in one go: it is then done in pieces of its columns, which change no bit of a column's sums, or,
// where no row is longer than DG_STATIC_CHUNK (or the chunks leave no room for four columns), without splitting rows.
//
// Sharing: all calls on a device use the same array.  Nothing in it has to start at zero - every scratch row is fully
// written by the chunk kernel before the finishing kernel reads it - so no clearing is done between calls, but two
// calls that overlap in time on the GPU (different streams) race on it.  Serialise them on one stream.
//
// Set-up: the array's name below is a host-side handle, not a device address.  The address is looked up once per device
// with cudaGetSymbolAddress while that device is current, and cached.  With CUDA's lazy module loading that first lookup
// is also the moment the 16 MiB array is materialised on the device (it can fail for lack of memory, and may synchronise).
// dg_static_scratch_prepare() does the lookup on its own: call it once per device where an allocation is still acceptable
// (next to dg_plan_create, before the host's pool reserves the rest of the memory, before any stream capture); after it,
// dg_spmm_csr_static touches neither the allocator nor the module loader.  Without it the first product call on a device
// does the lookup.
//
// The entry always runs the row kernels (the streaming family sizes its scratch differently) and its products are not
// counted by dg_profile_begin / dg_profile_end.
#include <mutex>
#include "dg_internal.h"

#define DG_STATIC_SCRATCH_FLOATS (4 * 1024 * 1024)
#define DG_MAX_DEVICES 64

static __device__ __align__(256) float g_static_scratch[DG_STATIC_SCRATCH_FLOATS];

namespace {
std::mutex g_lookup_mutex;
float* g_scratch_address[DG_MAX_DEVICES] = {nullptr};

// Device address of g_static_scratch on `device`, which must be the current device.
int static_scratch_address(int device, float** out)
{
    if (device < 0 || device >= DG_MAX_DEVICES) return DG_ERR_STATE;
    std::lock_guard<std::mutex> lock(g_lookup_mutex);
    if (!g_scratch_address[device]) {
        float* ptr = nullptr;
        DG_CUDA(cudaGetSymbolAddress((void**)&ptr, g_static_scratch));
        if (!ptr) return DG_ERR_STATE;
        g_scratch_address[device] = ptr;
    }
    *out = g_scratch_address[device];
    return DG_OK;
}
}  // namespace

extern "C" int64_t dg_static_scratch_capacity(void) { return DG_STATIC_SCRATCH_FLOATS; }

extern "C" int dg_static_scratch_prepare(void)
try {
    int device = -1;
    DG_CUDA(cudaGetDevice(&device));
    float* unused = nullptr;
    return static_scratch_address(device, &unused);
} catch (...) {
    return dg_exception();
}

extern "C" int dg_spmm_csr_static(const dg_plan* plan, const float* val, const float* B, int64_t ldb, float* C,
                                  int64_t ldc, int32_t F, float alpha, float beta, uint32_t flags,
                                  const float* row_scale, const float* bias, void* stream)
try {
    int rc = dg_check_spmm_args(plan, val, B, ldb, C, ldc, F, flags, row_scale, bias);   // also checks the current device
    if (rc) return rc;
    const int64_t chunks = plan->n_chunks;
    const bool fits = chunks * F <= DG_STATIC_SCRATCH_FLOATS;
    if (!fits && plan->static_chunks * F > DG_STATIC_SCRATCH_FLOATS) return DG_ERR_SCRATCH;
    float* scratch = nullptr;
    if ((rc = static_scratch_address(plan->device, &scratch))) return rc;
    const bool split = fits || (plan->max_row_nnz > DG_STATIC_CHUNK && chunks * 4 <= DG_STATIC_SCRATCH_FLOATS);
    const int32_t piece = fits || !split ? F : (int32_t)(DG_STATIC_SCRATCH_FLOATS / chunks / 4 * 4);
    for (int32_t c0 = 0; c0 < F && rc == DG_OK; c0 += piece) {
        const int32_t width = F - c0 < piece ? F - c0 : piece;
        rc = dg_spmm_launch_rows(plan, val, B ? B + c0 : B, ldb, C + c0, ldc, width, alpha, beta, flags, row_scale, bias ? bias + c0 : bias, scratch,
                                 split ? chunks * width : 0, (cudaStream_t)stream, 0, split);
    }
    return rc;
} catch (...) {
    return dg_exception();
}
