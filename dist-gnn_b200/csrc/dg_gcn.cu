// A whole GCN on one rank from one host call.
//
// A training step on a small graph is bound by the host: some twenty launches of a few microseconds each, issued through
// an interpreter that needs ten times that between them (1.2 ms a step on the 10,000-node graph, 0.3 ms of it on the
// device).  These two functions issue the layers' products and transforms back to back.
#include <algorithm>
#include "dg_internal.h"

namespace {

int64_t pad4(int64_t w) { return (w + 3) / 4 * 4; }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// The plan's scratch for every width of the network, the backward pass's among them, before the first product: grown width by
// width, the first pass waited for the device and went to the allocator up to three times in its middle.
int prepare(const dg_gcn_net* a, void* stream)
{
    int64_t widest = 0;
    for (int l = 0; l <= a->layers; ++l) widest = std::max(widest, pad4(a->dims[l]));
    return dg_spmm_prepare(a->plan, (int32_t)widest, (cudaStream_t)stream);
}

struct Marks {          // ids of the points between the regions of one call; a failed record is reported by its negative id
    int32_t* at;
    void* stream;
    void operator()() { if (at) *at++ = dg_mark_record(stream); }
};

int check_net(const dg_gcn_net* a, bool backward)
{
    if (!a || !a->plan || !a->dims || !a->act || !a->ld_act || !a->z) return DG_ERR_NULL;
    if (a->layers < 1 || a->n < 0 || a->plan->m != a->n || a->plan->k != a->n) return DG_ERR_DIMS;
    if (!backward && !a->fwd_split) return DG_ERR_NULL;
    if (backward && (!a->dw || !a->grad || !a->tn_scratch || (a->layers > 1 && (!a->bwd_split || !a->g)))) return DG_ERR_NULL;
    for (int l = 0; l <= a->layers; ++l)
        if (a->dims[l] < 1) return DG_ERR_DIMS;
    if (!a->x || a->ldx % 4 || a->ldx < pad4(a->dims[0]) || !aligned16(a->x) || !aligned16(a->z)) return DG_ERR_DIMS;
    for (int l = 0; l < a->layers; ++l) {
        if (!a->act[l]) return DG_ERR_NULL;
        const bool hidden = l + 1 < a->layers;
        if (a->ld_act[l] < a->dims[l + 1]) return DG_ERR_DIMS;
        if (hidden && (a->ld_act[l] % 4 || a->ld_act[l] < pad4(a->dims[l + 1]) || !aligned16(a->act[l]))) return DG_ERR_DIMS;
        if (!backward && !a->fwd_split[l]) return DG_ERR_NULL;
        if (backward && l > 0 && !a->bwd_split[l]) return DG_ERR_NULL;
    }
    if (backward && (a->ld_grad % 4 || a->ld_grad < pad4(a->dims[a->layers]) || !aligned16(a->grad) || (a->g && !aligned16(a->g)))) return DG_ERR_DIMS;
    return DG_OK;
}

int product(const dg_gcn_net* a, const float* b, int64_t ldb, int32_t width, void* stream)
{
    return dg_spmm_csr(a->plan, a->val, b, ldb, a->z, width, width, 1.f, 0.f, 0u, nullptr, nullptr, stream);
}

}  // namespace

extern "C" int dg_gcn_forward(const dg_gcn_net* a, void* stream)
try {
    int rc = check_net(a, false);
    if (rc || a->n == 0) return rc;
    if ((rc = prepare(a, stream))) return rc;
    Marks mark{a->marks, stream};
    mark();
    const float* in = a->x;
    int64_t ld_in = a->ldx;
    for (int l = 0; l < a->layers; ++l) {
        const int32_t K = a->dims[l], N = a->dims[l + 1];
        const int64_t width = pad4(K);
        if ((rc = product(a, in, ld_in, (int32_t)width, stream))) return rc;
        mark();
        const float* head = a->fwd_split[l];
        rc = dg_dense_nt_masked(a->z, width, head, head + (int64_t)N * width, width, a->act[l], a->ld_act[l], a->n, N, K, l + 1 < a->layers,
                                nullptr, 0, stream);
        if (rc) return rc;
        mark();
        in = a->act[l];
        ld_in = a->ld_act[l];
    }
    return DG_OK;
} catch (...) {
    return dg_exception();
}

extern "C" int dg_gcn_backward(const dg_gcn_net* a, void* stream)
try {
    int rc = check_net(a, true);
    if (rc || a->n == 0) return rc;
    if ((rc = prepare(a, stream))) return rc;
    Marks mark{a->marks, stream};
    mark();
    const float* g = a->grad;
    int64_t ld_g = a->ld_grad;
    for (int l = a->layers - 1; l >= 0; --l) {
        const int32_t K = a->dims[l], N = a->dims[l + 1];
        const int64_t width = pad4(N);
        const float* in = l ? a->act[l - 1] : a->x;
        const int64_t ld_in = l ? a->ld_act[l - 1] : a->ldx;
        if ((rc = product(a, g, ld_g, (int32_t)width, stream))) return rc;
        mark();
        if (l > 0) {        // the next gradient; g itself has been read by the product above
            const float* head = a->bwd_split[l];
            rc = dg_dense_nt_masked(a->z, width, head, head + (int64_t)K * width, width, a->g, pad4(K), a->n, K, N, 0, in, ld_in, stream);
            if (rc) return rc;
        }
        if (a->dw[l] && (rc = dg_dense_tn(in, ld_in, a->z, width, a->dw[l], N, a->n, K, N, a->tn_scratch, a->tn_scratch_floats, a->max_ctas, stream)))
            return rc;
        mark();
        g = a->g;
        ld_g = pad4(K);
    }
    return DG_OK;
} catch (...) {
    return dg_exception();
}
