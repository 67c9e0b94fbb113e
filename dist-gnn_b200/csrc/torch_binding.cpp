// Native side of the training path's hot calls: what a PyTorch program issues per step, without the interpreter in between.
//
// A training step on a small graph is bound by the host.  Issued from Python, autograd nodes, argument conversions and views
// cost three times what the step's kernels take (10,000-node graph: 0.4 ms of host work for 0.12 ms of kernels).  Here the
// one-rank network, the loss of the train rows and the local product are C++ autograd nodes and functions over the C ABI
// of include/dist_gnn_b200.h; torch owns memory, streams and the graph, as everywhere in this package.
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <atomic>
#include <mutex>
#include <unordered_map>
#include "dist_gnn_b200.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

std::atomic<int64_t> g_launches{0};       // dense-transform launches since the last take_launches()

void check(int code)
{
    if (code != DG_OK) throw std::runtime_error("dist_gnn_b200 error " + std::to_string(code) + ": " + dg_strerror(code));
}

void* stream_of(const Tensor& t) { return (void*)at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
int64_t pad4(int64_t w) { return (w + 3) / 4 * 4; }

// ---- time marks of regions that no Python code sees: kept until the timer they belong to asks ---------------------------
// One list per call: the points between its products and transforms, which alternate.  A region read out one by one from the
// interpreter was 5 us of host work, a quarter of a small training step; here it is what cudaEventElapsedTime takes.
struct Regions {
    std::vector<int32_t> marks;
    bool backward;                        // every layer then counts an all-reduce that a rank without peers has not to do
};
std::mutex g_regions_mu;
std::unordered_map<int64_t, std::vector<Regions>> g_regions;

void add_regions(int64_t timer, std::vector<int32_t>&& marks, bool backward)
{
    std::lock_guard<std::mutex> lock(g_regions_mu);
    g_regions[timer].push_back({std::move(marks), backward});
}
int64_t pending_regions(int64_t timer)
{
    std::lock_guard<std::mutex> lock(g_regions_mu);
    int64_t n = 0;
    const auto it = g_regions.find(timer);
    if (it != g_regions.end())
        for (const Regions& r : it->second) n += (int64_t)r.marks.size() - 1;
    return n;
}
// (seconds, regions) of the products, the transforms and the all-reduces since the last call.  The device has passed the marks.
std::vector<std::pair<double, int64_t>> resolve_regions(int64_t timer)
{
    std::vector<Regions> calls;
    {
        std::lock_guard<std::mutex> lock(g_regions_mu);
        const auto it = g_regions.find(timer);
        if (it != g_regions.end()) {
            calls = std::move(it->second);
            g_regions.erase(it);
        }
    }
    std::vector<std::pair<double, int64_t>> sums(3, {0.0, 0});
    int failed = DG_OK;
    for (const Regions& r : calls) {
        for (size_t i = 0; i + 1 < r.marks.size(); ++i) {
            auto& sum = sums[i & 1];
            ++sum.second;
            float ms = 0.f;
            if (r.marks[i] < 0 || r.marks[i + 1] < 0) continue;
            const int rc = dg_mark_elapsed(r.marks[i], r.marks[i + 1], &ms);
            if (rc != DG_OK) failed = rc;
            else sum.first += ms / 1000.0;
        }
        for (int32_t id : r.marks)
            if (id >= 0) dg_mark_release(id);
        if (r.backward) sums[2].second += (int64_t)r.marks.size() / 2;
    }
    check(failed);
    return sums;
}

// ---- a plan that the autograd graph can keep alive ----------------------------------------------------------------------
struct PlanRef {
    dg_plan* plan;
    Tensor col, values;                   // borrowed by the plan
    PlanRef(int64_t handle, Tensor c, Tensor v) : plan(reinterpret_cast<dg_plan*>(handle)), col(std::move(c)), values(std::move(v)) {}
    PlanRef(const PlanRef&) = delete;
    ~PlanRef() { dg_plan_destroy(plan); }
};

// ---- the local product --------------------------------------------------------------------------------------------------
int64_t operand(const Tensor& t, int64_t rows, const char* what)
{
    if (!t.defined() || !t.is_cuda() || t.scalar_type() != at::kFloat || t.dim() != 2)
        throw std::runtime_error(std::string(what) + " must be a 2-D fp32 CUDA tensor");
    if (t.size(0) != rows || (t.size(1) > 1 && t.stride(1) != 1)) {
        std::ostringstream s;
        s << what << " has shape " << t.sizes() << " / strides " << t.strides() << ", expected " << rows << " rows, unit column stride";
        throw std::runtime_error(s.str());
    }
    return t.size(0) > 1 ? t.stride(0) : std::max<int64_t>(t.size(1), 1);
}
const float* vector_ptr(const std::optional<Tensor>& t, const char* what)
{
    if (!t.has_value()) return nullptr;
    if (!t->is_cuda()) throw std::runtime_error(std::string(what) + " must be a CUDA tensor: this library has no CPU path");
    if (t->scalar_type() != at::kFloat || !t->is_contiguous()) throw std::runtime_error(std::string(what) + " must be a contiguous torch.float32 tensor");
    return t->data_ptr<float>();
}

void spmm(const std::shared_ptr<PlanRef>& ref, int64_t m, int64_t k, int64_t val, const Tensor& B, const Tensor& C, double alpha, double beta,
          const std::optional<Tensor>& row_scale, const std::optional<Tensor>& bias, bool relu)
{
    const int64_t ldb = operand(B, k, "B"), ldc = operand(C, m, "C");
    if (B.size(1) != C.size(1)) throw std::runtime_error("B and C differ in width");
    const float *scale = vector_ptr(row_scale, "row_scale"), *shift = vector_ptr(bias, "bias");
    const uint32_t flags = (scale ? DG_EPI_ROW_SCALE : 0u) | (shift ? DG_EPI_BIAS : 0u) | (relu ? DG_EPI_RELU : 0u);
    c10::cuda::CUDAGuard guard(ref->values.device());
    check(dg_spmm_csr(ref->plan, reinterpret_cast<const float*>(val), B.data_ptr<float>(), ldb, C.data_ptr<float>(), ldc, (int32_t)B.size(1), (float)alpha,
                      (float)beta, flags, scale, shift, stream_of(ref->values)));
}

// ---- operands with rows of whole 16-byte pieces ---------------------------------------------------------------------------
// t [n x w] as [n x pad4(w)] where it can be read that way in place (the columns beyond w are read and their results dropped).
bool readable_padded(const Tensor& t, int64_t width)
{
    const int64_t n = t.size(0), ld = t.stride(0);
    if (t.stride(1) != 1 || ld % 4 || ld < width || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15)) return false;
    return width == t.size(1) || t.storage_offset() + (n - 1) * ld + width <= (int64_t)(t.storage().nbytes() / 4);
}
Tensor padded_copy(const Tensor& t)
{
    const Tensor src = (t.size(1) > 1 && t.stride(1) != 1) || t.stride(0) < t.size(1) ? t.contiguous() : t;
    Tensor wide = at::empty({t.size(0), pad4(t.size(1))}, t.options());
    check(dg_pad_rows(src.data_ptr<float>(), src.size(0) > 1 ? src.stride(0) : src.size(1), src.size(0), (int32_t)src.size(1), wide.data_ptr<float>(),
                      wide.size(1), stream_of(t)));
    return wide;
}

// ---- partial results of weight gradients ------------------------------------------------------------------------------------
// A product's own, from torch's allocator: products on two streams may run at the same time, and the memory serves the next one on its stream.
int tn_ctas(const Tensor& x) { return at::cuda::getDeviceProperties(x.get_device())->multiProcessorCount; }
int64_t tn_floats(int64_t Km, int64_t Nn, int ctas)
{
    return ctas * ((std::min<int64_t>(Km, 256) + 127) / 128 * 128) * ((std::min<int64_t>(Nn, 256) + 15) / 16 * 16);
}
std::pair<Tensor, int> tn_scratch(const Tensor& x, int64_t Km, int64_t Nn)
{
    const int ctas = tn_ctas(x);
    return {at::empty({tn_floats(Km, Nn, ctas)}, x.options()), ctas};
}

// ---- the whole GCN on one rank ----------------------------------------------------------------------------------------------
struct Net {                              // shapes and buffers of one call
    std::vector<int32_t> dims;
    std::vector<float*> act;
    std::vector<int64_t> ld_act;
    std::vector<int32_t> marks;
    dg_gcn_net net{};
    Net(const PlanRef& plan, const Tensor& x, const std::vector<int32_t>& d, std::vector<float*> a) : dims(d), act(std::move(a)), marks(2 * d.size() - 1, -1)
    {
        const int L = (int)dims.size() - 1;
        for (int l = 0; l < L; ++l) ld_act.push_back(l + 1 < L ? pad4(dims[l + 1]) : dims[l + 1]);
        net.plan = plan.plan;
        net.val = plan.values.data_ptr<float>();
        net.dims = dims.data();
        net.x = x.data_ptr<float>();
        net.ldx = x.size(0) > 1 ? x.stride(0) : pad4(dims[0]);
        net.act = act.data();
        net.ld_act = ld_act.data();
        net.marks = marks.data();
        net.n = (int32_t)x.size(0);
        net.layers = L;
    }
};

struct GcnNode : public torch::autograd::Node {
    std::shared_ptr<PlanRef> plan;
    SavedVariable features;               // only to notice that they were changed in place
    std::vector<SavedVariable> weights;
    Tensor x, hidden, splits;
    std::vector<int32_t> dims;
    std::vector<int64_t> act_start, bwd_split;
    int64_t timer = 0;

    std::string name() const override { return "OneRankGcnBackward"; }
    void release_variables() override
    {
        features.reset_data();
        for (auto& w : weights) w.reset_data();
        x.reset(), hidden.reset(), splits.reset();
    }
    variable_list apply(variable_list&& grads) override
    {
        const int L = (int)dims.size() - 1;
        variable_list out((size_t)L);
        if (!grads[0].defined()) return out;
        TORCH_CHECK(x.defined(), "Trying to backward through the graph a second time");
        features.unpack();
        std::vector<Tensor> w;
        for (auto& s : weights) w.push_back(s.unpack());
        c10::cuda::CUDAGuard guard(x.device());
        const int64_t n = x.size(0), width = pad4(dims[L]);
        Tensor g = grads[0].scalar_type() == at::kFloat ? grads[0] : grads[0].to(at::kFloat);
        if (!readable_padded(g, width)) g = width == g.size(1) ? g.contiguous() : padded_copy(g);
        std::vector<float*> act;
        float* base = hidden.data_ptr<float>();
        for (int l = 0; l + 1 < L; ++l) act.push_back(base + act_start[l]);
        act.push_back(x.data_ptr<float>());               // the last activation is not read
        Net call(*plan, x, dims, act);
        int64_t widest = 0, widest_hidden = 0;
        for (int l = 1; l <= L; ++l) widest = std::max(widest, pad4(dims[l]));
        for (int l = 1; l < L; ++l) widest_hidden = std::max(widest_hidden, pad4(dims[l]));
        Tensor work = at::empty({n * (widest + widest_hidden)}, x.options());
        call.net.z = work.data_ptr<float>();
        call.net.g = L > 1 ? call.net.z + n * widest : nullptr;
        std::vector<const float*> split((size_t)L, nullptr);
        for (int l = 1; l < L; ++l) split[l] = splits.data_ptr<float>() + bwd_split[l];
        std::vector<float*> dw((size_t)L, nullptr);
        int64_t launches = 0;
        auto panels = [](int64_t d) { return (d + 255) / 256; };
        for (int l = 0; l < L; ++l) {
            if (l > 0) launches += panels(dims[l]);
            if (!task_should_compute_output((size_t)l)) continue;
            out[l] = at::empty_like(w[l]);
            dw[l] = out[l].data_ptr<float>();
            launches += 2 * panels(dims[l]) * panels(dims[l + 1]);
        }
        call.net.grad = g.data_ptr<float>();
        call.net.ld_grad = n > 1 ? g.stride(0) : width;
        call.net.dw = dw.data();
        call.net.bwd_split = split.data();
        const int ctas = tn_ctas(x);
        int64_t partials = 0;
        for (int l = 0; l < L; ++l)
            if (dw[l]) partials = std::max(partials, tn_floats(dims[l], dims[l + 1], ctas));
        Tensor partial = at::empty({std::max<int64_t>(partials, 1)}, x.options());
        call.net.tn_scratch = partial.data_ptr<float>();
        call.net.tn_scratch_floats = partial.numel();
        call.net.max_ctas = ctas;
        check(dg_gcn_backward(&call.net, stream_of(x)));
        g_launches += launches;
        add_regions(timer, std::move(call.marks), true);
        return out;
    }
};

Tensor gcn(const std::shared_ptr<PlanRef>& plan, const Tensor& features, const Tensor& x, const std::vector<Tensor>& weights, int64_t timer)
{
    const int L = (int)weights.size();
    const int64_t n = x.size(0);
    bool train = false;
    for (const Tensor& w : weights) train = train || w.requires_grad();
    train = train && at::GradMode::is_enabled();
    c10::cuda::CUDAGuard guard(x.device());
    Tensor out, hidden, splits;
    std::vector<int64_t> act_start, fwd_split((size_t)L), bwd_split((size_t)L, -1);
    std::vector<int32_t> dims(1, (int32_t)features.size(1));
    for (const Tensor& w : weights) dims.push_back((int32_t)w.size(1));
    {
        at::AutoDispatchBelowADInplaceOrView below;
        // all weights split by one launch: W^T for the forward pass, W for the backward pass of every layer but the first
        int64_t floats = 0;
        for (int l = 0; l < L; ++l) {
            fwd_split[l] = floats;
            floats += 2 * dims[l + 1] * pad4(dims[l]);
            if (train && l > 0) {
                bwd_split[l] = floats;
                floats += 2 * dims[l] * pad4(dims[l + 1]);
            }
        }
        splits = at::empty({floats}, x.options());
        std::vector<dg_split_job> jobs;
        float* sbase = splits.data_ptr<float>();
        for (int l = 0; l < L; ++l) {
            const float* w = weights[l].data_ptr<float>();
            const int32_t K = dims[l], N = dims[l + 1];
            float* f = sbase + fwd_split[l];
            jobs.push_back({w, N, f, f + N * pad4(K), pad4(K), N, K, 1, 0});
            if (bwd_split[l] >= 0) {
                float* b = sbase + bwd_split[l];
                jobs.push_back({w, N, b, b + K * pad4(N), pad4(N), K, N, 0, 0});
            }
        }
        check(dg_dense_split_operands(jobs.data(), (int32_t)jobs.size(), stream_of(x)));
        // hidden activations in one buffer: side by side while a backward pass will read them, else every layer over the last
        int64_t sum = 0, widest_in = 0, widest_hidden = 0;
        for (int l = 0; l < L; ++l) widest_in = std::max(widest_in, pad4(dims[l]));
        for (int l = 1; l < L; ++l) {
            act_start.push_back(train ? sum : 0);
            sum += n * pad4(dims[l]);
            widest_hidden = std::max(widest_hidden, pad4(dims[l]));
        }
        hidden = at::empty({train ? sum : n * widest_hidden}, x.options());
        out = at::empty({n, dims[L]}, x.options());
        Tensor z = at::empty({n * widest_in}, x.options());
        std::vector<float*> act;
        for (int64_t s : act_start) act.push_back(hidden.data_ptr<float>() + s);
        act.push_back(out.data_ptr<float>());
        Net call(*plan, x, dims, act);
        std::vector<const float*> heads;
        for (int64_t s : fwd_split) heads.push_back(sbase + s);
        call.net.z = z.data_ptr<float>();
        call.net.fwd_split = heads.data();
        check(dg_gcn_forward(&call.net, stream_of(x)));
        int64_t launches = 1;
        for (int l = 1; l <= L; ++l) launches += (dims[l] + 255) / 256;
        g_launches += launches;
        add_regions(timer, std::move(call.marks), false);
    }
    if (train) {
        auto node = std::shared_ptr<GcnNode>(new GcnNode(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(weights));
        node->plan = plan;
        node->features = SavedVariable(features, false);
        for (const Tensor& w : weights) node->weights.emplace_back(w, false);
        node->x = x.detach();
        node->hidden = hidden;
        node->splits = splits;
        node->dims = dims;
        node->act_start = act_start;
        node->bwd_split = bwd_split;
        node->timer = timer;
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ---- mean cross-entropy of the rows with a target ------------------------------------------------------------------------------
struct RowLossNode : public torch::autograd::Node {
    SavedVariable logits;
    Tensor targets, lse;
    int64_t count = 0;

    std::string name() const override { return "RowCrossEntropyBackward"; }
    void release_variables() override
    {
        logits.reset_data();
        targets.reset(), lse.reset();
    }
    variable_list apply(variable_list&& grads) override
    {
        if (!grads[0].defined()) return {Tensor()};
        TORCH_CHECK(lse.defined(), "Trying to backward through the graph a second time");
        const Tensor x = logits.unpack();
        c10::cuda::CUDAGuard guard(x.device());
        const Tensor up = grads[0].contiguous();
        const int64_t n = x.size(0), C = x.size(1), width = pad4(C);
        Tensor grad = at::empty({n, width}, x.options());
        check(dg_rows_cross_entropy_grad(x.data_ptr<float>(), n > 1 ? x.stride(0) : C, n, (int32_t)C, targets.data_ptr<int32_t>(), count, lse.data_ptr<float>(),
                                         up.data_ptr<float>(), grad.data_ptr<float>(), width, stream_of(x)));
        return {width == C ? grad : grad.narrow(1, 0, C)};
    }
};

Tensor row_cross_entropy(const Tensor& x, const Tensor& targets, int64_t count)
{
    if (!x.is_cuda() || x.scalar_type() != at::kFloat || x.dim() != 2 || (x.size(1) > 1 && x.stride(1) != 1) || (x.size(0) > 1 && x.stride(0) < x.size(1)))
        throw std::runtime_error("logits must be a row-major fp32 CUDA matrix");
    if (!targets.is_cuda() || targets.scalar_type() != at::kInt || !targets.is_contiguous() || targets.numel() != x.size(0))
        throw std::runtime_error("targets must be a contiguous int32 CUDA tensor with one entry per row");
    const bool train = x.requires_grad() && at::GradMode::is_enabled();
    c10::cuda::CUDAGuard guard(x.device());
    Tensor loss, lse;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        const int64_t n = x.size(0), parts = dg_rows_loss_scratch();
        lse = at::empty({n}, x.options());
        const Tensor sums = at::empty({parts}, x.options().dtype(at::kDouble));
        loss = at::empty({}, x.options());
        check(dg_rows_cross_entropy(x.data_ptr<float>(), n > 1 ? x.stride(0) : x.size(1), n, (int32_t)x.size(1), targets.data_ptr<int32_t>(), count,
                                    lse.data_ptr<float>(), sums.data_ptr<double>(), loss.data_ptr<float>(), stream_of(x)));
    }
    if (train) {
        auto node = std::shared_ptr<RowLossNode>(new RowLossNode(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(x));
        node->logits = SavedVariable(x, false);
        node->targets = targets;
        node->lse = lse;
        node->count = count;
        torch::autograd::set_history(loss, node);
    }
    return loss;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m)
{
    py::class_<PlanRef, std::shared_ptr<PlanRef>>(m, "PlanRef").def(py::init<int64_t, Tensor, Tensor>());
    m.def("spmm", &spmm);
    m.def("gcn", &gcn);
    m.def("readable_padded", &readable_padded);
    m.def("tn_scratch", &tn_scratch);
    m.def("row_cross_entropy", &row_cross_entropy);
    m.def("pending_regions", &pending_regions);
    m.def("resolve_regions", &resolve_regions);
    m.def("take_launches", [] { return g_launches.exchange(0); });
}
