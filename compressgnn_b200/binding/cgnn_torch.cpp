// Native host path of the layers: the operators of include/cgnn_b200.h called on torch tensors, with
// their autograd nodes, in C++.
//
// What bounds it is host time: a small propagation's six kernels take 26 us on the device.  Issued from Python it
// takes 135 us (argument checks, ctypes conversions, torch.empty calls and two autograd functions, the backward one
// behind a GIL hand-over), from here 62: the allocations and the launches.  Nothing below computes anything
// the C ABI does not.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/utils/pybind.h>

#include <mutex>
#include <tuple>
#include <vector>

#include "../../include/cgnn_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

void check(int rc) {
    if (rc != CGNN_OK) TORCH_CHECK(false, "cgnn_b200: ", cgnn_last_error());
}

int dtype_code(const Tensor &t) {
    if (t.scalar_type() == at::kFloat) return CGNN_F32;
    TORCH_CHECK(t.scalar_type() == at::kDouble, "only float32 and float64 are supported");
    return CGNN_F64;
}

cgnn_stream_t current_stream(const Tensor &t) {
    return reinterpret_cast<cgnn_stream_t>(c10::cuda::getCurrentCUDAStream(t.get_device()).stream());
}

void *data(const Tensor &t) { return t.defined() && t.numel() ? t.data_ptr() : nullptr; }

// These operators carry no forward-mode derivative: a dual number is refused, its tangent never dropped.
void refuse_dual(const char *what, at::TensorList inputs) {
    for (const Tensor &t : inputs)
        TORCH_CHECK_NOT_IMPLEMENTED(!torch::autograd::isFwGradDefined(t), what,
                                    " does not support forward-mode automatic differentiation");
}

// Is the current stream of the current device being captured?
bool capturing() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }

// Runs `fill`, which makes a buffer that launches on any stream will read from now on, and returns when the buffer is
// complete.  While the current stream is captured the buffer is made on another one: the captured graph may be
// replayed late, after other users of the buffer, or never.
template <typename Fill>
auto complete(int device, Fill &&fill) {
    c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(device);
    c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    if (capturing()) stream = c10::cuda::getStreamFromPool(false, device);
    const c10::cuda::CUDAStreamGuard guard(stream);
    auto made = fill();
    C10_CUDA_CHECK(cudaStreamSynchronize(stream));
    return made;
}

// Owner of a native plan and of its scratch: one zero-initialised buffer per (width, dtype, stream), since
// a launch leaves the ticket words zero, launches on one stream are ordered, and those that hand each other
// sums in the scratch are kept together by the plan.
class Plan {
  public:
    Plan(intptr_t handle, int device) : plan_(reinterpret_cast<cgnn_plan *>(handle)), device_(device) {
        int64_t info[8];
        check(cgnn_plan_info(plan_, info));
        rows = info[0];
        nnz = info[1];
        check(cgnn_plan_source_rows(plan_, source_rows));
    }
    Plan(const Plan &) = delete;
    ~Plan() { cgnn_plan_destroy(plan_); }

    const cgnn_plan *get() const { return plan_; }
    intptr_t address() const { return reinterpret_cast<intptr_t>(plan_); }
    int device() const { return device_; }

    std::pair<void *, size_t> scratch(int64_t width, int code, cgnn_stream_t stream) {
        std::lock_guard<std::mutex> held(lock_);
        for (const auto &s : scratch_)
            if (s.width == width && s.code == code && s.stream == stream) return {s.buffer.data_ptr(), s.buffer.numel()};
        const int64_t bytes = std::max<int64_t>((int64_t)cgnn_plan_scratch_bytes(plan_, width, code), 16);
        const c10::cuda::CUDAGuard guard(device_);
        auto zeros = [&] { return at::zeros({bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device_)); };
        const Tensor buffer = capturing() ? complete(device_, zeros) : zeros();
        TORCH_CHECK(buffer.data_ptr() != nullptr, "the operators of compressgnn_b200 need tensors with memory, not fake ones");
        buffer.record_stream(c10::cuda::getCurrentCUDAStream(device_));
        scratch_.push_back({width, code, stream, buffer});
        return {scratch_.back().buffer.data_ptr(), scratch_.back().buffer.numel()};
    }
    std::pair<intptr_t, size_t> scratch_py(int64_t width, int code, intptr_t stream) {
        auto s = scratch(width, code, reinterpret_cast<cgnn_stream_t>(stream));
        return {reinterpret_cast<intptr_t>(s.first), s.second};
    }

    int64_t rows = 0, nnz = 0;
    int64_t source_rows[2] = {0, 0};

  private:
    struct Scratch {
        int64_t width;
        int code;
        cgnn_stream_t stream;
        Tensor buffer;
    };
    cgnn_plan *plan_;
    int device_;
    std::mutex lock_;
    std::vector<Scratch> scratch_;
};
using PlanPtr = std::shared_ptr<Plan>;

// ---------------------------------------------------------------------------------------------
// compressed propagation
// ---------------------------------------------------------------------------------------------
// The launch tables of one graph: per direction the plans in launch order (rules, levels, vertices) with
// the value arrays behind them, brought into plan order once per element type.
class Propagation : public std::enable_shared_from_this<Propagation> {
  public:
    using Launch = std::pair<PlanPtr, std::vector<Tensor>>;
    Propagation(int64_t vertices, int64_t rules, std::vector<Launch> forward, std::vector<Launch> backward)
        : vertices_(vertices), rules_(rules) {
        launches_[0] = std::move(forward);
        launches_[1] = std::move(backward);
        for (auto &dir : launches_) {
            TORCH_CHECK(dir.size() >= 2, "a pass has a rule launch and a vertex launch");
            for (auto &launch : dir)
                TORCH_CHECK(launch.first && launch.first->device() == device(), "the plans must lie on one device");
        }
    }
    int device() const { return launches_[0].front().first->device(); }

    // Launches first .. last of one direction (last < 0: to the end) on the current stream.
    Tensor run(const Tensor &x_in, bool backward, const Tensor &out_in, const Tensor &rule_in, int first, int last) {
        TORCH_CHECK(x_in.is_cuda(), "compressgnn_b200 runs on CUDA tensors only (no CPU propagation path)");
        TORCH_CHECK(x_in.get_device() == device(), "the feature matrix is on cuda:", (int)x_in.get_device(),
                    " and the graph on cuda:", device());
        const Tensor x = x_in.contiguous();
        TORCH_CHECK(x.dim() == 2, "the feature matrix must have two dimensions");
        const c10::cuda::OptionalCUDAGuard guard(x.device());
        const int64_t width = x.size(1);
        Tensor out = out_in;
        if (!out.defined()) out = at::empty({vertices_, width}, x.options());
        else
            TORCH_CHECK(out.device() == x.device() && out.dim() == 2 && out.size(0) == vertices_ && out.size(1) == width &&
                            out.scalar_type() == x.scalar_type() && out.is_contiguous(),
                        "out does not match the graph and the feature matrix");
        if (out.numel() == 0) return out;
        // The rule matrix starts a whole number of rows away from x, so that the fused vertex pass reads both
        // through one base pointer and a row index (see cgnn_spmm_pair).
        Tensor rule = rule_in;
        char *rule_ptr = nullptr;
        if (rule.defined()) {
            TORCH_CHECK(rule.device() == x.device() && rule.dim() == 2 && rule.size(0) == rules_ && rule.size(1) == width &&
                            rule.scalar_type() == x.scalar_type() && rule.is_contiguous(),
                        "rule buffer does not match the graph and the feature matrix");
            rule_ptr = static_cast<char *>(data(rule));
        } else if (rules_ > 0) {
            rule = at::empty({(rules_ + 1) * width}, x.options());
            const int64_t row_bytes = width * x.element_size();
            rule_ptr = static_cast<char *>(rule.data_ptr());
            int64_t shift = (reinterpret_cast<intptr_t>(x.data_ptr()) - reinterpret_cast<intptr_t>(rule_ptr)) % row_bytes;
            rule_ptr += shift < 0 ? shift + row_bytes : shift;
        }
        const Table &t = table(backward, width, x);
        TORCH_CHECK(x.size(0) >= t.x_rows && rules_ >= t.rule_rows,
                    "propagate: the graph refers to rows beyond the feature or rule matrix");
        const int n = (int)t.plans.size();
        check(cgnn_propagate(n, t.plans.data(), t.values.data(), t.scratch.data(), t.scratch_bytes.data(), t.code, width,
                             x.data_ptr(), rule_ptr, out.data_ptr(), backward ? 1 : 0, first, last < 0 ? n - 1 : last,
                             t.stream));
        return out;
    }

    Tensor apply(const Tensor &x, bool backward);

  private:
    struct Table {
        bool backward;
        int64_t width;
        int code;
        cgnn_stream_t stream;
        int64_t x_rows, rule_rows;
        std::vector<const cgnn_plan *> plans;
        std::vector<const void *> values;
        std::vector<void *> scratch;
        std::vector<size_t> scratch_bytes;
    };

    // The value arrays of one direction in plan order.  Every stream reads the same ones, so they are complete before
    // the first launch that does.
    const std::vector<Tensor> &ordered(bool backward, const Tensor &x, int code) {
        auto &have = ordered_[backward][code];
        if (!have.empty()) return have;
        have = complete(x.get_device(), [&] {
            std::vector<Tensor> arrays;
            for (auto &launch : launches_[backward]) {
                Tensor dst = at::empty({launch.first->nnz}, x.options());
                if (launch.first->nnz) {
                    Tensor v0 = launch.second[0].to(x.scalar_type()).contiguous(), v1;
                    int64_t given = v0.numel();
                    if (launch.second.size() > 1) {
                        v1 = launch.second[1].to(x.scalar_type()).contiguous();
                        given += v1.numel();
                    }
                    TORCH_CHECK(given == launch.first->nnz, "values do not match the plan's entries");
                    check(cgnn_plan_permute_values(launch.first->get(), code, data(v0), data(v1), dst.data_ptr(),
                                                   current_stream(x)));
                }
                arrays.push_back(dst);
            }
            return arrays;
        });
        return have;
    }

    const Table &table(bool backward, int64_t width, const Tensor &x) {
        const int code = dtype_code(x);
        const cgnn_stream_t stream = current_stream(x);
        std::lock_guard<std::mutex> guard(lock_);
        for (const auto &t : tables_)
            if (t->backward == backward && t->width == width && t->code == code && t->stream == stream) return *t;
        auto t = std::make_unique<Table>();
        t->backward = backward;
        t->width = width;
        t->code = code;
        t->stream = stream;
        const auto &values = ordered(backward, x, code);
        const auto &launches = launches_[backward];
        for (size_t i = 0; i < launches.size(); ++i) {
            auto s = launches[i].first->scratch(width, code, stream);
            t->plans.push_back(launches[i].first->get());
            t->values.push_back(data(values[i]));
            values[i].record_stream(c10::cuda::getCurrentCUDAStream(x.get_device()));
            t->scratch.push_back(s.first);
            t->scratch_bytes.push_back(s.second);
        }
        const int64_t *last = launches.back().first->source_rows;
        t->x_rows = std::max(launches.front().first->source_rows[0], last[backward ? 0 : 1]);
        t->rule_rows = last[backward ? 1 : 0];
        tables_.push_back(std::move(t));
        return *tables_.back();
    }

    int64_t vertices_, rules_;
    std::vector<Launch> launches_[2];
    std::vector<Tensor> ordered_[2][2];
    std::mutex lock_;
    std::vector<std::unique_ptr<Table>> tables_;
};

// What arrives for an output whose consumer returned no gradient: zeros, as autograd functions get them.
Tensor materialized(Node &node, const Tensor &grad) { return grad.defined() ? grad : node.input_metadata(0).zeros_like(); }

struct PropagateBackward : public Node {
    std::shared_ptr<Propagation> graph;
    bool backward = false;  // direction of the pass this node differentiates
    variable_list apply(variable_list &&grads) override {
        if (!task_should_compute_output(0)) return {Tensor()};
        return {graph->apply(materialized(*this, grads[0]), !backward)};
    }
    std::string name() const override { return "CompressgnnPropagateBackward"; }
};

template <typename N>
std::shared_ptr<N> new_node() {
    return std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
}

// One direction with autograd (its derivative is the other direction).
Tensor Propagation::apply(const Tensor &x, bool backward) {
    refuse_dual("the propagation", {x});
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        out = run(x, backward, Tensor(), Tensor(), 0, -1);
    }
    if (torch::autograd::compute_requires_grad(x)) {
        auto node = new_node<PropagateBackward>();
        node->graph = shared_from_this();
        node->backward = backward;
        node->set_next_edges(torch::autograd::collect_next_edges(x));
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ---------------------------------------------------------------------------------------------
// bucket mean, Linear, reconstruction
// ---------------------------------------------------------------------------------------------
Tensor mean(const Tensor &x, const Tensor &counts, Plan &plan) {
    Tensor out = at::empty({counts.numel(), x.size(1)}, x.options());
    const int code = dtype_code(x);
    const cgnn_stream_t stream = current_stream(x);
    auto s = plan.scratch(x.size(1), code, stream);
    check(cgnn_cluster_mean(plan.get(), code, x.size(1), data(x), counts.const_data_ptr<int32_t>(), data(out), s.first,
                            s.second, stream));
    return out;
}

Tensor mean_backward(const Tensor &grad, const Tensor &index, const Tensor &counts) {
    Tensor out = at::empty({index.numel(), grad.size(1)}, grad.options());
    if (out.numel() == 0) return out;
    Tensor scaled = at::empty_like(grad);
    check(cgnn_cluster_mean_backward(dtype_code(grad), index.numel(), grad.size(1), grad.size(0), data(grad),
                                     index.const_data_ptr<int64_t>(), counts.const_data_ptr<int32_t>(), data(out),
                                     data(scaled), current_stream(grad)));
    return out;
}

Tensor reconstruct(const Tensor &reps, const Tensor &index, const Tensor &bias, bool relu, double p, uint64_t seed) {
    Tensor out = at::empty({index.numel(), reps.size(1)}, reps.options());
    if (out.numel() == 0) return out;
    const int code = dtype_code(reps);
    if (p > 0.0)
        check(cgnn_cluster_reconstruct_dropout(code, index.numel(), reps.size(1), reps.size(0), data(reps),
                                               index.const_data_ptr<int64_t>(), data(bias), p, seed, data(out),
                                               current_stream(reps)));
    else
        check(cgnn_cluster_reconstruct(code, index.numel(), reps.size(1), reps.size(0), data(reps),
                                       index.const_data_ptr<int64_t>(), data(bias), relu ? 1 : 0, data(out),
                                       current_stream(reps)));
    return out;
}

// relu: 0, 1 (mask row per node) or 2 (one mask row per group), as in cgnn_cluster_reconstruct_backward.
std::pair<Tensor, Tensor> reconstruct_backward(const Tensor &grad, const Tensor &output, int64_t groups, int relu,
                                               bool want_bias, Plan &plan) {
    const int64_t width = grad.size(1);
    Tensor out = at::empty({groups, width}, grad.options()), bias;
    if (want_bias) bias = at::empty({width}, grad.options());
    TORCH_CHECK(plan.rows == groups && plan.nnz == grad.size(0), "reconstruct backward: plan does not match index/groups");
    const int code = dtype_code(grad);
    const cgnn_stream_t stream = current_stream(grad);
    auto s = plan.scratch(width, code, stream);
    check(cgnn_cluster_reconstruct_backward(plan.get(), code, width, data(grad), relu ? data(output) : nullptr, relu,
                                            data(out), data(bias), s.first, s.second, stream));
    return {out, bias};
}

// a^T b for tall a [K, M] and b [K, N]: the weight gradient over the representatives.  The package's kernel splits K
// over the GPU; it takes fp32 at full precision with up to a GPU of output tiles (64 x 128), beyond which the
// library's tiles fill the GPU without a split, and leaves a caller who allowed TF32 products to the library.  (128 x 256 over
// 64 k rows: 158 us there, 90 here; beyond 148 tiles neither side is measured and the library stays.)
// The precision is asked for by the query that answers for all of torch's switches: the older one raises once the
// newer switch has been used.
bool full_precision_products() {
    const auto precision = at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL);
    return precision == at::Float32Precision::NONE || precision == at::Float32Precision::IEEE;
}

Tensor matmul_tn(const Tensor &a, const Tensor &b) {
    const int64_t K = a.size(0), M = a.size(1), N = b.size(1);
    const int64_t tiles = ((M + 63) / 64) * ((N + 127) / 128);
    if (a.scalar_type() != at::kFloat || tiles > 148 || tiles == 0 || !full_precision_products())
        return at::mm(a.t(), b);
    Tensor out = at::empty({M, N}, a.options());
    const size_t bytes = cgnn_matmul_tn_scratch_bytes(K, M, N);
    const Tensor scratch = at::empty({(int64_t)bytes}, a.options().dtype(at::kByte));
    check(cgnn_matmul_tn(K, M, N, static_cast<const float *>(data(a)), static_cast<const float *>(data(b)),
                         static_cast<float *>(data(out)), data(scratch), bytes, current_stream(a)));
    return out;
}

// A fresh 63-bit key from torch's host generator (follows torch.manual_seed; no device synchronisation):
// the draw of torch.randint(0, 2**63 - 1, (1,)).
uint64_t dropout_key() {
    return (uint64_t)at::randint(0, std::numeric_limits<int64_t>::max(), {1}, at::TensorOptions().dtype(at::kLong))
        .const_data_ptr<int64_t>()[0];
}

void check_matrix(const Tensor &x) {
    TORCH_CHECK(x.is_cuda() && x.dim() == 2, "Expected contiguous CUDA matrix");
    TORCH_CHECK(x.scalar_type() == at::kFloat || x.scalar_type() == at::kDouble, "Only float32 and float64 are supported");
}

void check_index(const Tensor &index, const Tensor &like) {
    TORCH_CHECK(index.device() == like.device() && index.dim() == 1 && index.is_contiguous() &&
                    index.scalar_type() == at::kLong,
                "Expected contiguous int64 index on input device");
}

void check_counts(const Tensor &counts, const Tensor &like) {
    TORCH_CHECK(counts.device() == like.device() && counts.dim() == 1 && counts.is_contiguous() &&
                    counts.scalar_type() == at::kInt && counts.numel() >= 1,
                "Expected nonempty int32 counts on input device");
}

void check_bias(const Tensor &bias, int64_t width, const Tensor &like) {
    if (bias.defined())
        TORCH_CHECK(bias.device() == like.device() && bias.scalar_type() == like.scalar_type() && bias.dim() == 1 &&
                        bias.numel() == width,
                    "Invalid reconstruction bias");
}

// (Saved tensors are unpacked with .contiguous(): what a saved-tensor hook hands back may have other strides.)
// The gradients of these nodes are final: differentiating them again raises.  That takes an incoming gradient that
// is differentiated itself; with a constant one the result is a constant.
variable_list first_order(variable_list &&result, const variable_list &incoming) {
    if (!torch::autograd::compute_requires_grad(incoming)) return std::move(result);
    variable_list wrapped;
    for (auto &t : result) {
        if (t.defined()) {
            auto error = std::make_shared<torch::autograd::Error>(
                "trying to differentiate twice a function that was marked with @once_differentiable");
            t = t.detach().requires_grad_();
            error->set_next_edges(torch::autograd::collect_next_edges(t));
            Tensor out = t.detach();
            torch::autograd::set_history(out, error);
            wrapped.push_back(out);
        } else {
            wrapped.push_back(t);
        }
    }
    return wrapped;
}

struct MeanBackward : public Node {
    SavedVariable index_, counts_;
    variable_list apply(variable_list &&grads) override {
        if (!task_should_compute_output(0)) return {Tensor()};
        Tensor dx;
        {
            at::NoGradGuard no_grad;
            const Tensor grad = materialized(*this, grads[0]).contiguous();
            const c10::cuda::OptionalCUDAGuard guard(grad.device());
            dx = mean_backward(grad, index_.unpack().contiguous(), counts_.unpack().contiguous());
        }
        return first_order({dx}, grads);
    }
    void release_variables() override {
        index_.reset_data();
        counts_.reset_data();
    }
    std::string name() const override { return "CompressgnnMeanBackward"; }
};

Tensor mean_autograd(const Tensor &x_in, const Tensor &index, const Tensor &counts, const PlanPtr &plan) {
    refuse_dual("the bucket mean", {x_in});
    check_matrix(x_in);
    check_index(index, x_in);
    check_counts(counts, x_in);
    TORCH_CHECK(index.numel() == x_in.size(0), "Input/index length mismatch");
    TORCH_CHECK(x_in.numel() == 0 || (plan && plan->rows == counts.numel() && plan->nnz == index.numel()),
                "cluster_mean: plan does not match index/count");
    const c10::cuda::OptionalCUDAGuard guard(x_in.device());
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor x = x_in.contiguous();
        out = x.numel() ? mean(x, counts, *plan) : at::zeros({counts.numel(), x.size(1)}, x.options());
    }
    if (torch::autograd::compute_requires_grad(x_in)) {
        auto node = new_node<MeanBackward>();
        node->index_ = SavedVariable(index, false);
        node->counts_ = SavedVariable(counts, false);
        node->set_next_edges(torch::autograd::collect_next_edges(x_in));
        torch::autograd::set_history(out, node);
    }
    return out;
}

// plan == null: the index did not come from an assignment; its plan is built when the backward needs it.
PlanPtr plan_for(const PlanPtr &plan, const Tensor &index, int64_t groups) {
    if (plan) return plan;
    pybind11::gil_scoped_acquire gil;
    return pybind11::module_::import("compressgnn_b200.runtime")
        .attr("index_plan")(index, groups)
        .attr("native")
        .cast<PlanPtr>();
}

std::pair<Tensor, Tensor> backward_or_zero(const Tensor &grad, const Tensor &output, int64_t groups, int relu,
                                           bool want_bias, const PlanPtr &plan) {
    if (grad.numel()) return reconstruct_backward(grad, output, groups, relu, want_bias, *plan);
    return {at::zeros({groups, grad.size(1)}, grad.options()),
            want_bias ? at::zeros({grad.size(1)}, grad.options()) : Tensor()};
}

struct ReconstructBackward : public Node {
    SavedVariable index_, output_;
    PlanPtr plan;
    int64_t groups = 0;
    bool relu = false, has_bias = false;
    double p = 0.0;
    variable_list apply(variable_list &&grads) override {
        std::pair<Tensor, Tensor> r;
        {
            at::NoGradGuard no_grad;
            const Tensor grad = materialized(*this, grads[0]).contiguous();
            const c10::cuda::OptionalCUDAGuard guard(grad.device());
            const Tensor output = relu ? output_.unpack(shared_from_this()).contiguous() : Tensor();
            const Tensor index = index_.unpack().contiguous();
            const PlanPtr segments = grad.numel() ? plan_for(plan, index, groups) : plan;
            // Without dropout the rows of a group are identical and one mask row per group suffices; with it every
            // row has its own zeros (dropped or clamped alike): exact mask, sums rescaled.
            r = backward_or_zero(grad, output, groups, relu ? (p > 0.0 ? 1 : 2) : 0, has_bias, segments);
            if (p > 0.0) {
                r.first.mul_(1.0 / (1.0 - p));
                if (has_bias) r.second.mul_(1.0 / (1.0 - p));
            }
        }
        return first_order({r.first, r.second}, grads);
    }
    void release_variables() override {
        index_.reset_data();
        output_.reset_data();
    }
    std::string name() const override { return "CompressgnnReconstructBackward"; }
};

Tensor reconstruct_autograd(const Tensor &src, const Tensor &index_in, const c10::optional<Tensor> &bias_in, bool relu,
                            double p, const PlanPtr &plan) {
    check_matrix(src);
    const Tensor index = index_in.contiguous();
    check_index(index, src);
    const Tensor bias = bias_in.has_value() ? *bias_in : Tensor();
    refuse_dual("the reconstruction", {src, bias});
    check_bias(bias, src.size(1), src);
    TORCH_CHECK(p >= 0.0 && p < 1.0, "dropout probability must lie in [0, 1)");
    TORCH_CHECK(p == 0.0 || relu, "the fused dropout follows a ReLU (the backward reads its mask off the zeros)");
    const c10::cuda::OptionalCUDAGuard guard(src.device());
    const uint64_t seed = p > 0.0 ? dropout_key() : 0;
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        out = reconstruct(src.contiguous(), index, bias.defined() ? bias.contiguous() : bias, relu, p, seed);
    }
    if (torch::autograd::compute_requires_grad(src, bias)) {
        auto node = new_node<ReconstructBackward>();
        node->plan = plan;
        node->groups = src.size(0);
        node->relu = relu;
        node->has_bias = bias.defined();
        node->p = p;
        node->index_ = SavedVariable(index, false);
        node->set_next_edges(torch::autograd::collect_next_edges(src, bias));
        torch::autograd::set_history(out, node);
        if (relu) node->output_ = SavedVariable(out, true);
    }
    return out;
}

// act(dropout)(Linear(bucket means of x)) spread back over the nodes: the three modules of a layer
// (ref: model/compressgnn/gcn.py:27-34) as one autograd node.
struct TransformBackward : public Node {
    SavedVariable index_, counts_, reps_, weight_, output_;
    PlanPtr plan;
    bool relu = false;
    double p = 0.0;
    variable_list apply(variable_list &&grads) override {
        Tensor dx, dw, db;
        {
            at::NoGradGuard no_grad;
            const Tensor grad = materialized(*this, grads[0]).contiguous();
            const c10::cuda::OptionalCUDAGuard guard(grad.device());
            // all of them, needed or not: one that was modified in place since the forward pass is an error
            const Tensor index = index_.unpack().contiguous(), counts = counts_.unpack().contiguous();
            const Tensor reps = reps_.unpack().contiguous(), weight = weight_.unpack();
            const Tensor output = relu ? output_.unpack(shared_from_this()).contiguous() : Tensor();
            auto r = backward_or_zero(grad, output, reps.size(0), relu ? (p > 0.0 ? 1 : 2) : 0, true, plan);
            if (p > 0.0) {
                r.first.mul_(1.0 / (1.0 - p));
                r.second.mul_(1.0 / (1.0 - p));
            }
            if (task_should_compute_output(1)) dw = matmul_tn(r.first, reps);
            if (task_should_compute_output(0))
                dx = mean_backward(at::mm(r.first, weight), index, counts);
            if (task_should_compute_output(2)) db = r.second;
        }
        return first_order({dx, dw, db}, grads);
    }
    void release_variables() override {
        for (SavedVariable *v : {&index_, &counts_, &reps_, &weight_, &output_}) v->reset_data();
    }
    std::string name() const override { return "CompressgnnTransformBackward"; }
};

Tensor transform_autograd(const Tensor &x_in, const Tensor &index, const Tensor &counts, const PlanPtr &plan,
                          const Tensor &weight, const c10::optional<Tensor> &bias_in, bool relu, double p) {
    check_matrix(x_in);
    check_index(index, x_in);
    check_counts(counts, x_in);
    TORCH_CHECK(index.numel() == x_in.size(0), "Input/index length mismatch");
    // (without columns the mean needs no plan, but the backward sums gradients as wide as the layer's output)
    TORCH_CHECK(x_in.size(0) == 0 || (plan && plan->rows == counts.numel() && plan->nnz == index.numel()),
                "transform: plan does not match index/count");
    const Tensor bias = bias_in.has_value() ? *bias_in : Tensor();
    refuse_dual("the transformation", {x_in, weight, bias});
    check_bias(bias, weight.size(0), x_in);
    TORCH_CHECK(p >= 0.0 && p < 1.0, "dropout probability must lie in [0, 1)");
    TORCH_CHECK(p == 0.0 || relu, "the fused dropout follows a ReLU (the backward reads its mask off the zeros)");
    const c10::cuda::OptionalCUDAGuard guard(x_in.device());
    Tensor reps, out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        reps = x_in.numel() ? mean(x_in.contiguous(), counts, *plan) : at::zeros({counts.numel(), x_in.size(1)}, x_in.options());
        const Tensor lin = at::mm(reps, weight.t());
        const uint64_t seed = p > 0.0 ? dropout_key() : 0;
        out = reconstruct(lin, index, bias.defined() ? bias.contiguous() : bias, relu, p, seed);
    }
    if (torch::autograd::compute_requires_grad(x_in, weight, bias)) {
        auto node = new_node<TransformBackward>();
        node->plan = plan;
        node->relu = relu;
        node->p = p;
        node->index_ = SavedVariable(index, false);
        node->counts_ = SavedVariable(counts, false);
        node->reps_ = SavedVariable(reps, false);
        node->weight_ = SavedVariable(weight, false);
        node->set_next_edges(torch::autograd::collect_next_edges(x_in, weight, bias));
        torch::autograd::set_history(out, node);
        if (relu) node->output_ = SavedVariable(out, true);
    }
    return out;
}

// ---------------------------------------------------------------------------------------------
// assignment
// ---------------------------------------------------------------------------------------------
std::tuple<Tensor, Tensor, int64_t, PlanPtr> assign(const Tensor &x, const Tensor &planes, int bits, const Tensor &workspace) {
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    at::AutoDispatchBelowADInplaceOrView below;
    const cgnn_stream_t stream = current_stream(x);
    const int64_t n = x.size(0);
    const auto ints = x.options().dtype(at::kInt).requires_grad(false);
    Tensor codes = at::empty({n}, ints), ids = at::empty({n}, ints.dtype(at::kLong));
    check(cgnn_cluster_codes(dtype_code(x), data(x), data(planes), n, x.size(1), bits, codes.data_ptr<int32_t>(), stream));
    int64_t active = 0;
    check(cgnn_cluster_assign(codes.data_ptr<int32_t>(), n, bits, workspace.data_ptr(), workspace.numel(),
                              ids.data_ptr<int64_t>(), &active, stream));
    Tensor counts = at::empty({active + 1}, ints);
    cgnn_plan *plan = nullptr;
    check(cgnn_cluster_assign_export(workspace.data_ptr(), n, active, counts.data_ptr<int32_t>(), &plan, 0, stream));
    return {ids, counts, active, std::make_shared<Plan>(reinterpret_cast<intptr_t>(plan), x.get_device())};
}

}  // namespace

namespace py = pybind11;

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    using nogil = py::call_guard<py::gil_scoped_release>;
    py::class_<Plan, PlanPtr>(m, "Plan")
        .def(py::init<intptr_t, int>())
        .def_property_readonly("handle", &Plan::address)
        .def("scratch", &Plan::scratch_py, nogil());
    py::class_<Propagation, std::shared_ptr<Propagation>>(m, "Propagation")
        .def(py::init<int64_t, int64_t, std::vector<Propagation::Launch>, std::vector<Propagation::Launch>>())
        .def("apply", &Propagation::apply, nogil())
        .def("run",
             [](Propagation &p, const Tensor &x, bool backward, const c10::optional<Tensor> &out,
                const c10::optional<Tensor> &rule_out, int first, int last) {
                 at::NoGradGuard no_grad;
                 return p.run(x, backward, out.value_or(Tensor()), rule_out.value_or(Tensor()), first, last);
             },
             py::arg("x"), py::arg("backward"), py::arg("out") = py::none(), py::arg("rule_out") = py::none(),
             py::arg("first") = 0, py::arg("last") = -1, nogil());
    m.def("mean", &mean_autograd, nogil());
    m.def("reconstruct", &reconstruct_autograd, nogil());
    m.def("transform", &transform_autograd, nogil());
    m.def("assign", &assign, nogil());
    m.def("matmul_tn", [](const Tensor &a, const Tensor &b) {
        TORCH_CHECK(a.is_cuda() && a.device() == b.device() && a.scalar_type() == b.scalar_type() && a.dim() == 2 &&
                        b.dim() == 2 && a.size(0) == b.size(0) && a.is_contiguous() && b.is_contiguous(),
                    "Expected contiguous CUDA matrices with equal row counts");
        const c10::cuda::OptionalCUDAGuard guard(a.device());
        at::NoGradGuard no_grad;
        return matmul_tn(a, b);
    }, nogil());
}
