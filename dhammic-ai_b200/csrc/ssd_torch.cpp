// Host path of the operators: argument checks, allocations, autograd nodes and the calls into the C ABI (include/ssd_b200.h), native
// so that a call costs the CPU about 12 us per launch: forward + backward of one scan on the fp32 kernels, nine launches, take
// the host 110 us.  (As Python autograd functions over ctypes about 200 us, more than the GPU needs for any call below some
// 300 MB.)
//
// Every operator is one autograd node.  A forward runs without recording; when a gradient is wanted the node keeps its inputs
// as saved variables (so that an input overwritten in place is noticed) and the buffers the kernels left for the backward.
// All work goes to the current stream of the tensors' device; nothing here synchronises unless the status check is on.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <atomic>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>

#include "../../include/ssd_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// What Python callers see as AssertionError (the checks the reference makes with `assert`).
struct AssertionFailed : std::runtime_error {
    using std::runtime_error::runtime_error;
};
#define SSD_ASSERT(cond, ...) \
    do {                      \
        if (!(cond)) throw AssertionFailed(c10::str(__VA_ARGS__)); \
    } while (0)

// The exception type that belongs to a return code of the C ABI.
void check(int rc) {
    if (rc >= 0) return;
    const std::string msg = ssd_b200_last_error();
    if (rc == SSD_B200_EINVAL && msg.find("not divisible by chunk_size") != std::string::npos) throw AssertionFailed(msg);
    TORCH_CHECK_VALUE(rc != SSD_B200_EINVAL, msg);
    TORCH_CHECK_NOT_IMPLEMENTED(rc != SSD_B200_EUNSUPPORTED, msg);
    TORCH_CHECK(false, "ssd_b200 error ", rc, ": ", msg);
}

// Switches of the Python layer that belong to a call.
struct Options {
    int path;          // SSD_B200_PATH_*
    bool save_states;  // keep the forward's states for the backward
};
// Synchronise after every call and report a bounded wait that ran out.  Read when a pass runs, so that the switch holds for the
// backward of a forward that ran before it was set.
std::atomic<bool> g_check_status{false};

int dtype_code(const Tensor& t) {
    if (t.scalar_type() == at::kFloat) return SSD_B200_F32;
    if (t.scalar_type() == at::kBFloat16) return SSD_B200_BF16;
    TORCH_CHECK(false, "ssd_b200 supports float32 and bfloat16 tensors, got ", t.scalar_type());
}

// Contiguous and, where the storage starts between two 16-byte boundaries, copied to a fresh one (TMA needs them).
Tensor dense(const Tensor& t) {
    Tensor c = t.contiguous();
    return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15) ? c.clone() : c;
}
Tensor dense_as(const Tensor& t, at::ScalarType type) { return dense(t.scalar_type() == type ? t : t.to(type)); }
Tensor f32(const Tensor& t) { return t.to(at::kFloat).contiguous(); }
Tensor cast(const Tensor& t, at::ScalarType type) { return t.defined() && t.scalar_type() != type ? t.to(type) : t; }

template <class T = void>
T* ptr(const Tensor& t) {
    return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}
Tensor get(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

Tensor empty_f32(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().dtype(at::kFloat)); }
Tensor bytes(size_t n, const Tensor& like) {
    return at::empty({static_cast<int64_t>(n < 256 ? 256 : n)}, like.options().dtype(at::kByte));
}

void check_inputs(const Tensor& x, const Tensor& B, const Tensor& C) {
    SSD_ASSERT(x.is_cuda() && B.is_cuda() && C.is_cuda(), "ssd_b200 runs on CUDA tensors only (no CPU fallback)");
    TORCH_CHECK_VALUE(x.dim() == 4 && B.dim() == 4 && C.dim() == 4, "expected x (b,T,h,p) and B, C (b,T,g,n)");
    TORCH_CHECK_VALUE(B.sizes() == C.sizes() && B.size(0) == x.size(0) && B.size(1) == x.size(1), "shape mismatch: x ", x.sizes(), ", B ",
                      B.sizes(), ", C ", C.sizes());
    TORCH_CHECK(x.scalar_type() == B.scalar_type() && B.scalar_type() == C.scalar_type(),
                "expected x, B and C to have the same dtype, got ", x.scalar_type(), ", ", B.scalar_type(), ", ", C.scalar_type());
    TORCH_CHECK_VALUE(B.device() == x.device() && C.device() == x.device(), "x, B and C are on different devices");
}

// A tensor whose values a kernel reads by x's sizes: on x's device, and with as many values as those sizes have.
void check_like(const char* name, const Tensor& t, const Tensor& x, int64_t numel) {
    if (!t.defined()) return;
    SSD_ASSERT(t.is_cuda(), "ssd_b200 runs on CUDA tensors only (no CPU fallback): ", name);
    TORCH_CHECK_VALUE(t.device() == x.device(), name, " is on ", t.device(), ", x on ", x.device());
    TORCH_CHECK_VALUE(t.numel() == numel, name, " has shape ", t.sizes(), ": expected ", numel, " values for x ", x.sizes());
}

ssd_b200_shape make_shape(const Tensor& x, int a_dtype, const Tensor& B, int64_t chunk, int path) {
    return {SSD_B200_ABI_VERSION, dtype_code(x), a_dtype, path, x.size(0), x.size(1), x.size(2), x.size(3), B.size(3), B.size(2), chunk};
}

// The workspace of a call, or the least it runs with where the device has no room for the whole.
Tensor workspace(const ssd_b200_shape& s, int pass, const Tensor& like) {
    const size_t n = ssd_b200_workspace_bytes(&s, pass), least = ssd_b200_workspace_min_bytes(&s, pass);
    if (n == 0) check(ssd_b200_resolve_path(&s));
    try {
        return bytes(n, like);
    } catch (const c10::OutOfMemoryError&) {
        if (least >= n) throw;
    }
    return bytes(least, like);
}

void check_status(const ssd_b200_shape& s, const Tensor& ws) {
    if (g_check_status.load(std::memory_order_relaxed)) check(ssd_b200_device_status(&s, ptr(ws), stream_of(ws)));
}

// The operators have reverse-mode derivatives only.  A tangent would be dropped without a word (the kernels see values), which the
// caller would read as a zero derivative.
void refuse_tangents(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(),
                                    "ssd_b200 operators have no jvp: they cannot be used with forward-mode AD");
}

bool wants_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// The per-position and per-head arguments of the forms with dt and A_head.
void check_coefficients(const Tensor& x, const Tensor& dt, const Tensor& A_head, const Tensor& D, const Tensor& init, int64_t n) {
    check_like("dt", dt, x, x.size(0) * x.size(1) * x.size(2));
    check_like("A_head", A_head, x, x.size(2));
    check_like("D", D, x, x.size(2));
    check_like("initial_states", init, x, x.size(0) * x.size(2) * x.size(3) * n);
}

// The inputs of one scan in the form the kernels read (see ssd_b200_fwd_args for the forms), and what its forward leaves.
struct Scan {
    ssd_b200_shape shape{};
    Tensor x, a, dt, A_head, D, B, C, init, skip;  // undefined = not given
    Tensor cum, states;
};

struct ScanOut {
    Tensor y, final_state;
};

ScanOut scan_forward(Scan& s, int64_t chunk, const Options& o, const Tensor& cum_in, bool want_states, const Tensor& ysq = {}) {
    const int64_t b = s.x.size(0), T = s.x.size(1), h = s.x.size(2), p = s.x.size(3), n = s.B.size(3);
    SSD_ASSERT(chunk > 0 && T % chunk == 0, "sequence length ", T, " not divisible by chunk_size ", chunk);
    s.shape = make_shape(s.x, s.a.defined() ? dtype_code(s.a) : SSD_B200_F32, s.B, chunk, o.path);
    ScanOut out{at::empty_like(s.x), empty_f32({b, h, p, n}, s.x)};
    if (cum_in.defined()) {
        s.cum = f32(cum_in);
        TORCH_CHECK_VALUE(s.cum.sizes() == at::IntArrayRef({b, h, T / chunk, chunk}), "A_cumsum cache has shape ", s.cum.sizes(), ", expected ",
                          at::IntArrayRef({b, h, T / chunk, chunk}));
    } else {
        s.cum = empty_f32({b, h, T / chunk, chunk}, s.x);
    }
    const Tensor ws = workspace(s.shape, SSD_B200_PASS_FWD, s.x);
    if (want_states && o.save_states)
        if (const size_t nb = ssd_b200_states_bytes(&s.shape)) s.states = bytes(nb, s.x);
    ssd_b200_fwd_args a{};
    a.shape = s.shape;
    a.x = ptr(s.x); a.a = ptr(s.a); a.dt = ptr<float>(s.dt); a.A_head = ptr<float>(s.A_head); a.D = ptr<float>(s.D);
    a.B = ptr(s.B); a.C = ptr(s.C); a.init = ptr<float>(s.init); a.y = ptr(out.y); a.final_state = ptr<float>(out.final_state);
    a.a_cumsum = ptr<float>(s.cum); a.cumsum_is_input = cum_in.defined(); a.workspace = ptr(ws); a.workspace_bytes = ws.numel();
    a.states = ptr(s.states); a.ysq = ptr<float>(ysq); a.skip = ptr<float>(s.skip);
    check(ssd_b200_fwd(&a, stream_of(s.x)));
    check_status(s.shape, ws);
    return out;
}

struct ScanGrads {
    Tensor dx, dB, dC, da, ddt, dA_head, dD, dinit, dskip;
};

ScanGrads scan_backward(const Scan& s, const Tensor& dy, const Tensor& dfinal, bool cached) {
    const int64_t b = s.x.size(0), T = s.x.size(1), h = s.x.size(2);
    const bool operator_form = s.a.defined(), mamba2 = !operator_form, scaled = operator_form && s.dt.defined();
    ScanGrads g;
    g.dx = at::empty_like(s.x);
    g.dB = at::empty_like(s.B);
    g.dC = at::empty_like(s.C);
    if (operator_form && !cached) g.da = empty_f32({b, T, h}, s.x);
    if (mamba2 || scaled) g.ddt = empty_f32({b, T, h}, s.x);
    if (mamba2) g.dA_head = empty_f32({h}, s.x);
    if (s.D.defined()) g.dD = empty_f32({h}, s.x);
    if (scaled) g.dskip = empty_f32({b, T, h}, s.x);
    if (s.init.defined()) g.dinit = at::empty_like(s.init);
    const Tensor ws = workspace(s.shape, SSD_B200_PASS_BWD, s.x);
    ssd_b200_bwd_args a{};
    a.shape = s.shape;
    a.x = ptr(s.x); a.a = ptr(s.a); a.dt = ptr<float>(s.dt); a.A_head = ptr<float>(s.A_head); a.D = ptr<float>(s.D);
    a.B = ptr(s.B); a.C = ptr(s.C); a.init = ptr<float>(s.init); a.a_cumsum = ptr<float>(s.cum); a.dy = ptr(dy);
    a.dfinal = ptr<float>(dfinal); a.dx = ptr(g.dx); a.dB = ptr(g.dB); a.dC = ptr(g.dC); a.da = ptr<float>(g.da);
    a.ddt = ptr<float>(g.ddt); a.dA_head = ptr<float>(g.dA_head); a.dD = ptr<float>(g.dD); a.dinit = ptr<float>(g.dinit);
    a.cumsum_is_input = cached; a.workspace = ptr(ws); a.workspace_bytes = ws.numel(); a.states = ptr(s.states);
    a.skip = ptr<float>(s.skip); a.dskip = ptr<float>(g.dskip);
    check(ssd_b200_bwd(&a, stream_of(s.x)));
    check_status(s.shape, ws);
    return g;
}

// A node's hold on the scan it differentiates: inputs as saved variables, buffers as they are.
struct SavedScan {
    ssd_b200_shape shape{};
    SavedVariable x, a, dt, A_head, D, B, C, init, skip, cum;
    Tensor states;
    void save(const Scan& s) {
        shape = s.shape;
        x = SavedVariable(s.x, false); a = SavedVariable(s.a, false); dt = SavedVariable(s.dt, false);
        A_head = SavedVariable(s.A_head, false); D = SavedVariable(s.D, false); B = SavedVariable(s.B, false);
        C = SavedVariable(s.C, false); init = SavedVariable(s.init, false); skip = SavedVariable(s.skip, false);
        cum = SavedVariable(s.cum, false);
        states = s.states;
    }
    Scan load() const {
        return {shape, x.unpack(), a.unpack(), dt.unpack(), A_head.unpack(), D.unpack(), B.unpack(), C.unpack(), init.unpack(),
                skip.unpack(), cum.unpack(), states};
    }
    void release() {
        for (SavedVariable* v : {&x, &a, &dt, &A_head, &D, &B, &C, &init, &skip, &cum}) v->reset_data();
        states.reset();
    }
};

// A node with saved variables.  Two threads can run backward through one graph, so unpacking and releasing take the node's lock; a
// second backward through a freed graph is reported as torch reports it.
struct SavingNode : Node {
    bool released = false;
    virtual void release_saved() = 0;
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        release_saved();
        released = true;
    }
    // What `unpack` returns: the saved tensors, taken out while nobody releases them.
    template <class F>
    auto unpacked(F&& unpack) {
        std::lock_guard<std::mutex> lock(mutex_);
        TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
        return unpack();
    }
};
struct ScanNode : SavingNode {
    SavedScan saved;
    void release_saved() override { saved.release(); }
    Scan load() {
        return unpacked([&] { return saved.load(); });
    }
};

// A node behind the given inputs (undefined ones get no edge).
template <class N, class... Inputs>
std::shared_ptr<N> link_node(const Inputs&... inputs) {
    auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(inputs...));
    return node;
}
template <class N, class... Inputs>
std::shared_ptr<N> new_node(const Scan& s, const Inputs&... inputs) {
    auto node = link_node<N>(inputs...);
    node->saved.save(s);
    return node;
}

Tensor dfinal_of(const Tensor& g) { return g.defined() ? f32(g) : Tensor(); }

// ---------------------------------------------------------------------------------------------------- Mamba-2 form
struct Mamba2Node : ScanNode {
    at::ScalarType dt_type, A_type, D_type;
    std::vector<int64_t> init_shape;
    std::string name() const override { return "SSDMamba2Backward"; }
    variable_list apply(variable_list&& grads) override {
        at::NoGradGuard no_grad;
        const Scan s = load();
        c10::cuda::CUDAGuard guard(s.x.device());
        const Tensor dy = grads[0].defined() ? dense_as(grads[0], s.x.scalar_type()) : at::zeros_like(s.x);
        const ScanGrads g = scan_backward(s, dy, dfinal_of(grads[1]), false);
        return {g.dx, cast(g.ddt, dt_type), cast(g.dA_head, A_type), g.dB, g.dC, cast(g.dD, D_type),
                g.dinit.defined() ? g.dinit.view(init_shape) : Tensor()};
    }
};

std::tuple<Tensor, Tensor> mamba2(const Tensor& x, const Tensor& dt, const Tensor& A_head, const Tensor& B, const Tensor& C, const OptTensor& D_,
                                  int64_t chunk, const OptTensor& init_, int path, bool save_states) {
    const Options o{path, save_states};
    const Tensor D = get(D_), init = get(init_);
    refuse_tangents({&x, &dt, &A_head, &B, &C, &D, &init});
    check_inputs(x, B, C);
    check_coefficients(x, dt, A_head, D, init, B.size(3));
    c10::cuda::CUDAGuard guard(x.device());
    const bool grad = wants_grad({&x, &dt, &A_head, &B, &C, &D, &init});
    Scan s;
    ScanOut out;
    {
        at::NoGradGuard no_grad;
        s.x = dense(x); s.dt = f32(dt); s.A_head = f32(A_head); s.B = dense(B); s.C = dense(C);
        if (D.defined()) s.D = f32(D);
        if (init.defined()) s.init = f32(init.reshape({x.size(0), x.size(2), x.size(3), B.size(3)}));
        out = scan_forward(s, chunk, o, {}, grad);
    }
    if (grad) {
        auto node = new_node<Mamba2Node>(s, x, dt, A_head, B, C, D, init);
        node->dt_type = dt.scalar_type();
        node->A_type = A_head.scalar_type();
        if (D.defined()) node->D_type = D.scalar_type();
        if (init.defined()) node->init_shape = init.sizes().vec();
        torch::autograd::set_history(out.y, node);
        torch::autograd::set_history(out.final_state, node);
    }
    return {out.y, out.final_state};
}

// ---------------------------------------------------------------------------------------------------- operator form
struct OperatorNode : ScanNode {
    at::ScalarType A_type, init_type;
    std::vector<int64_t> init_shape;
    bool cached = false;
    std::string name() const override { return "FusedSSDScanBackward"; }
    variable_list apply(variable_list&& grads) override {
        at::NoGradGuard no_grad;
        const Scan s = load();
        c10::cuda::CUDAGuard guard(s.x.device());
        const Tensor dy = grads[0].defined() ? dense_as(grads[0], s.x.scalar_type()) : at::zeros_like(s.x);
        const ScanGrads g = scan_backward(s, dy, dfinal_of(grads[1]), cached);
        return {g.dx, cast(g.da, A_type), g.dB, g.dC, g.dinit.defined() ? cast(g.dinit.view(init_shape), init_type) : Tensor()};
    }
};

// (Y, final state in x's dtype, A_cumsum); `cum_in` is the A_cumsum of an earlier call (then A gets no gradient, as in the reference)
std::tuple<Tensor, Tensor, Tensor> operator_scan(const Tensor& x, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk,
                                                 const OptTensor& init_, const OptTensor& cum_in, int path, bool save_states) {
    const Options o{path, save_states};
    const Tensor init = get(init_), cached = get(cum_in);
    refuse_tangents({&x, &A, &B, &C, &init, &cached});
    check_inputs(x, B, C);
    check_like("A", A, x, x.size(0) * x.size(1) * x.size(2));
    check_like("initial_states", init, x, x.size(0) * x.size(2) * x.size(3) * B.size(3));
    check_like("A_cumsum", cached, x, x.size(0) * x.size(1) * x.size(2));
    c10::cuda::CUDAGuard guard(x.device());
    const bool grad = wants_grad({&x, &A, &B, &C, &init});
    Scan s;
    ScanOut out;
    {
        at::NoGradGuard no_grad;
        s.x = dense(x); s.a = A.contiguous(); s.B = dense(B); s.C = dense(C);
        if (init.defined()) s.init = f32(init.reshape({x.size(0), x.size(2), x.size(3), B.size(3)}));
        out = scan_forward(s, chunk, o, cached, grad);
        out.final_state = cast(out.final_state, x.scalar_type());
    }
    if (grad) {
        auto node = new_node<OperatorNode>(s, x, A, B, C, init);
        node->A_type = A.scalar_type();
        node->cached = cum_in.has_value();
        if (init.defined()) {
            node->init_shape = init.sizes().vec();
            node->init_type = init.scalar_type();
        }
        torch::autograd::set_history(out.y, node);
        torch::autograd::set_history(out.final_state, node);
    }
    // (sums that came in leave without the graph that made them: they get no gradient here)
    return {out.y, out.final_state, cached.defined() ? s.cum.detach() : s.cum};
}

// ---------------------------------------------------------------------------------------------------- norm and gate
// Rows of `cols` values (of zero columns: none, which the C ABI refuses).
int64_t rows_of(const Tensor& t, int64_t cols) { return cols ? t.numel() / cols : 0; }

struct NormGrads {
    Tensor dx, dz, dw;
};
NormGrads norm_backward(const Tensor& x, const Tensor& w, const Tensor& z, const Tensor& dout, const Tensor& rstd) {
    const int64_t D = w.numel(), rows = rstd.numel();
    NormGrads g{at::empty_like(x), z.defined() ? at::empty_like(z) : Tensor(), empty_f32({D}, x)};
    const Tensor ws = empty_f32({static_cast<int64_t>(ssd_b200_rmsnorm_ws_floats(rows, D))}, x);
    check(ssd_b200_rmsnorm_bwd(dtype_code(x), rows, D, ptr(x), ptr<float>(w), ptr(z), ptr(dout), ptr<float>(rstd), ptr(g.dx), ptr(g.dz),
                               ptr<float>(g.dw), ptr<float>(ws), stream_of(x)));
    return g;
}

struct NormNode : SavingNode {
    SavedVariable x, w, z, rstd;
    at::ScalarType w_type, z_type;
    std::string name() const override { return "FusedRMSNormBackward"; }
    void release_saved() override {
        for (SavedVariable* v : {&x, &w, &z, &rstd}) v->reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor()};
        at::NoGradGuard no_grad;
        const auto [xv, wv, zv, rv] = unpacked([&] { return std::tuple(x.unpack(), w.unpack(), z.unpack(), rstd.unpack()); });
        c10::cuda::CUDAGuard guard(xv.device());
        const NormGrads g = norm_backward(xv, wv, zv, cast(grads[0].contiguous(), xv.scalar_type()), rv);
        return {g.dx, cast(g.dw, w_type), cast(g.dz, z_type)};
    }
};

Tensor rmsnorm(const Tensor& x, const Tensor& weight, double eps, const OptTensor& z_) {
    const Tensor z = get(z_);
    refuse_tangents({&x, &weight, &z});
    SSD_ASSERT(x.is_cuda() && weight.is_cuda(), "FusedRMSNorm requires CUDA tensors");
    const int64_t D = x.size(-1);
    SSD_ASSERT(weight.dim() == 1 && weight.size(0) == D, "weight shape ", weight.sizes(), " mismatches D=", D);
    if (z.defined()) SSD_ASSERT(z.is_cuda() && z.sizes() == x.sizes(), "gate shape ", z.sizes(), " vs x ", x.sizes());
    check_like("weight", weight, x, D);
    check_like("gate", z, x, x.numel());
    c10::cuda::CUDAGuard guard(x.device());
    Tensor xc, zc, w, out, rstd;
    {
        at::NoGradGuard no_grad;
        xc = x.contiguous();
        w = f32(weight);
        if (z.defined()) zc = cast(z.contiguous(), x.scalar_type());
        const int64_t rows = rows_of(xc, D);
        out = at::empty_like(xc);
        rstd = empty_f32({rows}, x);
        check(ssd_b200_rmsnorm_fwd(dtype_code(xc), rows, D, static_cast<float>(eps), ptr(xc), ptr<float>(w), ptr(zc), ptr(out), ptr<float>(rstd), stream_of(x)));
    }
    if (wants_grad({&x, &weight, &z})) {
        auto node = link_node<NormNode>(x, weight, z);
        node->x = SavedVariable(xc, false); node->w = SavedVariable(w, false);
        node->z = SavedVariable(zc, false); node->rstd = SavedVariable(rstd, false);
        node->w_type = weight.scalar_type();
        if (z.defined()) node->z_type = z.scalar_type();
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ---------------------------------------------------------------------------------------------------- scan + norm + gate
// The scan followed by the block's output stage, out = rmsnorm(y over all heads) * silu(z)
// (src/mamba_base_engine.py:189-191).  The forward walk leaves the per-half-row sums of y^2 behind, from its fp32 values: the
// statistic carries no rounding of y to its storage type, and the norm reads y once however wide the row.
struct GatedNode : ScanNode {
    SavedVariable y, z, w, rstd;
    at::ScalarType dt_type, A_type, D_type, z_type, w_type;
    std::vector<int64_t> init_shape, z_shape, w_shape;
    std::string name() const override { return "SSDMamba2GatedBackward"; }
    void release_saved() override {
        ScanNode::release_saved();
        for (SavedVariable* v : {&y, &z, &w, &rstd}) v->reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        at::NoGradGuard no_grad;
        const auto [s, yv, wv, zv, rv] = unpacked([&] { return std::tuple(saved.load(), y.unpack(), w.unpack(), z.unpack(), rstd.unpack()); });
        c10::cuda::CUDAGuard guard(s.x.device());
        const Tensor dout = grads[0].defined() ? dense_as(grads[0], s.x.scalar_type()) : at::zeros_like(s.x);
        const NormGrads n = norm_backward(yv, wv, zv, dout, rv);
        const ScanGrads g = scan_backward(s, n.dx, dfinal_of(grads[1]), false);
        return {g.dx, cast(g.ddt, dt_type), cast(g.dA_head, A_type), g.dB, g.dC, cast(g.dD, D_type), cast(n.dz.view(z_shape), z_type),
                cast(n.dw.view(w_shape), w_type), g.dinit.defined() ? g.dinit.view(init_shape) : Tensor()};
    }
};

std::tuple<Tensor, Tensor> mamba2_gated(const Tensor& x, const Tensor& dt, const Tensor& A_head, const Tensor& B, const Tensor& C, const OptTensor& D_,
                                        const Tensor& z, const Tensor& weight, double eps, int64_t chunk, const OptTensor& init_, int path,
                                        bool save_states) {
    const Options o{path, save_states};
    const Tensor D = get(D_), init = get(init_);
    refuse_tangents({&x, &dt, &A_head, &B, &C, &D, &z, &weight, &init});
    check_inputs(x, B, C);
    check_coefficients(x, dt, A_head, D, init, B.size(3));
    check_like("norm_weight", weight, x, x.size(2) * x.size(3));
    check_like("z", z, x, x.numel());
    SSD_ASSERT(z.is_cuda() && z.dim() >= 2 && z.size(0) == x.size(0) && z.size(1) == x.size(1) && z.numel() == x.numel(),
               "the gate must have the size of y: ", z.sizes(), " vs ", x.sizes());
    c10::cuda::CUDAGuard guard(x.device());
    const bool grad = wants_grad({&x, &dt, &A_head, &B, &C, &D, &z, &weight, &init});
    const int64_t b = x.size(0), T = x.size(1), h = x.size(2), p = x.size(3), rows = b * T, Dn = h * p;
    Scan s;
    ScanOut scan;
    Tensor zc, w, out, rstd;
    {
        at::NoGradGuard no_grad;
        s.x = dense(x); s.dt = f32(dt); s.A_head = f32(A_head); s.B = dense(B); s.C = dense(C);
        if (D.defined()) s.D = f32(D);
        if (init.defined()) s.init = f32(init.reshape({b, h, p, B.size(3)}));
        const ssd_b200_shape probe = make_shape(s.x, SSD_B200_F32, s.B, chunk, path);
        const int rp = ssd_b200_resolve_path(&probe);
        check(rp);
        Tensor ysq;
        if (rp == SSD_B200_PATH_TC && T % 128 == 0) ysq = empty_f32({rows * h * 2}, x);
        scan = scan_forward(s, chunk, o, {}, grad, ysq);
        zc = cast(z.contiguous(), x.scalar_type());
        w = f32(weight);
        out = at::empty_like(scan.y);
        rstd = empty_f32({rows}, x);
        const int dtc = dtype_code(scan.y);
        if (ysq.defined())
            check(ssd_b200_rmsnorm_fwd_presummed(dtc, rows, Dn, static_cast<float>(eps), ptr(scan.y), ptr<float>(w), ptr(zc), ptr<float>(ysq), h,
                                                 ptr(out), ptr<float>(rstd), stream_of(x)));
        else
            check(ssd_b200_rmsnorm_fwd(dtc, rows, Dn, static_cast<float>(eps), ptr(scan.y), ptr<float>(w), ptr(zc), ptr(out), ptr<float>(rstd), stream_of(x)));
    }
    if (grad) {
        auto node = new_node<GatedNode>(s, x, dt, A_head, B, C, D, z, weight, init);
        node->y = SavedVariable(scan.y, false); node->z = SavedVariable(zc, false);
        node->w = SavedVariable(w, false); node->rstd = SavedVariable(rstd, false);
        node->dt_type = dt.scalar_type(); node->A_type = A_head.scalar_type();
        node->z_type = z.scalar_type(); node->w_type = weight.scalar_type();
        node->z_shape = z.sizes().vec();
        node->w_shape = weight.sizes().vec();
        if (D.defined()) node->D_type = D.scalar_type();
        if (init.defined()) node->init_shape = init.sizes().vec();
        torch::autograd::set_history(out, node);
        torch::autograd::set_history(scan.final_state, node);
    }
    return {out, scan.final_state};
}

// ---------------------------------------------------------------------------------------------------- Mamba-3 form
// The reference block's two scans as one, see mamba3.py.  `fused`: the scan takes the input weight w and the skip
// coefficient per position (tensor-core path); otherwise x * w is written and the scan runs in plain operator form.
struct Mamba3Node : ScanNode {
    ssd_b200_shape block{};  // ungrouped shape of the element-wise kernels
    SavedVariable x, dt, lam, A_head, D, B, C, cum, sdot;
    at::ScalarType ang_type, dt_type, A_type, D_type, raw_type, lam_type;
    bool fused = false;
    std::string name() const override { return "SSDMamba3Backward"; }
    void release_saved() override {
        ScanNode::release_saved();
        for (SavedVariable* v : {&x, &dt, &lam, &A_head, &D, &B, &C, &cum, &sdot}) v->reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        at::NoGradGuard no_grad;
        const auto [s, xv, dtv, lamv, Ah, Dv, Bv, Cv, cumv, sd] = unpacked([&] {
            return std::tuple(saved.load(), x.unpack(), dt.unpack(), lam.unpack(), A_head.unpack(), D.unpack(), B.unpack(), C.unpack(), cum.unpack(),
                              sdot.unpack());
        });
        c10::cuda::CUDAGuard guard(xv.device());
        const int64_t b = xv.size(0), T = xv.size(1), h = xv.size(2), n = Bv.size(3);
        const Tensor dy = grads[0].defined() ? dense_as(grads[0], xv.scalar_type()) : at::zeros_like(xv);
        ScanGrads g = scan_backward(s, dy, {}, false);
        // fused: dx is complete; dw = <dX, x> and dyx = <dy, x> come from the scan's own row sums
        Tensor dx = g.dx, dxw, dw = g.ddt, dyx = g.dskip;
        if (!fused) {
            dxw = g.dx;
            dx = at::empty_like(xv);
            dw = empty_f32({b, T, h}, xv);
            dyx = at::empty_like(dw);
        }
        const Tensor dB = at::empty_like(Bv), dC = at::empty_like(Cv);
        const Tensor dang = at::empty({b, T, h, n / 2}, xv.options().dtype(ang_type));
        const Tensor dcum = ssd_b200_m3_dcum_ws_floats(&block, ptr(Bv), ptr(Cv), ptr<float>(cumv), ptr(g.dB), ptr(g.dC)) ? empty_f32({b, T, h, n / 2}, xv) : Tensor();
        const Tensor seg = empty_f32({b * ((T + 127) / 128) * h * (n / 2)}, xv);
        void* st = stream_of(xv);
        check(ssd_b200_m3_prologue_bwd(&block, ptr(xv), ptr(dy), ptr<float>(dtv), ptr<float>(lamv), ptr<float>(Dv), ptr(Bv), ptr(Cv), ptr<float>(cumv),
                                       ptr<float>(sd), ptr(dxw), ptr(g.dB), ptr(g.dC), ptr(dx), ptr<float>(dw), ptr<float>(dyx), ptr(dB), ptr(dC),
                                       ptr(dang), dtype_code(dang), ptr<float>(dcum), ptr<float>(seg), st));
        // chain rule through w = lam dt + u, u[t] = (1 - lam[t+1]) dt[t+1], the diagonal term -u s x and
        // a = dt A_head, with the two per-head sums, in one kernel on the (b,T,h) tensors
        const Tensor dlam = at::empty_like(dw), ddt = at::empty_like(dw), dAh = empty_f32({h}, xv);
        const Tensor dD = Dv.defined() ? empty_f32({h}, xv) : Tensor();
        const Tensor ws = empty_f32({static_cast<int64_t>(ssd_b200_m3_chain_ws_floats(&block))}, xv);
        check(ssd_b200_m3_chain_bwd(&block, ptr<float>(dw), ptr<float>(dyx), ptr<float>(sd), ptr<float>(dtv), ptr<float>(lamv), ptr<float>(g.da),
                                    ptr<float>(Ah), ptr<float>(dlam), ptr<float>(ddt), ptr<float>(dAh), ptr<float>(dD), ptr<float>(ws), st));
        return {dx, cast(ddt, dt_type), cast(dAh, A_type), dB, dC, cast(dD, D_type), cast(dang, raw_type), cast(dlam, lam_type)};
    }
};

Tensor mamba3(const Tensor& x, const Tensor& dt, const Tensor& A_head, const Tensor& B, const Tensor& C, const OptTensor& D_, const Tensor& raw_angles,
              const Tensor& lam, int64_t chunk, int path, bool save_states) {
    const Options o{path, save_states};
    const Tensor D = get(D_);
    refuse_tangents({&x, &dt, &A_head, &B, &C, &D, &raw_angles, &lam});
    check_inputs(x, B, C);
    check_coefficients(x, dt, A_head, D, {}, B.size(3));
    check_like("lam", lam, x, x.size(0) * x.size(1) * x.size(2));
    TORCH_CHECK_VALUE(B.size(3) % 2 == 0, "d_state must be even for the pairwise rotation, got ", B.size(3));
    check_like("raw_angles", raw_angles, x, x.size(0) * x.size(1) * x.size(2) * (B.size(3) / 2));
    c10::cuda::CUDAGuard guard(x.device());
    const bool grad = wants_grad({&x, &dt, &A_head, &B, &C, &D, &raw_angles, &lam});
    const int64_t b = x.size(0), T = x.size(1), h = x.size(2), g = B.size(2), n = B.size(3);
    Scan s;
    ScanOut out;
    Tensor xc, dtc, lamc, Ah, Dc, Bc, Cc, ang, cum, sdot;
    ssd_b200_shape block;
    bool fused;
    {
        at::NoGradGuard no_grad;
        xc = dense(x); Bc = dense(B); Cc = dense(C);
        // angles keep their own precision: fp32 angles (the reference's dt * theta product) are summed as given
        ang = dense(raw_angles);
        if (ang.scalar_type() != at::kFloat && ang.scalar_type() != x.scalar_type()) ang = ang.to(at::kFloat);
        dtc = f32(dt); lamc = f32(lam); Ah = f32(A_head);
        if (D.defined()) Dc = f32(D);
        block = make_shape(xc, SSD_B200_F32, Bc, T, SSD_B200_PATH_AUTO);
        ssd_b200_shape probe = block;  // the scan sees one head per group (per-head rotated B, C)
        probe.ngroups = h;
        probe.chunk = chunk;
        fused = ssd_b200_resolve_path(&probe) == SSD_B200_PATH_TC;
        s.a = empty_f32({b, T, h}, x);
        s.B = at::empty({b, T, h, n}, xc.options());
        s.C = at::empty_like(s.B);
        sdot = empty_f32({b, T, g}, x);
        cum = empty_f32({b, T, h, n / 2}, x);
        const Tensor seg = empty_f32({b * ((T + 127) / 128) * h * (n / 2)}, x);
        if (fused) {
            s.x = xc;
            s.dt = at::empty_like(s.a);
            s.skip = at::empty_like(s.a);
        } else {
            s.x = at::empty_like(xc);
        }
        check(ssd_b200_m3_prologue_fwd(&block, ptr(xc), ptr<float>(dtc), ptr<float>(lamc), ptr<float>(Ah), ptr(Bc), ptr(Cc), ptr(ang), dtype_code(ang),
                                       fused ? nullptr : ptr(s.x), ptr<float>(s.a), ptr(s.B), ptr(s.C), ptr<float>(sdot), ptr<float>(cum),
                                       ptr<float>(seg), ptr<float>(Dc), ptr<float>(s.dt), ptr<float>(s.skip), stream_of(x)));
        out = scan_forward(s, chunk, o, {}, grad);
        if (!fused)
            check(ssd_b200_m3_skip_fwd(&block, ptr(out.y), ptr(xc), ptr<float>(Dc), ptr<float>(dtc), ptr<float>(lamc), ptr<float>(sdot), ptr(out.y),
                                       stream_of(x)));
    }
    if (grad) {
        auto node = new_node<Mamba3Node>(s, x, dt, A_head, B, C, D, raw_angles, lam);
        node->block = block;
        node->x = SavedVariable(xc, false); node->dt = SavedVariable(dtc, false); node->lam = SavedVariable(lamc, false);
        node->A_head = SavedVariable(Ah, false); node->D = SavedVariable(Dc, false); node->B = SavedVariable(Bc, false);
        node->C = SavedVariable(Cc, false); node->cum = SavedVariable(cum, false); node->sdot = SavedVariable(sdot, false);
        node->ang_type = ang.scalar_type(); node->dt_type = dt.scalar_type(); node->A_type = A_head.scalar_type();
        node->raw_type = raw_angles.scalar_type(); node->lam_type = lam.scalar_type();
        if (D.defined()) node->D_type = D.scalar_type();
        node->fused = fused;
        torch::autograd::set_history(out.y, node);
    }
    return out.y;
}

// ---------------------------------------------------------------------------------------------------- rotation
struct RopeNode : SavingNode {
    SavedVariable x, ang;
    at::ScalarType ang_type;
    bool broadcast = false;
    std::string name() const override { return "FusedRoPEBackward"; }
    void release_saved() override {
        x.reset_data();
        ang.reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        if (!grads[0].defined()) return {Tensor(), Tensor()};
        at::NoGradGuard no_grad;
        const auto [xv, av] = unpacked([&] { return std::tuple(x.unpack(), ang.unpack()); });
        c10::cuda::CUDAGuard guard(xv.device());
        const Tensor dy = cast(grads[0].contiguous(), xv.scalar_type());
        const Tensor dx = at::empty_like(xv), dang = at::empty_like(av);
        check(ssd_b200_rope_bwd(dtype_code(xv), xv.size(0), xv.size(1), xv.size(2), xv.size(3), broadcast, ptr(xv), ptr<float>(av), ptr(dy), ptr(dx),
                                ptr<float>(dang), stream_of(xv)));
        return {dx, cast(dang, ang_type)};
    }
};

Tensor rope(const Tensor& x, const Tensor& angles) {
    refuse_tangents({&x, &angles});
    SSD_ASSERT(x.is_cuda() && angles.is_cuda(), "rotation runs on the GPU only: x and angles must be CUDA tensors");
    SSD_ASSERT(x.dim() == 4 && angles.dim() == 4, "x must be (B,T,H,D) and angles (B,T,1 or H,D/2); got ", x.dim(), " and ", angles.dim(),
               " dimensions");
    const int64_t B = x.size(0), T = x.size(1), H = x.size(2), D = x.size(3), aH = angles.size(2);
    SSD_ASSERT(D % 2 == 0, "pairs are rotated, so the last dimension of x must be even (it is ", D, ")");
    SSD_ASSERT(angles.size(0) == B && angles.size(1) == T && angles.size(3) == D / 2, "angles ", angles.sizes(), " do not fit x ", x.sizes(),
               ": want (", B, ", ", T, ", 1 or ", H, ", ", D / 2, ")");
    SSD_ASSERT(aH == 1 || aH == H, "angles carry ", aH, " heads; give 1 (shared by all heads) or ", H, " (one set per head)");
    check_like("angles", angles, x, B * T * aH * (D / 2));
    c10::cuda::CUDAGuard guard(x.device());
    Tensor xc, ang, out;
    {
        at::NoGradGuard no_grad;
        xc = x.contiguous();
        ang = f32(angles);
        out = at::empty_like(xc);
        check(ssd_b200_rope_fwd(dtype_code(xc), B, T, H, D, aH == 1, ptr(xc), ptr<float>(ang), ptr(out), stream_of(x)));
    }
    if (wants_grad({&x, &angles})) {
        auto node = link_node<RopeNode>(x, angles);
        node->x = SavedVariable(xc, false);
        node->ang = SavedVariable(ang, false);
        node->ang_type = angles.scalar_type();
        node->broadcast = aH == 1;
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ---------------------------------------------------------------------------------------------------- coefficients
struct TrapezoidNode : SavingNode {
    SavedVariable dt_raw, lam_raw, bias, alog;
    at::ScalarType bias_type, alog_type, lam_type;
    std::string name() const override { return "FusedTrapezoidalBackward"; }
    void release_saved() override {
        for (SavedVariable* v : {&dt_raw, &lam_raw, &bias, &alog}) v->reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        at::NoGradGuard no_grad;
        const auto [d, l, bv, av] = unpacked([&] { return std::tuple(dt_raw.unpack(), lam_raw.unpack(), bias.unpack(), alog.unpack()); });
        c10::cuda::CUDAGuard guard(d.device());
        const int64_t H = d.size(-1), rows = rows_of(d, H);
        Tensor g[4];
        for (int i = 0; i < 4; ++i) g[i] = grads[i].defined() ? cast(grads[i].contiguous(), d.scalar_type()) : at::zeros_like(d);
        const Tensor dd = at::empty_like(d), dl = at::empty_like(d), db = empty_f32({H}, d), da = empty_f32({H}, d);
        const Tensor ws = empty_f32({static_cast<int64_t>(ssd_b200_trapezoid_ws_floats(rows, H))}, d);
        check(ssd_b200_trapezoid_bwd(dtype_code(d), rows, H, ptr(d), ptr(l), ptr<float>(bv), ptr<float>(av), ptr(g[0]), ptr(g[1]), ptr(g[2]), ptr(g[3]),
                                     ptr(dd), ptr(dl), ptr<float>(db), ptr<float>(da), ptr<float>(ws), stream_of(d)));
        return {dd, cast(dl, lam_type), cast(db, bias_type), cast(da, alog_type)};
    }
};

std::tuple<Tensor, Tensor, Tensor, Tensor> trapezoid(const Tensor& dt_raw, const Tensor& lam_raw, const Tensor& dt_bias, const Tensor& A_log) {
    refuse_tangents({&dt_raw, &lam_raw, &dt_bias, &A_log});
    SSD_ASSERT(dt_raw.is_cuda() && lam_raw.is_cuda() && dt_bias.is_cuda() && A_log.is_cuda(),
               "the coefficient kernel runs on the GPU only: all four arguments must be CUDA tensors");
    SSD_ASSERT(dt_raw.sizes() == lam_raw.sizes(), "dt_raw and lam_raw must have one shape, got ", dt_raw.sizes(), " and ", lam_raw.sizes());
    SSD_ASSERT(dt_raw.dim() >= 1, "dt_raw needs a trailing head dimension");
    const int64_t H = dt_raw.size(-1);
    SSD_ASSERT(dt_bias.dim() == 1 && dt_bias.size(0) == H, "dt_bias must be (", H, ",), got ", dt_bias.sizes());
    SSD_ASSERT(A_log.dim() == 1 && A_log.size(0) == H, "A_log must be (", H, ",), got ", A_log.sizes());
    check_like("lam_raw", lam_raw, dt_raw, dt_raw.numel());
    check_like("dt_bias", dt_bias, dt_raw, H);
    check_like("A_log", A_log, dt_raw, H);
    c10::cuda::CUDAGuard guard(dt_raw.device());
    Tensor d, l, bias, alog, o[4];
    {
        at::NoGradGuard no_grad;
        const at::ScalarType type = dt_raw.scalar_type();
        d = dt_raw.contiguous();
        l = cast(lam_raw.contiguous(), type);
        // the reference rounds the parameters to the working dtype before use (src/kernels/trapezoidal.py:241-243)
        bias = f32(cast(dt_bias.contiguous(), type));
        alog = f32(cast(A_log.contiguous(), type));
        for (Tensor& t : o) t = at::empty_like(d);
        check(ssd_b200_trapezoid_fwd(dtype_code(d), rows_of(d, H), H, ptr(d), ptr(l), ptr<float>(bias), ptr<float>(alog), ptr(o[0]), ptr(o[1]), ptr(o[2]),
                                     ptr(o[3]), stream_of(d)));
    }
    if (wants_grad({&dt_raw, &lam_raw, &dt_bias, &A_log})) {
        auto node = link_node<TrapezoidNode>(dt_raw, lam_raw, dt_bias, A_log);
        node->dt_raw = SavedVariable(d, false); node->lam_raw = SavedVariable(l, false);
        node->bias = SavedVariable(bias, false); node->alog = SavedVariable(alog, false);
        node->bias_type = dt_bias.scalar_type(); node->alog_type = A_log.scalar_type(); node->lam_type = lam_raw.scalar_type();
        for (Tensor& t : o) torch::autograd::set_history(t, node);
    }
    return {o[0], o[1], o[2], o[3]};
}

}  // namespace

PYBIND11_MODULE(ssd_torch, m) {
    // (the exceptions of a backward surface through torch's own engine, which knows the c10 types)
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const AssertionFailed& e) {
            PyErr_SetString(PyExc_AssertionError, e.what());
        } catch (const c10::ValueError& e) {
            PyErr_SetString(PyExc_ValueError, e.what_without_backtrace());
        } catch (const c10::NotImplementedError& e) {
            PyErr_SetString(PyExc_NotImplementedError, e.what_without_backtrace());
        }
    });
    const auto nogil = py::call_guard<py::gil_scoped_release>();
    m.def("set_check_status", [](bool on) { g_check_status.store(on, std::memory_order_relaxed); });
    m.def("mamba2", &mamba2, nogil);
    m.def("operator_scan", &operator_scan, nogil);
    m.def("mamba2_gated", &mamba2_gated, nogil);
    m.def("mamba3", &mamba3, nogil);
    m.def("rmsnorm", &rmsnorm, nogil);
    m.def("rope", &rope, nogil);
    m.def("trapezoid", &trapezoid, nogil);
}
