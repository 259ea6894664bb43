// Inference forward of the ViG and HierViG models in C++: the same sequence of library calls, GEMMs and kernels as the Python
// modules, without their per-step cost.  A ViG forward is about 100 launches; in Python they took 3.2 ms, five times the
// kernels' time for one 224 x 224 image.
//
// A Plan is built by the Python layer (vig_b200/native.py) from a model's modules and stays valid while nothing it was built
// from changes: it watches every parameter (identity, version, address, type, strides), every module's children, hooks, plain
// attributes and overridden forwards, and answers None as soon as one differs, so that the caller rebuilds it or runs the
// modules themselves.  The check is some hundred pointer comparisons.
#include "host.h"
#include <cuda_runtime_api.h>
#include <limits>
#include <shared_mutex>
#include <unordered_map>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/CUDAGraph.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAException.h>
#include <ATen/ops/empty.h>

namespace vig_host {
namespace {

using OptT = std::optional<Tensor>;

// ---- library calls on tensors --------------------------------------------------------------------------------------
struct Ctx { void* stream; int32_t* status; int code; };
struct Chained {                                             // launches of this scope may overlap the end of the kernel before them, or may not
    const int was;
    explicit Chained(bool on) : was(api.vig_chain_launches(on)) {}
    ~Chained() { api.vig_chain_launches(was); }
};

Tensor dwconv(const Ctx& c, const Tensor& x, const Tensor& taps, const Tensor& bias, int64_t h, int64_t w, bool act) {
    Tensor y = at::empty_like(x);
    ok(api.vig_dwconv3x3_fwd(ptr(x), ptr(taps), ptr(bias), ptr(y), x.size(0), h, w, x.size(2), act, c.code, c.status, c.stream), "vig_dwconv3x3_fwd");
    return y;
}
std::pair<Tensor, Tensor> add_rmsnorm(const Ctx& c, const Tensor& x, const Tensor& w, const Tensor& res, double eps, bool prenorm) {
    const int64_t N = x.size(-1);
    Tensor y = at::empty_like(x), r = prenorm && res.defined() ? at::empty_like(x) : Tensor();
    ok(api.vig_add_rmsnorm_fwd(ptr(x), ptr(res), ptr(w), ptr(y), ptr(r), x.numel() / N, N, (float)eps, c.code, c.stream), "vig_add_rmsnorm_fwd");
    return {y, r};
}
Tensor layernorm(const Ctx& c, const Tensor& x, const Tensor& w, const Tensor& b, double eps, bool swish, const Tensor& pre_bias) {
    const int64_t N = x.size(-1);
    Tensor y = at::empty_like(x);
    ok(api.vig_layernorm_act_fwd(ptr(x), ptr(pre_bias), ptr(w), ptr(b), ptr(y), x.numel() / N, N, (float)eps, swish, c.code, c.stream), "vig_layernorm_act_fwd");
    return y;
}
Tensor token_mean(const Ctx& c, const Tensor& x) {
    Tensor y = at::empty({x.size(0), x.size(2)}, x.options());
    ok(api.vig_token_mean_fwd(ptr(x), ptr(y), x.size(0), x.size(1), x.size(2), c.code, c.stream), "vig_token_mean_fwd");
    return y;
}
// a matrix that TMA can read; the GEMM library takes others too
bool on16(const Tensor& w) { return (reinterpret_cast<uintptr_t>(ptr(w)) & 15) == 0; }
// swiglu(x W^T): one kernel where it is the faster one, GEMM + activation kernel otherwise
Tensor mlp_in(const Ctx& c, const Tensor& x, const Tensor& w) {
    const int64_t K = x.size(-1), I = w.size(0) / 2, M = x.numel() / K;
    Tensor out = at::empty({x.size(0), x.size(1), I}, x.options());
    if (on16(w) && api.vig_linear_swiglu_preferred(M, K, I, c.code)) {
        ok(api.vig_linear_swiglu_fwd(ptr(x), K, ptr(w), ptr(out), I, M, K, I, c.code, c.status, c.stream), "vig_linear_swiglu_fwd");
        return out;
    }
    const Tensor z = at::linear(x, w);
    ok(api.vig_swiglu_fwd(ptr(z), (uint8_t*)ptr(z) + I * z.element_size(), ptr(out), M, I, 2 * I, I, c.code, c.stream), "vig_swiglu_fwd");
    return out;
}
// r = x W^T + residual, h = RMSNorm(r): one kernel where it is the faster one
std::pair<Tensor, Tensor> linear_add_rmsnorm(const Ctx& c, const Tensor& x, const Tensor& w, const Tensor& res, const Tensor& nw, double eps) {
    const int64_t K = x.size(-1), N = w.size(0), M = x.numel() / K;
    if (!on16(w) || !api.vig_linear_add_rmsnorm_preferred(M, K, N, c.code)) return add_rmsnorm(c, at::linear(x, w), nw, res, eps, true);
    Tensor h = at::empty({x.size(0), x.size(1), N}, x.options()), r = at::empty({x.size(0), x.size(1), N}, x.options());
    ok(api.vig_linear_add_rmsnorm_fwd(ptr(x), K, ptr(w), ptr(res), ptr(nw), ptr(r), ptr(h), M, K, N, (float)eps, c.code, c.status, c.stream), "vig_linear_add_rmsnorm_fwd");
    return {h, r};
}

// ---- the attention module ------------------------------------------------------------------------------------------
struct Attn {
    // taps, w_z, b_z: derived weights, made by ``pack`` when the first forward gets here, so that the GPU works on the blocks
    // before meanwhile (all of them ahead of the first launch: 64 images of 1024 x 1024 waited 1.5 of 14 ms)
    mutable Tensor taps, w_z, b_z;
    mutable py::object pack;
    Tensor conv_b, gn_w, ln_w, o_w;
    int64_t H, dk, dv;
    bool act_conv, out_act;
    double eps, out_scale, norm, clamp;

    struct Scanned { Tensor o, xs, z; };                     // scan output [B,L,H,dv], conv output, stacked projection
    Scanned scan(const Ctx& c, const Tensor& x, int64_t h, int64_t w) const {
        // the first launch behind the kernels that make the weights reads them, and waits for their end like any other
        std::optional<Chained> apart;
        if (!w_z.defined()) { apart.emplace(false); std::tie(taps, w_z, b_z) = pack().cast<std::tuple<Tensor, Tensor, Tensor>>(); }
        const int64_t B = x.size(0), L = x.size(1), kd = H * dk, vd = H * dv;
        Tensor xs, z;
        if (api.vig_conv_proj_preferred(B * L, (int)x.size(2), (int)w_z.size(0), c.code) && on16(x) && on16(taps) && on16(w_z) && on16(b_z) && (!conv_b.defined() || on16(conv_b))) {
            xs = at::empty_like(x);
            z = at::empty({B, L, w_z.size(0)}, x.options());
            ok(api.vig_conv_proj_fwd(ptr(x), ptr(taps), ptr(conv_b), ptr(w_z), ptr(b_z), ptr(xs), ptr(z), B, h, w, x.size(2), w_z.size(0), act_conv, c.code, c.stream), "vig_conv_proj_fwd");
            apart.reset();
        } else {
            xs = dwconv(c, x, taps, conv_b, h, w, act_conv);
            apart.reset();
            const int64_t M = B * L, K = x.size(2), N = w_z.size(0);
            if (on16(w_z) && on16(b_z) && api.vig_linear_pair_preferred(M, K, N, c.code)) {
                z = at::empty({B, L, N}, x.options());
                ok(api.vig_linear_pair_fwd(ptr(xs), K, ptr(w_z), ptr(b_z), ptr(z), N, M, K, N, c.code, c.status, c.stream), "vig_linear_pair_fwd");
            } else {
                z = at::linear(xs, w_z, b_z);
            }
        }
        const int64_t W = z.size(2);
        auto view = [&](int64_t col, int64_t d) { return z.as_strided({B, H, L, d}, {L * W, d, W, 1}, z.storage_offset() + col); };
        Tensor o = at::empty({B, L, H, dv}, x.options());
        bi_gla_into(view(0, dk), view(kd, dk), view(2 * kd, dv), view(2 * kd + 2 * vd, dk), view(3 * kd + 2 * vd, dk),
                    o.as_strided({B, H, L, dv}, {L * vd, dv, vd, 1}), -1.0, out_scale, norm, clamp, {}, {}, {}, {}, 3, VIG_IMPL_AUTO);
        return {o, xs, z};
    }
    const void* gate_logits(const Tensor& z) const { return (const uint8_t*)ptr(z) + (2 * H * dk + H * dv) * z.element_size(); }

    // everything up to (not including) the output projection; h [B,L,C] contiguous
    Tensor forward(const Ctx& c, const Tensor& x, int64_t h, int64_t w) const {
        const auto [o, xs, z] = scan(c, x, h, w);
        const int64_t B = x.size(0), L = x.size(1), vd = H * dv, W = z.size(2);
        const int64_t so[3] = {L * vd, dv, vd};
        Tensor y = at::empty({B, L, vd}, x.options());
        ok(api.vig_gate_inject_fwd(ptr(o), so, ptr(xs), gate_logits(z), ptr(gn_w), ptr(ln_w), ptr(y), vd, W, vd, B, H, L, dv,
                                   (float)eps, out_act, c.code, c.stream), "vig_gate_inject_fwd");
        return y;
    }
};

// ---- what a plan was built from --------------------------------------------------------------------------------------
struct Watch {
    struct Item { py::object dict, key, value; };
    struct Param { Tensor t; int64_t version; void* data; at::ScalarType type; std::vector<int64_t> sizes, strides; };
    std::vector<Item> items;
    std::vector<std::pair<py::object, Py_ssize_t>> sizes;
    std::vector<std::pair<py::object, py::object>> absent;
    std::vector<Param> params;

    void item(py::object d, py::object k, py::object v) { items.push_back({d, k, v}); }
    void size(py::object d) { sizes.emplace_back(d, PyDict_Size(d.ptr())); }
    void missing(py::object d, py::object k) { absent.emplace_back(d, k); }
    void param(const Tensor& t, bool values) { params.push_back({t, values ? (int64_t)t._version() : -1, values ? t.data_ptr() : nullptr, t.scalar_type(), t.sizes().vec(), t.strides().vec()}); }
    // a module's plain attributes, parameters (values: what is in them too), children, hooks and the forward it overrides or not
    void module(py::handle m, bool values) {
        const py::dict d = m.attr("__dict__");
        const py::str fwd("forward");
        for (auto kv : d) {
            const std::string name = py::cast<std::string>(kv.first);
            PyObject* v = kv.second.ptr();
            if (name[0] != '_' && (v == Py_None || PyBool_Check(v) || PyLong_Check(v) || PyFloat_Check(v) || PyUnicode_Check(v) || PyTuple_Check(v)))
                item(d, py::reinterpret_borrow<py::object>(kv.first), py::reinterpret_borrow<py::object>(kv.second));
        }
        for (const char* table : {"_parameters", "_modules"}) {
            const py::dict t = d[table];
            for (auto kv : t) {
                item(t, py::reinterpret_borrow<py::object>(kv.first), py::reinterpret_borrow<py::object>(kv.second));
                if (table[1] == 'p' && !kv.second.is_none()) param(kv.second.cast<Tensor>(), values);
            }
            size(t);
        }
        for (const char* h : {"_forward_hooks", "_forward_pre_hooks"}) size(d[h]);
        if (PyObject* own = PyDict_GetItem(d.ptr(), fwd.ptr())) item(d, fwd, py::reinterpret_borrow<py::object>(own));
        else missing(d, fwd);
    }
    bool same() const {
        for (const auto& i : items) if (PyDict_GetItem(i.dict.ptr(), i.key.ptr()) != i.value.ptr()) return false;
        for (const auto& s : sizes) if (PyDict_Size(s.first.ptr()) != s.second) return false;
        for (const auto& a : absent) if (PyDict_GetItem(a.first.ptr(), a.second.ptr())) return false;
        for (const auto& p : params)
            if (p.t.scalar_type() != p.type || p.t.sizes() != p.sizes || p.t.strides() != p.strides || (p.version >= 0 && ((int64_t)p.t._version() != p.version || p.t.data_ptr() != p.data))) return false;
        return true;
    }
};

// The device's error word looked at without stalling the stream: the value copied by an earlier forward, if it has landed.
struct StatusPeek {
    int32_t* host = nullptr;
    cudaEvent_t event = nullptr;
    bool pending = false, drop = false;                  // drop: the value under way has been reported and cleared
    static StatusPeek& of(int device) { static StatusPeek s[64]; return s[device]; }
    int poll(bool capturing) {
        if (capturing || !pending || cudaEventQuery(event) != cudaSuccess) return 0;
        pending = false;
        if (drop) { drop = false; return 0; }
        return *host;
    }
    void snapshot(int device, cudaStream_t st, bool capturing) {
        if (capturing || pending) return;
        if (!host) {
            if (cudaHostAlloc(reinterpret_cast<void**>(&host), sizeof(int32_t), cudaHostAllocDefault) != cudaSuccess) { host = nullptr; return; }
            if (cudaEventCreateWithFlags(&event, cudaEventDisableTiming) != cudaSuccess) return;
        }
        if (!event || cudaMemcpyAsync(host, status_ptr(device), sizeof(int32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess) return;
        pending = cudaEventRecord(event, st) == cudaSuccess;
    }
};

struct Conv {
    Tensor w, b;                                         // bias may be undefined
    int64_t stride = 1, pad = 0;
    // NHWC in, NHWC out
    Tensor forward(const Tensor& x, bool with_bias) const {
        const Tensor y = at::conv2d(x.permute({0, 3, 1, 2}), w, with_bias && b.defined() ? OptT(b) : std::nullopt, {stride, stride}, {pad, pad});
        return y.permute({0, 2, 3, 1}).contiguous();
    }
};

struct PlanBase {
    Watch watch;
    at::ScalarType type = at::kBFloat16;
    at::Device device = at::Device(at::kCPU);
    Tensor head_w, head_b;
    py::object on_status;                                // called with the error word's value when an earlier forward left one

    bool takes(const Tensor& x) const {
        return x.is_cuda() && x.device() == device && x.scalar_type() == type && x.dim() == 4 && x.size(1) == 3 && x.numel() > 0 &&
               !(at::GradMode::is_enabled()) && !at::autocast::is_autocast_enabled(at::kCUDA) && !c10::impl::TorchDispatchModeTLS::any_modes_set() && status_known(device.index()) && watch.same();
    }
    Tensor finish(const Tensor& pooled) const { return at::linear(pooled, head_w, head_b.defined() ? OptT(head_b) : std::nullopt); }
    // One forward.  ``work``: a measure of the activations (tokens x channels).  Launched one by one, a forward of 50 to 150
    // kernels spends 5 - 10 us a launch on the host (through the GEMM library), which small forwards wait for, and 1.4 us
    // between kernels on the device, 7 % of one of three milliseconds (128 images of 224 x 224, width 384: 3465 -> 3220 us; 64
    // through the hierarchical model 3380 -> 3100; 64 of 1024 x 1024, width 192: 11.6 -> 11.45 ms).  So a shape that comes a
    // second time on a stream is captured into a CUDA graph, behind that call's own launches and while they run (2 - 4 ms of
    // host time), and replayed from the third call on.  The first kernel, which reads the images, stays outside and writes the
    // graph's input, so that nothing is copied.  The graph and its memory (about 45 bytes per activation element, GRAPH_WORK
    // elements in all per plan: 3 GB, and 32 MB of GEMM workspace) belong to this plan, one per shape and stream, the least recently used given back first,
    // and go with it.  Larger forwards gain little (8 of 2048 x 2048: 0.4 %) and would hold more.
    static constexpr int64_t GRAPH_WORK = 64 << 20;
    static constexpr size_t GRAPHS = 8, SHAPES = 64;
    struct Shape {
        int64_t B, H, W;
        cudaStream_t stream;
        bool operator==(const Shape& o) const { return B == o.B && H == o.H && W == o.W && stream == o.stream; }
    };
    // Calls of a shape since its graph was last given back, and how many of them are worth a capture: twice as many every time,
    // so that shapes which push each other out are not captured for ever.
    struct Seen { Shape shape; int64_t calls, worth; uint64_t used; };
    struct Captured {
        Shape shape;
        int64_t work;
        uint64_t used;
        std::unique_ptr<at::cuda::CUDAGraph> graph;
        std::unique_ptr<at::cuda::CUDAEvent> done;       // behind the last replay: the graph's memory is not given back before
        Tensor in, out, held;                            // held: what the graph reads and the plan may replace
        std::vector<c10::DataPtr> scratch;               // the GEMM library's workspaces that its kernels write
        // Also while the caller captures a graph of its own, where waiting for an event would spoil that capture but for the
        // relaxed mode: the event was recorded outside it
        ~Captured() {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (done) { try { done->synchronize(); } catch (...) {} }
            graph.reset();
            cudaThreadExchangeStreamCaptureMode(&mode);
        }
    };
    bool graphs = true;
    std::vector<Seen> seen;
    std::vector<std::unique_ptr<Captured>> captured;
    uint64_t clock = 0;
    int64_t captures = 0;

    template <typename V> static size_t oldest(const V& v) {
        auto used = [](const auto& e) { if constexpr (std::is_same_v<std::decay_t<decltype(e)>, Seen>) return e.used; else return e->used; };
        size_t at = 0;
        for (size_t i = 1; i < v.size(); ++i) if (used(v[i]) < used(v[at])) at = i;
        return at;
    }
    Captured* find(const Shape& s) {
        for (auto& e : captured) if (e->shape == s) { e->used = ++clock; return e.get(); }
        return nullptr;
    }
    Seen& record(const Shape& s) {
        for (Seen& e : seen) if (e.shape == s) { e.used = ++clock; return e; }
        if (seen.size() >= SHAPES) seen.erase(seen.begin() + oldest(seen));
        seen.push_back({s, 0, 2, ++clock});
        return seen.back();
    }
    void make_room(int64_t work) {
        for (;;) {
            int64_t held = work;
            for (const auto& e : captured) held += e->work;
            if (captured.empty() || (held <= GRAPH_WORK && captured.size() < GRAPHS)) return;
            const size_t i = oldest(captured);
            Seen& e = record(captured[i]->shape);
            e.calls = 0;
            e.worth *= 2;
            captured.erase(captured.begin() + i);
        }
    }
    // A stream of its own to capture on: no one else's work is ever on it
    at::cuda::CUDAStream capture_stream() const {
        static std::unordered_map<int, cudaStream_t>* streams = new std::unordered_map<int, cudaStream_t>();
        auto it = streams->find(device.index());
        if (it == streams->end()) {
            cudaStream_t st = nullptr;
            C10_CUDA_CHECK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
            it = streams->emplace(device.index(), st).first;
        }
        return at::cuda::getStreamFromExternal(it->second, device.index());
    }
    // The GEMM library's workspaces for ``st``, out of torch's tables.  They are made on the first GEMM on a stream, so those of
    // a capture come from the graph's own memory pool, and taken out here they are the graph's alone: graphs that run side by
    // side on two streams share no scratch, and nobody else gives it back.
    static void take_scratch(cudaStream_t st, std::vector<c10::DataPtr>& into) {
        for (auto* table : {&at::cuda::cublas_handle_stream_to_workspace(), &at::cuda::cublaslt_handle_stream_to_workspace()}) {
            std::unique_lock<std::shared_mutex> lock(table->mutex);
            for (auto it = table->map.begin(); it != table->map.end();) {
                if (std::get<1>(it->first) != static_cast<void*>(st)) { ++it; continue; }
                into.push_back(std::move(it->second));
                it = table->map.erase(it);
            }
        }
    }
    // in: what the first kernel of this call wrote; the graph keeps it as its input
    template <typename F> void capture(const Shape& s, int64_t work, const Tensor& in, Tensor held, F rest, const Ctx& c) {
        make_room(work);
        const at::cuda::CUDAStream on = capture_stream();
        std::vector<c10::DataPtr> stale;
        take_scratch(on.stream(), stale);                    // of a capture that failed half way
        c10::cuda::CUDAStreamGuard guard(on);
        auto e = std::make_unique<Captured>();
        e->shape = s; e->work = work; e->used = ++clock; e->in = in; e->held = std::move(held);
        auto g = std::make_unique<at::cuda::CUDAGraph>();
        bool failed = false;
        g->capture_begin({0, 0}, cudaStreamCaptureModeThreadLocal);
        try { e->out = rest(Ctx{on.stream(), c.status, c.code}, in); } catch (...) { failed = true; }
        try { g->capture_end(); } catch (...) { failed = true; }
        take_scratch(on.stream(), e->scratch);
        if (failed) { record(s).worth = std::numeric_limits<int64_t>::max() / 2; return; }
        e->graph = std::move(g);
        e->done = std::make_unique<at::cuda::CUDAEvent>();
        captured.push_back(std::move(e));
        ++captures;
    }

    // ``first(c, images, y)``: the first kernel, into y (allocated if undefined); ``rest(c, y)``: everything behind it; ``held()``:
    // a tensor made for this shape before both, which the plan keeps for the last shape only
    template <typename F, typename R, typename G> OptT run(const Tensor& x, int64_t work, F first, R rest, G held) {
        if (!takes(x)) return std::nullopt;
        c10::cuda::CUDAGuard guard(device);
        at::NoGradGuard ng;
        auto st = at::cuda::getCurrentCUDAStream();
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(st.stream(), &cap);
        const bool capturing = cap != cudaStreamCaptureStatusNone;
        StatusPeek& peek = StatusPeek::of(device.index());
        if (const int v = peek.poll(capturing)) { on_status(v); }
        const Tensor kept = held();
        const Ctx c{st.stream(), status_ptr(device.index()), type == at::kBFloat16 ? VIG_DTYPE_BF16 : VIG_DTYPE_F16};
        const Chained chained(true);
        const bool replays = graphs && !capturing && work <= GRAPH_WORK;
        const Shape shape{x.size(0), x.size(2), x.size(3), st.stream()};
        Captured* e = replays ? find(shape) : nullptr;
        Tensor y;
        if (e) {
            first(c, x.contiguous(), e->in);
            e->graph->replay();
            y = e->out.clone();
            e->done->record(st);
        } else {
            Tensor t;
            first(c, x.contiguous(), t);
            y = rest(c, t);
            if (replays) {
                Seen& r = record(shape);
                if (++r.calls >= r.worth) capture(shape, work, t, kept, rest, c);
            }
        }
        peek.snapshot(device.index(), st.stream(), capturing);
        return y;
    }
};

// ---- ViG -----------------------------------------------------------------------------------------------------------
struct VigBlock {
    Tensor n1, n2, gate_w, down_w;
    double e1, e2;
    Attn attn;
};

struct VigPlan : PlanBase {
    // stem: first convolution as one kernel with its LayerNorm (w_gemm) where the library has it, or as a 2x2 convolution over
    // unfolded cells (w_cells) followed by the LayerNorm kernel; second convolution and LayerNorm
    Tensor w_gemm, b1, ln1_w, ln1_b, ln2_w, ln2_b;
    Conv cells, conv2;
    double ln1_e, ln2_e;
    int64_t C = 0;
    bool fused_norms = false;
    std::vector<VigBlock> blocks;
    Tensor norm_w;
    double norm_e;
    py::object pos_fn;                                   // (h, w) -> [1, h*w, C], the module's own cache
    mutable Tensor pos;
    mutable int64_t pos_h = 0, pos_w = 0;

    OptT forward(const Tensor& x) {
        const int64_t H = x.dim() == 4 ? x.size(2) : 0, W = x.dim() == 4 ? x.size(3) : 0;
        if (H % 8 || W % 8 || H == 0) return std::nullopt;
        return run(x, x.size(0) * ((H + 15) / 16) * ((W + 15) / 16) * C, [&](const Ctx& c, const Tensor& img, Tensor& f) { first(c, img, f); },
                   [&, B = x.size(0)](const Ctx& c, const Tensor& f) { return rest(c, f, B, H, W); }, [&] { return position((H / 8 + 1) / 2, (W / 8 + 1) / 2); });
    }
    Tensor position(int64_t h, int64_t w) const {
        if (!pos.defined() || pos_h != h || pos_w != w) {
            pos = pos_fn(py::make_tuple(h, w)).cast<Tensor>().to(type).contiguous();
            pos_h = h; pos_w = w;
        }
        return pos;
    }
    bool folds(const Ctx& c, int64_t B, int64_t H, int64_t W) const { return w_gemm.defined() && api.vig_stem_conv_ln_supported(B, H / 8, W / 8, 192, C / 2, c.code); }
    void first(const Ctx& c, const Tensor& img, Tensor& f) const {       // 8 x 8 pixel cells, with a border of cells for the 2 x 2 convolution
        const int64_t B = img.size(0), H = img.size(2), W = img.size(3), edge = folds(c, B, H, W) ? 0 : 1;
        if (!f.defined()) f = at::empty({B, H / 8 + edge, W / 8 + edge, 192}, img.options());
        if (edge) ok(api.vig_stem_unfold_fwd(ptr(img), ptr(f), B, 3, H, W, 8, c.code, c.stream), "vig_stem_unfold_fwd");
        else ok(api.vig_stem_fold_fwd(ptr(img), ptr(f), B, 3, H, W, c.code, c.stream), "vig_stem_fold_fwd");
    }
    Tensor rest(const Ctx& c, const Tensor& f, int64_t B, int64_t H, int64_t W) const {
        Tensor y;
        if (folds(c, B, H, W)) {
            y = at::empty({B, H / 8, W / 8, C / 2}, f.options());
            ok(api.vig_stem_conv_ln_fwd(ptr(f), ptr(w_gemm), ptr(b1), ptr(ln1_w), ptr(ln1_b), ptr(y), B, H / 8, W / 8, 192, C / 2, (float)ln1_e, 1, c.code, c.status,
                                        c.stream), "vig_stem_conv_ln_fwd");
        } else {
            y = layernorm(c, cells.forward(f, false), ln1_w, ln1_b, ln1_e, true, b1);
        }
        y = conv2.forward(y, false);
        const int64_t h = y.size(1), w = y.size(2), L = h * w, rows = B * L;
        const Tensor pos = position(h, w);
        Tensor tok = at::empty({B, L, C}, f.options());
        if (fused_norms) {
            Tensor n = at::empty({B, L, C}, f.options());
            ok(api.vig_layernorm_act_add_rmsnorm_fwd(ptr(y), ptr(conv2.b), ptr(ln2_w), ptr(ln2_b), ptr(pos), L, ptr(tok), ptr(blocks[0].n1), (float)blocks[0].e1,
                                                     ptr(n), rows, C, (float)ln2_e, 0, c.code, c.stream), "vig_layernorm_act_add_rmsnorm_fwd");
            for (size_t i = 0; i < blocks.size(); ++i) {
                const VigBlock& b = blocks[i];
                const bool last = i + 1 == blocks.size();
                const int64_t I = b.down_w.size(1);
                const Tensor& next_w = last ? norm_w : blocks[i + 1].n1;
                const double next_e = last ? norm_e : blocks[i + 1].e1;
                if (on16(b.attn.o_w) && on16(b.gate_w) && on16(b.down_w) && api.vig_block_tail_preferred(rows, b.attn.H, b.attn.dv, I, c.code)) {
                    const auto [o, xs, z] = b.attn.scan(c, n, h, w);
                    Tensor r = at::empty_like(tok), hn = at::empty_like(tok);
                    ok(api.vig_block_tail_fwd(ptr(o), ptr(xs), b.attn.gate_logits(z), z.size(2), ptr(b.attn.gn_w), ptr(b.attn.ln_w), (float)b.attn.eps, b.attn.out_act,
                                              ptr(b.attn.o_w), ptr(tok), ptr(b.n2), (float)b.e2, ptr(b.gate_w), ptr(b.down_w), ptr(next_w), (float)next_e, ptr(r),
                                              ptr(hn), rows, b.attn.H, b.attn.dv, I, c.code, c.status, c.stream), "vig_block_tail_fwd");
                    tok = r; n = hn;
                    continue;
                }
                std::tie(n, tok) = linear_add_rmsnorm(c, b.attn.forward(c, n, h, w), b.attn.o_w, tok, b.n2, b.e2);
                std::tie(n, tok) = linear_add_rmsnorm(c, mlp_in(c, n, b.gate_w), b.down_w, tok, next_w, next_e);
            }
            return finish(token_mean(c, n));
        }
        ok(api.vig_layernorm_act_add_fwd(ptr(y), ptr(conv2.b), ptr(ln2_w), ptr(ln2_b), ptr(pos), L, ptr(tok), rows, C, (float)ln2_e, 0, c.code, c.stream),
           "vig_layernorm_act_add_fwd");
        Tensor branch;                                   // the residual add of a branch rides in the next norm
        for (const VigBlock& b : blocks) {
            Tensor n, r;
            std::tie(n, r) = branch.defined() ? add_rmsnorm(c, branch, b.n1, tok, b.e1, true) : add_rmsnorm(c, tok, b.n1, {}, b.e1, false);
            if (r.defined()) tok = r;
            std::tie(n, tok) = add_rmsnorm(c, at::linear(b.attn.forward(c, n, h, w), b.attn.o_w), b.n2, tok, b.e2, true);
            branch = at::linear(mlp_in(c, n, b.gate_w), b.down_w);
        }
        return finish(token_mean(c, add_rmsnorm(c, branch, norm_w, tok, norm_e, false).first));
    }
};

// ---- HierViG -------------------------------------------------------------------------------------------------------
struct Norm { Tensor w, b; double eps = 0; };
// r = x + residual (optional), LayerNorm(r) with an activation: {LayerNorm, r}
std::pair<Tensor, Tensor> add_layernorm(const Ctx& c, const Tensor& x, const Tensor& res, const Norm& n, int act, const Tensor& pre_bias = {}) {
    const int64_t N = x.size(-1);
    Tensor y = at::empty_like(x), r = res.defined() ? at::empty_like(x) : Tensor();
    ok(api.vig_add_layernorm_fwd(ptr(x), ptr(pre_bias), ptr(res), ptr(n.w), ptr(n.b), ptr(y), ptr(r), x.numel() / N, N, (float)n.eps, act, c.code, c.stream), "vig_add_layernorm_fwd");
    return {y, r};
}

struct HierBlock {
    Norm n1, n2;
    Attn attn;
    bool gated = false;
    Tensor fc1_w, fc1_b, fc2_w, fc2_b;
};
struct HierStage {
    std::vector<HierBlock> blocks;
    bool down = false;
    Conv conv;
    Norm norm;
};

struct HierPlan : PlanBase {
    std::vector<std::tuple<Conv, bool, Norm, int>> embed;   // convolution, whether a LayerNorm follows, the norm, activation (0 / 2 = GELU)
    std::vector<HierStage> stages;
    Tensor first_w;                                          // [O,3,3,3] where the embedding's first convolution has a kernel of its own
    Norm last;

    OptT forward(const Tensor& x) {
        return run(x, x.dim() == 4 ? x.size(0) * ((x.size(2) + 3) / 4) * ((x.size(3) + 3) / 4) * std::get<0>(embed.back()).w.size(0) : 0, [&](const Ctx& c, const Tensor& img, Tensor& y) { first(c, img, y); },
                   [&](const Ctx& c, const Tensor& y) { return rest(c, y); }, [] { return Tensor(); });
    }
    void first(const Ctx& c, const Tensor& img, Tensor& y) const {
        const int64_t B = img.size(0), H = img.size(2), W = img.size(3);
        if (first_w.defined()) {                             // the first convolution with its norm and activation, from the image as it is
            const auto& [conv, has_norm, norm, act] = embed[0];
            const int64_t O = first_w.size(0);
            if (!y.defined()) y = at::empty({B, (H + 1) / 2, (W + 1) / 2, O}, img.options());
            const Tensor w = first_w.contiguous();
            ok(api.vig_embed_conv_ln_fwd(ptr(img), ptr(w), ptr(conv.b), ptr(norm.w), ptr(norm.b), ptr(y), B, H, W, O, (float)norm.eps, act == 2, c.code, c.stream),
               "vig_embed_conv_ln_fwd");
        } else {                                             // channels-last
            if (!y.defined()) y = at::empty({B, H, W, img.size(1)}, img.options());
            y.copy_(img.permute({0, 2, 3, 1}));
        }
    }
    Tensor rest(const Ctx& c, const Tensor& first_out) const {
        Tensor y = first_out;
        for (size_t i = first_w.defined() ? 1 : 0; i < embed.size(); ++i) {
            const auto& [conv, has_norm, norm, act] = embed[i];
            y = conv.forward(y, !has_norm);                      // the bias rides in the norm
            if (has_norm) y = add_layernorm(c, y, {}, norm, act, conv.b).first;
            else if (act == 2) y = at::gelu(y);
        }
        int64_t h = y.size(1), w = y.size(2);
        Tensor x = y.view({y.size(0), h * w, y.size(3)}), branch;
        for (const HierStage& st : stages) {
            for (const HierBlock& b : st.blocks) {
                Tensor n, r;
                std::tie(n, r) = add_layernorm(c, branch.defined() ? branch : x, branch.defined() ? x : Tensor(), b.n1, 0);   // the branch's add rides in the norm
                if (r.defined()) x = r;
                std::tie(n, x) = add_layernorm(c, at::linear(b.attn.forward(c, n, h, w), b.attn.o_w), x, b.n2, 0);
                branch = b.gated ? at::linear(mlp_in(c, n, b.fc1_w), b.fc2_w)
                                 : at::linear(at::gelu(at::linear(n, b.fc1_w, b.fc1_b)), b.fc2_w, b.fc2_b);
            }
            if (st.down) {
                if (branch.defined()) { x = x + branch; branch = Tensor(); }
                y = st.conv.forward(x.view({x.size(0), h, w, x.size(2)}), false);
                h = y.size(1); w = y.size(2);
                x = add_layernorm(c, y.view({y.size(0), h * w, y.size(3)}), {}, st.norm, 0, st.conv.b).first;
            }
        }
        const Tensor n = branch.defined() ? add_layernorm(c, branch, x, last, 0).first : add_layernorm(c, x, {}, last, 0).first;
        return finish(token_mean(c, n));
    }
};

// ---- plans from Python dictionaries ----------------------------------------------------------------------------------
Tensor tensor_of(const py::dict& d, const char* key) { return d.contains(key) && !d[key].is_none() ? d[key].cast<Tensor>() : Tensor(); }
Attn attn_of(const py::dict& d) {
    Attn a;
    a.pack = d["pack"]; a.conv_b = tensor_of(d, "conv_b");
    a.gn_w = tensor_of(d, "gn_w"); a.ln_w = tensor_of(d, "ln_w"); a.o_w = tensor_of(d, "o_w");
    a.H = d["H"].cast<int64_t>(); a.dk = d["dk"].cast<int64_t>(); a.dv = d["dv"].cast<int64_t>();
    a.act_conv = d["act_conv"].cast<bool>(); a.out_act = d["out_act"].cast<bool>();
    a.eps = d["eps"].cast<double>(); a.out_scale = d["out_scale"].cast<double>(); a.norm = d["norm"].cast<double>(); a.clamp = d["clamp"].cast<double>();
    return a;
}
Norm norm_of(const py::dict& d) { return {tensor_of(d, "w"), tensor_of(d, "b"), d["eps"].cast<double>()}; }
Conv conv_of(const py::dict& d) { return {tensor_of(d, "w"), tensor_of(d, "b"), d["stride"].cast<int64_t>(), d["pad"].cast<int64_t>()}; }
void base_of(PlanBase& p, const py::dict& d) {
    p.head_w = tensor_of(d, "head_w"); p.head_b = tensor_of(d, "head_b");
    p.type = p.head_w.scalar_type(); p.device = p.head_w.device();
    p.on_status = d["on_status"];
    p.graphs = d["graphs"].cast<bool>();
}

VigPlan* make_vig(const py::dict& d) {
    auto p = std::make_unique<VigPlan>();
    base_of(*p, d);
    p->w_gemm = tensor_of(d, "w_gemm"); p->b1 = tensor_of(d, "b1");
    const Norm n1 = norm_of(d["ln1"]), n2 = norm_of(d["ln2"]);
    p->ln1_w = n1.w; p->ln1_b = n1.b; p->ln1_e = n1.eps; p->ln2_w = n2.w; p->ln2_b = n2.b; p->ln2_e = n2.eps;
    p->cells = conv_of(d["cells"]); p->conv2 = conv_of(d["conv2"]);
    p->C = p->conv2.w.size(0);
    p->fused_norms = d["fused_norms"].cast<bool>();
    p->norm_w = tensor_of(d, "norm_w"); p->norm_e = d["norm_e"].cast<double>();
    p->pos_fn = d["pos_fn"];
    for (auto item : d["blocks"].cast<py::list>()) {
        const py::dict b = item.cast<py::dict>();
        p->blocks.push_back({tensor_of(b, "n1"), tensor_of(b, "n2"), tensor_of(b, "gate_w"), tensor_of(b, "down_w"), b["e1"].cast<double>(), b["e2"].cast<double>(),
                             attn_of(b["attn"])});
    }
    return p.release();
}

HierPlan* make_hier(const py::dict& d) {
    auto p = std::make_unique<HierPlan>();
    base_of(*p, d);
    for (auto item : d["embed"].cast<py::list>()) {
        const py::dict e = item.cast<py::dict>();
        const bool has = !e["norm"].is_none();
        p->embed.emplace_back(conv_of(e["conv"]), has, has ? norm_of(e["norm"]) : Norm(), e["act"].cast<int>());
    }
    p->first_w = tensor_of(d, "first_w");
    for (auto item : d["stages"].cast<py::list>()) {
        const py::dict s = item.cast<py::dict>();
        HierStage st;
        for (auto bi : s["blocks"].cast<py::list>()) {
            const py::dict b = bi.cast<py::dict>();
            st.blocks.push_back({norm_of(b["n1"]), norm_of(b["n2"]), attn_of(b["attn"]), b["gated"].cast<bool>(), tensor_of(b, "fc1_w"), tensor_of(b, "fc1_b"),
                                 tensor_of(b, "fc2_w"), tensor_of(b, "fc2_b")});
        }
        if (!s["conv"].is_none()) { st.down = true; st.conv = conv_of(s["conv"]); st.norm = norm_of(s["norm"]); }
        p->stages.push_back(std::move(st));
    }
    p->last = norm_of(d["last"]);
    return p.release();
}

}  // namespace

void bind_model(py::module_& m) {
    m.def("drop_status", [](int device) {                // the error word was read and cleared otherwise
        if (device < 0 || device >= 64) return;
        StatusPeek& peek = StatusPeek::of(device);
        peek.drop = peek.pending;
    });
    auto watch = [](auto& cls) {
        using P = typename std::decay_t<decltype(cls)>::type;
        cls.def("watch_item", [](P& p, py::object d, py::object k, py::object v) { p.watch.item(d, k, v); })
            .def("watch_size", [](P& p, py::object d) { p.watch.size(d); })
            .def("watch_modules", [](P& p, const py::list& ms) { for (auto m : ms) p.watch.module(m, true); })
            .def("graphs", [](const P& p) { return p.captured.size(); })
            .def("captures", [](const P& p) { return p.captures; })
            .def("valid", [](const P& p) { return p.watch.same(); })
            .def("forward", &P::forward);
    };
    // what a model without a plan was refused for
    py::class_<Watch>(m, "Refusal")
        .def(py::init<>())
        .def("watch_item", [](Watch& w, py::object d, py::object k, py::object v) { w.item(d, k, v); })
        .def("watch_size", [](Watch& w, py::object d) { w.size(d); })
        .def("watch_modules", [](Watch& w, const py::list& ms) { for (auto m : ms) w.module(m, false); })
        .def("valid", &Watch::same)
        .def("forward", [](const Watch&, py::object) { return py::none(); });
    py::class_<VigPlan> vig(m, "VigPlan");
    vig.def(py::init(&make_vig));
    watch(vig);
    py::class_<HierPlan> hier(m, "HierPlan");
    hier.def(py::init(&make_hier));
    watch(hier);
}

}  // namespace vig_host
