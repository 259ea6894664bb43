// Operator entry points of the Python layer in C++: argument checks, output and workspace allocation, the library call and the
// autograd node.  In Python these took 40 us a call (170 us forward + backward), more than the kernels of small calls.
// Anything out of the ordinary -- an argument the checks reject, an option only the Python layer implements -- answers None,
// and the caller takes the Python path, which raises or handles it.
#include "host.h"
#include <dlfcn.h>
#include <torch/csrc/autograd/custom_function.h>

namespace vig_host {

Api api;
static Tensor* const g_status = new Tensor[64];         // never destroyed: outlives the interpreter and the CUDA context's teardown

int32_t* status_ptr(int device) { return device >= 0 && device < 64 && g_status[device].defined() ? g_status[device].data_ptr<int32_t>() : nullptr; }
bool status_known(int device) { return status_ptr(device) != nullptr; }

static void init(const std::string& path) {
    void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (!h) throw std::runtime_error(std::string("cannot open the kernel library: ") + dlerror());
#define X(name)                                                                                          \
    api.name = reinterpret_cast<decltype(api.name)>(dlsym(h, #name));                                     \
    if (!api.name) throw std::runtime_error(std::string("the kernel library lacks ") + #name);
    VIG_HOST_API(X)
#undef X
}

static void set_status(int device, const Tensor& t) {
    if (device < 0 || device >= 64) throw std::runtime_error("device index");
    g_status[device] = t;
}

void bi_gla_into(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gf, const Tensor& gb, const Tensor& o, double scale, double out_scale,
                 double norm, double clamp, const Tensor& init_f, const Tensor& init_b, const Tensor& final_f, const Tensor& final_b, int dir_mask, int impl) {
    const int B = k.size(0), H = k.size(1), L = k.size(2), dk = k.size(3), dv = v.size(3), code = dtype_code(k);
    const size_t n = api.vig_bigla_workspace_bytes(B, H, L, dk, dv, code, impl);
    Tensor ws;
    if (n) ws = at::empty({(int64_t)n}, k.options().dtype(at::kByte));
    const S3 sq(q), sk(k), sv(v), sf(gf), sb(gb), so(o);
    ok(api.vig_bigla_fwd(ptr(q), ptr(k), ptr(v), ptr(gf), ptr(gb), ptr(o), B, H, L, dk, dv, code, q.defined() ? sq.s : nullptr, sk.s, sv.s,
                         gf.defined() ? sf.s : nullptr, gb.defined() ? sb.s : nullptr, o.defined() ? so.s : nullptr, (float)scale, (float)out_scale,
                         (float)norm, (float)clamp, (const float*)ptr(init_f), (const float*)ptr(init_b), (float*)ptr(final_f), (float*)ptr(final_b),
                         nullptr, nullptr, dir_mask, impl, ptr(ws), n, status_ptr(k.get_device()), stream()), "vig_bigla_fwd");
}

// one dtype, one device, matching shapes, contiguous last dimension
static bool scan_args_ok(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gf, const Tensor& gb, int dir_mask) {
    if (!k.defined() || !v.defined() || !q.defined() || k.dim() != 4 || v.dim() != 4 || dir_mask < 1 || dir_mask > 3) return false;
    if (dtype_code(k) < 0 || !k.is_cuda() || !status_known(k.get_device())) return false;
    for (int i = 0; i < 3; ++i) if (v.size(i) != k.size(i)) return false;
    auto same = [&](const Tensor& t, const Tensor& like) {
        return t.scalar_type() == k.scalar_type() && t.device() == k.device() && t.dim() == 4 && t.sizes() == like.sizes() && (t.stride(3) == 1 || t.size(3) == 1);
    };
    if (!same(q, k) || !same(k, k) || !same(v, v)) return false;
    if (((dir_mask & 1) != 0) != gf.defined() || ((dir_mask & 2) != 0) != gb.defined()) return false;
    return (!gf.defined() || same(gf, k)) && (!gb.defined() || same(gb, k));
}

static bool bwd_dims(int64_t dk, int64_t dv) {
    return (dk == 16 && dv == 32) || (dk == 32 && dv == 32) || (dk == 32 && dv == 64) || (dk == 64 && dv == 64) || (dk == 64 && dv == 128);
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct BiGla : torch::autograd::Function<BiGla> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& gf,
                          const std::optional<Tensor>& gb, double scale, double out_scale, double norm, double clamp, int64_t dir_mask, int64_t impl) {
        at::AutoDispatchBelowADInplaceOrView guard;
        const Tensor f = gf ? *gf : Tensor(), b = gb ? *gb : Tensor();
        c10::cuda::CUDAGuard dev(k.device());
        Tensor o = at::empty({k.size(0), k.size(1), k.size(2), v.size(3)}, v.options());
        bi_gla_into(q, k, v, f, b, o, scale, out_scale, norm, clamp, {}, {}, {}, {}, (int)dir_mask, (int)impl);
        ctx->save_for_backward({q, k, v, f, b});
        ctx->saved_data["scale"] = scale; ctx->saved_data["out_scale"] = out_scale; ctx->saved_data["norm"] = norm; ctx->saved_data["clamp"] = clamp;
        ctx->saved_data["mask"] = dir_mask;
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grad_out) {
        const auto saved = ctx->get_saved_variables();
        // a saved-tensor hook may hand a tensor back in another layout
        auto rows = [](const Tensor& t) { return t.defined() && t.stride(3) != 1 && t.size(3) != 1 ? t.contiguous() : t; };
        const Tensor q = rows(saved[0]), k = rows(saved[1]), v = rows(saved[2]), gf = rows(saved[3]), gb = rows(saved[4]);
        Tensor d = grad_out[0];
        variable_list none(11);
        if (!d.defined()) return none;
        c10::cuda::CUDAGuard dev(k.device());
        d = rows(d);
        const int B = k.size(0), H = k.size(1), L = k.size(2), dk = k.size(3), dv = v.size(3), mask = (int)ctx->saved_data["mask"].toInt();
        const Tensor dq = at::empty({B, H, L, dk}, k.options()), dkk = at::empty({B, H, L, dk}, k.options()), dvv = at::empty({B, H, L, dv}, k.options());
        Tensor df, db;
        if (mask & 1) df = at::empty({B, H, L, dk}, k.options());
        if (mask & 2) db = at::empty({B, H, L, dk}, k.options());
        const size_t n = api.vig_bigla_bwd_full_workspace_bytes(B, H, L, dk, dv);
        const Tensor ws = at::empty({(int64_t)n}, k.options().dtype(at::kByte));
        const S3 sq(q), sk(k), sv(v), sf(gf), sb(gb), sd(d);
        ok(api.vig_bigla_bwd_full(ptr(q), ptr(k), ptr(v), ptr(gf), ptr(gb), ptr(d), ptr(dq), ptr(dkk), ptr(dvv), ptr(df), ptr(db), 0, B, H, L, dk, dv,
                                  dtype_code(k), sq.s, sk.s, sv.s, gf.defined() ? sf.s : nullptr, gb.defined() ? sb.s : nullptr, sd.s,
                                  (float)ctx->saved_data["scale"].toDouble(), (float)ctx->saved_data["out_scale"].toDouble(),
                                  (float)ctx->saved_data["norm"].toDouble(), (float)ctx->saved_data["clamp"].toDouble(), mask, ptr(ws), n, stream()),
           "vig_bigla_bwd_full");
        none[0] = dq; none[1] = dkk; none[2] = dvv; none[3] = df; none[4] = db;
        return none;
    }
};

using OptT = std::optional<Tensor>;
static Tensor get(const OptT& t) { return t ? *t : Tensor(); }
static bool wants_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts) if (t->defined() && t->requires_grad()) return true;
    return false;
}

// the plain call: both or one direction, no states; differentiable
static OptT bi_gla(const OptT& q_, const OptT& k_, const OptT& v_, const OptT& gf_, const OptT& gb_, double scale, double out_scale, double norm,
                   double clamp, int64_t dir_mask, int64_t impl) {
    const Tensor q = get(q_), k = get(k_), v = get(v_), gf = get(gf_), gb = get(gb_);
    if (!scan_args_ok(q, k, v, gf, gb, (int)dir_mask)) return std::nullopt;
    if (wants_grad({&q, &k, &v, &gf, &gb})) {
        if (!bwd_dims(k.size(3), v.size(3))) return std::nullopt;
        return BiGla::apply(q, k, v, gf.defined() ? OptT(gf) : std::nullopt, gb.defined() ? OptT(gb) : std::nullopt, scale, out_scale, norm, clamp, dir_mask, impl);
    }
    c10::cuda::CUDAGuard dev(k.device());
    Tensor o = at::empty({k.size(0), k.size(1), k.size(2), v.size(3)}, v.options());
    bi_gla_into(q, k, v, gf, gb, o, scale, out_scale, norm, clamp, {}, {}, {}, {}, (int)dir_mask, (int)impl);
    return o;
}

// gates of both directions stacked along the batch: [2B,H,L,dk]
static OptT bi_gla_stacked(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, double scale, double out_scale) {
    const int64_t B = q.dim() == 4 ? q.size(0) : 0;
    if (g.dim() != 4 || B == 0 || g.size(0) != 2 * B) return std::nullopt;
    return bi_gla(q, k, v, g.narrow(0, 0, B), g.narrow(0, B, B), scale, out_scale, 0.0, std::nan(""), 3, VIG_IMPL_AUTO);
}

// one direction, continued from a state and / or returning the final one (not differentiable)
static std::optional<std::pair<Tensor, OptT>> scan(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, double scale, const OptT& init, bool want_final,
                                                   bool reverse) {
    const Tensor none, &gf = reverse ? none : g, &gb = reverse ? g : none;
    if (!scan_args_ok(q, k, v, gf, gb, reverse ? 2 : 1)) return std::nullopt;
    const bool states = init || want_final;
    const Tensor h0 = get(init);
    if (wants_grad({&q, &k, &v, &g})) {
        if (states || !bwd_dims(k.size(3), v.size(3))) return std::nullopt;
        return std::make_pair(BiGla::apply(q, k, v, gf.defined() ? OptT(gf) : std::nullopt, gb.defined() ? OptT(gb) : std::nullopt, scale, 1.0, 0.0, std::nan(""),
                                           (int64_t)(reverse ? 2 : 1), (int64_t)VIG_IMPL_AUTO), OptT());
    }
    const std::vector<int64_t> hs{k.size(0), k.size(1), k.size(3), v.size(3)};
    if (h0.defined() && (h0.scalar_type() != at::kFloat || !h0.is_contiguous() || h0.device() != k.device() || h0.sizes() != hs)) return std::nullopt;
    c10::cuda::CUDAGuard dev(k.device());
    Tensor o = at::empty({k.size(0), k.size(1), k.size(2), v.size(3)}, v.options()), fin;
    if (want_final) fin = at::empty(hs, k.options().dtype(at::kFloat));
    bi_gla_into(q, k, v, gf, gb, o, scale, 1.0, 0.0, std::nan(""), reverse ? none : h0, reverse ? h0 : none, reverse ? none : fin, reverse ? fin : none,
                reverse ? 2 : 1, VIG_IMPL_AUTO);
    return std::make_pair(o, fin.defined() ? OptT(fin) : OptT());
}

}  // namespace vig_host

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    using namespace vig_host;
    m.def("init", &init);
    m.def("set_status", &set_status);
    m.def("bi_gla", &bi_gla);
    m.def("bi_gla_stacked", &bi_gla_stacked);
    m.def("scan", &scan);
    bind_model(m);
}
