// The host half of the operators whose kernels are shorter than the Python around them: argument checks, output allocation, the
// library call and the autograd nodes, in C++. A call of a few microseconds on the GPU spent 15 us in Python, a training pass of
// the scan (B16 T512 D704: 104 us of kernels) 160, most of it in the autograd functions' Python frames. The C ABI stays what the
// kernels are reached by; this file only prepares its arguments, and ops.py / scan_kernel.py / assoc_kernel.py call it.
#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/extension.h>

#include "../../include/pragnosia_b200.h"

namespace {
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int CHUNK = 64;
// Bytes of per-chunk states the fp32 plain prefill takes at most: more chains or chunks than that go one group after the other. Without
// a limit 768 chains of 4096 tokens took 805 MB for 3.41 ms; 3.49 at 256 MiB, 3.66 at 64, 5.2 at 16.
constexpr long long FP32_SCRATCH = 256LL << 20;

void check(int status, const char *what) {
    if (status == PGB_OK) return;
    std::string msg = std::string(what) + ": " + pgb_status_string(status);
    if (status == PGB_ERR_CUDA) msg += std::string(" [") + pgb_last_cuda_error() + "]";
    throw std::runtime_error(msg);
}
void need_cuda(const Tensor &t) {
    if (t.defined() && !t.is_cuda()) throw std::runtime_error("pragnosia_b200 ops run on CUDA tensors only (there is no CPU path)");
}
template <typename... P> void need_cuda(const Tensor &t, const P &...rest) { need_cuda(t); need_cuda(rest...); }

// an absent tensor is an undefined one from here on
Tensor opt(const OptTensor &t) { return t.has_value() ? *t : Tensor(); }
OptTensor some(const Tensor &t) { return t.defined() ? OptTensor(t) : OptTensor(); }
Tensor f32c(const Tensor &t) {
    if (!t.defined() || (t.scalar_type() == at::kFloat && t.is_contiguous())) return t;
    return t.to(at::kFloat).contiguous();
}
Tensor as(const Tensor &t, at::ScalarType dt) { return !t.defined() || t.scalar_type() == dt ? t : t.to(dt); }
Tensor like(const Tensor &t, at::ScalarType dt) { return as(t, dt).contiguous(); }
float *fp(const Tensor &t) { return t.defined() ? static_cast<float *>(t.data_ptr()) : nullptr; }
void *vp(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }
int code(const Tensor &t) { return t.scalar_type() == at::kFloat ? PGB_F32 : PGB_BF16; }
bool io_type(at::ScalarType t) { return t == at::kFloat || t == at::kBFloat16; }
Tensor alloc(const Tensor &ref, at::IntArrayRef shape, at::ScalarType dt) { return at::empty(shape, ref.options().dtype(dt).requires_grad(false)); }
Tensor bytes(const Tensor &ref, long long n) { return alloc(ref, {n}, at::kByte); }

// the library reads CUDA's current device and is handed that device's current stream
struct OnDevice {
    c10::cuda::CUDAGuard guard;
    void *stream;
    explicit OnDevice(const Tensor &t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

// ------------------------------------------------------------------------------------------------ lambda scan
// The angle as fp32 with unit stride over D and either zero (batch, time) strides -- one angle per channel, read as such -- or
// the dense strides.
struct Angle { Tensor t; long long sb, st; };
Angle angle_view(const Tensor &ang, int64_t B, int64_t T, int64_t D) {
    Tensor a = as(ang, at::kFloat);
    if (a.dim() == 1) a = a.expand({B, T, D});
    TORCH_CHECK_VALUE(a.sizes() == at::IntArrayRef({B, T, D}), "lambda_scan: u, logmag, ang must share the shape (B,T,D)");
    if (D > 1 && a.stride(2) != 1) a = a.contiguous();
    long long sb = B > 1 ? a.stride(0) : 0, st = T > 1 ? a.stride(1) : 0;
    if (!(sb == 0 && st == 0) && !(st == D && sb == T * D)) { a = a.contiguous(); sb = T * D; st = D; }
    return {a, sb, st};
}

struct LambdaOut { Tensor y, hr, hi, hia; };
LambdaOut lambda_fwd(const Tensor &u, const Tensor &lm, const Tensor &ang, const Tensor &h0r_, const Tensor &h0i_, int segments, bool keep) {
    need_cuda(u, lm, ang, h0r_, h0i_);
    TORCH_CHECK_VALUE(u.dim() == 3 && lm.sizes() == u.sizes(), "lambda_scan: u, logmag, ang must share the shape (B,T,D)");
    const int64_t B = u.size(0), T = u.size(1), D = u.size(2);
    OnDevice dev(u);
    const Tensor u32 = f32c(u), lm32 = f32c(lm), h0r = f32c(h0r_), h0i = f32c(h0i_);
    const Angle a = angle_view(ang, B, T, D);
    LambdaOut r{alloc(u, {B, T, D}, at::kFloat), alloc(u, {B, D}, at::kFloat), alloc(u, {B, D}, at::kFloat), Tensor()};
    if (keep) {
        r.hia = alloc(u, {B, T, D}, at::kFloat);
        check(pgb_lambda_scan_fwd_train(fp(u32), fp(lm32), fp(a.t), a.sb, a.st, fp(h0r), fp(h0i), fp(r.y), fp(r.hia), fp(r.hr), fp(r.hi), B, T, D,
                                        dev.stream), "pgb_lambda_scan_fwd_train");
    } else {
        check(pgb_lambda_scan_fwd_ex(fp(u32), fp(lm32), fp(a.t), a.sb, a.st, fp(h0r), fp(h0i), fp(r.y), fp(r.hr), fp(r.hi), B, T, D, segments,
                                     dev.stream), "pgb_lambda_scan_fwd");
    }
    return r;
}
struct LambdaGrads { Tensor du, dlm, dan, d0r, d0i; };
LambdaGrads lambda_bwd(const Tensor &g_, const Tensor &u_, const Tensor &lm_, const Tensor &ang, const Tensor &hr_, const Tensor &hi_, const Tensor &gli_,
                       bool want_dh0) {
    need_cuda(g_, u_, lm_, ang, hr_, hi_);
    const int64_t B = u_.size(0), T = u_.size(1), D = u_.size(2);
    OnDevice dev(u_);
    const Tensor g = f32c(g_), u = f32c(u_), lm = f32c(lm_), hr = f32c(hr_), hi = f32c(hi_), gli = f32c(gli_);
    const Angle a = angle_view(ang, B, T, D);
    LambdaGrads r{alloc(u, {B, T, D}, at::kFloat), alloc(u, {B, T, D}, at::kFloat), alloc(u, {B, T, D}, at::kFloat), Tensor(), Tensor()};
    if (want_dh0) { r.d0r = alloc(u, {B, D}, at::kFloat); r.d0i = alloc(u, {B, D}, at::kFloat); }
    check(pgb_lambda_scan_bwd(fp(g), fp(u), fp(lm), fp(a.t), a.sb, a.st, fp(hr), fp(hi), fp(gli), fp(r.du), fp(r.dlm), fp(r.dan), fp(r.d0r), fp(r.d0i),
                              B, T, D, dev.stream), "pgb_lambda_scan_bwd");
    return r;
}

// Differentiable scan (the reference's _Scan, src/scan_kernel.py:105-140): the forward keeps Im h for the adjoint.
struct LambdaScan : torch::autograd::Function<LambdaScan> {
    static variable_list forward(AutogradContext *ctx, const Tensor &u, const Tensor &lm, const Tensor &ang, const OptTensor &h0r, const OptTensor &h0i) {
        LambdaOut r = lambda_fwd(u, lm, ang, opt(h0r), opt(h0i), 0, true);
        ctx->save_for_backward({u, lm, ang, r.y, r.hia});
        ctx->set_materialize_grads(false);                            // no gradient arrived: undefined, not a tensor of zeros to add
        ctx->saved_data["dh0"] = h0r.has_value();
        return {r.y, r.hr, r.hi};
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        Tensor g = grads[0].defined() ? as(grads[0], at::kFloat) : at::zeros_like(s[3]);
        if (grads[1].defined()) {
            g = g.clone();
            g.select(1, g.size(1) - 1).add_(as(grads[1], at::kFloat));
        }
        LambdaGrads r = lambda_bwd(g, s[0], s[1], s[2], s[3], s[4], grads[2], ctx->saved_data["dh0"].toBool());
        return {r.du, r.dlm, r.dan, r.d0r, r.d0i};
    }
};

bool wants_grad(const Tensor &t) { return t.defined() && t.requires_grad(); }

// (Re h, Re h_T, Im h_T) in u's type; differentiable where a gradient is wanted
std::tuple<Tensor, Tensor, Tensor> scan(const Tensor &u, const Tensor &lm, const Tensor &ang, const OptTensor &h0r, const OptTensor &h0i) {
    const at::ScalarType dt = u.scalar_type();
    if (at::GradMode::is_enabled() && (wants_grad(u) || wants_grad(lm) || wants_grad(ang) || wants_grad(opt(h0r)) || wants_grad(opt(h0i)))) {
        need_cuda(u, lm, ang, opt(h0r), opt(h0i));
        variable_list r = LambdaScan::apply(as(u, at::kFloat), as(lm, at::kFloat), as(ang, at::kFloat), some(as(opt(h0r), at::kFloat)),
                                            some(as(opt(h0i), at::kFloat)));
        return {as(r[0], dt), as(r[1], dt), as(r[2], dt)};
    }
    LambdaOut r = lambda_fwd(u, lm, ang, opt(h0r), opt(h0i), 0, false);
    return {as(r.y, dt), as(r.hr, dt), as(r.hi, dt)};
}

// ------------------------------------------------------------------------------------------------ prep
struct PrepIn { Tensor q, k, v, gate, theta, pos; long long gsb, gst; };
PrepIn prep_in(const Tensor &qp_, const Tensor &kp_, const Tensor &vp_, const Tensor &gl_, const Tensor &theta, const Tensor &pos) {
    need_cuda(qp_, kp_, vp_, theta, pos);
    TORCH_CHECK_VALUE(qp_.dim() == 4 && kp_.sizes() == qp_.sizes() && vp_.sizes() == qp_.sizes(), "prep: qp, kp, vp must share the shape (B,T,H,D)");
    const at::ScalarType dt = io_type(qp_.scalar_type()) ? qp_.scalar_type() : at::kFloat;
    const int64_t per = std::max<int64_t>(1, qp_.size(3) / 32);       // channels a lane moves in one access: strides must keep it aligned
    auto strided = [&](Tensor t) {
        t = as(t, dt);
        const bool ok = t.stride(3) == 1 && t.stride(0) % per == 0 && t.stride(1) % per == 0 && t.stride(2) % per == 0;
        return ok ? t : t.contiguous();
    };
    PrepIn p{strided(qp_), strided(kp_), strided(vp_), as(gl_, dt), f32c(theta), as(pos, at::kLong).contiguous(), 0, 0};
    if (p.k.strides() != p.q.strides() || p.v.strides() != p.q.strides()) { p.q = p.q.contiguous(); p.k = p.k.contiguous(); p.v = p.v.contiguous(); }
    if (p.gate.defined()) {
        if (p.gate.stride(2) != 1) p.gate = p.gate.contiguous();
        p.gsb = p.gate.stride(0); p.gst = p.gate.stride(1);
    }
    return p;
}
std::tuple<Tensor, Tensor, Tensor> prep_fwd(const Tensor &qp, const Tensor &kp, const Tensor &vp_, const OptTensor &gl, const Tensor &theta, const Tensor &pos,
                                            bool out_bf16) {
    const PrepIn p = prep_in(qp, kp, vp_, opt(gl), theta, pos);
    const int64_t B = p.q.size(0), T = p.q.size(1), H = p.q.size(2), D = p.q.size(3);
    OnDevice dev(p.q);
    const at::ScalarType dt = out_bf16 ? at::kBFloat16 : at::kFloat;
    Tensor q = alloc(p.q, {B, H, T, D}, dt), k = alloc(p.q, {B, H, T, D}, dt), v = alloc(p.q, {B, H, T, D}, dt);
    check(pgb_aspin_prep_fwd(vp(p.q), vp(p.k), vp(p.v), code(p.q), p.q.stride(0), p.q.stride(1), p.q.stride(2), vp(p.gate), p.gsb, p.gst, fp(p.theta),
                             static_cast<const long long *>(vp(p.pos)), vp(q), vp(k), vp(v), code(q), B, T, H, D, dev.stream), "pgb_aspin_prep_fwd");
    return {q, k, v};
}
using PrepGrads = std::tuple<Tensor, Tensor, Tensor, OptTensor, OptTensor>;
PrepGrads prep_bwd(const Tensor &qp, const Tensor &kp, const Tensor &vp_, const OptTensor &gl, const Tensor &theta, const Tensor &pos, const Tensor &dq_,
                   const Tensor &dk_, const Tensor &dv_, bool want_theta) {
    need_cuda(dq_, dk_, dv_);
    const PrepIn p = prep_in(qp, kp, vp_, opt(gl), theta, pos);
    const int64_t B = p.q.size(0), T = p.q.size(1), H = p.q.size(2), D = p.q.size(3);
    OnDevice dev(p.q);
    const at::ScalarType gt = io_type(dq_.scalar_type()) ? dq_.scalar_type() : at::kFloat, dt = p.q.scalar_type();
    const Tensor dq = like(dq_, gt), dk = like(dk_, gt), dv = like(dv_, gt);
    Tensor dqp = alloc(p.q, {B, T, H, D}, dt), dkp = alloc(p.q, {B, T, H, D}, dt), dvp = alloc(p.q, {B, T, H, D}, dt), dgl, part;
    if (p.gate.defined()) dgl = alloc(p.q, {B, T, H}, at::kFloat);
    if (want_theta) part = alloc(p.q, {B * pgb_aspin_prep_bwd_tiles(T), H, D / 2}, at::kFloat);
    check(pgb_aspin_prep_bwd(vp(p.q), vp(p.k), vp(p.v), code(p.q), p.q.stride(0), p.q.stride(1), p.q.stride(2), vp(p.gate), p.gsb, p.gst, fp(p.theta),
                             static_cast<const long long *>(vp(p.pos)), vp(dq), vp(dk), vp(dv), code(dq), vp(dqp), vp(dkp), vp(dvp), fp(dgl), fp(part), B, T, H,
                             D, dev.stream), "pgb_aspin_prep_bwd");
    return {dqp, dkp, dvp, some(dgl), want_theta ? OptTensor(part.sum(0)) : OptTensor()};
}

// The backward kernels have no derivative of their own: with create_graph a second differentiation through `grads` raises instead of
// leaving its share out.
variable_list once(const char *what, const variable_list &saved, variable_list grads, const variable_list &incoming) {
    auto wants = [](const variable_list &l) { return std::any_of(l.begin(), l.end(), wants_grad); };
    if (!at::GradMode::is_enabled() || !(wants(saved) || wants(incoming))) return grads;
    const auto node = std::make_shared<torch::autograd::Error>(std::string("Trying to backward through the gradient of ") + what + ": it has no derivative",
                                                               torch::autograd::collect_next_edges(saved, incoming));
    for (Tensor &g : grads)
        if (g.defined()) torch::autograd::set_history(g, node);
    return grads;
}

// prep with its backward kernel
struct Prep : torch::autograd::Function<Prep> {
    static variable_list forward(AutogradContext *ctx, const Tensor &qp, const Tensor &kp, const Tensor &vp_, const OptTensor &gl, const Tensor &theta,
                                 const Tensor &pos) {
        ctx->save_for_backward({qp, kp, vp_, opt(gl), theta, pos});
        ctx->saved_data["theta"] = theta.requires_grad();
        auto [q, k, v] = prep_fwd(qp, kp, vp_, gl, theta, pos, true);
        return {q, k, v};
    }
    static variable_list backward(AutogradContext *ctx, variable_list g) {
        const variable_list s = ctx->get_saved_variables();
        auto [dq, dk, dv, dgl, dth] = prep_bwd(s[0], s[1], s[2], some(s[3]), s[4], s[5], g[0], g[1], g[2], ctx->saved_data["theta"].toBool());
        return once("pragnosia_b200 prep", s, {as(dq, s[0].scalar_type()), as(dk, s[1].scalar_type()), as(dv, s[2].scalar_type()),
                    dgl ? as(*dgl, s[3].scalar_type()) : Tensor(), dth ? as(*dth, s[4].scalar_type()) : Tensor(), Tensor()}, g);
    }
};
using Three = std::optional<std::tuple<Tensor, Tensor, Tensor>>;
// nullopt: a tracer, a torch_dispatch mode (fake tensors, make_fx, selective checkpointing), a functorch transform or a tensor subclass
// wants to see the registered operators
template <typename... P> bool plain(const P &...ts) {
    using c10::DispatchKey;
    const c10::DispatchKeySet special{DispatchKey::Python, DispatchKey::FuncTorchBatched, DispatchKey::FuncTorchGradWrapper};
    return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::tracer::impl::is_dispatch_enabled() &&
           !c10::impl::tls_is_dispatch_key_included(DispatchKey::FuncTorchDynamicLayerFrontMode) &&
           (... && (!ts.defined() || !ts.key_set().has_any(special)));
}
Three prep_diff(const Tensor &qp, const Tensor &kp, const Tensor &vp_, const OptTensor &gl, const Tensor &theta, const Tensor &pos) {
    if (!plain(qp, kp, vp_, opt(gl), theta, pos)) return std::nullopt;
    variable_list r = Prep::apply(qp, kp, vp_, gl, theta, pos);
    return std::make_tuple(r[0], r[1], r[2]);
}

// ------------------------------------------------------------------------------------------------ associative scan
// the tensor the final state is written to: a new one, or the caller's (which may be the S0 it passed: every (sequence, head)
// reads its entering state before it writes its final one)
Tensor state_out(const OptTensor &S_out, const Tensor &ref, int64_t B, int64_t H, int64_t D) {
    if (!S_out.has_value()) return alloc(ref, {B, H, D, D}, at::kFloat);
    TORCH_CHECK_VALUE(S_out->scalar_type() == at::kFloat && S_out->is_contiguous() && S_out->sizes() == at::IntArrayRef({B, H, D, D}),
                      "S_out must be a contiguous fp32 (B,H,D,D) tensor");
    return *S_out;
}
// The plain rule in fp32 with the chunks of a sequence side by side (prefill_fp32_chunk.cu), in groups whose scratch is bounded: whole
// batch rows, or some heads of one, or (a chain that is too long by itself) one chain piece by piece with its state handed on. False:
// the scratch could not be had, nothing was launched.
bool prefill_fp32_grouped(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &la, const Tensor &S0, const Tensor &theta, const Tensor &shift,
                          double shift_host, const Tensor &o, const Tensor &S, const Tensor &sent, void *stream) {
    const long long B = q.size(0), H = q.size(1), T = q.size(2), D = q.size(3), NC = (T + CHUNK - 1) / CHUNK;
    const long long chunk = pgb_aspin_prefill_fp32_scratch_bytes(1, 1, CHUNK, D), chain = pgb_aspin_prefill_fp32_scratch_bytes(1, 1, T, D);
    const long long chains = std::min(B * H, std::max(1LL, FP32_SCRATCH / chain)), piece = chain <= FP32_SCRATCH ? T : FP32_SCRATCH / chunk * CHUNK;
    const long long nb = std::max(1LL, chains / H), nh = std::min(chains, H);
    const long long n = pgb_aspin_prefill_fp32_scratch_bytes(nb, nh, std::min(piece, T), D);
    Tensor scratch;
    try {
        scratch = bytes(q, n);
    } catch (const c10::OutOfMemoryError &) {
        return false;
    }
    char *out = static_cast<char *>(vp(o));
    for (long long b = 0; b < B; b += nb)
        for (long long h = 0; h < H; h += nh)
            for (long long t = 0; t < T; t += piece) {
                const long long c = b * H + h, Bn = std::min(nb, B - b), Hn = std::min(nh, H - h), Tn = std::min(piece, T - t), row = c * T + t;
                const float *first = t > 0 ? fp(S) + c * D * D : S0.defined() ? fp(S0) + c * D * D : nullptr;
                check(pgb_aspin_prefill_fp32_fwd(fp(q) + row * D, fp(k) + row * D, fp(v) + row * D, fp(la) + row, first,
                                                 t == 0 && theta.defined() ? fp(theta) + h * (D / 2) : nullptr, fp(shift), shift_host,
                                                 out + row * D * o.element_size(), code(o), fp(S) + c * D * D,
                                                 sent.defined() ? static_cast<char *>(vp(sent)) + (c * NC + t / CHUNK) * D * D * 2 : nullptr, vp(scratch), n,
                                                 Bn, Hn, Tn, D, stream), "pgb_aspin_prefill_fp32_fwd");
            }
    return true;
}
using ScanOut = std::tuple<Tensor, Tensor, OptTensor>;
// out_type: -1 = q's (fp32 where q is neither fp32 nor bf16), else a dtype code
ScanOut prefill(const Tensor &q_, const Tensor &k_, const Tensor &v_, const Tensor &la_, const OptTensor &beta_, const OptTensor &S0_, const OptTensor &theta_,
                const OptTensor &shift_dev_, double shift_host, bool want_sent, int precision, int out_type, const OptTensor &S_out) {
    need_cuda(q_, k_, v_, la_, opt(shift_dev_));
    const int64_t B = q_.size(0), H = q_.size(1), T = q_.size(2), D = q_.size(3);
    OnDevice dev(q_);
    const at::ScalarType dt = io_type(q_.scalar_type()) ? q_.scalar_type() : at::kFloat;
    const Tensor q = like(q_, dt), k = like(k_, dt), v = like(v_, dt), la = f32c(la_), beta = f32c(opt(beta_)), S0 = f32c(opt(S0_)), theta = opt(theta_),
                 shift = opt(shift_dev_);
    const at::ScalarType ot = out_type < 0 ? dt : out_type == PGB_F32 ? at::kFloat : at::kBFloat16;
    Tensor o = alloc(q, {B, H, T, D}, ot), S = state_out(S_out, q, B, H, D), sent;
    if (want_sent) sent = alloc(q, {B, H, (T + CHUNK - 1) / CHUNK, D, D}, at::kBFloat16);
    const int oc = code(o);
    if (beta.defined() && dt == at::kBFloat16 && precision != PGB_PREFILL_FP32 && B * H <= 65535) {
        // delta rule on the tensor cores: the chunk inverses go through a scratch buffer
        long long n = want_sent ? pgb_aspin_delta_scratch_bytes(B, H, T) : pgb_aspin_delta_prefill_scratch_bytes(B, H, T, D);
        Tensor scratch;
        try {
            scratch = bytes(q, n);
        } catch (const c10::OutOfMemoryError &) {                     // without the segments' share, then
            const long long least = pgb_aspin_delta_scratch_bytes(B, H, T);
            if (n == least) throw;
            scratch = bytes(q, n = least);
        }
        check(pgb_aspin_delta_prefill_fwd(vp(q), vp(k), vp(v), fp(la), fp(beta), fp(S0), fp(theta), fp(shift), shift_host, vp(o), oc, fp(S), vp(sent),
                                          vp(scratch), n, B, H, T, D, dev.stream), "pgb_aspin_delta_prefill_fwd");
        return {o, S, some(sent)};
    }
    if (!beta.defined() && dt == at::kBFloat16 && precision != PGB_PREFILL_FP32 && D == 64 && !(S0.defined() && S0.is_same_size(S) && S0.data_ptr() == S.data_ptr())) {
        const long long n = pgb_aspin_prefill_segments_scratch_bytes(B, H, T, D); // few long chains, or few in the last round: their segments side by side
        if (n > 0) {
            const Tensor scratch = bytes(q, n);
            check(pgb_aspin_prefill_segments_fwd(vp(q), vp(k), vp(v), fp(la), fp(S0), fp(theta), fp(shift), shift_host, vp(o), oc, fp(S), vp(sent),
                                                 vp(scratch), n, B, H, T, D, dev.stream), "pgb_aspin_prefill_segments_fwd");
            return {o, S, some(sent)};
        }
    }
    // fp32 plain rule: the chunks side by side, also where the chains alone fill the GPU (1024 chains of 8 chunks: 616 us against the
    // walk's 776; 24 of 64: 134 against 1258). A single chunk a chain at D = 64 is the walk's: 96 .. 1024 chains 31 .. 121 us against 32 .. 130.
    if (!beta.defined() && dt == at::kFloat && precision != PGB_PREFILL_TENSOR && B > 0 && H > 0 && T > 0 && B * H <= 65535 && (D == 64 || D == 128) &&
        !(D == 64 && T <= CHUNK && 2 * B * H > at::cuda::getCurrentDeviceProperties()->multiProcessorCount) &&
        prefill_fp32_grouped(q, k, v, la, S0, theta, shift, shift_host, o, S, sent, dev.stream))
        return {o, S, some(sent)};
    check(pgb_aspin_prefill_fwd(vp(q), vp(k), vp(v), code(q), fp(la), fp(beta), fp(S0), fp(theta), fp(shift), shift_host, vp(o), oc, fp(S), vp(sent), B, H, T,
                                D, precision, dev.stream), "pgb_aspin_prefill_fwd");
    return {o, S, some(sent)};
}

// The scan with what its backward reads: (o, S, sent, W, X); bf16 q, k, v, fp32 la, beta, all contiguous; W and X with the delta rule.
struct TrainOut { Tensor o, S, sent, W, X; };
TrainOut train_fwd(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &la, const Tensor &beta, const Tensor &S0) {
    need_cuda(q, k, v, la, beta, S0);
    const int64_t B = q.size(0), H = q.size(1), T = q.size(2), D = q.size(3);
    OnDevice dev(q);
    if (!beta.defined()) {
        const long long n = pgb_aspin_prefill_segments_scratch_bytes(B, H, T, D);
        TrainOut r{alloc(q, {B, H, T, D}, at::kBFloat16), alloc(q, {B, H, D, D}, at::kFloat), alloc(q, {B, H, (T + CHUNK - 1) / CHUNK, D, D}, at::kBFloat16),
                   Tensor(), Tensor()};
        const Tensor scratch = n > 0 ? bytes(q, n) : Tensor();
        check(pgb_aspin_prefill_train_fwd(vp(q), vp(k), vp(v), fp(la), fp(S0), vp(r.o), fp(r.S), vp(r.sent), vp(scratch), n, B, H, T, D, dev.stream),
              "pgb_aspin_prefill_train_fwd");
        return r;
    }
    const long long n = pgb_aspin_delta_scratch_bytes(B, H, T);
    TrainOut r{alloc(q, {B, H, T, D}, at::kBFloat16), alloc(q, {B, H, D, D}, at::kFloat), alloc(q, {B, H, (T + CHUNK - 1) / CHUNK, D, D}, at::kBFloat16),
               alloc(q, {B, H, T, D}, at::kBFloat16), bytes(q, n)};
    check(pgb_aspin_delta_prefill_train_fwd(vp(q), vp(k), vp(v), fp(la), fp(beta), fp(S0), vp(r.o), fp(r.S), vp(r.sent), vp(r.W), vp(r.X), n, B, H, T, D,
                                            dev.stream), "pgb_aspin_delta_prefill_train_fwd");
    return r;
}
struct TrainGrads { Tensor dq, dk, dv, dla, dbe, dS0; };
TrainGrads train_bwd(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &la, const Tensor &beta, const Tensor &sent, const Tensor &W, const Tensor &X,
                     const Tensor &dout_, const Tensor &dsent_, const Tensor &dS_, bool want_dS0) {
    need_cuda(q, k, v, la, beta, sent, dout_);
    const int64_t B = q.size(0), H = q.size(1), T = q.size(2), D = q.size(3);
    OnDevice dev(q);
    const Tensor dout = like(dout_, at::kBFloat16), dsent = f32c(dsent_), dS = f32c(dS_);
    TrainGrads r{alloc(q, {B, H, T, D}, at::kBFloat16), alloc(q, {B, H, T, D}, at::kBFloat16), alloc(q, {B, H, T, D}, at::kBFloat16),
                 alloc(q, {B, H, T}, at::kFloat), Tensor(), Tensor()};
    if (beta.defined()) r.dbe = alloc(q, {B, H, T}, at::kFloat);
    if (want_dS0) r.dS0 = alloc(q, {B, H, D, D}, at::kFloat);
    const long long n = pgb_aspin_train_scratch_bytes(B, H, T, D, beta.defined());
    const Tensor scratch = bytes(q, n);
    check(pgb_aspin_train_bwd(vp(q), vp(k), vp(v), fp(la), fp(beta), vp(sent), vp(W), vp(X), vp(dout), fp(dsent), fp(dS), vp(r.dq), vp(r.dk), vp(r.dv),
                              fp(r.dla), fp(r.dbe), fp(r.dS0), vp(scratch), n, B, H, T, D, dev.stream), "pgb_aspin_train_bwd");
    return r;
}

// The scan of bf16 operands with all its gradients as one library call each way (train_chunk.cu): (o, final state, state entering
// each chunk), each of them differentiable. No beta: the plain rule.
struct Scan : torch::autograd::Function<Scan> {
    static variable_list forward(AutogradContext *ctx, const Tensor &q_, const Tensor &k_, const Tensor &v_, const Tensor &la, const OptTensor &beta,
                                 const OptTensor &S0) {
        const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous(), la32 = f32c(la), be32 = f32c(opt(beta));
        TrainOut r = train_fwd(q, k, v, la32, be32, f32c(opt(S0)));
        ctx->save_for_backward({q, k, v, la32, be32, r.sent, r.W, r.X});
        ctx->set_materialize_grads(false);
        auto &d = ctx->saved_data;
        d["la"] = static_cast<int64_t>(la.scalar_type());
        if (beta) d["beta"] = static_cast<int64_t>(beta->scalar_type());
        if (S0) d["S0"] = static_cast<int64_t>(S0->scalar_type());
        d["dS0"] = S0.has_value() && S0->requires_grad();
        return {r.o, r.S, r.sent};
    }
    static variable_list backward(AutogradContext *ctx, variable_list g) {
        const variable_list s = ctx->get_saved_variables();
        auto &d = ctx->saved_data;
        auto type = [&](const char *n) { return static_cast<at::ScalarType>(d[n].toInt()); };
        TrainGrads r = train_bwd(s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], g[0].defined() ? g[0] : at::zeros_like(s[0]), g[2], g[1], d["dS0"].toBool());
        return once("pragnosia_b200 scan", s, {r.dq, r.dk, r.dv, as(r.dla, type("la")), r.dbe.defined() ? as(r.dbe, type("beta")) : Tensor(),
                    r.dS0.defined() ? as(r.dS0, type("S0")) : Tensor()}, g);
    }
};
Three scan_diff(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &la, const OptTensor &beta, const OptTensor &S0) {
    if (!plain(q, k, v, la, opt(beta), opt(S0))) return std::nullopt;
    variable_list r = Scan::apply(q, k, v, la, beta, S0);
    return std::make_tuple(r[0], r[1], r[2]);
}
}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    using nogil_t = pybind11::call_guard<pybind11::gil_scoped_release>;             // as a ctypes call would: other threads run meanwhile
    const nogil_t nogil;
    m.def("lambda_scan", [](const Tensor &u, const Tensor &lm, const Tensor &ang, const OptTensor &h0r, const OptTensor &h0i, int segments, bool keep) {
        LambdaOut r = lambda_fwd(u, lm, ang, opt(h0r), opt(h0i), segments, keep);
        return std::make_tuple(r.y, r.hr, r.hi, some(r.hia));
    }, nogil);
    m.def("lambda_scan_bwd", [](const Tensor &g, const Tensor &u, const Tensor &lm, const Tensor &ang, const Tensor &hr, const Tensor &hi, const OptTensor &gli,
                                bool want_dh0) {
        LambdaGrads r = lambda_bwd(g, u, lm, ang, hr, hi, opt(gli), want_dh0);
        return std::make_tuple(r.du, r.dlm, r.dan, some(r.d0r), some(r.d0i));
    }, nogil);
    m.def("scan", &scan, nogil);
    m.def("prep", &prep_fwd, nogil);
    m.def("prep_bwd", &prep_bwd, nogil);
    m.def("prep_diff", &prep_diff, nogil);
    m.def("prefill", &prefill, nogil);
    m.def("scan_train_fwd", [](const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &la, const OptTensor &beta, const OptTensor &S0) {
        TrainOut r = train_fwd(q, k, v, la, opt(beta), opt(S0));
        return std::make_tuple(r.o, r.S, r.sent, some(r.W), some(r.X));
    }, nogil);
    m.def("scan_train_bwd", [](const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &la, const OptTensor &beta, const Tensor &sent, const OptTensor &W,
                               const OptTensor &X, const Tensor &dout, const OptTensor &dsent, const OptTensor &dS, bool want_dS0) {
        TrainGrads r = train_bwd(q, k, v, la, opt(beta), sent, opt(W), opt(X), dout, opt(dsent), opt(dS), want_dS0);
        return std::make_tuple(r.dq, r.dk, r.dv, r.dla, some(r.dbe), some(r.dS0));
    }, nogil);
    m.def("scan_diff", &scan_diff, nogil);
}
