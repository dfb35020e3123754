// Tensor-level front end of the C ABI for the calls that decode loops and short prompts make: argument checks, output
// allocation, the current stream and the call, in native code.  Through Python and ctypes the same work took 30 to 40 us a
// call (a decode step of one sequence runs 3 us on the GPU, one of sixteen 25), so these calls were bound by it.
//
// Every function returns the status of the C ABI first; the Python wrappers (ops.py) raise on it.  Inputs are normalised as
// there: activations of one dtype, states in fp32, contiguous where the ABI has no strides.  Nothing is kept between calls.
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include "xlstm_cuda.h"

namespace {

using at::Tensor;
using OptTensor = c10::optional<Tensor>;

void need_cuda(const Tensor &t) {
    if (!t.is_cuda()) throw std::runtime_error("xlstm_cuda kernels need CUDA tensors (no CPU fallback exists)");
}
void need_cuda(const OptTensor &t) {
    if (t) need_cuda(*t);
}
// The ABI takes bare pointers: whatever could make a kernel read beyond a tensor is refused here.
void need(bool ok, const char *what) {
    if (!ok) throw py::value_error(what);
}
void need_type(const Tensor &t, at::ScalarType type, const char *what) {
    if (t.scalar_type() != type) throw py::type_error(what);
}
int dtype_code(const Tensor &t) {
    if (t.scalar_type() == at::kBFloat16) return XLSTM_BF16;
    if (t.scalar_type() == at::kFloat) return XLSTM_F32;
    throw py::type_error(std::string("xlstm_cuda kernels take float32 or bfloat16 activations, got ") + at::toString(t.scalar_type()));
}
// Launches run without the interpreter's lock, as calls through ctypes do: a full launch queue stalls this thread alone.
template <typename Call> int unlocked(Call &&call) {
    py::gil_scoped_release release;
    return call();
}
void *stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
const void *ptr(const OptTensor &t) { return t ? t->data_ptr() : nullptr; }
const float *fptr(const OptTensor &t) { return t ? static_cast<const float *>(t->data_ptr()) : nullptr; }
float *fptr(const Tensor &t) { return static_cast<float *>(t.data_ptr()); }
OptTensor cast_contiguous(const OptTensor &t, at::ScalarType dt) {
    return t ? OptTensor(t->to(dt).contiguous()) : OptTensor();
}

struct State {
    OptTensor C, n, m;
    // C, which a step of a settled state reads early, is a copy made here, by the launch right before the step's: not settled,
    // whatever the caller says
    bool converted;
    State(const OptTensor &c, const OptTensor &nn, const OptTensor &mm, int64_t B, int64_t NH, int64_t dqk, int64_t dv)
        : C(cast_contiguous(c, at::kFloat)), n(cast_contiguous(nn, at::kFloat)), m(cast_contiguous(mm, at::kFloat)) {
        need(C.has_value() == n.has_value() && C.has_value() == m.has_value(), "a state is (C, n, m), all three or None");
        if (C) {
            need_cuda(C); need_cuda(n); need_cuda(m);
            need(C->numel() == B * NH * dqk * dv && n->numel() == B * NH * dqk && m->numel() == B * NH,
                 "state of another size than [B,NH,dqk,dv], [B,NH,dqk], [B,NH]");
            m = m->reshape({B, NH});
        }
        converted = c && !C->is_same(*c);
    }
    int step_flags(bool settled) const { return settled && C && !converted ? XLSTM_STEP_STATE_SETTLED : 0; }
};
struct NewState {
    Tensor C, n, m;
    NewState(const Tensor &q, const State &st, int64_t B, int64_t NH, int64_t dqk, int64_t dv, bool inplace) {
        const auto f32 = q.options().dtype(at::kFloat);
        C = inplace && st.C ? *st.C : at::empty({B, NH, dqk, dv}, f32);
        n = at::empty({B, NH, dqk}, f32);
        m = at::empty({B, NH}, f32);
    }
};

void step_inputs(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &i, const Tensor &f, int64_t B, int64_t NH,
                 int64_t dqk, int64_t dv) {
    need_type(k, q.scalar_type(), "q, k and v of one dtype");
    need_type(v, q.scalar_type(), "q, k and v of one dtype");
    need(k.numel() == B * NH * dqk && v.numel() == B * NH * dv && i.numel() == B * NH && f.numel() == B * NH,
         "k, v or gates of another size than q: [B,NH,dqk], [B,NH,dv], [B,NH]");
}
// v is read four elements at a time
Tensor aligned4(const Tensor &t) {
    return reinterpret_cast<uintptr_t>(t.data_ptr()) % (4 * t.element_size()) ? t.clone() : t;
}

bool aligned16(const Tensor &t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

// q, k: [B, NH, dqk], v: [B, NH, dv], i, f: [B, NH], or the same with a token dimension of one ([B, NH, 1, d], [B, NH, 1])
py::tuple mlstm_step(Tensor q, Tensor k, Tensor v, Tensor i, Tensor f, const OptTensor &C0, const OptTensor &n0,
                     const OptTensor &m0, double eps, bool inplace, double gate_cap, bool state_settled) {
    for (const Tensor *t : {&q, &k, &v, &i, &f}) need_cuda(*t);
    const bool token_dim = q.dim() == 4;
    if (q.dim() != 3 && !(token_dim && q.size(2) == 1))
        throw py::value_error("mlstm_step takes q as [B, NH, dqk] or [B, NH, 1, dqk]");
    const int64_t B = q.size(0), NH = q.size(1), dqk = q.size(-1), dv = v.size(-1);
    const int dt = dtype_code(q);
    step_inputs(q, k, v, i, f, B, NH, dqk, dv);
    q = q.contiguous(); k = k.contiguous(); v = aligned4(v.contiguous());
    i = i.to(q.scalar_type()).contiguous(); f = f.to(q.scalar_type()).contiguous();
    const State st(C0, n0, m0, B, NH, dqk, dv);
    const Tensor h = token_dim ? at::empty({B, NH, 1, dv}, q.options()) : at::empty({B, NH, dv}, q.options());
    const NewState out(q, st, B, NH, dqk, dv, inplace);
    const int flags = st.step_flags(state_settled);
    const int rc = unlocked([&] {
        return xlstm_mlstm_step_ex(q.data_ptr(), k.data_ptr(), v.data_ptr(), i.data_ptr(), f.data_ptr(), fptr(st.C), fptr(st.n),
                                   fptr(st.m), h.data_ptr(), fptr(out.C), fptr(out.n), fptr(out.m), (int)B, (int)NH, (int)dqk,
                                   (int)dv, (float)eps, (float)gate_cap, flags, dt, stream());
    });
    return py::make_tuple(rc, h, out.C, out.n, out.m);
}

bool dense_heads(const Tensor &t) { return t.stride(2) == 1 && (t.size(1) == 1 || t.stride(1) == t.size(2)); }

struct Stepped {
    int rc;
    Tensor y;
    NewState state;
    py::tuple tuple() const { return py::make_tuple(rc, y, state.C, state.n, state.m); }
};
Stepped step_gated(Tensor q, Tensor k, Tensor v, Tensor i, Tensor f, Tensor ogate, const OptTensor &norm_weight,
                   const OptTensor &C0, const OptTensor &n0, const OptTensor &m0, double eps, double norm_eps,
                   bool inplace, double gate_cap, bool state_settled) {
    for (const Tensor *t : {&q, &k, &v, &i, &f, &ogate}) need_cuda(*t);
    need_cuda(norm_weight);
    if (q.dim() != 3) throw py::value_error("mlstm_step_gated takes q as [B, NH, dqk]");
    const int64_t B = q.size(0), NH = q.size(1), dqk = q.size(2), dv = v.size(-1);
    const int dt = dtype_code(q);
    const auto type = q.scalar_type();
    step_inputs(q, k, v, i, f, B, NH, dqk, dv);
    i = i.to(type); f = f.to(type);
    if (i.dim() != 2) i = i.reshape({B, NH});
    if (f.dim() != 2) f = f.reshape({B, NH});
    const bool in_place = dense_heads(q) && dense_heads(k) && dense_heads(v) && i.stride(1) == 1 && f.stride(1) == 1 &&
                          (B == 1 || (i.stride(0) == f.stride(0) && v.stride(0) % 4 == 0)) &&
                          reinterpret_cast<uintptr_t>(v.data_ptr()) % (4 * v.element_size()) == 0;
    if (!in_place) {
        q = q.contiguous(); k = k.contiguous(); v = aligned4(v.contiguous()); i = i.contiguous(); f = f.contiguous();
    }
    const int64_t pitch[4] = {B == 1 ? 0 : q.stride(0), B == 1 ? 0 : k.stride(0), B == 1 ? 0 : v.stride(0), B == 1 ? 0 : i.stride(0)};
    Tensor og = ogate.to(type);
    need(og.numel() == B * NH * dv && (!norm_weight || norm_weight->numel() == NH * dv),
         "output gate or norm weight of another size than [B,NH*dv], [NH*dv]");
    if (og.dim() != 2 || og.stride(1) != 1 || og.size(1) != NH * dv) og = og.reshape({B, NH * dv}).contiguous();
    int64_t ld = B > 1 ? og.stride(0) : NH * dv;
    if (ld < NH * dv) { og = og.contiguous(); ld = NH * dv; }
    const OptTensor w = cast_contiguous(norm_weight, type);
    const State st(C0, n0, m0, B, NH, dqk, dv);
    const Tensor y = at::empty({B, NH * dv}, q.options());
    const NewState out(q, st, B, NH, dqk, dv, inplace);
    const int flags = st.step_flags(state_settled);
    const int rc = unlocked([&] {
        return xlstm_mlstm_step_gated_rows(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), i.data_ptr(), f.data_ptr(), pitch, fptr(st.C), fptr(st.n), fptr(st.m),
            og.data_ptr(), ld, ptr(w), (float)norm_eps, y.data_ptr(), fptr(out.C), fptr(out.n), fptr(out.m), (int)B, (int)NH,
            (int)dqk, (int)dv, (float)eps, (float)gate_cap, flags, dt, stream());
    });
    return {rc, y, out};
}
py::tuple mlstm_step_gated(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &i, const Tensor &f, const Tensor &ogate,
                           const OptTensor &norm_weight, const OptTensor &C0, const OptTensor &n0, const OptTensor &m0, double eps,
                           double norm_eps, bool inplace, double gate_cap, bool state_settled) {
    return step_gated(q, k, v, i, f, ogate, norm_weight, C0, n0, m0, eps, norm_eps, inplace, gate_cap, state_settled).tuple();
}

py::tuple mlstm_chunkwise(Tensor q, Tensor k, Tensor v, Tensor i, Tensor f, const OptTensor &C0, const OptTensor &n0,
                          const OptTensor &m0, int64_t chunk_size, double eps, OptTensor workspace, const OptTensor &h_out,
                          double gate_cap) {
    for (const Tensor *t : {&q, &k, &v, &i, &f}) need_cuda(*t);
    if (q.dim() != 4) throw py::value_error("mlstm_chunkwise takes q as [B, NH, S, dqk]");
    const int64_t B = q.size(0), NH = q.size(1), S = q.size(2), dqk = q.size(3), dv = v.size(-1);
    const int dt = dtype_code(q);
    const auto type = q.scalar_type();
    auto fix = [](const Tensor &t) { return t.stride(-1) == 1 ? t : t.contiguous(); };
    auto covers = [](const Tensor &t, at::IntArrayRef s) {
        bool ok = t.dim() >= (int64_t)s.size();
        for (size_t d = 0; ok && d < s.size(); ++d) ok = t.size(d) >= s[d];
        return ok;
    };
    need(covers(k, {B, NH, S, dqk}) && covers(v, {B, NH, S, dv}) && covers(i, {B, NH, S}) && covers(f, {B, NH, S}),
         "k, v or gates smaller than q: [B,NH,S,dqk], [B,NH,S,dv], [B,NH,S]");
    need_cuda(h_out); need_cuda(workspace);
    q = fix(q); k = fix(k.to(type)); v = fix(v.to(type));
    i = i.to(type); f = f.to(type);
    if (i.strides() != f.strides()) { i = i.contiguous(); f = f.contiguous(); }
    const State st(C0, n0, m0, B, NH, dqk, dv);
    const Tensor h = h_out ? *h_out : at::empty({B, NH, S, dv}, q.options());
    const NewState out(q, st, B, NH, dqk, dv, false);
    int64_t strides[15];
    const Tensor *ts[5] = {&q, &k, &v, &h, &i};
    for (int t = 0; t < 5; ++t)
        for (int d = 0; d < 3; ++d) strides[3 * t + d] = ts[t]->stride(d);
    const size_t need = xlstm_mlstm_chunkwise_workspace_bytes((int)B, (int)NH, (int)S, (int)dqk, (int)dv, (int)chunk_size, dt);
    if (need && (!workspace || workspace->nbytes() < need)) workspace = at::empty({(int64_t)need}, q.options().dtype(at::kByte));
    const size_t bytes = workspace ? workspace->nbytes() : 0;
    void *ws = workspace ? workspace->data_ptr() : nullptr;
    const int rc = unlocked([&] {
        return xlstm_mlstm_chunkwise_fwd_gatecap(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), i.data_ptr(), f.data_ptr(), fptr(st.C), fptr(st.n), fptr(st.m),
            h.data_ptr(), fptr(out.C), fptr(out.n), fptr(out.m), (int)B, (int)NH, (int)S, (int)dqk, (int)dv, (int)chunk_size,
            (float)eps, (float)gate_cap, dt, strides, ws, bytes, stream());
    });
    return py::make_tuple(rc, h, out.C, out.n, out.m);
}

// rows of x as [M, K] bf16 and the output [.., N]
std::vector<int64_t> with_last(const Tensor &x, int64_t n) {
    auto s = x.sizes().vec();
    s.back() = n;
    return s;
}

struct Result {
    int rc;
    Tensor y;
    const char *what;   // the call that gave rc
    py::tuple tuple() const { return py::make_tuple(rc, y); }
};
Result linear(const Tensor &weight, const Tensor &x, const OptTensor &bias, const OptTensor &norm_weight, double norm_eps,
              const OptTensor &residual, bool swiglu_pair, int64_t max_rows, bool weights_settled) {
    need_cuda(weight); need_cuda(x); need_cuda(bias); need_cuda(norm_weight); need_cuda(residual);
    if (weight.scalar_type() != at::kBFloat16) throw py::type_error("linear_token and linear_rows are bf16 kernels");
    const int64_t K = x.size(-1);
    need(weight.dim() == 2 && weight.size(1) == K, "weight must be [N, K] for rows of K elements");
    need(!swiglu_pair || weight.size(0) % 2 == 0, "a SwiGLU pair has as many gate rows as up rows");
    need(!bias || bias->numel() == weight.size(0), "bias must have one element per weight row");
    need(!norm_weight || norm_weight->numel() == K, "norm weight must have K elements");
    const Tensor x2 = x.reshape({-1, K}).to(at::kBFloat16).contiguous();
    const int64_t M = x2.size(0);
    if (M > max_rows)
        throw py::value_error("this Linear takes at most " + std::to_string(max_rows) + " rows, got " + std::to_string(M));
    const Tensor w = weight.contiguous();
    const int64_t N = swiglu_pair ? w.size(0) / 2 : w.size(0);
    const OptTensor b = cast_contiguous(bias, at::kBFloat16), nw = cast_contiguous(norm_weight, at::kBFloat16);
    need(!residual || residual->numel() == M * N, "residual must have the size of the result");
    const OptTensor r = residual ? cast_contiguous(residual->reshape({-1, N}), at::kBFloat16) : OptTensor();
    const Tensor y = at::empty(with_last(x, N), x.options().dtype(at::kBFloat16));
    const int epi = swiglu_pair ? 2 : (r ? 1 : 0);
    // a dense copy made here is written by the launch right before the call
    const int flags = weights_settled && w.is_same(weight) ? XLSTM_LINEAR_WEIGHTS_SETTLED : 0;
    const bool token = max_rows <= 4;
    const int rc = unlocked([&] {
        return token
            ? xlstm_linear_token(w.data_ptr(), x2.data_ptr(), ptr(b), ptr(nw), (float)norm_eps, ptr(r), y.data_ptr(), (int)M,
                                 (int)N, (int)K, epi, XLSTM_BF16, stream())
            : xlstm_linear_rows_norm(w.data_ptr(), x2.data_ptr(), ptr(b), ptr(nw), (float)norm_eps, ptr(r), y.data_ptr(), (int)M,
                                     (int)N, (int)K, epi, flags, XLSTM_BF16, stream());
    });
    return {rc, y, token ? "xlstm_linear_token" : "xlstm_linear_rows_norm"};
}
py::tuple linear_token(const Tensor &weight, const Tensor &x, const OptTensor &bias, const OptTensor &norm_weight,
                       double norm_eps, const OptTensor &residual, bool swiglu_pair, int64_t max_rows, bool weights_settled) {
    return linear(weight, x, bias, norm_weight, norm_eps, residual, swiglu_pair, max_rows, weights_settled).tuple();
}

Result norm(const Tensor &x, const OptTensor &weight, double eps) {
    need_cuda(x); need_cuda(weight);
    const int64_t cols = x.size(-1);
    need(!weight || weight->numel() == cols, "norm weight must have one element per column");
    const Tensor xc = x.contiguous();
    const OptTensor w = cast_contiguous(weight, xc.scalar_type());
    const Tensor y = at::empty_like(xc);
    const int dt = dtype_code(xc);
    const int rc = unlocked([&] {
        return xlstm_rms_norm(xc.data_ptr(), ptr(w), y.data_ptr(), cols ? xc.numel() / cols : 0, (int)cols, (float)eps, dt,
                              stream());
    });
    return {rc, y, "xlstm_rms_norm"};
}
py::tuple rms_norm(const Tensor &x, const OptTensor &weight, double eps) { return norm(x, weight, eps).tuple(); }

py::tuple add_rms_norm(const Tensor &x, const Tensor &residual, const OptTensor &weight, double eps) {
    need_cuda(x); need_cuda(residual); need_cuda(weight);
    const int64_t cols = x.size(-1);
    need(residual.numel() == x.numel() && (!weight || weight->numel() == cols),
         "residual of another size than x, or norm weight of another size than a row");
    const Tensor xc = x.contiguous(), rc_ = residual.to(x.scalar_type()).contiguous();
    const OptTensor w = cast_contiguous(weight, xc.scalar_type());
    const Tensor s = at::empty_like(xc), y = at::empty_like(xc);
    const int dt = dtype_code(xc);
    const int rc = unlocked([&] {
        return xlstm_add_rms_norm(xc.data_ptr(), rc_.data_ptr(), ptr(w), s.data_ptr(), y.data_ptr(),
                                  cols ? xc.numel() / cols : 0, (int)cols, (float)eps, dt, stream());
    });
    return py::make_tuple(rc, s, y);
}

// One token of B sequences through an mLSTM block, launch after launch as mLSTMBlock._token_step describes them: W, b are the
// merged input projections, ffn the gate and up projections.  rows: the Linears for up to 16 rows, else those for up to 4; the
// norms are in them (more than 48 KB of rows, or rows or a norm weight off 16 bytes: launches of their own, which take both).
// Through Python the seven launches of a block took 140 us of host time, as much as the GPU has work for 16 sequences of 4096.
py::tuple token_block(const Tensor &x, const Tensor &W, const OptTensor &b, const OptTensor &norm_w, double norm_eps, int64_t NH,
                      int64_t dqk, int64_t dv, const OptTensor &C0, const OptTensor &n0, const OptTensor &m0,
                      const OptTensor &head_norm_w, double eps, double head_norm_eps, bool inplace, double gate_cap,
                      const Tensor &out_w, const OptTensor &out_b, const OptTensor &ffn_norm_w, double ffn_norm_eps,
                      const Tensor &ffn, const Tensor &down_w, const OptTensor &down_b, bool rows) {
    need(x.dim() == 2 && W.dim() == 2 && W.size(0) == 2 * NH * dqk + 2 * NH * dv + 2 * NH,
         "token_block takes x as [B, D] and W as the merged q, k, v, i, f and o projections");
    const OptTensor none;
    auto failed = [&](int rc, const char *call) { return py::make_tuple(rc, call, x, none, none, none); };
    // settled: the launch before the Linear is one of this block's, none of which writes weights
    auto project = [&](const Tensor &w, const Tensor &in, const OptTensor &bias, const OptTensor &nw, double ne, const OptTensor &res,
                       bool pair, bool settled) -> Result {
        if (!rows) return linear(w, in, bias, nw, ne, res, pair, 4, false);
        const bool fits = in.size(0) * (2 * in.size(1) + 64) + 2 * in.size(1) <= XLSTM_LINEAR_NORM_BYTES;
        if (!nw || (fits && aligned16(in) && aligned16(*nw))) return linear(w, in, bias, nw, ne, res, pair, 16, settled);
        const Result n = norm(in, nw, ne);
        if (n.rc) return n;
        return linear(w, n.y, bias, none, 0.0, res, pair, 16, true);
    };
    const Result y = project(W, x, b, norm_w, norm_eps, none, false, false);
    if (y.rc) return failed(y.rc, y.what);
    int64_t at = 0;
    auto columns = [&](int64_t n) {
        const Tensor t = y.y.narrow(1, at, n);
        at += n;
        return t;
    };
    const int64_t B = x.size(0);
    const Tensor q = columns(NH * dqk).view({B, NH, dqk}), k = columns(NH * dqk).view({B, NH, dqk}), v = columns(NH * dv).view({B, NH, dv});
    const Tensor i = columns(NH), f = columns(NH), o = columns(NH * dv);
    // the launch before the step is the projection above: the state is settled
    const Stepped st = step_gated(q, k, v, i, f, o, head_norm_w, C0, n0, m0, eps, head_norm_eps, inplace, gate_cap, true);
    if (st.rc) return failed(st.rc, "xlstm_mlstm_step_gated_rows");
    const Result x1 = project(out_w, st.y, out_b, none, 0.0, x, false, true);
    if (x1.rc) return failed(x1.rc, x1.what);
    const Result act = project(ffn, x1.y, none, ffn_norm_w, ffn_norm_eps, none, true, true);
    if (act.rc) return failed(act.rc, act.what);
    const Result x3 = project(down_w, act.y, down_b, none, 0.0, x1.y, false, true);
    return py::make_tuple(x3.rc, x3.what, x3.y, st.state.C, st.state.n, st.state.m);
}

// LayerNorm of each of `groups` column blocks of the rows of x; the status says if the kernel does not take the layout
py::tuple layer_norm(const Tensor &x, const Tensor &weight, const Tensor &bias, double eps, int64_t groups) {
    need_cuda(x); need_cuda(weight); need_cuda(bias);
    const int64_t width = x.size(-1);
    need(groups > 0 && width % groups == 0, "a row must split into equal groups");
    need(weight.numel() == width && bias.numel() == width, "norm weight and bias must have one element per column");
    const Tensor xc = x.contiguous();
    const Tensor w = weight.to(xc.scalar_type()).contiguous(), b = bias.to(xc.scalar_type()).contiguous();
    const Tensor y = at::empty_like(xc);
    const int dt = dtype_code(xc);
    const int rc = unlocked([&] {
        return xlstm_layer_norm(xc.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), width ? xc.numel() / width : 0,
                                (int)groups, (int)(width / groups), (float)eps, dt, stream());
    });
    return py::make_tuple(rc, y);
}

// Gates i, f, o of the packaged sLSTM for all tokens of x [B, S, C]
py::tuple slstm_gates(const Tensor &x, const Tensor &conv_w, const OptTensor &conv_b, const std::vector<Tensor> &w,
                      const std::vector<Tensor> &b, double gate_cap) {
    need_cuda(x); need_cuda(conv_w); need_cuda(conv_b);
    need(x.dim() == 3 && w.size() == 3 && b.size() == 3, "slstm_gates takes x as [B, S, C] and three weights and biases (i, f, o)");
    const int64_t B = x.size(0), S = x.size(1), C = x.size(2), NH = w[0].size(0), K = conv_w.size(-1);
    const int dt = dtype_code(x);
    const auto type = x.scalar_type();
    need(conv_w.numel() == C * K && (!conv_b || conv_b->numel() == C), "convolution weight or bias of another size than [C,K], [C]");
    const Tensor xc = x.contiguous(), cw = conv_w.to(type).contiguous();
    const OptTensor cb = cast_contiguous(conv_b, type);
    std::vector<Tensor> keep, gates;
    const void *wp[3], *bp[3];
    void *gp[3];
    for (int k = 0; k < 3; ++k) {
        need_cuda(w[k]); need_cuda(b[k]);
        need(w[k].numel() == NH * C && b[k].numel() == NH, "gate weight or bias of another size than [NH,C], [NH]");
        keep.push_back(w[k].to(type).contiguous());
        wp[k] = keep.back().data_ptr();
        keep.push_back(b[k].to(type).contiguous());
        bp[k] = keep.back().data_ptr();
        gates.push_back(at::empty({B, S, NH}, x.options()));
        gp[k] = gates.back().data_ptr();
    }
    const int rc = unlocked([&] {
        return xlstm_slstm_gates(xc.data_ptr(), cw.data_ptr(), ptr(cb), wp, bp, gp, (int)B, (int)S, (int)C, (int)K, (int)NH,
                                 (float)gate_cap, dt, stream());
    });
    return py::make_tuple(rc, gates[0], gates[1], gates[2]);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("mlstm_step", &mlstm_step);
    m.def("mlstm_step_gated", &mlstm_step_gated);
    m.def("mlstm_chunkwise", &mlstm_chunkwise);
    m.def("linear_token", &linear_token);
    m.def("rms_norm", &rms_norm);
    m.def("add_rms_norm", &add_rms_norm);
    m.def("token_block", &token_block);
    m.def("layer_norm", &layer_norm);
    m.def("slstm_gates", &slstm_gates);
}
