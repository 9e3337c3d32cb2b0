// The host side of the calls that training and decoding make most: views, output tensors, device
// and stream look-ups and the call into the C ABI, in one step out of Python. The same work through
// ctypes costs several times the kernels of a small call (q/k/v with LoRA at 810 tokens: 16 launches
// of 86 us GPU time in all took 668 us from Python). Argument checks that need the quant state, and the
// autograd functions, stay in Python; nothing is kept here between calls.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/utils/pybind.h>

#include <optional>
#include <utility>
#include <vector>

#include "../../include/nf4b200.h"

namespace py = pybind11;
using at::Tensor;
using Opt = std::optional<Tensor>;
using Opts = std::vector<Opt>;

namespace {

constexpr int64_t RANK = 16;
constexpr int MAX_GROUP = 4, MAX_BATCH = 8;

// A non-zero status becomes the package's own exception. (The calls run without the interpreter lock.)
void check(int rc) {
    if (rc == 0) return;
    const py::gil_scoped_acquire lock;
    py::module_::import("hackaton_b200._lib").attr("check")(rc);
}

void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

const void* ptr(const Opt& t) { return t.has_value() ? t->const_data_ptr() : nullptr; }

const nf4b200_weight* weight(int64_t address) { return reinterpret_cast<const nf4b200_weight*>(address); }

// Where the tensors of a weight lie and how often each has been written (inference tensors do not count
// that), in a form that compares as a whole.
py::bytes stamps(const Tensor& packed, const Tensor& absmax, const Tensor& code, const Opt& absmax2, const Opt& code2,
                 const Opt& offset) {
    const Tensor none;
    const Tensor* all[] = {&packed, &absmax, &code, absmax2 ? &*absmax2 : &none, code2 ? &*code2 : &none,
                           offset ? &*offset : &none};
    int64_t r[12];
    int n = 0;
    for (const Tensor* t : all) {
        r[n++] = t->defined() ? reinterpret_cast<int64_t>(t->const_data_ptr()) : 0;
        r[n++] = t->defined() && !t->is_inference() ? t->_version() : -1;
    }
    return py::bytes(reinterpret_cast<const char*>(r), sizeof r);
}

// [..., cols] -> 2-D view with contiguous rows, 16-byte aligned and 8 elements apart (copied only if the
// layout forces it; columns that are no eights stay where they are).
Tensor rows_view(const Tensor& t, int64_t cols) {
    const auto aligned = [](const Tensor& v) { return (reinterpret_cast<uintptr_t>(v.const_data_ptr()) & 15) == 0; };
    Tensor v = t.dim() == 2 && t.size(1) == cols ? t : t.reshape({-1, cols});
    if (v.stride(1) == 1 && v.stride(0) % 8 == 0 && aligned(v) && v.stride(0) >= cols) return v;
    v = v.contiguous();
    // (a tensor that counts as contiguous keeps its address, and a single row its stride)
    if (cols % 8 == 0 && (!aligned(v) || v.stride(0) != cols)) v = v.clone(at::MemoryFormat::Contiguous);
    return v;
}

// Output with the leading dimensions of `like` and `cols` columns.
Tensor output(const Tensor& like, int64_t cols, at::ScalarType type = at::kHalf) {
    at::DimVector shape(like.sizes().begin(), like.sizes().end());
    shape.back() = cols;
    return at::empty(shape, like.options().dtype(type).memory_format(c10::nullopt));
}

// Scratch of one call on the current stream (see hackaton_b200.nf4.scratch_bytes): the allocator hands it
// out again only behind the work of that stream.
struct Scratch {
    Tensor buffer;
    Scratch(int64_t bytes, const Tensor& like) {
        if (bytes > 0) buffer = at::empty({bytes}, like.options().dtype(at::kByte).memory_format(c10::nullopt));
    }
    void* get() const { return buffer.defined() ? buffer.data_ptr() : nullptr; }
};

// What a kernel reads besides its input has to be there: a rank-16 pair of `rows` and `cols`, a bias.
void check_pair(const Opt& a, int64_t rows, const Opt& b, int64_t cols) {
    TORCH_CHECK(a.has_value() == b.has_value() &&
                    (!a.has_value() || (a->numel() >= rows * RANK && b->numel() >= cols * RANK)),
                "rank-16 pair does not reach over ", rows, " rows and ", cols, " columns");
}

void check_bias(const Opt& bias, int64_t cols) {
    TORCH_CHECK(!bias.has_value() || bias->numel() >= cols, "bias of ", bias->numel(), " values for ", cols, " outputs");
}

Opt half(const Opt& t) {
    if (!t.has_value()) return t;
    return t->to(at::kHalf).contiguous();
}

Tensor linear_fwd(int64_t w, const Tensor& x, const Opt& bias, const Opt& xa, const Opt& lora_b, int64_t ws_bytes) {
    const nf4b200_weight* q = weight(w);
    if (x.numel() == 0) return output(x, q->n_rows);
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor x2 = rows_view(x, q->n_cols);
    check_pair(xa, x2.size(0), lora_b, q->n_rows);
    check_bias(bias, q->n_rows);
    Tensor y = output(x, q->n_rows);
    const Opt b = half(bias);
    const Scratch ws(ws_bytes, x);
    check(nf4b200_linear_fwd(q, x2.const_data_ptr(), x2.size(0), x2.stride(0), ptr(b), ptr(xa), ptr(lora_b),
                             y.data_ptr(), q->n_rows, ws.get(), (size_t)ws_bytes, stream_of(x)));
    return y;
}

Tensor linear_bwd_dx(int64_t w, const Tensor& dy, const Opt& u, const Opt& lora_a, int64_t ws_bytes) {
    const nf4b200_weight* q = weight(w);
    if (dy.numel() == 0) return output(dy, q->n_cols);
    const c10::cuda::CUDAGuard guard(dy.device());
    const Tensor g2 = rows_view(dy, q->n_rows);
    check_pair(u, g2.size(0), lora_a, q->n_cols);
    Tensor dx = output(dy, q->n_cols);
    const Scratch ws(ws_bytes, dy);
    check(nf4b200_linear_bwd_dx(q, g2.const_data_ptr(), g2.size(0), g2.stride(0), ptr(u), ptr(lora_a), dx.data_ptr(),
                                q->n_cols, ws.get(), (size_t)ws_bytes, stream_of(dy)));
    return dx;
}

std::vector<Tensor> linear_fwd_group(const std::vector<int64_t>& ws_addr, const Tensor& x, const Opts& biases,
                                     const Opts& xas, const Opts& lora_bs, int64_t ws_bytes) {
    const int n = (int)ws_addr.size();
    TORCH_CHECK(n >= 1 && n <= MAX_GROUP, "a group holds 1..", MAX_GROUP, " projections, got ", n);
    std::vector<Tensor> ys;
    for (const int64_t address : ws_addr) ys.push_back(output(x, weight(address)->n_rows));
    if (x.numel() == 0) return ys;
    const c10::cuda::CUDAGuard guard(x.device());
    const nf4b200_weight* q[MAX_GROUP];
    const void *b[MAX_GROUP], *a[MAX_GROUP], *l[MAX_GROUP];
    void* y[MAX_GROUP];
    int64_t ld[MAX_GROUP];
    Opts keep;
    const Tensor x2 = rows_view(x, weight(ws_addr[0])->n_cols);
    for (int i = 0; i < n; ++i) {
        q[i] = weight(ws_addr[i]);
        check_pair(xas[i], x2.size(0), lora_bs[i], q[i]->n_rows);
        check_bias(biases[i], q[i]->n_rows);
        keep.push_back(half(biases[i]));
        b[i] = ptr(keep.back());
        a[i] = ptr(xas[i]);
        l[i] = ptr(lora_bs[i]);
        y[i] = ys[i].data_ptr();
        ld[i] = q[i]->n_rows;
    }
    const Scratch ws(ws_bytes, x);
    check(nf4b200_linear_fwd_group(n, q, x2.const_data_ptr(), x2.size(0), x2.stride(0), b, a, l, y, ld,
                                   ws.get(), (size_t)ws_bytes, stream_of(x)));
    return ys;
}

Tensor linear_bwd_dx_group(const std::vector<int64_t>& ws_addr, const std::vector<Tensor>& grads, const Opts& us,
                           const Opts& lora_as, int64_t ws_bytes) {
    const int n = (int)ws_addr.size();
    TORCH_CHECK(n >= 1 && n <= MAX_GROUP && (int)grads.size() == n, "a group holds 1..", MAX_GROUP, " projections");
    if (grads[0].numel() == 0) return output(grads[0], weight(ws_addr[0])->n_cols);
    const c10::cuda::CUDAGuard guard(grads[0].device());
    const nf4b200_weight* q[MAX_GROUP];
    const void *g[MAX_GROUP], *u[MAX_GROUP], *a[MAX_GROUP];
    int64_t ld[MAX_GROUP];
    std::vector<Tensor> keep;
    for (int i = 0; i < n; ++i) {
        q[i] = weight(ws_addr[i]);
        keep.push_back(rows_view(grads[i], q[i]->n_rows));
        g[i] = keep.back().const_data_ptr();
        ld[i] = keep.back().stride(0);
        TORCH_CHECK(keep.back().size(0) == keep[0].size(0), "gradients differ in their number of rows");
        check_pair(us[i], keep[0].size(0), lora_as[i], q[i]->n_cols);
        u[i] = ptr(us[i]);
        a[i] = ptr(lora_as[i]);
    }
    const int64_t m = keep[0].size(0), cols = q[0]->n_cols;
    Tensor dx = output(grads[0], cols);
    const Scratch ws(ws_bytes, dx);
    check(nf4b200_linear_bwd_dx_group(n, q, g, m, ld, u, a, dx.data_ptr(), cols, ws.get(), (size_t)ws_bytes, stream_of(dx)));
    return dx;
}

// A LoRA factor as the side kernel reads it: contiguous, 16-byte aligned fp32 or fp16.
Tensor factor(const Tensor& t) {
    Tensor p = t.detach();
    if (p.scalar_type() != at::kFloat && p.scalar_type() != at::kHalf) p = p.to(at::kHalf);
    p = p.contiguous();
    return (reinterpret_cast<uintptr_t>(p.const_data_ptr()) & 15) == 0 ? p : p.clone();
}

// (products, p16s, b16s, b16ts): see hackaton_b200.lora.lora_side.
std::tuple<std::vector<Tensor>, std::vector<Tensor>, std::vector<Tensor>, Opts>
lora_side(const std::vector<Tensor>& inputs, const std::vector<Tensor>& ps, const std::vector<double>& scalings,
          const std::vector<Tensor>& bs, bool transpose, const Opt& zero) {
    const int n = (int)inputs.size();
    TORCH_CHECK(n >= 1 && n <= MAX_BATCH && (int)ps.size() == n && (int)scalings.size() == n &&
                (bs.empty() || (int)bs.size() == n), "lora_side: 1..", MAX_BATCH, " adapters, one factor each");
    const c10::cuda::CUDAGuard guard(inputs[0].device());
    const auto options = inputs[0].options().dtype(at::kHalf);
    nf4b200_lora_item items[MAX_BATCH] = {};
    std::vector<Tensor> keep, products, p16s, b16s;
    Opts b16ts;
    int64_t m = -1;
    bool whole = true;   // every input in whole 16-byte pieces, as the side kernel reads it
    for (int i = 0; i < n; ++i) {
        const int64_t c = inputs[i].size(-1);
        const Tensor i2 = rows_view(inputs[i], c), p = factor(ps[i]);
        TORCH_CHECK(p.dim() == 2 && p.size(0) == RANK && p.size(1) == c, "lora_side: factor ", p.sizes(), " for ", c,
                    " columns");
        if (m < 0) m = i2.size(0);
        TORCH_CHECK(i2.size(0) == m, "lora_side: inputs differ in their number of rows");
        nf4b200_lora_item& it = items[i];
        it.in = i2.const_data_ptr(); it.c = c; it.ld_in = i2.stride(0);
        whole = whole && c % 8 == 0 && it.ld_in % 8 == 0 && (reinterpret_cast<uintptr_t>(it.in) & 15) == 0;
        it.p = p.const_data_ptr(); it.p_f32 = p.scalar_type() == at::kFloat;
        it.scaling = (float)scalings[i];
        products.push_back(at::empty({m, RANK}, options));
        it.out = products.back().data_ptr();
        p16s.push_back(it.p_f32 ? at::empty({RANK, c}, options) : p);
        it.p16 = it.p_f32 ? p16s.back().data_ptr() : nullptr;
        keep.push_back(i2);
        keep.push_back(p);
        if (bs.empty()) continue;
        const Tensor b = factor(bs[i]);
        TORCH_CHECK(b.dim() == 2 && b.size(1) == RANK, "lora_side: second factor ", b.sizes());
        const int64_t rows = b.size(0);
        it.b = b.const_data_ptr(); it.n = rows; it.b_f32 = b.scalar_type() == at::kFloat;
        b16s.push_back(it.b_f32 ? at::empty({rows, RANK}, options) : b);
        it.b16 = it.b_f32 ? b16s.back().data_ptr() : nullptr;
        b16ts.push_back(transpose ? Opt(at::empty({RANK, rows}, options)) : Opt());
        it.b16t = transpose ? b16ts.back()->data_ptr() : nullptr;
        keep.push_back(b);
    }
    if (m == 0 || !whole) {   // nothing to multiply, or columns that are not eights: copies and zeros by torch
        for (int i = 0; i < n; ++i) {
            if (items[i].p_f32) p16s[i].copy_(ps[i].detach());
            if (m > 0)
                check(nf4b200_lora_down(items[i].in, m, items[i].c, items[i].ld_in, p16s[i].const_data_ptr(),
                                        items[i].c, 1, items[i].scaling, items[i].out, stream_of(inputs[0])));
            if (bs.empty()) continue;
            if (items[i].b_f32) b16s[i].copy_(bs[i].detach());
            if (transpose) b16ts[i]->copy_(bs[i].detach().t());
        }
        if (zero.has_value()) zero->zero_();
    } else {
        check(nf4b200_lora_side(n, items, m, zero.has_value() ? zero->data_ptr() : nullptr,
                                zero.has_value() ? (size_t)zero->numel() * 4 : 0, stream_of(inputs[0])));
    }
    return {products, p16s, b16s, b16ts};
}

int64_t grad_piece(int64_t c) { return (c * RANK + 63) / 64 * 64; }   // 256-byte aligned pieces

// Adds the gradients zᵀ . s to pieces of the zeroed buffer `flat`, [16, C] or [C, 16] each.
std::vector<Tensor> lora_grad_batch(const std::vector<Tensor>& zs, const std::vector<Tensor>& ss,
                                    const std::vector<bool>& rank_major, const Tensor& flat) {
    const int n = (int)zs.size();
    TORCH_CHECK(n >= 1 && n <= MAX_BATCH && (int)ss.size() == n && (int)rank_major.size() == n,
                "lora_grad_batch: 1..", MAX_BATCH, " problems");
    const c10::cuda::CUDAGuard guard(zs[0].device());
    const void *z[MAX_BATCH], *s[MAX_BATCH];
    float* out[MAX_BATCH];
    int64_t m[MAX_BATCH], c[MAX_BATCH], ld[MAX_BATCH], sr[MAX_BATCH], sc[MAX_BATCH];
    std::vector<Tensor> keep, outs;
    int64_t at = 0;
    for (int i = 0; i < n; ++i) {
        c[i] = zs[i].size(-1);
        keep.push_back(rows_view(zs[i], c[i]));
        z[i] = keep.back().const_data_ptr();
        m[i] = keep.back().size(0);
        ld[i] = keep.back().stride(0);
        s[i] = ss[i].const_data_ptr();
        const bool rm = rank_major[i];
        TORCH_CHECK(at + c[i] * RANK <= flat.numel(), "lora_grad_batch: buffer too small");
        outs.push_back(rm ? flat.as_strided({RANK, c[i]}, {c[i], 1}, flat.storage_offset() + at)
                          : flat.as_strided({c[i], RANK}, {RANK, 1}, flat.storage_offset() + at));
        out[i] = static_cast<float*>(outs.back().data_ptr());
        sr[i] = rm ? c[i] : 1;
        sc[i] = rm ? 1 : RANK;
        at += grad_piece(c[i]);
    }
    if (m[0] > 0)
        check(nf4b200_lora_grad_batch(n, z, m, c, ld, s, out, sr, sc, stream_of(zs[0])));
    return outs;
}

int dtype_code(at::ScalarType t) { return t == at::kHalf ? NF4B200_F16 : NF4B200_F32; }

// (normalised rows, 1/rms, sum or None)
std::tuple<Tensor, Tensor, Opt> rmsnorm_fwd(const Tensor& x2, const Opt& delta2, const Tensor& weight, double eps,
                                            bool to_half) {
    const c10::cuda::CUDAGuard guard(x2.device());
    const int64_t rows = x2.size(0), hidden = x2.size(1);
    Tensor out = at::empty({rows, hidden}, x2.options().dtype(to_half ? at::kHalf : at::kFloat));
    Tensor rstd = at::empty({rows}, x2.options().dtype(at::kFloat));
    Opt total;
    if (delta2.has_value()) total = at::empty_like(x2);
    check(nf4b200_rmsnorm_fwd(x2.const_data_ptr(), ptr(delta2), weight.const_data_ptr(),
                              total.has_value() ? total->data_ptr() : nullptr, out.data_ptr(),
                              dtype_code(out.scalar_type()), rstd.data_ptr(), rows, hidden, (float)eps, stream_of(x2)));
    return {out, rstd, total};
}

Tensor rmsnorm_bwd(const Tensor& x2, const Tensor& weight, const Tensor& rstd, const Tensor& dy2, const Opt& d_total,
                   const Opt& dx16) {
    const c10::cuda::CUDAGuard guard(x2.device());
    Tensor dx = at::empty_like(x2);
    check(nf4b200_add_rmsnorm_bwd(x2.const_data_ptr(), weight.const_data_ptr(), rstd.const_data_ptr(),
                                  dy2.const_data_ptr(), dtype_code(dy2.scalar_type()), ptr(d_total), dx.data_ptr(),
                                  dx16.has_value() ? dx16->data_ptr() : nullptr, x2.size(0), x2.size(1),
                                  stream_of(x2)));
    return dx;
}

struct Rotation {   // everything about one rotation that is not a tensor
    int64_t tokens, seq, heads, kv_heads, dim, batch_stride;
    bool padded, f32;
};

void rotate(const Rotation& r, const Tensor (&src)[3], Tensor (&dst)[3], const Tensor& cos, const Tensor& sin,
            const Tensor& b_idx, const Tensor& t_idx, bool backward) {
    check(nf4b200_qkv_rotate(src[0].const_data_ptr(), src[1].const_data_ptr(), src[2].const_data_ptr(),
                             dst[0].data_ptr(), dst[1].data_ptr(), dst[2].data_ptr(), cos.const_data_ptr(),
                             sin.const_data_ptr(), r.batch_stride, cos.stride(1), b_idx.const_data_ptr(),
                             t_idx.const_data_ptr(), r.tokens, r.seq, (int)r.heads, (int)r.kv_heads, (int)r.dim,
                             r.padded ? 1 : 0, backward ? 1 : 0, r.f32 ? NF4B200_F32 : NF4B200_F16,
                             stream_of(dst[0])));
}

// (q, k, v heads, and what the gradient needs: cos, sin, b_idx, t_idx as the kernel read them, geometry)
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Rotation>
rotate_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cos_in, const Tensor& sin_in,
           const Tensor& b_in, const Tensor& t_in, int64_t batch, int64_t seq, int64_t heads, int64_t kv_heads,
           int64_t dim, bool padded) {
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor cos = cos_in.contiguous(), sin = sin_in.contiguous();
    const Tensor b_idx = b_in.to(at::kInt).contiguous(), t_idx = t_in.to(at::kInt).contiguous();
    Rotation r = {q.size(0), seq, heads, kv_heads, dim, cos.size(0) == 1 ? 0 : cos.stride(0), padded,
                  q.scalar_type() == at::kFloat};
    const Tensor src[3] = {q.contiguous(), k.contiguous(), v.contiguous()};
    const auto options = q.options().dtype(at::kHalf);
    Tensor dst[3];
    for (auto& d : dst)   // padded: positions no token maps to stay zero
        d = padded ? at::zeros({batch, heads, seq, r.dim}, options) : at::empty({r.tokens, heads, r.dim}, options);
    rotate(r, src, dst, cos, sin, b_idx, t_idx, false);
    return {dst[0], dst[1], dst[2], cos, sin, b_idx, t_idx, r};
}

std::tuple<Tensor, Tensor, Tensor> rotate_bwd(const Tensor& gq, const Tensor& gk, const Tensor& gv, const Tensor& cos,
                                              const Tensor& sin, const Tensor& b_idx, const Tensor& t_idx,
                                              const Rotation& r) {
    const c10::cuda::CUDAGuard guard(gq.device());
    const Tensor src[3] = {gq.to(at::kHalf).contiguous(), gk.to(at::kHalf).contiguous(),
                           gv.to(at::kHalf).contiguous()};
    const auto options = gq.options().dtype(r.f32 ? at::kFloat : at::kHalf);
    Tensor dst[3];
    for (int i = 0; i < 3; ++i) dst[i] = at::empty({r.tokens, (i == 0 ? r.heads : r.kv_heads) * r.dim}, options);
    rotate(r, src, dst, cos, sin, b_idx, t_idx, true);
    return {dst[0], dst[1], dst[2]};
}

}  // namespace

// What the module was compiled against; the build looks for the text in the file.
#ifndef NF4B200_HOST_TARGET
#define NF4B200_HOST_TARGET "unknown"
#endif
const char BUILT_FOR[] = "built for " NF4B200_HOST_TARGET ";";

PYBIND11_MODULE(_host, m) {
    m.attr("built_for") = py::str(BUILT_FOR + sizeof "built for " - 1, sizeof NF4B200_HOST_TARGET - 1);
    py::class_<Rotation>(m, "Rotation");
    m.def("stamps", &stamps);
    // An allocation or a launch can block (cudaMalloc, a full launch queue): other Python threads go on.
    using unlocked = py::call_guard<py::gil_scoped_release>;
    m.def("linear_fwd", &linear_fwd, unlocked());
    m.def("linear_bwd_dx", &linear_bwd_dx, unlocked());
    m.def("linear_fwd_group", &linear_fwd_group, unlocked());
    m.def("linear_bwd_dx_group", &linear_bwd_dx_group, unlocked());
    m.def("lora_side", &lora_side, unlocked());
    m.def("lora_grad_batch", &lora_grad_batch, unlocked());
    m.def("rmsnorm_fwd", &rmsnorm_fwd, unlocked());
    m.def("rmsnorm_bwd", &rmsnorm_bwd, unlocked());
    m.def("rotate_fwd", &rotate_fwd, unlocked());
    m.def("rotate_bwd", &rotate_bwd, unlocked());
}
