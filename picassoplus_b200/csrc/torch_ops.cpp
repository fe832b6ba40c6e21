// The host path of the operators as a torch extension: argument checks, output and workspace allocation, kernel
// launches through the C ABI and the autograd nodes, without the interpreter in between.  A small mesh's step is a
// dozen launches of a few microseconds each; from Python (one autograd.Function, one ctypes call, several allocations
// and device guards per operator) the host needs 20 to 40 us per launch and sets the step's time, from here 2 to 3.
// The kernels stay in libpicasso_b200.so: this file calls the functions of include/picasso_b200.h like any C host.
//
// Autograd nodes are plain torch::autograd::Node subclasses: forward runs below the autograd dispatch keys, the node
// keeps SavedVariables (so an input overwritten between forward and backward is reported, as with the Python
// Functions), backward runs on the engine's thread without the GIL.
#include <torch/extension.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <mutex>
#include <stdexcept>
#include <string>

#include "../../include/picasso_b200.h"

namespace {

using at::Tensor;
using torch::autograd::edge_list;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

[[noreturn]] void fail(const std::string& text) { throw std::runtime_error(text); }

void call(int rc, const char* name) {
    if (rc != PB200_OK) fail(std::string(name) + " failed (" + std::to_string(rc) + "): " + pb200_last_error());
}

void check(const Tensor& t, const char* name, int64_t dims, at::ScalarType type) {
    if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor");
    if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
    if (t.dim() != dims) fail(std::string(name) + " must have dimension of " + std::to_string(dims));
    if (t.scalar_type() != type)
        fail(std::string(name) + " must have dtype " + c10::toString(type) + ", got " + c10::toString(t.scalar_type()));
}

bool misaligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) != 0; }
// The tensor-core kernels copy rows with 16-byte vector and bulk copies; a contiguous view that starts off a 16-byte
// boundary (a slice of a larger tensor) is moved to fresh storage.
Tensor aligned(const Tensor& t) { return misaligned(t) ? t.clone() : t; }

// Everything a call needs from the current device: guard, stream, allocation.
struct Scope {
    c10::cuda::CUDAGuard guard;
    at::TensorOptions f32;
    void* stream;
    explicit Scope(const Tensor& t)
        : guard(t.device()), f32(t.options().dtype(at::kFloat).requires_grad(false)),
          stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
    Tensor floats(at::IntArrayRef shape) const { return at::empty(shape, f32); }
    Tensor bytes(size_t n) const { return at::empty({(int64_t)(n > 0 ? n : 1)}, f32.dtype(at::kByte)); }
};

const float* fp(const Tensor& t) { return t.defined() ? static_cast<const float*>(t.data_ptr()) : nullptr; }
float* fpm(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
const int32_t* ip(const Tensor& t) { return t.defined() ? static_cast<const int32_t*>(t.data_ptr()) : nullptr; }
Tensor or_undefined(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
SavedVariable keep(const Tensor& t) { return SavedVariable(t, /*is_output=*/false); }

template <typename N, typename... Inputs>
std::shared_ptr<N> node_for(const Inputs&... inputs) {
    auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(inputs...));
    return node;
}

// ------------------------------------------------------------------------------------------------- raw operators
Tensor v2f_forward(const Scope& s, const Tensor& input, const Tensor& filter, const Tensor& face) {
    const int64_t Nv = input.size(0), C = input.size(1), r = filter.size(2), Nf = face.size(0);
    Tensor out = s.floats({Nf, C * r});
    call(pb200_vertex2facet_forward(Nf, Nv, (int)C, (int)r, fp(input), fp(filter), ip(face), fpm(out), s.stream),
         "pb200_vertex2facet_forward");
    return out;
}

void v2f_backward(const Scope& s, const Tensor& g, const Tensor& input, const Tensor& filter, const Tensor& face,
                  const Tensor& rowptr, const Tensor& entries, Tensor& gin, Tensor& gf) {
    const int64_t Nv = input.size(0), C = input.size(1), r = filter.size(2), Nf = face.size(0);
    gin = s.floats({Nv, C});
    gf = s.floats({3, C, r});
    const size_t nb = pb200_vertex2facet_backward_workspace_bytes(Nf, Nv, (int)C, (int)r);
    Tensor ws = s.bytes(nb);
    call(pb200_vertex2facet_backward(Nf, Nv, (int)C, (int)r, fp(g), fp(input), fp(filter), ip(face), ip(rowptr), ip(entries),
                                     fpm(gin), fpm(gf), ws.data_ptr(), nb, s.stream),
         "pb200_vertex2facet_backward");
}

Tensor f2v_forward(const Scope& s, const Tensor& input, const Tensor& filter, const Tensor& coeff, const Tensor& nf_count,
                   const Tensor& rowptr, const Tensor& entries) {
    const int64_t Nf = input.size(0), C = input.size(1), K = filter.size(0), r = filter.size(2), NvOut = nf_count.size(0);
    Tensor out = s.floats({NvOut, C * r});
    const size_t nb = pb200_facet2vertex_forward_workspace_bytes(Nf, (int)C, (int)r, (int)K);
    Tensor ws = s.bytes(nb);
    call(pb200_facet2vertex_forward(Nf, NvOut, (int)C, (int)r, (int)K, fp(input), fp(filter), fp(coeff), ip(nf_count),
                                    ip(rowptr), ip(entries), fpm(out), ws.data_ptr(), nb, s.stream),
         "pb200_facet2vertex_forward");
    return out;
}

void f2v_backward(const Scope& s, const Tensor& g, const Tensor& input, const Tensor& filter, const Tensor& coeff,
                  const Tensor& face, const Tensor& nf_count, const Tensor& vt_map, Tensor& gin, Tensor& gf) {
    const int64_t Nf = input.size(0), C = input.size(1), K = filter.size(0), r = filter.size(2);
    gin = s.floats({Nf, C});
    gf = s.floats({K, C, r});
    const size_t nb = pb200_facet2vertex_backward_workspace_bytes(Nf, (int)C, (int)r, (int)K);
    Tensor ws = s.bytes(nb);
    call(pb200_facet2vertex_backward(Nf, vt_map.size(0), nf_count.size(0), (int)C, (int)r, (int)K, fp(g), fp(input), fp(filter),
                                     fp(coeff), ip(face), ip(nf_count), ip(vt_map), fpm(gin), fpm(gf), ws.data_ptr(), nb,
                                     s.stream),
         "pb200_facet2vertex_backward");
}

Tensor f2f_forward(const Scope& s, const Tensor& input, const Tensor& filter, const Tensor& bary, const Tensor& cum,
                   int precision) {
    const int64_t NiK = input.size(0), Cin = input.size(1), Cout = filter.size(0), F = filter.size(2), Nf = cum.size(0);
    Tensor out = s.floats({Nf, Cout});
    const size_t nb = pb200_facet2facet_forward_workspace_bytes(Nf, NiK, (int)Cin, (int)Cout, (int)F, precision);
    Tensor ws = s.bytes(nb);
    call(pb200_facet2facet_forward(Nf, NiK, (int)Cin, (int)Cout, (int)F, fp(input), fp(filter), fp(bary), ip(cum), fpm(out),
                                   precision, ws.data_ptr(), nb, s.stream),
         "pb200_facet2facet_forward");
    return out;
}

Tensor f2f_one_sample_forward(const Scope& s, const Tensor& input, const Tensor& filter, const Tensor& weights,
                              const Tensor& weights_padded, int precision) {
    const int64_t Nf = input.size(0), Cin = input.size(1), Cout = filter.size(0), F = filter.size(2);
    Tensor out = s.floats({Nf, Cout});
    const size_t nb = pb200_facet2facet_one_sample_forward_workspace_bytes(Nf, (int)Cin, (int)Cout, (int)F, precision);
    Tensor ws = s.bytes(nb);
    call(pb200_facet2facet_one_sample_forward(Nf, (int)Cin, (int)Cout, (int)F, fp(input), fp(filter), fp(weights),
                                              fp(weights_padded), fpm(out), precision, ws.data_ptr(), nb, s.stream),
         "pb200_facet2facet_one_sample_forward");
    return out;
}

void f2f_backward(const Scope& s, const Tensor& g, const Tensor& input, const Tensor& filter, const Tensor& bary,
                  const Tensor& bary_padded, const Tensor& cum, int precision, Tensor& gin, Tensor& gf) {
    const int64_t NiK = input.size(0), Cin = input.size(1), Cout = filter.size(0), F = filter.size(2), Nf = cum.size(0);
    gin = s.floats({NiK, Cin});
    gf = s.floats({Cout, Cin, F});
    const size_t nb = pb200_facet2facet_backward_workspace_bytes(Nf, NiK, (int)Cin, (int)Cout, (int)F, precision);
    Tensor ws = s.bytes(nb);
    call(pb200_facet2facet_backward_padded(Nf, NiK, (int)Cin, (int)Cout, (int)F, fp(g), fp(input), fp(filter), fp(bary),
                                           fp(bary_padded), ip(cum), fpm(gin), fpm(gf), precision, ws.data_ptr(), nb, s.stream),
         "pb200_facet2facet_backward_padded");
}

// --------------------------------------------------------------------------------------------------------- checks
void check_v2f(const Tensor& input, const Tensor& filter, const Tensor& face) {
    check(input, "input", 2, at::kFloat);
    check(filter, "filter", 3, at::kFloat);
    check(face, "face", 2, at::kInt);
    if (filter.size(0) != 3 || filter.size(1) != input.size(1))
        fail("3 filters required, or input Channel size error of the filter");
    if (face.size(0) > 0 && face.size(1) != 3) fail("face must have shape (NfIn, 3)");
}

void check_f2v(const Tensor& input, const Tensor& filter, const Tensor& coeff, const Tensor& face, const Tensor& nf_count,
               const Tensor& vt_map) {
    check(input, "input", 2, at::kFloat);
    check(filter, "filter", 3, at::kFloat);
    check(coeff, "coeff", 2, at::kFloat);
    check(face, "face", 2, at::kInt);
    check(nf_count, "nf_count", 1, at::kInt);
    check(vt_map, "vt_map", 1, at::kInt);
    if (filter.size(1) != input.size(1)) fail("Input Channel size error of the filter");
    if (coeff.size(0) != input.size(0) || coeff.size(1) != filter.size(0)) fail("coeff must have shape (NfIn, filter_size)");
    if (face.size(0) != input.size(0) || (face.size(0) > 0 && face.size(1) != 3)) fail("face must have shape (NfIn, 3)");
}

void check_f2f(const Tensor& input, const Tensor& filter, const Tensor& bary) {
    check(input, "input", 2, at::kFloat);
    check(filter, "filter", 3, at::kFloat);
    check(bary, "bary_coeff", 2, at::kFloat);
    if (filter.size(1) != input.size(1)) fail("input Channel size error of the filter.");
    if (filter.size(2) > 50) fail("A maximum of 50 filters are supported in face2face convolution.");
    if (bary.size(1) != filter.size(2)) fail("Dimension of bary_coeff mismatches number of filters.");
    if (bary.size(0) != input.size(0)) fail("The shape of bary_coeff should be (NiK, Dim)).");
}

Tensor upstream(const variable_list& grads) { return grads[0].contiguous(); }

// ---------------------------------------------------------------------------------------------------------- nodes
struct V2F : Node {
    SavedVariable input, filter, face, rowptr, entries;
    variable_list apply(variable_list&& grads) override {
        variable_list out(2);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack();
        Scope s(x);
        v2f_backward(s, upstream(grads), x, filter.unpack(), face.unpack(), rowptr.unpack(), entries.unpack(), out[0], out[1]);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&input, &filter, &face, &rowptr, &entries}) v->reset_data();
    }
    std::string name() const override { return "VertexToFacetBackward"; }
};

struct F2V : Node {
    SavedVariable input, filter, coeff, face, nf_count, vt_map;
    variable_list apply(variable_list&& grads) override {
        variable_list out(2);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack();
        Scope s(x);
        f2v_backward(s, upstream(grads), x, filter.unpack(), coeff.unpack(), face.unpack(), nf_count.unpack(), vt_map.unpack(),
                     out[0], out[1]);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&input, &filter, &coeff, &face, &nf_count, &vt_map}) v->reset_data();
    }
    std::string name() const override { return "FacetToVertexBackward"; }
};

// facet2facet, general (cum = running sample count) or with one sample per face (cum = 1, 2, ..., Nf)
struct F2F : Node {
    SavedVariable input, filter, bary, bary_padded, cum;
    int precision = 0;
    variable_list apply(variable_list&& grads) override {
        variable_list out(2);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack();
        Scope s(x);
        f2f_backward(s, aligned(upstream(grads)), aligned(x), filter.unpack(), aligned(bary.unpack()), bary_padded.unpack(),
                     cum.unpack(), precision, out[0], out[1]);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&input, &filter, &bary, &bary_padded, &cum}) v->reset_data();
    }
    std::string name() const override { return "FacetToFacetBackward"; }
};

// vertex2facet -> facet2facet with one row per face -> facet2vertex
struct ConvBlock : Node {
    SavedVariable x, corners, spatial, filter, filter_out, y, z, weights, weights_padded, one_each, face, coeff, nf_count, vt_map,
        rowptr, entries;
    int precision = 0;
    variable_list apply(variable_list&& grads) override {
        variable_list out(4);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor xin = x.unpack(), sp = spatial.unpack(), fc = face.unpack(), eye = corners.unpack();
        Scope s(xin);
        Tensor gz, gy, gs;
        f2v_backward(s, upstream(grads), z.unpack(), filter_out.unpack(), coeff.unpack(), fc, nf_count.unpack(), vt_map.unpack(),
                     gz, out[3]);
        f2f_backward(s, gz, y.unpack(), filter.unpack(), weights.unpack(), weights_padded.unpack(), one_each.unpack(), precision,
                     gy, out[2]);
        gz.reset();
        v2f_backward(s, gy, xin, sp, fc, rowptr.unpack(), entries.unpack(), out[0], gs);
        if (task_should_compute_output(1)) {
            const int64_t K = eye.size(1), C = sp.size(1);
            out[1] = s.floats({K, C});
            call(pb200_corner_filter_backward((int)K, (int)C, fp(eye), fp(gs), fpm(out[1]), s.stream),
                 "pb200_corner_filter_backward");
        }
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&x, &corners, &spatial, &filter, &filter_out, &y, &z, &weights, &weights_padded, &one_each, &face,
                                 &coeff, &nf_count, &vt_map, &rowptr, &entries})
            v->reset_data();
    }
    std::string name() const override { return "ConvBlockBackward"; }
};

// ---------------------------------------------------------------------------------------------- differentiable calls
// rowptr / entries: the vertex CSR of `face` over the input vertices; needed (and looked at) only when a gradient is
Tensor vertex2facet(const Tensor& input, const Tensor& filter, const Tensor& face, const OptTensor& rowptr,
                    const OptTensor& entries) {
    check_v2f(input, filter, face);
    std::shared_ptr<V2F> node;
    if (torch::autograd::compute_requires_grad(input, filter)) node = node_for<V2F>(input, filter);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        out = v2f_forward(s, input, filter, face);
    }
    if (node) {
        node->input = keep(input);
        node->filter = keep(filter);
        node->face = keep(face);
        node->rowptr = keep(or_undefined(rowptr));
        node->entries = keep(or_undefined(entries));
        torch::autograd::set_history(out, node);
    }
    return out;
}

Tensor facet2vertex(const Tensor& input, const Tensor& filter, const Tensor& coeff, const Tensor& face, const Tensor& nf_count,
                    const Tensor& vt_map, const Tensor& rowptr, const Tensor& entries) {
    check_f2v(input, filter, coeff, face, nf_count, vt_map);
    std::shared_ptr<F2V> node;
    if (torch::autograd::compute_requires_grad(input, filter)) node = node_for<F2V>(input, filter);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        out = f2v_forward(s, input, filter, coeff, nf_count, rowptr, entries);
    }
    if (node) {
        node->input = keep(input);
        node->filter = keep(filter);
        node->coeff = keep(coeff);
        node->face = keep(face);
        node->nf_count = keep(nf_count);
        node->vt_map = keep(vt_map);
        torch::autograd::set_history(out, node);
    }
    return out;
}

Tensor facet2facet(const Tensor& input, const Tensor& filter, const Tensor& bary, const Tensor& cum, int precision) {
    check_f2f(input, filter, bary);
    check(cum, "num_texture", 1, at::kInt);
    std::shared_ptr<F2F> node;
    if (torch::autograd::compute_requires_grad(input, filter)) node = node_for<F2F>(input, filter);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        out = f2f_forward(s, aligned(input), filter, bary, cum, precision);
    }
    if (node) {
        node->input = keep(input);
        node->filter = keep(filter);
        node->bary = keep(bary);
        node->bary_padded = keep(Tensor());
        node->cum = keep(cum);
        node->precision = precision;
        torch::autograd::set_history(out, node);
    }
    return out;
}

void check_weights(const Tensor& weights, const OptTensor& padded, int64_t Nf, int64_t F) {
    check(weights, "weights", 2, at::kFloat);
    if (weights.size(0) != Nf || weights.size(1) != F) fail("weights must have shape (NfIn, number of filters)");
    if (padded.has_value() && (padded->dim() != 2 || padded->size(0) != Nf || padded->size(1) != pb200_padded_row_floats((int)F)))
        fail("weights_padded must have shape (NfIn, padded row length)");
}

void check_shared_rows(const Tensor& rows, const Tensor& filter, const Tensor& weights, const OptTensor& padded) {
    check(rows, "input", 2, at::kFloat);
    check(filter, "filter", 3, at::kFloat);
    if (filter.size(1) != rows.size(1)) fail("input Channel size error of the filter.");
    if (filter.size(2) > 50) fail("A maximum of 50 filters are supported in face2face convolution.");
    check_weights(weights, padded, rows.size(0), filter.size(2));
}

Tensor facet2facet_shared_rows(const Tensor& rows_in, const Tensor& filter_in, const Tensor& weights, const Tensor& one_each,
                               const OptTensor& weights_padded, int precision) {
    const Tensor rows = rows_in.contiguous(), filter = filter_in.contiguous();
    check_shared_rows(rows, filter, weights, weights_padded);
    std::shared_ptr<F2F> node;
    if (torch::autograd::compute_requires_grad(rows, filter)) node = node_for<F2F>(rows, filter);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(rows);
        out = f2f_one_sample_forward(s, aligned(rows), filter, aligned(weights), or_undefined(weights_padded), precision);
    }
    if (node) {
        node->input = keep(rows);
        node->filter = keep(filter);
        node->bary = keep(weights);
        node->bary_padded = keep(or_undefined(weights_padded));
        node->cum = keep(one_each);
        node->precision = precision;
        torch::autograd::set_history(out, node);
    }
    return out;
}

Tensor conv_block(const Tensor& x, const Tensor& wv_in, const Tensor& wf_in, const Tensor& wo, const Tensor& corners_in,
                  const Tensor& face, const Tensor& weights, const Tensor& one_each, const OptTensor& weights_padded,
                  const Tensor& coeff, const Tensor& nf_count, const Tensor& vt_map, const OptTensor& v_rowptr,
                  const OptTensor& v_entries, const Tensor& f_rowptr, const Tensor& f_entries, int precision) {
    std::shared_ptr<ConvBlock> node;
    if (torch::autograd::compute_requires_grad(x, wv_in, wf_in, wo)) node = node_for<ConvBlock>(x, wv_in, wf_in, wo);
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor wv = wv_in.contiguous(), wf = wf_in.contiguous(), corners = corners_in.contiguous();
    check(x, "input", 2, at::kFloat);
    check(face, "face", 2, at::kInt);
    check(corners, "sh_eye", 2, at::kFloat);
    check(wv, "Wv", 2, at::kFloat);
    const int64_t C = x.size(1), K = corners.size(1);
    if (corners.size(0) != 3 || wv.size(0) != K || wv.size(1) != C) fail("Wv must have shape (number of bases, in_channels)");
    if (face.size(0) > 0 && face.size(1) != 3) fail("face must have shape (NfIn, 3)");
    Scope s(x);
    const Tensor w = aligned(weights);
    Tensor spatial = s.floats({3, C, 1});
    call(pb200_corner_filter((int)K, (int)C, fp(corners), fp(wv), fpm(spatial), s.stream), "pb200_corner_filter");
    Tensor y = v2f_forward(s, x, spatial, face);
    check_shared_rows(y, wf, w, weights_padded);
    Tensor z = f2f_one_sample_forward(s, y, wf, w, or_undefined(weights_padded), precision);
    check_f2v(z, wo, coeff, face, nf_count, vt_map);
    Tensor out = f2v_forward(s, z, wo, coeff, nf_count, f_rowptr, f_entries);
    if (node) {
        node->x = keep(x);
        node->corners = keep(corners);
        node->spatial = keep(spatial);
        node->filter = keep(wf);
        node->filter_out = keep(wo);
        node->y = keep(y);
        node->z = keep(z);
        node->weights = keep(w);
        node->weights_padded = keep(or_undefined(weights_padded));
        node->one_each = keep(one_each);
        node->face = keep(face);
        node->coeff = keep(coeff);
        node->nf_count = keep(nf_count);
        node->vt_map = keep(vt_map);
        node->rowptr = keep(or_undefined(v_rowptr));
        node->entries = keep(or_undefined(v_entries));
        node->precision = precision;
        torch::autograd::set_history(out, node);
    }
    return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.doc() = "Native host path of picassoplus_b200 (see torch_ops.cpp).";
    m.def("vertex2facet", &vertex2facet);
    m.def("facet2vertex", &facet2vertex);
    m.def("facet2facet", &facet2facet);
    m.def("facet2facet_shared_rows", &facet2facet_shared_rows);
    m.def("conv_block", &conv_block);
}
