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

#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/Event.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <array>
#include <list>
#include <mutex>
#include <stdexcept>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

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

// Everything a call needs from the current device: guard, stream, allocation.  Autocast stays out: AutoDispatchBelow... leaves its
// keys on, and a product that torch rounds to half precision under it would come back as half the bytes that the kernels behind
// it read and write.  The kernels choose their operands' precision themselves.
thread_local c10::DeviceIndex call_device = -1;              // of the innermost Scope
// scratch memory of a call: back to the allocator, for work behind it on the call's stream, when it goes out of scope
struct Workspace {
    c10::DataPtr memory;
    void* data_ptr() const { return memory.get(); }
};
struct Scope {
    c10::cuda::CUDAGuard guard;
    const c10::DeviceIndex outer = std::exchange(call_device, guard.current_device().index());
    c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::DispatchKey::AutocastCUDA};
    at::TensorOptions f32;
    void* stream;
    explicit Scope(const Tensor& t)
        : guard(t.device()), f32(t.options().dtype(at::kFloat).requires_grad(false)),
          stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
    ~Scope() { call_device = outer; }
    // Straight from torch's allocator, past the dispatcher: a pass makes a dozen of them and more, 1.7 us each through at::empty
    // (a training step of one shape of 642 vertices 150 -> 140 us, of an encoder on two of 162 1 020 -> 965)
    Tensor floats(at::IntArrayRef shape) const { return empty(shape, at::kFloat); }
    Tensor ints(at::IntArrayRef shape) const { return empty(shape, at::kInt); }
    Workspace bytes(size_t n) const { return Workspace{c10::cuda::CUDACachingAllocator::get()->allocate(n > 0 ? n : 1)}; }

private:
    Tensor empty(at::IntArrayRef shape, at::ScalarType type) const {
        return Tensor(at::detail::empty_cuda(shape, type, c10::Device(c10::kCUDA, guard.current_device().index()), std::nullopt));
    }
};

// Addresses for a kernel: whatever way a tensor came in, one of another type, device or layout goes no further
void* address(const Tensor& t, at::ScalarType type) {
    if (!t.defined()) return nullptr;
    if (t.scalar_type() != type || !t.is_cuda() || t.get_device() != call_device || !t.is_contiguous())
        fail(std::string("expected a contiguous ") + c10::toString(type) + " tensor on the call's CUDA device, got " +
             c10::toString(t.scalar_type()) + " on " + t.device().str());
    return t.data_ptr();
}
const float* fp(const Tensor& t) { return static_cast<const float*>(address(t, at::kFloat)); }
float* fpm(const Tensor& t) { return static_cast<float*>(address(t, at::kFloat)); }
const int32_t* ip(const Tensor& t) { return static_cast<const int32_t*>(address(t, at::kInt)); }
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

// what a backward pass says of an adjacency that could not be made (topology.for_backward)
constexpr const char* BAD_FACE = "face holds an index outside the vertex range";
constexpr const char* BAD_PAIR = "nn_index holds an index outside the input points";

void v2f_backward(const Scope& s, const Tensor& g, const Tensor& input, const Tensor& filter, const Tensor& face,
                  const Tensor& rowptr, const Tensor& entries, Tensor& gin, Tensor& gf) {
    const int64_t Nv = input.size(0), C = input.size(1), r = filter.size(2), Nf = face.size(0);
    if (!rowptr.defined()) fail(BAD_FACE);
    gin = s.floats({Nv, C});
    gf = s.floats({3, C, r});
    const size_t nb = pb200_vertex2facet_backward_workspace_bytes(Nf, Nv, (int)C, (int)r);
    const Workspace ws = s.bytes(nb);
    call(pb200_vertex2facet_backward(Nf, Nv, (int)C, (int)r, fp(g), fp(input), fp(filter), ip(face), ip(rowptr), ip(entries),
                                     fpm(gin), fpm(gf), ws.data_ptr(), nb, s.stream),
         "pb200_vertex2facet_backward");
}

Tensor f2v_forward(const Scope& s, const Tensor& input, const Tensor& filter, const Tensor& coeff, const Tensor& nf_count,
                   const Tensor& rowptr, const Tensor& entries) {
    const int64_t Nf = input.size(0), C = input.size(1), K = filter.size(0), r = filter.size(2), NvOut = nf_count.size(0);
    Tensor out = s.floats({NvOut, C * r});
    const size_t nb = pb200_facet2vertex_forward_workspace_bytes(Nf, (int)C, (int)r, (int)K);
    const Workspace ws = s.bytes(nb);
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
    const Workspace ws = s.bytes(nb);
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
    const Workspace ws = s.bytes(nb);
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
    const Workspace ws = s.bytes(nb);
    call(pb200_facet2facet_one_sample_forward(Nf, (int)Cin, (int)Cout, (int)F, fp(input), fp(filter), fp(weights),
                                              fp(weights_padded), fpm(out), precision, ws.data_ptr(), nb, s.stream),
         "pb200_facet2facet_one_sample_forward");
    return out;
}

void f2f_backward(const Scope& s, const Tensor& g, const Tensor& input, const Tensor& filter, const Tensor& bary,
                  const Tensor& bary_padded, const Tensor& cum, int precision, Tensor& gin, Tensor& gf, bool want_gin) {
    const int64_t NiK = input.size(0), Cin = input.size(1), Cout = filter.size(0), F = filter.size(2), Nf = cum.size(0);
    if (want_gin) gin = s.floats({NiK, Cin});
    gf = s.floats({Cout, Cin, F});
    const size_t nb = pb200_facet2facet_backward_workspace_bytes(Nf, NiK, (int)Cin, (int)Cout, (int)F, precision);
    const Workspace ws = s.bytes(nb);
    if (want_gin)
        call(pb200_facet2facet_backward_padded(Nf, NiK, (int)Cin, (int)Cout, (int)F, fp(g), fp(input), fp(filter), fp(bary),
                                               fp(bary_padded), ip(cum), fpm(gin), fpm(gf), precision, ws.data_ptr(), nb, s.stream),
             "pb200_facet2facet_backward_padded");
    else
        call(pb200_facet2facet_filter_gradient(Nf, NiK, (int)Cin, (int)Cout, (int)F, fp(g), fp(input), fp(bary), fp(bary_padded), ip(cum),
                                               fpm(gf), precision, ws.data_ptr(), nb, s.stream),
             "pb200_facet2facet_filter_gradient");
}

// one sample per face (one_each = 1, 2, ..., Nf)
void f2f_one_sample_backward(const Scope& s, const Tensor& g, const Tensor& input, const Tensor& filter, const Tensor& weights,
                             const Tensor& weights_padded, const Tensor& one_each, int precision, Tensor& gin, Tensor& gf) {
    const int64_t Nf = input.size(0), Cin = input.size(1), Cout = filter.size(0), F = filter.size(2);
    gin = s.floats({Nf, Cin});
    gf = s.floats({Cout, Cin, F});
    const size_t nb = pb200_facet2facet_backward_workspace_bytes(Nf, Nf, (int)Cin, (int)Cout, (int)F, precision);
    const Workspace ws = s.bytes(nb);
    call(pb200_facet2facet_one_sample_backward(Nf, (int)Cin, (int)Cout, (int)F, fp(g), fp(input), fp(filter), fp(weights),
                                               fp(weights_padded), ip(one_each), fpm(gin), fpm(gf), precision, ws.data_ptr(), nb, s.stream),
         "pb200_facet2facet_one_sample_backward");
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
    bool one_sample = false;
    variable_list apply(variable_list&& grads) override {
        variable_list out(2);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack();
        Scope s(x);
        if (one_sample)
            f2f_one_sample_backward(s, aligned(upstream(grads)), aligned(x), filter.unpack(), aligned(bary.unpack()), bary_padded.unpack(),
                                    cum.unpack(), precision, out[0], out[1]);
        else
            f2f_backward(s, aligned(upstream(grads)), aligned(x), filter.unpack(), aligned(bary.unpack()), bary_padded.unpack(),
                     cum.unpack(), precision, out[0], out[1], task_should_compute_output(0));
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
        f2f_one_sample_backward(s, gz, y.unpack(), filter.unpack(), weights.unpack(), weights_padded.unpack(), one_each.unpack(),
                                precision, gy, out[2]);
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
        node->one_sample = true;
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

// ------------------------------------------------------------------------------------------------------------ layers
// What stands behind the operator of a layer: product with depth_weights, bias, ReLU or nothing, batch normalisation.
enum NormMode { NORM_NONE = 0, NORM_BATCH = 1, NORM_RUNNING = 2 };
struct Tail {
    int mode = NORM_NONE;
    bool relu = false;
    Tensor gamma, beta, running_mean, running_var, batches;
    double momentum = 0, eps = 0;
};
void check_tail(const Tail& t, int64_t Cout) {
    for (const Tensor* x : {&t.gamma, &t.beta, &t.running_mean, &t.running_var})
        if (x->defined() && x->numel() != Cout) fail("batch normalisation must have one value per output channel");
}

// Mean and 1 / deviation of every channel
struct NormStats { Tensor mean, invstd; };
void bump(const Tensor& t) { if (t.defined()) t.unsafeGetTensorImpl()->bump_version(); }
int64_t* counter(const Tensor& t) { return static_cast<int64_t*>(address(t, at::kLong)); }

// Statistics of activated rows with torch's own reduction (norm.cu says why); it moves the running statistics too.
NormStats batch_stats(const Scope& s, const Tail& t, const Tensor& act) {
    NormStats st;
    Tensor var;
    std::tie(st.mean, var) = at::batch_norm_update_stats(act, t.running_mean, t.running_var, t.momentum);
    st.invstd = s.floats({act.size(1)});
    call(pb200_norm_invstd((int)act.size(1), fp(var), (float)t.eps, counter(t.batches), fpm(st.invstd), s.stream), "pb200_norm_invstd");
    bump(t.running_mean);
    bump(t.running_var);
    bump(t.batches);
    return st;
}

// Statistics from the partials of pb200_bias_act_stats
NormStats finalize(const Scope& s, const Tail& t, int64_t C, int nparts, const Tensor& partial) {
    NormStats st{s.floats({C}), s.floats({C})};
    call(pb200_norm_finalize(nparts, (int)C, fp(partial), (float)t.eps, (float)t.momentum, fpm(t.running_mean), fpm(t.running_var),
                             counter(t.batches), fpm(st.mean), fpm(st.invstd), s.stream),
         "pb200_norm_finalize");
    bump(t.running_mean);
    bump(t.running_var);
    bump(t.batches);
    return st;
}

Tensor normalise(const Scope& s, const Tail& t, const Tensor& act, const NormStats& st) {
    Tensor out = s.floats(act.sizes());
    call(pb200_norm_apply(act.size(0), (int)act.size(1), fp(act), fp(st.mean), fp(st.invstd), fp(t.gamma), fp(t.beta), fpm(out), s.stream),
         "pb200_norm_apply");
    return out;
}

// The per-channel factors that take a gradient back through the normalisation, each array on a 16-byte boundary, and the
// gradients of gamma and beta
struct NormGrads {
    Tensor buffer, gamma, beta;
    pb200_norm_gradient factors = {nullptr, nullptr, nullptr, nullptr};
};
NormGrads norm_backward(const Scope& s, const Tensor& g, const Tensor& act, const NormStats& st, const Tensor& gamma) {
    const int64_t rows = act.size(0), C = act.size(1), pitch = (C + 3) / 4 * 4;
    NormGrads r{s.floats({3, pitch}), s.floats({C}), s.floats({C})};
    float *scale = fpm(r.buffer), *k1 = scale + pitch, *k2 = k1 + pitch;
    Tensor partial = s.floats({pb200_norm_parts(rows, (int)C), 2, C});
    call(pb200_norm_backward_reduce(rows, (int)C, fp(g), fp(act), fp(st.mean), fp(st.invstd), fp(gamma), fpm(partial), fpm(r.gamma),
                                    fpm(r.beta), scale, k1, k2, s.stream),
         "pb200_norm_backward_reduce");
    r.factors = {fp(st.mean), scale, k1, k2};
    return r;
}

// The gradient in front of the activation, as an array of its own, and its column sums
void masked_gradient(const Scope& s, const Tensor& g, const Tensor& act, const NormGrads& n, bool relu, Tensor& gm, Tensor& bias) {
    const int64_t rows = act.size(0), C = act.size(1);
    gm = s.floats({rows, C});
    bias = s.floats({1, C});
    Tensor partial = s.floats({pb200_norm_parts(rows, (int)C), C});
    call(pb200_norm_backward_apply(rows, (int)C, fp(g), fp(act), n.factors.mean, n.factors.scale, n.factors.k1, n.factors.k2, relu ? 1 : 0,
                                   fpm(gm), fpm(partial), fpm(bias), s.stream),
         "pb200_norm_backward_apply");
}

// The pointwise stage of a forward pass.  `launch` runs the operator's layer entry with the extras it is handed; what
// the backward pass needs stays in `act`, `features` and `stats`.
struct Staged { Tensor out, act, features; NormStats stats; };
// What a pass that keeps no features may spend on gathered rows (2 M rows of 128 channels); larger ones gather inside the product.
constexpr int64_t GATHER_BYTES = int64_t(1) << 30;
// Whether that much can be had without making room: from what the allocator holds and nobody uses, else from a device that has
// plenty.  An allocation that fails gives every cached block back to the driver first, and a pass would pay for that call after call.
bool has_room(size_t bytes) {
    using c10::CachingAllocator::StatType;
    constexpr auto ALL = static_cast<size_t>(StatType::AGGREGATE);
    const auto stats = c10::cuda::CUDACachingAllocator::getDeviceStats(call_device);
    const int64_t reserved = stats.reserved_bytes[ALL].current, need = (int64_t)bytes;
    if (reserved - stats.active_bytes[ALL].current >= need) return true;
    size_t free = 0, total = 0;
    c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    if (cudaMemGetInfo(&free, &total) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    const double allowed = c10::cuda::CUDACachingAllocator::getMemoryFraction(call_device) * (double)total - (double)reserved;
    return (double)free >= 4. * (double)need && allowed >= 4. * (double)need;
}
template <typename Launch>
Staged run_stage(const Scope& s, const Tail& t, int64_t rows, int64_t C, int64_t Cout, bool keep_features, bool gathers, Launch&& launch) {
    check_tail(t, Cout);
    Staged r;
    r.act = s.floats({rows, Cout});
    pb200_pointwise_extra x = {};
    Workspace scratch;
    if (keep_features) {
        r.features = s.floats({rows, C});
        x.features = fpm(r.features);
    } else if (gathers && rows <= GATHER_BYTES / 4 / C) {
        try {
            if (has_room((size_t)(4 * rows * C))) {
                scratch = s.bytes((size_t)(4 * rows * C));
                x.features = static_cast<float*>(scratch.data_ptr());
            }
        } catch (const c10::Error&) {      // no memory after all, an allocator without figures: the kernel that needs no room is still there
        }
    }
    if (t.mode == NORM_RUNNING) {
        x.mean = fp(t.running_mean); x.var = fp(t.running_var); x.gamma = fp(t.gamma); x.beta = fp(t.beta); x.eps = (float)t.eps;
    }
    launch(fpm(r.act), &x);
    r.out = r.act;
    if (t.mode == NORM_BATCH) {
        r.stats = batch_stats(s, t, r.act);
        r.out = normalise(s, t, r.act, r.stats);
    }
    return r;
}

struct StageGrads { Tensor features, weights, bias, gamma, beta; };

// Gradients of out = norm(act(features @ weights + bias)) for upstream g.
StageGrads stage_backward(const Scope& s, const Tensor& g_in, const Tensor& act, const Tensor& features, const Tensor& weights,
                          const NormStats& st, const Tensor& gamma, bool relu, bool want_features, int precision) {
    const int64_t rows = act.size(0), C = weights.size(0), Cout = act.size(1);
    StageGrads r;
    const Tensor g = aligned(g_in);
    const bool normed = st.mean.defined();
    NormGrads n;
    if (normed) {
        n = norm_backward(s, g, act, st, gamma);
        r.gamma = n.gamma;
        r.beta = n.beta;
    }
    Tensor gm = g;
    if (Cout % 8 == 0 && rows > 0 && want_features) {
        r.features = s.floats({rows, C});
        if (relu || normed) gm = s.floats({rows, Cout});
        const size_t nb = pb200_masked_rows_matmul_workspace_bytes((int)Cout, precision);
        const Workspace ws = s.bytes(nb);
        call(pb200_gradient_rows_matmul(rows, (int)Cout, (int)C, fp(g), relu || normed ? fp(act) : nullptr, relu ? 1 : 0,
                                        normed ? &n.factors : nullptr, fp(weights), 1, fpm(r.features),
                                        gm.is_same(g) ? nullptr : fpm(gm), precision, ws.data_ptr(), nb, s.stream),
             "pb200_gradient_rows_matmul");
    } else {
        if (rows > 0 && (relu || normed)) masked_gradient(s, g, act, n, relu, gm, r.bias);
        if (want_features) r.features = at::matmul(gm, weights.t());
    }
    if (C % 4 == 0 && Cout % 4 == 0 && rows > 0) {
        const Tensor a = aligned(features);
        r.weights = s.floats({C, Cout});
        r.bias = s.floats({1, Cout});
        const size_t nb = pb200_rows_contract_workspace_bytes(rows, (int)C, (int)Cout);
        const Workspace ws = s.bytes(nb);
        call(pb200_rows_contract(rows, (int)C, (int)Cout, fp(a), fp(gm), fpm(r.weights), fpm(r.bias), precision, ws.data_ptr(), nb,
                                 s.stream),
             "pb200_rows_contract");
    } else {
        r.weights = at::matmul(features.t(), gm);
        if (!r.bias.defined()) r.bias = gm.sum(0, true);
    }
    return r;
}

// one value per output channel; a single value stands for all
Tensor flat(const Tensor& bias, int64_t Cout) {
    if (!bias.defined()) return bias;
    if (bias.numel() == 1 && Cout != 1) return bias.reshape({1}).expand({Cout}).contiguous();
    if (bias.numel() != Cout) fail("biases must have one value per output channel");
    return bias.reshape({-1}).contiguous();
}
void check_stage(const Tensor& weights, int64_t C) {
    check(weights, "depth_weights", 2, at::kFloat);
    if (weights.size(0) != C) fail("depth_weights must have shape (channels, out_channels)");
}
// gradients that the node's edges ask for only
#define PUT(i, t) do { if (task_should_compute_output(i)) out[i] = (t); } while (0)

struct V2FLayer : Node {
    SavedVariable input, filter, corners, face, rowptr, entries, weights, act, features, mean, invstd, gamma;
    bool relu = false, sorted = true;                          // sorted: there are rowptr and entries
    int precision = 0;
    variable_list apply(variable_list&& grads) override {
        variable_list out(6);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack(), eye = corners.unpack();
        Scope s(x);
        if (!sorted) fail(BAD_FACE);
        StageGrads r = stage_backward(s, upstream(grads), act.unpack(shared_from_this()), features.unpack(), weights.unpack(), NormStats{mean.unpack(), invstd.unpack()},
                                      gamma.unpack(), relu,
                                      task_should_compute_output(0) || task_should_compute_output(1), precision);
        if (r.features.defined()) {
            Tensor gf;
            v2f_backward(s, r.features, x, filter.unpack(), face.unpack(), rowptr.unpack(), entries.unpack(), out[0], gf);
            if (task_should_compute_output(1)) {
                out[1] = s.floats({eye.size(1), x.size(1)});
                call(pb200_corner_filter_backward((int)eye.size(1), (int)x.size(1), fp(eye), fp(gf), fpm(out[1]), s.stream),
                     "pb200_corner_filter_backward");
            }
        }
        PUT(2, r.weights);
        PUT(3, r.bias);
        PUT(4, r.gamma);
        PUT(5, r.beta);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&input, &filter, &corners, &face, &rowptr, &entries, &weights, &act, &features, &mean, &invstd, &gamma}) v->reset_data();
    }
    std::string name() const override { return "VertexToFacetLayerBackward"; }
};

struct F2VLayer : Node {
    SavedVariable input, filter, coeff, face, nf_count, vt_map, weights, act, features, mean, invstd, gamma;
    bool relu = false;
    int precision = 0;
    variable_list apply(variable_list&& grads) override {
        variable_list out(6);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack();
        Scope s(x);
        StageGrads r = stage_backward(s, upstream(grads), act.unpack(shared_from_this()), features.unpack(), weights.unpack(), NormStats{mean.unpack(), invstd.unpack()},
                                      gamma.unpack(), relu,
                                      task_should_compute_output(0) || task_should_compute_output(1), precision);
        if (r.features.defined())
            f2v_backward(s, r.features, x, filter.unpack(), coeff.unpack(), face.unpack(), nf_count.unpack(), vt_map.unpack(), out[0],
                         out[1]);
        PUT(2, r.weights);
        PUT(3, r.bias);
        PUT(4, r.gamma);
        PUT(5, r.beta);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&input, &filter, &coeff, &face, &nf_count, &vt_map, &weights, &act, &features, &mean, &invstd, &gamma}) v->reset_data();
    }
    std::string name() const override { return "FacetToVertexLayerBackward"; }
};

struct RowsLayer : Node {
    SavedVariable rows, weights, act, mean, invstd, gamma;
    bool relu = false;
    int precision = 0;
    variable_list apply(variable_list&& grads) override {
        variable_list out(5);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = rows.unpack();
        Scope s(x);
        StageGrads r = stage_backward(s, upstream(grads), act.unpack(shared_from_this()), x, weights.unpack(), NormStats{mean.unpack(), invstd.unpack()},
                                      gamma.unpack(), relu,
                                      task_should_compute_output(0), precision);
        PUT(0, r.features);
        PUT(1, r.weights);
        PUT(2, r.bias);
        PUT(3, r.gamma);
        PUT(4, r.beta);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&rows, &weights, &act, &mean, &invstd, &gamma}) v->reset_data();
    }
    std::string name() const override { return "RowsLayerBackward"; }
};

struct F2FLayer : Node {
    SavedVariable input, filter, bary, cum, act, mean, invstd, gamma;
    bool relu = false;
    int precision = 0;
    variable_list apply(variable_list&& grads) override {
        variable_list out(5);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack(), a = act.unpack(shared_from_this()), g = aligned(upstream(grads));
        const NormStats st{mean.unpack(), invstd.unpack()};
        Scope s(x);
        NormGrads n;
        if (st.mean.defined()) {
            n = norm_backward(s, g, a, st, gamma.unpack());
            out[3] = n.gamma;
            out[4] = n.beta;
        }
        const Tensor w = filter.unpack();
        const int64_t Nf = a.size(0), NiK = x.size(0), Cin = x.size(1), Cout = w.size(0), F = w.size(2);
        const Tensor weights = aligned(bary.unpack());
        if (!task_should_compute_output(0) &&
            pb200_facet2facet_layer_gradient_fused(Nf, NiK, (int)Cin, (int)Cout, (int)F, fp(weights), precision)) {
            out[1] = s.floats(w.sizes());
            out[2] = s.floats({1, Cout});
            const size_t nb = pb200_facet2facet_layer_filter_gradient_workspace_bytes(Nf, (int)Cout, (int)F);
            const Workspace ws = s.bytes(nb);
            const Tensor samples = aligned(x), ends = cum.unpack();
            call(pb200_facet2facet_layer_filter_gradient(Nf, NiK, (int)Cin, (int)Cout, (int)F, fp(g), fp(a), relu,
                                                         st.mean.defined() ? &n.factors : nullptr, fp(samples), fp(weights), ip(ends), fpm(out[1]),
                                                         fpm(out[2]), precision, ws.data_ptr(), nb, s.stream),
                 "pb200_facet2facet_layer_filter_gradient");
            return out;
        }
        Tensor gm;
        masked_gradient(s, g, a, n, relu, gm, out[2]);
        f2f_backward(s, gm, aligned(x), w, weights, Tensor(), cum.unpack(), precision, out[0], out[1],
                     task_should_compute_output(0));
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&input, &filter, &bary, &cum, &act, &mean, &invstd, &gamma}) v->reset_data();
    }
    std::string name() const override { return "FacetToFacetLayerBackward"; }
};

Tail make_tail(bool relu, int mode, const OptTensor& gamma, const OptTensor& beta, const OptTensor& mean, const OptTensor& var,
               const OptTensor& batches, double momentum, double eps) {
    return Tail{mode, relu, or_undefined(gamma), or_undefined(beta), or_undefined(mean), or_undefined(var), or_undefined(batches),
                momentum, eps};
}
#define TAIL_PARAMS bool relu, int norm_mode, const OptTensor &gamma, const OptTensor &beta, const OptTensor &running_mean, \
        const OptTensor &running_var, const OptTensor &batches, double momentum, double eps, int precision
#define TAIL_ARGS relu, norm_mode, gamma, beta, running_mean, running_var, batches, momentum, eps

// vertex2facet with the filter corners @ spatial_weights, then the pointwise stage
Tensor v2f_layer(const Tensor& x_in, const Tensor& face, const OptTensor& rowptr, const OptTensor& entries, const Tensor& corners,
                 const Tensor& spatial, const Tensor& weights_in, const OptTensor& bias_in, TAIL_PARAMS) {
    const Tail t = make_tail(TAIL_ARGS);
    const Tensor bias0 = or_undefined(bias_in);
    std::shared_ptr<V2FLayer> node;
    if (torch::autograd::compute_requires_grad(x_in, spatial, weights_in, bias0, t.gamma, t.beta))
        node = node_for<V2FLayer>(x_in, spatial, weights_in, bias0, t.gamma, t.beta);
    at::AutoDispatchBelowADInplaceOrView below;
    check(x_in, "input", 2, at::kFloat);
    check(face, "face", 2, at::kInt);
    check(spatial.contiguous(), "spatial_weights", 2, at::kFloat);
    check_stage(weights_in, x_in.size(1));
    const int64_t Nv = x_in.size(0), C = x_in.size(1), Nf = face.size(0), Cout = weights_in.size(1), K = corners.size(1);
    if (spatial.size(0) != K || spatial.size(1) != C) fail("spatial_weights must have shape (number of bases, channels)");
    if (Nf > 0 && face.size(1) != 3) fail("face must have shape (NfIn, 3)");
    Scope s(x_in);
    const Tensor x = aligned(x_in), bias = flat(bias0, Cout);
    // the library product, whose rounding the separate modules share (norm.cu says why bits matter between layers)
    const Tensor filter = at::matmul(corners, spatial).view({3, C, 1});
    const size_t nb = pb200_vertex2facet_pointwise_workspace_bytes((int)C, precision);
    const Workspace ws = s.bytes(nb);
    Staged r = run_stage(s, t, Nf, C, Cout, (bool)node, pb200_vertex2facet_layer_wants_features(Nf, (int)C, (int)Cout), [&](float* out, const pb200_pointwise_extra* extra) {
        call(pb200_vertex2facet_layer_forward(Nf, Nv, (int)C, (int)Cout, fp(x), fp(filter), ip(face), fp(weights_in), fp(bias), relu, out,
                                              precision, extra, ws.data_ptr(), nb, s.stream),
             "pb200_vertex2facet_layer_forward");
    });
    if (node) {
        node->input = keep(x);
        node->filter = keep(filter);
        node->corners = keep(corners);
        node->face = keep(face);
        node->rowptr = keep(or_undefined(rowptr));
        node->sorted = rowptr.has_value();
        node->entries = keep(or_undefined(entries));
        node->weights = keep(weights_in);
        node->features = keep(r.features);
        node->mean = keep(r.stats.mean);
        node->invstd = keep(r.stats.invstd);
        node->gamma = keep(t.gamma);
        node->relu = relu;
        node->precision = precision;
        torch::autograd::set_history(r.out, node);
        node->act = SavedVariable(r.act, r.act.is_same(r.out));
    }
    return r.out;
}

Tensor f2v_layer(const Tensor& x_in, const Tensor& face, const Tensor& nf_count, const Tensor& vt_map, const Tensor& rowptr,
                 const Tensor& entries, const Tensor& coeff, const Tensor& filter_in, const Tensor& weights, const OptTensor& bias_in,
                 TAIL_PARAMS) {
    const Tail t = make_tail(TAIL_ARGS);
    const Tensor bias0 = or_undefined(bias_in);
    std::shared_ptr<F2VLayer> node;
    if (torch::autograd::compute_requires_grad(x_in, filter_in, weights, bias0, t.gamma, t.beta))
        node = node_for<F2VLayer>(x_in, filter_in, weights, bias0, t.gamma, t.beta);
    at::AutoDispatchBelowADInplaceOrView below;
    check_f2v(x_in, filter_in, coeff, face, nf_count, vt_map);
    check_stage(weights, x_in.size(1));
    const int64_t Nf = x_in.size(0), C = x_in.size(1), K = filter_in.size(0), NvOut = nf_count.size(0), Cout = weights.size(1);
    if (filter_in.size(2) != 1) fail("filter must have shape (K, C, 1)");
    Scope s(x_in);
    const Tensor x = aligned(x_in), filter = aligned(filter_in), bias = flat(bias0, Cout);
    const size_t nb = pb200_facet2vertex_pointwise_workspace_bytes(Nf, (int)C, precision);
    const Workspace ws = s.bytes(nb);
    Staged r = run_stage(s, t, NvOut, C, Cout, (bool)node, pb200_layer_wants_features(NvOut), [&](float* out, const pb200_pointwise_extra* extra) {
        call(pb200_facet2vertex_layer_forward(Nf, NvOut, (int)C, (int)K, (int)Cout, fp(x), fp(filter), fp(coeff), ip(nf_count), ip(rowptr),
                                              ip(entries), fp(weights), fp(bias), relu, out, precision, extra, ws.data_ptr(), nb, s.stream),
             "pb200_facet2vertex_layer_forward");
    });
    if (node) {
        node->input = keep(x);
        node->filter = keep(filter);
        node->coeff = keep(coeff);
        node->face = keep(face);
        node->nf_count = keep(nf_count);
        node->vt_map = keep(vt_map);
        node->weights = keep(weights);
        node->features = keep(r.features);
        node->mean = keep(r.stats.mean);
        node->invstd = keep(r.stats.invstd);
        node->gamma = keep(t.gamma);
        node->relu = relu;
        node->precision = precision;
        torch::autograd::set_history(r.out, node);
        node->act = SavedVariable(r.act, r.act.is_same(r.out));
    }
    return r.out;
}

Tensor rows_layer(const Tensor& rows_in, const Tensor& weights, const OptTensor& bias_in, TAIL_PARAMS) {
    const Tail t = make_tail(TAIL_ARGS);
    const Tensor bias0 = or_undefined(bias_in);
    std::shared_ptr<RowsLayer> node;
    if (torch::autograd::compute_requires_grad(rows_in, weights, bias0, t.gamma, t.beta))
        node = node_for<RowsLayer>(rows_in, weights, bias0, t.gamma, t.beta);
    at::AutoDispatchBelowADInplaceOrView below;
    check(rows_in, "inputs", 2, at::kFloat);
    check(weights, "weights", 2, at::kFloat);
    const int64_t N = rows_in.size(0), C = rows_in.size(1), Cout = weights.size(1);
    if (weights.size(0) != C) fail("weights must have shape (in_channels, out_channels)");
    Scope s(rows_in);
    const Tensor rows = aligned(rows_in), bias = flat(bias0, Cout);
    const size_t nb = pb200_masked_rows_matmul_workspace_bytes((int)C, precision);
    const Workspace ws = s.bytes(nb);
    Staged r = run_stage(s, t, N, C, Cout, false, false, [&](float* out, const pb200_pointwise_extra* extra) {
        call(pb200_rows_layer_forward(N, (int)C, (int)Cout, fp(rows), fp(weights), fp(bias), relu, out, precision, extra, ws.data_ptr(), nb,
                                      s.stream),
             "pb200_rows_layer_forward");
    });
    if (node) {
        node->rows = keep(rows);
        node->weights = keep(weights);
        node->mean = keep(r.stats.mean);
        node->invstd = keep(r.stats.invstd);
        node->gamma = keep(t.gamma);
        node->relu = relu;
        node->precision = precision;
        torch::autograd::set_history(r.out, node);
        node->act = SavedVariable(r.act, r.act.is_same(r.out));
    }
    return r.out;
}

// out = the normalisation of activated rows (act itself without one) by the statistics of the batch, from their partials, or the
// running ones; the batch's statistics
NormStats normalise_by(const Scope& s, const Tail& t, const Tensor& act, int parts, const Tensor& partial, Tensor& out) {
    const int64_t C = act.size(1);
    out = act;
    NormStats st;
    if (t.mode == NORM_BATCH) {
        st = finalize(s, t, C, parts, partial);
        out = normalise(s, t, act, st);
    } else if (t.mode == NORM_RUNNING) {
        const NormStats running{t.running_mean, s.floats({C})};
        call(pb200_norm_invstd((int)C, fp(t.running_var), (float)t.eps, nullptr, fpm(running.invstd), s.stream), "pb200_norm_invstd");
        out = normalise(s, t, act, running);
    }
    return st;
}

// act <- activation(act + bias) in place, out = its normalisation (act itself without one); the statistics used
NormStats bias_act_norm(const Scope& s, const Tail& t, const Tensor& act, const Tensor& bias, Tensor& out) {
    const int64_t rows = act.size(0), C = act.size(1);
    check_tail(t, C);
    Tensor partial = s.floats({pb200_norm_parts(rows, (int)C), 3, C});
    int parts = 0;
    call(pb200_bias_act_stats(rows, (int)C, fpm(act), fp(bias), t.relu, fpm(partial), &parts, s.stream), "pb200_bias_act_stats");
    return normalise_by(s, t, act, parts, partial, out);
}

// facet2facet over the samples of every face (`counts` per face), then bias, ReLU or nothing, normalisation
Tensor f2f_layer(const Tensor& input, const Tensor& filter, const Tensor& bary, const Tensor& counts, const Tensor& bias0, TAIL_PARAMS) {
    const Tail t = make_tail(TAIL_ARGS);
    std::shared_ptr<F2FLayer> node;
    if (torch::autograd::compute_requires_grad(input, filter, bias0, t.gamma, t.beta))
        node = node_for<F2FLayer>(input, filter, bias0, t.gamma, t.beta);
    at::AutoDispatchBelowADInplaceOrView below;
    check_f2f(input, filter, bary);
    Scope s(input);
    const Tensor cum = at::cumsum(counts, 0, at::kInt), bias = flat(bias0, filter.size(0));
    check(cum, "num_texture", 1, at::kInt);
    const int64_t NiK = input.size(0), Cin = input.size(1), Cout = filter.size(0), F = filter.size(2), Nf = cum.size(0);
    check_tail(t, Cout);
    const Tensor x = aligned(input), act = s.floats({Nf, Cout}), partial = s.floats({pb200_norm_parts(Nf, (int)Cout), 3, Cout});
    const size_t nb = pb200_facet2facet_forward_workspace_bytes(Nf, NiK, (int)Cin, (int)Cout, (int)F, precision);
    const Workspace ws = s.bytes(nb);
    int parts = 0;
    call(pb200_facet2facet_layer_forward(Nf, NiK, (int)Cin, (int)Cout, (int)F, fp(x), fp(filter), fp(bary), ip(cum), fp(bias), relu, fpm(act),
                                         fpm(partial), &parts, precision, ws.data_ptr(), nb, s.stream),
         "pb200_facet2facet_layer_forward");
    Tensor out;
    const NormStats st = normalise_by(s, t, act, parts, partial, out);
    if (node) {
        node->input = keep(input);
        node->filter = keep(filter);
        node->bary = keep(bary);
        node->cum = keep(cum);
        node->mean = keep(st.mean);
        node->invstd = keep(st.invstd);
        node->gamma = keep(t.gamma);
        node->relu = relu;
        node->precision = precision;
        torch::autograd::set_history(out, node);
        node->act = SavedVariable(act, act.is_same(out));
    }
    return out;
}

// ------------------------------------------------------------------------------------------- pooling over clusters
struct Pool : Node {
    enum Kind { MAX, AVG, UNPOOL } kind = MAX;
    SavedVariable max_index, vt_replace;
    Tensor key, rowptr, members;                               // cluster arrays of the cache: never written in place
    std::vector<int64_t> in_shape;
    variable_list apply(variable_list&& grads) override {
        variable_list out(1);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor g = upstream(grads);
        Scope s(g);
        out[0] = s.floats(in_shape);
        const int64_t n = in_shape[0], C = in_shape[1], m = g.size(0);
        if (kind == MAX)
            call(pb200_mesh_max_pool_backward_clusters(n, m, (int)C, ip(max_index.unpack()), fp(g), ip(key), ip(rowptr), fpm(out[0]), s.stream),
                 "pb200_mesh_max_pool_backward_clusters");
        else if (kind == AVG)
            call(pb200_mesh_avg_pool_backward(n, m, (int)C, fp(g), ip(vt_replace.unpack()), ip(key), fpm(out[0]), s.stream),
                 "pb200_mesh_avg_pool_backward");
        else
            call(pb200_mesh_unpool_backward(n, m, (int)C, fp(g), ip(rowptr), ip(members), fpm(out[0]), s.stream),
                 "pb200_mesh_unpool_backward");
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        max_index.reset_data();
        vt_replace.reset_data();
        key.reset(); rowptr.reset(); members.reset();
    }
    std::string name() const override { return "MeshPoolBackward"; }
};

std::shared_ptr<Pool> pool_node(Pool::Kind kind, const Tensor& input, const Tensor& key, const Tensor& rowptr, const Tensor& members) {
    std::shared_ptr<Pool> node;
    if (torch::autograd::compute_requires_grad(input)) {
        node = node_for<Pool>(input);
        node->kind = kind;
        node->in_shape = input.sizes().vec();
        node->key = key; node->rowptr = rowptr; node->members = members;
    }
    return node;
}

Tensor max_pool(const Tensor& input, int64_t nv_out, const Tensor& key, const Tensor& rowptr, const Tensor& members) {
    auto node = pool_node(Pool::MAX, input, key, rowptr, members);
    Tensor out, index;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        const int64_t C = input.size(1);
        out = s.floats({nv_out, C});
        index = s.ints({nv_out, C});
        call(pb200_mesh_max_pool_forward(input.size(0), nv_out, (int)C, fp(input), ip(rowptr), ip(members), fpm(out),
                                         static_cast<int32_t*>(index.data_ptr()), s.stream),
             "pb200_mesh_max_pool_forward");
    }
    if (node) {
        node->max_index = keep(index);
        torch::autograd::set_history(out, node);
    }
    return out;
}

Tensor avg_pool(const Tensor& input, int64_t nv_out, const Tensor& vt_replace, const Tensor& key, const Tensor& rowptr,
                const Tensor& members) {
    auto node = pool_node(Pool::AVG, input, key, rowptr, members);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        out = s.floats({nv_out, input.size(1)});
        call(pb200_mesh_avg_pool_forward(input.size(0), nv_out, (int)input.size(1), fp(input), ip(vt_replace), ip(rowptr), ip(members),
                                         fpm(out), s.stream),
             "pb200_mesh_avg_pool_forward");
    }
    if (node) {
        node->vt_replace = keep(vt_replace);
        torch::autograd::set_history(out, node);
    }
    return out;
}

Tensor unpool(const Tensor& input, int64_t nv_fine, const Tensor& key, const Tensor& rowptr, const Tensor& members) {
    auto node = pool_node(Pool::UNPOOL, input, key, rowptr, members);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        out = s.floats({nv_fine, input.size(1)});
        call(pb200_mesh_unpool_forward(input.size(0), nv_fine, (int)input.size(1), fp(input), ip(key), fpm(out), s.stream),
             "pb200_mesh_unpool_forward");
    }
    if (node) torch::autograd::set_history(out, node);
    return out;
}

struct SegmentMean : Node {
    Tensor ends;                                               // of the cache: never written in place
    int64_t rows = 0, channels = 0;
    variable_list apply(variable_list&& grads) override {
        variable_list out(1);
        if (!grads[0].defined()) return out;
        const Tensor g = upstream(grads);
        Scope s(g);
        out[0] = s.floats({rows, channels});
        call(pb200_segment_mean_backward(rows, (int)g.size(0), (int)channels, fp(g), ends.data_ptr<int64_t>(), fpm(out[0]), s.stream),
             "pb200_segment_mean_backward");
        return out;
    }
    std::string name() const override { return "SegmentMeanBackward"; }
};

Tensor segment_mean(const Tensor& input, const Tensor& ends) {
    std::shared_ptr<SegmentMean> node;
    if (torch::autograd::compute_requires_grad(input)) node = node_for<SegmentMean>(input);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        const int64_t N = input.size(0), C = input.size(1), B = ends.size(0);
        out = s.floats({B, C});
        const size_t nb = pb200_segment_mean_workspace_bytes(N, (int)B, (int)C);
        const Workspace ws = s.bytes(nb);
        call(pb200_segment_mean(N, (int)B, (int)C, fp(input), ends.data_ptr<int64_t>(), fpm(out), ws.data_ptr(), nb, s.stream),
             "pb200_segment_mean");
    }
    if (node) {
        node->ends = ends;
        node->rows = input.size(0);
        node->channels = input.size(1);
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ----------------------------------------------------------------------------------------------- point-cloud convolution
// The neighbour pairs and the two groupings of them (rowptr / members by output and by input point)
struct Pairs { Tensor nn_count, nn_index, bin_index, bin_coeff; };
int bins_per_pair(const Pairs& q) { return q.bin_coeff.defined() ? (int)q.bin_index.size(1) : 1; }

void check_pairs(const Tensor& input, const Tensor& filter, const Pairs& q) {
    check(input, "input", 2, at::kFloat);
    check(filter, "filter", 3, at::kFloat);
    check(q.nn_count, "nn_count", 1, at::kInt);
    check(q.nn_index, "nn_index", 2, at::kInt);
    check(q.bin_index, "bin_index", q.bin_coeff.defined() ? 2 : 1, at::kInt);
    if (q.bin_coeff.defined()) {
        check(q.bin_coeff, "bin_coeff", 2, at::kFloat);
        if (q.bin_coeff.sizes() != q.bin_index.sizes()) fail("bin_coeff and bin_index must have the same shape");
    }
    if (filter.size(1) != input.size(1)) fail("Input Channel size error of the filter");
    if (q.nn_index.size(0) > 0 && q.nn_index.size(1) != 2) fail("nn_index must have shape (pairs, 2)");
    if (q.bin_index.size(0) != q.nn_index.size(0)) fail("bin_index must have one row per neighbor pair");
}

Tensor pairs_forward(const Scope& s, const Tensor& input, const Tensor& filter, const Pairs& q, const Tensor& rowptr, const Tensor& members) {
    const int64_t Np = input.size(0), C = input.size(1), F = filter.size(0), r = filter.size(2), Mp = q.nn_count.size(0);
    Tensor out = s.floats({Mp, C * r});
    call(pb200_pcloud_conv3d_forward(Np, Mp, q.nn_index.size(0), (int)F, (int)C, (int)r, bins_per_pair(q), fp(input), fp(filter),
                                     ip(q.nn_count), ip(q.nn_index), ip(q.bin_index), fp(q.bin_coeff), ip(rowptr), ip(members), fpm(out),
                                     s.stream),
         "pb200_pcloud_conv3d_forward");
    return out;
}

void pairs_backward(const Scope& s, const Tensor& g, const Tensor& input, const Tensor& filter, const Pairs& q, const Tensor& rowptr,
                    const Tensor& members, Tensor& gin, Tensor& gf) {
    const int64_t Np = input.size(0), C = input.size(1), F = filter.size(0), r = filter.size(2), Mp = q.nn_count.size(0), n = q.nn_index.size(0);
    if (!rowptr.defined()) fail(BAD_PAIR);
    gin = s.floats({Np, C});
    gf = s.floats({F, C, r});
    const size_t nb = pb200_pcloud_conv3d_backward_workspace_bytes(n, (int)F, (int)C, (int)r);
    const Workspace ws = s.bytes(nb);
    call(pb200_pcloud_conv3d_backward(Np, Mp, n, (int)F, (int)C, (int)r, bins_per_pair(q), fp(g), fp(input), fp(filter), ip(q.nn_count),
                                      ip(q.nn_index), ip(q.bin_index), fp(q.bin_coeff), ip(rowptr), ip(members), fpm(gin), fpm(gf),
                                      ws.data_ptr(), nb, s.stream),
         "pb200_pcloud_conv3d_backward");
}

struct PairsNode : Node {
    SavedVariable input, filter, nn_count, nn_index, bin_index, bin_coeff, rowptr, members;
    bool sorted = true;                                        // there are rowptr and members
    void keep_pairs(const Tensor& x, const Tensor& f, const Pairs& q, const Tensor& by_in_rowptr, const Tensor& by_in_members) {
        input = keep(x);
        filter = keep(f);
        nn_count = keep(q.nn_count);
        nn_index = keep(q.nn_index);
        bin_index = keep(q.bin_index);
        bin_coeff = keep(q.bin_coeff);
        rowptr = keep(by_in_rowptr);
        sorted = by_in_rowptr.defined();
        members = keep(by_in_members);
    }
    void pairs_gradient(const Scope& s, const Tensor& g, const Tensor& x, Tensor& gin, Tensor& gf) {
        pairs_backward(s, g, x, filter.unpack(), Pairs{nn_count.unpack(), nn_index.unpack(), bin_index.unpack(), bin_coeff.unpack()},
                       rowptr.unpack(), members.unpack(), gin, gf);
    }
    variable_list apply(variable_list&& grads) override {
        variable_list out(2);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack();
        Scope s(x);
        pairs_gradient(s, upstream(grads), x, out[0], out[1]);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&input, &filter, &nn_count, &nn_index, &bin_index, &bin_coeff, &rowptr, &members}) v->reset_data();
    }
    std::string name() const override { return "PointConvBackward"; }
};

// convolution, product with depth_weights (fp32), bias, ReLU or nothing, normalisation
struct PointLayer : PairsNode {
    SavedVariable features, weights, act, mean, invstd, gamma;
    bool relu = false;
    variable_list apply(variable_list&& grads) override {
        variable_list out(6);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor x = input.unpack(), a = act.unpack(shared_from_this()), w = weights.unpack(), feats = features.unpack(),
                     g = aligned(upstream(grads));
        const NormStats st{mean.unpack(), invstd.unpack()};
        Scope s(x);
        if (!sorted) fail(BAD_PAIR);
        NormGrads n;
        if (st.mean.defined()) {
            n = norm_backward(s, g, a, st, gamma.unpack());
            out[4] = n.gamma;
            out[5] = n.beta;
        }
        Tensor gm;
        masked_gradient(s, g, a, n, relu, gm, out[3]);
        const int64_t rows = a.size(0), M = w.size(0), N = w.size(1);
        out[2] = s.floats({M, N});
        const size_t nb = pb200_rows_contract_f32_workspace_bytes(rows, (int)M, (int)N);
        const Workspace ws = s.bytes(nb);
        call(pb200_rows_contract_f32(rows, (int)M, (int)N, fp(feats), fp(gm), fpm(out[2]), ws.data_ptr(), nb, s.stream),
             "pb200_rows_contract_f32");
        if (task_should_compute_output(0) || task_should_compute_output(1))
            pairs_gradient(s, at::matmul(gm, w.t()), x, out[0], out[1]);
        return out;
    }
    void release_variables() override {
        PairsNode::release_variables();
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* v : {&features, &weights, &act, &mean, &invstd, &gamma}) v->reset_data();
    }
    std::string name() const override { return "PointLayerBackward"; }
};

Tensor point_conv(const Tensor& input, const Tensor& filter, const Tensor& nn_count, const Tensor& nn_index, const Tensor& bin_index,
                  const OptTensor& bin_coeff, const Tensor& out_rowptr, const Tensor& out_members, const OptTensor& in_rowptr,
                  const OptTensor& in_members) {
    const Pairs q{nn_count, nn_index, bin_index, or_undefined(bin_coeff)};
    check_pairs(input, filter, q);
    std::shared_ptr<PairsNode> node;
    if (torch::autograd::compute_requires_grad(input, filter)) node = node_for<PairsNode>(input, filter);
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Scope s(input);
        out = pairs_forward(s, input, filter, q, out_rowptr, out_members);
    }
    if (node) {
        node->keep_pairs(input, filter, q, or_undefined(in_rowptr), or_undefined(in_members));
        torch::autograd::set_history(out, node);
    }
    return out;
}

Tensor point_layer(const Tensor& input, const Tensor& filter, const Tensor& nn_count, const Tensor& nn_index, const Tensor& bin_index,
                   const OptTensor& bin_coeff, const Tensor& out_rowptr, const Tensor& out_members, const OptTensor& in_rowptr,
                   const OptTensor& in_members, const Tensor& weights_in, const Tensor& bias0, bool relu, int norm_mode, const OptTensor& gamma,
                   const OptTensor& beta, const OptTensor& running_mean, const OptTensor& running_var, const OptTensor& batches,
                   double momentum, double eps) {
    const Tail t = make_tail(TAIL_ARGS);
    const Pairs q{nn_count, nn_index, bin_index, or_undefined(bin_coeff)};
    check_pairs(input, filter, q);
    std::shared_ptr<PointLayer> node;
    if (torch::autograd::compute_requires_grad(input, filter, weights_in, bias0, t.gamma, t.beta))
        node = node_for<PointLayer>(input, filter, weights_in, bias0, t.gamma, t.beta);
    at::AutoDispatchBelowADInplaceOrView below;
    Scope s(input);
    const Tensor weights = weights_in.contiguous();
    check_stage(weights, filter.size(1) * filter.size(2));
    Tensor feats = pairs_forward(s, input, filter, q, out_rowptr, out_members);
    Tensor act = at::matmul(feats, weights), out;
    const NormStats st = bias_act_norm(s, t, act, flat(bias0, weights.size(1)), out);
    if (node) {
        node->keep_pairs(input, filter, q, or_undefined(in_rowptr), or_undefined(in_members));
        node->features = keep(feats);
        node->weights = keep(weights);
        node->mean = keep(st.mean);
        node->invstd = keep(st.invstd);
        node->gamma = keep(t.gamma);
        node->relu = relu;
        torch::autograd::set_history(out, node);
        node->act = SavedVariable(act, act.is_same(out));
    }
    return out;
}

// -------------------------------------------------------------------------------------------------------- decimation
Tensor on_device(const std::vector<int64_t>& values, const Tensor& like) {
    return at::tensor(values, at::TensorOptions().dtype(at::kInt)).to(like.device());
}
std::vector<int64_t> on_host(const Tensor& t) {
    const Tensor h = t.cpu().contiguous();
    const int32_t* p = h.data_ptr<int32_t>();
    return std::vector<int64_t>(p, p + h.numel());
}

// The pass loop of mesh_decimation (picasso/mesh/pi_modules/decimate.py:5-48) with one synchronisation per pass: the host
// reads the samples' new sizes, which it needs to allocate the result, and decides on the next pass by them.
// target_in: vertices to keep, one number per sample or one for all.  Without it the sizes are known to the caller already:
// nv_host / mf_host / target_host are the values of nv_in / mf_in and the target.
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, std::vector<int64_t>, std::vector<int64_t>>
mesh_decimation(const Tensor& vertex_in, const Tensor& face_in, const Tensor& geometry_in, const Tensor& nv_in, const Tensor& mf_in,
                const OptTensor& target_in, bool use_area, double wgt_bnd, std::vector<int64_t> nv_host, std::vector<int64_t> mf_host,
                std::vector<int64_t> target_host) {
    c10::InferenceMode inference(false);
    at::NoGradGuard no_grad;
    if (nv_in.dim() != 1 || mf_in.dim() != 1) fail("nvIn and mfIn must have dimension of 1");
    const int64_t B = nv_in.size(0);
    if (target_in.has_value()) {
        const Tensor& t = *target_in;
        if (t.dim() > 1) fail("the vertices to keep must have dimension of 1");
        if (t.dim() == 1 && t.device() != nv_in.device()) fail("the vertices to keep must be on the device of nvIn");
        if (nv_in.device() == mf_in.device() && nv_in.device() == t.device()) {                   // one copy to the host
            const std::vector<int64_t> all = on_host(at::cat({nv_in.to(at::kInt), mf_in.to(at::kInt), t.reshape({-1}).to(at::kInt)}));
            nv_host.assign(all.begin(), all.begin() + B);
            mf_host.assign(all.begin() + B, all.begin() + B + mf_in.size(0));
            target_host.assign(all.begin() + B + mf_in.size(0), all.end());
        } else {
            nv_host = on_host(nv_in.to(at::kInt));
            mf_host = on_host(mf_in.to(at::kInt));
            target_host = on_host(t.reshape({-1}).to(at::kInt));
        }
    }
    if (target_host.size() == 1) target_host.assign(B, target_host[0]);
    if ((int64_t)nv_host.size() != B || (int64_t)target_host.size() != B)
        fail("nvIn and the vertices to keep must have one entry per sample");
    auto sum = [](const std::vector<int64_t>& v) { int64_t t = 0; for (int64_t x : v) t += x; return t; };
    auto more = [&] { for (int64_t k = 0; k < B; ++k) if (nv_host[k] > target_host[k]) return true; return false; };
    Tensor rep, map;
    if (!more()) {
        const auto i32 = vertex_in.options().dtype(at::kInt).requires_grad(false);
        rep = at::zeros({vertex_in.size(0)}, i32);
        map = at::arange(vertex_in.size(0), i32);
        return {vertex_in, face_in, geometry_in, nv_in, mf_in, rep, map, nv_host, mf_host};
    }
    if (mf_in.size(0) != B || (int64_t)mf_host.size() != B) fail("mfIn must have one entry per sample");
    for (int64_t k = 0; k < B; ++k)
        if (nv_host[k] < 0 || mf_host[k] < 0) fail("mesh_simplify: nvIn / mfIn must not be negative");
    Tensor vertex = vertex_in.contiguous(), face = face_in.contiguous(), geometry = geometry_in.contiguous();
    check(vertex, "vertexIn", 2, at::kFloat);
    check(face, "faceIn", 2, at::kInt);
    check(geometry, "planeIn", 2, at::kFloat);
    if (vertex.size(1) < 3) fail("The shape of input vertex should be (Nv, 3+)).");
    if (face.size(1) != 3) fail("The shape of input face should be (Nf, 3)).");
    if (geometry.size(0) != face.size(0) || geometry.size(1) != 5) fail("The shape of input face normals should be (Nf, 5)).");
    for (const Tensor& t : {face, geometry, nv_in, mf_in})
        if (t.device() != vertex.device()) fail("vertexIn, faceIn, planeIn, nvIn and mfIn must be on one CUDA device");
    if (sum(nv_host) != vertex.size(0) || sum(mf_host) != face.size(0))
        fail("mesh_simplify: nvIn / mfIn must be the samples' vertex and face counts");
    Scope s(vertex);
    const auto i32 = s.f32.dtype(at::kInt);
    const int64_t D = vertex.size(1);
    Tensor nv = nv_in, mf = mf_in;
    const bool there = target_in.has_value() && target_in->dim() == 1 && target_in->size(0) == B;
    const Tensor target = there ? target_in->to(at::kInt).contiguous() : on_device(target_host, vertex);
    while (more()) {
        const int64_t Nv = vertex.size(0), Nf = face.size(0);
        const Tensor sizes = s.ints({2 * B + 1}), vt_replace = s.ints({Nv}), vt_map = s.ints({Nv});
        int32_t* sz = sizes.data_ptr<int32_t>();
        const size_t nb = pb200_mesh_simplify_workspace_bytes(B, Nv, Nf);
        const Workspace ws = s.bytes(nb);
        const Tensor nv32 = nv.to(at::kInt).contiguous(), mf32 = mf.to(at::kInt).contiguous();
        int64_t most = 0;
        for (int64_t m : mf_host) most = m > most ? m : most;
        call(pb200_decimate_begin(use_area, (float)wgt_bnd, B, D, Nv, Nf, most, ip(nv32), ip(mf32), ip(target), fp(vertex), ip(face),
                                  fp(geometry), sz, sz + B, sz + 2 * B, vt_replace.data_ptr<int32_t>(), vt_map.data_ptr<int32_t>(),
                                  ws.data_ptr(), nb, s.stream),
             "pb200_decimate_begin");
        const std::vector<int64_t> now = on_host(sizes);
        if (now[2 * B] == PB200_EINDEX) fail("mesh_simplify: face holds a vertex id outside [0, Nv)");
        if (now[2 * B] == 1) fail("mesh_simplify: a face joins vertices of two samples");
        if (now[2 * B] != 0) fail("mesh_simplify: a wait inside the clustering kernel ran out");
        bool removed = false;
        for (int64_t k = 0; k < B; ++k) removed |= now[k] < nv_host[k];
        if (!removed) break;               // nothing left to contract (no candidate edges): the reference would loop forever
        nv_host.assign(now.begin(), now.begin() + B);
        mf_host.assign(now.begin() + B, now.begin() + 2 * B);
        const int64_t Nv2 = sum(nv_host), Nf2 = sum(mf_host);
        Tensor vertex2 = s.floats({Nv2, D}), face2 = s.ints({Nf2, 3}), geometry2 = s.floats({Nf2, 5});
        // an empty result still needs addresses for the checks of the call; nothing is written there
        float* const nowhere = static_cast<float*>(ws.data_ptr());
        call(pb200_decimate_finish(B, D, Nv, Nf, fp(vertex), ip(vt_replace), ip(vt_map), Nv2 ? fpm(vertex2) : nowhere,
                                   Nf2 ? face2.data_ptr<int32_t>() : sz, Nf2 ? fpm(geometry2) : nowhere, ws.data_ptr(), nb, s.stream),
             "pb200_decimate_finish");
        if (!rep.defined()) {
            rep = vt_replace;
            map = vt_map;
        } else {
            const int64_t nvA = rep.size(0);
            Tensor rep2 = s.ints({nvA}), map2 = s.ints({nvA}), work = s.ints({Nv + 2});
            int32_t* w = work.data_ptr<int32_t>();
            call(pb200_combine_clusters(nvA, Nv, ip(rep), ip(map), ip(vt_replace), ip(vt_map), rep2.data_ptr<int32_t>(),
                                        map2.data_ptr<int32_t>(), w + Nv + 1, w, sizeof(int32_t) * (size_t)(Nv + 1), s.stream),
                 "pb200_combine_clusters");
            rep = rep2;
            map = map2;
        }
        vertex = vertex2;
        face = face2;
        geometry = geometry2;
        nv = sizes.narrow(0, 0, B);
        mf = sizes.narrow(0, B, B);
    }
    if (!rep.defined()) {                  // not even the first pass found an edge
        rep = at::zeros({vertex.size(0)}, i32);
        map = at::arange(vertex.size(0), i32);
        return {vertex_in, face_in, geometry_in, nv, mf, rep, map, nv_host, mf_host};
    }
    return {vertex, face, geometry, nv, mf, rep, map, nv_host, mf_host};
}

// One mesh level: what topology.prepare_level returns, with the status word of the CSR build.
std::tuple<OptTensor, OptTensor, Tensor, Tensor, Tensor, Tensor, Tensor>
level_prepare(const Tensor& vertex, const Tensor& face, const OptTensor& vt_map, int64_t nv_out, int L, bool orient, bool want_geometry,
              bool want_normals) {
    c10::InferenceMode inference(false);         // the structure is kept (topology.py)
    at::NoGradGuard no_grad;
    Scope s(face);
    const auto i32 = s.f32.dtype(at::kInt);
    const int64_t nv_in = vertex.size(0), nf = face.size(0), K = (int64_t)(L + 1) * (L + 1);
    OptTensor geometry, normals;
    if (want_geometry) geometry = s.floats({nf, 5});
    if (want_normals) normals = s.floats({nf, 3});
    Tensor coeff = s.floats({nf, K}), nf_count = s.ints({nv_out}), rowptr = s.ints({nv_out + 1}),
           entries = s.ints({nf > 0 ? 3 * nf : 1}), status = s.ints({1});
    const size_t nb = pb200_vertex_csr_workspace_bytes(nf, nv_out);
    const Workspace ws = s.bytes(nb);
    call(pb200_level_prepare(nf, nv_in, nv_out, (int)vertex.size(1), fp(vertex), ip(face), vt_map.has_value() ? ip(*vt_map) : nullptr, L,
                             orient ? 1 : 0, geometry.has_value() ? fpm(*geometry) : nullptr, normals.has_value() ? fpm(*normals) : nullptr,
                             fpm(coeff), nf_count.data_ptr<int32_t>(), rowptr.data_ptr<int32_t>(), entries.data_ptr<int32_t>(),
                             status.data_ptr<int32_t>(), ws.data_ptr(), nb, s.stream),
         "pb200_level_prepare");
    return {geometry, normals, coeff, nf_count, rowptr, entries, status};
}

// -------------------------------------------------------------------------------------------------- topology cache
// Structures derived from index tensors (CSRs, sample means, running totals), found again by the tensors they were made
// from.  An entry is named by kind, addresses, row counts, row strides, types and two numbers; it is good while the index tensors' storages are the ones it
// was made from (weak references: the cache does not keep a batch's tensors alive, and memory that was freed and handed out
// again is another storage) and their version counters have not moved.  Entries of storages that are gone are dropped at
// the next insertion: a program that brings a new batch every step holds the structures of the batches it holds, no more.
// Otherwise least recently used ones go when the bytes exceed the budget.  A structure used on a stream other than the one
// it was made on waits there for its kernels and is recorded there, so that dropping it is safe at any time.  One made while a
// graph is captured exists when that graph has run and is good inside that capture only.  All calls run under the GIL.
struct TopologyCache {
    struct Source {
        c10::weak_intrusive_ptr<c10::StorageImpl> storage;
        int64_t version;
        explicit Source(const Tensor& t) : storage(t.storage().getWeakStorageImpl()), version(t._version()) {}
        bool is(const Tensor& t) const {
            return !storage.expired() && storage._unsafe_get_target() == t.storage().unsafeGetStorageImpl() && version == (int64_t)t._version();
        }
    };
    struct Entry {
        std::vector<Source> sources;
        std::vector<Tensor> tensors;
        py::object value;
        int64_t bytes;
        c10::cuda::CUDAStream stream;
        unsigned long long capture;              // id of the capture it was made in, 0: none
        c10::Event ready;                        // behind the kernels that make it
        bool complete = false;                   // they are known to have run
    };
    using Key = std::array<int64_t, 12>;
    struct Hash {
        size_t operator()(const Key& k) const {
            uint64_t h = 0x9e3779b97f4a7c15ull;
            for (int64_t x : k) h = (h ^ (uint64_t)x) * 0xff51afd7ed558ccdull, h ^= h >> 32;
            return (size_t)h;
        }
    };
    using List = std::list<std::pair<Key, Entry>>;
    List recent;                                 // least recently used first
    std::unordered_map<Key, List::iterator, Hash> at;
    int64_t bytes = 0, budget = 2ll << 30;

    static Key key(int kind, const Tensor& a, const OptTensor& b, int64_t m, int64_t n) {
        Key k{kind, a.device().index(), (int64_t)a.data_ptr(), a.size(0), a.stride(0), (int64_t)a.scalar_type(), m, n, -1, -1, -1, -1};
        if (b.has_value()) k[8] = (int64_t)b->data_ptr(), k[9] = b->size(0), k[10] = b->stride(0), k[11] = (int64_t)b->scalar_type();
        return k;
    }
    static unsigned long long capture_id(c10::cuda::CUDAStream stream) {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        unsigned long long id = 0;
        C10_CUDA_CHECK(cudaStreamGetCaptureInfo(stream.stream(), &status, &id));
        return status == cudaStreamCaptureStatusActive ? id : 0;
    }
    // orders work on `now` behind the kernels that make e; false: they belong to another capture
    static bool order(Entry& e, c10::cuda::CUDAStream now) {
        if (e.capture != 0) {
            if (capture_id(now) != e.capture) return false;
            if (now != e.stream) e.ready.block(now.unwrap());
            return true;
        }
        if (now == e.stream || e.complete) return true;
        c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);     // a capture elsewhere must not mind the query
        e.complete = e.ready.query();
        if (!e.complete && capture_id(now) != 0) {       // a captured stream cannot wait for what lies outside: the host does
            e.ready.synchronize();
            e.complete = true;
        }
        if (!e.complete) e.ready.block(now.unwrap());
        return true;
    }
    void erase(List::iterator it) {
        bytes -= it->second.bytes;
        at.erase(it->first);
        recent.erase(it);
    }
    // what inference mode made counts no versions: nothing tells whether it has been overwritten since
    static bool versioned(const Tensor& a, const OptTensor& b) { return !a.is_inference() && !(b.has_value() && b->is_inference()); }
    Entry* find(const Key& k, const Tensor& a, const OptTensor& b) {
        if (!versioned(a, b)) return nullptr;
        auto it = at.find(k);
        if (it == at.end()) return nullptr;
        Entry& e = it->second->second;
        if (!e.sources[0].is(a) || (b.has_value() && !e.sources[1].is(*b))) return nullptr;
        const auto now = c10::cuda::getCurrentCUDAStream(a.device().index());
        if (!order(e, now)) return nullptr;
        recent.splice(recent.end(), recent, it->second);
        if (now != e.stream)
            for (const Tensor& t : e.tensors) t.record_stream(now);
        return &e;
    }
    void put(const Key& k, const Tensor& a, const OptTensor& b, std::vector<Tensor> tensors, py::object value, int64_t size, bool complete) {
        auto old = at.find(k);
        if (old != at.end()) erase(old->second);
        for (auto it = recent.begin(); it != recent.end();) {
            auto here = it++;
            bool gone = false;
            for (const Source& src : here->second.sources) gone |= src.storage.expired();
            if (gone) erase(here);
        }
        if (budget <= 0 || !versioned(a, b)) return;
        const auto now = c10::cuda::getCurrentCUDAStream(a.device().index());
        Entry e{{Source(a)}, std::move(tensors), std::move(value), size, now, capture_id(now), c10::Event(c10::DeviceType::CUDA)};
        if (b.has_value()) e.sources.emplace_back(*b);
        e.complete = complete && e.capture == 0;
        if (!e.complete) e.ready.record(now.unwrap());
        at[k] = recent.insert(recent.end(), {k, std::move(e)});
        bytes += size;
        while (!recent.empty() && bytes > budget) erase(recent.begin());
    }
};
TopologyCache& cache() {
    static TopologyCache* c = new TopologyCache();          // never destroyed: it holds Python objects
    return *c;
}
py::object cache_find(int kind, const Tensor& a, const OptTensor& b, int64_t m, int64_t n) {
    TopologyCache::Entry* e = cache().find(TopologyCache::key(kind, a, b, m, n), a, b);
    return e ? e->value : py::object(py::none());
}
// complete: the caller has waited for the kernels that make the structure
void cache_put(int kind, const Tensor& a, const OptTensor& b, int64_t m, int64_t n, std::vector<Tensor> tensors, py::object value,
               int64_t bytes, bool complete) {
    cache().put(TopologyCache::key(kind, a, b, m, n), a, b, std::move(tensors), std::move(value), bytes, complete);
}
void cache_budget(int64_t n) {
    TopologyCache& c = cache();
    c.budget = n;
    while (!c.recent.empty() && c.bytes > c.budget) c.erase(c.recent.begin());
}
py::tuple cache_stats() { return py::make_tuple(cache().recent.size(), cache().bytes, cache().budget); }
void cache_clear() {
    cache().at.clear();
    cache().recent.clear();
    cache().bytes = 0;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.doc() = "Native host path of picassoplus_b200 (see torch_ops.cpp).";
    m.def("vertex2facet", &vertex2facet);
    m.def("facet2vertex", &facet2vertex);
    m.def("facet2facet", &facet2facet);
    m.def("facet2facet_shared_rows", &facet2facet_shared_rows);
    m.def("conv_block", &conv_block);
    m.def("v2f_layer", &v2f_layer);
    m.def("f2v_layer", &f2v_layer);
    m.def("rows_layer", &rows_layer);
    m.def("f2f_layer", &f2f_layer);
    m.def("point_conv", &point_conv);
    m.def("point_layer", &point_layer);
    m.def("max_pool", &max_pool);
    m.def("avg_pool", &avg_pool);
    m.def("unpool", &unpool);
    m.def("segment_mean", &segment_mean);
    // it waits for the GPU once per pass: other threads of the interpreter go on meanwhile
    m.def("mesh_decimation", &mesh_decimation, py::call_guard<py::gil_scoped_release>());
    m.def("level_prepare", &level_prepare);
    m.def("cache_find", &cache_find);
    m.def("cache_put", &cache_put);
    m.def("cache_budget", &cache_budget);
    m.def("cache_stats", &cache_stats);
    m.def("cache_clear", &cache_clear);
}
