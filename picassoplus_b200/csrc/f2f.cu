// facet2facet entry points: argument checks and the choice between the fp32 FFMA path
// (every shape, fp32-faithful) and the tensor-core path.
#include "common.cuh"

namespace pb {
size_t f2f_simt_fwd_ws(int64_t Nf, int Cin, int Cout, int F);
size_t f2f_simt_bwd_ws(int64_t Nf, int Cin, int Cout, int F);
int f2f_simt_forward(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* input, const float* filter,
                     const float* bary, const int32_t* cum, float* output, void* ws, cudaStream_t stream);
int f2f_simt_backward(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* gout, const float* input,
                      const float* filter, const float* bary, const int32_t* cum, float* gin, float* gfilter,
                      void* ws, cudaStream_t stream, bool want_gin, bool want_gfilter);
namespace small {
bool supported(int Cin, int Cout, int F);
int forward(int64_t Nf, int Cin, int Cout, int F, const float* input, const float* filter, const float* bary, const int32_t* cum,
            float* output, cudaStream_t stream);
size_t workspace_bytes(int64_t Nf, int Cin, int Cout, int F);
int backward_filter(int64_t Nf, int Cin, int Cout, int F, const float* gout, const float* input, const float* bary, const int32_t* cum,
                    float* gfilter, void* ws, cudaStream_t stream);
}  // namespace small
namespace rgb {
bool supported(int Cin, int F, const float* bary);
bool forward_alone(int Cout, int F);
bool gradient_alone(int Cout);
bool layer_forward(int Cout);
bool layer_gradient(int Cout);
int forward(int64_t Nf, int Cout, int F, const float* input, const float* filter, const float* bary, const int32_t* cum, const float* bias,
            int relu, float* output, float* stats, int most, int* nparts, cudaStream_t stream);
size_t workspace_bytes(int64_t Nf, int Cout, int F);
int backward_filter(int64_t Nf, int Cout, int F, const float* gout, const float* act, int relu, const pb200_norm_gradient* norm,
                    const float* input, const float* bary, const int32_t* cum, float* gfilter, float* gbias, void* ws, cudaStream_t stream);
}  // namespace rgb
namespace tc {
bool fwd_supported(int Cin, int Cout, int F);
size_t fwd_workspace_bytes(int64_t NiK, int Cin, int Cout, int F, int precision);
int forward(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* input, const float* filter,
            const float* bary, const int32_t* cum, float* output, int precision, void* ws, cudaStream_t stream);
int check_async_error(const char* where);
namespace gin {
bool supported(int Cin, int Cout, int F);
bool fits(int Cin, int Cout, int F, int precision);
size_t workspace_bytes(int Cin, int Cout, int F, int precision);
int backward_input(int64_t Nf, int Cin, int Cout, int F, const float* gout, const float* filter, const float* bary,
                   const float* bary_p, int Fp, const int32_t* cum, float* gin, int precision, void* ws,
                   cudaStream_t stream, bool transposed);
}  // namespace gin
namespace one {
bool supported(int Cn, int Ck, int F, int precision);
size_t workspace_bytes(int Cn, int Ck, int F, int precision);
int run(int64_t Nf, int Cn, int Ck, int F, const float* rows, const float* filter, const float* w, int Fp, float* out, int precision,
        void* ws, cudaStream_t stream, bool forward);
}  // namespace one
namespace onef {
bool supported(int Cin, int Cout, int F, int precision);
size_t workspace_bytes(int64_t Nf, int Cin, int Cout, int F, int precision);
int backward_filter(int64_t Nf, int Cin, int Cout, int F, const float* gout, const float* input, const float* w, float* gfilter,
                    int precision, void* ws, cudaStream_t stream);
}  // namespace onef
namespace gfilter {
bool supported(int Cin, int Cout, int F);
bool fits(int64_t Nf, int Cin, int Cout, int F, int precision);
size_t workspace_bytes(int64_t Nf, int Cin, int Cout, int F, int precision);
int backward_filter(int64_t Nf, int Cin, int Cout, int F, const float* gout, const float* input, const float* bary_p,
                    int Fp, const int32_t* cum, float* gfilter, int precision, void* ws, cudaStream_t stream);
}  // namespace gfilter
int padded_F(int F);
size_t padded_bary_bytes(int64_t NiK, int F);
int pad_bary(int64_t NiK, int F, const float* bary, float* dst, cudaStream_t stream);
int padded_channels(int Cin);
size_t padded_input_bytes(int64_t NiK, int Cin);
int pad_input(int64_t NiK, int Cin, const float* input, float* dst, cudaStream_t stream);
}  // namespace tc
}  // namespace pb

using namespace pb;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static bool use_tc_fwd(int Cin, int Cout, int F, int precision) {
    return precision != PB200_PREC_FP32_FFMA && tc::fwd_supported(Cin, Cout, F);
}
// Few input channels: fp32 kernels of their own in every tensor-core mode.  Meshes of less than 4096 faces stay on the
// tensor-core kernels: test_every_channel_count_runs_on_the_tensor_cores pins those for a small mesh of three channels.  The line is
// not where the two sides meet (4000 faces: 26 us on the tensor cores, 9 here); a training step of that size is host work.  The filter
// gradient's products outgrow the multiply-add units where the tensor cores' padding wastes less (1 758 000 faces, three channels:
// 16 bases, 32 outputs 358 against 876 us, 25 bases, 64 outputs 1376 against 1066); forward there are no partial sums to keep and the
// line lies further out (278 against 907 us, 1006 against 1168).
static bool use_small(int64_t Nf, int Cin, int Cout, int F, int precision) {
    return precision != PB200_PREC_FP32_FFMA && Nf >= 4096 && small::supported(Cin, Cout, F) && Cin * Cout * F <= 5000;
}
static bool use_small_gf(int64_t Nf, int Cin, int Cout, int F, int precision) {
    return use_small(Nf, Cin, Cout, F, precision) && Cin * Cout * F <= 3600;
}
static bool use_tc_gf(int64_t Nf, int Cin, int Cout, int F, int precision) {
    return precision != PB200_PREC_FP32_FFMA && tc::gfilter::supported(Cin, Cout, F) &&
           tc::gfilter::fits(Nf, Cin, Cout, F, precision);
}
static bool use_tc_gin(int Cin, int Cout, int F, int precision) {
    return precision != PB200_PREC_FP32_FFMA && tc::gin::supported(Cin, Cout, F) && tc::gin::fits(Cin, Cout, F, precision);
}

static bool f2f_sizes_ok(int64_t Nf, int64_t NiK, int Cin, int Cout, int F) {
    return Nf >= 0 && NiK >= 0 && Cin > 0 && Cout > 0 && F > 0 && F <= 50 && NiK < (1LL << 31) && Nf < (1LL << 31);
}

extern "C" {

size_t pb200_facet2facet_forward_workspace_bytes(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, int precision) {
    if (!f2f_sizes_ok(Nf, NiK, Cin, Cout, F)) return 0;
    if (use_small(Nf, Cin, Cout, F, precision)) return 256;
    if (use_tc_fwd(Cin, Cout, F, precision)) return tc::fwd_workspace_bytes(NiK, Cin, Cout, F, precision);
    return f2f_simt_fwd_ws(Nf, Cin, Cout, F);
}

int pb200_facet2facet_forward(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* input,
                              const float* filter, const float* bary, const int32_t* numInterior, float* output,
                              int precision, void* workspace, size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(f2f_sizes_ok(Nf, NiK, Cin, Cout, F), PB200_EINVAL,
               "facet2facet_forward: bad sizes (F must be in 1..50)");
    PB_REQUIRE(precision >= PB200_PREC_FP32 && precision <= PB200_PREC_FP32_TF32X3, PB200_EINVAL,
               "facet2facet_forward: unknown precision %d", precision);
    if (Nf == 0) return PB200_OK;
    PB_REQUIRE(filter && numInterior && output && (NiK == 0 || (input && bary)), PB200_EINVAL,
               "facet2facet_forward: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_facet2facet_forward_workspace_bytes(Nf, NiK, Cin, Cout, F, precision),
               PB200_EWORKSPACE, "facet2facet_forward: workspace too small");
    if (use_small(Nf, Cin, Cout, F, precision)) {
        if (rgb::supported(Cin, F, bary) && rgb::forward_alone(Cout, F))
            return rgb::forward(Nf, Cout, F, input, filter, bary, numInterior, nullptr, 0, output, nullptr, 0, nullptr, stream);
        return small::forward(Nf, Cin, Cout, F, input, filter, bary, numInterior, output, stream);
    }
    if (use_tc_fwd(Cin, Cout, F, precision)) {
        PB_REQUIRE(NiK == 0 || aligned16(input), PB200_EINVAL, "facet2facet_forward: input must be 16-byte aligned");
        PB_REQUIRE(aligned16(workspace), PB200_EINVAL, "facet2facet_forward: workspace must be 16-byte aligned");
        return tc::forward(Nf, NiK, Cin, Cout, F, input, filter, bary, numInterior, output, precision, workspace,
                           stream);
    }
    return f2f_simt_forward(Nf, NiK, Cin, Cout, F, input, filter, bary, numInterior, output, workspace, stream);
}

int pb200_facet2facet_layer_forward(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* input, const float* filter,
                                    const float* bary, const int32_t* numInterior, const float* bias, int relu, float* act,
                                    float* partial, int* nparts, int precision, void* workspace, size_t workspace_bytes, void* stream) {
    PB_REQUIRE(f2f_sizes_ok(Nf, NiK, Cin, Cout, F) && Nf > 0, PB200_EINVAL, "facet2facet_layer_forward: bad sizes (F must be in 1..50)");
    PB_REQUIRE(partial && nparts, PB200_EINVAL, "facet2facet_layer_forward: null pointer");
    if (use_small(Nf, Cin, Cout, F, precision) && rgb::supported(Cin, F, bary) && rgb::layer_forward(Cout)) {
        PB_REQUIRE(filter && numInterior && act && (NiK == 0 || (input && bary)), PB200_EINVAL, "facet2facet_layer_forward: null pointer");
        return rgb::forward(Nf, Cout, F, input, filter, bary, numInterior, bias, relu, act, partial, pb200_norm_parts(Nf, Cout), nparts,
                            (cudaStream_t)stream);
    }
    const int rc = pb200_facet2facet_forward(Nf, NiK, Cin, Cout, F, input, filter, bary, numInterior, act, precision, workspace, workspace_bytes,
                                             stream);
    return rc ? rc : pb200_bias_act_stats(Nf, Cout, act, bias, relu, partial, nparts, stream);
}

int pb200_facet2facet_layer_gradient_fused(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* bary, int precision) {
    return Nf > 0 && f2f_sizes_ok(Nf, NiK, Cin, Cout, F) && use_small_gf(Nf, Cin, Cout, F, precision) &&
                   rgb::supported(Cin, F, bary) && rgb::layer_gradient(Cout) ? 1 : 0;
}

int pb200_facet2facet_layer_filter_gradient(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* gradOutput, const float* act,
                                            int relu, const pb200_norm_gradient* norm, const float* input, const float* bary,
                                            const int32_t* numInterior, float* gradFilter, float* gradBias, int precision,
                                            void* workspace, size_t workspace_bytes, void* stream) {
    PB_REQUIRE(pb200_facet2facet_layer_gradient_fused(Nf, NiK, Cin, Cout, F, bary, precision), PB200_EINVAL,
               "facet2facet_layer_filter_gradient: sizes that the fused gradient is not for");
    PB_REQUIRE(gradOutput && act && gradFilter && gradBias && numInterior && (NiK == 0 || (input && bary)) &&
                   (!norm || (norm->mean && norm->scale && norm->k1 && norm->k2)),
               PB200_EINVAL, "facet2facet_layer_filter_gradient: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= rgb::workspace_bytes(Nf, Cout, F), PB200_EWORKSPACE,
               "facet2facet_layer_filter_gradient: workspace too small");
    return rgb::backward_filter(Nf, Cout, F, gradOutput, act, relu, norm, input, bary, numInterior, gradFilter, gradBias, workspace,
                                (cudaStream_t)stream);
}

size_t pb200_facet2facet_layer_filter_gradient_workspace_bytes(int64_t Nf, int Cout, int F) {
    return Nf > 0 && Cout > 0 && F > 0 ? rgb::workspace_bytes(Nf, Cout, F) : 0;
}

// One sample per face: output[f,co] = sum_d weights[f,d] * (sum_ci input[f,ci] * filter[co,ci,d]).  The inner
// sum is a plain GEMM over the input rows (no face operand of F * Cin products to build, split and store) and
// the outer one an epilogue over the accumulator: the input-gradient kernel with the channel roles exchanged.
static bool one_sample_on_gin(int Cin, int Cout, int F, int precision) {
    return tc::one::supported(Cout, Cin, F, precision) || use_tc_gin(Cout, Cin, F, precision);
}
// workspace of the one-sample product (Cn channels out of Ck): its own kernel, else the input-gradient kernel's
static size_t one_sample_ws(int Cn, int Ck, int F, int precision) {
    return tc::one::supported(Cn, Ck, F, precision) ? tc::one::workspace_bytes(Cn, Ck, F, precision)
                                                    : tc::gin::workspace_bytes(Cn, Ck, F, precision);
}

size_t pb200_facet2facet_one_sample_forward_workspace_bytes(int64_t Nf, int Cin, int Cout, int F, int precision) {
    if (!f2f_sizes_ok(Nf, Nf, Cin, Cout, F)) return 0;
    if (one_sample_on_gin(Cin, Cout, F, precision))
        return one_sample_ws(Cout, Cin, F, precision) + tc::padded_bary_bytes(Nf, F);
    return align_up(sizeof(int32_t) * (size_t)(Nf > 0 ? Nf : 1), 256) +
           pb200_facet2facet_forward_workspace_bytes(Nf, Nf, Cin, Cout, F, precision);
}

__global__ void count_up_kernel(int64_t n, int32_t* out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (int32_t)(i + 1);
}

int pb200_facet2facet_one_sample_forward(int64_t Nf, int Cin, int Cout, int F, const float* input, const float* filter,
                                         const float* weights, const float* weightsPadded, float* output, int precision,
                                         void* workspace, size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(f2f_sizes_ok(Nf, Nf, Cin, Cout, F), PB200_EINVAL, "facet2facet_one_sample_forward: bad sizes (F must be in 1..50)");
    PB_REQUIRE(precision >= PB200_PREC_FP32 && precision <= PB200_PREC_FP32_TF32X3, PB200_EINVAL,
               "facet2facet_one_sample_forward: unknown precision %d", precision);
    if (Nf == 0) return PB200_OK;
    PB_REQUIRE(input && filter && weights && output, PB200_EINVAL, "facet2facet_one_sample_forward: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_facet2facet_one_sample_forward_workspace_bytes(Nf, Cin, Cout, F, precision),
               PB200_EWORKSPACE, "facet2facet_one_sample_forward: workspace too small");
    char* w = (char*)workspace;
    if (one_sample_on_gin(Cin, Cout, F, precision)) {
        PB_REQUIRE(aligned16(input) && aligned16(weights) && aligned16(workspace), PB200_EINVAL,
                   "facet2facet_one_sample_forward: input, weights and workspace must be 16-byte aligned");
        const float* wp = weights;
        const int Fp = tc::padded_F(F);
        if (F % 4 != 0 && weightsPadded) {
            PB_REQUIRE(aligned16(weightsPadded), PB200_EINVAL,
                       "facet2facet_one_sample_forward: weightsPadded must be 16-byte aligned");
            wp = weightsPadded;
        } else if (F % 4 != 0) {
            float* dst = (float*)(w + one_sample_ws(Cout, Cin, F, precision));
            int rc = tc::pad_bary(Nf, F, weights, dst, stream);
            if (rc) return rc;
            wp = dst;
        }
        if (tc::one::supported(Cout, Cin, F, precision))
            return tc::one::run(Nf, Cout, Cin, F, input, filter, wp, Fp, output, precision, w, stream, true);
        return tc::gin::backward_input(Nf, Cout, Cin, F, input, filter, weights, wp, Fp, nullptr, output, precision, w,
                                       stream, true);
    }
    int32_t* one_each = (int32_t*)w;
    w += align_up(sizeof(int32_t) * (size_t)Nf, 256);
    PB_LAUNCH("count_up", count_up_kernel, persistent_blocks(Nf, 256, 8), 256, 0, stream, Nf, one_each);
    return pb200_facet2facet_forward(Nf, Nf, Cin, Cout, F, input, filter, weights, one_each, output, precision, w,
                                     workspace_bytes - (size_t)(w - (char*)workspace), stream_);
}

// room for the filter image of either input-gradient kernel
static size_t gin_ws(int Cin, int Cout, int F, int precision) {
    const size_t a = tc::gin::workspace_bytes(Cin, Cout, F, precision);
    const size_t b = tc::one::supported(Cin, Cout, F, precision) ? tc::one::workspace_bytes(Cin, Cout, F, precision) : 0;
    return a > b ? a : b;
}

// room for the partial sums of either filter-gradient kernel
static size_t gf_ws(int64_t Nf, int Cin, int Cout, int F, int precision) {
    if (use_small_gf(Nf, Cin, Cout, F, precision)) return small::workspace_bytes(Nf, Cin, Cout, F);
    const size_t a = tc::gfilter::workspace_bytes(Nf, Cin, Cout, F, precision);
    const size_t b = tc::onef::supported(Cin, Cout, F, precision) ? tc::onef::workspace_bytes(Nf, Cin, Cout, F, precision) : 0;
    return a > b ? a : b;
}

size_t pb200_facet2facet_backward_workspace_bytes(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, int precision) {
    if (!f2f_sizes_ok(Nf, NiK, Cin, Cout, F)) return 0;
    const bool tg = use_tc_gin(Cin, Cout, F, precision), sf = use_small_gf(Nf, Cin, Cout, F, precision);
    const bool tf = sf || use_tc_gf(Nf, Cin, Cout, F, precision);
    size_t n = (tg && tf) ? 0 : f2f_simt_bwd_ws(Nf, Cin, Cout, F);
    if (tg) n += gin_ws(Cin, Cout, F, precision);
    if (tf) n += gf_ws(Nf, Cin, Cout, F, precision);
    if (tg || tf) n += tc::padded_bary_bytes(NiK, F);
    if (tf && !sf) n += tc::padded_input_bytes(NiK, Cin);
    return n;
}

}  // extern "C"

// baryPadded: optional copy of bary with rows padded to padded_F(F) floats (pad columns zero), as pb200_pad_rows
// makes it; given, the tensor-core kernels read it instead of padding bary into the workspace on every call
static int f2f_backward_impl(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* gradOutput,
                             const float* input, const float* filter, const float* bary, const float* baryPadded,
                             const int32_t* numInterior, float* gradInput, float* gradFilter, int precision,
                             void* workspace, size_t workspace_bytes, void* stream_, bool want_gin, bool one_each) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(f2f_sizes_ok(Nf, NiK, Cin, Cout, F), PB200_EINVAL,
               "facet2facet_backward: bad sizes (F must be in 1..50)");
    PB_REQUIRE(precision >= PB200_PREC_FP32 && precision <= PB200_PREC_FP32_TF32X3, PB200_EINVAL,
               "facet2facet_backward: unknown precision %d", precision);
    PB_REQUIRE(gradFilter, PB200_EINVAL, "facet2facet_backward: null pointer");
    if (Nf == 0) {
        PB_CUDA(cudaMemsetAsync(gradFilter, 0, sizeof(float) * (size_t)Cout * Cin * F, stream));
        return PB200_OK;
    }
    PB_REQUIRE(gradOutput && (filter || !want_gin) && numInterior && (NiK == 0 || (input && bary && (gradInput || !want_gin))), PB200_EINVAL,
               "facet2facet_backward: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_facet2facet_backward_workspace_bytes(Nf, NiK, Cin, Cout, F, precision),
               PB200_EWORKSPACE, "facet2facet_backward: workspace too small");
    const bool tg = use_tc_gin(Cin, Cout, F, precision), sf = use_small_gf(Nf, Cin, Cout, F, precision);
    const bool tf = sf || use_tc_gf(Nf, Cin, Cout, F, precision);
    if (tg || tf)
        PB_REQUIRE(aligned16(gradOutput) && aligned16(workspace) && (NiK == 0 || (aligned16(input) && aligned16(bary))),
                   PB200_EINVAL, "facet2facet_backward: gradOutput, input, bary and workspace must be 16-byte aligned");
    char* w = (char*)workspace;
    void* simt_ws = w;
    if (!(tg && tf)) w += f2f_simt_bwd_ws(Nf, Cin, Cout, F);
    // both tensor-core kernels read bary rows with 16-byte loads: rows padded to 4 floats
    const float* bary_p = bary;
    const int Fp = tc::padded_F(F);
    if (((tg && want_gin) || (tf && !sf)) && F % 4 != 0 && NiK > 0) {
        if (baryPadded) {
            PB_REQUIRE(aligned16(baryPadded), PB200_EINVAL, "facet2facet_backward: baryPadded must be 16-byte aligned");
            bary_p = baryPadded;
        } else {
            char* wp = w + (tg ? gin_ws(Cin, Cout, F, precision) : 0) +
                       (tf ? gf_ws(Nf, Cin, Cout, F, precision) : 0);
            int rc = tc::pad_bary(NiK, F, bary, (float*)wp, stream);
            if (rc) return rc;
            bary_p = (const float*)wp;
        }
    }
    if (tg) {
        if (NiK > 0 && want_gin) {
            int rc = one_each && tc::one::supported(Cin, Cout, F, precision)
                         ? tc::one::run(Nf, Cin, Cout, F, gradOutput, filter, bary_p, Fp, gradInput, precision, w, stream, false)
                         : tc::gin::backward_input(Nf, Cin, Cout, F, gradOutput, filter, bary, bary_p, Fp, numInterior, gradInput,
                                                   precision, w, stream, false);
            if (rc) return rc;
        }
        w += gin_ws(Cin, Cout, F, precision);
    }
    if (sf) {
        int rc = rgb::supported(Cin, F, bary) && rgb::gradient_alone(Cout)
                     ? rgb::backward_filter(Nf, Cout, F, gradOutput, nullptr, 0, nullptr, input, bary, numInterior, gradFilter, nullptr, w, stream)
                     : small::backward_filter(Nf, Cin, Cout, F, gradOutput, input, bary, numInterior, gradFilter, w, stream);
        if (rc) return rc;
    } else if (tf && one_each && tc::onef::supported(Cin, Cout, F, precision)) {
        int rc = tc::onef::backward_filter(Nf, Cin, Cout, F, gradOutput, input, bary_p, gradFilter, precision, w, stream);
        if (rc) return rc;
    } else if (tf) {
        // the filter-gradient kernel reads 16 input channels per CTA with 16-byte copies: channel counts that
        // are not a multiple of 16 go through a zero-padded copy at the end of the workspace
        const float* input_p = input;
        if (Cin % 16 != 0 && NiK > 0) {
            char* wx = (char*)workspace + pb200_facet2facet_backward_workspace_bytes(Nf, NiK, Cin, Cout, F, precision) -
                       tc::padded_input_bytes(NiK, Cin);
            int rc = tc::pad_input(NiK, Cin, input, (float*)wx, stream);
            if (rc) return rc;
            input_p = (const float*)wx;
        }
        int rc = tc::gfilter::backward_filter(Nf, Cin, Cout, F, gradOutput, input_p, bary_p, Fp, numInterior, gradFilter,
                                              precision, w, stream);
        if (rc) return rc;
    }
    if ((tg || !want_gin) && tf) return PB200_OK;
    return f2f_simt_backward(Nf, NiK, Cin, Cout, F, gradOutput, input, filter, bary, numInterior, gradInput,
                             gradFilter, simt_ws, stream, !tg && want_gin, !tf);
}

extern "C" {

int pb200_facet2facet_backward(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* gradOutput,
                               const float* input, const float* filter, const float* bary,
                               const int32_t* numInterior, float* gradInput, float* gradFilter, int precision,
                               void* workspace, size_t workspace_bytes, void* stream) {
    return f2f_backward_impl(Nf, NiK, Cin, Cout, F, gradOutput, input, filter, bary, nullptr, numInterior, gradInput,
                             gradFilter, precision, workspace, workspace_bytes, stream, true, false);
}

int pb200_facet2facet_backward_padded(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* gradOutput,
                                      const float* input, const float* filter, const float* bary, const float* baryPadded,
                                      const int32_t* numInterior, float* gradInput, float* gradFilter, int precision,
                                      void* workspace, size_t workspace_bytes, void* stream) {
    return f2f_backward_impl(Nf, NiK, Cin, Cout, F, gradOutput, input, filter, bary, baryPadded, numInterior, gradInput,
                             gradFilter, precision, workspace, workspace_bytes, stream, true, false);
}

// for callers whose samples are data (raw textures): the input gradient, a third of the backward pass, is left out
int pb200_facet2facet_filter_gradient(int64_t Nf, int64_t NiK, int Cin, int Cout, int F, const float* gradOutput,
                                      const float* input, const float* bary, const float* baryPadded, const int32_t* numInterior,
                                      float* gradFilter, int precision, void* workspace, size_t workspace_bytes, void* stream) {
    return f2f_backward_impl(Nf, NiK, Cin, Cout, F, gradOutput, input, nullptr, bary, baryPadded, numInterior, nullptr, gradFilter,
                             precision, workspace, workspace_bytes, stream, false, false);
}

int pb200_facet2facet_one_sample_backward(int64_t Nf, int Cin, int Cout, int F, const float* gradOutput, const float* input,
                                          const float* filter, const float* weights, const float* weightsPadded, const int32_t* oneEach,
                                          float* gradInput, float* gradFilter, int precision, void* workspace, size_t workspace_bytes,
                                          void* stream) {
    return f2f_backward_impl(Nf, Nf, Cin, Cout, F, gradOutput, input, filter, weights, weightsPadded, oneEach, gradInput, gradFilter,
                             precision, workspace, workspace_bytes, stream, true, true);
}

int pb200_padded_row_floats(int F) { return F > 0 ? tc::padded_F(F) : 0; }

int pb200_pad_rows(int64_t N, int F, const float* rows, float* out, void* stream) {
    PB_REQUIRE(N >= 0 && F > 0, PB200_EINVAL, "pad_rows: bad sizes");
    if (N == 0) return PB200_OK;
    PB_REQUIRE(rows && out, PB200_EINVAL, "pad_rows: null pointer");
    PB_REQUIRE(aligned16(out), PB200_EINVAL, "pad_rows: out must be 16-byte aligned");
    return tc::pad_bary(N, F, rows, out, (cudaStream_t)stream);
}

}  // extern "C"
