// Launches of gemv_generic_step.cuh: the linears of a decoder step over weights that no tensor-core GEMV serves.
#include "common.cuh"
#include "gemv_generic_step.cuh"

using namespace ab2;

namespace ab2 {
bool qlinear_w4a16_mma_eligible(const ab2_qweight *w, ab2_dtype dtype);
bool qlinear_i8_stream_eligible(const ab2_qweight *w, ab2_dtype dtype, int M);
bool qlinear_q4km_stream_eligible(const ab2_qweight *w, ab2_dtype dtype, int M);
namespace {

constexpr size_t GEN_STEP_MAX_SMEM = 40 * 1024;

template <int FMT, typename T, int MT>
cudaError_t launch_step(const GenericStepArgs &a, int epi, cudaStream_t s) {
    const int outs = epi == GEN_SWIGLU ? a.w.N / 2 : a.w.N;
    const dim3 grid((outs + GEN_STEP_WARPS - 1) / GEN_STEP_WARPS), block(GEN_STEP_WARPS * 32);
    const size_t smem = a.norm_w ? (size_t)a.M * a.w.K * 4 : 0;
    if (epi == GEN_ADD) return launch_kernel(gemv_generic_step_kernel<FMT, T, MT, GEN_ADD, false>, grid, block, 0, s, a);
    if (epi == GEN_SWIGLU) return launch_kernel(gemv_generic_step_kernel<FMT, T, MT, GEN_SWIGLU, true>, grid, block, smem, s, a);
    return launch_kernel(gemv_generic_step_kernel<FMT, T, MT, GEN_STORE, true>, grid, block, smem, s, a);
}

template <int FMT, typename T>
cudaError_t launch_step_tokens(const GenericStepArgs &a, int epi, cudaStream_t s) {
    if (a.M == 1) return launch_step<FMT, T, 1>(a, epi, s);
    return a.M <= 4 ? launch_step<FMT, T, 4>(a, epi, s) : launch_step<FMT, T, 8>(a, epi, s);
}

template <typename T>
cudaError_t launch_step_fmt(int fmt, const GenericStepArgs &a, int epi, cudaStream_t s) {
    switch (fmt) {
    case FMT_I8: return launch_step_tokens<FMT_I8, T>(a, epi, s);
    case FMT_I4_AFFINE: return launch_step_tokens<FMT_I4_AFFINE, T>(a, epi, s);
    case FMT_Q4KM: return launch_step_tokens<FMT_Q4KM, T>(a, epi, s);
    default: return launch_step_tokens<FMT_W4A16, T>(a, epi, s);
    }
}

int step_linear(const ab2_qweight *w, ab2_dtype dtype, GenericStepArgs a, int epi, cudaStream_t s) {
    a.w = gemv_args_of(w);
    cudaError_t e = dtype == AB2_F32 ? launch_step_fmt<float>(w->fmt, a, epi, s) : launch_step_fmt<__nv_bfloat16>(w->fmt, a, epi, s);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "GEMV launch failed: %s", cudaGetErrorString(e));
    return AB2_OK;
}

}  // namespace

// Whether a step of M tokens takes this path: up to 8 tokens that would go to the generic kernel one by one, their
// normed copies in shared memory.
bool qlinear_step_eligible(const ab2_qweight *w, ab2_dtype dtype, int M) {
    return w->fmt != FMT_BF16 && (dtype == AB2_F32 || dtype == AB2_BF16) && M <= 8 && w->K % 8 == 0 && (size_t)M * w->K * 4 <= GEN_STEP_MAX_SMEM &&
           !(w->fmt == FMT_I4_AFFINE && w->group % 8 != 0) && !qlinear_w4a16_mma_eligible(w, dtype) && !qlinear_i8_stream_eligible(w, dtype, M) &&
           !qlinear_q4km_stream_eligible(w, dtype, M);
}

// y = RMSNorm(x; norm_w) . W^T, or its gated unit over a gate|up weight
int qlinear_step_norm(const ab2_qweight *w, const void *x, const float *norm_w, float eps, int M, ab2_dtype dtype, bool swiglu, void *y, cudaStream_t s) {
    GenericStepArgs a = {};
    a.x = x; a.norm_w = norm_w; a.eps = eps; a.y = y; a.M = M;
    return step_linear(w, dtype, a, swiglu ? GEN_SWIGLU : GEN_STORE, s);
}

// y = resid + x . W^T (resid may be y)
int qlinear_step_add(const ab2_qweight *w, const void *x, const void *resid, int M, ab2_dtype dtype, void *y, cudaStream_t s) {
    GenericStepArgs a = {};
    a.x = x; a.resid = resid; a.y = y; a.M = M;
    return step_linear(w, dtype, a, GEN_ADD, s);
}

}  // namespace ab2
