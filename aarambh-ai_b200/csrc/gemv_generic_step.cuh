// The linears of a decoder step over any weight format and type, up to 8 tokens, with what surrounds them: the RMSNorm
// of the input in the prologue, the residual addition or the gated unit at the end.  The arithmetic of
// gemv_generic_kernel, rms_norm_kernel and the element-wise kernels, in one launch of what were two or three.
//
// A decoder of width 384 is bound by launches: its weights stream in less time than a launch takes.  A CTA is four
// warps, a row (or a gate row and its up row) each; the warp requests its first words of the weight before the
// dependency wait, and every CTA norms the tokens for itself.  One step of the 6-layer f32 decoder, with chained launches:
// 171 us in 65 launches before, 90 us in 33.
#pragma once

#include "gemv_generic.cuh"
#include "ops.cuh"

namespace ab2 {

enum GenericEpilogue : int { GEN_STORE = 0, GEN_ADD = 1, GEN_SWIGLU = 2 };

struct GenericStepArgs {
    GemvArgs w;
    const void *x;         // [M][K]
    const float *norm_w;   // with NORM
    const void *resid;     // GEN_ADD: [M][N], may be y
    void *y;               // [M][N], GEN_SWIGLU: [M][N / 2]
    float eps;
    int M;
};

constexpr int GEN_STEP_WARPS = 4;

template <int FMT, typename T, int MT, int EPI, bool NORM>
__global__ void __launch_bounds__(GEN_STEP_WARPS * 32) gemv_generic_step_kernel(GenericStepArgs a) {
    constexpr int ROWS = EPI == GEN_SWIGLU ? 2 : 1, THREADS = GEN_STEP_WARPS * 32;
    extern __shared__ __align__(16) float xs[];   // NORM: [M][K] normed, rounded to T
    __shared__ float warp_sums[MT][GEN_STEP_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * GEN_STEP_WARPS + warp, outs = a.w.N / ROWS, words = a.w.K >> 3;
    const bool live = n < outs;
    // U words of a lane are in flight together; those of the first round are requested, and turned into weights, before
    // the wait
    constexpr int U = MT == 1 ? 4 / ROWS : MT == 4 ? 2 : 1;
    float w[U][ROWS][8];
    auto weights = [&](int word0) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                if (live && word0 + 32 * u < words) dequant_word<FMT>(a.w, n + r * outs, word0 + 32 * u, w[u][r]);
            }
    };
    weights(lane);
    float4 ng[2];
    if (NORM && MT == 1 && words <= THREADS && (int)threadIdx.x < words) {
        ng[0] = *reinterpret_cast<const float4 *>(a.norm_w + threadIdx.x * 8);
        ng[1] = *reinterpret_cast<const float4 *>(a.norm_w + threadIdx.x * 8 + 4);
    }
    pdl_wait();
    pdl_launch_dependents();
    const T *x = (const T *)a.x;
    if (NORM && MT == 1 && words <= THREADS) {
        // one token of at most 1024 columns stays in registers between the two passes
        float v[8], sum = 0.f;
        const int i = threadIdx.x;
        if (i < words) {
            Vec8<T>::load(x + (size_t)i * 8, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) sum = fmaf(v[j], v[j], sum);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) warp_sums[0][warp] = sum;
        __syncthreads();
        sum = 0.f;
#pragma unroll
        for (int k = 0; k < GEN_STEP_WARPS; ++k) sum += warp_sums[0][k];
        const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)a.w.K), a.eps)));
        if (i < words) {
            const float g[8] = {ng[0].x, ng[0].y, ng[0].z, ng[0].w, ng[1].x, ng[1].y, ng[1].z, ng[1].w};
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = to_f32(from_f32<T>(__fmul_rn(__fmul_rn(v[j], inv), g[j])));
            float4 *dst = reinterpret_cast<float4 *>(xs + (size_t)i * 8);
            dst[0] = make_float4(v[0], v[1], v[2], v[3]);
            dst[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
        __syncthreads();
    } else if (NORM) {
        for (int m = 0; m < a.M; ++m) {
            float sum = 0.f;
            for (int i = threadIdx.x; i < words; i += THREADS) {
                float v[8];
                Vec8<T>::load(x + (size_t)m * a.w.K + (size_t)i * 8, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) sum = fmaf(v[j], v[j], sum);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0) warp_sums[m][warp] = sum;
        }
        __syncthreads();
        for (int m = 0; m < a.M; ++m) {
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < GEN_STEP_WARPS; ++i) sum += warp_sums[m][i];
            const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)a.w.K), a.eps)));
            for (int i = threadIdx.x; i < words; i += THREADS) {
                float v[8];
                Vec8<T>::load(x + (size_t)m * a.w.K + (size_t)i * 8, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = to_f32(from_f32<T>(__fmul_rn(__fmul_rn(v[j], inv), a.norm_w[i * 8 + j])));
                float4 *dst = reinterpret_cast<float4 *>(xs + (size_t)m * a.w.K + (size_t)i * 8);
                dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                dst[1] = make_float4(v[4], v[5], v[6], v[7]);
            }
        }
        __syncthreads();
    }
    if (!live) return;
    float acc[ROWS][MT];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;
    for (int word0 = lane; word0 < words; word0 += 32 * U) {
        if (word0 != lane) weights(word0);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < a.M) {
                float xv[U][8];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (word0 + 32 * u < words) {
                        if (NORM) Vec8<float>::load(xs + (size_t)m * a.w.K + (size_t)(word0 + 32 * u) * 8, xv[u]);
                        else Vec8<T>::load(x + (size_t)m * a.w.K + (size_t)(word0 + 32 * u) * 8, xv[u]);
                    }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (word0 + 32 * u < words) {
#pragma unroll
                        for (int r = 0; r < ROWS; ++r)
#pragma unroll
                            for (int j = 0; j < 8; ++j) acc[r][m] = fmaf(xv[u][j], w[u][r][j], acc[r][m]);
                    }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        if (m >= a.M) break;
        float v[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            v[r] = acc[r][m];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[r] += __shfl_xor_sync(0xffffffffu, v[r], o);
        }
        if (lane == 0) {
            const size_t at = (size_t)m * outs + n;
            T *y = (T *)a.y;
            if (EPI == GEN_STORE) y[at] = from_f32<T>(v[0]);
            else if (EPI == GEN_ADD) y[at] = from_f32<T>(__fadd_rn(to_f32(((const T *)a.resid)[at]), to_f32(from_f32<T>(v[0]))));
            else y[at] = from_f32<T>(swiglu_value(to_f32(from_f32<T>(v[0])), to_f32(from_f32<T>(v[ROWS - 1]))));
        }
    }
}

}  // namespace ab2
