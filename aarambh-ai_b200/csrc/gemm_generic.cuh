// Fused dequantise + GEMM on CUDA cores with f32 arithmetic, for every weight format and activation type: what
// gemv_generic.cuh computes, for more tokens than a warp per row serves well.  A CTA owns TM tokens x TN channels;
// weights are formed exactly as there and meet the activations in shared memory, 32 columns at a time, the next
// 32 on their way in registers meanwhile.
//
// Bound by f32 FMA where the tiles fill the machine, by the latency of its few steps where they do not (a decoder of
// width 384 has 12 steps).  The 24 linears of the 6-layer f32 decoder at 200 tokens (Q4_K_M-style): 3497 us by a warp per row,
// 478 us here.
// Each 32 columns are summed apart and then added, so the longest chain of additions is K / 32 + 32.
#pragma once

#include "gemv_generic.cuh"

namespace ab2 {

constexpr int GG_TK = 32;

template <int FMT, typename T, int TM, int TN>
__global__ void __launch_bounds__(TM * TN / 16) gemm_generic_kernel(GemvArgs a, const T *__restrict__ x, T *__restrict__ y, int M) {
    constexpr int THREADS = TM * TN / 16;              // 4 x 4 outputs each
    constexpr int WV = TN * (GG_TK / 8) / THREADS, XV = TM * (GG_TK / 8) / THREADS;  // words of 8 per thread and step
    static_assert(WV * THREADS == TN * GG_TK / 8 && XV * THREADS == TM * GG_TK / 8, "whole words per thread");
    __shared__ __align__(16) float xs[GG_TK][TM + 4], ws[GG_TK][TN + 4];
    const int tid = threadIdx.x, n0 = blockIdx.x * TN;
    const int words = a.K >> 3, steps = (words + GG_TK / 8 - 1) / (GG_TK / 8);
    const int tx = tid % (TN / 4), ty = tid / (TN / 4);
    for (int m0 = blockIdx.y * TM; m0 < M; m0 += gridDim.y * TM) {  // once, but for more tokens than a grid has rows of tiles
        float wr[WV][8], xr[XV][8];
        // a thread fetches word `i % 4` of row `i / 4`; what lies outside is zero
        auto fetch = [&](int step) {
#pragma unroll
            for (int u = 0; u < WV; ++u) {
                const int i = tid + u * THREADS, word = step * (GG_TK / 8) + i % (GG_TK / 8), n = n0 + i / (GG_TK / 8);
                if (word < words && n < a.N) dequant_word<FMT>(a, n, word, wr[u]);
                else
#pragma unroll
                    for (int j = 0; j < 8; ++j) wr[u][j] = 0.f;
            }
#pragma unroll
            for (int u = 0; u < XV; ++u) {
                const int i = tid + u * THREADS, word = step * (GG_TK / 8) + i % (GG_TK / 8), m = m0 + i / (GG_TK / 8);
                if (word < words && m < M) Vec8<T>::load(x + (size_t)m * a.K + (size_t)word * 8, xr[u]);
                else
#pragma unroll
                    for (int j = 0; j < 8; ++j) xr[u][j] = 0.f;
            }
        };
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
        fetch(0);
        for (int step = 0; step < steps; ++step) {
#pragma unroll
            for (int u = 0; u < WV; ++u)
#pragma unroll
                for (int j = 0; j < 8; ++j) ws[((tid + u * THREADS) % (GG_TK / 8)) * 8 + j][(tid + u * THREADS) / (GG_TK / 8)] = wr[u][j];
#pragma unroll
            for (int u = 0; u < XV; ++u)
#pragma unroll
                for (int j = 0; j < 8; ++j) xs[((tid + u * THREADS) % (GG_TK / 8)) * 8 + j][(tid + u * THREADS) / (GG_TK / 8)] = xr[u][j];
            __syncthreads();
            if (step + 1 < steps) fetch(step + 1);
            float part[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[i][j] = 0.f;
#pragma unroll
            for (int k = 0; k < GG_TK; ++k) {
                const float4 xv = *reinterpret_cast<const float4 *>(&xs[k][ty * 4]), wv = *reinterpret_cast<const float4 *>(&ws[k][tx * 4]);
                const float xa[4] = {xv.x, xv.y, xv.z, xv.w}, wa[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) part[i][j] = fmaf(xa[i], wa[j], part[i][j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j];
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
                if (m < M && n < a.N) y[(size_t)m * a.N + n] = from_f32<T>(acc[i][j]);
            }
    }
}

}  // namespace ab2
