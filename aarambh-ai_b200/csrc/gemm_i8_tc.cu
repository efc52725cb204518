// W8A16 GEMM for many tokens (prefill) on the 5th-generation tensor cores: INT8 symmetric
// weights with one f32 scale per output channel (per-output-channel absmax,
// crates/aarambh-studio-quant/src/qat.rs:140-169; a per-tensor scale, absmax.rs:7-24, is the same
// with the scale replicated; the reference dequantises such weights at load,
// crates/aarambh-studio-weights/src/gguf.rs:187-212, and multiplies dense), bf16 activations.
//
//   Y[M, N] = X[M, K] . W^T,   W = codes[N][K] (int8, row-major) * scale[N]
//
// Same skeleton as the W4A16 kernel (gemm_w4a16_tc.cu): the 128 output channels of a tile are the
// M dimension of tcgen05.mma, the tokens its N dimension, one persistent CTA per SM with
// specialised warps.  What differs:
//   warp 0      one lane loads a 128-channel x 128-K tile of codes per ring slot with one TMA
//               tile copy (128-byte swizzle, so that the row-per-thread reads below do not
//               collide on shared-memory banks)
//   warps 2-17  thread = channel: two codes at a time go into the low bytes of 16-bit halves (PRMT); the low
//               7 bits and the sign bit are each the mantissa of a bf16 between 128 and 256 (two logic ops),
//               whose difference is the code, exactly.  The codes enter the MMA unscaled;
//   warps 18-21 the epilogue multiplies the f32 accumulator by the channel's f32 scale - the
//               product is rounded once, where the reference rounds q * scale to the model
//               dtype before its matmul.
// Every wait on an mbarrier is bounded; on a time-out the CTA records AB2_ERR_TIMEOUT, walks
// through the rest of its work, frees its tensor memory and returns.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "tcgen05_util.cuh"

using namespace ab2;
using namespace ab2::tc;

namespace ab2 {
int device_status_word(int **out);
int device_sm_count();
namespace {

constexpr int TC_MAX_STAGES = 6, TC_MAX_WSLOTS = 6;
constexpr int TC_WSLOT_BYTES = 128 * 128;  // 128 channels x 128 codes
constexpr int TC_OUT_BYTES = 4 * 32 * 32 * 2;  // an epilogue warp's 32 tokens x 32 channels on their way out
constexpr int TC_A_COLS = 32;  // tensor-memory columns of 64 K-elements: two bf16 per column, a lane per channel
constexpr int TC_SETS = 4;  // sets of four convert warps on stages of their own
constexpr int TC_THREADS = (2 + 4 * TC_SETS + 4 + 1) * 32;  // weight producer, MMA, convert, epilogue, activation producer

struct TcShared {
    uint64_t wfull[TC_MAX_WSLOTS], wempty[TC_MAX_WSLOTS];
    uint64_t full[TC_MAX_STAGES], empty[TC_MAX_STAGES];
    uint64_t accfull[2], accempty[2];  // two accumulators: the epilogue of a tile overlaps the next tile's MMAs
    uint32_t tmem_base;
    int failed;
};

// Stages of 64 K-elements: the weight tile in tensor memory, the activation tile in shared memory, with one pair of
// barriers, so that the issuing warp waits once per stage (a wait costs it about 150 cycles even when the stage is
// ready).  A weight tile in shared memory would be written and read there besides the activations, at 256 tokens 112
// KB a stage instead of 80.  256 tokens leave room for one accumulator: the MMAs of a tile wait for the last one's to be stored.
// The slots hold 128 channels x 128 codes each.
template <int NTOK>
__host__ __device__ constexpr int tc_stages() { return NTOK > 192 ? 5 : NTOK > 128 ? 4 : 6; }
template <int NTOK>
__host__ __device__ constexpr int tc_wslots() { return NTOK > 192 ? 2 : TC_MAX_WSLOTS; }
template <int NTOK>
__host__ __device__ constexpr int tc_accs() { return NTOK > 192 ? 1 : 2; }
template <int NTOK>
__host__ __device__ constexpr uint32_t tc_cols() { return tc_accs<NTOK>() * NTOK + tc_stages<NTOK>() * TC_A_COLS > 256 ? 512 : 256; }

template <int NTOK>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_i8_tc_kernel(const __grid_constant__ CUtensorMap wmap, const float *__restrict__ scales,
                  const __grid_constant__ CUtensorMap xmap, __nv_bfloat16 *__restrict__ y, int N, int K, int M, int *status) {
    constexpr int B_BYTES = NTOK * 128;
    constexpr int TC_STAGES = tc_stages<NTOK>(), TC_WSLOTS = tc_wslots<NTOK>(), ACCS = tc_accs<NTOK>();
    static_assert(ACCS * NTOK + TC_STAGES * TC_A_COLS <= 512, "tensor memory");
    static_assert(TC_WSLOTS % (TC_SETS / 2) == 0 && TC_STAGES >= TC_SETS, "one pair of sets per slot; no set a lap ahead of a stage");
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NTOK >> 3) << 17) | ((128u >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *b_st = smem;                            // [TC_STAGES][B_BYTES]
    uint8_t *w_ring = b_st + TC_STAGES * B_BYTES;    // [TC_WSLOTS][TC_WSLOT_BYTES]
    __nv_bfloat16 *stage = (__nv_bfloat16 *)(w_ring + TC_WSLOTS * TC_WSLOT_BYTES);  // [4 epilogue warps][32 tokens][32 channels]
    TcShared *sh = (TcShared *)((uint8_t *)stage + TC_OUT_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = K >> 7;
    const int n_tiles = (N + 127) >> 7, m_tiles = (M + NTOK - 1) / NTOK;
    const int items = n_tiles * m_tiles;
    volatile int *failed = &sh->failed;

    if (threadIdx.x == 0) {
        for (int i = 0; i < TC_WSLOTS; ++i) { bar_init(&sh->wfull[i], 1); bar_init(&sh->wempty[i], 8); }
        for (int i = 0; i < TC_STAGES; ++i) { bar_init(&sh->full[i], 4 + 1); bar_init(&sh->empty[i], 1); }
        for (int i = 0; i < 2; ++i) { bar_init(&sh->accfull[i], 1); bar_init(&sh->accempty[i], 4); }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {  // tensor-memory allocation is a whole-warp operation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(sptr(&sh->tmem_base)), "r"(tc_cols<NTOK>()));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    pdl_wait();  // the setup above overlaps the end of the preceding kernel
    pdl_launch_dependents();
    const uint32_t tmem = sh->tmem_base, tmem_a = tmem + (uint32_t)(ACCS * NTOK);

    if (warp == 0) {
        // ---------------------------------------------------------- producer of the codes
        if (lane == 0) {
            uint32_t wuse = 0;
            for (int it = blockIdx.x; it < items && !*failed; it += gridDim.x) {
                const int nt = it / m_tiles;
                for (int g = 0; g < G && !*failed; ++g, ++wuse) {
                    const int ws = wuse % TC_WSLOTS;
                    if (!bar_wait(&sh->wempty[ws], ((wuse / TC_WSLOTS) & 1) ^ 1, failed)) break;
                    bar_expect_tx(&sh->wfull[ws], TC_WSLOT_BYTES);  // rows past N arrive as zeros and count
                    tma_load_2d(w_ring + ws * TC_WSLOT_BYTES, &wmap, g * 128, nt * 128, &sh->wfull[ws]);
                }
            }
        }
    } else if (warp == TC_THREADS / 32 - 1) {
        // ---------------------------------------------------------- producer of the activation tiles
        if (lane == 0) {
            uint32_t suse = 0;
            for (int it = blockIdx.x; it < items && !*failed; it += gridDim.x) {
                const int mt = it % m_tiles;
                for (int ks = 0; ks < 2 * G && !*failed; ++ks, ++suse) {
                    const int st = suse % TC_STAGES;
                    if (!bar_wait(&sh->empty[st], ((suse / TC_STAGES) & 1) ^ 1, failed)) break;
                    bar_expect_tx(&sh->full[st], B_BYTES);
                    tma_load_2d(b_st + st * B_BYTES, &xmap, ks * 64, mt * NTOK, &sh->full[st]);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------- MMA issue
        uint32_t suse = 0, tuse = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++tuse) {
            const int ab = tuse % ACCS;
            bar_wait(&sh->accempty[ab], ((tuse / ACCS) & 1) ^ 1, failed);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t tacc = tmem + (uint32_t)(ab * NTOK);
            for (int ks = 0; ks < 2 * G; ++ks, ++suse) {
                const int st = suse % TC_STAGES;
                warp_wait(&sh->full[st], (suse / TC_STAGES) & 1, failed);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                if (elect_one()) {
                    umma_stage_ts(tacc, tmem_a + (uint32_t)(st * TC_A_COLS), umma_desc(sptr(b_st + st * B_BYTES)), IDESC, ks == 0);
                    umma_commit(&sh->empty[st]);  // the stage is free when the MMAs retire
                }
                __syncwarp();
            }
            if (elect_one()) umma_commit(&sh->accfull[ab]);
            __syncwarp();
        }
    } else if (warp < 2 + 4 * TC_SETS) {
        // ---------------------------------------------------------- codes -> bf16
        // a set of four warps takes the same half (64 K-elements, one stage) of every second group
        const int t = (warp & 3) * 32 + lane, set = (warp - 2) >> 2, half = set & 1;  // channel: the warp's lanes of tensor memory
        uint32_t gbase = 0;  // groups before this tile
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            for (uint32_t wuse = gbase + ((set >> 1) + TC_SETS - gbase % (TC_SETS / 2)) % (TC_SETS / 2); wuse < gbase + (uint32_t)G; wuse += TC_SETS / 2) {
                const int ws = wuse % TC_WSLOTS;
                bar_wait(&sh->wfull[ws], (wuse / TC_WSLOTS) & 1, failed);
                // row t of the slot: 128 codes in eight 16-byte chunks, chunk c stored at c ^ (t & 7)
                const uint8_t *wrow = w_ring + ws * TC_WSLOT_BYTES + t * 128;
                uint4 raw[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) raw[i] = *reinterpret_cast<const uint4 *>(wrow + (((4 * half + i) ^ (t & 7)) << 4));
                // one arrival per warp, fed by the loads of all its lanes
                const uint32_t held = __reduce_or_sync(0xffffffffu, raw[0].x ^ raw[1].x ^ raw[2].x ^ raw[3].x);
                if (lane == 0) bar_arrive_after(&sh->wempty[ws], held, (uint32_t)K & 1u);
                const uint32_t suse = 2 * wuse + half;
                const int s = suse % TC_STAGES;
                const bool free = warp_wait(&sh->empty[s], ((suse / TC_STAGES) & 1) ^ 1, failed);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                uint32_t o[32];  // two bf16 each
#pragma unroll
                for (int i = 0; i < 4; ++i) {  // 16 codes
                    const uint32_t w4[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        // two codes into the low bytes of 16-bit halves; code = (128 + its low 7 bits) - (128 + its
                        // sign's 128), both of which are a bf16 with those bits as mantissa: exact
                        const uint32_t p = __byte_perm(w4[j >> 1], 0u, j & 1 ? 0x4342 : 0x4140);
                        o[8 * i + j] = bf16x2_add_((p & 0x007F007Fu) | 0x43004300u, (p & 0x00800080u) | 0xC300C300u);
                    }
                }
                tmem_st32(tmem_a + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(s * TC_A_COLS), o);
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0 && free) bar_arrive(&sh->full[s]);
            }
            gbase += (uint32_t)G;
        }
    } else if (warp < TC_THREADS / 32 - 1) {
        // ---------------------------------------------------------- epilogue
        const int quad = warp & 3;
        const bool aligned = rows_in_16_bytes(y, N);
        uint32_t tuse = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++tuse) {
            const int nt = it / m_tiles, mt = it % m_tiles;
            const int ab = tuse % ACCS;
            bar_wait(&sh->accfull[ab], (tuse / ACCS) & 1, failed);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int n = nt * 128 + quad * 32 + lane;
            const float sc = n < N ? __ldg(scales + n) : 0.f;
#pragma unroll 1
            for (int c = 0; c < NTOK / 32 && mt * NTOK + c * 32 < M; ++c) {
                uint32_t v[32];
                const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(ab * NTOK + c * 32);
                __syncwarp();  // the tensor-memory load is a whole-warp operation
                tmem_ld32(v, taddr);
                if (aligned) {
                    __nv_bfloat16 *out = stage + quad * 1024;
#pragma unroll
                    for (int j = 0; j < 32; ++j) out[j * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[j]) * sc);
                    const int tok = mt * NTOK + c * 32, n0 = nt * 128 + quad * 32;
                    flush_rows<32>(out, y + (size_t)tok * N + n0, N, M - tok, N - n0, lane);
                } else if (n < N) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const int tok = mt * NTOK + c * 32 + j;
                        if (tok < M) y[(size_t)tok * N + n] = __float2bfloat16_rn(__uint_as_float(v[j]) * sc);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&sh->accempty[ab]);
        }
    }

    // ---- teardown: every warp arrives here (all waits are bounded)
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && sh->failed) atomicExch(status, (int)AB2_ERR_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tc_cols<NTOK>()));
    }
}

template <int NTOK>
int launch_i8_tc(const ab2_qweight *w, const void *x, int M, void *y, cudaStream_t s) {
    int *status = nullptr;
    int rc = device_status_word(&status);
    if (rc != AB2_OK) return rc;
    CUtensorMap xmap, wmap;
    rc = make_x_map(&xmap, x, M, w->K, NTOK);
    if (rc != AB2_OK) return rc;
    rc = make_bytes_map(&wmap, w->codes, w->N, w->K);
    if (rc != AB2_OK) return rc;
    const size_t smem = 1024 + tc_stages<NTOK>() * NTOK * 128 + tc_wslots<NTOK>() * TC_WSLOT_BYTES + TC_OUT_BYTES + sizeof(TcShared);
    static bool configured[64] = {false};  // the attribute is per device
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    if (!configured[dev]) {
        AB2_CUDA(cudaFuncSetAttribute(gemm_i8_tc_kernel<NTOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured[dev] = true;
    }
    const int items = ((w->N + 127) / 128) * ((M + NTOK - 1) / NTOK);
    const int grid = std::min(items, device_sm_count());
    cudaError_t e = launch_kernel(gemm_i8_tc_kernel<NTOK>, dim3(grid), dim3(TC_THREADS), smem, s, wmap, (const float *)w->scales, xmap, (__nv_bfloat16 *)y, w->N, w->K, M, status);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "INT8 GEMM launch failed: %s", cudaGetErrorString(e));
    AB2_LAUNCH_CHECK();
    return AB2_OK;
}

}  // namespace

// Whether the tensor-core path serves this weight and token count: INT8 codes whose rows start on
// 16-byte boundaries, K in whole 128-element slots.
bool qlinear_i8_tc_eligible(const ab2_qweight *w, ab2_dtype dtype, int M) {
    return w->fmt == FMT_I8 && dtype == AB2_BF16 && M > 8 && w->K % 128 == 0 && ((uintptr_t)w->codes & 15) == 0;
}

// Y[M][N] = X[M][K] . W^T on the tcgen05 path (INT8 codes, f32 scale per channel, bf16 activations).
int qlinear_i8_tc(const ab2_qweight *w, const void *x, int M, void *y, cudaStream_t s) {
    AB2_REQUIRE(((uintptr_t)x & 15) == 0, AB2_ERR_BAD_ALIGN, "activations must be 16-byte aligned");
    // Measured: rounds of 18 / 21 / 28 us of tiles of 128 / 192 / 256 tokens over K = 4096, 61 / 72 / 86 over K = 14336; a
    // tile of 32 takes what one of 128 does but for its stores.
    static const GemmTileCost costs[] = {{32, 0.5, 0.53}, {128, 1.0, 0.54}, {192, 1.5, 0.62}, {256, 6.0, 0.70}};
    switch (choose_gemm_tile(costs, M, w->N, w->K / 128, device_sm_count(), 1).ntok) {
    case 32: return launch_i8_tc<32>(w, x, M, y, s);
    case 128: return launch_i8_tc<128>(w, x, M, y, s);
    case 192: return launch_i8_tc<192>(w, x, M, y, s);
    default: return launch_i8_tc<256>(w, x, M, y, s);
    }
}

}  // namespace ab2
