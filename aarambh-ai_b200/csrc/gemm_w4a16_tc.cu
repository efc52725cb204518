// W4A16 (group 128, bf16) GEMM for many tokens (prefill, batched decode) on the
// 5th-generation tensor cores: tcgen05.mma with the accumulator in tensor memory.
//
//   Y[M, N] = X[M, K] . W^T,  W packed 4-bit in tile-major blocks (w4a16_layout.cuh)
//
// The product is formed transposed: the 128 output channels of a tile are the M
// dimension of the MMA (operand A = dequantised weights), the tokens its N
// dimension (operand B = activations), so any token count is a legal N and the
// weights are dequantised once per (channel tile, token tile).  One CTA per SM,
// persistent over tiles, warp-specialised:
//   warp 0      producer of the packed weights: one ring slot per quantisation
//               group, lane b issues the bulk copy of 16-channel block b
//   warp 22     producer of the activations: TMA tile loads of X (128-byte
//               swizzle) into the operand-B stages
//   warp 1      allocates tensor memory, issues tcgen05.mma (K = 16 per
//               instruction, 64 per stage), commits stage / accumulator barriers.
//   warps 2-17  dequantise, four sets of four warps on stages of their own; thread = output channel; nibbles -> bf16 (128 + q by
//               one logic op, minus (128 + z) exactly, times the bf16 scale, i.e.
//               the round-to-nearest bf16 of (q - z) * s) written to the
//               operand-A stage in tensor memory, a lane per channel
//   warps 18-21 epilogue: tcgen05.ld of the accumulator, bf16 rows of Y by way of shared memory
// Every wait on an mbarrier is bounded; on a time-out the CTA records
// AB2_ERR_TIMEOUT, walks through the rest of its work, frees its tensor memory and returns.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "tcgen05_util.cuh"
#include "w4a16_layout.cuh"

using namespace ab2;
using namespace ab2::tc;

namespace ab2 {
int device_status_word(int **out);
int device_sm_count();
void launch_splitk_reduce(const float *part, __nv_bfloat16 *y, int M, int N, int ksplit, cudaStream_t s);
namespace {

constexpr int TC_MAX_STAGES = 6, TC_MAX_WSLOTS = 10;
constexpr int TC_BLOCK_WORDS = 272;   // 16 rows x 16 code words + 16 parameter words
constexpr int TC_WSLOT_BYTES = 8 * TC_BLOCK_WORDS * 4;  // 8 row tiles of 16 = 128 channels
constexpr int TC_OUT_BYTES = 4 * 32 * 32 * 2;  // an epilogue warp's 32 tokens x 32 channels on their way out
constexpr int TC_A_COLS = 32;  // tensor-memory columns of 64 K-elements: two bf16 per column, a lane per channel
constexpr int TC_SETS = 4;  // sets of four unpack warps; a set takes every TC_SETS-th stage
constexpr int TC_UNPACK_WARPS = 4 * TC_SETS;
constexpr int TC_THREADS = (2 + TC_UNPACK_WARPS + 4 + 1) * 32;

struct TcShared {
    uint64_t wfull[TC_MAX_WSLOTS], wempty[TC_MAX_WSLOTS];
    uint64_t full[TC_MAX_STAGES], empty[TC_MAX_STAGES];
    uint64_t accfull[2], accempty[2];  // two accumulators: the epilogue of a tile overlaps the next tile's MMAs
    uint32_t tmem_base;
    int failed;
};

// Stages of 64 K-elements: the weight tile in tensor memory, the activation tile in shared memory, with one pair of
// barriers, so that the issuing warp waits once per stage (a wait costs it about 150 cycles even when the stage is
// ready).  A weight tile in shared memory would be written and read there besides the activations, at 256 tokens 104
// KB a stage instead of 72.  256 tokens leave room for one accumulator: the MMAs of a tile wait for the last one's to be stored.
// The slots of packed weights, one quantisation group each, are even in number: a slot is then read by one pair of sets
// only.  With three, a pair could reach its next use of a slot while the group between, the other pair's, was still on
// its way - copies may land out of order - and take the barrier's older phase for the one it waits for.
template <int NTOK>
__host__ __device__ constexpr int tc_stages() { return NTOK > 192 ? 5 : NTOK > 128 ? 4 : 6; }
template <int NTOK>
__host__ __device__ constexpr int tc_wslots() { return NTOK > 192 ? 6 : TC_MAX_WSLOTS; }
template <int NTOK>
__host__ __device__ constexpr int tc_accs() { return NTOK > 192 ? 1 : 2; }
template <int NTOK>
__host__ __device__ constexpr uint32_t tc_cols() { return tc_accs<NTOK>() * NTOK + tc_stages<NTOK>() * TC_A_COLS > 256 ? 512 : 256; }

template <int NTOK>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_w4a16_tc_kernel(const uint32_t *__restrict__ wt, const __grid_constant__ CUtensorMap xmap,
                     __nv_bfloat16 *__restrict__ y, int N, int K, int M, int *status, int ksplit, float *part) {
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
    const int G = K >> 7, tiles16 = (N + 15) >> 4;
    const int n_tiles = (N + 127) >> 7, m_tiles = (M + NTOK - 1) / NTOK;
    // an item is (channel tile, token tile, K split): with fewer tiles than SMs the groups of a tile are
    // divided over `ksplit` CTAs, which leave f32 partial sums in `part` [ksplit][M][N] for a reduce pass
    const int items = n_tiles * m_tiles * ksplit;
#define TC_ITEM(it)                                                                    \
    const int ksp = (it) % ksplit, tile_ = (it) / ksplit;                              \
    const int nt = tile_ / m_tiles, mt = tile_ % m_tiles;                              \
    const int g0 = (int)((long long)ksp * G / ksplit), g1 = (int)((long long)(ksp + 1) * G / ksplit); \
    (void)ksp; (void)nt; (void)mt; (void)g0; (void)g1;
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
        // ---------------------------------------------------------- producer of the packed weights
        // One slot per quantisation group; lane b issues the bulk copy of block b, so the eight
        // copies of a group leave in parallel instead of one after the other from a single thread.
        uint32_t wuse = 0;
        int ok = 1;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            TC_ITEM(it)
            const int nblk = min(8, tiles16 - nt * 8);
            for (int g = g0; g < g1; ++g, ++wuse) {
                const int ws = wuse % TC_WSLOTS;
                if (lane == 0) {
                    ok = bar_wait(&sh->wempty[ws], ((wuse / TC_WSLOTS) & 1) ^ 1, failed) ? 1 : 0;
                    if (ok) bar_expect_tx(&sh->wfull[ws], (uint32_t)nblk * TC_BLOCK_WORDS * 4);
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                if (lane < nblk)
                    bulk_copy(w_ring + ws * TC_WSLOT_BYTES + lane * TC_BLOCK_WORDS * 4,
                              wt + ((size_t)(nt * 8 + lane) * G + g) * TC_BLOCK_WORDS, TC_BLOCK_WORDS * 4, &sh->wfull[ws]);
            }
        }
    } else if (warp == TC_THREADS / 32 - 1) {
        // ---------------------------------------------------------- producer of the activation tiles
        if (lane == 0) {
            uint32_t suse = 0;
            for (int it = blockIdx.x; it < items && !*failed; it += gridDim.x) {
                TC_ITEM(it)
                for (int ks = 2 * g0; ks < 2 * g1 && !*failed; ++ks, ++suse) {
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
            TC_ITEM(it)
            for (int ks = 2 * g0; ks < 2 * g1; ++ks, ++suse) {
                const int st = suse % TC_STAGES;
                warp_wait(&sh->full[st], (suse / TC_STAGES) & 1, failed);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                if (elect_one()) {
                    umma_stage_ts(tacc, tmem_a + (uint32_t)(st * TC_A_COLS), umma_desc(sptr(b_st + st * B_BYTES)), IDESC, ks == 2 * g0);
                    umma_commit(&sh->empty[st]);  // the stage is free when the MMAs retire
                }
                __syncwarp();
            }
            if (elect_one()) umma_commit(&sh->accfull[ab]);
            __syncwarp();
        }
    } else if (warp < 2 + TC_UNPACK_WARPS) {
        // ---------------------------------------------------------- dequantise
        const int t = (warp & 3) * 32 + lane, set = (warp - 2) >> 2;  // channel within the tile: the warp's lanes of tensor memory
        const int blk = t >> 4, r = t & 15, half = set & 1;
        uint32_t gbase = 0;  // groups before this tile
        uint32_t k_mask = 0x000F000Fu, k_magic = 0x43004300u;
        asm volatile("" : "+r"(k_mask), "+r"(k_magic));
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            TC_ITEM(it)
            // the set's groups: every (TC_SETS / 2)-th of the CTA's sequence of groups
            for (uint32_t wuse = gbase + ((set >> 1) + TC_SETS - gbase % (TC_SETS / 2)) % (TC_SETS / 2); wuse < gbase + (uint32_t)(g1 - g0); wuse += TC_SETS / 2) {
                const int ws = wuse % TC_WSLOTS;
                bar_wait(&sh->wfull[ws], (wuse / TC_WSLOTS) & 1, failed);
                const uint32_t *bw = (const uint32_t *)(w_ring + ws * TC_WSLOT_BYTES) + blk * TC_BLOCK_WORDS;
                const uint4 pw[2] = {*reinterpret_cast<const uint4 *>(bw + r * 16 + half * 8), *reinterpret_cast<const uint4 *>(bw + r * 16 + half * 8 + 4)};
                const uint32_t pr = bw[256 + r];
                // one arrival per warp, fed by the loads of all its lanes
                const uint32_t held = __reduce_or_sync(0xffffffffu, pw[0].x ^ pw[1].x ^ pr);
                if (lane == 0) bar_arrive_after(&sh->wempty[ws], held, (uint32_t)K & 1u);
                const uint32_t sc2 = __byte_perm(pr, pr, 0x1010);  // bf16x2 (scale, scale)
                const uint32_t nz2 = __byte_perm(pr, pr, 0x3232);  // bf16x2 -(128 + z)
                const uint32_t suse = 2 * wuse + half;
                const int s = suse % TC_STAGES;
                const bool free = warp_wait(&sh->empty[s], ((suse / TC_STAGES) & 1) ^ 1, failed);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                uint32_t o[32];  // two bf16 each
#pragma unroll
                for (int c = 0; c < 8; ++c) {  // chunk c = 8 consecutive k = one code word
                    const uint4 q4 = pw[c >> 2];
                    const uint32_t word = (c & 3) == 0 ? q4.x : (c & 3) == 1 ? q4.y : (c & 3) == 2 ? q4.z : q4.w;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t v;
                        const uint32_t shv = j ? (word >> (4 * j)) : word;
                        asm("lop3.b32 %0, %1, %2, %3, 0xEA;\n" : "=r"(v) : "r"(shv), "r"(k_mask), "r"(k_magic));
                        o[4 * c + j] = bf16x2_mul_(bf16x2_add_(v, nz2), sc2);
                    }
                }
                tmem_st32(tmem_a + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(s * TC_A_COLS), o);
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0 && free) bar_arrive(&sh->full[s]);
            }
            gbase += (uint32_t)(g1 - g0);
        }
    } else if (warp < TC_THREADS / 32 - 1) {
        // ---------------------------------------------------------- epilogue
        const int quad = warp & 3;
        const bool aligned = rows_in_16_bytes(y, N);
        uint32_t tuse = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++tuse) {
            TC_ITEM(it)
            const int ab = tuse % ACCS;
            bar_wait(&sh->accfull[ab], (tuse / ACCS) & 1, failed);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int n = nt * 128 + quad * 32 + lane;
#pragma unroll 1
            for (int c = 0; c < NTOK / 32 && mt * NTOK + c * 32 < M; ++c) {
                uint32_t v[32];
                const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(ab * NTOK + c * 32);
                __syncwarp();  // the tensor-memory load is a whole-warp operation
                tmem_ld32(v, taddr);
                if (ksplit > 1) {  // a split is chosen for rows_in_16_bytes only
                    float *out = reinterpret_cast<float *>(stage + quad * 1024);
                    const int tok = mt * NTOK + c * 32, n0 = nt * 128 + quad * 32;
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        out[(j & 15) * 32 + lane] = __uint_as_float(v[j]);
                        if ((j & 15) == 15)
                            flush_rows_f32<16>(out, [&](int i) { return part + ((size_t)ksp * M + tok + j - 15 + i) * N + n0; }, M - tok - (j - 15), N - n0, lane);
                    }
                } else if (aligned) {
                    __nv_bfloat16 *out = stage + quad * 1024;
#pragma unroll
                    for (int j = 0; j < 32; ++j) out[j * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[j]));
                    const int tok = mt * NTOK + c * 32, n0 = nt * 128 + quad * 32;
                    flush_rows<32>(out, y + (size_t)tok * N + n0, N, M - tok, N - n0, lane);
                } else if (n < N) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const int tok = mt * NTOK + c * 32 + j;
                        if (tok < M) {
                            y[(size_t)tok * N + n] = __float2bfloat16_rn(__uint_as_float(v[j]));
                        }
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

// y[i] = bf16(sum over splits of part[s][i]): eight elements per thread
__global__ void splitk_reduce_kernel(const float *__restrict__ part, __nv_bfloat16 *__restrict__ y, size_t n8, size_t stride, int ksplit) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n8) return;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < ksplit; ++s) {
        const float4 a = reinterpret_cast<const float4 *>(part + s * stride)[2 * i];
        const float4 b = reinterpret_cast<const float4 *>(part + s * stride)[2 * i + 1];
        acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
        acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        o[j] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(acc[2 * j])) |
               ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(acc[2 * j + 1])) << 16);
    reinterpret_cast<uint4 *>(y)[i] = make_uint4(o[0], o[1], o[2], o[3]);
}

constexpr size_t TC_SPLIT_MAX_BYTES = (size_t)128 << 20;

template <int NTOK>
int launch_tc(const ab2_qweight *w, const void *x, int M, void *y, int ksplit, float *part, cudaStream_t s) {
    int *status = nullptr;
    int rc = device_status_word(&status);
    if (rc != AB2_OK) return rc;
    CUtensorMap map;
    rc = make_x_map(&map, x, M, w->K, NTOK);
    if (rc != AB2_OK) return rc;
    const size_t smem = 1024 + tc_stages<NTOK>() * NTOK * 128 + tc_wslots<NTOK>() * TC_WSLOT_BYTES + TC_OUT_BYTES + sizeof(TcShared);
    static bool configured[64] = {false};  // the attribute is per device
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    if (!configured[dev]) {
        AB2_CUDA(cudaFuncSetAttribute(gemm_w4a16_tc_kernel<NTOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured[dev] = true;
    }
    const int tiles = ((w->N + 127) / 128) * ((M + NTOK - 1) / NTOK);
    const int items = tiles * ksplit;
    const int grid = std::min(items, device_sm_count());
    cudaError_t e = launch_kernel(gemm_w4a16_tc_kernel<NTOK>, dim3(grid), dim3(TC_THREADS), smem, s, (const uint32_t *)w->codes, map, (__nv_bfloat16 *)y, w->N, w->K, M,
                                  status, ksplit, part);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "W4A16 GEMM launch failed: %s", cudaGetErrorString(e));
    if (ksplit > 1) launch_splitk_reduce(part, (__nv_bfloat16 *)y, M, w->N, ksplit, s);
    AB2_LAUNCH_CHECK();
    return AB2_OK;
}

}  // namespace

// y[M][N] = bf16(sum of the splits' part[ksplit][M][N]); rows_in_16_bytes(y, N)
void launch_splitk_reduce(const float *part, __nv_bfloat16 *y, int M, int N, int ksplit, cudaStream_t s) {
    const size_t n8 = (size_t)M * N / 8;
    launch_kernel(splitk_reduce_kernel, dim3((unsigned)((n8 + 255) / 256)), dim3(256), 0, s, part, y, n8, (size_t)M * N, ksplit);  // checked by the caller
}

// Y[M][N] = X[M][K] . W^T on the tcgen05 path (W4A16, group 128, bf16).
int qlinear_w4a16_tc(const ab2_qweight *w, const void *x, int M, void *y, cudaStream_t s) {
    AB2_REQUIRE(((uintptr_t)x & 15) == 0 && (w->K * 2) % 16 == 0, AB2_ERR_BAD_ALIGN, "activations must be 16-byte aligned");
    // Measured: rounds of 19.7 / 22.3 / 27.1 us of tiles of 128 / 192 / 256 tokens over K = 4096 (28672 channels, 2048 tokens),
    // 68 / 73 / 85 over K = 14336; a tile of 32 takes what one of 128 does but for its stores.  Splitting K (few tiles:
    // 512 tokens on the 4096 x 14336 weight are 64 of 256) needs rows that the reduce pass can store in 16-byte
    // pieces and a workspace; a recorded launch, in whose graph that would be memory nodes, goes without.
    static const GemmTileCost costs[] = {{32, 0.5, 0.58}, {128, 1.0, 0.605}, {192, 2.2, 0.63}, {256, 4.0, 0.72}};
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool recorded = cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
    static const bool no_split = getenv("AB2_GEMM_NO_SPLITK") != nullptr;
    const bool split = !recorded && !no_split && rows_in_16_bytes(y, w->N) && (size_t)4 * M * w->N * sizeof(float) <= TC_SPLIT_MAX_BYTES;
    GemmTileChoice c = choose_gemm_tile(costs, M, w->N, w->K / 128, device_sm_count(), split ? 4 : 1);
    ScratchLease ws(s);
    if (c.ksplit > 1 && !ws.take((size_t)c.ksplit * M * w->N * sizeof(float)))
        c = choose_gemm_tile(costs, M, w->N, w->K / 128, device_sm_count(), 1);
    float *part = (float *)ws.ptr;
    switch (c.ntok) {
    case 32: return launch_tc<32>(w, x, M, y, c.ksplit, part, s);
    case 128: return launch_tc<128>(w, x, M, y, c.ksplit, part, s);
    case 192: return launch_tc<192>(w, x, M, y, c.ksplit, part, s);
    default: return launch_tc<256>(w, x, M, y, c.ksplit, part, s);
    }
}

}  // namespace ab2
