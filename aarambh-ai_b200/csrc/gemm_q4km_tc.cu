// Q4_K_M-style block weights (256 values per block, 4-bit codes, f16 scale and minimum,
// crates/aarambh-studio-quant/src/gguf_quant.rs:39-49: w = q * scale + min), bf16 activations, many tokens: the
// prompts and larger batches of a GGUF-loaded model on the 5th-generation tensor cores.
//
//   y[t][n] = sum over blocks b of  scale[n][b] * (sum_k (q[n][k] - 8) x[t][k]) + (min[n][b] + 8 scale[n][b]) * X[t][b],
//
// X the sum of a token's activations over a block.  The codes enter the MMA as exact small integers, around 0 and not from 0 on: the
// two parts would otherwise be sums of up to 16 times the result whose difference it is.  A block is 256
// steps of K, after which its accumulator leaves tensor memory and the scale and the minimum are applied in f32, so
// no weight is rounded.  A first kernel forms X and a copy of the activations whose groups of 8 are ordered
// 0,4,1,5,2,6,3,7, the order in which one shift and one mask take codes out of a word of the reference's layout.
//
// As in the other tcgen05 kernels the 128 channels of a tile are the M dimension of the MMA and NTOK tokens its N
// dimension, one persistent CTA per SM:
//   warp 0       producer of the codes: a TMA tile of 128 channels x one block per slot
//   warp 1       MMA issue; two accumulators, a block each in turn
//   warps 2-9    unpack, two sets of four warps on alternate stages of 64 K-elements, thread = channel; the integers go
//                to tensor memory (through shared memory, which the MMAs read too, the kernel took 5 to 11 % longer)
//   warps 10-17  epilogue, thread = channel and half of the tokens, running sums in registers
//   warp 18      producer of the activation tiles and of X
// With fewer tiles than SMs the blocks of a tile are divided over several CTAs; their f32 sums meet in a reduce pass.
// What bounds it is the unpack and the per-block epilogue (about 450 cycles a stage against the MMA's 257 at 128
// tokens).  14336 x 4096 at 300 tokens: 3329 us on CUDA cores,
// 73 us here (482 TFLOP/s); 3072 x 2048: 421 -> 20 us, at 9 tokens 17 -> 11.
// Every wait on an mbarrier is bounded; on a time-out the CTA records AB2_ERR_TIMEOUT, walks through the rest
// of its work, frees its tensor memory and returns.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "tcgen05_util.cuh"

using namespace ab2;
using namespace ab2::tc;

namespace ab2 {
int device_status_word(int **out);
int device_sm_count();
void launch_splitk_reduce(const float *part, __nv_bfloat16 *y, int M, int N, int ksplit, cudaStream_t s);
namespace {

constexpr int QB_MAX_STAGES = 6, QB_MAX_WSLOTS = 6;
constexpr int QB_A_COLS = 32;              // tensor-memory columns of 64 K-elements: two bf16 per column, a lane per channel
constexpr int QB_WSLOT_BYTES = 128 * 128;  // 128 channels x 256 codes
constexpr int QB_UNPACK_WARPS = 8, QB_EPI_WARPS = 8;
constexpr int QB_OUT_BYTES = QB_EPI_WARPS * 16 * 32 * 2;  // an epilogue warp's 16 tokens x 32 channels on their way out
constexpr int QB_THREADS = (2 + QB_UNPACK_WARPS + QB_EPI_WARPS + 1) * 32;

template <int NTOK>
__host__ __device__ constexpr int qb_stages() { return NTOK > 64 ? 5 : 6; }
template <int NTOK>
__host__ __device__ constexpr int qb_wslots() { return NTOK > 64 ? 3 : NTOK > 32 ? 4 : QB_MAX_WSLOTS; }

struct QbShared {
    uint64_t wfull[QB_MAX_WSLOTS], wempty[QB_MAX_WSLOTS];
    uint64_t full[QB_MAX_STAGES], empty[QB_MAX_STAGES];
    uint64_t accfull[2], accempty[2], xsfull[2];
    uint32_t tmem_base;
    int failed;
    alignas(16) float xsum[2][128];
};

struct QbArgs {
    const uint32_t *params;  // [N][KB]
    const float *xsum;       // [KB][Mp]
    __nv_bfloat16 *y;
    float *part;             // [ksplit][M][N] with a K split
    int N, KB, M, Mp, ksplit;
};

// A warp per (token, block): the block's sum and its activations in the order of the unpacked codes.
__global__ void __launch_bounds__(256) q4km_prepare_kernel(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ xp, float *__restrict__ xsum,
                                                           int M, int Mp, int K) {
    const int b = blockIdx.x, lane = threadIdx.x & 31;
    pdl_wait();
    pdl_launch_dependents();
    for (int t = blockIdx.y * 8 + (threadIdx.x >> 5); t < Mp; t += gridDim.y * 8) {
        float sum = 0.f;
        if (t < M) {
            const size_t at = (size_t)t * K + b * 256 + lane * 8;
            const uint4 v = *reinterpret_cast<const uint4 *>(x + at);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) sum += __uint_as_float(w[j] << 16) + __uint_as_float(w[j] & 0xffff0000u);
            *reinterpret_cast<uint4 *>(xp + at) = make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632),
                                                             __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) xsum[(size_t)b * Mp + t] = sum;
    }
}

template <int NTOK>
__global__ void __launch_bounds__(QB_THREADS, 1)
gemm_q4km_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, QbArgs a, int *status) {
    constexpr int STAGES = qb_stages<NTOK>(), WSLOTS = qb_wslots<NTOK>(), B_BYTES = NTOK * 128;
    constexpr uint32_t ACC_COLS = 2 * NTOK, TMEM_COLS = ACC_COLS + STAGES * QB_A_COLS > 256 ? 512 : 256;
    static_assert(ACC_COLS + STAGES * QB_A_COLS <= 512, "accumulators and operand stages fit");
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NTOK >> 3) << 17) | ((128u >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    uint8_t *b_st = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // [STAGES][B_BYTES]
    uint8_t *w_ring = b_st + STAGES * B_BYTES;                                     // [WSLOTS][QB_WSLOT_BYTES]
    __nv_bfloat16 *stage = (__nv_bfloat16 *)(w_ring + WSLOTS * QB_WSLOT_BYTES);  // [QB_EPI_WARPS][16][32]
    QbShared *sh = (QbShared *)((uint8_t *)stage + QB_OUT_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = (a.N + 127) >> 7, m_tiles = (a.M + NTOK - 1) / NTOK, items = n_tiles * m_tiles * a.ksplit;
    volatile int *failed = &sh->failed;
    // item: (channel tile, token tile, share of the blocks)
    auto item = [&](int it, int &nt, int &mt, int &sp, int &b0, int &b1) {
        sp = it % a.ksplit;
        mt = it / a.ksplit % m_tiles;
        nt = it / a.ksplit / m_tiles;
        b0 = (int)((long long)sp * a.KB / a.ksplit);
        b1 = (int)((long long)(sp + 1) * a.KB / a.ksplit);
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < WSLOTS; ++i) { bar_init(&sh->wfull[i], 1); bar_init(&sh->wempty[i], QB_UNPACK_WARPS); }
        for (int i = 0; i < STAGES; ++i) { bar_init(&sh->full[i], 4 + 1); bar_init(&sh->empty[i], 1); }
        for (int i = 0; i < 2; ++i) { bar_init(&sh->accfull[i], 1); bar_init(&sh->accempty[i], QB_EPI_WARPS); bar_init(&sh->xsfull[i], 1); }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {  // tensor-memory allocation is a whole-warp operation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(sptr(&sh->tmem_base)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    pdl_wait();  // the setup above overlaps the end of the preceding kernel
    pdl_launch_dependents();
    const uint32_t tmem = sh->tmem_base, tmem_a = tmem + ACC_COLS;
    int nt, mt, sp, b0, b1;

    if (warp == 0) {
        // ---------------------------------------------------------- producer of the codes
        if (lane == 0) {
            uint32_t wuse = 0;
            for (int it = blockIdx.x; it < items && !*failed; it += gridDim.x) {
                item(it, nt, mt, sp, b0, b1);
                for (int b = b0; b < b1 && !*failed; ++b, ++wuse) {
                    const int ws = wuse % WSLOTS;
                    if (!bar_wait(&sh->wempty[ws], ((wuse / WSLOTS) & 1) ^ 1, failed)) break;
                    bar_expect_tx(&sh->wfull[ws], QB_WSLOT_BYTES);  // rows past N arrive as zeros and count
                    tma_load_2d(w_ring + ws * QB_WSLOT_BYTES, &wmap, b * 128, nt * 128, &sh->wfull[ws]);
                }
            }
        }
    } else if (warp == QB_THREADS / 32 - 1) {
        // ---------------------------------------------------------- producer of the activation tiles and their sums
        if (lane == 0) {
            uint32_t suse = 0, buse = 0;
            for (int it = blockIdx.x; it < items && !*failed; it += gridDim.x) {
                item(it, nt, mt, sp, b0, b1);
                for (int b = b0; b < b1 && !*failed; ++b, ++buse) {
                    const int ab = buse & 1;
                    if (!bar_wait(&sh->accempty[ab], ((buse >> 1) & 1) ^ 1, failed)) break;
                    bar_expect_tx(&sh->xsfull[ab], NTOK * 4);
                    bulk_copy(sh->xsum[ab], a.xsum + (size_t)b * a.Mp + mt * NTOK, NTOK * 4, &sh->xsfull[ab]);
                    for (int q = 0; q < 4; ++q, ++suse) {
                        const int st = suse % STAGES;
                        if (!bar_wait(&sh->empty[st], ((suse / STAGES) & 1) ^ 1, failed)) break;
                        bar_expect_tx(&sh->full[st], B_BYTES);
                        tma_load_2d(b_st + st * B_BYTES, &xmap, b * 256 + q * 64, mt * NTOK, &sh->full[st]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------- MMA issue
        uint32_t suse = 0, buse = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            item(it, nt, mt, sp, b0, b1);
            for (int b = b0; b < b1; ++b, ++buse) {
                const int ab = buse & 1;
                bar_wait(&sh->accempty[ab], ((buse >> 1) & 1) ^ 1, failed);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                for (int q = 0; q < 4; ++q, ++suse) {
                    const int st = suse % STAGES;
                    warp_wait(&sh->full[st], (suse / STAGES) & 1, failed);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    if (elect_one()) {
                        umma_stage_ts(tmem + (uint32_t)(ab * NTOK), tmem_a + (uint32_t)(st * QB_A_COLS), umma_desc(sptr(b_st + st * B_BYTES)), IDESC, q == 0);
                        umma_commit(&sh->empty[st]);
                        if (q == 3) umma_commit(&sh->accfull[ab]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < 2 + QB_UNPACK_WARPS) {
        // ---------------------------------------------------------- unpack: codes -> bf16 integers
        const int t = (warp & 3) * 32 + lane, set = (warp - 2) >> 2;  // channel: the warp's lanes of tensor memory
        uint32_t wuse = 0;
        uint32_t k_mask = 0x000F000Fu, k_magic = 0x43004300u, k_off = 0xC308C308u;  // -136: code - 8 from 128 + code
        asm volatile("" : "+r"(k_mask), "+r"(k_magic), "+r"(k_off));
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            item(it, nt, mt, sp, b0, b1);
            for (int b = b0; b < b1; ++b, ++wuse) {
                const int ws = wuse % WSLOTS;
                bar_wait(&sh->wfull[ws], (wuse / WSLOTS) & 1, failed);
                // row t of the slot: 256 codes in eight 16-byte chunks, chunk c stored at c ^ (t & 7); the set takes quarters
                // set and set + 2 of the block
                const uint8_t *wrow = w_ring + ws * QB_WSLOT_BYTES + t * 128;
                uint4 raw[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) raw[i] = *reinterpret_cast<const uint4 *>(wrow + (((2 * set + (i & 1) + 4 * (i >> 1)) ^ (t & 7)) << 4));
                const uint32_t held = __reduce_or_sync(0xffffffffu, raw[0].x ^ raw[1].x ^ raw[2].x ^ raw[3].x);
                if (lane == 0) bar_arrive_after(&sh->wempty[ws], held, (uint32_t)a.KB >> 30);
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    const uint32_t suse = 4 * wuse + set + 2 * h;
                    const int st = suse % STAGES;
                    const bool free = warp_wait(&sh->empty[st], ((suse / STAGES) & 1) ^ 1, failed);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    uint32_t o[32];  // two bf16 each
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint4 q4 = h ? raw[2 + (c >> 2)] : raw[c >> 2];
                        const uint32_t word = (c & 3) == 0 ? q4.x : (c & 3) == 1 ? q4.y : (c & 3) == 2 ? q4.z : q4.w;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {  // codes j and j + 4
                            uint32_t v;
                            const uint32_t shv = j ? (word >> (4 * j)) : word;
                            asm("lop3.b32 %0, %1, %2, %3, 0xEA;\n" : "=r"(v) : "r"(shv), "r"(k_mask), "r"(k_magic));
                            o[4 * c + j] = bf16x2_add_(v, k_off);
                        }
                    }
                    tmem_st32(tmem_a + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(st * QB_A_COLS), o);
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0 && free) bar_arrive(&sh->full[st]);
                }
            }
        }
    } else {
        // ---------------------------------------------------------- epilogue
        constexpr int COLS = NTOK / 2;  // tokens of a thread
        const bool aligned = rows_in_16_bytes(a.y, a.N);
        const int quad = warp & 3, half = (warp - 2 - QB_UNPACK_WARPS) >> 2;
        uint32_t buse = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            item(it, nt, mt, sp, b0, b1);
            const int n = nt * 128 + quad * 32 + lane;
            const uint32_t *prm = a.params + (size_t)min(n, a.N - 1) * a.KB;
            float acc[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
            uint32_t next = __ldg(prm + b0);
            for (int b = b0; b < b1; ++b, ++buse) {
                const int ab = buse & 1;
                const uint32_t param = next;
                if (b + 1 < b1) next = __ldg(prm + b + 1);
                bar_wait(&sh->xsfull[ab], (buse >> 1) & 1, failed);
                warp_wait(&sh->accfull[ab], (buse >> 1) & 1, failed);
                const float s = f16_bits_to_f32((uint16_t)(param & 0xffffu)), m = fmaf(8.f, s, f16_bits_to_f32((uint16_t)(param >> 16)));
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const float *xs = sh->xsum[ab] + half * COLS;
                const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(ab * NTOK + half * COLS);
#pragma unroll
                for (int c = 0; c < COLS / 8; ++c) {
                    uint32_t v[8];
                    tmem_ld8(v, taddr + 8 * c);
#pragma unroll
                    for (int j = 0; j < 8; j += 4) {
                        const float4 X = *reinterpret_cast<const float4 *>(xs + 8 * c + j);
                        acc[8 * c + j] += fmaf(s, __uint_as_float(v[j]), m * X.x);
                        acc[8 * c + j + 1] += fmaf(s, __uint_as_float(v[j + 1]), m * X.y);
                        acc[8 * c + j + 2] += fmaf(s, __uint_as_float(v[j + 2]), m * X.z);
                        acc[8 * c + j + 3] += fmaf(s, __uint_as_float(v[j + 3]), m * X.w);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                // the arrival also gives X's slot back: its loads have fed the sums
                uint32_t held = 0;
#pragma unroll
                for (int j = 0; j < COLS; j += 4) held ^= __float_as_uint(acc[j]);
                held = __reduce_or_sync(0xffffffffu, held);
                if (lane == 0) bar_arrive_after(&sh->accempty[ab], held, (uint32_t)a.KB >> 30);
            }
            const int t0 = mt * NTOK + half * COLS;
            if (aligned && a.ksplit == 1) {
                __nv_bfloat16 *out = stage + (warp - 2 - QB_UNPACK_WARPS) * 512;
#pragma unroll
                for (int j = 0; j < COLS; ++j) {
                    out[(j & 15) * 32 + lane] = __float2bfloat16_rn(acc[j]);
                    if ((j & 15) == 15) flush_rows<16>(out, a.y + (size_t)(t0 + j - 15) * a.N + n - lane, a.N, a.M - t0 - (j - 15), a.N - (n - lane), lane);
                }
                continue;
            }
#pragma unroll
            for (int j = 0; j < COLS; ++j)
                if (n < a.N && t0 + j < a.M) {
                    if (a.ksplit > 1) a.part[((size_t)sp * a.M + t0 + j) * a.N + n] = acc[j];
                    else a.y[(size_t)(t0 + j) * a.N + n] = __float2bfloat16_rn(acc[j]);
                }
            __syncwarp();
        }
    }

    // ---- teardown: every warp arrives here (all waits are bounded)
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && sh->failed) atomicExch(status, (int)AB2_ERR_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// Tokens of a tile: one tile of 32 or 64 where it takes all of them; else 128, which unpack a weight for the most tokens.
int qb_tokens(int M) { return M <= 32 ? 32 : M <= 64 ? 64 : 128; }

struct QbPlan {
    int Mp, tiles, ksplit;
    size_t xp_bytes, xs_bytes, part_bytes;
};
QbPlan qb_plan(const ab2_qweight *w, int M, int ntok, bool whole_rows) {
    const int KB = w->K / 256;
    QbPlan p;
    p.Mp = (M + ntok - 1) / ntok * ntok;
    p.tiles = ((w->N + 127) / 128) * (p.Mp / ntok);
    // as many shares of K as make one wave of items, at least two blocks each; the reduce pass stores rows in 16-byte pieces
    p.ksplit = whole_rows ? std::max(1, std::min(std::min(8, KB / 2), device_sm_count() / p.tiles)) : 1;
    p.xp_bytes = ((size_t)M * w->K * 2 + 255) & ~(size_t)255;
    p.xs_bytes = ((size_t)KB * p.Mp * 4 + 255) & ~(size_t)255;
    p.part_bytes = p.ksplit > 1 ? (size_t)p.ksplit * M * w->N * 4 : 0;
    return p;
}

template <int NTOK>
int launch_qb(const ab2_qweight *w, const void *x, int M, void *y, cudaStream_t s) {
    int *status = nullptr;
    int rc = device_status_word(&status);
    if (rc != AB2_OK) return rc;
    const QbPlan p = qb_plan(w, M, NTOK, rows_in_16_bytes(y, w->N));
    const int N = w->N, K = w->K, KB = K / 256, Mp = p.Mp, tiles = p.tiles, sms = device_sm_count();
    const size_t smem = 1024 + qb_stages<NTOK>() * NTOK * 128 + qb_wslots<NTOK>() * QB_WSLOT_BYTES + QB_OUT_BYTES + sizeof(QbShared);
    static_assert(1024 + qb_stages<NTOK>() * NTOK * 128 + qb_wslots<NTOK>() * QB_WSLOT_BYTES + QB_OUT_BYTES + sizeof(QbShared) <= 227 * 1024, "shared memory of a CTA");
    static bool configured[64] = {false};  // the attribute is per device
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    if (!configured[dev]) {
        AB2_CUDA(cudaFuncSetAttribute(gemm_q4km_tc_kernel<NTOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured[dev] = true;
    }
    int ksplit = p.ksplit;
    ScratchLease ws(s);
    if (ksplit > 1 && !ws.take(p.xp_bytes + p.xs_bytes + p.part_bytes)) ksplit = 1;
    if (!ws.ptr && !ws.take(p.xp_bytes + p.xs_bytes)) return AB2_ERR_UNSUPPORTED;  // the CUDA-core kernel needs none
    __nv_bfloat16 *xp = (__nv_bfloat16 *)ws.ptr;
    float *xsum = (float *)((char *)ws.ptr + p.xp_bytes), *part = (float *)((char *)ws.ptr + p.xp_bytes + p.xs_bytes);
    CUtensorMap wmap, xmap;
    rc = make_x_map(&xmap, xp, M, K, NTOK);
    if (rc == AB2_OK) rc = make_bytes_map(&wmap, w->codes, N, K / 2);
    if (rc != AB2_OK) return rc;
    launch_kernel(q4km_prepare_kernel, dim3(KB, std::min((Mp + 7) / 8, 65535)), dim3(256), 0, s, (const __nv_bfloat16 *)x, xp, xsum, M, Mp, K);  // checked with the next
    const QbArgs a = {w->block_params, xsum, (__nv_bfloat16 *)y, part, N, KB, M, Mp, ksplit};
    cudaError_t e = launch_kernel(gemm_q4km_tc_kernel<NTOK>, dim3(std::min(tiles * ksplit, sms)), dim3(QB_THREADS), smem, s, wmap, xmap, a, status);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "Q4_K_M GEMM launch failed: %s", cudaGetErrorString(e));
    if (ksplit > 1) launch_splitk_reduce(part, (__nv_bfloat16 *)y, M, N, ksplit, s);
    AB2_LAUNCH_CHECK();
    return AB2_OK;
}

}  // namespace

bool qlinear_q4km_tc_eligible(const ab2_qweight *w, ab2_dtype dtype) { return w->fmt == FMT_Q4KM && dtype == AB2_BF16 && w->K % 256 == 0; }

// AB2_ERR_UNSUPPORTED where its scratch is not to be had.
int qlinear_q4km_tc(const ab2_qweight *w, const void *x, int M, void *y, cudaStream_t s) {
    switch (qb_tokens(M)) {
    case 32: return launch_qb<32>(w, x, M, y, s);
    case 64: return launch_qb<64>(w, x, M, y, s);
    default: return launch_qb<128>(w, x, M, y, s);
    }
}

// The most that a call of M tokens leases.
size_t qlinear_q4km_tc_scratch(const ab2_qweight *w, int M) {
    const QbPlan p = qb_plan(w, M, qb_tokens(M), w->N % 8 == 0);
    return p.xp_bytes + p.xs_bytes + p.part_bytes;
}

}  // namespace ab2
