// bf16 linears of 5 to 32 tokens on the 5th-generation tensor cores: y = epilogue(x W^T) and act = glu(x Wg^T, x Wu^T).
// Every weight crosses HBM once, and the activations the chip once per 128 output channels (the GEMV's CTAs of 16 channels
// read them eight times as often, which bound it: 32 tokens x 2048 are as many bytes as its weights).
//
// The 128 output channels of a tile are the M dimension of tcgen05.mma, the tokens (padded to 16 or 32) its N dimension.
// A unit is a tile's next 64 of K: 16 KB of weights (gate and up: 32) and 2 or 4 KB of activations.  One CTA per SM:
//   warp 0      weights (TMA, 128-byte swizzle, requests of 256 bytes to DRAM), from before the wait on the preceding kernel on
//   warp 1      MMA issue (one elected thread), two accumulators in tensor memory
//   warps 2-9   epilogue: two per tensor-memory quadrant, each for 16 tokens
//   warp 10     activations (TMA, boxes of 16 rows)
//
// Small weights (tiles for at most half of the SMs) have a cluster of CTAs per tile, which deal its K out.  Each CTA writes its f32
// sums of a share of the tokens into the shared memory of the CTA that finishes that share, and adds up what the others
// wrote to its own, in the order of K.  (Over global memory, with one CTA adding the parts of 9 to 18, the chain of fence,
// counter and reads took 14 to 19 us at 2048 x 2048 where this takes 10.)  The cluster is the largest of which enough run
// at once: 16 of 8 CTAs do not, and 128 CTAs in two rounds took 14.6 us.
//
// Larger weights: every CTA takes whole tiles where the last round of tiles is nearly full (or one round uses 96 SMs or more,
// enough to draw on all of HBM); else the units of all tiles are one sequence of which it takes a contiguous range, and a
// tile cut by a range's end is finished by the CTA that arrives last: f32 parts wait in a slot of each contributor, a
// counter per tile tells who is last, and the parts are added in the contributors' order.
//
// What bounds it: HBM for large weights (0.8 of the copy rate and 9 us a launch alone); for small ones the chain of launch,
// first activations, products, exchange.  us, launches one after another over cold weights (channels x K), GEMV -> this kernel, 9 / 32
// tokens: 4096 x 14336 30 / 46 -> 26 / 27; 14336 x 4096 34 / 56 -> 26 / 29; 32000 x 4096 58 / 98 -> 48 / 52.
// With requests of 128 bytes to DRAM 32000 x 4096 took 3 us longer.
// Built, measured and not kept: the experts' linears of a mixture in this form (units of all experts in one sequence, the
// activations of all tokens multiplied and the pairs' columns picked from tensor memory): 8 rows x 8 layers of 32
// experts 6170 -> 6370 us for 8 steps, 32 rows of the latent stack 7940 -> 8160.
// Every wait on an mbarrier is bounded; on a time-out the CTA records AB2_ERR_TIMEOUT, walks through the rest of its
// work (which brings the counters back to zero), frees its tensor memory and returns.
#include <cuda.h>

#include <algorithm>

#include "gemv_w4a16_mma.cuh"
#include "linear_bf16.cuh"
#include "tcgen05_util.cuh"

using namespace ab2;
using namespace ab2::tc;

namespace ab2 {
int device_status_word(int **out);
int device_sm_count();
namespace {

constexpr int GF_TOK = 32, GF_EPI_WARPS = 8, GF_THREADS = (3 + GF_EPI_WARPS) * 32;
constexpr int GF_W_BYTES = 128 * 128, GF_X_BYTES = GF_TOK * 128, GF_BOX_ROWS = 16;
// 184 KB: what is left of an SM takes the CTAs of the short kernels before, so that the weights' copies start during them
constexpr int GF_RING_BYTES = 184 * 1024;
constexpr int GF_MAX_STAGES = 9;

struct GfShared {
    uint64_t full[GF_MAX_STAGES], empty[GF_MAX_STAGES];
    uint64_t accfull[2], accempty[2], parts;
    uint32_t tmem_base;
    int failed, last;
};

template <int MODE> __host__ __device__ constexpr bool gf_dual() { return MODE == LIN_GLU; }
// The cluster form: CTAs of a cluster share one tile and hand their parts over in shared memory, PER x 16 KB of each.
constexpr int GF_MAX_CLUSTER = 8;
template <int MODE> __host__ __device__ constexpr int gf_stage_bytes() { return (gf_dual<MODE>() ? 2 : 1) * GF_W_BYTES + GF_X_BYTES; }
template <int MODE, bool CLUSTER> __host__ __device__ constexpr int gf_part_bytes() { return CLUSTER ? (gf_dual<MODE>() ? 2 : 1) * GF_TOK * 128 * 4 : 0; }
template <int MODE, bool CLUSTER> __host__ __device__ constexpr int gf_stages() { return (GF_RING_BYTES - gf_part_bytes<MODE, CLUSTER>()) / gf_stage_bytes<MODE>(); }
static_assert(gf_stages<LIN_DENSE, false>() == GF_MAX_STAGES, "barriers for the deepest ring");

// How the units of `tiles` tiles of `ks` units each are dealt out to `ctas` CTAs: whole tiles, or ranges that may cross them.
// Both sides measured at 4096 of K, us: 112 tiles 27 whole, 31 in ranges; 250 tiles 50.5, 51.8 (2048 of K 29.6, 32.0);
// 75 tiles 25.5, 24.4 (32 tokens 29.4, 25.6); 168 tiles 49, 39; 219 tiles 51, 47; 313 tiles 73, 63.
struct GfRange {
    int tiles, ks, ctas;
    bool whole;
    __host__ __device__ static bool in_whole(int tiles, int ctas) {
        const int rounds = (tiles + ctas - 1) / ctas;
        return rounds == 1 ? tiles * 20 >= ctas * 13 : rounds * ctas * 5 <= tiles * 6;
    }
    __device__ __forceinline__ GfRange(int tiles_, int ks_, int ctas_) : tiles(tiles_), ks(ks_), ctas(ctas_), whole(in_whole(tiles_, ctas_)) {}
    __device__ __forceinline__ int begin(int c) const {
        return whole ? (int)((long long)c * tiles / ctas) * ks : (int)((long long)c * tiles * ks / ctas);
    }
    // the CTA with a unit, where ranges may cross tiles
    __device__ __forceinline__ int owner(int unit) const { return (int)(((long long)(unit + 1) * ctas - 1) / ((long long)tiles * ks)); }
};

__device__ __forceinline__ uint32_t cluster_ctas() {
    uint32_t n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(n));
    return n;
}
__device__ __forceinline__ void peer_store(uint32_t remote, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;\n" ::"r"(remote), "r"(v) : "memory");
}
__device__ __forceinline__ void tensormap_prefetch(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(map) : "memory");
}
// A wait for the cluster's arrivals, which make its stores to this CTA's shared memory visible.
__device__ __forceinline__ void cluster_wait(uint64_t *b, uint32_t parity, volatile int *failed) {
    const uint32_t addr = sptr(b);
    const unsigned long long t0 = wall_ns();
    for (uint32_t done = 0; !__all_sync(0xffffffffu, done);) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (!done && wall_ns() - t0 > 4000000000ull) {  // longer than a peer's own waits
            *failed = 1;
            done = 1;
        }
    }
}

// partials: two slots of W4DG_MAX_SLOT_FLOATS per CTA; counters: one per tile, zero on entry and exit.
template <int MODE, bool CLUSTER>
__global__ void __launch_bounds__(GF_THREADS, 1)
gemm_bf16_few_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap w2map, const __grid_constant__ CUtensorMap xmap,
                     LinArgs a, float *partials, int *counters, int *status) {
    constexpr bool DUAL = gf_dual<MODE>();
    constexpr int STAGES = gf_stages<MODE, CLUSTER>(), STAGE_BYTES = gf_stage_bytes<MODE>(), PER = DUAL ? 2 : 1;
    constexpr uint32_t ACC_COLS = PER * GF_TOK, TMEM_COLS = 2 * ACC_COLS;
    static_assert(PER * GF_TOK * 128 <= W4DG_MAX_SLOT_FLOATS, "a slot holds a tile's sums");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *ring = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *part_buf = ring + STAGES * STAGE_BYTES;   // [contributor][its share of the tokens][gate, up][128] f32
    GfShared *sh = (GfShared *)(part_buf + gf_part_bytes<MODE, CLUSTER>());
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KS = (a.K + 63) >> 6, n_tiles = (a.N + 127) >> 7;
    volatile int *failed = &sh->failed;

    if (threadIdx.x == 32) {
        tensormap_prefetch(&wmap);
        if (DUAL) tensormap_prefetch(&w2map);
        tensormap_prefetch(&xmap);
    }
    if (threadIdx.x == 0) {
        if (CLUSTER) bar_init(&sh->parts, cluster_ctas() * GF_EPI_WARPS);
        for (int i = 0; i < STAGES; ++i) { bar_init(&sh->full[i], 2); bar_init(&sh->empty[i], 1); }
        for (int i = 0; i < 2; ++i) { bar_init(&sh->accfull[i], 1); bar_init(&sh->accempty[i], GF_EPI_WARPS); }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(sptr(&sh->tmem_base)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncwarp();
    if (CLUSTER) cluster_sync_all();  // peers arrive at `parts`
    else __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = sh->tmem_base;
    if (warp != 0) {  // the weights are constants
        pdl_wait();
        pdl_launch_dependents();
    }
    const GfRange rg(n_tiles, KS, (int)gridDim.x);
    const int peers = CLUSTER ? (int)cluster_ctas() : 1, rank = CLUSTER ? (int)cluster_rank() : 0;
    const int tile0 = (int)blockIdx.x / peers;
    const int u0 = CLUSTER ? tile0 * KS + rank * KS / peers : rg.begin(blockIdx.x);
    const int u1 = CLUSTER ? tile0 * KS + (rank + 1) * KS / peers : rg.begin(blockIdx.x + 1);

    if (warp == 0) {
        // ---------------------------------------------------------- weights
        if (lane == 0) {
            for (int u = u0, use = 0; u < u1; ++u, ++use) {
                const int tile = u / KS, ks = u - tile * KS, s = use % STAGES;
                if (!bar_wait(&sh->empty[s], ((use / STAGES) & 1) ^ 1, failed)) break;
                uint8_t *st = ring + s * STAGE_BYTES;
                bar_expect_tx(&sh->full[s], PER * GF_W_BYTES);  // what lies past a tensor arrives as zeros and counts
                tma_load_2d(st, &wmap, ks * 64, tile * 128, &sh->full[s]);
                if (DUAL) tma_load_2d(st + GF_W_BYTES, &w2map, ks * 64, tile * 128, &sh->full[s]);
            }
        }
    } else if (warp == 2 + GF_EPI_WARPS) {
        // ---------------------------------------------------------- activations
        if (lane == 0) {
            const int boxes = (a.M + GF_BOX_ROWS - 1) / GF_BOX_ROWS;
            for (int u = u0, use = 0; u < u1; ++u, ++use) {
                const int ks = u % KS, s = use % STAGES;
                if (!bar_wait(&sh->empty[s], ((use / STAGES) & 1) ^ 1, failed)) break;
                uint8_t *st = ring + s * STAGE_BYTES + PER * GF_W_BYTES;
                bar_expect_tx(&sh->full[s], boxes * (GF_BOX_ROWS * 128));
                for (int b = 0; b < boxes; ++b) tma_load_2d(st + b * (GF_BOX_ROWS * 128), &xmap, ks * 64, b * GF_BOX_ROWS, &sh->full[s]);
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------- MMA issue
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((a.M + 15) / 16 * 2) << 17) | ((128u >> 4) << 24);
        int use = 0, seg = 0;
        for (int u = u0; u < u1; ++seg) {
            const int tile = u / KS, end = min(u1, (tile + 1) * KS), ab = seg & 1;
            warp_wait(&sh->accempty[ab], ((seg >> 1) & 1) ^ 1, failed);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t tacc = tmem + (uint32_t)ab * ACC_COLS;
            for (bool first = true; u < end; ++u, ++use, first = false) {
                const int s = use % STAGES;
                warp_wait(&sh->full[s], (use / STAGES) & 1, failed);
                if (elect_one()) {
                    const uint32_t a0 = sptr(ring + s * STAGE_BYTES);
                    const uint64_t xd = umma_desc(a0 + PER * GF_W_BYTES);
                    umma_stage(tacc, umma_desc(a0), xd, idesc, first);
                    if (DUAL) umma_stage(tacc + GF_TOK, umma_desc(a0 + GF_W_BYTES), xd, idesc, first);
                    umma_commit(&sh->empty[s]);
                }
                __syncwarp();
            }
            if (elect_one()) umma_commit(&sh->accfull[ab]);
            __syncwarp();
        }
    } else {
        // ---------------------------------------------------------- epilogue
        const int quad = warp & 3, j0 = ((warp - 2) >> 2) * 16, row = quad * 32 + lane;
        const int cnt = min(a.M - j0, 16);  // tokens of this warp, none where it is negative
        int seg = 0;
        for (int u = u0; u < u1; ++seg) {
            const int tile = u / KS, end = min(u1, (tile + 1) * KS), ab = seg & 1, n = tile * 128 + row;
            const bool whole = u == tile * KS && end == (tile + 1) * KS;
            u = end;
            warp_wait(&sh->accfull[ab], (seg >> 1) & 1, failed);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)ab * ACC_COLS;
            uint32_t v[32];
            if (DUAL) tmem_ld16_pair(v, taddr + j0, taddr + GF_TOK + j0);
            else tmem_ld16(*reinterpret_cast<uint32_t(*)[16]>(v), taddr + j0);
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&sh->accempty[ab]);

            auto put = [&](int t, float z, float up) {
                if (n >= a.N) return;
                if (DUAL) {
                    ((__nv_bfloat16 *)a.y)[(size_t)t * a.N + n] = __float2bfloat16_rn(glu_value(a.glu, z, up, a.limit));
                } else {
                    const size_t o = (size_t)t * a.ldy + n;
                    if (a.epi == LIN_F32) ((float *)a.y)[o] = softcap_value(z, a.cap);
                    else ((__nv_bfloat16 *)a.y)[o] = __float2bfloat16_rn(a.epi == LIN_ACT ? lin_act_value(z, n < a.act_n) : z);
                }
            };
            if (CLUSTER) {
                // every CTA finishes a share of the tokens: the others' sums of them are written into its shared memory
                const int share = (a.M + peers - 1) / peers;   // peers * share <= 32, as peers divides 32
                const uint32_t buf = sptr(part_buf) + row * 4;
                uint32_t to = peer_addr(buf, (uint32_t)min(j0 / share, peers - 1));
                int p = j0 / share, slot = rank * share + j0 - p * share;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (j >= cnt) break;
                    peer_store(to + slot * (PER * 512), v[j]);
                    if (DUAL) peer_store(to + slot * (PER * 512) + 512, v[16 + j]);
                    if (++slot == (rank + 1) * share) {
                        slot = rank * share;
                        if (++p < peers) to = peer_addr(buf, (uint32_t)p);
                    }
                }
                __syncwarp();
                if (lane < peers) peer_arrive(peer_addr(sptr(&sh->parts), (uint32_t)lane));
                cluster_wait(&sh->parts, 0, failed);
                const int t1 = min(a.M, (rank + 1) * share);
                for (int t = rank * share + (j0 >> 4); t < t1; t += 2) {
                    const float *src = reinterpret_cast<const float *>(part_buf) + (t - rank * share) * (PER * 128) + row;
                    float z[2] = {0.f, 0.f};
#pragma unroll
                    for (int c = 0; c < GF_MAX_CLUSTER; ++c) {
                        if (c >= peers) break;
                        z[0] += src[c * share * (PER * 128)];
                        if (DUAL) z[1] += src[c * share * (PER * 128) + 128];
                    }
                    put(t, z[0], z[1]);
                }
                continue;
            }
            if (!whole) {
                const int c_first = rg.owner(tile * KS), c_last = rg.owner(tile * KS + KS - 1);
                // slot 1: the tile that the range ends inside
                auto slot = [&](int c) { return partials + ((size_t)c * 2 + (c == c_first ? 1 : 0)) * W4DG_MAX_SLOT_FLOATS + j0 * PER * 128 + row; };
                float *mine = slot(blockIdx.x);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (j >= cnt) break;
                    __stcg(mine + j * PER * 128, __uint_as_float(v[j]));
                    if (DUAL) __stcg(mine + (j * PER + 1) * 128, __uint_as_float(v[16 + j]));
                }
                __threadfence();
                asm volatile("bar.sync 1, 256;\n" ::: "memory");
                if (threadIdx.x == 64) sh->last = atomicAdd(&counters[tile], 1) == c_last - c_first;
                asm volatile("bar.sync 1, 256;\n" ::: "memory");
                if (!sh->last) continue;
                __threadfence();
                if (threadIdx.x == 64) counters[tile] = 0;
                float f[16 * PER];
#pragma unroll
                for (int j = 0; j < 16 * PER; ++j) f[j] = 0.f;
                // the loads of two contributors (gate and up: of one) are under way together
                constexpr int TOGETHER = DUAL ? 1 : 2;
                for (int c = c_first; c <= c_last; c += TOGETHER) {
                    float p[TOGETHER][16 * PER];
#pragma unroll
                    for (int i = 0; i < TOGETHER; ++i) {
                        const float *src = slot(min(c + i, c_last));
#pragma unroll
                        for (int j = 0; j < 16 * PER; ++j) p[i][j] = j / PER < cnt ? __ldcg(src + j * 128) : 0.f;
                    }
#pragma unroll
                    for (int i = 0; i < TOGETHER; ++i)
                        if (c + i <= c_last)
#pragma unroll
                            for (int j = 0; j < 16 * PER; ++j) f[j] += p[i][j];
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    v[j] = __float_as_uint(f[j * PER]);
                    if (DUAL) v[16 + j] = __float_as_uint(f[j * PER + PER - 1]);
                }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (j < cnt) put(j0 + j, __uint_as_float(v[j]), DUAL ? __uint_as_float(v[16 + j]) : 0.f);
        }
    }

    // ---- teardown: every warp arrives here (all waits are bounded)
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncwarp();
    if (CLUSTER) cluster_sync_all();  // nobody leaves while peers may still write to it
    else __syncthreads();
    if (threadIdx.x == 0 && sh->failed) atomicExch(status, (int)AB2_ERR_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// Clusters of `size` CTAs that run side by side; a GPC's last SMs may not make one up, so fewer than SMs / size.
template <int MODE>
int clusters_at_once(int size, size_t smem) {
    static int known[64][GF_MAX_CLUSTER + 1] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (known[dev][size] == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(size); cfg.blockDim = dim3(GF_THREADS); cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = size; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_bf16_few_kernel<MODE, true>, &cfg) != cudaSuccess) (void)cudaGetLastError();
        known[dev][size] = n > 0 ? n : -1;
    }
    return known[dev][size];
}

template <int MODE, bool CLUSTER>
constexpr size_t gf_smem_bytes() { return 1024 + (size_t)gf_stages<MODE, CLUSTER>() * gf_stage_bytes<MODE>() + gf_part_bytes<MODE, CLUSTER>() + sizeof(GfShared); }

// CTAs of a tile's cluster: the most of which all tiles' run side by side.
template <int MODE>
int gf_cluster(int tiles, int K) {
    int cluster = GF_MAX_CLUSTER;
    while (cluster > 2 && (cluster > (K + 63) / 64 || tiles > clusters_at_once<MODE>(cluster, gf_smem_bytes<MODE, true>()))) cluster >>= 1;
    return cluster;
}

template <int MODE, bool CLUSTER>
int launch_few(const LinArgs &a, int ctas, const DecodeGemmScratch &sc, cudaStream_t s) {
    int cluster = 1;
    int *status = nullptr;
    int rc = device_status_word(&status);
    if (rc != AB2_OK) return rc;
    CUtensorMap wmap, w2map, xmap;
    rc = make_rows_map(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.w, a.N, a.K, a.K, 128, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc == AB2_OK) rc = make_rows_map(&w2map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, gf_dual<MODE>() ? a.w2 : a.w, a.N, a.K, a.K, 128, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc == AB2_OK) rc = make_x_map(&xmap, a.x, a.M, a.K, GF_BOX_ROWS, MODE == LIN_DENSE ? a.ldx : a.K);
    if (rc != AB2_OK) return rc;
    constexpr size_t smem = gf_smem_bytes<MODE, CLUSTER>();
    static bool configured[64] = {false};  // the attribute is per device
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    if (!configured[dev]) {
        AB2_CUDA(cudaFuncSetAttribute(gemm_bf16_few_kernel<MODE, CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured[dev] = true;
    }
    if (CLUSTER) {
        const int n_tiles = (a.N + 127) / 128;
        cluster = gf_cluster<MODE>(n_tiles, a.K);
        ctas = cluster * n_tiles;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas); cfg.blockDim = dim3(GF_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_pdl_launch ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_bf16_few_kernel<MODE, CLUSTER>, wmap, w2map, xmap, a, sc.partials, sc.counters, status);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "bf16 decode GEMM launch failed: %s", cudaGetErrorString(e));
    return AB2_OK;
}

}  // namespace

bool gemm_bf16_few(const LinArgs &a, int mode, cudaStream_t s, int *rc) {
    if (a.M < 1 || a.M > GF_TOK || (mode != LIN_DENSE && mode != LIN_GLU) || (mode == LIN_DENSE && (a.batch > 1 || a.epi == LIN_GATE))) return false;
    const int tiles = (a.N + 127) / 128, KS = (a.K + 63) / 64, sms = device_sm_count(), k = (mode == LIN_GLU ? 2 : 1) * a.K;
    if (2 * tiles <= sms) {
        if (KS < 2) return false;
        // Pairs of CTAs that leave a quarter of the SMs idle: us, GEMV / this kernel at 9 tokens, 4608 x 4096 15.0, 17.8, 6144 x 4096 16.9,
        // 17.7, 5120 x 8192 25.6, 28.7, but 7168 x 4096 23.8, 18.3 (at 32 tokens 31, 18; 6144 x 4096 30, 18).
        if (mode == LIN_DENSE && a.M <= 16 && 8 * tiles < 3 * sms && gf_cluster<LIN_DENSE>(tiles, a.K) == 2) return false;
        *rc = mode == LIN_DENSE ? launch_few<LIN_DENSE, true>(a, 0, {}, s) : launch_few<LIN_GLU, true>(a, 0, {}, s);
        return true;
    }
    const int ctas = tiles < sms && GfRange::in_whole(tiles, sms) ? tiles : sms;
    ScratchLease lease(s);  // given back once the launch stands
    DecodeGemmScratch sc = {};
    if (!GfRange::in_whole(tiles, ctas)) {
        // Handing parts over costs about 6 us, which short ranges do not win back.  us, GEMV / this kernel: 80 tiles, 1024 of K at 32 tokens
        // 16.3, 18.3 (2048: 24.4, 20.5); 2048 of K at 9 tokens 16.0, 20.4 (4096: 27, 26.4); 4096 of K at 5 tokens 24.9, 26.4; 160
        // tiles, 1024 of K at 9 tokens 15.9, 18.4 (2048: 24.0, 24.7; at 32 tokens 24.4, 18.5).
        const int least = tiles < sms ? (a.M > 16 ? 1024 : a.M > 8 ? 2048 : 4096) : a.M > 16 ? 0 : 1024;
        if (k <= least || (long long)tiles * KS > 0x7fffffffll || !decode_gemm_scratch(s, tiles, &lease, &sc)) return false;
    }
    *rc = mode == LIN_DENSE ? launch_few<LIN_DENSE, false>(a, ctas, sc, s) : launch_few<LIN_GLU, false>(a, ctas, sc, s);
    return true;
}

}  // namespace ab2
