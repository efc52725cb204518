// tcgen05 / TMA building blocks shared by the W4A16 tensor-memory kernels
// (internal header): mbarrier helpers with bounded waits, bulk and tensor-map
// copies, the K-major 128-byte-swizzle shared-memory descriptors, the bf16 MMA
// issue and commit, and the host-side tensor map of a [rows][K] bf16 matrix.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace ab2 {
namespace tc {

__device__ __forceinline__ uint32_t sptr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }


__device__ __forceinline__ void bar_init(uint64_t *b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(sptr(b)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(sptr(b)) : "memory");
}
// Arrival that hands a shared-memory slot back to a producer of asynchronous copies.  The arrival
// must not leave while a load of the slot is still under way (the copy that follows it may land
// first): `held` is a value every such load has fed, `hidden_zero` a zero the compiler cannot see
// (derived from a kernel argument); the address of the arrival takes in held & hidden_zero, so the
// instruction waits for the loads.
__device__ __forceinline__ void bar_arrive_after(uint64_t *b, uint32_t held, uint32_t hidden_zero) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(sptr(b) + (held & hidden_zero)) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(sptr(b)), "r"(bytes) : "memory");
}
// Bounded wait (two seconds of wall clock, read from %globaltimer; a probe may itself
// sleep for a while, so counting probes bounds nothing); also gives up as soon as another
// warp of the CTA has failed.
__device__ __forceinline__ unsigned long long wall_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool bar_wait(uint64_t *b, uint32_t parity, volatile int *failed) {
    const uint32_t addr = sptr(b);
    unsigned long long t0 = 0;
    for (int spin = 0;; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
        if ((spin & 31) == 31) {  // the timer is a slow register: read only once a wait has lasted
            if (*failed) return false;
            const unsigned long long now = wall_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > 2000000000ull) break;
        }
    }
    *failed = 1;
    return false;
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::
                     "r"(sptr(dst)), "l"(src), "r"(bytes), "r"(sptr(bar)) : "memory");
}
// 2-D tile load: coordinates (k element, token row); completion counted on `bar`.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::
            "r"(sptr(dst)), "l"(map), "r"(sptr(bar)), "r"(x), "r"(y) : "memory");
}

// ---- pairs of CTAs (a cluster of two) that multiply one tile: cta_group::2
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// The address of CTA `rank`'s variable that lies where `local` does in this CTA.
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local), "r"(rank));
    return remote;
}
__device__ __forceinline__ void peer_arrive(uint32_t remote) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(remote) : "memory");
}
// A tile into this CTA's memory, counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::
            "r"(sptr(dst)), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}

// 3-D tile load: coordinates (element, row, matrix).
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n" ::
            "r"(sptr(dst)), "l"(map), "r"(sptr(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
// 4-D tile load: coordinates from the innermost on.
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int x, int y, int z, int w, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n" ::
            "r"(sptr(dst)), "l"(map), "r"(sptr(bar)), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: 8-row groups are
// 1024 bytes apart, the start address advances by 32 bytes per K = 16 step.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;             // leading byte offset (unused for swizzled K-major): 1
    d |= (uint64_t)(1024 >> 4) << 32;   // stride byte offset: 8 rows x 128 bytes
    d |= (uint64_t)1 << 46;             // descriptor version
    d |= (uint64_t)2 << 61;             // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::
            "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(sptr(bar)) : "memory");
}

// M- or N-major operand, 128-byte swizzle: 64 elements of M per row of K, 8 rows a group of 1024 bytes,
// the next 64 elements `lbo` bytes further.
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t saddr, uint32_t lbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)(lbo >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// One lane of a converged warp, always the same one.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n selp.u32 %0, 1, 0, e;\n}\n" : "=r"(p));
    return p;
}
// The four K = 16 steps of a stage of 64 K-elements, by one thread.  Its branch is taken with elect_one(): behind
// `lane == 0` the compiler cannot know that a single thread is active and feeds the instruction's uniform operands
// lane by lane.  Descriptors count in 16 bytes.
__device__ __forceinline__ void umma_stage(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool first) {
#pragma unroll
    for (int k = 0; k < 4; ++k) umma_bf16(tmem_d, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, !first || k > 0);
}
// The same by the first CTA of a pair for both: 256 rows of A and the columns of B, half of each in either's shared memory.
__device__ __forceinline__ void umma_stage_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool first) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::
                "r"(tmem_d), "l"(adesc + (uint64_t)(2 * k)), "l"(bdesc + (uint64_t)(2 * k)), "r"(idesc), "r"((uint32_t)(!first || k > 0)) : "memory");
}
// Arrives at the barrier in both CTAs of the pair.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(sptr(bar)), "h"((uint16_t)3) : "memory");
}
// The first operand in tensor memory: 128 lanes, two bf16 per column.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::
            "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// The four K = 16 steps of a stage whose first operand lies in 32 columns of tensor memory.
__device__ __forceinline__ void umma_stage_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, bool first) {
#pragma unroll
    for (int k = 0; k < 4; ++k) umma_bf16_ts(tmem_d, tmem_a + (uint32_t)(8 * k), bdesc + (uint64_t)(2 * k), idesc, !first || k > 0);
}
#define AB2_REGS8(c, v) c(v[0]), c(v[1]), c(v[2]), c(v[3]), c(v[4]), c(v[5]), c(v[6]), c(v[7])
#define AB2_REGS16(c, v) AB2_REGS8(c, v), c(v[8]), c(v[9]), c(v[10]), c(v[11]), c(v[12]), c(v[13]), c(v[14]), c(v[15])
#define AB2_REGS32(c, v) \
    c(v[0]), c(v[1]), c(v[2]), c(v[3]), c(v[4]), c(v[5]), c(v[6]), c(v[7]), c(v[8]), c(v[9]), c(v[10]), c(v[11]), c(v[12]), c(v[13]), c(v[14]), c(v[15]), \
    c(v[16]), c(v[17]), c(v[18]), c(v[19]), c(v[20]), c(v[21]), c(v[22]), c(v[23]), c(v[24]), c(v[25]), c(v[26]), c(v[27]), c(v[28]), c(v[29]), c(v[30]), c(v[31])
// 8, 16 or 32 columns of the warp's lanes; the registers pass through the wait, so that nothing computed from them can
// move ahead of it.
__device__ __forceinline__ void tmem_ld8(uint32_t (&v)[8], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n" : AB2_REGS8("=r", v) : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" : AB2_REGS8("+r", v)::"memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t (&v)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : AB2_REGS16("=r", v) : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" : AB2_REGS16("+r", v)::"memory");
}
__device__ __forceinline__ void tmem_ld32_start(uint32_t (&v)[32], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : AB2_REGS32("=r", v) : "r"(addr));
}
__device__ __forceinline__ void tmem_ld32_wait(uint32_t (&v)[32]) { asm volatile("tcgen05.wait::ld.sync.aligned;\n" : AB2_REGS32("+r", v)::"memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t (&v)[32], uint32_t addr) {
    tmem_ld32_start(v, addr);
    tmem_ld32_wait(v);
}
// 16 columns from each of two places
__device__ __forceinline__ void tmem_ld16_pair(uint32_t (&v)[32], uint32_t addr, uint32_t addr2) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : AB2_REGS16("=r", v) : "r"(addr));
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : AB2_REGS16("=r", (v + 16)) : "r"(addr2));
    tmem_ld32_wait(v);
}
__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};\n" ::AB2_REGS32("r", v), "r"(addr)
        : "memory");
}
// A wait of a whole warp, with one answer for it.  Lanes that left a loop after a wait while others went on would leave those
// waiting for them in the warp's next collective instruction for good.  So the warps of the GEMMs that execute any do not
// leave: after a time-out they walk through the rest of their work, whose waits then give up at once, over whatever the
// buffers hold, and the status word says that the output is void.  (They do not arrive at a barrier with copies under way
// unless the stage was theirs: arrivals beyond its count are undefined.)  Leaving by a vote after each wait is sound too, but the INT8
// GEMM took 225 us with it on 14336 x 4096 at 2048 tokens, 213 with lanes that left alone, and takes 205 so.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *failed) { return __all_sync(0xffffffffu, bar_wait(bar, parity, failed)); }

__device__ __forceinline__ uint32_t bf16x2_add_(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.bf16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t bf16x2_mul_(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
    return d;
}


// Whether rows of N bf16 at y can be stored in pieces of 16 bytes.  A caller's y need only lie on an element.
__host__ __device__ __forceinline__ bool rows_in_16_bytes(const void *y, int N) { return (N & 7) == 0 && ((uintptr_t)y & 15) == 0; }

// T tokens x the warp's 32 channels, rounded to bf16, wait in `stage` ([T][32], the warp's own) and go out to rows of
// `ld` elements: `rows` and `cols` of them exist.  Stored straight from the lanes, 32 instructions of 64 bytes for 32
// tokens, they took 50 to 60 ns a token, and those of the last round of tiles are not hidden behind MMAs.
// y lies on a 16-byte boundary; ld and cols are multiples of 8.
template <int T>
__device__ __forceinline__ void flush_rows(const __nv_bfloat16 *stage, __nv_bfloat16 *y, long long ld, int rows, int cols, int lane) {
    __syncwarp();
    const int n = (lane & 3) * 8, row = lane >> 2;
#pragma unroll
    for (int i = 0; i < T; i += 8) {
        const uint4 q = *reinterpret_cast<const uint4 *>(stage + (i + row) * 32 + n);
        if (i + row < rows && n < cols) *reinterpret_cast<uint4 *>(y + (i + row) * ld + n) = q;
    }
    __syncwarp();
}

// The same for T tokens of f32 ([T][32]); row(j), called by the whole warp, is where token j's channels of the warp start.
template <int T, class Row>
__device__ __forceinline__ void flush_rows_f32(const float *stage, Row row, int rows, int cols, int lane) {
    __syncwarp();
    const int n = (lane & 7) * 4, r = lane >> 3;
#pragma unroll
    for (int i = 0; i < T; i += 4) {
        const float4 q = *reinterpret_cast<const float4 *>(stage + (i + r) * 32 + n);
        float *y = row(i + r);
        if (i + r < rows && n < cols) *reinterpret_cast<float4 *>(y + n) = q;
    }
    __syncwarp();
}

// What a tile of ntok tokens by 128 channels takes: `fixed` us and `group` us per 128 of K.
struct GemmTileCost { int ntok; double fixed, group; };
// Tile and K split of a GEMM over G groups: rounds of items on the SMs times an item's time.  A split of at most `splits`
// fits one round; its parts are written and read as f32 at about 4 TB/s by a pass that takes 4 us more.
struct GemmTileChoice { int ntok, ksplit; };
template <int COUNT>
inline GemmTileChoice choose_gemm_tile(const GemmTileCost (&costs)[COUNT], int M, int N, int G, int sms, int splits) {
    GemmTileChoice best = {costs[0].ntok, 1};
    double best_us = 1e30;
    for (const GemmTileCost &c : costs) {
        const long long tiles = (long long)((N + 127) / 128) * ((M + c.ntok - 1) / c.ntok);
        for (int ks = 1; ks <= splits && (ks == 1 || (tiles * ks <= sms && G / ks >= 4)); ++ks) {
            const double rounds = (double)((tiles * ks + sms - 1) / sms);
            const double us = rounds * (c.fixed + c.group * ((G + ks - 1) / ks)) + (ks > 1 ? 4.0 + (double)ks * M * N * 8 / 4e6 : 0.0);
            if (us < best_us) { best_us = us; best = {c.ntok, ks}; }
        }
    }
    return best;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline int tensor_map_encoder(EncodeTiledFn *out) {
    static EncodeTiledFn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        AB2_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
        AB2_REQUIRE(fn != nullptr && qres == cudaDriverEntryPointSuccess, AB2_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is unavailable");
        encode = (EncodeTiledFn)fn;
    }
    *out = encode;
    return AB2_OK;
}

// Tensor map of `rows` rows of `cols` elements that lie `ld` elements apart, read in boxes of 128 bytes x box_rows
// (128-byte swizzle).
inline int make_rows_map(CUtensorMap *map, CUtensorMapDataType type, int elem, const void *p, int rows, int cols, long long ld, int box_rows,
                         CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_L2_128B) {
    EncodeTiledFn encode;
    int rc = tensor_map_encoder(&encode);
    if (rc != AB2_OK) return rc;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * elem};
    cuuint32_t box[2] = {(cuuint32_t)(128 / elem), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode(map, type, 2, const_cast<void *>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    AB2_REQUIRE(r == CUDA_SUCCESS, AB2_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    return AB2_OK;
}

// Tensor map of a [M][K] bf16 matrix whose rows lie `ld` elements apart (0: K), read in boxes of 64 x ntok.
inline int make_x_map(CUtensorMap *map, const void *x, int M, int K, int ntok, long long ld = 0) {
    return make_rows_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, M, K, ld > 0 ? ld : K, ntok);
}

// Tensor map of `mats` bf16 matrices of `rows` rows x `cols`, rows `ld` and matrices `z` elements apart, read in boxes
// of 64 x box_rows of one matrix.
inline int make_mats_map(CUtensorMap *map, const void *p, int mats, int rows, int cols, long long ld, long long z, int box_rows) {
    EncodeTiledFn encode;
    int rc = tensor_map_encoder(&encode);
    if (rc != AB2_OK) return rc;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)mats};
    cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)z * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    AB2_REQUIRE(r == CUDA_SUCCESS, AB2_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    return AB2_OK;
}

// Tensor map of [N][bytes] bytes, read in boxes of 128 x 128.
inline int make_bytes_map(CUtensorMap *map, const void *p, int N, int bytes) {
    return make_rows_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p, N, bytes, bytes, 128);
}


}  // namespace tc
}  // namespace ab2
