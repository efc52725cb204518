// Flash-decode attention over INT8 and bf16 caches on the warp-level tensor cores (head_dim 128,
// up to 8 query heads per KV head): the throughput path for long contexts and
// large batches, where CUDA cores are bound by conversions and multiplications rather than by HBM.
//
// Per 16 cached tokens a warp issues 16 MMAs for Q.K^T (A = the group's query
// heads as the 16 rows, constant in registers; B = K^T straight from the
// token rows) and 8 MMAs for P.V (A = V^T obtained from the natural [token][d]
// rows with ldmatrix.trans, on byte pairs for INT8; B = P^T, which is exactly the score
// fragment the first MMA left in this thread's registers).  int8 codes become
// fp16 by one shift or none and one logic op a pair (0x6400 | (code ^ 0x80) = 1152 + code, exact)
// and one exact fp16 subtraction of 1152 on the otherwise idle FMA pipe; the
// per-token K scale multiplies the f32 score, the per-token V scale is folded
// into P.  Over a bf16 cache P enters as three bf16 terms, the rounded value and what rounding
// left of it twice over (together all of its 24 bits), hence 24 MMAs for P.V.
// Accumulation is f32; softmax is the same online form as the reference
// (crates/aarambh-studio-kernel/src/cpu/parallel_attn.rs:189-234), in blocks of
// 16 keys.
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "kv_cache.cuh"
#include "tcgen05_util.cuh"

using namespace ab2;
using namespace ab2::tc;

namespace ab2 {
int device_status_word(int **out);
int device_sm_count();
namespace {

struct MmaAttnArgs {
    KvView kv;
    const void *q;  // head (row, head) at row * q_stride + head * 128
    long long q_stride;
    int row0, nrows, h, rep, dtype;
    // CTAs of a KV head that are resident at once; most splits of a row; fewest tokens of a split; rows of up to that many are not split
    int slots, nsplit, min_tokens, whole_tokens;
    int pending;    // appended, not yet committed tokens per row: they are attended too
    bool whole;     // no row is split: a CTA's row is its index
    float scale;
    float *part_acc, *part_ml;  // [row][head][nsplit]
    int *counters;  // [row][kv head] splits that have arrived, zero at rest
    void *out;
};

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                              uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t f16x2_sub1152(uint32_t v) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(d) : "r"(v), "r"(0xE480E480u));  // + (-1152, -1152)
    return d;
}
// bytes i and j of the sign-flipped word as fp16x2 (code_i, code_j), exact
template <int I, int J>
__device__ __forceinline__ uint32_t i8_pair_f16(uint32_t flipped) {
    return f16x2_sub1152(__byte_perm(flipped, 0x64646464u, (4 << 12) | (J << 8) | (4 << 4) | I));
}
__device__ __forceinline__ float q_as_f32(const void *p, int dtype, size_t i) {
    if (dtype == AB2_F32) return ((const float *)p)[i];
    if (dtype == AB2_F16) return __half2float(((const __half *)p)[i]);
    return __bfloat162float(((const __nv_bfloat16 *)p)[i]);
}
__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}
__device__ __forceinline__ void st_out(void *p, int dtype, size_t i, float v) {
    if (dtype == AB2_F32) ((float *)p)[i] = v;
    else if (dtype == AB2_F16) ((__half *)p)[i] = __float2half_rn(v);
    else ((__nv_bfloat16 *)p)[i] = __float2bfloat16_rn(v);
}

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a)) | ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(b)) << 16);
}
__device__ __forceinline__ float bf16_rest(float v) { return v - __bfloat162float(__float2bfloat16_rn(v)); }
// The codes of bytes 0 and 2, and of bytes 1 and 3, as fp16x2, exact.  Mask and magic number come in registers, so that they
// meet in one logic op.
struct I8Pairs {
    uint32_t mask = 0x00FF00FFu, magic = 0x64806480u;
    __device__ __forceinline__ I8Pairs() { asm volatile("" : "+r"(mask), "+r"(magic)); }
    __device__ __forceinline__ uint32_t even(uint32_t w) const {
        uint32_t d;
        asm("lop3.b32 %0, %1, %2, %3, 0x6A;\n" : "=r"(d) : "r"(w), "r"(mask), "r"(magic));  // (w & mask) ^ magic
        return f16x2_sub1152(d);
    }
    __device__ __forceinline__ uint32_t odd(uint32_t w) const { return even(w >> 8); }
};

__device__ __forceinline__ uint32_t transposed(uint32_t v) {  // an 8 x 8 matrix of 16-bit values over the warp
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ void ldmatrix_trans(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}

// What bounds it: HBM from some 10,000 tokens of a batch on, the chain of a launch (lengths, first copies, MMAs, merge) below.
// INT8 rows cost the instructions that turn codes into fp16 besides, half of what the schedulers can issue.  So nothing else is
// spent on a block that can be avoided: a warp's ring of AT_STAGES blocks of 16 tokens is filled by tensor-map copies of one
// lane, two blocks ahead; their 128-byte swizzle keeps fragment reads free of bank conflicts; keys are the rows of the first
// product, so that no half of an MMA is padding, and a transpose in registers makes its result the second one's operand; the
// reference score moves rarely; exponentials are powers of two of scores scaled once.  394 instructions a block of INT8 tokens;
// 583 with cp.async and queries as rows.  Sixteen warps of an INT8 launch share an SM, eight of a bf16 one.
// us in a graph, 32 / 8 heads, the kernels before (for bf16 on CUDA cores) -> now: INT8 8 x 16384 74 -> 52 (0.82 of the copy rate; a call of
// its own 75 -> 55), 64 x 4096 119 -> 93, 32 x 700 17.4 -> 15.6, 1 x 4096 24 -> 12.3, 1 x 256 7.9 -> 5.5; bf16 64 x 2048 225 -> 84 (0.99), 8 x 8192
// 160 -> 49, 32 x 700 53 -> 20, 1 x 4096 27 -> 12.6, 1 x 256 14.7 -> 6.9.
// Error against 64 bits over 40 drawn batches to that of the kernels before: bf16 rows 1.00000001 (two terms of the weights in one
// accumulator 1.0000008; the third and accumulators of their own take 3 % of the time), INT8 rows with bf16 queries 0.999995, with f32
// queries 1.0006, single batches 0.987 to 1.006.  Exponentials of scores scaled by log2 e, which are 2 ulp off, don't show in it.
constexpr int AT_STAGES = 3, AT_TOK = 16, AT_HD = 128;
template <int KVD, bool MANY>  // MANY: short rows, many of them
struct AtShape {
    static constexpr bool I8 = KVD == AB2_KV_INT8;
    static constexpr int WARPS = (I8 ? 8 : 4) / (MANY ? 2 : 1), STRIDE = WARPS * AT_TOK;  // a warp takes every WARPS-th block
    static constexpr int TILES = I8 ? 1 : 2;                     // tiles of 16 tokens x 128 bytes that hold the keys, or values, of a block
    static constexpr int BLOCK = TILES * AT_TOK * 128, STAGE = 2 * BLOCK, WARP = AT_STAGES * STAGE;
    static constexpr int SCALES = I8 ? AT_STAGES * 2 * AT_TOK * 4 : 0;  // of a warp
    static constexpr int SMEM = 1024 + WARPS * (WARP + SCALES);
    static constexpr int CTAS = MANY ? 4 : 2;                    // of an SM
    static_assert(WARP >= 8 * AT_HD * 4, "the warps' sums are merged in the rings' place");
};

// byte offset of 16-byte chunk `ch` of token `tok` in a block, as the copies' swizzle places it
__device__ __forceinline__ int at_chunk(int tok, int ch) { return (ch >> 3) * (AT_TOK * 128) + tok * 128 + (((ch & 7) ^ (tok & 7)) << 4); }

__device__ __forceinline__ float exp2_approx(float v) {  // 2 ulp; 0 for -inf
    float r;
    asm("ex2.approx.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}

// The share of a CTA: splits of every row, as many as its tokens ask for, dealt out in the rows' order.  The tokens of a split
// are the fewest with which the splits of all rows are resident at once (equal splits per row left a quarter of the SMs' time
// unused where rows are ragged).  Found by every warp for itself, from the lengths as they are when the launch runs.
struct AtShare {
    int rrow, split, splits, t0, t1;  // rrow < 0: none
};
__device__ __forceinline__ AtShare at_share(const MmaAttnArgs &a, int cta, int lane) {
    auto len_of = [&](int r) { return r < a.nrows ? a.kv.lens[kv_row(a.kv, a.row0, r)] + a.pending : 0; };
    const int len0 = len_of(lane);  // the first 32 rows stay in a register
    unsigned total = 0, most = 0;   // in 16s
    for (int r0 = 0; r0 < a.nrows; r0 += 32) {
        const unsigned n = (unsigned)((r0 ? len_of(r0 + lane) : len0) + 15) / 16;
        total += __reduce_add_sync(0xffffffffu, n);
        most = max(most, __reduce_max_sync(0xffffffffu, n));
    }
    unsigned per = max(max((total + a.slots - 1) / a.slots, (most + a.nsplit - 1) / a.nsplit), (unsigned)a.min_tokens / 16);
    if (most <= (unsigned)a.whole_tokens / 16) per = most;
    for (; per < most; per += max(1u, per / 8)) {
        unsigned ctas = 0;
        for (int r0 = 0; r0 < a.nrows; r0 += 32)
            ctas += __reduce_add_sync(0xffffffffu, ((unsigned)((r0 ? len_of(r0 + lane) : len0) + 15) / 16 + per - 1) / per);
        if (ctas <= (unsigned)a.slots) break;
    }
    int before = 0;
    for (int r0 = 0; r0 < a.nrows; r0 += 32) {
        const int len = r0 ? len_of(r0 + lane) : len0;
        const unsigned blocks = (unsigned)(len + 15) / 16, n0 = (blocks + per - 1) / per;
        const unsigned even = n0 ? (blocks + n0 - 1) / n0 : 1;  // the row's splits are alike
        const int n = (int)((blocks + even - 1) / even);
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, cta < before + upto);
        if (hit) {
            const int src = __ffs(hit) - 1;
            const int first = __shfl_sync(0xffffffffu, before + upto - n, src), rlen = __shfl_sync(0xffffffffu, len, src);
            const int tokens = __shfl_sync(0xffffffffu, (int)even * 16, src);
            AtShare w;
            w.rrow = r0 + src; w.split = cta - first; w.splits = __shfl_sync(0xffffffffu, n, src);
            w.t0 = w.split * tokens; w.t1 = min(rlen, w.t0 + tokens);
            return w;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return AtShare{-1, 0, 0, 0, 0};
}

// grid (CTAs of a KV head, kv heads); head_dim 128.
template <int KVD, bool MANY>
__global__ void __launch_bounds__(32 * AtShape<KVD, MANY>::WARPS, AtShape<KVD, MANY>::CTAS)
attn_decode_mma_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, MmaAttnArgs a, int *status) {
    using S = AtShape<KVD, MANY>;
    constexpr int HD = AT_HD;
    constexpr bool I8 = S::I8;
    extern __shared__ uint8_t at_smem_raw[];
    __shared__ float wm[S::WARPS][8], wl[S::WARPS][8];
    __shared__ float weight[8][AB2_KV_MAX_SPLITS];
    __shared__ uint64_t full[S::WARPS][AT_STAGES];
    __shared__ int last_flag, failed_flag;
    uint8_t *at_smem = (uint8_t *)(((uintptr_t)at_smem_raw + 1023) & ~(uintptr_t)1023);
    volatile int *failed = &failed_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    if (threadIdx.x == 0) {
        failed_flag = 0;
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&kmap) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&vmap) : "memory");
    }
    if (lane == 0) {
        // the copies' bytes, and the scales of every lane
        for (int i = 0; i < AT_STAGES; ++i) bar_init(&full[warp][i], I8 ? 33 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    __syncthreads();
    pdl_wait();  // inputs come from the preceding kernel of the step
    pdl_launch_dependents();
    AtShare w;
    if (a.whole) {
        w.rrow = (int)blockIdx.x; w.split = 0; w.splits = 1;
        w.t0 = 0; w.t1 = a.kv.lens[kv_row(a.kv, a.row0, w.rrow)] + a.pending;
    } else {
        w = at_share(a, (int)blockIdx.x, lane);
        if (w.rrow < 0) return;
    }
    const int kvhead = blockIdx.y, rrow = w.rrow, row = kv_row(a.kv, a.row0, rrow), t0 = w.t0, t1 = w.t1;
    const size_t head_base = ((size_t)row * a.kv.kvh + kvhead) * a.kv.cap;
    uint8_t *ring = at_smem + warp * S::WARP;
    float *scales = reinterpret_cast<float *>(at_smem + S::WARPS * S::WARP) + warp * (S::SCALES / 4);
    const uint32_t ring_s = sptr(ring);
    const float *sc_src = nullptr;
    if constexpr (I8) sc_src = (lane < 16 ? a.kv.ks : a.kv.vs) + head_base;

    // Tokens past the end come along as whatever the cache holds there: their scores are masked below, their values' weight is 0.
    // Codes are finite whatever they are; scales past the end are not read, bf16 values past the end are cleared.
    auto fetch = [&](int base, int st) {
        if (lane == 0) {
            uint8_t *dst = ring + st * S::STAGE;
            bar_expect_tx(&full[warp][st], S::STAGE);
#pragma unroll
            for (int i = 0; i < S::TILES; ++i) {
                tma_load_2d(dst + i * (AT_TOK * 128), &kmap, i * 64, (int)head_base + base, &full[warp][st]);
                tma_load_2d(dst + S::BLOCK + i * (AT_TOK * 128), &vmap, i * 64, (int)head_base + base, &full[warp][st]);
            }
        }
        if constexpr (I8) {
            const float *src = sc_src + min(base + (lane & 15), t1 - 1);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sptr(scales + st * 32 + lane)), "l"(src) : "memory");
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(sptr(&full[warp][st])) : "memory");
        }
    };
    const int first = t0 + warp * AT_TOK;
#pragma unroll
    for (int i = 0; i < AT_STAGES - 1; ++i)
        if (first + S::STRIDE * i < t1) fetch(first + S::STRIDE * i, i);

    // ---- Q fragments (B operand): column g = query head g of the group.  Which of a row's elements a k index stands for is the
    // same in both operands: k-step s of lane column c covers d = c*32 + 4s + {0,2} (first register) and {1,3} over INT8 rows, {0,1}
    // and {2,3} over bf16 rows, whose 16-byte chunks columns 2 and 3 take in another order (no bank met twice).  Heads >= rep are zero.
    uint32_t qb[8][2];
    {
        const size_t q0 = (size_t)rrow * a.q_stride + ((size_t)kvhead * a.rep + g) * HD + c * 32;
        uint32_t qw[16] = {};  // the 32 elements as bf16, in the order they lie
        const bool wide = a.dtype == AB2_BF16 && (((uintptr_t)a.q | (uintptr_t)(a.q_stride * 2)) & 15) == 0;
        if (wide && g < a.rep) {
            const uint4 *qp = reinterpret_cast<const uint4 *>((const __nv_bfloat16 *)a.q + q0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 v = qp[I8 ? i : i ^ (c & 2)];
                qw[4 * i] = v.x; qw[4 * i + 1] = v.y; qw[4 * i + 2] = v.z; qw[4 * i + 3] = v.w;
            }
        }
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            float v0 = __uint_as_float(qw[2 * s] << 16), v1 = __uint_as_float(qw[2 * s] & 0xffff0000u);
            float v2 = __uint_as_float(qw[2 * s + 1] << 16), v3 = __uint_as_float(qw[2 * s + 1] & 0xffff0000u);
            if (!wide && g < a.rep) {
                const size_t at = q0 + 4 * (I8 ? s : s ^ (c & 2) << 1);
                v0 = q_as_f32(a.q, a.dtype, at); v1 = q_as_f32(a.q, a.dtype, at + 1);
                v2 = q_as_f32(a.q, a.dtype, at + 2); v3 = q_as_f32(a.q, a.dtype, at + 3);
            }
            qb[s][0] = I8 ? pack_f16(v0, v2) : pack_bf16(v0, v1);
            qb[s][1] = I8 ? pack_f16(v1, v3) : pack_bf16(v2, v3);
        }
    }

    // Of heads 2c, 2c+1: reference score; this lane's tokens' sum.  The reference starts at the lowest finite value, so that blocks
    // of scores of -inf weigh nothing.
    float m_ref[2] = {-FLT_MAX, -FLT_MAX}, l_part[2] = {0.f, 0.f};
    float o[8][4];               // [d chunk][fragment]: rows d, columns heads 2c, 2c+1
    float rest[I8 ? 1 : 8][4];   // the same of what P's rounding to bf16 left: apart, since it is 0 or below 0 where a value may be infinite
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            o[i][j] = 0.f;
            if constexpr (!I8) rest[i][j] = 0.f;
        }

    const I8Pairs i8;
    // places in a block, from its start; further chunks are exclusive-ors away
    const uint32_t k_at = at_chunk(g, I8 ? 2 * c : 4 * c + (c & 2)), lm = lane >> 3, v_at = S::BLOCK + at_chunk((lm & 1) * 8 + (lane & 7), lm >> 1);
    const float scale2 = a.scale * 1.4426950408889634f;  // scores in powers of two
    int stage = 0, ahead = AT_STAGES - 1;
    uint32_t lap = 0;
    for (int base = first; base < t1; base += S::STRIDE) {
        bar_wait(&full[warp][stage], lap, failed);
        __syncwarp();  // every lane has left the stage that is filled next: the MMAs took its loads in
        if (base + S::STRIDE * (AT_STAGES - 1) < t1) fetch(base + S::STRIDE * (AT_STAGES - 1), ahead);
        const uint32_t kst = (uint32_t)(stage * S::STAGE) + k_at, vs = ring_s + stage * S::STAGE + v_at;
        const float *sc = scales + stage * 32;
        if constexpr (!I8) {
            if (base + AT_TOK > t1) {  // the last block: no value past the end may be infinite or NaN
                for (int i = lane; i < AT_TOK * 16; i += 32)
                    if (base + (i >> 4) >= t1) *reinterpret_cast<uint4 *>(ring + stage * S::STAGE + S::BLOCK + at_chunk(i >> 4, i & 15)) = make_uint4(0, 0, 0, 0);
                __syncwarp();
            }
        }
        if (++stage == AT_STAGES) { stage = 0; lap ^= 1; }
        if (++ahead == AT_STAGES) ahead = 0;

        // ---- S^T = K.Q^T: rows tokens g, g + 8 (fragments 0,1 and 2,3), columns heads 2c, 2c+1
        float sv[4] = {0.f, 0.f, 0.f, 0.f}, sv2[4] = {0.f, 0.f, 0.f, 0.f};  // two chains of MMAs
#pragma unroll
        for (int i = 0; i < 2 * S::TILES; ++i) {  // this thread's 32 elements of the two tokens
            const uint8_t *kp = ring + (kst ^ (i << 4));
            const uint4 ka = *reinterpret_cast<const uint4 *>(kp), kb = *reinterpret_cast<const uint4 *>(kp + 8 * 128);
            if constexpr (I8) {
                const uint32_t wa[4] = {ka.x, ka.y, ka.z, ka.w}, wb[4] = {kb.x, kb.y, kb.z, kb.w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    mma_f16_16816(j & 1 ? sv2 : sv, i8.even(wa[j]), i8.even(wb[j]), i8.odd(wa[j]), i8.odd(wb[j]), qb[4 * i + j][0], qb[4 * i + j][1]);
            } else {
                mma_bf16_16816(sv, ka.x, kb.x, ka.y, kb.y, qb[2 * i][0], qb[2 * i][1]);
                mma_bf16_16816(sv2, ka.z, kb.z, ka.w, kb.w, qb[2 * i + 1][0], qb[2 * i + 1][1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) sv[i] += sv2[i];
        // ---- weights 2^(score - reference) of the heads' 16 tokens
        float va = 1.f, vb = 1.f;  // V scales of tokens g, g + 8
        {
            float fa = scale2, fb = scale2;
            if constexpr (I8) { fa *= sc[g]; fb *= sc[g + 8]; va = sc[16 + g]; vb = sc[24 + g]; }
            sv[0] *= fa; sv[1] *= fa; sv[2] *= fb; sv[3] *= fb;
        }
        if (base + AT_TOK > t1) {
            if (base + g >= t1) sv[0] = sv[1] = -INFINITY;
            if (base + g + 8 >= t1) sv[2] = sv[3] = -INFINITY;
        }
        // The reference moves when a score passes it; over bf16 rows 2^8 ahead, so that it seldom has to after the first blocks (fp16
        // weights have no bits to spare for that).  No weight is above 1: it would overflow fp16 with its token's scale, and f32 sums
        // of large bf16 values.
        constexpr float AHEAD = I8 ? 0.f : 8.f;
        if (__any_sync(0xffffffffu, !(fmaxf(sv[0], sv[2]) <= m_ref[0]) || !(fmaxf(sv[1], sv[3]) <= m_ref[1]))) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float m = fmaxf(sv[e], sv[2 + e]);
#pragma unroll
                for (int x = 4; x < 32; x <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
                m = m > m_ref[e] ? m + AHEAD : m_ref[e];
                const float corr = exp2_approx(m_ref[e] - m);
                l_part[e] *= corr;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    o[i][e] *= corr; o[i][2 + e] *= corr;
                    if constexpr (!I8) { rest[i][e] *= corr; rest[i][2 + e] *= corr; }
                }
                m_ref[e] = m;
            }
        }
        float pv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pv[i] = exp2_approx(sv[i] - m_ref[i & 1]);  // 0 for tokens past the end
        l_part[0] += pv[0] + pv[2];
        l_part[1] += pv[1] + pv[3];

        // ---- O^T += V^T . P^T; P^T (B operand) is the transpose of what the first product left here
        // ldmatrix x4.trans: matrices (tokens 0-7, chunk dc), (8-15, dc), (0-7, dc+1), (8-15, dc+1)
        if constexpr (I8) {
            // times the V scale of their token
            const uint32_t pb0 = transposed(pack_f16(pv[0] * va, pv[1] * va)), pb1 = transposed(pack_f16(pv[2] * vb, pv[3] * vb));
#pragma unroll
            for (int dp = 0; dp < 4; ++dp) {
                uint32_t r0, r1, r2, r3;
                ldmatrix_trans(r0, r1, r2, r3, vs ^ (dp << 5));
                // rows g: d = chunk*16 + 2g (bytes 0, 2); rows g+8: d + 1 (bytes 1, 3)
                mma_f16_16816(o[2 * dp], i8.even(r0), i8.odd(r0), i8.even(r1), i8.odd(r1), pb0, pb1);
                mma_f16_16816(o[2 * dp + 1], i8.even(r2), i8.odd(r2), i8.even(r3), i8.odd(r3), pb0, pb1);
            }
        } else {
            uint32_t pb[3][2];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                pb[i][0] = transposed(pack_bf16(pv[0], pv[1]));
                pb[i][1] = transposed(pack_bf16(pv[2], pv[3]));
#pragma unroll
                for (int j = 0; j < 4; ++j) pv[j] = bf16_rest(pv[j]);
            }
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
                uint32_t r0, r1, r2, r3;
                ldmatrix_trans(r0, r1, r2, r3, (vs + (ch >> 2) * (AT_TOK * 128)) ^ ((ch & 3) << 5));
                // rows g: d = chunk*16 + g; rows g+8: d + 8
                mma_bf16_16816(o[ch], r0, r2, r1, r3, pb[0][0], pb[0][1]);
                mma_bf16_16816(rest[ch], r0, r2, r1, r3, pb[2][0], pb[2][1]);
                mma_bf16_16816(rest[ch], r0, r2, r1, r3, pb[1][0], pb[1][1]);
            }
        }
    }
    if constexpr (!I8) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (fabsf(o[i][j]) <= FLT_MAX) o[i][j] += rest[i][j];  // infinite: of an infinite value, as it stands
    }
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) l_part[e] += __shfl_xor_sync(0xffffffffu, l_part[e], x);

    // ---- merge the warps
    if (threadIdx.x == 0 && *failed) atomicExch(status, (int)AB2_ERR_TIMEOUT);
    __syncthreads();  // the rings are free: every copy was waited for
    float *wacc = reinterpret_cast<float *>(at_smem);  // [S::WARPS][8][HD]
    if (g < 2) { wm[warp][2 * c + g] = g ? m_ref[1] : m_ref[0]; wl[warp][2 * c + g] = g ? l_part[1] : l_part[0]; }
#pragma unroll
    for (int ch = 0; ch < 8; ++ch) {
        const int d = ch * 16 + (I8 ? 2 * g : g), d2 = d + (I8 ? 1 : 8);
        float *h0 = wacc + (warp * 8 + 2 * c) * HD, *h1 = h0 + HD;
        h0[d] = o[ch][0]; h0[d2] = o[ch][2];
        h1[d] = o[ch][1]; h1[d2] = o[ch][3];
    }
    __syncthreads();
    const size_t pi0 = ((size_t)row * a.h + kvhead * a.rep) * a.nsplit;  // the group's first part
    for (int i = threadIdx.x; i < a.rep * HD; i += 32 * S::WARPS) {
        const int hh = i / HD, d = i % HD;
        float M = wm[0][hh];
#pragma unroll
        for (int i2 = 1; i2 < S::WARPS; ++i2) M = fmaxf(M, wm[i2][hh]);
        float L = 0.f, A = 0.f;
#pragma unroll
        for (int i2 = 0; i2 < S::WARPS; ++i2) {
            const float e = exp2f(wm[i2][hh] - M);
            L += e * wl[i2][hh];
            A += e * wacc[(i2 * 8 + hh) * HD + d];
        }
        if (w.splits == 1) {
            st_out(a.out, a.dtype, ((size_t)rrow * a.h + kvhead * a.rep + hh) * HD + d, A * (1.0f / L));
        } else {
            const size_t pi = pi0 + (size_t)hh * a.nsplit + w.split;
            a.part_acc[pi * HD + d] = A;
            if (d == 0) { a.part_ml[pi * 2] = M; a.part_ml[pi * 2 + 1] = L; }
        }
    }
    if (w.splits == 1) return;
    // ---- merge the splits: by the CTA that arrives last, in the splits' order
    __threadfence();
    __syncthreads();
    int *counter = a.counters + row * a.kv.kvh + kvhead;
    if (threadIdx.x == 0) last_flag = atomicAdd(counter, 1) == w.splits - 1;
    __syncthreads();
    if (!last_flag) return;
    __threadfence();
    if (threadIdx.x == 0) *counter = 0;
    for (int hh = warp; hh < a.rep; hh += S::WARPS) {  // what each split's sums count, two splits a lane
        const float2 *ml = reinterpret_cast<const float2 *>(a.part_ml) + pi0 + (size_t)hh * a.nsplit;
        const float2 none = make_float2(-INFINITY, 0.f);
        const float2 x = lane < w.splits ? __ldcg(ml + lane) : none, y = lane + 32 < w.splits ? __ldcg(ml + lane + 32) : none;
        float M = fmaxf(x.x, y.x);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        const float ex = x.x == -INFINITY ? 0.f : exp2f(x.x - M), ey = y.x == -INFINITY ? 0.f : exp2f(y.x - M);
        float L = ex * x.y + ey * y.y;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        const float inv = 1.0f / L;
        weight[hh][lane] = ex * inv;
        weight[hh][lane + 32] = ey * inv;
    }
    __syncthreads();
    for (int hh = warp; hh < a.rep; hh += S::WARPS) {  // a warp a head, four dimensions a lane
        const float4 *p = reinterpret_cast<const float4 *>(a.part_acc + (pi0 + (size_t)hh * a.nsplit) * HD) + lane;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int s = 0; s < w.splits; ++s) {
            const float4 v = __ldcg(p + s * (HD / 4));
            const float e = weight[hh][s];
            sum.x += e * v.x; sum.y += e * v.y; sum.z += e * v.z; sum.w += e * v.w;
        }
        const size_t at = ((size_t)rrow * a.h + kvhead * a.rep + hh) * HD + lane * 4;
        st_out(a.out, a.dtype, at, sum.x); st_out(a.out, a.dtype, at + 1, sum.y);
        st_out(a.out, a.dtype, at + 2, sum.z); st_out(a.out, a.dtype, at + 3, sum.w);
    }
}

// ---------------------------------------------------------------------------
// Causal attention of S new queries per sequence over the INT8 cache (prefill
// chunks, speculative verification): GroupedQueryAttention::forward at S > 1
// (crates/aarambh-studio-nn/src/attention.rs:170-226) with the causal cut of
// dispatch.rs:145-160 (query i sees keys up to kv_len - q_len + i).
//
// Same tensor-core arithmetic as the decode kernel above with the roles of the
// MMA rows changed: a warp owns 16 consecutive queries of ONE query head (the A
// rows of Q.K^T), walks the keys 16 at a time up to the causal limit of its last
// query, keeps the online softmax of its 16 rows in registers and accumulates
// O^T = V^T . P^T for queries 0-7 and 8-15 with the same V^T fragments.  The warps
// of a CTA are the query heads of one KV head on the same 16 queries, so the K
// rows and V blocks they fetch are the same bytes (cache hits after the first).
// No cross-warp merge and no context split: every (head, query tile) is a warp.
// ---------------------------------------------------------------------------
struct PrefillAttnArgs {
    KvView kv;
    const void *q;
    void *out;
    AttnStrides st;
    int S, pending, row0, rep, dtype;
    float scale;
};

__global__ void __launch_bounds__(128) attn_prefill_mma_kernel(PrefillAttnArgs a) {
    constexpr int HD = 128;
    __shared__ alignas(128) uint8_t vst[4][2][16 * HD];  // per warp, double-buffered V block (swizzled 16-byte chunks)
    pdl_wait();
    pdl_launch_dependents();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    if (warp >= a.rep) return;  // no barrier below: a spare warp may leave
    const int qt = blockIdx.x, kvhead = blockIdx.y, rrow = blockIdx.z, row = kv_row(a.kv, a.row0, rrow);
    const int head = kvhead * a.rep + warp;
    const int q_lo = qt * 16;
    // keys visible to query i: [0, first + i]; first = cached + appended - S
    const int first = a.kv.lens[row] + a.pending - a.S;
    const int kmax = first + min(a.S, q_lo + 16);  // keys the tile's last query sees
    const size_t head_base = ((size_t)row * a.kv.kvh + kvhead) * a.kv.cap;
    const int8_t *kbase = (const int8_t *)a.kv.k + head_base * HD;
    const int8_t *vbase = (const int8_t *)a.kv.v + head_base * HD;
    const float *ksc = a.kv.ks + head_base, *vsc = a.kv.vs + head_base;

    // ---- Q fragments: rows g and g + 8 = queries q_lo + g, q_lo + g + 8; k-step s covers
    // d = c*32 + 4s + {0,1} (a0 / a1) and {2,3} (a2 / a3)
    uint32_t qa0[8], qa1[8], qa2[8], qa3[8];
    {
        const int qa = q_lo + g, qb = q_lo + g + 8;
        const size_t ba = (size_t)((long long)rrow * a.st.q_b + (long long)qa * a.st.q_s + (long long)head * a.st.q_h) + c * 32;
        const size_t bb = (size_t)((long long)rrow * a.st.q_b + (long long)qb * a.st.q_s + (long long)head * a.st.q_h) + c * 32;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (qa < a.S)
                for (int j = 0; j < 4; ++j) v[j] = q_as_f32(a.q, a.dtype, ba + 4 * s + j);
            if (qb < a.S)
                for (int j = 0; j < 4; ++j) v[4 + j] = q_as_f32(a.q, a.dtype, bb + 4 * s + j);
            qa0[s] = pack_f16(v[0], v[1]); qa2[s] = pack_f16(v[2], v[3]);
            qa1[s] = pack_f16(v[4], v[5]); qa3[s] = pack_f16(v[6], v[7]);
        }
    }
    const int end_a = first + q_lo + g + 1, end_b = end_a + 8;  // exclusive key limits of this thread's two rows

    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    float o[8][2][4];  // [d chunk][queries 0-7 / 8-15][fragment]: rows d, d + 1; columns queries 2c, 2c + 1
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2)
#pragma unroll
            for (int j = 0; j < 4; ++j) o[i][h2][j] = 0.f;

    auto stage_v = [&](int base, int buf) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = lane + 32 * i, tok = idx >> 3, ch = idx & 7;
            const int src_tok = min(base + tok, kmax - 1);
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&vst[warp][buf][tok * HD + ((ch ^ (tok & 7)) << 4)]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(vbase + (size_t)src_tok * HD + ch * 16));
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    auto load_k = [&](int base, uint4 (&kr)[4], float (&sc)[8]) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int tok = min(base + nt * 8 + g, kmax - 1);
            const uint4 *p = reinterpret_cast<const uint4 *>(kbase + (size_t)tok * HD + c * 32);
            kr[2 * nt] = p[0];
            kr[2 * nt + 1] = p[1];
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int tok = min(base + nt * 8 + 2 * c + e, kmax - 1);
                sc[nt * 2 + e] = ksc[tok];
                sc[4 + nt * 2 + e] = vsc[tok];
            }
    };

    int buf = 0;
    uint4 kr[4];
    float sc[8];
    if (kmax > 0) { stage_v(0, 0); load_k(0, kr, sc); }
    for (int base = 0; base < kmax; base += 16) {
        uint4 kr_n[4];
        float sc_n[8];
        const int nxt = base + 16;
        if (nxt < kmax) { stage_v(nxt, buf ^ 1); load_k(nxt, kr_n, sc_n); }

        // ---- S = Q.K^T for two 8-token tiles (rows g: fragments 0,1; rows g + 8: fragments 2,3)
        float s_frag[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
            for (int j = 0; j < 4; ++j) s_frag[nt][j] = 0.f;
            const uint32_t w[8] = {kr[2 * nt].x ^ 0x80808080u, kr[2 * nt].y ^ 0x80808080u, kr[2 * nt].z ^ 0x80808080u,
                                   kr[2 * nt].w ^ 0x80808080u, kr[2 * nt + 1].x ^ 0x80808080u, kr[2 * nt + 1].y ^ 0x80808080u,
                                   kr[2 * nt + 1].z ^ 0x80808080u, kr[2 * nt + 1].w ^ 0x80808080u};
#pragma unroll
            for (int s = 0; s < 8; ++s)
                mma_f16_16816(s_frag[nt], qa0[s], qa1[s], qa2[s], qa3[s], i8_pair_f16<0, 1>(w[s]), i8_pair_f16<2, 3>(w[s]));
        }
        // ---- online softmax of rows g and g + 8 over the 16 tokens (causal: token < row limit)
        float pv[2][4], corr[2];
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            const int lim = h2 ? end_b : end_a;
            float sv[4], bm = -INFINITY;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const bool valid = base + nt * 8 + 2 * c + e < lim;
                    sv[nt * 2 + e] = valid ? s_frag[nt][2 * h2 + e] * sc[nt * 2 + e] * a.scale : -INFINITY;
                    bm = fmaxf(bm, sv[nt * 2 + e]);
                }
            bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
            bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
            const float m_new = fmaxf(m_run[h2], bm);
            // a row with no visible key yet keeps m = -inf; exp(-inf - -inf) must not become NaN
            corr[h2] = m_new == -INFINITY ? 1.f : expf(m_run[h2] - m_new);
            float psum = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                pv[h2][i] = m_new == -INFINITY ? 0.f : expf(sv[i] - m_new);
                psum += pv[h2][i];
            }
            psum += __shfl_xor_sync(0xffffffffu, psum, 1);
            psum += __shfl_xor_sync(0xffffffffu, psum, 2);
            l_run[h2] = l_run[h2] * corr[h2] + psum;
            m_run[h2] = m_new;
        }
        // P^T fragments (B operand of P.V) for queries 0-7 and 8-15, times the V scale of their token
        uint32_t pb0[2], pb1[2];
        float c0[2], c1[2];
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            pb0[h2] = pack_f16(pv[h2][0] * sc[4], pv[h2][1] * sc[5]);
            pb1[h2] = pack_f16(pv[h2][2] * sc[6], pv[h2][3] * sc[7]);
            // rescale factors of the queries this thread's output columns belong to (rows 2c, 2c + 1 of the half)
            c0[h2] = __shfl_sync(0xffffffffu, corr[h2], (2 * c) * 4);
            c1[h2] = __shfl_sync(0xffffffffu, corr[h2], (2 * c + 1) * 4);
        }

        // ---- O^T += V^T . P^T  (V block staged in shared memory)
        if (nxt < kmax) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncwarp();
        const uint32_t vs_base = (uint32_t)__cvta_generic_to_shared(&vst[warp][buf][0]);
        const int lm = lane >> 3, lr = lane & 7, ltok = (lm & 1) * 8 + lr;
#pragma unroll
        for (int dp = 0; dp < 4; ++dp) {
            const int ch = 2 * dp + (lm >> 1);
            const uint32_t addr = vs_base + ltok * HD + ((ch ^ (ltok & 7)) << 4);
            uint32_t r0, r1, r2, r3;
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                         : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
            r0 ^= 0x80808080u; r1 ^= 0x80808080u; r2 ^= 0x80808080u; r3 ^= 0x80808080u;
#pragma unroll
            for (int hc = 0; hc < 2; ++hc) {
                const uint32_t lo = hc ? r2 : r0, hi = hc ? r3 : r1;
                const uint32_t va0 = i8_pair_f16<0, 2>(lo), va1 = i8_pair_f16<1, 3>(lo), va2 = i8_pair_f16<0, 2>(hi), va3 = i8_pair_f16<1, 3>(hi);
#pragma unroll
                for (int h2 = 0; h2 < 2; ++h2) {
                    float (&acc)[4] = o[2 * dp + hc][h2];
                    acc[0] *= c0[h2]; acc[1] *= c1[h2]; acc[2] *= c0[h2]; acc[3] *= c1[h2];
                    mma_f16_16816(acc, va0, va1, va2, va3, pb0[h2], pb1[h2]);
                }
            }
        }
        __syncwarp();
        if (nxt < kmax) {
#pragma unroll
            for (int i = 0; i < 4; ++i) kr[i] = kr_n[i];
#pragma unroll
            for (int i = 0; i < 8; ++i) sc[i] = sc_n[i];
        }
        buf ^= 1;
    }

    // ---- normalise and store: this thread holds dims (d, d + 1), d = ch*16 + 2g, of queries 2c, 2c + 1 of each half
#pragma unroll
    for (int h2 = 0; h2 < 2; ++h2) {
        const float l0 = __shfl_sync(0xffffffffu, l_run[h2], (2 * c) * 4), l1 = __shfl_sync(0xffffffffu, l_run[h2], (2 * c + 1) * 4);
        const float i0 = l0 > 0.f ? 1.0f / l0 : 0.f, i1 = l1 > 0.f ? 1.0f / l1 : 0.f;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int qi = q_lo + 8 * h2 + 2 * c + e;
            if (qi >= a.S) continue;
            const size_t ob = (size_t)((long long)rrow * a.st.o_b + (long long)qi * a.st.o_s + (long long)head * a.st.o_h);
            const float inv = e ? i1 : i0;
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
                const int d = ch * 16 + 2 * g;
                st_out(a.out, a.dtype, ob + d, o[ch][h2][e] * inv);
                st_out(a.out, a.dtype, ob + d + 1, o[ch][h2][2 + e] * inv);
            }
        }
    }
}

}  // namespace

template <int KVD, bool MANY>
static int launch_decode_mma(const MmaAttnArgs &a, dim3 grid, cudaStream_t s) {
    using S = AtShape<KVD, MANY>;
    constexpr int smem = S::SMEM;
    static bool configured[64] = {false};  // the attribute is per device
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    if (!configured[dev]) {
        AB2_CUDA(cudaFuncSetAttribute(attn_decode_mma_kernel<KVD, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured[dev] = true;
    }
    int *status = nullptr;
    int rc = device_status_word(&status);
    if (rc != AB2_OK) return rc;
    CUtensorMap kmap, vmap;
    const long long rows = (long long)a.kv.B * a.kv.kvh * a.kv.cap;
    AB2_REQUIRE(rows < (1ll << 31), AB2_ERR_UNSUPPORTED, "decode attention serves caches of less than 2^31 rows");
    const CUtensorMapDataType type = KVD == AB2_KV_INT8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int elem = KVD == AB2_KV_INT8 ? 1 : 2;
    rc = make_rows_map(&kmap, type, elem, a.kv.k, (int)rows, AT_HD, AT_HD, AT_TOK);
    if (rc == AB2_OK) rc = make_rows_map(&vmap, type, elem, a.kv.v, (int)rows, AT_HD, AT_HD, AT_TOK);
    if (rc != AB2_OK) return rc;
    cudaError_t e = launch_kernel(attn_decode_mma_kernel<KVD, MANY>, grid, dim3(32 * S::WARPS), smem, s, kmap, vmap, a, status);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "decode attention launch failed: %s", cudaGetErrorString(e));
    return AB2_OK;
}

// Whether the kernel serves the cache and the queries' type: INT8 rows take queries rounded to fp16 whatever their type, bf16 rows
// take bf16 queries as they are.
bool attention_decode_mma_serves(const ab2_kv *kv, ab2_dtype dtype) {
    return kv->hd == AT_HD && kv->h / kv->kvh <= 8 && (kv->dtype == AB2_KV_INT8 || (kv->dtype == AB2_KV_BF16 && dtype == AB2_BF16));
}

int attention_decode_mma_device(const ab2_kv *kv, int layer, const void *q, void *out, int row0, int nrows,
                                float scale, ab2_dtype dtype, int max_len, int nsplit, float *part_acc, float *part_ml,
                                int pending, long long q_stride, cudaStream_t s) {
    MmaAttnArgs a;
    a.kv = kv_view(kv, layer);
    a.q = q; a.out = out; a.row0 = row0; a.nrows = nrows; a.h = kv->h; a.rep = kv->h / kv->kvh; a.nsplit = nsplit;
    a.dtype = (int)dtype; a.scale = scale; a.part_acc = part_acc; a.part_ml = part_ml; a.counters = kv->counters;
    a.pending = pending; a.q_stride = q_stride;
    // A split costs its arrival and the merge, about 3 us: as long as 512 tokens of a CTA of its own.
    a.min_tokens = 256; a.whole_tokens = 512;
    // Short rows, more of them than the larger CTAs that are resident at once: CTAs of half the warps, twice as many.  us, 8 / 8 heads,
    // larger and smaller: INT8 48 x 16 8.0, 5.0, 64 x 256 12.2, 10.8; bf16 96 x 4 11.2, 8.5, 64 x 256 17.0, 15.4; but long rows bf16 96 x 1500
    // 93, 108, INT8 64 x 4096 ragged 72, 83.
    const bool many = max_len <= a.whole_tokens && nrows * kv->kvh > 2 * device_sm_count();
    a.slots = std::max(1, device_sm_count() * 2 / kv->kvh);
    // What the launch would find from lengths that the host can bound: no CTA has to read all rows' lengths.
    a.whole = nsplit == 1 || max_len <= a.whole_tokens;
    const dim3 grid((unsigned)(a.whole ? nrows : std::max<long long>(nrows, std::min<long long>(a.slots, (long long)nrows * nsplit))), kv->kvh);
    if (kv->dtype == AB2_KV_INT8) return many ? launch_decode_mma<AB2_KV_INT8, true>(a, grid, s) : launch_decode_mma<AB2_KV_INT8, false>(a, grid, s);
    return many ? launch_decode_mma<AB2_KV_BF16, true>(a, grid, s) : launch_decode_mma<AB2_KV_BF16, false>(a, grid, s);
}

// S > 1 queries per row over an INT8 cache, head_dim 128, 1..4 query heads per KV head: the
// tensor-core causal kernel.  AB2_ERR_UNSUPPORTED otherwise (the caller keeps the general kernel).
int attention_prefill_mma_device(const ab2_kv *kv, int layer, const void *q, void *out, int S, int pending, int row0,
                                 int nrows, float scale, ab2_dtype dtype, AttnStrides st, cudaStream_t s) {
    const int rep = kv->h / kv->kvh;
    if (kv->dtype != AB2_KV_INT8 || kv->hd != 128 || rep > 4 || S < 2) return AB2_ERR_UNSUPPORTED;
    PrefillAttnArgs a;
    a.kv = kv_view(kv, layer);
    a.q = q; a.out = out; a.st = st; a.S = S; a.pending = pending; a.row0 = row0; a.rep = rep;
    a.dtype = (int)dtype; a.scale = scale;
    cudaError_t e = launch_kernel(attn_prefill_mma_kernel, dim3((S + 15) / 16, kv->kvh, nrows), dim3(128), 0, s, a);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "prefill attention launch failed: %s", cudaGetErrorString(e));
    return AB2_OK;
}

}  // namespace ab2
