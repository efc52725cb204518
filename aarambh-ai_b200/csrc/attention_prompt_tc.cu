// Causal attention of a prompt portion in bf16 on the 5th-generation tensor cores, over keys and values laid
// out position by position (PromptAttnArgs): projected latents, the cache of a dense decoder (bf16 rows as they are,
// INT8 codes after one pass that widens them), the ring of a window layer (copied straight where it wraps).  A CTA
// owns 128 queries of a head and walks the keys in its sight 128 at a time:
//
//   S[128 queries][128 keys] = Q . K^T         both K-major in shared memory
//   O[128 queries][vdim]    += (P_hi + P_lo) . V   P in tensor memory, V N-major in shared memory
//
// The softmax weights enter as two bf16 terms, the rounded weight and what rounding left, so the product carries
// them to about 16 significant bits.
//
//   warp 0       TMA producer: K and V tiles, two of each in flight
//   warp 1       MMA issue of the scores;   warp 2   MMA issue of the sums
//   warps 4-7    softmax of the even key tiles, a thread per query, with sums O_0 of their own
//   warps 8-11   softmax of the odd key tiles, with O_1; the two halves are merged at the end
// Tensor memory: S_0, S_1 (128 columns each; the weights take the place of the scores), O_0, O_1.  The
// weights are relative to a maximum per query that moves only when a score exceeds it by 2^8; then the query's
// sums are rescaled in tensor memory.
// The chain scores - softmax - sums of a half bounds it, about 2 us a tile of 128 x 128 against the 0.8 us of its
// MMAs.  32 / 8 heads of 128: 3001 tokens over an INT8 cache 787 us on the warp-level tensor cores, 222 + 11 (widening) here;
// 1000 tokens behind 500 over a bf16 cache 1344 us on CUDA cores, 50 here; 2048 tokens of 16 / 4 heads with a window of
// 1024: 114 -> 48.  Below 16 queries a CTA would be nearly empty; short contexts and many short sequences stay with the other kernels
// (prompt_tc_pays).
// The MMA multiplies a tile of values whole, a hidden one by a weight of 0, so an Inf or a NaN in it would reach queries
// that do not see it.  A query whose sums came out as either is computed again on CUDA cores over the keys in its sight.
// Every wait on an mbarrier is bounded; on a time-out the CTA records AB2_ERR_TIMEOUT, stops issuing
// work, frees its tensor memory and returns.
#include <algorithm>
#include <cstring>

#include "kv_cache.cuh"
#include "stack.cuh"
#include "tcgen05_util.cuh"

using namespace ab2;
using namespace ab2::tc;

namespace ab2 {
int device_status_word(int **out);
int device_sm_count();
namespace {

constexpr int PT_Q = 128, PT_KEYS = 128, PT_THREADS = 384, PT_BOX = 128 * 128;  // a box is 128 rows of 64 elements
constexpr int PT_SMEM = 227 * 1024;
constexpr int PT_MIN_QUERIES = 16;  // fewer go to the kernels that read the cache as it is
constexpr float PT_SLACK = 8.f;  // powers of two a score may exceed the query's maximum by

struct PtShared {
    uint64_t kfull[2], kempty[2], vfull[2], vempty[2], sfull[2], pfull[2], odone[2];
    uint32_t tmem_base;
    int failed;
    float top[2][PT_Q], sum[2][PT_Q];
    uint32_t again[2][4];  // queries to compute again, a bit each: by half of the warps and quarter of the queries
    // scales of a tile's keys and values: a half's tile is read from one buffer while its next is written to the other
    alignas(16) float ks[2][2][PT_KEYS], vs[2][2][PT_KEYS];
};

struct PtArgs {
    PromptAttnArgs a;
    int main_boxes, tail_boxes, v_boxes;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
// One tile of keys for the warp's 32 queries, a lane each: scores to weights in tensor memory.  With EDGE the keys
// before `lo` and past `lim` are out of sight.  With SCALED a score is multiplied by its key's scale and a weight, after it has been
// counted, by its value's.  o_blocks blocks of 32 columns hold sums so far.
template <bool EDGE, bool SCALED>
__device__ __forceinline__ void softmax_tile(uint32_t s_addr, uint32_t o_addr, float sl, int lo, int lim, const float *ks, const float *vs, int o_blocks, float &top,
                                             float &sum) {
    // two buffers: the next 32 scores are on their way while these are looked at
    uint32_t v[2][32];
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
    tmem_ld32_start(v[0], s_addr);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        tmem_ld32_wait(v[c & 1]);
        tmem_ld32_start(v[(c + 1) & 1], s_addr + 32 * ((c + 1) & 3));  // the last one fetches the first again
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
            float f[4] = {__uint_as_float(v[c & 1][k]), __uint_as_float(v[c & 1][k + 1]), __uint_as_float(v[c & 1][k + 2]), __uint_as_float(v[c & 1][k + 3])};
            if (SCALED) {
                const float4 q = *reinterpret_cast<const float4 *>(ks + 32 * c + k);
                f[0] *= q.x; f[1] *= q.y; f[2] *= q.z; f[3] *= q.w;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], EDGE && (32 * c + k + e > lim || 32 * c + k + e < lo) ? -INFINITY : f[e]);
        }
    }
    tmem_ld32_wait(v[0]);
    const float best = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl;  // the scale is positive
    const float now = best > top + PT_SLACK ? best : top;
    if (__any_sync(0xffffffffu, now != top)) {
        const float corr = ex2(top - now);
        sum *= corr;
        top = now;
        // the scores came after the products of this half's last tile: its sums stand still
#pragma unroll 1
        for (int c = 0; c < o_blocks; ++c) {
            uint32_t o[32];
            tmem_ld32(o, o_addr + 32 * c);
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * corr);
            tmem_st32(o_addr + 32 * c, o);
        }
    }
    float part_sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (c > 0) tmem_ld32_wait(v[c & 1]);
        if (c < 3) tmem_ld32_start(v[(c + 1) & 1], s_addr + 32 * (c + 1));
        uint32_t w[32];
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
            float f[4] = {__uint_as_float(v[c & 1][k]), __uint_as_float(v[c & 1][k + 1]), __uint_as_float(v[c & 1][k + 2]), __uint_as_float(v[c & 1][k + 3])};
            if (SCALED) {
                const float4 q = *reinterpret_cast<const float4 *>(ks + 32 * c + k);
                f[0] *= q.x; f[1] *= q.y; f[2] *= q.z; f[3] *= q.w;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                f[e] = ex2(fmaf(f[e], sl, -top));
                if (EDGE && (32 * c + k + e > lim || 32 * c + k + e < lo)) f[e] = 0.f;
            }
            part_sum[(k >> 1) & 3] += f[0] + f[1];
            part_sum[((k >> 1) + 1) & 3] += f[2] + f[3];
            if (SCALED) {
                const float4 q = *reinterpret_cast<const float4 *>(vs + 32 * c + k);
                f[0] *= q.x; f[1] *= q.y; f[2] *= q.z; f[3] *= q.w;
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const int i = (k + e) >> 1;
                const __nv_bfloat162 h = __floats2bfloat162_rn(f[e], f[e + 1]);
                w[i] = *reinterpret_cast<const uint32_t *>(&h);
                const __nv_bfloat162 l = __floats2bfloat162_rn(f[e] - __uint_as_float(w[i] << 16), f[e + 1] - __uint_as_float(w[i] & 0xffff0000u));
                w[16 + i] = *reinterpret_cast<const uint32_t *>(&l);
            }
        }
        tmem_st32(s_addr + 32 * c, w);
    }
    sum += (part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3]);
}

// Where a sequence's keys are: its first query is row `first` of those that are counted from its first key in sight, the keys of a head
// are matrix z, whose row y0 that key is, and its scales start at `scales`.
struct PtWhere {
    int seq, first, z, y0;
    size_t scales;
};
__device__ __forceinline__ PtWhere pt_where(const PromptAttnArgs &a, int seq, int kv_head) {
    const int kvh = a.rep > 1 ? a.heads / a.rep : a.heads, row = a.rows ? a.rows[a.row0 + seq] : a.row0 + seq;
    const int at = a.lens ? a.lens[row] + a.pending - a.S : a.first, base = a.window ? max(0, at - a.window + 1) : 0;
    PtWhere w;
    w.seq = seq;
    w.first = at - base;
    w.z = a.k_z ? (a.gathered ? seq : row) * kvh + kv_head : 0;
    w.y0 = a.ring ? base % a.ring : 0;
    w.scales = ((size_t)row * kvh + kv_head) * a.scale_z;
    return w;
}

// A query's output over the keys of rows [from, to], by one warp: a lane has every 32nd dimension.  Where the fast path's
// sums were sound this gives the same value, otherwise what a sum over the keys in sight alone gives.
__device__ __noinline__ void attend_again(const PromptAttnArgs &a, int head, int qi, int from, int to, int lane) {
    constexpr int QD = 6, VD = 4;  // dim + tail_dims <= 192 (what shared memory holds), vdim <= 128
    const int dims = a.dim + a.tail_dims;
    const int kv_head = a.rep > 1 ? head / a.rep : head;
    const PtWhere at = pt_where(a, blockIdx.z, kv_head);
    const __nv_bfloat16 *q = a.q + at.seq * a.q_row + (size_t)qi * a.q_stride + (size_t)head * dims;
    const __nv_bfloat16 *k = a.k + (size_t)at.z * a.k_z + (size_t)kv_head * a.k_head + (size_t)at.y0 * a.k_stride;
    const __nv_bfloat16 *v = a.v + (size_t)at.z * a.v_z + (size_t)kv_head * a.v_head + (size_t)at.y0 * a.v_stride;
    float qv[QD], acc[VD] = {}, top = -INFINITY, sum = 0.f;
#pragma unroll
    for (int i = 0; i < QD; ++i) qv[i] = lane + 32 * i < dims ? __bfloat162float(q[lane + 32 * i]) : 0.f;
    for (int key = from; key <= to; ++key) {
        float s = 0.f, vv[VD];
#pragma unroll
        for (int i = 0; i < QD; ++i) {
            const int d = lane + 32 * i;
            if (d < dims) s = fmaf(qv[i], __bfloat162float(d < a.dim ? k[(size_t)key * a.k_stride + d] : a.tail[(size_t)key * a.tail_stride + d - a.dim]), s);
        }
#pragma unroll
        for (int i = 0; i < VD; ++i) vv[i] = lane + 32 * i < a.vdim ? __bfloat162float(v[(size_t)key * a.v_stride + lane + 32 * i]) : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        s *= a.scale;
        if (a.k_scale) s *= a.k_scale[at.scales + key];
        const float best = fmaxf(top, s), keep = top == best ? 1.f : expf(top - best);
        float w = s == -INFINITY ? 0.f : expf(s - best);
        sum = sum * keep + w;
        if (a.v_scale) w *= a.v_scale[at.scales + key];
#pragma unroll
        for (int i = 0; i < VD; ++i) acc[i] = fmaf(w, vv[i], acc[i] * keep);
        top = best;
    }
    float scale = sum > 0.f ? 1.f / sum : 1.f;  // a NaN is in acc
    if (a.gate) scale /= 1.f + expf(-__bfloat162float(a.gate[(size_t)qi * a.gate_stride + head]));
#pragma unroll
    for (int i = 0; i < VD; ++i)
        if (lane + 32 * i < a.vdim) a.out[at.seq * a.out_row + (size_t)qi * a.out_stride + (size_t)head * a.vdim + lane + 32 * i] = __float2bfloat16_rn(acc[i] * scale);
}

template <bool SCALED>
__global__ void __launch_bounds__(PT_THREADS, 1)
prompt_tc_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap vmap, const __grid_constant__ PtArgs p, int *status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *qbuf = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const PromptAttnArgs &a = p.a;
    const int kboxes = p.main_boxes + p.tail_boxes;
    uint8_t *kbuf = qbuf + kboxes * PT_BOX, *vbuf = kbuf + 2 * kboxes * PT_BOX;
    PtShared *sh = (PtShared *)(vbuf + 2 * p.v_boxes * PT_BOX);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head = blockIdx.x;
    const int q_lo = ((int)gridDim.y - 1 - (int)blockIdx.y) * PT_Q;  // the longest walks of every head first
    const int kv_head = a.rep > 1 ? head / a.rep : head;
    volatile int *failed = &sh->failed;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            bar_init(&sh->kfull[i], 1); bar_init(&sh->kempty[i], 1); bar_init(&sh->vfull[i], 1); bar_init(&sh->vempty[i], 1);
            bar_init(&sh->sfull[i], 1); bar_init(&sh->pfull[i], 4); bar_init(&sh->odone[i], 1);
        }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(sptr(&sh->tmem_base)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    pdl_wait();
    pdl_launch_dependents();
    const PtWhere where = pt_where(a, blockIdx.z, kv_head);
    const int first = where.first;
    // tiles of keys in sight of the first query (from t0 on) to that of the last
    const int t0 = a.window ? max(0, first + q_lo - a.window + 1) / PT_KEYS : 0;
    const int tiles = (first + min(a.S, q_lo + PT_Q) + PT_KEYS - 1) / PT_KEYS - t0;
    auto load_k = [&](int j) {
        uint8_t *dst = kbuf + (j & 1) * kboxes * PT_BOX;
        bar_expect_tx(&sh->kfull[j & 1], (uint32_t)(kboxes * PT_BOX));
        for (int b = 0; b < p.main_boxes; ++b) tma_load_3d(dst + b * PT_BOX, &kmap, kv_head * a.k_head + b * 64, where.y0 + (t0 + j) * PT_KEYS, where.z, &sh->kfull[j & 1]);
        for (int b = 0; b < p.tail_boxes; ++b) tma_load_2d(dst + (p.main_boxes + b) * PT_BOX, &tmap, b * 64, (t0 + j) * PT_KEYS, &sh->kfull[j & 1]);
    };
    auto load_v = [&](int j) {
        uint8_t *dst = vbuf + (j & 1) * p.v_boxes * PT_BOX;
        bar_expect_tx(&sh->vfull[j & 1], (uint32_t)(p.v_boxes * PT_BOX));
        for (int b = 0; b < p.v_boxes; ++b) tma_load_3d(dst + b * PT_BOX, &vmap, kv_head * a.v_head + b * 64, where.y0 + (t0 + j) * PT_KEYS, where.z, &sh->vfull[j & 1]);
    };
    if (threadIdx.x == 0)
        for (int j = 0; j < min(2, tiles); ++j) { load_k(j); load_v(j); }
    // the queries, in boxes like the keys; what a head or the portion does not have is zero
    for (int i = threadIdx.x; i < kboxes * PT_Q * 8; i += PT_THREADS) {
        const int ch = i & 7, r = (i >> 3) % PT_Q, b = (i >> 3) / PT_Q;
        const int d = (b < p.main_boxes ? b : b - p.main_boxes) * 64 + ch * 8;
        const bool in = q_lo + r < a.S && d < (b < p.main_boxes ? a.dim : a.tail_dims);
        const uint4 v = in ? *reinterpret_cast<const uint4 *>(a.q + where.seq * a.q_row + (size_t)(q_lo + r) * a.q_stride + (size_t)head * (a.dim + a.tail_dims) + (b < p.main_boxes ? d : a.dim + d))
                           : make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4 *>(qbuf + b * PT_BOX + r * 128 + ((ch ^ (r & 7)) << 4)) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = sh->tmem_base, tmem_o = tmem + 2 * PT_KEYS;  // O_0 and O_1 128 columns apart
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
    if (warp == 0) {
        // ---------------------------------------------------------- TMA producer
        if (lane == 0)
            for (int j = 2; j < tiles && !*failed; ++j) {
                if (!bar_wait(&sh->kempty[j & 1], ((j >> 1) & 1) ^ 1, failed)) break;
                load_k(j);
                if (!bar_wait(&sh->vempty[j & 1], ((j >> 1) & 1) ^ 1, failed)) break;
                load_v(j);
            }
    } else if (warp == 1) {
        // ---------------------------------------------------------- scores
        const uint32_t idesc = IDESC | ((uint32_t)(PT_KEYS >> 3) << 17);
        for (int j = 0; j < tiles; ++j) {
            if (!warp_wait(&sh->kfull[j & 1], (j >> 1) & 1, failed)) break;
            // the weights that lie in this score buffer have been multiplied
            if (j >= 2 && !warp_wait(&sh->odone[j & 1], ((j >> 1) - 1) & 1, failed)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (elect_one()) {
                for (int b = 0; b < kboxes; ++b) {
                    const uint64_t qd = umma_desc(sptr(qbuf + b * PT_BOX)), kd = umma_desc(sptr(kbuf + ((j & 1) * kboxes + b) * PT_BOX));
#pragma unroll
                    for (int k = 0; k < 4; ++k)  // descriptors count in 16 bytes
                        umma_bf16(tmem + (uint32_t)((j & 1) * PT_KEYS), qd + (uint64_t)(2 * k), kd + (uint64_t)(2 * k), idesc, (b | k) != 0);
                }
                umma_commit(&sh->kempty[j & 1]);
                umma_commit(&sh->sfull[j & 1]);
            }
            __syncwarp();
        }
    } else if (warp == 2) {
        // ---------------------------------------------------------- sums
        const uint32_t idesc = IDESC | (1u << 16) | ((uint32_t)(p.v_boxes * 64 >> 3) << 17);
        for (int j = 0; j < tiles; ++j) {
            if (!warp_wait(&sh->vfull[j & 1], (j >> 1) & 1, failed) || !warp_wait(&sh->pfull[j & 1], (j >> 1) & 1, failed)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (elect_one()) {
                const uint64_t vd = umma_desc_mn(sptr(vbuf + (j & 1) * p.v_boxes * PT_BOX), PT_BOX);
                const uint32_t w = tmem + (uint32_t)((j & 1) * PT_KEYS), o = tmem_o + (uint32_t)((j & 1) * 128);
#pragma unroll
                for (int k = 0; k < PT_KEYS / 16; ++k) {
                    const uint32_t at = w + (uint32_t)((k >> 1) * 32 + (k & 1) * 8);  // 32 keys: 16 columns of rounded weights, 16 of the rest
                    umma_bf16_ts(o, at, vd + (uint64_t)(k * (2048 >> 4)), idesc, j >= 2 || k > 0);
                    umma_bf16_ts(o, at + 16, vd + (uint64_t)(k * (2048 >> 4)), idesc, 1);
                }
                umma_commit(&sh->vempty[j & 1]);
                umma_commit(&sh->odone[j & 1]);
            }
            __syncwarp();
        }
    } else if (warp >= 4) {
        // ---------------------------------------------------------- softmax
        const int part = (warp - 4) >> 2, quad = warp & 3, r = quad * 32 + lane;
        const int pos = first + q_lo + r;
        const uint32_t quad_addr = (uint32_t)(quad * 32) << 16, s_addr = tmem + quad_addr + (uint32_t)(part * PT_KEYS), o_addr = tmem_o + quad_addr + (uint32_t)(part * 128);
        const float sl = a.scale * 1.44269504088896341f;  // scores in powers of two
        float top = -1e30f, sum = 0.f;
        bool ok = true;
        // the thread fetches the scales of key r of its half's next tile
        const int rows = first + a.S;
        auto scale_of = [&](const float *p, int j) { const int k = (t0 + j) * PT_KEYS + r; return j < tiles && k < rows ? __ldg(p + where.scales + k) : 0.f; };
        float ks_next = SCALED ? scale_of(a.k_scale, part) : 0.f, vs_next = SCALED ? scale_of(a.v_scale, part) : 0.f;
        for (int j = part; j < tiles; j += 2) {
            const int buf = (j >> 1) & 1;
            if (SCALED) {
                sh->ks[part][buf][r] = ks_next;
                sh->vs[part][buf][r] = vs_next;
                ks_next = scale_of(a.k_scale, j + 2);
                vs_next = scale_of(a.v_scale, j + 2);
                asm volatile("barrier.cta.sync %0, 128;\n" ::"r"(2 + part) : "memory");
            }
            ok = warp_wait(&sh->sfull[part], (j >> 1) & 1, failed);
            if (!SCALED && !ok) break;  // with scales the warps go on to their barrier together; what they write is not read
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int at = (t0 + j) * PT_KEYS;
            const bool edge = at + PT_KEYS - 1 > first + q_lo || (a.window && at < first + q_lo + PT_Q - a.window);
            const int lim = pos - at, lo = a.window ? lim - a.window + 1 : -0x40000000;  // keys of the tile in sight
            const int o_blocks = j >= 2 ? p.v_boxes * 2 : 0;
            if (edge) softmax_tile<true, SCALED>(s_addr, o_addr, sl, lo, lim, sh->ks[part][buf], sh->vs[part][buf], o_blocks, top, sum);
            else softmax_tile<false, SCALED>(s_addr, o_addr, sl, lo, lim, sh->ks[part][buf], sh->vs[part][buf], o_blocks, top, sum);
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&sh->pfull[part]);
        }
        sh->top[part][r] = top;
        sh->sum[part][r] = sum;
        const int mine = (tiles - part + 1) / 2;  // tiles of this half
        if (ok && mine > 0) ok = warp_wait(&sh->odone[part], (mine - 1) & 1, failed);
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        asm volatile("barrier.cta.sync 1, 256;\n" ::: "memory");
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        uint32_t again = 0;
        if (!__any_sync(0xffffffffu, *failed)) {
            float poison = 0.f;  // stays 0 unless an output is Inf or NaN
            // both halves of the warps store: value boxes of 64 dimensions in turn
            const float t0 = sh->top[0][r], t1 = sh->top[1][r], t = fmaxf(t0, t1);
            float f0 = ex2(t0 - t), f1 = tiles > 1 ? ex2(t1 - t) : 0.f;
            float scale = 1.f / (f0 * sh->sum[0][r] + f1 * sh->sum[1][r]);
            const int qi = q_lo + r;
            if (a.gate && qi < a.S) scale /= 1.f + expf(-__bfloat162float(a.gate[(size_t)qi * a.gate_stride + head]));
            f0 *= scale;
            f1 *= scale;
            __nv_bfloat16 *dst = a.out + where.seq * a.out_row + (size_t)qi * a.out_stride + (size_t)head * a.vdim;
#pragma unroll 1
            for (int c = part; c < p.v_boxes * 2; c += 2) {
                uint32_t v[32], w[32];
                __syncwarp();
                tmem_ld32(v, tmem_o + quad_addr + 32 * c);
                if (tiles > 1) tmem_ld32(w, tmem_o + quad_addr + 128 + 32 * c);
                else
#pragma unroll
                    for (int k = 0; k < 32; ++k) w[k] = 0u;
#pragma unroll
                for (int k = 0; k < 32; k += 8) {
                    uint32_t o[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int n = k + 2 * e;
                        const float x = f0 * __uint_as_float(v[n]) + f1 * __uint_as_float(w[n]), y = f0 * __uint_as_float(v[n + 1]) + f1 * __uint_as_float(w[n + 1]);
                        poison = fmaf(y, 0.f, fmaf(x, 0.f, poison));
                        const __nv_bfloat162 q = __floats2bfloat162_rn(x, y);
                        o[e] = *reinterpret_cast<const uint32_t *>(&q);
                    }
                    if (qi < a.S && 32 * c + k < a.vdim) *reinterpret_cast<uint4 *>(dst + 32 * c + k) = make_uint4(o[0], o[1], o[2], o[3]);
                }
            }
            again = __ballot_sync(0xffffffffu, qi < a.S && poison != 0.f);  // NaN is not 0
        }
        if (lane == 0) sh->again[part][quad] = again;
        asm volatile("barrier.cta.sync 1, 256;\n" ::: "memory");
        for (int i = 0, n = 0; i < 4; ++i)
            for (uint32_t rows_left = sh->again[0][i] | sh->again[1][i]; rows_left; rows_left &= rows_left - 1, ++n)
                if ((n & 7) == warp - 4) {
                    const int at = q_lo + 32 * i + __ffs(rows_left) - 1, to = first + at;
                    attend_again(a, head, at, a.window ? max(0, to - a.window + 1) : 0, to, lane);
                }
    }

    // ---- teardown: every warp arrives here (all waits are bounded)
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && sh->failed) atomicExch(status, (int)AB2_ERR_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
    }
}

size_t prompt_tc_smem(const PtArgs &p) { return 1024 + (size_t)(3 * (p.main_boxes + p.tail_boxes) + 2 * p.v_boxes) * PT_BOX + sizeof(PtShared); }

template <bool SCALED>
int launch_prompt(const PtArgs &p, const CUtensorMap &kmap, const CUtensorMap &tmap, const CUtensorMap &vmap, int *status, cudaStream_t s) {
    static bool configured[64] = {false};  // the attribute is per device
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    if (!configured[dev]) {
        AB2_CUDA(cudaFuncSetAttribute(prompt_tc_kernel<SCALED>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM));
        configured[dev] = true;
    }
    cudaError_t e = launch_kernel(prompt_tc_kernel<SCALED>, dim3(p.a.heads, (p.a.S + PT_Q - 1) / PT_Q, std::max(1, p.a.nrows)), dim3(PT_THREADS), prompt_tc_smem(p), s, kmap, tmap, vmap, p, status);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "prompt attention launch failed: %s", cudaGetErrorString(e));
    return AB2_OK;
}

// The keys and values in sight of every sequence and head, one after the other: INT8 codes as the bf16 integers they are, or the rows
// of a ring of `cap` slots.  blockIdx.y is the head, z the sequence's keys or values; 16 bytes of the output a thread.
struct PtGather {
    PromptAttnArgs a;      // whose sequences; k and v are the copies, `n` rows a matrix
    const void *src[2];
    int ld[2];             // elements of a row, a multiple of 8
    long long src_z[2];    // elements between matrices of the source
    int n, cap;
};
template <bool INT8>
__global__ void __launch_bounds__(256) prompt_gather_kernel(const __grid_constant__ PtGather g) {
    pdl_wait();
    pdl_launch_dependents();
    const int w = blockIdx.z & 1, seq = blockIdx.z >> 1, per = (w ? g.ld[1] : g.ld[0]) >> 3;
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= (size_t)g.n * per) return;
    const PromptAttnArgs &a = g.a;
    const int r = (int)(i / per), c = (int)(i % per) * 8, row = a.rows ? a.rows[a.row0 + seq] : a.row0 + seq;
    const int at = a.lens ? a.lens[row] + a.pending - a.S : a.first, base = a.window ? max(0, at - a.window + 1) : 0;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);  // past a shorter sequence: multiplied by weights of 0
    if (r < at + a.S - base) {
        const size_t from = ((size_t)row * gridDim.y + blockIdx.y) * (w ? g.src_z[1] : g.src_z[0]) + (size_t)((base + r) % g.cap) * (per * 8) + c;
        if (INT8) {
            const uint2 q = *reinterpret_cast<const uint2 *>((const int8_t *)(w ? g.src[1] : g.src[0]) + from);
            // a code is the difference of two bf16 between 128 and 256, as in the INT8 GEMM
            auto pair = [](uint32_t x, uint32_t sel) {
                const uint32_t b = __byte_perm(x, 0u, sel);
                return bf16x2_add_((b & 0x007F007Fu) | 0x43004300u, (b & 0x00800080u) | 0xC300C300u);
            };
            v = make_uint4(pair(q.x, 0x4140), pair(q.x, 0x4342), pair(q.y, 0x4140), pair(q.y, 0x4342));
        } else {
            v = *reinterpret_cast<const uint4 *>((const __nv_bfloat16 *)(w ? g.src[1] : g.src[0]) + from);
        }
    }
    __nv_bfloat16 *dst = const_cast<__nv_bfloat16 *>(w ? a.v : a.k);
    *reinterpret_cast<uint4 *>(dst + (((size_t)seq * gridDim.y + blockIdx.y) * g.n + r) * (per * 8) + c) = v;
}

// The attention of `p` over gathered keys and values, `g` saying where they come from and how many (at most) a sequence has in sight, `heads` of
// them a sequence: as many sequences at a time as SCRATCH_ROWS_BYTES hold, one at least.  AB2_ERR_UNSUPPORTED where there is no
// memory for them: the kernels that read the cache as it is need none.
constexpr size_t SCRATCH_ROWS_BYTES = (size_t)160 << 20;  // what the scratch pool keeps
int attention_gathered(PtGather g, PromptAttnArgs p, bool int8, int heads, cudaStream_t s) {
    const size_t kb = (size_t)heads * g.n * g.ld[0] * 2, vb = (size_t)heads * g.n * g.ld[1] * 2;  // multiples of 16 bytes
    const int nrows = std::max(1, p.nrows), at_once = (int)std::min<size_t>(nrows, std::max<size_t>(1, SCRATCH_ROWS_BYTES / (kb + vb)));
    ScratchLease ws(s);
    if (!ws.take(at_once * (kb + vb))) return AB2_ERR_UNSUPPORTED;
    const int row0 = p.row0;
    p.k = (__nv_bfloat16 *)ws.ptr;
    p.v = (__nv_bfloat16 *)((char *)ws.ptr + at_once * kb);
    p.k_stride = g.ld[0]; p.v_stride = g.ld[1];
    p.k_z = (long long)g.n * g.ld[0]; p.v_z = (long long)g.n * g.ld[1];
    p.key_rows = g.n; p.ring = 0; p.gathered = true;
    for (int done = 0; done < nrows; done += at_once) {
        const int now = std::min(at_once, nrows - done);
        p.nrows = now; p.mats = now * heads; p.row0 = row0 + done;
        g.a = p;
        const dim3 grid((unsigned)(((size_t)g.n * (std::max(g.ld[0], g.ld[1]) / 8) + 255) / 256), heads, 2 * now);
        cudaError_t e = int8 ? launch_kernel(prompt_gather_kernel<true>, grid, dim3(256), 0, s, g) : launch_kernel(prompt_gather_kernel<false>, grid, dim3(256), 0, s, g);
        if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "prompt attention launch failed: %s", cudaGetErrorString(e));
        int rc = prompt_tc_attention(p, s);
        if (rc != AB2_OK) return rc;
        p.q += now * p.q_row;
        p.out += now * p.out_row;
    }
    return AB2_OK;
}

// Which kernel takes a prompt: the faster one by what they take, in us, measured (launches in a row) over 1 to 32 sequences of 16 to 2048
// queries behind 0 to 4096 tokens, 16 / 4 heads of 64 and 32 / 8 of 128 (caches) and windows of 128, 1024 and 2048 over 8 / 2 to 32 / 8
// heads.  The estimates are within a third of the times and pick the slower kernel, by at most 7 %, in 4 of 330 cases.  Examples, this kernel
// against the other: INT8 cache, 32 / 8 x 128, 1 x 16 queries alone 22 / 10, behind 512 tokens 27 / 41; 32 x 64 behind 512 194 / 208, alone
// 86 / 42; bf16 cache, 32 x 16 alone 66 / 37, behind 512 118 / 391; window 1024 of 16 / 4 x 128, 1 x 64 alone 30 / 19, 1 x 512 25 / 30.
struct KeyWalk {
    double mean;       // tiles of keys that a tile of queries walks
    int most, tiles;   // and tiles of queries
};
KeyWalk key_walk(int first, int S, int window, int queries, int keys) {
    KeyWalk w = {0.0, 0, 0};
    for (int lo = 0; lo < S; lo += queries, ++w.tiles) {
        const int from = window ? std::max(0, first + lo - window + 1) / keys : 0, n = (first + std::min(S, lo + queries) + keys - 1) / keys - from;
        w.mean += n;
        w.most = std::max(w.most, n);
    }
    w.mean /= w.tiles;
    return w;
}
// A CTA has its SM to itself; the `gathered` bytes that a pass before it moves go at 4 TB/s.
double prompt_tc_us(const PromptAttnArgs &p, int first, bool scaled, double gathered) {
    const KeyWalk w = key_walk(first, p.S, p.window, PT_Q, PT_KEYS);
    const bool wide = std::max(p.dim, p.vdim) > 64;
    const int rounds = (int)(((long long)p.heads * p.nrows * w.tiles + device_sm_count() - 1) / device_sm_count());
    const double one = scaled ? (wide ? 10.6 : 8.9) : (wide ? 9.4 : 8.3), more = scaled ? (wide ? 2.45 : 1.9) : (wide ? 1.7 : 1.15);
    const double full = (scaled ? 4.0 : 2.5) * std::min(p.S, PT_Q) / PT_Q;  // queries and outputs of a round that waits for the one before
    const double us = rounds == 1 ? one + more * (w.most - 1) : rounds * (one + full + more * (w.mean - 1));
    return us + (gathered > 0 ? 5 + gathered / 4e6 : 0);
}
// window_attn_mma_kernel: tiles of 64 queries and 64 keys, several CTAs an SM.
double window_mma_us(const PromptAttnArgs &p, int first) {
    const KeyWalk w = key_walk(first, p.S, p.window, 64, 64);
    const bool wide = std::max(p.dim, p.vdim) > 64;
    return std::max(2 + (wide ? 1.75 : 1.15) * w.most, (double)p.heads * p.nrows * w.tiles * (wide ? 0.017 + 0.0145 * w.mean : 0.008 + 0.0075 * w.mean));
}
// The kernels that read a cache as it is: attn_prefill_mma_kernel (16 queries, 16 keys a step) and attn_split_kernel (a CTA a query).
double cache_other_us(const PromptAttnArgs &p, int first, bool int8) {
    const int kvh = p.heads / p.rep;
    const double keys = first + (p.S + 1) / 2.0;
    if (int8 && p.dim == 128 && p.rep <= 4) {
        const double steps = keys / 16, ctas = (double)p.nrows * kvh * ((p.S + 15) / 16);
        return std::max(6 + 1.04 * steps, ctas * (0.033 + 0.0053 * steps));
    }
    const bool wide = p.dim > 64;
    const double key = int8 ? (wide ? 1.2e-4 : 7.3e-5) : (wide ? 1.67e-4 : 9.4e-5), alone = int8 ? (wide ? 0.05 : 0.0385) : (wide ? 0.042 : 0.031);
    return std::max(6.5 + alone * keys, (double)p.nrows * p.S * kvh * ((wide ? 0.008 : 0.006) + key * keys));
}
bool prompt_tc_pays(double here, double other) {
    static const char *force = getenv("AB2_PROMPT_ATTN");  // measurement and test switch: tc, other
    return force ? strcmp(force, "tc") == 0 : here < other;
}

// The host's lengths are those of the rows when the launch runs, unless the launch is recorded to run again.
bool lengths_known(cudaStream_t s) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
}

}  // namespace

bool prompt_tc_serves(const PromptAttnArgs &a) {
    const PtArgs p = {a, (a.dim + 63) / 64, (a.tail_dims + 63) / 64, (a.vdim + 63) / 64};
    return a.scale >= 0.f && a.dim % 8 == 0 && a.tail_dims % 8 == 0 && a.vdim % 8 == 0 && p.v_boxes <= 2 && prompt_tc_smem(p) <= PT_SMEM && a.q_stride % 8 == 0 &&
           a.k_stride % 8 == 0 && a.v_stride % 8 == 0 && a.tail_stride % 8 == 0 && a.k_head % 8 == 0 && a.v_head % 8 == 0 && a.out_stride % 8 == 0 &&
           a.k_z % 8 == 0 && a.v_z % 8 == 0 && a.q_row % 8 == 0 && a.out_row % 8 == 0 &&
           (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.tail | (uintptr_t)a.out) & 15) == 0;
}

int prompt_tc_attention(const PromptAttnArgs &a, cudaStream_t s) {
    const PtArgs p = {a, (a.dim + 63) / 64, (a.tail_dims + 63) / 64, (a.vdim + 63) / 64};
    int *status = nullptr;
    int rc = device_status_word(&status);
    CUtensorMap kmap, tmap, vmap;
    const int heads = a.heads / std::max(1, a.rep), L = a.k_z ? a.key_rows : a.first + a.S;
    const int mats = a.k_z ? a.mats : 1, kcols = a.k_z ? a.dim : (heads - 1) * a.k_head + a.dim, vcols = a.k_z ? a.vdim : (heads - 1) * a.v_head + a.vdim;
    if (rc == AB2_OK) rc = make_mats_map(&kmap, a.k, mats, L, kcols, a.k_stride, a.k_z ? a.k_z : L * a.k_stride, PT_KEYS);
    if (rc == AB2_OK) rc = a.tail_dims > 0 ? make_x_map(&tmap, a.tail, L, a.tail_dims, PT_KEYS, a.tail_stride) : make_x_map(&tmap, a.k, L, a.dim, PT_KEYS, a.k_stride);
    if (rc == AB2_OK) rc = make_mats_map(&vmap, a.v, mats, L, vcols, a.v_stride, a.k_z ? a.v_z : L * a.v_stride, PT_KEYS);
    if (rc != AB2_OK) return rc;
    return a.k_scale ? launch_prompt<true>(p, kmap, tmap, vmap, status, s) : launch_prompt<false>(p, kmap, tmap, vmap, status, s);
}

int prompt_tc_cached(const ab2_kv *kv, int layer, const void *q, void *out, int S, int pending, int row0, int nrows, float scale,
                     ab2_dtype dtype, const AttnStrides &st, cudaStream_t s) {
    const int hd = kv->hd;
    const bool int8 = kv->dtype == AB2_KV_INT8;
    if (hd != 64 && hd != 128) return AB2_ERR_UNSUPPORTED;  // as for decode and fewer queries over such a cache: refused
    if (S < PT_MIN_QUERIES || dtype != AB2_BF16 || kv->dtype == AB2_KV_F32 || st.q_h != hd || st.o_h != hd || !lengths_known(s)) return AB2_ERR_UNSUPPORTED;
    int longest = 0;
    for (int i = 0; i < nrows; ++i) {
        const int L = kv->lens_host[kv_row_host(kv, row0, i)] + pending;
        if (L < S) return AB2_ERR_UNSUPPORTED;
        longest = std::max(longest, L);
    }
    const KvView v = kv_view(kv, layer);
    PromptAttnArgs p = {};
    p.q = (const __nv_bfloat16 *)q; p.out = (__nv_bfloat16 *)out;
    p.q_stride = st.q_s; p.out_stride = st.o_s; p.q_row = st.q_b; p.out_row = st.o_b;
    p.S = S; p.heads = kv->h; p.rep = kv->h / kv->kvh; p.dim = p.vdim = hd; p.scale = scale;
    p.nrows = nrows; p.row0 = row0; p.mats = kv->B * kv->kvh;
    p.k_stride = p.v_stride = hd;
    p.k_z = p.v_z = (long long)kv->cap * hd;
    // one sequence: its row and length are known here, so the kernel need not fetch them, and what lies past its keys reads as zeros
    if (nrows == 1) { p.row0 = kv_row_host(kv, row0, 0); p.first = longest - S; p.key_rows = longest; }
    else { p.lens = v.lens; p.rows = v.rows; p.pending = pending; p.key_rows = kv->cap; }
    if (!int8) { p.k = (const __nv_bfloat16 *)v.k; p.v = (const __nv_bfloat16 *)v.v; }
    if (!prompt_tc_serves(p)) return AB2_ERR_UNSUPPORTED;
    const double gathered = int8 ? 6.0 * nrows * kv->kvh * longest * hd : 0;  // codes read, bf16 written and read again
    if (!prompt_tc_pays(prompt_tc_us(p, longest - S, int8, gathered), cache_other_us(p, longest - S, int8))) return AB2_ERR_UNSUPPORTED;
    if (!int8) return prompt_tc_attention(p, s);
    p.k_scale = v.ks; p.v_scale = v.vs; p.scale_z = kv->cap;
    PtGather g = {};
    g.src[0] = v.k; g.src[1] = v.v;
    g.ld[0] = g.ld[1] = hd; g.src_z[0] = g.src_z[1] = p.k_z;
    g.n = longest; g.cap = kv->cap;
    return attention_gathered(g, p, true, kv->kvh, s);
}

int prompt_tc_window(const ab2_kv *kv, const WindowAttnArgs &a, int nrows, cudaStream_t s) {
    const KvLayer &l = a.kv.l;
    if (a.S < PT_MIN_QUERIES || !lengths_known(s)) return AB2_ERR_UNSUPPORTED;
    PromptAttnArgs p = {};
    int most = 0, longest = 0;  // keys in sight of a sequence, tokens before its queries
    bool wraps = false;
    for (int i = 0; i < nrows; ++i) {
        const int first = kv->lens_host[kv_row_host(kv, a.row0, i)], base = std::max(0, first - l.window + 1), n = first + a.S - base;
        if (l.window < first + a.S) p.window = l.window;
        most = std::max(most, n);
        longest = std::max(longest, first);
        wraps |= base % l.cap + n > l.cap;
    }
    p.q = (const __nv_bfloat16 *)a.q; p.q_stride = a.q_stride; p.q_row = a.S * a.q_stride;
    p.out = (__nv_bfloat16 *)a.out; p.out_stride = (long long)a.H * a.vdim; p.out_row = a.S * p.out_stride;
    p.S = a.S; p.heads = a.H; p.rep = a.rep; p.dim = a.dim; p.vdim = a.vdim; p.scale = a.scale;
    p.nrows = nrows; p.row0 = a.row0; p.mats = kv->B * l.kvh;
    p.k = (const __nv_bfloat16 *)l.k; p.v = (const __nv_bfloat16 *)l.v;
    p.k_stride = l.kds; p.v_stride = l.vds; p.k_z = (long long)l.cap * l.kds; p.v_z = (long long)l.cap * l.vds;
    p.key_rows = p.ring = l.cap;
    if (nrows == 1) { p.row0 = kv_row_host(kv, a.row0, 0); p.first = kv->lens_host[p.row0]; }
    else { p.lens = a.kv.lens; p.rows = a.kv.rows; }
    p.pending = a.S;
    if (!prompt_tc_serves(p)) return AB2_ERR_UNSUPPORTED;
    const double gathered = wraps ? 4.0 * nrows * l.kvh * most * (l.kds + l.vds) : 0;  // read, written; read again from L2
    if (!prompt_tc_pays(prompt_tc_us(p, longest, false, gathered), window_mma_us(p, longest))) return AB2_ERR_UNSUPPORTED;
    if (!wraps) return prompt_tc_attention(p, s);
    PtGather g = {};
    g.src[0] = l.k; g.src[1] = l.v;
    g.ld[0] = l.kds; g.ld[1] = l.vds; g.src_z[0] = p.k_z; g.src_z[1] = p.v_z;
    g.n = most; g.cap = l.cap;
    return attention_gathered(g, p, false, l.kvh, s);
}

}  // namespace ab2
