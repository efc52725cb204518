// W4A16 (group 128, bf16) decode GEMM for a few tokens (up to 64) on the 5th-generation
// tensor cores, built so that the packed weights cross HBM once and cost two and a
// quarter instructions per pair of codes whatever the token count.
//
//   Y[M, N] = X[M, K] . W^T,  W packed 4-bit in tile-major blocks (w4a16_layout.cuh)
//
// The 128 output channels of a channel tile are the M dimension of the MMA, the
// tokens (padded to NTOK) its N dimension.  Operand A is the integer q - zero over 128
// in bf16, not the dequantised weight.  A pair of codes masked out of its word is a
// pair of bf16 subnormals q 2^-133 (or, four bits higher, q 2^-129), so that one
// packed fma gives q / 128 - zero / 128, exactly: every value is an integer below 16
// times 2^-7.  Masks of two positions share a shift (a magic number in the place of the
// subnormals needs every code in the low bits, a shift for each pair but one).
// The unpack warps write the pairs to an operand stage in tensor memory.  The scale is
// applied per quantisation group in f32 by the epilogue warps: after the MMAs of a group
//   d[c][t] = sum_k x[t][k] (q[c][k] - zero[c]) / 128        (tensor memory)
// and the group adds scale[c] * d[c][t] to the running f32 output kept in the
// epilogue threads' registers (thread = channel); 128 comes in at the end.  Several
// accumulators rotate in tensor memory, so the epilogue of a group overlaps the MMAs
// of the next ones.
//
// Work is the sequence of (channel tile, group) units in tile-major order, cut
// into one contiguous range per CTA (one CTA per SM), so small weights are split
// over K.  A channel tile cut by a range boundary is finished by the CTA that
// arrives last: partial sums go to a global scratch slot per contributor, a
// counter per tile tells who is last, and the slots are added in contributor
// order.  One CTA per SM, warp-specialised; a stage holds one unit:
//   8 warps    unpack, two sets of four warps, a set takes every other unit; thread = channel
//   8 warps    epilogue, two groups of four warps, for every other unit or for the halves of 64 tokens:
//              tcgen05.ld of D, scale, running sums, the tile's final store (or partial + hand-over)
//   2 warps    tcgen05.mma issue and commits on alternate units
//   1 warp     packed weights: one tensor-map copy a unit
//   1 warp     activations: two 64-wide halves a unit, 128-byte swizzle
//
// What bounds it: the instructions of the unpack and epilogue warps (about 330 issue slots of each scheduler a unit, of
// which a unit takes 0.33 us; HBM would allow 0.2) and the serial chains through the barriers.  So every role waits at as
// few barriers a unit as can be: `full` of a stage collects the unpack warps' arrivals, the activations' bytes and the
// epilogue's word that the unit's accumulator is free again, and one commit (`done`) tells the unpack warps, the
// activations' producer and the epilogue.  Packed weights land with a 64-byte swizzle, so that 32 rows' 16-byte loads meet
// no bank twice.  4096 x 28672, 32 tokens: 42 us before (warp-level MMAs), 29 with one epilogue group and divisions in its
// loop, 25.5 with two groups and counted rings, 24.4 with subnormals.  Stages of two units (fewer waits, less in flight)
// took 31.7, four sets of unpack warps over four stages 28.
// Every wait on an mbarrier is bounded; on a time-out the CTA records
// AB2_ERR_TIMEOUT, walks through the rest of its work, frees its tensor memory and returns.
#include <algorithm>

#include "common.cuh"
#include "gemv_w4a16_mma.cuh"
#include "ops.cuh"
#include "tcgen05_util.cuh"

using namespace ab2;
using namespace ab2::tc;

namespace ab2 {
int device_status_word(int **out);
int device_sm_count();
namespace {

constexpr int DG_SLOT_BYTES = 8 * W4_BLOCK_WORDS * 4;  // eight 16-channel blocks of a unit: a multiple of the swizzle's 512 bytes
constexpr int DG_A_COLS = 64;     // tensor-memory columns of 128 K-elements: two bf16 per column, a lane per channel
constexpr int DG_WSLOTS = 12;     // depth of the packed-weight ring in units: ~100 KB in flight per SM
constexpr int DG_MMA_WARPS = 2;
constexpr int DG_PARAM_BUFS = 12;
static_assert(DG_SLOT_BYTES % 512 == 0, "a slot starts on the swizzle's period");

// A place in a ring of N, `by` places on at a time, with the parity of its lap; counted, since a division a unit shows in the chains.
template <int N>
struct DgRing {
    uint32_t at, lap = 0;
    __device__ __forceinline__ void next(uint32_t by) {
        at += by;
        if (at >= N) { at -= N; lap ^= 1; }
    }
};

template <int NTOK>
struct DgShape {
    static constexpr int SETS = 2;                                // sets of four unpack warps
    static constexpr int STAGES = NTOK > 32 ? 4 : 6;              // operand stages of one unit (64 columns of tensor memory, NTOK x 256 bytes of activations)
    static constexpr int ACC = 4;                                 // accumulators in tensor memory
    static constexpr int HALVES = NTOK > 32 ? 2 : 1;              // the epilogue's groups of four warps: two, for the halves of 64 tokens ...
    static constexpr int ALT = NTOK > 32 ? 1 : 2;                 // ... or for every other unit
    static constexpr int TOK = NTOK / HALVES;                     // tokens of an epilogue thread while it sums ...
    static constexpr int FIN = TOK / ALT;                         // ... and when it stores
    static constexpr int FIRST_EPI = 4 * SETS, FIRST_MMA = FIRST_EPI + 8, WARP_W = FIRST_MMA + DG_MMA_WARPS, WARP_X = WARP_W + 1;
    static constexpr int THREADS = 32 * (WARP_X + 1);
    static constexpr int X_BYTES = NTOK * 256, OUT_BYTES = 8 * FIN * 32 * 2, SWAP_BYTES = ALT > 1 ? NTOK * 128 * 4 : 0;
    // A parity wait cannot tell phase k from phase k + 2, so a warp must see every phase of the barriers it waits on: the stages
    // and slots that a unit uses must come back to the same warp, accumulators to the same epilogue warps.
    static_assert(STAGES % DG_MMA_WARPS == 0 && STAGES % SETS == 0 && DG_WSLOTS % SETS == 0 && STAGES % ALT == 0 && ACC % ALT == 0, "ring depths must be multiples of the warps' strides");
    static_assert(ACC <= STAGES && STAGES + ACC <= DG_PARAM_BUFS, "an accumulator's last unit is done with when its stage is filled; a parameter buffer's reader too");
    static_assert(ACC * NTOK + STAGES * DG_A_COLS <= 512, "accumulators and operand stages fit");
};

template <int NTOK>
struct DgShared {
    using S = DgShape<NTOK>;
    uint64_t wfull[DG_WSLOTS], wempty[DG_WSLOTS], full[S::STAGES], done[S::STAGES];
    uint32_t params[DG_PARAM_BUFS][128];  // scale | -(128 + zero) of a unit's 128 channels
    uint32_t tmem_base;
    int failed;
    int last_flag;
};

// Units [u0, u1) of a CTA.  parts > 0: that many CTAs for every channel tile, each a share of its groups.  Otherwise equal shares of all units.
struct DgRange {
    int total, ctas, G, parts;
    __device__ __forceinline__ int start(int cta) const {
        if (parts) return cta / parts * G + cta % parts * G / parts;
        const int base = total / ctas;
        return cta * base + min(cta, total - base * ctas);
    }
    __device__ __forceinline__ int owner(int u) const {  // whose range holds unit u, the first or last of a tile
        if (parts) return u / G * parts + (u % G ? parts - 1 : 0);
        const int base = total / ctas, rem = total - base * ctas, cut = rem * (base + 1);
        return u < cut ? u / (base + 1) : rem + (u - cut) / base;
    }
};

__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a)) | ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(b)) << 16);
}
__device__ __forceinline__ uint32_t bf16_pair_sum(uint32_t a, uint32_t b) {  // each half added in f32 and rounded
    return bf16_pair(__uint_as_float(a << 16) + __uint_as_float(b << 16), __uint_as_float(a & 0xffff0000u) + __uint_as_float(b & 0xffff0000u));
}

// What the warps that finish a channel tile store: TOK tokens from t0 on of the 32 channels from n0 on (lane = channel).
// Rows that lie on 16 bytes go out through `stage` in pieces of 16 bytes: 32 tokens stored straight from the lanes are 32
// instructions of 64 bytes and 1.7 us at the end of the launch.
template <int TOK, int EPI>
__device__ __forceinline__ void dg_store(const float (&acc)[TOK], __nv_bfloat16 *stage, __nv_bfloat16 *y, const __nv_bfloat16 *resid, int n0,
                                         int t0, int N, int M, bool aligned, int lane) {
    const int n = n0 + lane;
    if (EPI == W4_EPI_SWIGLU) {
        // channels come in 16s: 8 gate rows, then the 8 matching up rows (8 lanes further)
        const int half_n = N >> 1, col0 = n0 >> 1;  // 16 columns of the warp
#pragma unroll
        for (int j = 0; j < TOK; ++j) {
            const float g = __bfloat162float(__float2bfloat16_rn(acc[j]));
            const float u = __bfloat162float(__float2bfloat16_rn(__shfl_xor_sync(0xffffffffu, acc[j], 8)));
            const __nv_bfloat16 v = __float2bfloat16_rn(swiglu_value(g, u));
            const int c = (lane >> 4) * 8 + (lane & 7);
            if (lane & 8) continue;
            if (aligned) stage[j * 16 + c] = v;
            else if (t0 + j < M && col0 + c < half_n) y[(size_t)(t0 + j) * half_n + col0 + c] = v;
        }
        if (aligned) {
            __syncwarp();
#pragma unroll
            for (int i = lane; i < TOK * 2; i += 32) {
                const int j = i >> 1, c = (i & 1) * 8;
                if (t0 + j < M && col0 + c < half_n)
                    *reinterpret_cast<uint4 *>(y + (size_t)(t0 + j) * half_n + col0 + c) = *reinterpret_cast<const uint4 *>(stage + j * 16 + c);
            }
            __syncwarp();
        }
    } else if (EPI == W4_EPI_F32 || !aligned) {
#pragma unroll
        for (int j = 0; j < TOK; ++j) {
            if (t0 + j >= M || n >= N) continue;
            const size_t o = (size_t)(t0 + j) * N + n;
            float v = acc[j];
            if (EPI == W4_EPI_F32) {
                reinterpret_cast<float *>(y)[o] = v;
            } else {
                // the residual may alias the output: a thread reads and writes the same elements
                if (EPI == W4_EPI_ADD) v = __bfloat162float(resid[o]) + __bfloat162float(__float2bfloat16_rn(v));
                y[o] = __float2bfloat16_rn(v);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < TOK; ++j) stage[j * 32 + lane] = __float2bfloat16_rn(acc[j]);
        __syncwarp();
        const int c = (lane & 3) * 8;
#pragma unroll
        for (int j = lane >> 2; j < TOK; j += 8) {
            uint4 q = *reinterpret_cast<const uint4 *>(stage + j * 32 + c);
            if (t0 + j >= M || n0 + c >= N) continue;
            const size_t o = (size_t)(t0 + j) * N + n0 + c;
            if (EPI == W4_EPI_ADD) {
                const uint4 r = *reinterpret_cast<const uint4 *>(resid + o);
                q = make_uint4(bf16_pair_sum(r.x, q.x), bf16_pair_sum(r.y, q.y), bf16_pair_sum(r.z, q.z), bf16_pair_sum(r.w, q.w));
            }
            *reinterpret_cast<uint4 *>(y + o) = q;
        }
        __syncwarp();
    }
}

// partials: [gridDim.x][2][NTOK][128] f32; counters: one int per channel tile, zero on entry and exit.
template <int NTOK, int EPI>
__global__ void __launch_bounds__(DgShape<NTOK>::THREADS, 1)
gemv_w4a16_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                     __nv_bfloat16 *y, const __nv_bfloat16 *resid, int N, int K, int M, int parts, bool aligned, float *partials,
                     int *counters, int *status) {
    using S = DgShape<NTOK>;
    constexpr int HALF_BYTES = NTOK * 128;
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NTOK >> 3) << 17) | ((128u >> 4) << 24);
    constexpr uint32_t ACC_COLS = S::ACC * NTOK, TMEM_COLS = 512;
    static_assert(NTOK <= W4DG_MAX_TOKENS, "the caller's scratch holds two partial tiles per CTA");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *x_st = smem;                                    // [STAGES][X_BYTES]
    uint8_t *w_ring = x_st + S::STAGES * S::X_BYTES;         // [DG_WSLOTS][DG_SLOT_BYTES]
    __nv_bfloat16 *out = (__nv_bfloat16 *)(w_ring + DG_WSLOTS * DG_SLOT_BYTES);
    float4 *swap = (float4 *)((uint8_t *)out + S::OUT_BYTES);  // [NTOK / 4][128 channels]: what the epilogue's groups hand each other
    DgShared<NTOK> *sh = (DgShared<NTOK> *)((uint8_t *)swap + S::SWAP_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = K >> 7, n_tiles = (N + 127) >> 7;
    const DgRange rg = {n_tiles * G, (int)gridDim.x, G, parts};
    const int u0 = rg.start((int)blockIdx.x), units = rg.start((int)blockIdx.x + 1) - u0;
    volatile int *failed = &sh->failed;

    if (threadIdx.x == 0) {
        for (int i = 0; i < DG_WSLOTS; ++i) { bar_init(&sh->wfull[i], 1); bar_init(&sh->wempty[i], 4); }
        // a stage is full with its unit's weights (4 warps), activations (1) and free accumulator
        for (int i = 0; i < S::STAGES; ++i) { bar_init(&sh->full[i], 4 + 1 + 4 * S::HALVES); bar_init(&sh->done[i], 1); }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == S::FIRST_MMA) {  // tensor-memory allocation is a whole-warp operation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(sptr(&sh->tmem_base)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = sh->tmem_base, tmem_a = tmem + ACC_COLS;
    pdl_launch_dependents();  // the next kernel may start fetching its constant weights

    if (warp < S::FIRST_EPI) {
        // ---------------------------------------------------------- unpack: codes -> bf16 q - zero
        const int quad = warp & 3, set = warp >> 2;
        const int t = quad * 32 + lane;               // channel within the 128-channel tile
        const int line = (t >> 4) * 17 + (t & 15);    // 64-byte line of the slot that holds its codes; a block's 17th line is its parameters
        const uint32_t code_at = (uint32_t)line * 64, code_sw = (uint32_t)(line >> 1) & 3;
        const int pline = (t >> 4) * 17 + 16;
        const uint32_t param_at = (uint32_t)pline * 64 + ((((uint32_t)(t & 15) >> 2) ^ ((uint32_t)(pline >> 1) & 3)) << 4) + (t & 3) * 4;
        // opaque, so that the constants stay in registers
        uint32_t mask_lo = 0x000F000Fu, mask_hi = 0x00F000F0u, up_lo = 0x7E807E80u, up_hi = 0x7C807C80u;  // 2^126, 2^122
        asm volatile("" : "+r"(mask_lo), "+r"(mask_hi), "+r"(up_lo), "+r"(up_hi));
        const uint32_t tmem_w = tmem_a + ((uint32_t)(quad * 32) << 16);
        DgRing<DG_WSLOTS> ws = {(uint32_t)set};
        DgRing<S::STAGES> st = {(uint32_t)set};
        DgRing<DG_PARAM_BUFS> pb = {(uint32_t)set};
        for (int use = set; use < units; use += S::SETS, ws.next(S::SETS), st.next(S::SETS), pb.next(S::SETS)) {
            const uint8_t *slot = w_ring + ws.at * DG_SLOT_BYTES;
            bar_wait(&sh->wfull[ws.at], ws.lap, failed);
            uint4 p[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const uint4 *>(slot + code_at + ((i ^ code_sw) << 4));
            const uint32_t pr = *reinterpret_cast<const uint32_t *>(slot + param_at);
            const bool free = bar_wait(&sh->done[st.at], st.lap ^ 1, failed);
            __syncwarp();  // the tensor-memory stores are whole-warp operations
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            sh->params[pb.at][t] = pr;
            const uint32_t nz2 = bf16x2_fma(__byte_perm(pr, pr, 0x3232), 0x3C003C00u, 0x3F803F80u);  // 1 - (128 + zero) / 128 = -zero / 128
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t words[8] = {p[2 * h].x, p[2 * h].y, p[2 * h].z, p[2 * h].w, p[2 * h + 1].x, p[2 * h + 1].y, p[2 * h + 1].z, p[2 * h + 1].w};
                uint32_t o[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {  // 8 consecutive k = one code word
                    const uint32_t w0 = words[c], w8 = words[c] >> 8;
                    o[4 * c] = bf16x2_fma(w0 & mask_lo, up_lo, nz2);
                    o[4 * c + 1] = bf16x2_fma(w0 & mask_hi, up_hi, nz2);
                    o[4 * c + 2] = bf16x2_fma(w8 & mask_lo, up_lo, nz2);
                    o[4 * c + 3] = bf16x2_fma(w8 & mask_hi, up_hi, nz2);
                }
                tmem_st32(tmem_w + st.at * DG_A_COLS + h * 32, o);
            }
            // the stores took in every lane's loads of the slot: it can be filled again
            if (lane == 0 && free) bar_arrive(&sh->wempty[ws.at]);
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0 && free) bar_arrive(&sh->full[st.at]);
        }
    } else if (warp < S::FIRST_MMA) {
        // ---------------------------------------------------------- epilogue
        const int quad = warp & 3, grp = (warp - S::FIRST_EPI) >> 2;  // lanes of tensor memory, group
        const int row = quad * 32 + lane;                    // channel within the tile
        const int t_sum = S::HALVES > 1 ? grp * S::TOK : 0;  // first of the tokens that the thread sums, and of those that it stores
        const int t_fin = grp * S::FIN;
        __nv_bfloat16 *stage = out + (warp - S::FIRST_EPI) * S::FIN * 32;
        float acc[S::TOK];
#pragma unroll
        for (int j = 0; j < S::TOK; ++j) acc[j] = 0.f;
        if (lane == 0)
            for (int use = 0; use < S::ACC && use < units; ++use)
                if (use % S::ALT == grp % S::ALT) bar_arrive(&sh->full[use]);  // every accumulator is free
        // that these warps do not leave after a time-out also brings the counters of cut tiles back to zero
        const uint32_t tmem_d = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)t_sum;
        int use = S::ALT > 1 ? grp : 0;
        DgRing<S::STAGES> st = {(uint32_t)use};
        DgRing<S::ACC> ab = {(uint32_t)use};
        DgRing<DG_PARAM_BUFS> pb = {(uint32_t)use};
        int nt = u0 / G, g0 = u0 - nt * G;  // first of the tile's groups here
        for (int first = 0, end; first < units; first = end, ++nt, g0 = 0) {
            end = min(units, first + G - g0);
            for (; use < end; use += S::ALT, st.next(S::ALT), ab.next(S::ALT), pb.next(S::ALT)) {
                const bool ready = bar_wait(&sh->done[st.at], st.lap, failed);
                __syncwarp();  // the tensor-memory load is a whole-warp operation
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const float sc = __uint_as_float(sh->params[pb.at][row] << 16);
                constexpr int COLS = S::TOK < 32 ? 16 : 32;
                uint32_t d[COLS];
                if constexpr (COLS == 16) tmem_ld16(d, tmem_d + ab.at * NTOK);
                else tmem_ld32(d, tmem_d + ab.at * NTOK);
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                const uint32_t later = st.at + S::ACC;  // the stage of the unit that takes the accumulator next
                if (lane == 0 && ready && use + S::ACC < units) bar_arrive(&sh->full[later >= S::STAGES ? later - S::STAGES : later]);
#pragma unroll
                for (int j = 0; j < COLS; ++j) acc[j] = fmaf(sc, __uint_as_float(d[j]), acc[j]);
            }

            // ---- end of this CTA's share of channel tile nt
            float fin[S::FIN];
            if constexpr (S::ALT > 1) {  // even units' and odd units' sums: each group adds and stores half of the tokens
#pragma unroll
                for (int j = 0; j < S::FIN; j += 4) {
                    const int o = grp ? j : j + S::FIN;  // the other group's tokens
                    float4 v;
#pragma unroll
                    for (int q = 0; q < S::TOK; q += 4) if (q == o) v = make_float4(acc[q], acc[q + 1], acc[q + 2], acc[q + 3]);
                    swap[(o >> 2) * 128 + row] = v;
                }
                asm volatile("bar.sync 1, 256;\n" ::: "memory");
#pragma unroll
                for (int j = 0; j < S::FIN; j += 4) {
                    const float4 v = swap[((t_fin + j) >> 2) * 128 + row];
                    fin[j] = 128.f * (v.x + (grp ? acc[S::FIN + j] : acc[j]));
                    fin[j + 1] = 128.f * (v.y + (grp ? acc[S::FIN + j + 1] : acc[j + 1]));
                    fin[j + 2] = 128.f * (v.z + (grp ? acc[S::FIN + j + 2] : acc[j + 2]));
                    fin[j + 3] = 128.f * (v.w + (grp ? acc[S::FIN + j + 3] : acc[j + 3]));
                }
            } else {
#pragma unroll
                for (int j = 0; j < S::FIN; ++j) fin[j] = 128.f * acc[j];
            }
            bool finish = end - first == G;  // the whole tile is this CTA's
            if (!finish) {
                const int c_first = rg.owner(nt * G), c_last = rg.owner(nt * G + G - 1);
                const int which = (int)blockIdx.x == c_first ? 1 : 0;  // slot 1: the tile my range ends inside
                float4 *mine = reinterpret_cast<float4 *>(partials) + ((size_t)blockIdx.x * 2 + which) * (NTOK * 32) + (t_fin >> 2) * 128 + row;
#pragma unroll
                for (int j = 0; j < S::FIN; j += 4) __stcg(mine + j * 32, make_float4(fin[j], fin[j + 1], fin[j + 2], fin[j + 3]));
                __threadfence();
                asm volatile("bar.sync 1, 256;\n" ::: "memory");
                if (threadIdx.x == 32 * S::FIRST_EPI) sh->last_flag = atomicAdd(&counters[nt], 1) == c_last - c_first;
                asm volatile("bar.sync 1, 256;\n" ::: "memory");
                finish = sh->last_flag != 0;
                if (finish) {
                    __threadfence();
#pragma unroll
                    for (int j = 0; j < S::FIN; ++j) fin[j] = 0.f;
                    // in the order of the contributors; the loads of several are under way together
                    constexpr int TOGETHER = S::FIN > 16 ? 1 : S::FIN > 8 ? 2 : 4;
                    for (int c0 = c_first; c0 <= c_last; c0 += TOGETHER) {
                        float4 v[TOGETHER][S::FIN / 4];
#pragma unroll
                        for (int i = 0; i < TOGETHER; ++i) {
                            const int c = min(c0 + i, c_last);
                            const float4 *p = reinterpret_cast<const float4 *>(partials) + ((size_t)c * 2 + (c == c_first ? 1 : 0)) * (NTOK * 32) + (t_fin >> 2) * 128 + row;
#pragma unroll
                            for (int j = 0; j < S::FIN / 4; ++j) v[i][j] = __ldcg(p + j * 128);
                        }
#pragma unroll
                        for (int i = 0; i < TOGETHER; ++i) {
                            if (c0 + i > c_last) break;
#pragma unroll
                            for (int j = 0; j < S::FIN / 4; ++j) {
                                fin[4 * j] += v[i][j].x; fin[4 * j + 1] += v[i][j].y; fin[4 * j + 2] += v[i][j].z; fin[4 * j + 3] += v[i][j].w;
                            }
                        }
                    }
                    if (threadIdx.x == 32 * S::FIRST_EPI) counters[nt] = 0;
                }
            }
            if (finish) dg_store<S::FIN, EPI>(fin, stage, y, resid, nt * 128 + quad * 32, t_fin, N, M, aligned, lane);
            asm volatile("bar.sync 1, 256;\n" ::: "memory");  // the next tile's end writes `swap` and last_flag anew
#pragma unroll
            for (int j = 0; j < S::TOK; ++j) acc[j] = 0.f;
        }
    } else if (warp < S::WARP_W) {
        // ---------------------------------------------------------- MMA issue (alternate units per warp)
        const uint64_t xd0 = umma_desc(sptr(x_st));
        DgRing<S::STAGES> st = {(uint32_t)(warp - S::FIRST_MMA)};
        DgRing<S::ACC> ab = {(uint32_t)(warp - S::FIRST_MMA)};
        for (int use = warp - S::FIRST_MMA; use < units; use += DG_MMA_WARPS, st.next(DG_MMA_WARPS), ab.next(DG_MMA_WARPS)) {
            bar_wait(&sh->full[st.at], st.lap, failed);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (elect_one()) {
                const uint32_t td = tmem + ab.at * NTOK, ta = tmem_a + st.at * DG_A_COLS;
                const uint64_t xd = xd0 + (uint64_t)(st.at * (S::X_BYTES >> 4));
                umma_stage_ts(td, ta, xd, IDESC, true);
                umma_stage_ts(td, ta + 32, xd + (HALF_BYTES >> 4), IDESC, false);
                umma_commit(&sh->done[st.at]);
            }
            __syncwarp();
        }
    } else if (warp == S::WARP_W) {
        // ---------------------------------------------------------- producer of the packed weights
        if (lane == 0) {
            int nt = u0 / G, g = u0 - nt * G;
            for (int use = 0; use < units && !*failed; ++use, ++g) {
                const int ws = use % DG_WSLOTS;
                if (g == G) { g = 0; ++nt; }
                if (!bar_wait(&sh->wempty[ws], ((use / DG_WSLOTS) & 1) ^ 1, failed)) break;
                bar_expect_tx(&sh->wfull[ws], DG_SLOT_BYTES);  // blocks past the last tile are filled with zeros
                tma_load_4d(w_ring + ws * DG_SLOT_BYTES, &wmap, 0, 0, g, nt * 8, &sh->wfull[ws]);
            }
        }
    } else {
        // ---------------------------------------------------------- producer of the activation tiles
        if (lane == 0) {
            pdl_wait();  // the activations come from the preceding kernel
            int g = u0 % G;
            for (int use = 0; use < units && !*failed; ++use, ++g) {
                const int s = use % S::STAGES;
                if (g == G) g = 0;
                if (!bar_wait(&sh->done[s], ((use / S::STAGES) & 1) ^ 1, failed)) break;
                bar_expect_tx(&sh->full[s], S::X_BYTES);
                tma_load_2d(x_st + s * S::X_BYTES, &xmap, g * 128, 0, &sh->full[s]);
                tma_load_2d(x_st + s * S::X_BYTES + HALF_BYTES, &xmap, g * 128 + 64, 0, &sh->full[s]);
            }
        }
    }

    // ---- teardown: every warp arrives here (all waits are bounded)
    if (!(warp == S::WARP_X && lane == 0)) pdl_wait();  // every thread passes the wait before the grid counts as finished
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && sh->failed) atomicExch(status, (int)AB2_ERR_TIMEOUT);
    if (warp == S::FIRST_MMA) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// Tensor map of a weight's blocks as [16-channel tile][group][17 lines][64 bytes], read a unit (8 tiles of one group) at a time.
int make_w4_map(CUtensorMap *map, const ab2_qweight *w) {
    EncodeTiledFn encode;
    int rc = tensor_map_encoder(&encode);
    if (rc != AB2_OK) return rc;
    const cuuint64_t G = w->K / 128, block = W4_BLOCK_WORDS * 4;
    cuuint64_t dims[4] = {16, 17, G, (cuuint64_t)(w->N + 15) / 16};
    cuuint64_t strides[3] = {64, block, block * G};
    cuuint32_t box[4] = {16, 17, 1, 8};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, w->codes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    AB2_REQUIRE(r == CUDA_SUCCESS, AB2_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    return AB2_OK;
}

template <int NTOK>
constexpr size_t dg_smem_bytes() {
    using S = DgShape<NTOK>;
    return 1024 + S::STAGES * S::X_BYTES + DG_WSLOTS * DG_SLOT_BYTES + S::OUT_BYTES + S::SWAP_BYTES + sizeof(DgShared<NTOK>);
}

template <int NTOK, int EPI>
int launch_dg(const ab2_qweight *w, const void *x, int M, void *y, const void *resid, float *partials, int *counters,
              int max_ctas, cudaStream_t s) {
    int *status = nullptr;
    int rc = device_status_word(&status);
    if (rc != AB2_OK) return rc;
    CUtensorMap map, wmap;
    rc = make_x_map(&map, x, M, w->K, NTOK);
    if (rc == AB2_OK) rc = make_w4_map(&wmap, w);
    if (rc != AB2_OK) return rc;
    const size_t smem = dg_smem_bytes<NTOK>();
    static_assert(dg_smem_bytes<NTOK>() <= 227 * 1024, "shared memory of a CTA");
    static bool configured[64] = {false};  // the attribute is per device
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    if (!configured[dev]) {
        AB2_CUDA(cudaFuncSetAttribute(gemv_w4a16_tc_kernel<NTOK, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured[dev] = true;
    }
    // Equal shares of the units, or the same number of CTAs for every channel tile.  The latter's ranges are longer where the
    // tiles do not fill the SMs (a unit takes about 0.34 us), but a tile is finished by fewer CTAs, of its own if there is one,
    // and no CTA works on two cut tiles (32 tokens: 4096 x 4096 13.6 -> 11.0 us, 6144 x 4096 14.5 -> 12.2, 14336 x 4096 17.4 ->
    // 14.7 with 8 units more).
    const int G = w->K / 128, tiles = (w->N + 127) / 128, units = tiles * G, sms = std::min(max_ctas, device_sm_count());
    int grid = std::max(1, std::min(sms, units / 2)), parts = 0;
    if (tiles <= sms) {
        const int p = std::max(1, std::min(sms / tiles, G / 2));
        if ((G + p - 1) / p <= (units + grid - 1) / grid + 12) { parts = p; grid = tiles * p; }
    }
    const bool aligned = rows_in_16_bytes(y, EPI == W4_EPI_SWIGLU ? w->N / 2 : w->N) && (EPI != W4_EPI_ADD || ((uintptr_t)resid & 15) == 0);
    cudaError_t e = launch_kernel(gemv_w4a16_tc_kernel<NTOK, EPI>, dim3(grid), dim3(DgShape<NTOK>::THREADS), smem, s, wmap, map,
                                  (__nv_bfloat16 *)y, (const __nv_bfloat16 *)resid, w->N, w->K, M, parts, aligned, partials, counters, status);
    if (e != cudaSuccess) return fail(AB2_ERR_CUDA, "decode GEMM launch failed: %s", cudaGetErrorString(e));
    return AB2_OK;
}

}  // namespace

// Y = epilogue(X[M][K] . W^T) for 2..64 tokens; partials / counters are the caller's
// scratch (zeroed counters, one per 128-channel tile; two slots of W4DG_MAX_SLOT_FLOATS for every SM).
int qlinear_w4a16_tc_decode(const ab2_qweight *w, const void *x, int M, void *y, const void *resid, int epi,
                            float *partials, int *counters, int max_ctas, cudaStream_t s) {
    AB2_REQUIRE(M >= 1 && M <= W4DG_MAX_TOKENS, AB2_ERR_BAD_SHAPE, "the decode GEMM serves 1..%d tokens, got %d", W4DG_MAX_TOKENS, M);
    AB2_REQUIRE(((uintptr_t)x & 15) == 0 && (w->K * 2) % 16 == 0, AB2_ERR_BAD_ALIGN, "activations must be 16-byte aligned");
#define AB2_DG(NT)                                                                                              \
    switch (epi) {                                                                                              \
    case W4_EPI_STORE: return launch_dg<NT, W4_EPI_STORE>(w, x, M, y, resid, partials, counters, max_ctas, s);   \
    case W4_EPI_ADD: return launch_dg<NT, W4_EPI_ADD>(w, x, M, y, resid, partials, counters, max_ctas, s);       \
    case W4_EPI_SWIGLU: return launch_dg<NT, W4_EPI_SWIGLU>(w, x, M, y, resid, partials, counters, max_ctas, s); \
    case W4_EPI_F32: return launch_dg<NT, W4_EPI_F32>(w, x, M, y, resid, partials, counters, max_ctas, s);       \
    default: return fail(AB2_ERR_BAD_ARG, "unsupported epilogue %d", epi);                                       \
    }
    if (M <= 16) { AB2_DG(16) }
    if (M <= 32) { AB2_DG(32) }
    AB2_DG(64)
#undef AB2_DG
}

}  // namespace ab2
