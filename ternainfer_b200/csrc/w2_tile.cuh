// Medium batches on two-bit weights for sm_100a: tcgen05 int8 GEMM on single CTAs, weights expanded into tensor memory.
//
// A CTA owns 128 weight rows x NT tokens (a multiple of 16, at most 128) and one of S slices of K, the S CTAs of a tile forming a
// cluster.  The weight operand of tcgen05.mma may come from tensor memory: a decoder lane has one weight row, reads its
// 32 bytes of codes per 128 k from shared memory, expands them and writes 32 columns with two tcgen05.st.  Against expanding
// into shared memory (w2_pair.cuh before) that leaves the shared-memory port to the activations, and a launch needs
// half of an SM's tensor memory, shared memory and registers.  So the CTAs of the next launch run beside this one's, and all
// that does not depend on it - barriers, code copies, the expansion of the first six or seven stages - is done when it ends.
//
// 11 warps: 0-7 decode (warp w: rows 32 (w % 4) .. and one half of every stage of 256 k) and do the epilogue, 8 loads activations by TMA
// and allocates tensor memory, 9 streams codes (512 k, 2 KB per strip and copy) and stages the token scales, 10 issues the
// MMAs.  A stage's columns and activations share a ring slot, one barrier and one commit.  With S > 1 the partial sums are
// reduce-scattered through distributed shared memory in units of 8 tokens (st.async, counted by a barrier of the owner; a cluster
// barrier with release and acquire took three times as long), which their owners scale and store.  Every wait is bounded
// (status 4).  Shared memory is at least kTileMinSmem, so that no third CTA competes for tensor memory.
//
// What bounds it: an MMA of 128 rows x 32 k takes 50 cycles up to 64 tokens and a commit 150, so 270 cycles per 128 k of a CTA; around that
// the activations' first load, the exchange and the epilogue, each a chain of latencies.  us per call in a stream of different
// weights, before (mma.sync, pairs or the packed kernel, whichever was taken) and now: 13824 x 2560 at 16 / 48 / 128 tokens 6.9 / 10.0 / 10.9 and
// 5.2 / 6.0 / 7.5, 2560 x 2560 3.8 / 6.9 / 8.2 and 3.3 / 4.1 / 5.3, 2560 x 6912 5.7 / 11.6 / 15.7 and 4.4 / 5.4 / 6.9, 57344 x 8192 at 48 71 and 34.
#pragma once
#include <algorithm>

#include "spmm_large_m.cuh"
#include "w2_small.cuh"

namespace tsp {

constexpr int kTileRows = 128;
constexpr int kTileWorkers = 8;            // decoder warps: a stage is 2 x 128 k, four warps for each half
constexpr int kTileThreads = (kTileWorkers + 3) * 32;
constexpr int kTileMaxStages = 3;
constexpr int kTileCols = 256;             // tensor memory: accumulators, then 64 columns per stage
constexpr int kTileChunk = 4;              // block pairs (128 k) per copy of codes: two stages
constexpr int kTileSlots = 3;              // of codes, at most
constexpr int kTileSlotBytes = 8 * kTileChunk * 512;
constexpr int kTileMaxTokens = 128;
constexpr int kTileMinSmem = 80 * 1024;    // dynamic shared memory of a launch at least (ternaspmm.cu: most_tmem_columns)

constexpr int kTilePart = 8 * kTileRows * 4;   // bytes of a unit's partial sums

struct W2TileSmem {
    static constexpr int bar_full = 0;          // [3]  weights and activations of a stage are in place
    static constexpr int bar_empty = 32;        // [3]  the MMAs have read the stage
    static constexpr int bar_w = 64;            // [3]  codes of a slot have landed
    static constexpr int bar_w_free = 96;       // [3]  the decoder warps have read the slot
    static constexpr int bar_acc = 128;         // accumulators are complete
    static constexpr int bar_scl = 136;         // token scales are staged
    static constexpr int bar_parts = 144;       // the other CTAs' partial sums have arrived
    static constexpr int tmem_slot = 152;
    static constexpr int abort_flag = 156;
    static constexpr int scl_ok = 160;          // every scale lets tile_store take its usual path
    static constexpr int scl = 256;             // float[128] token scales, float[128] their reciprocals or the factors of the prefill form
    static constexpr int ring = 2048;           // codes, then activations; at the end the partial sums of other CTAs
};

struct W2TileParams {
    SpmmParams e;
    const uint8_t* w;                      // two-bit weights
    int nt, stages, slots;                 // tokens per tile, ring slots, slots of codes
};

// Pairs of fp32 values in packed instructions; quotient() of two.
__device__ __forceinline__ unsigned long long f32x2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 f32x2_mul(float2 a, float2 b) {
    unsigned long long r;
    float2 o;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f32x2(a.x, a.y)), "l"(f32x2(b.x, b.y)));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
    return o;
}
__device__ __forceinline__ float2 f32x2_fma(float2 a, float2 b, float2 c) {
    unsigned long long r;
    float2 o;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f32x2(a.x, a.y)), "l"(f32x2(b.x, b.y)), "l"(f32x2(c.x, c.y)));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
    return o;
}
__device__ __forceinline__ float2 quotient2(float2 acc, float2 s, float2 r) {
    const float2 q0 = f32x2_mul(acc, r);
    return f32x2_fma(f32x2_fma(make_float2(-q0.x, -q0.y), s, acc), r, q0);
}
// D[tmem] (+)= A[tmem] * B[smem]; M = 128
__device__ __forceinline__ void umma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p; }" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// a lane's 16 consecutive columns of its row
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
                 "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait(int (&v)[8]) {   // (names the registers: nothing that reads them may move ahead of the wait)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])::"memory");
}

// Codes of a row and one 64-column block, 16 columns per word -> 16 columns of tensor memory.
__device__ __forceinline__ void w2_expand_block(uint32_t taddr, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    uint32_t v[16];
    const uint32_t w[4] = {w0, w1, w2, w3};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t a[4];
        w2_decode(w[i], a);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[4 * i + j] = a[j];
    }
    tmem_st16(taddr, v);
}
// One decoder warp's part of up to two stages of 128 k, `stage_bytes` of codes and one ring slot apart: 32 rows, a lane each.
struct W2RowCodes {
    uint2 w[4];                            // columns 16q .. of block 0 and block 1
    __device__ __forceinline__ void load(uint32_t chunk0, const uint32_t (&off)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = lds64(chunk0 + off[q]);
    }
    __device__ __forceinline__ void expand(uint32_t taddr) const {
        w2_expand_block(taddr, w[0].x, w[1].x, w[2].x, w[3].x);
        w2_expand_block(taddr + 16, w[0].y, w[1].y, w[2].y, w[3].y);
    }
};
// Offset of a lane's codes inside a CTA's strips (each `strip_bytes` long) and the four chunks behind it.
__device__ __forceinline__ uint32_t w2_row_offset(int quarter, int lane, uint32_t strip_bytes, uint32_t (&off)[4]) {
    const int g = lane & 7;
#pragma unroll
    for (int q = 0; q < 4; ++q) off[q] = w2_chunk(g, q) + (lane & 8);
    return (uint32_t)(2 * quarter + (lane >> 4)) * strip_bytes;
}

// wait_or_abort for kernels with many waiting warps: suspended in the barrier (up to 20 us at a time) instead of polling, so
// that they do not take the others' issue slots.  What a wait needs beyond its first test stays out of the pipelines' loops.
__device__ __noinline__ bool wait_longer(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_test_suspended(bar, parity, 20000u)) return true;
    const unsigned long long t0 = global_timer_ns();
#pragma unroll 1
    for (uint32_t it = 0; it < (1u << 24); ++it) {
        if (mbar_test_suspended(bar, parity, 20000u)) return true;
        if (*abort_flag) return false;
        if (global_timer_ns() - t0 > kLgWaitLimitNs) break;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ bool wait_suspended(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return mbar_test_suspended(bar, parity, 20000u) || wait_longer(bar, parity, abort_flag);
}
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {   // the whole warp, one verdict
    if (__all_sync(0xffffffffu, mbar_test_suspended(bar, parity, 20000u))) return true;
    return __all_sync(0xffffffffu, wait_longer(bar, parity, abort_flag));
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{ .reg .pred q; elect.sync _|q, 0xffffffff; selp.u32 %0, 1, 0, q; }" : "=r"(p));
    return p != 0;
}

// A lane's row of four tokens and its neighbour's -> two words of both rows: tokens 0, 1 in the even lane, 2, 3 in the odd one.
__device__ __forceinline__ void pair_rows(uint32_t t01, uint32_t t23, bool odd, uint32_t& o0, uint32_t& o1) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? t01 : t23, 1);
    const uint32_t lo = odd ? other : t01, hi = odd ? t23 : other;   // rows 2i and 2i + 1
    o0 = __byte_perm(lo, hi, 0x5410), o1 = __byte_perm(lo, hi, 0x7632);
}
// 16 bytes into another CTA of the cluster, counted by a barrier there
__device__ __forceinline__ void st_async_v4(uint32_t cluster_addr, int a, int b, int c, int d, uint32_t cluster_bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(cluster_addr), "r"(a),
                 "r"(b), "r"(c), "r"(d), "r"(cluster_bar)
                 : "memory");
}

// ---- epilogue: U units of 8 tokens x 32 rows ---------------------------------------------------------
enum TileForm : int { FORM_FACTOR, FORM_QUOTIENT, FORM_GENERAL };   // ws / s in one factor; (acc / s) * ws; as scale_epilogue has it
struct TileOut {
    float ws_el;                           // weight scale of the lane's row
    int form, left, cols;
    bool wide, n_ok;
    size_t at;
};
// The residual as tile_store adds it: word 4u + j is of token c + 8u + (j & 1) + 4 (j >> 1) from the lane's first one.
template <int U>
__device__ __forceinline__ void tile_residual(const SpmmParams& p, const TileOut& o, int c, uint32_t* r) {
    if (!p.residual || !o.wide) return;
    const __nv_bfloat16* src = p.residual + o.at + (size_t)c * p.N;
#pragma unroll
    for (int j = 0; j < 4 * U; ++j) {
        const int t = (j & 1) + 4 * (j >> 1);
        if (c + t < o.left) r[j] = ld_cg_32(src + (size_t)t * p.N);
    }
}
// What is not on the usual path, out of its instruction stream: odd addresses, scales out of range, several scales in a tile.
__device__ __noinline__ void tile_store_general(const SpmmParams& p, float ws_el, int n_tokens, const int* v, const float* scl, long long at, bool live) {
#pragma unroll 1
    for (int j = 0; j < n_tokens; ++j) {
        const long long o = at + (long long)j * p.N;
        if (live) stg_b16(reinterpret_cast<__nv_bfloat16*>(p.out) + o,
                          __bfloat16_as_ushort(add_residual(scale_epilogue(v[j] >> 6, scl[j], ws_el, p.epilogue), p.residual, o)));
    }
}
template <int U>
__device__ __forceinline__ void tile_store(const SpmmParams& p, const TileOut& o, int c, int (&v)[U][8], const float* scl, const uint32_t* res) {
    const bool odd = threadIdx.x & 1;
    if (o.form == FORM_GENERAL) {
        int all[8 * U];
#pragma unroll
        for (int j = 0; j < 8 * U; ++j) all[j] = v[j >> 3][j & 7];
        const int behind = odd ? 2 : 0;
        tile_store_general(p, o.ws_el, min(8 * U, o.cols - c), all, scl, (long long)o.at + (long long)(c - behind) * p.N + odd, o.n_ok);
        return;
    }
    uint32_t f[U][4];                                        // tokens 2j, 2j + 1, rounded
    // The accumulators are 64 times the sums.  The quotient comes out 64 times too large and the weight scale takes that back: exact, as
    // a quotient is below 2^61 here and a bf16 divided by 64 is a float (a scale times 64 may not be: from 2^122 on it is infinite).
    const float2 ws2 = make_float2(o.ws_el * 0.015625f, o.ws_el * 0.015625f);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float4 aux = *reinterpret_cast<const float4*>(scl + kTileMaxTokens + 8 * u + 4 * j);
            float2 a = make_float2(__int2float_rn(v[u][4 * j]), __int2float_rn(v[u][4 * j + 1]));
            float2 b = make_float2(__int2float_rn(v[u][4 * j + 2]), __int2float_rn(v[u][4 * j + 3]));
            if (o.form == FORM_FACTOR) {
                a = f32x2_mul(a, make_float2(aux.x, aux.y)), b = f32x2_mul(b, make_float2(aux.z, aux.w));
            } else {
                const float4 sv = *reinterpret_cast<const float4*>(scl + 8 * u + 4 * j);
                a = f32x2_mul(quotient2(a, make_float2(sv.x, sv.y), make_float2(aux.x, aux.y)), ws2);
                b = f32x2_mul(quotient2(b, make_float2(sv.z, sv.w), make_float2(aux.z, aux.w)), ws2);
            }
            f[u][2 * j] = act_pack(a.x, a.y), f[u][2 * j + 1] = act_pack(b.x, b.y);
        }
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + o.at + (size_t)c * p.N;
    const size_t row = p.N;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        uint32_t w[4];
        pair_rows(f[u][0], f[u][1], odd, w[0], w[1]);
        pair_rows(f[u][2], f[u][3], odd, w[2], w[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (p.residual) w[j] = act_pack(act_lo(res[4 * u + j]) + act_lo(w[j]), act_hi(res[4 * u + j]) + act_hi(w[j]));
            const int t = 8 * u + (j & 1) + 4 * (j >> 1);
            if (c + t < o.left) stg_b32(out + t * row, w[j]);
        }
    }
}

__global__ void __launch_bounds__(kTileThreads, 2)
    w2_tile_kernel(const __grid_constant__ W2TileParams pp, const __grid_constant__ CUtensorMap tmap_x) {
    using L = W2TileSmem;
    extern __shared__ __align__(128) uint8_t smem[];
    const SpmmParams& p = pp.e;
    const uint32_t dyn = smem_u32(smem);
    const uint32_t sbase = (dyn + 1023u) & ~1023u;       // the same offset in every CTA of the cluster
    uint8_t* rest = smem + (sbase - dyn);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(rest + L::abort_flag);
    const float* scl = reinterpret_cast<const float*>(rest + L::scl);
    auto bar_full = [&](int s) { return sbase + L::bar_full + 8 * s; };
    auto bar_empty = [&](int s) { return sbase + L::bar_empty + 8 * s; };
    auto bar_w = [&](int s) { return sbase + L::bar_w + 8 * s; };
    auto bar_w_free = [&](int s) { return sbase + L::bar_w_free + 8 * s; };
    const uint32_t bar_acc = sbase + L::bar_acc, bar_scl = sbase + L::bar_scl, bar_parts = sbase + L::bar_parts;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = p.N, NT = pp.nt, ST = pp.stages, WS = pp.slots, S = gridDim.x, rank = blockIdx.x;
    const int n0 = blockIdx.y * kTileRows, t0 = blockIdx.z * NT, cols = min(NT, p.M - t0);
    const int KP = w2_pairs(p.K), kp0 = KP * rank / S, KB = KP * (rank + 1) / S - kp0;   // this CTA's block pairs of K
    const uint32_t codes = sbase + L::ring, xring = codes + WS * kTileSlotBytes, x_bytes = (uint32_t)NT * 128;   // (a stage has twice that)
    const int units = (cols + 7) >> 3, owned = (units - rank + S - 1) / S;   // 8 tokens each; unit u is finished by CTA u % S

    phase_mark(0);
    griddep_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) mbar_init(bar_full(s), kTileWorkers + 1), mbar_init(bar_empty(s), 1);   // the decoder warps and the loader
        for (int s = 0; s < WS; ++s) mbar_init(bar_w(s), 1), mbar_init(bar_w_free(s), kTileWorkers);
        mbar_init(bar_acc, 1), mbar_init(bar_scl, 1), mbar_init(bar_parts, 1);
        *abort_flag = 0;
        mbar_fence_init();
        if (S > 1 && owned > 0) mbar_arrive_expect_tx(bar_parts, (uint32_t)((S - 1) * owned * kTilePart));
    }
    if (warp == kTileWorkers) tmem_alloc(sbase + L::tmem_slot, kTileCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(rest + L::tmem_slot);
    const uint32_t a_tmem = tmem_base + kTileCols - (uint32_t)(ST * 64);   // behind the accumulators
    bool ok = true;
    phase_mark(1);

    if (warp == kTileWorkers) {
        // ------------------------------------------------ activations
        if (lane == 0) {
            griddep_wait();   // they come from earlier kernels of the stream
            uint32_t full = bar_full(0), empty = bar_empty(0), x = xring, parity = 1;
            int s = 0;
            for (int kb = 0; kb < KB; kb += 2) {
                if (!wait_suspended(empty, parity, abort_flag)) break;   // (passes in the first round)
                const bool two = kb + 1 < KB;
                mbar_arrive_expect_tx(full, two ? 2 * x_bytes : x_bytes);
                tma_load_2d(x, &tmap_x, (kp0 + kb) * 128, t0, full);
                if (two) tma_load_2d(x + x_bytes, &tmap_x, (kp0 + kb + 1) * 128, t0, full);
                full += 8, empty += 8, x += 2 * x_bytes;
                if (++s == ST) s = 0, full = bar_full(0), empty = bar_empty(0), x = xring, parity ^= 1u;
            }
        }
        __syncwarp();
    } else if (warp == kTileWorkers + 1) {
        // ------------------------------------------------ codes (immutable: no dependency wait), token scales
        const int live = min(8, (N - n0) >> 4);              // strips of a last, smaller row block
        const uint8_t* src = pp.w + ((size_t)((n0 >> 4) + lane) * KP + kp0) * 512;
        int s = 0;
        uint32_t parity = 1;
        auto copy = [&](int kb) {
            const uint32_t bytes = (uint32_t)min(kTileChunk, KB - kb) * 512;
            if (lane == 0) mbar_arrive_expect_tx(bar_w(s), (uint32_t)live * bytes);
            __syncwarp();
            if (lane < live) bulk_load(codes + s * kTileSlotBytes + lane * (kTileChunk * 512), src + (size_t)kb * 512, bytes, bar_w(s));
            if (++s == WS) s = 0, parity ^= 1u;
        };
        for (int kb = 0; kb < min(KB, WS * kTileChunk); kb += kTileChunk) copy(kb);
        griddep_wait();
        {
            const float ws0 = __bfloat162float(p.ws[ws_group(n0, p)]);
            bool in_range = true;
            for (int t = lane; t < NT; t += 32) {
                const float sv = t < cols ? __bfloat162float(p.s[t0 + t]) : 1.f;
                float aux = quotient_rcp(sv);
                if (p.epilogue == EPI_PREFILL) {
                    aux = sv != 0.f ? __fdiv_rn(ws0, sv) : 0.f;
                    // over 64, for sums that are 64 times theirs: exact in this range
                    aux = fabsf(aux) >= 0x1p-60f && fabsf(aux) <= 0x1p60f ? aux * 0.015625f : 0.f;
                }
                float* dst = reinterpret_cast<float*>(rest + L::scl) + t;
                dst[0] = sv, dst[kTileMaxTokens] = aux;
                in_range &= aux != 0.f;
            }
            in_range = __all_sync(0xffffffffu, in_range);
            if (lane == 0) *reinterpret_cast<int*>(rest + L::scl_ok) = in_range;
            __syncwarp();                                    // (a vote orders no memory: the other lanes' scales, before lane 0 releases them)
            if (lane == 0) mbar_arrive(bar_scl);
        }
        for (int kb = WS * kTileChunk; kb < KB; kb += kTileChunk) {
            if (!wait_warp(bar_w_free(s), parity, abort_flag)) break;
            copy(kb);
        }
    } else if (warp == kTileWorkers + 2) {
        // ------------------------------------------------ MMA issuer
        if (elect_one()) {
            // int8 x int8 -> int32, A in tensor memory, K-major B, M = 128, N = NT
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
            const uint64_t x_desc0 = umma_desc_sw128(xring);
            uint64_t x_desc = x_desc0;
            uint32_t a = a_tmem, full = bar_full(0), empty = bar_empty(0), parity = 0, accumulate = 0;
            int s = 0;
            for (int kb = 0; kb < KB; kb += 2) {
                if (!wait_suspended(full, parity, abort_flag)) break;
                tc_fence_after();
                if (kb == 0) phase_mark_here(3);
#pragma unroll
                for (int j = 0; j < 4; ++j) umma_i8_ts(tmem_base, a + 8 * j, x_desc + 2 * j, idesc, j ? 1u : accumulate);
                if (kb + 1 < KB) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_i8_ts(tmem_base, a + 32 + 8 * j, x_desc + (x_bytes >> 4) + 2 * j, idesc, 1u);
                }
                accumulate = 1;
                umma_commit(kb + 2 >= KB ? bar_acc : empty);
                a += 64, full += 8, empty += 8, x_desc += x_bytes >> 3;   // descriptor addresses count 16 bytes
                if (++s == ST) s = 0, a = a_tmem, full = bar_full(0), empty = bar_empty(0), x_desc = x_desc0, parity ^= 1u;
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------ decoders: a lane has a row, a warp one half of every stage
        const int quarter = warp & 3, group = warp >> 2;
        const uint32_t lanes = (uint32_t)(32 * quarter) << 16;
        uint32_t off[4];
        const uint32_t w_lane = codes + w2_row_offset(quarter, lane, kTileChunk * 512, off) + group * 512;
        uint32_t full = bar_full(0), empty = bar_empty(0), a = a_tmem + lanes + 32 * group, parity = 1, slot = 0;
        int s = 0, ws = 0, w_parity = 0;
        for (int kb = 0; kb < KB; kb += kTileChunk) {
            ok = wait_warp(bar_w(ws), w_parity, abort_flag);
            if (!ok) break;
            W2RowCodes w[2];
            w[0].load(w_lane + slot, off), w[1].load(w_lane + slot + 1024, off);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (kb + 2 * u >= KB) break;
                ok = wait_warp(empty, parity, abort_flag);   // (passes in the first round)
                if (!ok) break;
                tc_fence_after();
                w[u].expand(a);                              // (behind the last block pair: whatever the slot held, read by no MMA)
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(full);
                full += 8, empty += 8, a += 64;
                if (++s == ST) s = 0, full = bar_full(0), empty = bar_empty(0), a = a_tmem + lanes + 32 * group, parity ^= 1u;
            }
            if (!ok) break;
            if (lane == 0) mbar_arrive(bar_w_free(ws));
            slot += kTileSlotBytes;
            if (++ws == WS) ws = 0, slot = 0, w_parity ^= 1;
        }
        phase_mark(2);
        // ------------------------------------------------ epilogue
        griddep_wait();  // scales, residual and the output buffer may belong to the previous kernel
        const int n = n0 + 32 * quarter + lane;
        const bool n_ok = n < N, odd = lane & 1;             // (uniform over the warp: N is a multiple of 64)
        TileOut o;
        o.ws_el = n_ok ? __bfloat162float(p.ws[ws_group(n, p)]) : 0.f;
        o.form = p.epilogue != EPI_PREFILL ? FORM_QUOTIENT : ws_group(n0, p) == ws_group(min(n0 + kTileRows, N) - 1, p) ? FORM_FACTOR : FORM_GENERAL;
        o.wide = ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual)) & 3) == 0;
        o.n_ok = n_ok, o.cols = cols;
        o.left = n_ok ? cols - (odd ? 2 : 0) : 0;            // tokens, from this lane's first one
        o.at = (size_t)(t0 + (odd ? 2 : 0)) * N + (n & ~1);  // its pair of rows
        int c = S > 1 ? (rank + group * S) * 8 : group * 16; // this warp's first tokens
        uint32_t res[8];
        if (c < cols) tile_residual<2>(p, o, c, res);        // (more than a unit needs where S > 1)
        if (ok) ok = wait_warp(bar_scl, 0, abort_flag);
        if (!o.wide || !*reinterpret_cast<const volatile int*>(rest + L::scl_ok)) o.form = FORM_GENERAL;
        if (ok) ok = wait_warp(bar_acc, 0, abort_flag);
        tc_fence_after();
        phase_mark(4);
        const uint32_t acc = tmem_base + lanes;
        if (S > 1) {
            cluster_arrive_relaxed();                        // this CTA's rings are idle, its barriers initialised
            cluster_wait();
            for (int u = group; u < units && ok; u += 2) {
                const int owner = u % S;
                if (owner == rank) continue;
                int v[8];
                tmem_ld8(acc + (uint32_t)(u * 8), v);
                tmem_ld_wait(v);
                const uint32_t dst = map_to_rank(codes + (uint32_t)((u / S) * (S - 1) + rank - (rank > owner)) * kTilePart + (32 * quarter + lane) * 16, owner);
                const uint32_t bar = map_to_rank(bar_parts, owner);
                st_async_v4(dst, v[0], v[1], v[2], v[3], bar);
                st_async_v4(dst + kTilePart / 2, v[4], v[5], v[6], v[7], bar);
            }
            if (ok && owned > 0) ok = wait_warp(bar_parts, 0, abort_flag);
            phase_mark(5);
            uint32_t parts = codes + (uint32_t)(group * (S - 1) * kTilePart) + (32 * quarter + lane) * 16;
            for (; c < cols && ok; c += 16 * S) {
                int v[1][8];
                tmem_ld8(acc + (uint32_t)c, v[0]);
                tmem_ld_wait(v[0]);
#pragma unroll 2
                for (int r = 0; r < S - 1; ++r, parts += kTilePart) {
                    const uint4 lo = lds128(parts), hi = lds128(parts + kTilePart / 2);
                    v[0][0] += (int)lo.x, v[0][1] += (int)lo.y, v[0][2] += (int)lo.z, v[0][3] += (int)lo.w;
                    v[0][4] += (int)hi.x, v[0][5] += (int)hi.y, v[0][6] += (int)hi.z, v[0][7] += (int)hi.w;
                }
                parts += (S - 1) * kTilePart;                // the other group's unit
                tile_store<1>(p, o, c, v, scl + c, res);
                if (c + 16 * S < cols) tile_residual<1>(p, o, c + 16 * S, res);
            }
        } else {
            for (; c < cols && ok; c += 32) {                // two units at a time: a unit is a chain of latencies
                int v[2][8];
                tmem_ld8(acc + (uint32_t)c, v[0]), tmem_ld8(acc + (uint32_t)c + 8, v[1]);
                tmem_ld_wait(v[0]), tmem_ld_wait(v[1]);
                tile_store<2>(p, o, c, v, scl + c, res);
                if (c + 32 < cols) tile_residual<2>(p, o, c + 32, res);
            }
        }
        phase_mark(6);
    }
    if (S > 1 && warp >= kTileWorkers) {                     // (the workers' barrier)
        cluster_arrive_relaxed();
        cluster_wait();
    }
    if (*abort_flag) {                                       // copies and MMAs in flight end long before this
        if (tid == 0) atomicExch(p.status, ST_WAIT_TIMEOUT);
        const unsigned long long since = global_timer_ns();
        for (uint32_t it = 0; it < (1u << 20) && global_timer_ns() - since < 100ull * 1000; ++it) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kTileWorkers) tmem_dealloc(tmem_base, kTileCols);
    phase_mark(7);
}

// Tokens per tile and K slices of a call, and the time it takes, in us.  The CTAs of two to an SM (clusters leave some places empty) run
// at once, each KB = K / 128 / S block pairs long, 0.15 us each, 0.22 with two CTAs on an SM's tensor cores; a further round of CTAs costs
// its own start and end, and a cluster's exchange grows with S.  Tiles of more than 64 tokens have room for two stages only, 0.34 us per block
// pair, and pay where they save a round.  The constants of this and of w2_pair_plan_tile are fitted to 5400 measured plans of 582 calls of 9 to
// 4096 tokens (the layers of both models, their shards, and sizes drawn over the range): the plan chosen is 1.0 % slower than the best one in the mean,
// 1.1 % on calls that were left out of a fit.  us per call, S = 1 / 2 / 4 / 6 / 8: 2560 x 2560 at 48 tokens 5.2 / 4.4 / 4.1 / 4.4 / 5.4, 2560 x 6912 at 16 9.5 / 6.2 /
// 5.0 / 4.5 / 4.6, 1024 x 16384 at 16 19.5 / 11.1 / 7.1 / 6.1 / 5.3, 8192 x 8192 at 16 11.2 / 8.6 / 7.0 / 10.6 / 11.8 (384 CTAs with six slices); tiles of up to 64 / 128
// tokens: 2560 x 2560 at 1600 15.7 / 11.6, 8192 x 1024 at 512 10.9 / 7.7, 13824 x 2560 at 256 13.9 / 11.3.
struct W2TilePlan { int nt, splits; double us; };
inline W2TilePlan w2_tile_plan(int M, int N, int K, int sms) {
    const int tiles = (N + kTileRows - 1) / kTileRows, KP = w2_pairs(K);
    W2TilePlan best = {0, 0, 1e30};
    for (int most = 64; most <= kTileMaxTokens; most *= 2) {
        const int blocks = (M + most - 1) / most, nt = ((M + blocks - 1) / blocks + 15) & ~15;
        if (blocks > 65535 || tiles > 65535) continue;      // (the limits of a grid)
        for (int S = 1; S <= (nt > 64 ? 1 : std::min(8, KP)); ++S) {
            const long long ctas = (long long)tiles * blocks * S, at_once = S > 1 ? sms * 2 - sms / 4 : sms * 2;
            const long long rounds = (ctas + at_once - 1) / at_once, last = ctas - (rounds - 1) * at_once;
            const bool big = nt > 64;
            const double KB = (KP + S - 1) / S, alone = big ? 0.338 : 0.154, two = big ? 0.355 : 0.216;
            if (rounds > 1 && S > 1) break;                  // (a second round of clusters waits for whole ones to end)
            const double us = (big ? 0.75 + 0.0212 * nt : 1.3 + 0.025 * nt) + KB * ((rounds - 1) * two + (last > sms ? two : alone)) + (rounds - 1) * 3.05 +
                              (S > 1 ? 0.233 * S : 0.0) + (ctas > sms ? 0.27 : 0.0);
            if (us < best.us) best = {nt, S, us};
        }
    }
    return best;
}

}  // namespace tsp
