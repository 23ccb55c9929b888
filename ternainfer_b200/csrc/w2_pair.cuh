// Large batches on two-bit weights for sm_100a: tcgen05 int8 GEMM on CTA pairs whose weight operand is expanded into tensor memory.
//
// The packed format takes a decoder warp 0.12 instructions per weight, so the large-batch path that reads it decodes the
// weight once per call into a dense workspace (dense_prefill.cuh: 8 us for 13824 x 2560, and 16 times the bytes through
// L2 afterwards).  Two-bit codes (w2_small.cuh) expand with 7 instructions per 16 weights of a lane: eight decoder warps keep
// pace with the tensor cores, and neither the extra pass nor the workspace is needed.
//
// A pair (cluster of 2) owns a tile of 256 weight rows x NT tokens (CTA r: rows 128 r .. + 127 and half of the tokens) and walks over
// K in stages of 128 with tcgen05.mma.cta_group::2, whose A operand lies in tensor memory (w2_tile.cuh has the expansion).  Per CTA 27
// warps: warp 0 loads activation tiles by TMA, completing on the leader's barrier; warp 1 allocates tensor memory and, in the
// leader, issues the MMAs; warps 2-17 are the epilogue; warps 18-25 the decoders, two per quarter of the rows with every second stage
// each; warp 26 streams the two-bit weights of four stages at a time by cp.async.bulk, 2 KB per strip (the copy engine takes
// about 60 cycles per bulk copy whatever its size: 512-byte copies, eight per stage, were the bound at 700 cycles per stage).  A
// stage's two operands share ONE barrier and ONE commit: a commit costs the tensor pipe about
// 150 cycles (four MMAs of 50 and a commit 352, eight and a commit 540, N up to 64).  Every wait is bounded (status 4).
//
// Tensor memory holds two accumulator buffers of up to 192 columns and four to eight stages of weights, or one of 256 and eight; the
// eight activation slots in shared memory are a ring of their own, as deep as a TMA load from L2 is long (with four slots of
// both, 192 tokens took 0.33 us per stage; so 0.23).  With the operand expanded into shared memory a stage of 128 k was 0.26 us up to
// 128 tokens, whatever their number, and 0.29 at 256 (the port: stores, MMA reads, TMA); in tensor memory, and with less control code
// - waits that read the clock, issue loops run by whole warps: 300 cycles per stage alone - 0.164 at 64 tokens, 0.174 at 128 and 0.23 at 192 (tensor cores 0.20).
// us per call, before and now: 13824 x 2560 at 48 tokens (as pairs) 10.1 / 7.7, 3840 x 2560 at 333 10.4 / 8.2, 2560 x 6912 at 2048 35.7 / 25.8,
// 13824 x 2560 at 1226 35.7 / 33.0.
#pragma once
#include <algorithm>

#include "dense_pair.cuh"
#include "w2_tile.cuh"

namespace tsp {

constexpr int kW2PairDecoders = 8;
constexpr int kW2PairFirstDecoder = kLgFirstEpi + kPairEpiWarps;
constexpr int kW2PairThreads = (kW2PairFirstDecoder + kW2PairDecoders + 1) * 32;
constexpr int kW2OutStride = 80;           // bytes between two tokens of an output slice in shared memory: conflict-free
constexpr int kW2OutStageBytes = 16 * kW2OutStride;
constexpr int kW2PairMaxStages = 8;
constexpr int kW2PairSlots = 4;            // of two-bit weights: 128 rows x 512 k each
constexpr int kW2PairCols = 32;            // tensor-memory columns of a stage's weights: 128 k of four int8 each
constexpr int kW2PairChunk = 4;            // stages per slot
constexpr int kW2PairSlotBytes = kW2PairDecoders * kW2PairChunk * 512;

struct W2PairSmem {
    static constexpr int bar_full = 0;          // [8]  leader: both CTAs' weight rows and activation bytes of a stage are in place
    static constexpr int bar_empty = 64;        // [8]  each CTA: the MMAs have read the stage
    static constexpr int bar_acc_full = 128;    // [2]  each CTA: a tile's accumulators are complete
    static constexpr int bar_acc_empty = 144;   // [2]  leader: both CTAs' epilogues have read the buffer
    static constexpr int bar_w = 160;           // [4]  each CTA: two-bit weights of a slot have landed
    static constexpr int bar_w_free = 192;      // [4]  each CTA: the decoder warps have read the slot
    static constexpr int tmem_slot = 224;
    static constexpr int abort_flag = 228;
    static constexpr int scl = 256;             // float[64] scales and float[64] reciprocals per epilogue warp
    static constexpr int ostage = scl + kPairEpiWarps * 128 * 4;   // 1 KB per epilogue warp (output staging)
    static constexpr int w = (ostage + kPairEpiWarps * kW2OutStageBytes + 1023) / 1024 * 1024;
    static constexpr int stage = w + kW2PairSlots * kW2PairSlotBytes;   // activations, NT * 64 bytes per stage
    static constexpr int total = 1024 + stage + kW2PairMaxStages * 128 * kLgKStep;
};

// D[tmem of both CTAs] (+)= A[tmem of both CTAs] * B[smem of both CTAs]; M = 256, N and K = 32 from the descriptors
__device__ __forceinline__ void umma_i8_pair_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], [%1], %2, %3, p; }" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive on a barrier of any CTA of the cluster, releasing to this CTA's scope.  That suffices here, although the waiting MMA thread may
// be the peer's: what it is told is about tensor memory alone - a stage's weights are in it (decoders), an accumulator buffer has been
// read (epilogue).  Those accesses are complete, in the SM that they belong to, when tcgen05.wait::st or ::ld returns, before the
// arrival is issued, and tcgen05.fence::before_thread_sync, the barrier's phase and tcgen05.fence::after_thread_sync order the MMAs behind
// them.  The scope only says whose reads of ordinary memory see this thread's writes, and the MMA thread reads none of them: the
// activations are the copy engine's, counted by the same barrier.  Other forms cost more without saying more: released to the
// cluster 1200 cycles per stage, relaxed at cluster scope 13824 x 2560 at 1226 tokens 36.1 us instead of 33.0.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// bf16 epilogue of a slice of 16 tokens x 32 weight rows.  The accumulators come as 8x8 matrix fragments (rows = weight rows,
// columns = tokens; a lane has two neighbouring tokens of four rows), so that a lane needs four token scales instead of
// sixteen and stmatrix transposes on the way to shared memory: a third of the instructions of the row-per-lane form
// (store_slice16_wide).  ws_rows: weight scales of rows 8r + lane / 4; `ahead`: the residual as load_residual16 reads it.
// sc: [16] token scales, for FORM_FACTOR those of the whole product; rc: [16] their reciprocals, for FORM_QUOTIENT.
struct SliceAcc { int v[2][8]; };          // [16 rows][token half x (row half, token)]
__device__ __forceinline__ void load_slice16(uint32_t tmem, SliceAcc& a) {   // (waited for in store_slice16_matrix)
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(a.v[h][0]), "=r"(a.v[h][1]), "=r"(a.v[h][2]), "=r"(a.v[h][3]), "=r"(a.v[h][4]), "=r"(a.v[h][5]), "=r"(a.v[h][6]),
                       "=r"(a.v[h][7])
                     : "r"(tmem + ((uint32_t)(16 * h) << 16)));
}
template <int FORM>
__device__ __forceinline__ void store_slice16_matrix(const SpmmParams& p, SliceAcc& acc, const float* sc, const float* rc, long long o_row0,
                                                     int live, const float (&ws_rows)[4], uint32_t stage, int lane, const uint4 (&ahead)[2]) {
    float2 s[2], q[2];
    s[0] = *reinterpret_cast<const float2*>(sc + 2 * (lane & 3)), s[1] = *reinterpret_cast<const float2*>(sc + 8 + 2 * (lane & 3));
    if (FORM == FORM_QUOTIENT) q[0] = *reinterpret_cast<const float2*>(rc + 2 * (lane & 3)), q[1] = *reinterpret_cast<const float2*>(rc + 8 + 2 * (lane & 3));
#pragma unroll
    for (int h = 0; h < 2; ++h)            // (names the registers: nothing that reads them may move ahead of the wait)
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(acc.v[h][0]), "+r"(acc.v[h][1]), "+r"(acc.v[h][2]), "+r"(acc.v[h][3]), "+r"(acc.v[h][4]), "+r"(acc.v[h][5]),
                       "+r"(acc.v[h][6]), "+r"(acc.v[h][7])::"memory");
    uint32_t m[2][4];                                        // [token half][8 rows]: two tokens
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int a = acc.v[r >> 1][4 * t + 2 * (r & 1)] >> 6, b = acc.v[r >> 1][4 * t + 2 * (r & 1) + 1] >> 6;   // the operand holds 64 * weight
            const float2 ab = make_float2(__int2float_rn(a), __int2float_rn(b));
            float2 f;
            if (FORM == FORM_FACTOR) f = f32x2_mul(ab, s[t]);
            if (FORM == FORM_QUOTIENT) f = f32x2_mul(quotient2(ab, s[t], q[t]), make_float2(ws_rows[r], ws_rows[r]));
            if (FORM != FORM_GENERAL) m[t][r] = act_pack(f.x, f.y);
            else
                m[t][r] = (uint32_t)__bfloat16_as_ushort(scale_epilogue(a, s[t].x, ws_rows[r], p.epilogue)) |
                          ((uint32_t)__bfloat16_as_ushort(scale_epilogue(b, s[t].y, ws_rows[r], p.epilogue)) << 16);
        }
#pragma unroll
    for (int t = 0; t < 2; ++t) {                            // matrix r -> tokens 8t .. 8t+7, columns 8r .. 8r+7; lane l addresses row l % 8 of matrix l / 8
        const uint32_t addr = stage + (uint32_t)((8 * t + (lane & 7)) * kW2OutStride + (lane >> 3) * 16);
        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(m[t][0]), "r"(m[t][1]), "r"(m[t][2]),
                     "r"(m[t][3])
                     : "memory");
    }
    __syncwarp();
    const int part = lane & 3;
    uint4 d[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) d[i] = lds128(stage + (uint32_t)(((lane >> 2) + 8 * i) * kW2OutStride + part * 16));
    if (p.residual) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint32_t* dv = reinterpret_cast<uint32_t*>(&d[i]);
            const uint32_t* rv = reinterpret_cast<const uint32_t*>(&ahead[i]);
#pragma unroll
            for (int e = 0; e < 4; ++e) dv[e] = act_pack(act_lo(rv[e]) + act_lo(dv[e]), act_hi(rv[e]) + act_hi(dv[e]));
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = (lane >> 2) + 8 * i;
        if (row < live) stg_128(reinterpret_cast<__nv_bfloat16*>(p.out) + o_row0 + (long long)row * p.N + part * 8, d[i]);
    }
    __syncwarp();   // the staging area is free for the next slice
}

struct W2PairParams {
    SpmmParams e;
    const uint8_t* w;                      // two-bit weights
    int nt, stages;                        // tokens per tile: a multiple of 32 from 96 to 256; ring slots
    int a_stages;                          // of them, slots of weights in tensor memory
    int acc_bufs, acc_cols;                // accumulator buffers in tensor memory and the columns between them
};

// 512 columns of tensor memory hold the accumulators and, behind them, the weights of the stages in flight.
inline void w2_pair_plan(W2PairParams& pp) {
    pp.acc_bufs = pp.nt <= 192 ? 2 : 1;
    pp.acc_cols = pp.nt <= 128 ? 128 : pp.nt <= 192 ? 192 : 256;
    pp.stages = kW2PairMaxStages;
    pp.a_stages = std::min(pp.stages, (512 - pp.acc_bufs * pp.acc_cols) / kW2PairCols);
}

__global__ void __launch_bounds__(kW2PairThreads, 1)
    w2_pair_kernel(const __grid_constant__ W2PairParams pp, const __grid_constant__ CUtensorMap tmap_x) {
    using L = W2PairSmem;
    constexpr int WS = kW2PairSlots;
    extern __shared__ __align__(128) uint8_t smem[];
    const SpmmParams& p = pp.e;
    const uint32_t dyn = smem_u32(smem);
    const uint32_t sbase = (dyn + 1023u) & ~1023u;       // the same offset in both CTAs of the pair
    uint8_t* rest = smem + (sbase - dyn);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(rest + L::abort_flag);
    float* s_s = reinterpret_cast<float*>(rest + L::scl);
    auto bar_full = [&](int s) { return sbase + L::bar_full + 8 * s; };
    auto bar_empty = [&](int s) { return sbase + L::bar_empty + 8 * s; };
    auto bar_acc_full = [&](int b) { return sbase + L::bar_acc_full + 8 * b; };
    auto bar_acc_empty = [&](int b) { return sbase + L::bar_acc_empty + 8 * b; };
    auto bar_w = [&](int s) { return sbase + L::bar_w + 8 * s; };
    auto bar_w_free = [&](int s) { return sbase + L::bar_w_free + 8 * s; };

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = p.N, K = p.K, M = p.M, NT = pp.nt, ST = pp.stages;
    const uint32_t x_bytes = (uint32_t)NT * (kLgKStep / 2);   // this CTA's half of a stage's tokens
    const uint32_t stage0 = sbase + L::stage;
    const uint32_t crank = cluster_ctarank();            // 0 = leader
    const int pair = (int)blockIdx.x >> 1, npairs = (int)gridDim.x >> 1;
    const int KS = w2_pairs(K);                          // stages of 128 k = block pairs of the layout
    const int RB = (N + kPairRows - 1) / kPairRows;      // row block fastest: pairs that run side by side share the activation tile in L2
    const int n_tiles = RB * ((M + NT - 1) / NT);
    const int my_tiles = pair < n_tiles ? (n_tiles - 1 - pair) / npairs + 1 : 0;

    phase_mark(0);
    griddep_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(bar_full(s), 1 + kW2PairDecoders);   // the leader's loader thread (+ the TMA bytes of both CTAs), four decoder warps of each CTA
            mbar_init(bar_empty(s), 1);                        // tcgen05.commit
        }
        for (int s = 0; s < WS; ++s) mbar_init(bar_w(s), 1), mbar_init(bar_w_free(s), kW2PairDecoders);
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_acc_full(b), 1);                   // tcgen05.commit after a tile's last MMA
            mbar_init(bar_acc_empty(b), 2 * kPairEpiWarps);  // the epilogue warps of both CTAs
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc_pair(sbase + L::tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    cluster_arrive();                        // the peer's barriers exist before anything is sent to them
    cluster_wait();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(rest + L::tmem_slot);
    const int SA = pp.a_stages;
    const uint32_t a_tmem = tmem_base + 512u - (uint32_t)(SA * kW2PairCols);   // behind the accumulators
    bool ok = true;
    phase_mark(1);

    if (warp == 0) {
        // ------------------------------------------------ activation loader (both CTAs)
        if (lane == 0) {
            griddep_wait();   // the activations come from earlier kernels of the stream
            phase_mark(2);
            const uint32_t full0 = map_to_rank(bar_full(0), 0);
            uint32_t parity = 1;
            int s = 0;
            for (int ti = 0; ti < my_tiles && ok; ++ti) {
                const int t0 = ((pair + ti * npairs) / RB) * NT + (int)crank * (NT / 2);   // this CTA's tokens
                for (int ks = 0; ks < KS; ++ks) {
                    ok = wait_suspended(bar_empty(s), parity, abort_flag);   // (passes in the first round)
                    if (!ok) break;
                    if (crank == 0) mbar_arrive_expect_tx(bar_full(s), 2 * x_bytes);
                    tma_load_2d_pair(stage0 + s * x_bytes, &tmap_x, ks * kLgKStep, t0, full0 + 8 * s);
                    if (++s == ST) s = 0, parity ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------ MMA issuer (leader only)
        if (crank == 0 && elect_one()) {
            // int8 x int8 -> int32, A in tensor memory, K-major B, M = 256 over the pair, N = NT
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kPairRows >> 4) << 24);
            const uint64_t x_desc0 = umma_desc_sw128(stage0);
            uint64_t x_desc = x_desc0;
            uint32_t a = a_tmem, full = bar_full(0), empty = bar_empty(0), parity = 0, acc_parity = 1, d_tmem = tmem_base;
            int s = 0, sa = 0, buf = 0;
            for (int ti = 0; ti < my_tiles && ok; ++ti) {
                // both CTAs' epilogues must have drained this accumulator buffer (passes in the first round)
                ok = wait_suspended(bar_acc_empty(buf), acc_parity, abort_flag);
                if (!ok) break;
                tc_fence_after();
                for (int ks = 0; ks < KS; ++ks) {
                    ok = wait_suspended(full, parity, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    if (ti == 0 && ks == 0) phase_mark_here(3);
#pragma unroll
                    for (int j = 0; j < 4; ++j)   // four K=32 slices: eight columns of weights, 32 bytes inside the 128-byte swizzle row
                        umma_i8_pair_ts(d_tmem, a + 8 * j, x_desc + 2 * j, idesc, (ks | j) != 0);
                    umma_commit_pair(empty);     // frees the stage in both CTAs
                    a += kW2PairCols, full += 8, empty += 8, x_desc += x_bytes >> 4;   // descriptor addresses count 16 bytes
                    if (++sa == SA) sa = 0, a = a_tmem;
                    if (++s == ST) s = 0, full = bar_full(0), empty = bar_empty(0), x_desc = x_desc0, parity ^= 1u;
                }
                umma_commit_pair(bar_acc_full(buf));   // this tile's accumulators are complete in both CTAs
                d_tmem += pp.acc_cols;
                if (++buf == pp.acc_bufs) buf = 0, d_tmem = tmem_base, acc_parity ^= 1u;
            }
        }
        __syncwarp();
    } else if (warp == kW2PairFirstDecoder + kW2PairDecoders) {
        // ---------------------------------------------------------- two-bit weights (both CTAs, own 128 rows; immutable: no dependency wait)
        int s = 0, it = 0;
        for (int ti = 0; ti < my_tiles && ok; ++ti) {
            const int strip0 = ((pair + ti * npairs) % RB) * (kPairRows / 16) + (int)crank * 8;
            const int live = max(0, min(kW2PairDecoders, (N >> 4) - strip0));   // strips of a last, smaller row block
            const uint8_t* src = pp.w + (size_t)(strip0 + lane) * KS * 512;
            for (int ks = 0; ks < KS; ks += kW2PairChunk) {
                ok = wait_warp(bar_w_free(s), (it & 1) ^ 1, abort_flag);   // (passes in the first round)
                if (!ok) break;
                const uint32_t bytes = (uint32_t)min(kW2PairChunk, KS - ks) * 512;
                if (lane == 0) mbar_arrive_expect_tx(bar_w(s), (uint32_t)live * bytes);
                __syncwarp();
                if (lane < live)
                    bulk_load(sbase + L::w + s * kW2PairSlotBytes + lane * (kW2PairChunk * 512), src + (size_t)ks * 512, bytes, bar_w(s));
                if (++s == WS) s = 0, ++it;
            }
        }
    } else if (warp >= kW2PairFirstDecoder) {
        // ---------------------------------------------------------- decoders (both CTAs, own 128 weight rows)
        // a lane has a row, a warp 32 rows and every second stage of a tile
        const int quarter = warp & 3, group = (warp - kW2PairFirstDecoder) >> 2;
        uint32_t off[4];
        const uint32_t w_lane = sbase + L::w + w2_row_offset(quarter, lane, kW2PairChunk * 512, off) + group * 512;
        const uint32_t a_lane = a_tmem + ((uint32_t)(32 * quarter) << 16);
        const uint32_t full0 = map_to_rank(bar_full(0), 0);   // the leader's
        // A stage's weights go where those of SA stages before it were, whose MMAs have read them: positions in the ring of barriers
        // (two rounds being one turn) and in tensor memory, of the tile's first stage and of this warp's next one
        int base = 0, base_a = 0, ws = 0, w_parity = 0;
        for (int ti = 0; ti < my_tiles && ok; ++ti) {
            int pos = base + group, sa = base_a + group;
            if (pos >= 2 * ST) pos -= 2 * ST;
            if (sa >= SA) sa -= SA;
#pragma unroll 1
            for (int ks = group; ks < KS + group; ks += kW2PairChunk) {   // (every warp looks at every slot)
                ok = wait_warp(bar_w(ws), w_parity, abort_flag);
                if (!ok) break;
                static_assert(kW2PairChunk == 4 && kW2PairDecoders == 8, "two stages of a slot are a warp's");
                W2RowCodes w[2];
                w[0].load(w_lane + ws * kW2PairSlotBytes, off), w[1].load(w_lane + ws * kW2PairSlotBytes + 1024, off);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (ks + 2 * u >= KS) break;
                    const int s = pos >= ST ? pos - ST : pos;
                    int before = pos - SA;
                    if (before < 0) before += 2 * ST;
                    const bool second = before >= ST;
                    ok = wait_warp(bar_empty(second ? before - ST : before), second ? 1u : 0u, abort_flag);   // (passes for the first SA stages)
                    if (!ok) break;
                    tc_fence_after();
                    w[u].expand(a_lane + (uint32_t)(sa * kW2PairCols));
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(full0 + 8 * s);
                    pos += 2, sa += 2;
                    if (pos >= 2 * ST) pos -= 2 * ST;
                    if (sa >= SA) sa -= SA;
                }
                if (!ok) break;
                if (lane == 0) mbar_arrive(bar_w_free(ws));
                if (++ws == WS) ws = 0, w_parity ^= 1;
            }
            base = (base + KS) % (2 * ST), base_a = (base_a + KS) % SA;
        }
    } else {
        // ---------------------------------------------------------- epilogue (both CTAs, own 128 weight rows)
        griddep_wait();  // scales, residual and the output buffer may belong to the previous kernel
        const int quarter = warp & 3;          // the tensor-memory lanes a warp may read: 32 * (warp % 4)
        const int cg = (warp - kLgFirstEpi) >> 2;   // this warp's slices of 16 tokens: cg, cg + 4, ...
        float *s_w = s_s + (warp - kLgFirstEpi) * 128, *r_w = s_w + 64;
        const uint32_t ostage = sbase + L::ostage + (uint32_t)((warp - kLgFirstEpi) * kW2OutStageBytes);
        const bool wide = ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual)) & 15) == 0;
        int buf = 0, use = 0;
        for (int ti = 0; ti < my_tiles; ++ti) {
            const int tile = pair + ti * npairs;
            const int rb = tile % RB, t0 = (tile / RB) * NT;
            const int n = rb * kPairRows + (int)crank * 128 + 32 * quarter + lane;
            const bool n_ok = n < N;
            const int gsel = n_ok ? ws_group(n, p) : -1;
            const float ws_el = gsel >= 0 ? __bfloat162float(p.ws[gsel]) : 0.f;
            const int g0 = __shfl_sync(0xffffffffu, gsel, 0);
            const bool fast = p.epilogue == EPI_PREFILL && __all_sync(0xffffffffu, gsel == g0 || gsel < 0);
            const float ws0 = __shfl_sync(0xffffffffu, ws_el, 0);
            float ws_rows[4];                      // of the rows that store_slice16_matrix gives this lane
#pragma unroll
            for (int r = 0; r < 4; ++r) ws_rows[r] = __shfl_sync(0xffffffffu, ws_el, 8 * r + (lane >> 2));
            __syncwarp();                          // the previous tile's scales are no longer read
            bool in_range = p.epilogue != EPI_PREFILL;
            for (int i = lane; i < 64; i += 32) {  // token of local slot i: slice cg + 4 (i / 16)
                const int c = (cg + 4 * (i >> 4)) * 16 + (i & 15);
                const float sv = (c < NT && t0 + c < M) ? __bfloat162float(p.s[t0 + c]) : 1.f, rv = quotient_rcp(sv);
                s_w[i] = fast ? ((sv != 0.f) ? __fdiv_rn(ws0, sv) : 0.f) : sv;
                r_w[i] = rv;
                in_range &= rv != 0.f;
            }
            in_range = __all_sync(0xffffffffu, in_range);
            __syncwarp();                          // (a vote orders no memory: the lanes read each other's scales)
            const int cols = min(NT, M - t0);
            uint4 res[2], res_next[2];          // the residual is read one slice ahead
            auto residual_of = [&](int i, uint4 (&r)[2]) {
                const int c0 = (cg + 4 * i) * 16;
                if (wide && p.residual && c0 < cols)
                    load_residual16(p, (long long)(t0 + c0) * N + n - lane, n_ok ? min(16, M - t0 - c0) : 0, lane, r);
            };
            residual_of(0, res);
            ok = ok && wait_warp(bar_acc_full(buf), use & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (ti == 0 && warp == kLgFirstEpi && lane == 0) phase_mark_here(4);
#pragma unroll 1
            for (int i = 0; (cg + 4 * i) * 16 < cols; ++i) {
                const int c0 = (cg + 4 * i) * 16;
                const long long o0 = (long long)(t0 + c0) * N + n;
                const int live = n_ok ? min(16, M - t0 - c0) : 0;   // (n_ok is uniform over the warp: N is a multiple of 64)
                const uint32_t tmem = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(buf * pp.acc_cols + c0);
                if (wide) {
                    residual_of(i + 1, res_next);
                    SliceAcc acc;
                    load_slice16(tmem, acc);
                    if (fast) store_slice16_matrix<FORM_FACTOR>(p, acc, s_w + 16 * i, r_w + 16 * i, o0 - lane, live, ws_rows, ostage, lane, res);
                    else if (in_range) store_slice16_matrix<FORM_QUOTIENT>(p, acc, s_w + 16 * i, r_w + 16 * i, o0 - lane, live, ws_rows, ostage, lane, res);
                    else store_slice16_matrix<FORM_GENERAL>(p, acc, s_w + 16 * i, r_w + 16 * i, o0 - lane, live, ws_rows, ostage, lane, res);
                    res[0] = res_next[0], res[1] = res_next[1];
                } else {
                    int v[16];
                    tmem_ld16(tmem, v);
                    float sc[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] >>= 6, sc[j] = s_w[16 * i + j];   // (the operand holds 64 * weight)
                    store_slice16(p, v, sc, o0, live, fast, ws_el);
                }
            }
            tc_fence_before();
            __syncwarp();
            // the leader may overwrite this buffer
            if (lane == 0) mbar_arrive_remote(map_to_rank(bar_acc_empty(buf), 0));
            if (ti == 0 && warp == kLgFirstEpi && lane == 0) phase_mark_here(5);
            if (++buf == pp.acc_bufs) buf = 0, ++use;
        }
    }
    phase_mark(6);
    if (*abort_flag && tid == 0) atomicExch(p.status, ST_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    cluster_arrive_relaxed();   // neither CTA frees tensor memory or leaves while the other may still signal it
    cluster_wait();
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
    phase_mark(7);
}

// Tokens per tile of a call and the time it takes, in us: KS stages at the rate of the decoders and barriers (small tiles) or of the
// tensor cores, for each round of tiles over the pairs of the chip, and once what a launch needs around them (fitted with w2_tile_plan;
// 13824 x 2560 at 1226 tokens in tiles of 128 / 160 / 192 / 256: 37.1 / 33.0 / 33.6 / 41.9 us).  Above 192 tokens there is one accumulator buffer,
// and a tile's epilogue holds the next one up.
struct W2PairPlan { int nt; double us; };
inline W2PairPlan w2_pair_plan_tile(int M, int N, int K, int pairs) {
    const int RB = (N + kPairRows - 1) / kPairRows, KS = w2_pairs(K);
    W2PairPlan best = {0, 1e30};
    for (int nt = 96; nt <= 256; nt += 32) {              // (smaller ones never beat single tiles)
        const long long tiles = (long long)RB * ((M + nt - 1) / nt);
        const double rounds = (double)((tiles + pairs - 1) / pairs);
        const double us = 3.34 + 0.0158 * nt + rounds * KS * std::max(0.153 + 0.00017 * nt, 0.00106 * nt) + (rounds - 1) * (nt > 192 ? 4.7 : 0.68);
        if (us < best.us) best = {nt, us};
    }
    return best;
}

}  // namespace tsp
