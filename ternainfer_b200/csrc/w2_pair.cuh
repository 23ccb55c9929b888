// Large batches on two-bit weights for sm_100a: tcgen05 int8 GEMM on CTA pairs whose weight operand is expanded on chip.
//
// The packed format takes a decoder warp 0.12 instructions per weight, so the large-batch path that reads it decodes the
// weight once per call into a dense workspace (dense_prefill.cuh: 8 us for 13824 x 2560, and 16 times the bytes through
// L2 afterwards).  Two-bit codes (w2_small.cuh) expand with 33 instructions per 2048 weights: eight decoder warps keep
// pace with the tensor cores, and neither the extra pass nor the workspace is needed.
//
// A pair (cluster of 2) owns a tile of 256 weight rows x NT tokens (CTA r: rows 128 r .. + 127 and half of the tokens) and walks over
// K in stages of 128 with tcgen05.mma.cta_group::2.  Per CTA 27 warps: warp 0 loads activation tiles by TMA, completing
// on the leader's barrier; warp 1 allocates tensor memory and, in the leader, issues the MMAs; warps 2-17 are the epilogue;
// warps 18-25 the decoders, one per strip of 16 weight rows; warp 26 streams the two-bit weights of four stages at a time
// by cp.async.bulk, 2 KB per strip (the copy engine takes about 60 cycles per bulk copy whatever its size: 512-byte copies, eight
// per stage, were the bound at 700 cycles per stage).  A decoder warp reads 16 bytes per lane, makes four 16-byte stores into
// the 128-byte-swizzled K-major operand, makes them visible to the tensor cores' proxy and arrives on the leader's barrier.
// (That arrival has CTA scope: the stores stay in this CTA's shared memory and are ordered by the proxy fence.  Released
// to the cluster, it cost 1200 cycles per stage at any NT.)  A stage's two operands share a ring slot and ONE commit: the
// issuing thread is on the critical path (a second tcgen05.commit per stage cost 130 cycles of 520).  Up to eight slots, as
// many as shared memory holds at this NT.  Two accumulator buffers of NT columns.  Every wait is bounded (status 4).
//
// NT is chosen per call (w2_pair_tile): a launch lasts as many rounds of tiles over the pairs of the chip as its last pair
// has, so 2048 tokens x 2560 rows are 80 tiles of 256 - two rounds for 74 pairs - but 130 tiles of 160, two
// rounds of five eighths of the length.
#pragma once
#include "dense_pair.cuh"
#include "w2_small.cuh"

namespace tsp {

constexpr int kW2PairDecoders = 8;
constexpr int kW2PairFirstDecoder = kLgFirstEpi + kPairEpiWarps;
constexpr int kW2PairThreads = (kW2PairFirstDecoder + kW2PairDecoders + 1) * 32;
constexpr int kW2OutStride = 80;           // bytes between two tokens of an output slice in shared memory: conflict-free
constexpr int kW2OutStageBytes = 16 * kW2OutStride;
constexpr int kW2PairMaxStages = 8;
constexpr int kW2PairSlots = 2;            // of two-bit weights: 128 rows x 512 k each
constexpr int kW2PairChunk = 4;            // stages per slot
constexpr int kW2PairSlotBytes = kW2PairDecoders * kW2PairChunk * 512;

struct W2PairSmem {
    static constexpr int bar_full = 0;          // [8]  leader: both CTAs' weight rows and activation bytes of a stage are in place
    static constexpr int bar_empty = 64;        // [8]  each CTA: the MMAs have read the stage
    static constexpr int bar_acc_full = 128;    // [2]  each CTA: a tile's accumulators are complete
    static constexpr int bar_acc_empty = 144;   // [2]  leader: both CTAs' epilogues have read the buffer
    static constexpr int bar_w = 160;           // [2]  each CTA: two-bit weights of a slot have landed
    static constexpr int bar_w_free = 176;      // [2]  each CTA: the decoder warps have read the slot
    static constexpr int tmem_slot = 192;
    static constexpr int abort_flag = 196;
    static constexpr int scl = 256;             // float[64] per epilogue warp
    static constexpr int ostage = scl + kPairEpiWarps * 64 * 4;   // 1 KB per epilogue warp (output staging)
    static constexpr int w = (ostage + kPairEpiWarps * kW2OutStageBytes + 1023) / 1024 * 1024;
    static constexpr int stage = w + kW2PairSlots * kW2PairSlotBytes;   // [weights 16 KB][activations NT * 64 bytes] per stage
    static constexpr int total = 227 * 1024;
    static constexpr int stage_bytes = total - 1024 - stage;
};

// arrive on a barrier of any CTA of the cluster, ordering this CTA's accesses only
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// bf16 epilogue of a slice of 16 tokens x 32 weight rows.  The accumulators come as 8x8 matrix fragments (rows = weight rows,
// columns = tokens; a lane has two neighbouring tokens of four rows), so that a lane needs four token scales instead of
// sixteen and stmatrix transposes on the way to shared memory: a third of the instructions of the row-per-lane form
// (store_slice16_wide).  ws_rows: weight scales of rows 8r + lane / 4; `ahead`: the residual as load_residual16 reads it.
__device__ __forceinline__ void store_slice16_matrix(const SpmmParams& p, uint32_t tmem, const float* sc, long long o_row0, int live, bool fast,
                                                     const float (&ws_rows)[4], uint32_t stage, int lane, const uint4 (&ahead)[2]) {
    int v[2][8];                                             // [16 rows][token half x (row half, token)]
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[h][0]), "=r"(v[h][1]), "=r"(v[h][2]), "=r"(v[h][3]), "=r"(v[h][4]), "=r"(v[h][5]), "=r"(v[h][6]), "=r"(v[h][7])
                     : "r"(tmem + ((uint32_t)(16 * h) << 16)));
    const float2 s0 = *reinterpret_cast<const float2*>(sc + 2 * (lane & 3)), s1 = *reinterpret_cast<const float2*>(sc + 8 + 2 * (lane & 3));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    uint32_t m[2][4];                                        // [token half][8 rows]: two tokens
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int a = v[r >> 1][4 * t + 2 * (r & 1)] >> 6, b = v[r >> 1][4 * t + 2 * (r & 1) + 1] >> 6;   // the operand holds 64 * weight
            const float sa = t ? s1.x : s0.x, sb = t ? s1.y : s0.y;
            if (fast) {
                m[t][r] = act_pack(__fmul_rn(__int2float_rn(a), sa), __fmul_rn(__int2float_rn(b), sb));
            } else {
                m[t][r] = (uint32_t)__bfloat16_as_ushort(scale_epilogue(a, sa, ws_rows[r], p.epilogue)) |
                          ((uint32_t)__bfloat16_as_ushort(scale_epilogue(b, sb, ws_rows[r], p.epilogue)) << 16);
            }
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

__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{ .reg .pred q; elect.sync _|q, 0xffffffff; selp.u32 %0, 1, 0, q; }" : "=r"(p));
    return p != 0;
}

// wait_or_abort for the many warps of this kernel: suspended in the barrier (up to 20 us at a time) instead of polling, so
// that sixteen waiting epilogue warps do not take the decoders' issue slots.
__device__ __forceinline__ bool wait_suspended(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_test(bar, parity)) return true;
    const unsigned long long t0 = global_timer_ns();
    for (uint32_t it = 0; it < (1u << 24); ++it) {
        if (mbar_test_suspended(bar, parity, 20000u)) return true;
        if (*abort_flag) return false;
        if (global_timer_ns() - t0 > kLgWaitLimitNs) break;
    }
    *abort_flag = 1;
    return false;
}

struct W2PairParams {
    SpmmParams e;
    const uint8_t* w;                      // two-bit weights
    int nt, stages;                        // tokens per tile: a multiple of 32, at most 256; ring slots
};

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
    const uint32_t stage_bytes = kPairHalf + x_bytes, stage0 = sbase + L::stage;
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
            mbar_init(bar_full(s), 1 + 2 * kW2PairDecoders);   // the leader's loader thread (+ the TMA bytes of both CTAs), the decoder warps
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
    bool ok = true;
    phase_mark(1);

    if (warp == 0) {
        // ------------------------------------------------ activation loader (both CTAs)
        if (lane == 0) {
            griddep_wait();   // the activations come from earlier kernels of the stream
            phase_mark(2);
            int s = 0, it = 0;
            for (int ti = 0; ti < my_tiles && ok; ++ti) {
                const int t0 = ((pair + ti * npairs) / RB) * NT + (int)crank * (NT / 2);   // this CTA's tokens
                for (int ks = 0; ks < KS; ++ks) {
                    if (it > 0) ok = wait_suspended(bar_empty(s), (it - 1) & 1, abort_flag);
                    if (!ok) break;
                    if (crank == 0) mbar_arrive_expect_tx(bar_full(s), 2 * x_bytes);
                    tma_load_2d_pair(stage0 + s * stage_bytes + kPairHalf, &tmap_x, ks * kLgKStep, t0, map_to_rank(bar_full(s), 0));
                    if (++s == ST) s = 0, ++it;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------ MMA issuer (leader only): the warp runs the loop together, so
        // that addresses stay in uniform registers, and one elected lane issues
        if (crank == 0) {
            // int8 x int8 -> int32, K-major A and B, M = 256 over the pair, N = NT
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kPairRows >> 4) << 24);
            const bool elected = elect_one();
            const uint64_t a_desc0 = umma_desc_sw128(stage0), x_desc0 = umma_desc_sw128(stage0 + kPairHalf);
            int s = 0, it = 0;
            for (int ti = 0; ti < my_tiles; ++ti) {
                const int buf = ti & 1, use = ti >> 1;
                if (use > 0) {   // both CTAs' epilogues must have drained this accumulator buffer
                    ok = __all_sync(0xffffffffu, wait_suspended(bar_acc_empty(buf), (use - 1) & 1, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                }
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * 256);
                for (int ks = 0; ks < KS; ++ks) {
                    ok = __all_sync(0xffffffffu, wait_suspended(bar_full(s), it & 1, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                    if (ti == 0 && ks == 0 && lane == 0) phase_mark_here(3);
                    const uint32_t off = (uint32_t)s * (stage_bytes >> 4);   // descriptor addresses count 16 bytes
                    if (elected) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)   // four K=32 slices inside the 128-byte swizzle row
                            umma_i8_pair(d_tmem, a_desc0 + off + 2 * j, x_desc0 + off + 2 * j, idesc, (ks | j) != 0);
                        umma_commit_pair(bar_empty(s));     // frees the stage in both CTAs
                        if (ks == KS - 1) umma_commit_pair(bar_acc_full(buf));   // this tile's accumulators are complete in both CTAs
                    }
                    __syncwarp();
                    if (++s == ST) s = 0, ++it;
                }
                if (!ok) break;
            }
        }
    } else if (warp == kW2PairFirstDecoder + kW2PairDecoders) {
        // ---------------------------------------------------------- two-bit weights (both CTAs, own 128 rows; immutable: no dependency wait)
        int s = 0, it = 0;
        for (int ti = 0; ti < my_tiles && ok; ++ti) {
            const int strip0 = ((pair + ti * npairs) % RB) * (kPairRows / 16) + (int)crank * 8;
            const int live = max(0, min(kW2PairDecoders, (N >> 4) - strip0));   // strips of a last, smaller row block
            const uint8_t* src = pp.w + (size_t)(strip0 + lane) * KS * 512;
            for (int ks = 0; ks < KS; ks += kW2PairChunk) {
                if (it > 0) ok = wait_suspended(bar_w_free(s), (it - 1) & 1, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
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
        const int strip_in = warp - kW2PairFirstDecoder, g = lane >> 2, q = lane & 3;
        // row 16 strip + g (and + 8), 16-byte chunk (4 block + q) ^ g; lanes of odd g store block 1 first: no bank conflict
        const uint32_t a_row = stage0 + (uint32_t)((16 * strip_in + g) * 128);
        const uint32_t first = a_row + (((uint32_t)(4 * (g & 1) + q) ^ (uint32_t)g) << 4);
        const uint32_t second = a_row + (((uint32_t)(4 * ((g & 1) ^ 1) + q) ^ (uint32_t)g) << 4);
        const uint32_t w_lane = sbase + L::w + (uint32_t)(strip_in * (kW2PairChunk * 512) + lane * 16);
        const bool odd = g & 1;
        const uint32_t full0 = map_to_rank(bar_full(0), 0);   // the leader's
        int s = 0, it = 0, ws = 0, wit = 0;
        for (int ti = 0; ti < my_tiles && ok; ++ti) {
            const bool live = ((pair + ti * npairs) % RB) * (kPairRows / 16) + (int)crank * 8 + strip_in < (N >> 4);
#pragma unroll 1
            for (int ks = 0; ks < KS; ks += 2) {         // two stages per turn: one fence, and the latencies overlap
                const int in_slot = ks & (kW2PairChunk - 1);
                const bool two = ks + 1 < KS;
                if (in_slot == 0) {
                    ok = wait_suspended(bar_w(ws), wit & 1, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                uint4 w[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
                if (live) {
                    w[0] = lds128(w_lane + ws * kW2PairSlotBytes + in_slot * 512);
                    if (two) w[1] = lds128(w_lane + ws * kW2PairSlotBytes + in_slot * 512 + 512);
                }
                const int s0 = s, s1 = s + 1 == ST ? 0 : s + 1, it1 = it + (s + 1 == ST);
                if (it > 0) ok = wait_suspended(bar_empty(s0), (it - 1) & 1, abort_flag);
                if (two && it1 > 0) ok = ok && wait_suspended(bar_empty(s1), (it1 - 1) & 1, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (u == 1 && !two) break;
                    const uint4 v = odd ? make_uint4(w[u].z, w[u].w, w[u].x, w[u].y) : w[u];
                    uint32_t a[4], b[4];
                    const uint32_t off = (uint32_t)(u ? s1 : s0) * stage_bytes;
                    w2_decode(v.x, a), w2_decode(v.y, b);
                    sts128(first + off, make_uint4(a[0], a[2], b[0], b[2]));
                    sts128(first + off + 8 * 128, make_uint4(a[1], a[3], b[1], b[3]));
                    w2_decode(v.z, a), w2_decode(v.w, b);
                    sts128(second + off, make_uint4(a[0], a[2], b[0], b[2]));
                    sts128(second + off + 8 * 128, make_uint4(a[1], a[3], b[1], b[3]));
                }
                fence_proxy_async_smem();        // generic-proxy stores -> visible to the tensor cores' async proxy
                __syncwarp();
                const bool slot_done = in_slot == kW2PairChunk - 2 || ks + 2 >= KS;
                if (lane == 0) {
                    mbar_arrive_remote(full0 + 8 * s0);
                    if (two) mbar_arrive_remote(full0 + 8 * s1);
                    if (slot_done) mbar_arrive(bar_w_free(ws));
                }
                if (++s == ST) s = 0, ++it;
                if (two && ++s == ST) s = 0, ++it;
                if (slot_done && ++ws == WS) ws = 0, ++wit;
            }
        }
    } else {
        // ---------------------------------------------------------- epilogue (both CTAs, own 128 weight rows)
        griddep_wait();  // scales, residual and the output buffer may belong to the previous kernel
        const int quarter = warp & 3;          // the tensor-memory lanes a warp may read: 32 * (warp % 4)
        const int cg = (warp - kLgFirstEpi) >> 2;   // this warp's slices of 16 tokens: cg, cg + 4, ...
        float* s_w = s_s + (warp - kLgFirstEpi) * 64;
        const uint32_t ostage = sbase + L::ostage + (uint32_t)((warp - kLgFirstEpi) * kW2OutStageBytes);
        const bool wide = ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual)) & 15) == 0;
        for (int ti = 0; ti < my_tiles; ++ti) {
            const int tile = pair + ti * npairs;
            const int rb = tile % RB, t0 = (tile / RB) * NT;
            const int buf = ti & 1, use = ti >> 1;
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
            for (int i = lane; i < 64; i += 32) {  // token of local slot i: slice cg + 4 (i / 16)
                const int c = (cg + 4 * (i >> 4)) * 16 + (i & 15);
                const float sv = (c < NT && t0 + c < M) ? __bfloat162float(p.s[t0 + c]) : 1.f;
                s_w[i] = fast ? ((sv != 0.f) ? __fdiv_rn(ws0, sv) : 0.f) : sv;
            }
            __syncwarp();
            const int cols = min(NT, M - t0);
            uint4 res[2], res_next[2];          // the residual is read one slice ahead
            auto residual_of = [&](int i, uint4 (&r)[2]) {
                const int c0 = (cg + 4 * i) * 16;
                if (wide && p.residual && c0 < cols)
                    load_residual16(p, (long long)(t0 + c0) * N + n - lane, n_ok ? min(16, M - t0 - c0) : 0, lane, r);
            };
            residual_of(0, res);
            if (ok) ok = wait_suspended(bar_acc_full(buf), use & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);   // the tensor-memory loads below are warp-collective
            if (!ok) break;
            tc_fence_after();
            if (ti == 0 && warp == kLgFirstEpi && lane == 0) phase_mark_here(4);
#pragma unroll 1
            for (int i = 0; (cg + 4 * i) * 16 < cols; ++i) {
                const int c0 = (cg + 4 * i) * 16;
                const long long o0 = (long long)(t0 + c0) * N + n;
                const int live = n_ok ? min(16, M - t0 - c0) : 0;   // (n_ok is uniform over the warp: N is a multiple of 64)
                const uint32_t tmem = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(buf * 256 + c0);
                if (wide) {
                    residual_of(i + 1, res_next);
                    store_slice16_matrix(p, tmem, s_w + 16 * i, o0 - lane, live, fast, ws_rows, ostage, lane, res);
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
            // the leader may overwrite this buffer (CTA scope: a cluster release would wait for the output stores)
            if (lane == 0) mbar_arrive_remote(map_to_rank(bar_acc_empty(buf), 0));
            if (ti == 0 && warp == kLgFirstEpi && lane == 0) phase_mark_here(5);
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

// Tokens per tile for M tokens, RB row blocks, KS stages and `pairs` resident pairs: the shortest time of the busiest pair.
// Fitted to launches of 20 and 54 stages at 160, 192 and 256 tokens: a tile takes KS * (200 + 0.47 NT) + 20 NT ns (stage
// overheads, tensor cores, epilogue).  Measured since over 32 .. 256 tokens per tile (us per call, chosen / best): within 3 % for
// 13824 x 2560 from 48 to 512 tokens, and for the narrower layers up to 64 and from 256 on (2560 x 2560 at 512 10.3 / 9.9 is the
// widest); in between, one round of many small tiles is dearer than it says: 3840 x 2560 at 128 tokens 9.2 / 7.8
// (30 tiles of 64 instead of 60 of 32), 2560 x 2560 at 192 9.2 / 7.9, 4096 x 4096 at 128 12.5 / 10.5.
inline int w2_pair_tile(int M, int RB, int KS, int pairs) {
    int best = 32;
    double best_cost = 1e30;
    for (int nt = 32; nt <= 256; nt += 32) {
        const long long tiles = (long long)RB * ((M + nt - 1) / nt);
        const double cost = (double)((tiles + pairs - 1) / pairs) * (KS * (200.0 + 0.47 * nt) + 20.0 * nt);
        if (cost < best_cost) best = nt, best_cost = cost;
    }
    return best;
}

}  // namespace tsp
