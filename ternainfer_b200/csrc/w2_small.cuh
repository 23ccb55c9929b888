// Ternary linears on weights laid out once in two bits, for sm_100a: up to eight
// tokens with the activation front-end (RMSNorm, gate, int8 quantiser) inside the
// kernel; on int8 activations up to four, and up to eight for narrow layers (the others
// and more tokens: w2_tile.cuh, w2_pair.cuh).
//
// The packed checkpoint format (bitmap + sign stream) costs about 0.12 warp
// instructions per weight to decode, and that, not HBM, is what bounds the
// kernels that read it (spmm_small_m.cuh, spmm_list.cuh).  A module that keeps its
// weights for the life of a model can pay for that once: relayout_w2_kernel
// rewrites them as fixed-rate two-bit codes, which decode with one AND and at most one
// shift per four weights.
//
// Layout.  Strips of 16 weight rows; inside a strip, pairs of 64-column blocks, 512 bytes each: the 16 bytes at
// w2_chunk(g, q) are four words, row g in block 0, row g in block 1, row g + 8 in block 0, row g + 8 in block 1.  A word
// covers the columns 16q .. 16q + 15 of its block; byte e of it holds, from the top bits down, the codes of columns e, 4 + e, 8 + e and
// 12 + e.  Code = the weight in two's complement.  Where K is an odd multiple of 64 the second block of the last pair is zero.  A
// strip is ceil(K / 128) * 512 contiguous bytes, so any range of block pairs of a strip is one bulk copy.  Masking a shifted
// word with 0xC0C0C0C0 leaves 64 * weight in every signed byte, four neighbouring columns of a row: the A operand of an int8 MMA,
// as a lane of mma.sync holds it (lane 4g + q) and as a lane of tensor memory does (w2_tile.cuh: a lane per row).  The accumulators come
// out as 64 times the result and are shifted back exactly (|acc| < 2^31 for K < 2^18).
//
// Work split.  A CTA owns R strips and all of K; its
// warps split K.  Each warp streams its own part of the CTA's strips through its
// own ring of shared-memory slots by cp.async.bulk, so the weights of BitNet-2B-sized
// layers (10 - 60 KB per SM) are on chip before the programmatic-dependency wait
// returns, and several launches of a stream prefetch at the same time (a CTA takes
// what it needs of shared memory and at most half of the register file).
// After the wait a call is one chain of latencies: read the activations, norm and quantise
// them, MMAs, one reduction over the warps, store.  Hence the front-end in the kernel
// for the smallest calls: every CTA repeats it (a few microseconds of one row's
// arithmetic would cost more as a launch of its own than as redundant work).  At one token the
// chain of 3840 x 2560 is 5000 cycles: activations 460, norm and quantiser 2000, MMAs 1800, reduction and epilogue 750.  Partial
// sums go to a set per warp instead of shared atomics and quotients need no division where the scale allows it (us per call, before
// and now: 3840 x 2560 with the norm 3.5 / 3.3, 2560 x 6912 gated 5.5 / 5.1, quantiser and 4 rows 4.7 / 3.2, 8192 x 8192 at 4 rows 7.8 / 6.7).
// Measured and no better: the expansion without shifts into unsigned fields, a dry run of the code ahead of the dependency wait,
// twenty warps for K = 2560.
#pragma once
#include <cuda_bf16.h>

#include <algorithm>

#include "act_quant.cuh"
#include "spmm_small_m.cuh"

namespace tsp {

constexpr int kW2Warps = 10, kW2MaxWarps = 20;   // of a CTA that shares its SM with the next launch's, and of one that does not
constexpr uint32_t kW2Mask = 0xC0C0C0C0u;

struct W2Smem {   // shared-memory plan: byte offsets from the base of the dynamic segment
    int red, xq, res, ring, total;
    int red_stride, x_stride;
    int red_sets;     // partial sums: a set per warp, or one that the warps add to
};

struct W2Params {
    SpmmParams e;                     // shapes, scales, output and epilogue (its weight pointers are not used)
    const uint8_t* w;                 // two-bit weights, 16-byte aligned
    const __nv_bfloat16* xb;          // fused front-ends: bf16 activations [M][K] or [M][2K] (gated)
    const __nv_bfloat16* norm_w;      // norm weight [K]
    float eps;
    int strips_q, strips_r;           // CTA b owns strips_q strips, one more when b < strips_r
    int pairs_q, pairs_r;             // the same for the block pairs of K and the warps of a CTA
    int slots, chunk_pairs;           // ring slots per warp, block pairs per slot
    W2Smem smem;
};

// Warps of a CTA: as many as have a block pair of their own, at most ten (two CTAs of that size share the register file, so the
// next launch's CTA starts beside this one), evenly loaded; at least four for the front-end and the epilogue.  Up to twenty where a
// launch is long.
inline int w2_warps(int K, int most = kW2Warps) {
    const int KP = (K + 127) >> 7, per = (KP + most - 1) / most;
    return std::max(4, (KP + per - 1) / per);
}

// Front-end inside the kernel: none (int8 activations and scales given), the plain quantiser, RMSNorm + quantiser,
// gate + RMSNorm + quantiser.
enum W2FrontEnd : int { W2_INT8 = 0, W2_PLAIN = 1, W2_NORM = 2, W2_GATED = 3 };

// Byte offset of the chunk of rows g, g + 8 and columns 16q .. of both blocks.  The order of the chunks turns with the row, so that
// sixteen lanes with a row each and the same q (w2_tile.cuh) meet no bank twice either.
__device__ __forceinline__ int w2_chunk(int g, int q) { return g * 64 + ((q ^ (g >> 1)) << 4); }
__host__ __device__ inline int w2_pairs(int K) { return (K + 127) >> 7; }

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
                 : "memory");
}

// Wait for a phase of an mbarrier that this CTA's own copies complete, at most two seconds.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (uint32_t it = 0; it < (1u << 28); ++it) {
        if (mbar_test(bar, parity)) return true;
        if ((it & 255u) == 255u) {
            const unsigned long long now = global_timer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > 2000ull * 1000 * 1000) break;
        }
    }
    return false;
}

// Sixteen columns of a row -> four words of four columns each, 64 * weight per signed byte.
__device__ __forceinline__ void w2_decode(uint32_t w, uint32_t (&a)[4]) {
    a[0] = w & kW2Mask;
    a[1] = (w << 2) & kW2Mask;
    a[2] = (w << 4) & kW2Mask;
    a[3] = (w << 6) & kW2Mask;
}

// ---- packed format -> two-bit layout, once per weight: one warp per 64x64 tile -----------------------
__global__ void __launch_bounds__(256) relayout_w2_kernel(const SpmmParams p, uint8_t* __restrict__ w2) {
    const int lane = threadIdx.x & 31;
    const int KT = p.K >> 6;
    const long long tile = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tile >= (long long)(p.N >> 6) * KT) return;
    const TileHead h = load_head(p, tile, true, lane);
    const TileSigns sg = load_signs(p, h, true, lane);
    const uint32_t bm[4] = {h.bw.x, h.bw.y, h.bw.z, h.bw.w};
    const int rt = (int)(tile / KT), kt = (int)(tile - (long long)rt * KT);
    const int KP = w2_pairs(p.K);
    int pos = sg.pos;
#pragma unroll
    for (int r = 0; r < 4; ++r) {      // word r of the tile = rows 16r .. 16r+15 = one strip
        uint32_t sgn = __funnelshift_r(sg.lo[r], sg.hi[r], (uint32_t)pos), out[2] = {0u, 0u};
        pos += __popc(bm[r]);
#pragma unroll
        for (int b = 0; b < 32; ++b) { // nibble b/4 = 4 * step + field, element b%4 = byte
            if ((bm[r] >> b) & 1u) {       // (fields of a step: row g, row g + 8, the same four columns on)
                out[(b >> 2) & 1] |= (1u | ((sgn & 1u) << 1)) << (8 * (b & 3) + 6 - 2 * (2 * (b >> 4) + ((b >> 3) & 1)));
                sgn >>= 1;
            }
        }
        uint8_t* dst = w2 + (((size_t)rt * 4 + r) * KP + (kt >> 1)) * 512 + w2_chunk(lane >> 2, lane & 3) + (kt & 1) * 4;
        reinterpret_cast<uint32_t*>(dst)[0] = out[0], reinterpret_cast<uint32_t*>(dst)[2] = out[1];
        if (kt == KT - 1 && (KT & 1)) reinterpret_cast<uint32_t*>(dst)[1] = reinterpret_cast<uint32_t*>(dst)[3] = 0u;
    }
}

constexpr int kW2MaxSlots = 8;                       // ring slots per warp
constexpr int kW2MaxRows = 8;                        // tokens per call of this kernel (the columns of an MMA)
constexpr int kW2Scale = kW2MaxWarps * kW2MaxSlots * 8;           // behind the mbarriers: float s[32], quotient_rcp(s)[32], ws[4]
constexpr int kW2Partial = kW2Scale + 80 * 4;                     // of the front-ends: 8 x 32 partial sums, 8 x 32 maxima, 8 factors
constexpr int kW2ScratchBytes = kW2Partial + (2 * kW2MaxRows * 32 + kW2MaxRows) * 4;

// R strips per CTA at most, `tokens` rows of x, W warps, ring slots of `slot_bytes`
inline W2Smem w2_smem(int R, int tokens, int K, int W, int slots, int slot_bytes, bool residual) {
    W2Smem s;
    s.red_stride = R * 16 + 4;                       // conflict-free: token stride = 4 mod 16 words
    s.x_stride = (K & 127) ? K : K + 64;             // two tokens' 64-byte pieces on different banks
    s.red_sets = W * tokens * s.red_stride * 4 <= 16 * 1024 ? W : 1;
    int at = (kW2ScratchBytes + 127) & ~127;
    s.red = at;
    at += s.red_sets * tokens * s.red_stride * 4;
    at = (at + 127) & ~127;
    s.xq = at;
    at += ((tokens * s.x_stride + 64 + 127) & ~127);   // (a half pair reads 64 bytes past its row)
    s.res = at;                                      // residual of the CTA's outputs, bf16 [tokens][R * 16]
    if (residual) at += ((tokens * R * 32 + 127) & ~127);
    s.ring = at;
    at += W * slots * slot_bytes;
    s.total = at;
    return s;
}

// Four MMAs of a block pair of a strip: rows g, g + 8 of the strip by the tokens.
__device__ __forceinline__ void w2_mma_pair(int (&acc0)[4], int (&acc1)[4], const uint4& w, const uint4& x0, const uint4& x1) {
    uint32_t a[4], c[4];
    w2_decode(w.x, a), w2_decode(w.z, c);
    mma_s8_16x8x32(acc0, a[0], c[0], a[1], c[1], x0.x, x0.y);
    mma_s8_16x8x32(acc0, a[2], c[2], a[3], c[3], x0.z, x0.w);
    w2_decode(w.y, a), w2_decode(w.w, c);
    mma_s8_16x8x32(acc1, a[0], c[0], a[1], c[1], x1.x, x1.y);
    mma_s8_16x8x32(acc1, a[2], c[2], a[3], c[3], x1.z, x1.w);
}

// MW: warps at most.  RG: strips at a time, one or three (ternaspmm.cu has both rules).  VK, VR: vectors of a row per thread and rows at a time in
// the front-end.
template <int MW, int RG, int FE, int VK, int VR>
__global__ void __launch_bounds__(MW * 32, MW > kW2Warps ? 1 : 2) w2_small_kernel(const __grid_constant__ W2Params p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthreads = blockDim.x;
    const int g = lane >> 2, q = lane & 3;
    const int K = p.e.K, N = p.e.N, D = p.slots;
    const int mrows = p.e.M;
    const int b = blockIdx.x, strip0 = b * p.strips_q + min(b, p.strips_r), nstrips = p.strips_q + (b < p.strips_r);
    const int KP = w2_pairs(K), PC = p.chunk_pairs;           // block pairs of K, at most PC per ring slot
    const int p0 = warp * p.pairs_q + min(warp, p.pairs_r), p1 = p0 + p.pairs_q + (warp < p.pairs_r);
    const int slot_bytes = RG * PC * 512;
    const int NG = (nstrips + RG - 1) / RG;                   // groups of RG strips
    const W2Smem& L = p.smem;
    const uint32_t base = smem_u32(smem);
    int* red = reinterpret_cast<int*>(smem + L.red);
    float* scl = reinterpret_cast<float*>(smem + kW2Scale);
    const uint32_t bars = base + warp * (kW2MaxSlots * 8), ring = base + L.ring + warp * D * slot_bytes;
    const int red_stride = L.red_stride, red_sets = L.red_sets;

    phase_mark(0);
    griddep_launch_dependents();
    // ---- weights: complete before any kernel that this one may overtake began (ternaspmm_w2_relayout sees to it), so the ring
    // fills - and is waited for - before the dependency wait
    int f_gi = 0, f_c = p0, f_d = 0;                          // lane 0: the next chunk to fetch and its slot
    auto fetch = [&]() {
        const int c1 = min(f_c + PC, p1), nr = min(RG, nstrips - f_gi * RG);
        const uint32_t bytes = (uint32_t)(c1 - f_c) * 512;
        mbar_arrive_expect_tx(bars + 8 * f_d, bytes * nr);
        const uint8_t* src = p.w + ((size_t)(strip0 + f_gi * RG) * KP + f_c) * 512;
        for (int r = 0; r < nr; ++r)
            bulk_load(ring + f_d * slot_bytes + r * PC * 512, src + (size_t)r * KP * 512, bytes, bars + 8 * f_d);
        f_c = c1;
        if (f_c == p1) f_c = p0, ++f_gi;
        if (++f_d == D) f_d = 0;
    };
    if (lane == 0 && p0 < p1) {
        for (int d = 0; d < D; ++d) mbar_init(bars + 8 * d, 1);
        mbar_fence_init();
        for (int i = 0; i < D && f_gi < NG; ++i) fetch();
    }
    if (red_sets == 1 || p0 >= p1)                            // (a warp without a share of K leaves zeros)
        for (int i = red_sets == 1 ? tid : lane; i < mrows * red_stride; i += red_sets == 1 ? nthreads : 32)
            red[(red_sets == 1 ? 0 : warp * mrows * red_stride) + i] = 0;
    constexpr bool kGated = FE == W2_GATED;
    if ((FE == W2_NORM || FE == W2_GATED) && tid == 64 && b == 0) act_weight_ahead(p.norm_w, K);
    const int pairs = nstrips * 8, items = mrows * pairs;     // epilogue items: two columns of a token each
    const uint32_t inv_pairs = ((1u << 22) + pairs - 1) / pairs;   // i / pairs = i * inv >> 22 (i * pairs < 2^22)
    const bool res_smem = p.e.residual != nullptr && (reinterpret_cast<uintptr_t>(p.e.residual) & 15) == 0;
    const bool out_ok = (reinterpret_cast<uintptr_t>(p.e.out) & 3) == 0;

    __syncwarp();
    bool ok = true;
    if (p0 < p1)
        for (int d = 0; d < min(D, (p1 - p0 + PC - 1) / PC * NG); ++d) ok = ok && mbar_wait_bounded(bars + 8 * d, 0);
    phase_mark(1);
    griddep_wait();
    phase_mark(2);
    // ---- activations, scales, residual: everything is asked for before anything is waited for
    if (FE == W2_INT8) {                                // this warp's columns of the rows, 16 bytes a piece
        const int pieces = (min(p1 * 128, K) - p0 * 128) >> 4;
        for (int t = lane >> 4; t < mrows; t += 2)
            for (int i = lane & 15; i < pieces; i += 16)
                cp_async_16(base + L.xq + t * L.x_stride + p0 * 128 + i * 16, p.e.x + (size_t)t * K + p0 * 128 + i * 16);
    }
    if (res_smem) {
#pragma unroll 1
        for (int i = tid; i < mrows * nstrips * 2; i += nthreads) {   // 16 bytes a piece
            const int t = (int)((uint32_t)(i * 4) * inv_pairs >> 22), c = i * 4 - t * pairs;
            cp_async_16(base + L.res + (t * pairs + c) * 4, p.e.residual + (size_t)t * N + strip0 * 16 + c * 2);
        }
    }
    cp_async_commit();
    if (FE == W2_INT8 && tid < mrows) {
        const float s = __bfloat162float(p.e.s[tid]);
        scl[tid] = s, scl[32 + tid] = quotient_rcp(s);
    }
    if (tid >= 32 && tid < 36) scl[32 + tid] = __bfloat162float(p.e.ws[tid - 32]);
    const uint32_t x_lane = base + L.xq + min(g, mrows - 1) * L.x_stride + q * 16;   // (columns of absent tokens are not stored)
    if (FE == W2_INT8) {
        cp_async_wait_all();                                  // (the residual too)
        __syncwarp();                                         // (a warp reads the columns that it copied)
        if (red_sets == 1) __syncthreads();                   // red is zeroed
    } else {
        constexpr int kMode = FE == W2_PLAIN ? ACT_PLAIN : ACT_RMSNORM;
        float* part = reinterpret_cast<float*>(smem + kW2Partial);
        uint32_t* mxp = reinterpret_cast<uint32_t*>(part + kW2MaxRows * 32);
        float* rstd = reinterpret_cast<float*>(mxp + kW2MaxRows * 32);
#pragma unroll 1
        for (int t = 0; t < mrows; t += VR) {
            const uint32_t xrow = base + L.xq + t * L.x_stride;
            act_rows<kGated, kMode, VK, VR>(p.xb + (size_t)t * (kGated ? 2 * K : K), p.norm_w, p.eps, K, min(VR, mrows - t), part,
                                            mxp + (VR == 1 ? (t & 1) * 32 : 0), rstd, scl + t,
                                            [&](int r, int k0, const uint2& v) { sts64(xrow + r * L.x_stride + k0, v.x, v.y); });
        }
        __syncthreads();
    }

    phase_mark(3);
    int d = 0;
    uint32_t parity = 0;
    bool refilled = false;                                    // the slots of the first round have been waited for
    int* dst = red + (red_sets == 1 ? 0 : warp * mrows * red_stride) + 2 * q * red_stride + g;
    const bool t0_ok = 2 * q < mrows, t1_ok = 2 * q + 1 < mrows;
    const uint32_t w_lane = ring + w2_chunk(g, q);
    auto put = [&](const int (&a)[4], const int (&b)[4]) {    // (rows of absent tokens are not stored)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            int* at = dst + (c & 1) * red_stride + 8 * (c >> 1);
            if ((c & 1) ? t1_ok : t0_ok) {
                if (red_sets == 1) atomicAdd(at, a[c] + b[c]);
                else *at = a[c] + b[c];
            }
        }
        dst += 16;
    };
    auto next_slot = [&]() {                                  // after the last read of a slot: refill it, go on to the next
        __syncwarp();
        if (lane == 0 && f_gi < NG) fetch();
        if (++d == D) d = 0, parity ^= 1u, refilled = true;
    };
    const uint4 none = make_uint4(0, 0, 0, 0);
    // What a turn of a loop costs is its warps' chains and, the first time, its fetch (some 35 cycles for eight instructions).  One strip at a
    // time: at once where a warp's share of K is one or two block pairs, whose activations stay in registers, else a block pair per
    // turn (the next one's operands asked for ahead of it: 3 to 8 % slower; two per turn with accumulators of their own: no gain).  Three at a
    // time: two block pairs per turn.  (us per call, three / one at a time: 2560 x 2560 with the norm 3.3 / 3.1, 13824 x 2560 at 4 tokens
    // 4.3 / 4.5, 57344 x 8192 at 4 32.6 / 34.2.)
    if (RG == 1 && p1 - p0 <= 2 && p1 - p0 <= PC && p0 < p1) {
        const bool two = p1 - p0 == 2;
        const uint4 x0 = lds128(x_lane + p0 * 128), x1 = lds128(x_lane + p0 * 128 + 64);
        const uint4 x2 = two ? lds128(x_lane + p0 * 128 + 128) : none, x3 = two ? lds128(x_lane + p0 * 128 + 192) : none;
        const uint32_t second = two ? 512 : 0;
        uint4 w0 = lds128(w_lane), w1 = lds128(w_lane + second);
#pragma unroll 1
        for (int st = 0; st < nstrips; ++st) {
            next_slot();
            if (refilled && st + 1 < nstrips) ok = ok && mbar_wait_bounded(bars + 8 * d, parity);
            const uint4 n0 = lds128(w_lane + d * slot_bytes), n1 = lds128(w_lane + d * slot_bytes + second);
            int acc[4][4] = {};
            w2_mma_pair(acc[0], acc[1], w0, x0, x1);
            w2_mma_pair(acc[2], acc[3], w1, x2, x3);
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[0][c] += acc[2][c], acc[1][c] += acc[3][c];
            put(acc[0], acc[1]);
            w0 = n0, w1 = n1;
        }
    } else if (RG == 1) {
#pragma unroll 1
        for (int st = 0; st < nstrips && p0 < p1; ++st) {
            int acc[2][4] = {};
#pragma unroll 1
            for (int c0 = p0; c0 < p1; c0 += PC) {
                if (refilled) ok = ok && mbar_wait_bounded(bars + 8 * d, parity);
                uint32_t slot = w_lane + d * slot_bytes, xa = x_lane + c0 * 128;
                const uint32_t end = xa + min(PC, p1 - c0) * 128;
#pragma unroll 1
                for (; xa < end; slot += 512, xa += 128) w2_mma_pair(acc[0], acc[1], lds128(slot), lds128(xa), lds128(xa + 64));
                next_slot();
            }
            put(acc[0], acc[1]);
        }
    } else {
        // (a group's absent strips are computed from whatever the ring holds, an absent second pair from zeros, and neither is stored)
#pragma unroll 1
        for (int gi = 0; gi < NG && p0 < p1; ++gi) {
            int acc[RG][4] = {};
#pragma unroll 1
            for (int c0 = p0; c0 < p1; c0 += PC) {
                if (refilled) ok = ok && mbar_wait_bounded(bars + 8 * d, parity);
                const uint32_t slot = w_lane + d * slot_bytes;
                const int c1 = min(c0 + PC, p1);
#pragma unroll 1
                for (int pr = c0; pr < c1; pr += 2) {
                    uint4 x[2][2], w[2][RG];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int pu = u == 0 ? pr : min(pr + 1, c1 - 1);
                        x[u][0] = lds128(x_lane + pu * 128), x[u][1] = lds128(x_lane + pu * 128 + 64);
#pragma unroll
                        for (int r = 0; r < RG; ++r) w[u][r] = lds128(slot + (pu - c0) * 512 + r * PC * 512);
                        if (u > 0 && pr + 1 >= c1) x[u][0] = x[u][1] = none;
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int r = 0; r < RG; ++r) w2_mma_pair(acc[r], acc[r], w[u][r], x[u][0], x[u][1]);
                }
                next_slot();
            }
            const int nothing[4] = {};
#pragma unroll
            for (int r = 0; r < RG; ++r) {
                if (gi * RG + r >= nstrips) break;
                put(acc[r], nothing);
            }
        }
    }
    if (!ok) atomicExch(p.e.status, ST_WAIT_TIMEOUT);
    cp_async_wait_all();                                      // the residual
    phase_mark(5);
    __syncthreads();
    phase_mark(6);

    // ---- epilogue (one loop body: code that runs once is paid for in instruction fetches)
#pragma unroll 1
    for (int i = tid; i < items; i += nthreads) {
        const int t = (int)((uint32_t)i * inv_pairs >> 22), c = (i - t * pairs) * 2, n = strip0 * 16 + c;
        const int* src = red + t * red_stride + c;
        int2 v = make_int2(0, 0);
#pragma unroll 5
        for (int k = 0; k < red_sets; ++k) {
            const int2 o = *reinterpret_cast<const int2*>(src + k * mrows * red_stride);
            v.x += o.x, v.y += o.y;
        }
        v.x >>= 6, v.y >>= 6;
        const size_t o = (size_t)t * N + n;
        const float s = scl[t], rc = scl[32 + t], ws0 = scl[64 + ws_group(n, p.e)], ws1 = scl[64 + ws_group(n + 1, p.e)];
        __nv_bfloat16 r[2];
        if (p.e.epilogue == EPI_DECODE && rc != 0.f) {
            r[0] = __float2bfloat16_rn(__fmul_rn(quotient(__int2float_rn(v.x), s, rc), ws0));
            r[1] = __float2bfloat16_rn(__fmul_rn(quotient(__int2float_rn(v.y), s, rc), ws1));
        } else {
            r[0] = scale_epilogue(v.x, s, ws0, p.e.epilogue), r[1] = scale_epilogue(v.y, s, ws1, p.e.epilogue);
        }
        if (res_smem) {
            const uint32_t rv = lds32(base + L.res + i * 4);
            r[0] = __float2bfloat16_rn(act_lo(rv) + __bfloat162float(r[0])), r[1] = __float2bfloat16_rn(act_hi(rv) + __bfloat162float(r[1]));
        } else if (p.e.residual) {
            r[0] = add_residual(r[0], p.e.residual, (long long)o), r[1] = add_residual(r[1], p.e.residual, (long long)o + 1);
        }
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.e.out) + o;
        if (out_ok) stg_b32(out, (uint32_t)__bfloat16_as_ushort(r[0]) | ((uint32_t)__bfloat16_as_ushort(r[1]) << 16));
        else out[0] = r[0], out[1] = r[1];
    }
    phase_mark(7);
}

}  // namespace tsp
