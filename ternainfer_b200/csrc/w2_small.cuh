// Ternary linears on weights laid out once in two bits, for sm_100a: up to a few
// dozen tokens per pass, with the activation front-end (RMSNorm, gate, int8
// quantiser) optionally inside the kernel.
//
// The packed checkpoint format (bitmap + sign stream) costs about 0.12 warp
// instructions per weight to decode, and that, not HBM, is what bounds the
// kernels that read it (spmm_small_m.cuh, spmm_list.cuh).  A module that keeps its
// weights for the life of a model can pay for that once: relayout_w2_kernel
// rewrites them as fixed-rate two-bit codes in the order of the int8 MMA's A
// fragments, which decode with one AND and at most one shift per four weights.
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
// Work split.  A CTA owns R strips for a block of MT*8 tokens and all of K; its
// warps split K.  Each warp streams its own part of the CTA's strips through its
// own ring of shared-memory slots by cp.async.bulk, so the weights of BitNet-2B-sized
// layers (10 - 60 KB per SM) are on chip before the programmatic-dependency wait
// returns, and several launches of a stream prefetch at the same time (a CTA takes
// what it needs of shared memory and at most half of the register file).
// After the wait a call is one chain of latencies: read the activations, norm and quantise
// them, MMAs, one reduction over the warps, store.  Hence the front-end in the kernel
// for the smallest calls: every CTA repeats it (a few microseconds of one row's
// arithmetic would cost more as a launch of its own than as redundant work).
#pragma once
#include <cuda_bf16.h>

#include "act_quant.cuh"
#include "spmm_small_m.cuh"

namespace tsp {

constexpr int kW2MaxWarps = 10;
constexpr uint32_t kW2Mask = 0xC0C0C0C0u;

struct W2Smem {   // shared-memory plan: byte offsets from the base of the dynamic segment
    int red, xq, row, res, ring, total;
    int red_stride, x_stride;
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
constexpr int kW2MaxFusedRows = 8;                   // rows a front-end inside the kernel takes
constexpr int kW2Scale = kW2MaxWarps * kW2MaxSlots * 8;           // float s[32], ws[4] behind the mbarriers
constexpr int kW2Partial = kW2Scale + 48 * 4;                     // two sets (even and odd rows) of 32 partial sums, 32 maxima
constexpr int kW2ScratchBytes = kW2Partial + 2 * 64 * 4;

// R strips per CTA at most, `tokens` rows of x handled by a CTA (at most MT*8), W warps, ring slots of `slot_bytes`
inline W2Smem w2_smem(int R, int mt, int tokens, int K, int W, int slots, int slot_bytes, bool x_in_smem, int front_end,
                      bool residual) {
    W2Smem s;
    s.red_stride = R * 16 + 4;                       // conflict-free: token stride = 4 mod 16 words
    s.x_stride = (K & 127) ? K : K + 64;             // two tokens' 64-byte pieces on different banks
    int at = kW2ScratchBytes;
    s.red = at;
    at += mt * 8 * s.red_stride * 4;
    at = (at + 127) & ~127;
    s.xq = at;
    if (x_in_smem) at += ((tokens * s.x_stride + 64 + 127) & ~127);   // (a half pair reads 64 bytes past its row)
    s.row = at;                                      // a front-end's row (gated: both halves) and norm weight
    if (front_end != W2_INT8) at += ((K * (front_end == W2_GATED ? 6 : 4) + 127) & ~127);
    s.res = at;                                      // residual of the CTA's outputs, bf16 [tokens][R * 16]
    if (residual) at += ((tokens * R * 32 + 127) & ~127);
    s.ring = at;
    at += W * slots * slot_bytes;
    s.total = at;
    return s;
}

// XS: the CTA's int8 activations sit in shared memory (always with a front-end); otherwise fragments come straight from L2.
// Block pairs are taken U at a time, all their shared-memory loads first.  No branches inside: a group's absent strips and
// an absent second pair are computed from whatever the ring holds and from zeros, and not stored.
template <int MT, int RG, int U, int FE, bool XS>
__global__ void __launch_bounds__(kW2MaxWarps * 32, MT <= 2 ? 2 : 1) w2_small_kernel(const __grid_constant__ W2Params p) {
    static_assert(XS || FE == W2_INT8, "a front-end writes to shared memory");
    static_assert(XS || U == 1, "fragments from L2 are prefetched one pair ahead instead");
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthreads = blockDim.x;
    const int g = lane >> 2, q = lane & 3;
    const int K = p.e.K, N = p.e.N, D = p.slots;
    const int m0 = blockIdx.y * (MT * 8), mrows = min(p.e.M - m0, MT * 8);
    const int b = blockIdx.x, strip0 = b * p.strips_q + min(b, p.strips_r), nstrips = p.strips_q + (b < p.strips_r);
    const int KP = w2_pairs(K), PC = p.chunk_pairs;           // block pairs of K, at most PC per ring slot
    const int p0 = warp * p.pairs_q + min(warp, p.pairs_r), p1 = p0 + p.pairs_q + (warp < p.pairs_r);
    const int slot_bytes = RG * PC * 512;
    const W2Smem& L = p.smem;
    const uint32_t base = smem_u32(smem);
    int* red = reinterpret_cast<int*>(smem + L.red);
    float* scl = reinterpret_cast<float*>(smem + kW2Scale);
    const uint32_t bars = base + warp * (kW2MaxSlots * 8), ring = base + L.ring + warp * D * slot_bytes;
    const int NG = (nstrips + RG - 1) / RG;                   // groups of RG strips

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
    for (int i = tid; i < MT * 8 * L.red_stride; i += nthreads) red[i] = 0;
    constexpr bool kGated = FE == W2_GATED;
    const uint32_t row = base + L.row, wrow = row + K * (kGated ? 4 : 2);
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
    if (XS && FE == W2_INT8) {                                // this warp's columns of the rows, 16 bytes a piece
        const int pieces = (min(p1 * 128, K) - p0 * 128) >> 4;
        for (int t = lane >> 4; t < mrows; t += 2)
            for (int i = lane & 15; i < pieces; i += 16)
                cp_async_16(base + L.xq + t * L.x_stride + p0 * 128 + i * 16, p.e.x + (size_t)(m0 + t) * K + p0 * 128 + i * 16);
    }
    if (FE != W2_INT8) {
        const __nv_bfloat16* xr = p.xb + (size_t)m0 * (kGated ? 2 * K : K);
        act_row_copy(row, xr, K);
        if (kGated) act_row_copy(row + K * 2, xr + K, K);
        cp_async_commit();
        if (FE != W2_PLAIN) act_row_copy(wrow, p.norm_w, K);
    }
    if (res_smem) {
#pragma unroll 1
        for (int i = tid; i < mrows * nstrips * 2; i += nthreads) {   // 16 bytes a piece
            const int t = (int)((uint32_t)(i * 4) * inv_pairs >> 22), c = i * 4 - t * pairs;
            cp_async_16(base + L.res + (t * pairs + c) * 4, p.e.residual + (size_t)(m0 + t) * N + strip0 * 16 + c * 2);
        }
    }
    cp_async_commit();
    if (FE == W2_INT8 && tid < mrows) scl[tid] = __bfloat162float(p.e.s[m0 + tid]);
    if (tid >= 32 && tid < 36) scl[tid] = __bfloat162float(p.e.ws[tid - 32]);
    uint4 xn[2 * MT];                                         // direct fragments of the next pair
    auto load_x = [&](int pr, uint4* x) {                     // (columns of absent tokens are not stored)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            if (XS) {
                const uint32_t src = base + L.xq + min(mt * 8 + g, mrows - 1) * L.x_stride + pr * 128 + q * 16;
                x[2 * mt] = lds128(src);
                x[2 * mt + 1] = lds128(src + 64);
            } else {
                const int8_t* src = p.e.x + (size_t)(m0 + min(mt * 8 + g, mrows - 1)) * K + pr * 128 + q * 16;
                x[2 * mt] = ld_cg_128(src);
                x[2 * mt + 1] = ld_cg_128(src + (pr * 128 + 64 < K ? 64 : 0));   // (a half pair's second block has zero weights)
            }
        }
    };
    if (FE == W2_INT8) {
        if (!XS && p0 < p1) load_x(p0, xn);
        __syncthreads();                                      // red is zeroed, scales are staged
        if (XS) {
            cp_async_wait_all();                              // (the residual too)
            __syncwarp();
        }
    } else {
        constexpr int kMode = FE == W2_PLAIN ? ACT_PLAIN : ACT_RMSNORM;
        const int T = min(kActMaxThreads, max(64, ((K >> 3) + 31) & ~31));   // the fixed order of act_quant.cuh
#pragma unroll 1
        for (int t = 0; t < mrows; ++t) {
            float* part = reinterpret_cast<float*>(smem + kW2Partial) + (t & 1) * 64;
            const uint32_t xrow = base + L.xq + t * L.x_stride;
            if (t > 0) {                                      // (a thread's own vectors: the previous row's have been used)
                const __nv_bfloat16* xr = p.xb + (size_t)(m0 + t) * (kGated ? 2 * K : K);
                act_row_copy(row, xr, K);
                if (kGated) act_row_copy(row + K * 2, xr + K, K);
                cp_async_commit();
                cp_async_commit();                            // (no norm weight behind it)
            }
            const float s = act_row_finish<kGated, kMode>(row, wrow, p.eps, K, T, part, reinterpret_cast<uint32_t*>(part + 32), nullptr,
                                                          [&](int k0, const uint4& v) { sts64(xrow + k0, v.x, v.y); });
            if (tid == 0) scl[t] = s;
        }
        __syncthreads();
    }

    phase_mark(3);
    int d = 0;
    uint32_t parity = 0;
    bool refilled = false;                                    // the slots of the first round have been waited for
    for (int gi = 0; gi < NG && p0 < p1; ++gi) {
        constexpr int AC = RG * MT < 3 ? U : 1;               // separate accumulators per pair where there are few chains
        int acc[AC][RG][MT][4];
#pragma unroll
        for (int u = 0; u < AC; ++u)
#pragma unroll
            for (int r = 0; r < RG; ++r)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[u][r][mt][c] = 0;
        for (int c0 = p0; c0 < p1; c0 += PC) {
            if (refilled) ok = ok && mbar_wait_bounded(bars + 8 * d, parity);
            const uint32_t slot = ring + d * slot_bytes + w2_chunk(g, q);
            const int c1 = min(c0 + PC, p1);
#pragma unroll 1
            for (int pr = c0; pr < c1; pr += U) {
                uint4 x[U][2 * MT], w[U][RG];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int pu = u == 0 ? pr : min(pr + u, c1 - 1);
                    if (XS) {
                        load_x(pu, x[u]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 2 * MT; ++i) x[u][i] = xn[i];
                        if (p1 - p0 > 1) load_x(pr + 1 < p1 ? pr + 1 : p0, xn);
                    }
#pragma unroll
                    for (int r = 0; r < RG; ++r) w[u][r] = lds128(slot + (pu - c0) * 512 + r * PC * 512);
                    if (u > 0 && pr + u >= c1) {              // no second pair: zero activations
#pragma unroll
                        for (int i = 0; i < 2 * MT; ++i) x[u][i] = make_uint4(0, 0, 0, 0);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int r = 0; r < RG; ++r)
#pragma unroll
                        for (int blk = 0; blk < 2; ++blk) {
                            uint32_t a[4], b[4];              // rows g and g + 8
                            w2_decode(blk ? w[u][r].y : w[u][r].x, a), w2_decode(blk ? w[u][r].w : w[u][r].z, b);
#pragma unroll
                            for (int mt = 0; mt < MT; ++mt) {
                                const uint4 xv = x[u][2 * mt + blk];
                                mma_s8_16x8x32(acc[u % AC][r][mt], a[0], b[0], a[1], b[1], xv.x, xv.y);
                                mma_s8_16x8x32(acc[u % AC][r][mt], a[2], b[2], a[3], b[3], xv.z, xv.w);
                            }
                        }
            }
            __syncwarp();
            if (lane == 0 && f_gi < NG) fetch();              // into the slot just read
            if (++d == D) d = 0, parity ^= 1u, refilled = true;
        }
#pragma unroll
        for (int r = 0; r < RG; ++r) {
            const int strip = gi * RG + r;
            if (strip >= nstrips) break;
            int* dst = red + strip * 16 + g + 2 * q * L.red_stride;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    int v = acc[0][r][mt][c];
                    if (AC > 1) v += acc[AC - 1][r][mt][c];
                    if (mt * 8 + 2 * q + (c & 1) < mrows) atomicAdd(dst + (mt * 8 + (c & 1)) * L.red_stride + 8 * (c >> 1), v);
                }
        }
    }
    if (!ok) atomicExch(p.e.status, ST_WAIT_TIMEOUT);
    if (FE == W2_INT8 && !XS) cp_async_wait_all();            // the residual
    phase_mark(5);
    __syncthreads();
    phase_mark(6);

    // ---- epilogue (one loop body: code that runs once is paid for in instruction fetches)
#pragma unroll 1
    for (int i = tid; i < items; i += nthreads) {
        const int t = (int)((uint32_t)i * inv_pairs >> 22), c = (i - t * pairs) * 2, n = strip0 * 16 + c;
        const int v[2] = {red[t * L.red_stride + c] >> 6, red[t * L.red_stride + c + 1] >> 6};
        const size_t o = (size_t)(m0 + t) * N + n;
        __nv_bfloat16 r[2] = {scale_epilogue(v[0], scl[t], scl[32 + ws_group(n, p.e)], p.e.epilogue),
                              scale_epilogue(v[1], scl[t], scl[32 + ws_group(n + 1, p.e)], p.e.epilogue)};
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
