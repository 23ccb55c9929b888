// Attention glue of one decode step for sm_100a: RoPE on adjacent pairs, key / value append and attention of ONE new
// token per sequence over its cache, in one launch (model.py:205-243 of Gu-J/TernaInfer runs RoPE + cache update and
// xformers' attention there).
//
// What bounds it is latency: a step of a 600-token sequence reads 1.5 MB, a quarter of a microsecond, and the library
// kernels that did this job (a split kernel that also rotates and appends, and a combine kernel, outside of dependent
// launch) held a layer of the 30-layer model for 20 us.  A thread-block cluster of S <= 8 CTAs shares one key / value
// head of one sequence, each CTA an equal part of the cached keys, and combines through distributed shared memory, so
// nothing is left for a second launch.  Inside a CTA every warp runs alone over groups of 16 keys, with keys and values
// straight from global memory into mma.sync fragments: the head dimension of Q K^T is only a summation index, so a lane
// reads 16 consecutive bytes of a key and the query is permuted the same way; for P V a lane reads 32 consecutive bytes
// of four values and pairs them up with byte permutes.  The scores leave the first product in the registers in which the
// second one wants its A operand.  Running maximum and sum per warp, one merge per CTA (the new token's own key and
// value are one more partial result there), one over the cluster.  fp32 everywhere but the inputs, the rotated query,
// the probabilities of a group and the result.  Measured (60 caches in turn, 5 key / value heads): 1 sequence of 600 tokens
// 5.0 us, 8 of 1100 9.3 us, 16 of 2000 17.8 us (82 MB: 12.6 us at the copy rate); with the cache rows asked for ahead of
// the projections and a merge of one dimension per thread 5.6, 10.7, 19 us; with value tiles staged in shared memory and a
// CTA-wide softmax 6.0, 14.8, 32.9 us.
#pragma once
#include <cuda_bf16.h>

#include "spmm_small_m.cuh"

namespace tsp {

constexpr int kAttnD = 128;                // head dimension
constexpr int kAttnWarps = 4;

struct AttnParams {
    const __nv_bfloat16* qkv;              // [B][(H + 2 Hkv) * D], the new token's projections
    __nv_bfloat16 *k_cache, *v_cache;      // [B][L][Hkv][D], or [B][Hkv][L][D]
    const void *cos_row, *sin_row;         // [D / 2], the new token's rotation, bf16 (or fp32)
    const long long* pos;                  // position of the new token (the same in every sequence)
    __nv_bfloat16* out;                    // [B][H * D]
    int heads, kv_heads, max_len;
    float scale_log2;                      // log2(e) / sqrt(D)
    int* status;                           // BY_HEAD: told of a position outside of the cache
};

// D(16x8) += A(16x16) * B(16x8), bf16; rows8: rows 8-15 of A are zero
__device__ __forceinline__ void mma_bf16_rows8(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_full(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t bf16_pack(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float ex2_approx(float v) {                 // (weights below 2^-126 are zero)
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// (x, y) rotated by the angle whose cosine and sine are c, s
__device__ __forceinline__ uint32_t rope_pair(uint32_t xy, float c, float s) {
    const float x = bf16_lo(xy), y = bf16_hi(xy);
    return bf16_pack(x * c - y * s, x * s + y * c);
}
// the same as torch evaluates it: every product rounded
__device__ __forceinline__ uint32_t rope_pair_rounded(uint32_t xy, float c, float s) {
    const float x = bf16_lo(xy), y = bf16_hi(xy);
    return bf16_pack(__fsub_rn(__fmul_rn(x, c), __fmul_rn(y, s)), __fadd_rn(__fmul_rn(x, s), __fmul_rn(y, c)));
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// BY_HEAD: caches [B][Hkv][L][D] and an fp32 rotation whose products are rounded one by one: the layout and arithmetic of the
// default glue, which ran 27 torch kernels here (10 layers at 3 x 333 tokens: 932 us a token with them, 500 so).  index_copy_ refused a
// position outside of the cache, and so does this form: status 1, caches as they were, results NaN.
template <int GQ, bool BY_HEAD>
__global__ void __launch_bounds__(kAttnWarps * 32, 3) attn_decode_kernel(const AttnParams p) {
    constexpr int kParts = kAttnWarps + 1;                    // the warps' partial results and the new token's
    constexpr int kQStride = kAttnD + 8;                      // bf16 elements: conflict-free 16-byte reads
    constexpr int kOut = GQ * kAttnD, kThreads = kAttnWarps * 32;
    __shared__ __align__(16) __nv_bfloat16 qs[8 * kQStride];  // rotated queries, heads beyond GQ zero
    __shared__ __align__(16) float os[kParts][GQ][kAttnD];
    __shared__ float ms[kParts][8], ls[kParts][8];
    __shared__ __align__(16) __nv_bfloat16 kn[kAttnD];
    __shared__ __align__(16) float slot_o[kOut];
    __shared__ float slot_m[8][GQ], slot_l[8][GQ];   // pushed by the cluster's CTAs: [sender][outputs of this CTA], statistics
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int S = gridDim.x, rank = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;

    phase_mark(0);
    griddep_launch_dependents();
    cluster_arrive();                                         // (waited for before the first remote store)
    for (int i = tid; i < (8 - GQ) * kQStride / 2; i += kThreads) reinterpret_cast<uint32_t*>(qs)[GQ * kQStride / 2 + i] = 0u;
    const size_t row = BY_HEAD ? (size_t)kAttnD : (size_t)p.kv_heads * kAttnD;   // elements between two keys
    const size_t head0 = BY_HEAD ? ((size_t)b * p.kv_heads + hk) * p.max_len * kAttnD : ((size_t)b * p.max_len * p.kv_heads + hk) * kAttnD;
    const __nv_bfloat16* kc = p.k_cache + head0 + q * 8;      // this lane's 8 dimensions of every 32
    const __nv_bfloat16* vc = p.v_cache + head0 + g * 16;     // this lane's 16 dimensions
    const __nv_bfloat16* qkv = p.qkv + (size_t)b * (p.heads + 2 * p.kv_heads) * kAttnD;
    int gi = rank * kAttnWarps + warp;                        // this warp's group of 16 keys

    uint4 kf[2][4], vf[4][2];
    auto load_keys = [&](int grp) {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const __nv_bfloat16* src = kc + (size_t)min(grp * 16 + g + 8 * t, p.max_len - 1) * row;
#pragma unroll
            for (int c = 0; c < 4; ++c) kf[t][c] = ld_cg_128(src + c * 32);
        }
    };
    auto load_values = [&](int grp) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const __nv_bfloat16* src = vc + (size_t)min(grp * 16 + 2 * q + (t & 1) + 8 * (t >> 1), p.max_len - 1) * row;
            vf[t][0] = ld_cg_128(src), vf[t][1] = ld_cg_128(src + 8);
        }
    };
    phase_mark(1);
    griddep_wait();
    phase_mark(2);
    // Everything is asked for before the position is known (rows at and beyond it are masked below), the new token's
    // projections ahead of the cache rows: a warp's loads return in order, and 8 KB of keys and values per warp, 100 KB per SM,
    // take their time (8 sequences of 1100 tokens: the query was in place 2.8 us after the dependency, before).
    const long long pos_ll = *p.pos;
    constexpr int kPairs = (GQ + 1) * 64 / kThreads + ((GQ + 1) * 64 % kThreads != 0);   // rotated pairs per thread, query heads and the new key
    uint32_t xy[kPairs];
    float rc[kPairs], rs[kPairs];
#pragma unroll
    for (int k = 0; k < kPairs; ++k) {
        const int i = tid + k * kThreads, h = i >> 6, d = i & 63;
        if (h < GQ + (rank == 0)) {
            xy[k] = ld_cg_32(qkv + (size_t)(h < GQ ? hk * GQ + h : p.heads + hk) * kAttnD + 2 * d);
            if (BY_HEAD) rc[k] = static_cast<const float*>(p.cos_row)[d], rs[k] = static_cast<const float*>(p.sin_row)[d];
            else rc[k] = __bfloat162float(static_cast<const __nv_bfloat16*>(p.cos_row)[d]), rs[k] = __bfloat162float(static_cast<const __nv_bfloat16*>(p.sin_row)[d]);
        }
    }
    const uint2 vnew = *reinterpret_cast<const uint2*>(qkv + (size_t)(p.heads + p.kv_heads + hk) * kAttnD + lane * 4);
    if (gi * 16 < p.max_len) load_keys(gi), load_values(gi);
#pragma unroll
    for (int k = 0; k < kPairs; ++k) {
        const int i = tid + k * kThreads, h = i >> 6, d = i & 63;
        if (h < GQ + (rank == 0))
            (h < GQ ? reinterpret_cast<uint32_t*>(qs) + h * kQStride / 2 : reinterpret_cast<uint32_t*>(kn))[d] =
                BY_HEAD ? rope_pair_rounded(xy[k], rc[k], rs[k]) : rope_pair(xy[k], rc[k], rs[k]);
    }
    // cached keys 0 .. pos-1, the new one goes to row pos (clamped: a wrong position must not leave the cache)
    const int pos = (int)max(0ll, min(pos_ll, (long long)p.max_len - 1));
    const bool refused = BY_HEAD && pos_ll != pos;
    if (refused && tid == 0) atomicExch(p.status, ST_BAD_SHAPE);
    const int groups = (pos + 15) >> 4;
    __syncthreads();
    phase_mark(3);
    uint4 qf[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) qf[c] = *reinterpret_cast<const uint4*>(qs + g * kQStride + c * 32 + q * 8);

    // acc[i]: dimensions 16g + 2i (elements 0, 1) and 16g + 2i + 1 (2, 3) of heads 2q and 2q + 1; m, l: head g
    float acc[8][4], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 1
    for (; gi < groups; gi += S * kAttnWarps) {
        float sc[2][2][4];                                    // two chains per half of the group
#pragma unroll
        for (int t = 0; t < 4; ++t) sc[t >> 1][t & 1][0] = sc[t >> 1][t & 1][1] = sc[t >> 1][t & 1][2] = sc[t >> 1][t & 1][3] = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                mma_bf16_rows8(sc[t][0], qf[c].x, qf[c].y, kf[t][c].x, kf[t][c].y);
                mma_bf16_rows8(sc[t][1], qf[c].z, qf[c].w, kf[t][c].z, kf[t][c].w);
            }
        const int next = gi + S * kAttnWarps;
        if (next < groups) load_keys(next);
        float mx = m, pr[4];                                  // head g, keys 2q, 2q + 1 of either half
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int key = gi * 16 + 8 * (i >> 1) + 2 * q + (i & 1);
            pr[i] = key < pos ? (sc[i >> 1][0][i & 1] + sc[i >> 1][1][i & 1]) * p.scale_log2 : -INFINITY;
            mx = fmaxf(mx, pr[i]);
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float r = ex2_approx(m - mx);                        // (a group holds at least one key: mx is finite)
        m = mx, l *= r;
#pragma unroll
        for (int i = 0; i < 4; ++i) pr[i] = ex2_approx(pr[i] - mx), l += pr[i];
        const uint32_t b0 = bf16_pack(pr[0], pr[1]), b1 = bf16_pack(pr[2], pr[3]);   // as they are: keys x head g
        const float r0 = __shfl_sync(0xffffffffu, r, 8 * q), r1 = __shfl_sync(0xffffffffu, r, 8 * q + 4);
        if (gi * 16 + 16 > pos) {                             // rows that are not keys may hold anything: 0 * NaN
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (gi * 16 + 2 * q + (t & 1) + 8 * (t >> 1) >= pos) vf[t][0] = vf[t][1] = make_uint4(0, 0, 0, 0);
        }
        const uint32_t* v0 = reinterpret_cast<const uint32_t*>(vf[0]);
        const uint32_t* v1 = reinterpret_cast<const uint32_t*>(vf[1]);
        const uint32_t* v2 = reinterpret_cast<const uint32_t*>(vf[2]);
        const uint32_t* v3 = reinterpret_cast<const uint32_t*>(vf[3]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            acc[i][0] *= r0, acc[i][2] *= r0, acc[i][1] *= r1, acc[i][3] *= r1;
            mma_bf16_full(acc[i], __byte_perm(v0[i], v1[i], 0x5410), __byte_perm(v0[i], v1[i], 0x7632), __byte_perm(v2[i], v3[i], 0x5410),
                          __byte_perm(v2[i], v3[i], 0x7632), b0, b1);
        }
        if (next < groups) load_values(next);
    }
    phase_mark(4);
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    if (q == 0) ms[warp][g] = m, ls[warp][g] = l;
    // the new token's own key against every head, and its key and value into the cache
#pragma unroll 1
    for (int h = warp; h < GQ; h += kAttnWarps) {
        float d = -INFINITY;
        if (rank == 0) {
            const uint2 kv = *reinterpret_cast<const uint2*>(kn + lane * 4), qv = *reinterpret_cast<const uint2*>(qs + h * kQStride + lane * 4);
            d = bf16_lo(kv.x) * bf16_lo(qv.x) + bf16_hi(kv.x) * bf16_hi(qv.x) + bf16_lo(kv.y) * bf16_lo(qv.y) + bf16_hi(kv.y) * bf16_hi(qv.y);
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) d += __shfl_xor_sync(0xffffffffu, d, k);
            d *= p.scale_log2;
            const uint2 v = vnew;
            *reinterpret_cast<float4*>(&os[kAttnWarps][h][lane * 4]) = make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
            if (h == 0 && !refused) {
                *reinterpret_cast<uint2*>(p.k_cache + head0 + (size_t)pos * row + lane * 4) = kv;
                *reinterpret_cast<uint2*>(p.v_cache + head0 + (size_t)pos * row + lane * 4) = v;
            }
        }
        if (lane == 0) ms[kAttnWarps][h] = d, ls[kAttnWarps][h] = 1.f;
    }
    if (2 * q < GQ) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            *reinterpret_cast<float2*>(&os[warp][2 * q][16 * g + 2 * i]) = make_float2(acc[i][0], acc[i][2]);
            *reinterpret_cast<float2*>(&os[warp][2 * q + 1][16 * g + 2 * i]) = make_float2(acc[i][1], acc[i][3]);
        }
    }
    cluster_wait();                                           // every CTA of the cluster has started
    __syncthreads();
    // ---- merge the CTA's parts (a part without keys has maximum -inf and weight 0) and push them to the CTA that finishes them
    const int per = kOut / S, lg = 31 - __clz(per);           // outputs finished by a CTA, a power of two
#pragma unroll 1
    for (int h = warp; h < GQ; h += kAttnWarps) {             // a warp per head, four dimensions per lane
        float mk[kParts], lk[kParts], top = -INFINITY, sum = 0.f;
        float4 ok[kParts], o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < kParts; ++k) {
            mk[k] = ms[k][h], lk[k] = ls[k][h];
            ok[k] = k < kAttnWarps || rank == 0 ? *reinterpret_cast<const float4*>(&os[k][h][lane * 4]) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < kParts; ++k) top = fmaxf(top, mk[k]);
#pragma unroll
        for (int k = 0; k < kParts; ++k) {
            const float w = mk[k] == -INFINITY ? 0.f : ex2_approx(mk[k] - top);
            sum += w * lk[k];
            o.x += w * ok[k].x, o.y += w * ok[k].y, o.z += w * ok[k].z, o.w += w * ok[k].w;
        }
        const int i = h * kAttnD + lane * 4;                  // (per is at least 64: four outputs have one owner)
        st_cluster_v4(map_to_rank(smem_u32(&slot_o[rank * per + (i & (per - 1))]), i >> lg), __float_as_int(o.x), __float_as_int(o.y),
                      __float_as_int(o.z), __float_as_int(o.w));
        if (lane < S) {
            st_cluster_f32(map_to_rank(smem_u32(&slot_m[rank][h]), lane), top);
            st_cluster_f32(map_to_rank(smem_u32(&slot_l[rank][h]), lane), sum);
        }
    }
    phase_mark(5);
    cluster_arrive();
    cluster_wait();                                           // all parts have arrived; nothing remote is touched after this
    phase_mark(6);
    for (int j = tid; j < per; j += kThreads) {
        const int i = rank * per + j, h = i / kAttnD;
        float mr[8], lr[8], orr[8], top = -INFINITY, l_all = 0.f, o_all = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (r < S) mr[r] = slot_m[r][h], lr[r] = slot_l[r][h], orr[r] = slot_o[r * per + j];
            else mr[r] = -INFINITY, lr[r] = orr[r] = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) top = fmaxf(top, mr[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float w = mr[r] == -INFINITY ? 0.f : ex2_approx(mr[r] - top);
            l_all += w * lr[r], o_all += w * orr[r];
        }
        p.out[((size_t)b * p.heads + hk * GQ) * kAttnD + i] = __float2bfloat16_rn(refused ? NAN : o_all / l_all);
    }
    phase_mark(7);
}

}  // namespace tsp
