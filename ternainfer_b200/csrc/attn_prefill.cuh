// Attention glue of a prompt for sm_100a: RoPE on adjacent pairs, key / value append and causal attention of T new tokens per
// sequence over its cache (the prompt half of model.py:205-243 of Gu-J/TernaInfer).
//
// Two launches.  rope_append_kernel rotates the new keys and writes keys and values into the cache.
// attn_prefill_kernel is flash attention on mma.sync for grouped-query heads: a CTA takes 16 positions of the four query heads
// that share a key / value head - one head per warp -, so a tile of 64 keys and values is fetched once for 64 query rows.  The
// query is rotated on its way into the A fragments.  Tiles arrive by
// cp.async, double-buffered, in an XOR-swizzled layout that ldmatrix reads without bank conflicts; three CTAs per SM.
// Probabilities are rounded to bf16 for the second product, everything else accumulates in fp32.
// What bounds it is the chain of each warp at two to three warps per scheduler (tensor pipe 39 % of the active cycles, 58 % on
// the busiest SM, issue slots 28 %; stalls: fixed latencies, then fragment loads), and for short prompts the chain of the
// longest rows.  So instructions on that chain count: addresses that take one XOR per
// fragment, exponentials without range handling, an output that is rescaled only in tiles in which a row of the warp has a new
// maximum, CTAs sorted longest first over the whole launch, and two CTAs per item where there are few
// (ternaspmm_attn_prefill).  Both launches, 20 / 5 heads: 2 prompts of 613 tokens 35.9 -> 27.1 us (flash_attn's kv-cache
// kernel, which rotates and appends inside every CTA: 89 us), one of 1024 50.7 -> 30.3, of 4096 322 -> 263, 8 of 64 11.9 -> 8.6.
#pragma once
#include "attn_decode.cuh"

namespace tsp {

constexpr int kPfKeys = 64;                        // keys per tile
constexpr int kPfTile = kPfKeys * kAttnD * 2;      // bytes of a tile of keys or values

struct AttnPrefillParams {
    const __nv_bfloat16* qkv;              // [B][T][(H + 2 Hkv) * D]
    __nv_bfloat16 *k_cache, *v_cache;      // [B][L][Hkv][D]
    const __nv_bfloat16 *cos_tab, *sin_tab;   // [L][D / 2]
    const long long* pos;                  // positions of the new tokens, consecutive; pos[0] is read
    __nv_bfloat16* out;                    // [B][T][H * D]
    int T, heads, kv_heads, max_len;
    float scale_log2;
};

// One thread per 16 bytes: of a new key (rotated) and of the value beside it.
__global__ void __launch_bounds__(256) rope_append_kernel(const AttnPrefillParams p, long long items) {
    griddep_launch_dependents();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    griddep_wait();
    if (i >= items) return;
    const int c = (int)(i & 15);                                   // 8 dimensions
    const long long r = i >> 4;
    const int hk = (int)(r % p.kv_heads);
    const long long bt = r / p.kv_heads;
    const int b = (int)(bt / p.T), t = (int)(bt - (long long)b * p.T);
    const long long pos = *p.pos + t;
    if (pos < 0 || pos >= p.max_len) return;                       // (a wrong position must not leave the cache)
    const __nv_bfloat16* src = p.qkv + (size_t)bt * (p.heads + 2 * p.kv_heads) * kAttnD + (size_t)(p.heads + hk) * kAttnD + c * 8;
    const uint4 k = ld_cg_128(src), v = ld_cg_128(src + (size_t)p.kv_heads * kAttnD);
    const uint2 cs = *reinterpret_cast<const uint2*>(p.cos_tab + (size_t)pos * 64 + c * 4), sn = *reinterpret_cast<const uint2*>(p.sin_tab + (size_t)pos * 64 + c * 4);
    const size_t dst = (((size_t)b * p.max_len + pos) * p.kv_heads + hk) * kAttnD + c * 8;
    *reinterpret_cast<uint4*>(p.k_cache + dst) =
        make_uint4(rope_pair(k.x, bf16_lo(cs.x), bf16_lo(sn.x)), rope_pair(k.y, bf16_hi(cs.x), bf16_hi(sn.x)),
                   rope_pair(k.z, bf16_lo(cs.y), bf16_lo(sn.y)), rope_pair(k.w, bf16_hi(cs.y), bf16_hi(sn.y)));
    *reinterpret_cast<uint4*>(p.v_cache + dst) = v;
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// grid: items (16 positions of four query heads of a sequence), longest first, times S.  S = 2: the CTAs of a cluster take every
// other tile of keys, and each finishes two of the four heads.
template <int S>
__global__ void __launch_bounds__(128, 3) attn_prefill_kernel(const AttnPrefillParams p, int heads_x_batch) {
    extern __shared__ __align__(128) uint8_t smem[];               // [2 buffers][keys | values]
    const uint32_t base = smem_u32(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int item = blockIdx.x / S, rank = blockIdx.x % S, hb = item % heads_x_batch;
    const int qg = (p.T + 15) / 16 - 1 - item / heads_x_batch, h = hb % (p.heads / 4) * 4 + warp, hk = h / (p.heads / p.kv_heads), b = hb / (p.heads / 4);
    griddep_launch_dependents();
    const long long pos0_ll = *p.pos;
    const int pos0 = (int)max(0ll, min(pos0_ll, (long long)p.max_len - 1));
    const int t_first = qg * 16, t_last = min(t_first + 15, p.T - 1);
    const int n_keys = min(pos0 + t_last + 1, p.max_len), tiles = (n_keys + kPfKeys - 1) / kPfKeys;   // keys that the last row sees
    const size_t row = (size_t)p.kv_heads * kAttnD;
    const __nv_bfloat16* kc = p.k_cache + ((size_t)b * p.max_len * p.kv_heads + hk) * kAttnD;
    const __nv_bfloat16* vc = p.v_cache + ((size_t)b * p.max_len * p.kv_heads + hk) * kAttnD;

    // tiles: 16-byte chunk c of row r sits at c ^ (r & 7); this thread copies chunk tid & 15 of every eighth row
    const uint32_t f_dst = base + (uint32_t)((tid >> 4) * 256 + (((tid & 15) ^ ((tid >> 4) & 7)) << 4));
    const __nv_bfloat16 *f_k = kc + (tid & 15) * 8, *f_v = vc + (tid & 15) * 8;
    auto fetch = [&](int tile, int buf) {
#pragma unroll
        for (int k = 0; k < kPfKeys / 8; ++k) {
            const long long src = (long long)min(tile * kPfKeys + (tid >> 4) + 8 * k, n_keys - 1) * (int)row;
            cp_async_16(f_dst + buf * 2 * kPfTile + k * 2048, f_k + src);
            cp_async_16(f_dst + buf * 2 * kPfTile + kPfTile + k * 2048, f_v + src);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (rank < tiles) fetch(rank, 0);

    // ---- query fragments: rotated on the way through the second buffer (16 bytes a lane: two-byte pairs straight into the
    // fragments and their angles are 96 loads)
    uint32_t qa[8][4];
    const uint32_t qs = base + 2 * kPfTile + warp * 4096;
#pragma unroll 4
    for (int i = lane; i < 256; i += 32) {
        const int r = i >> 4, c = i & 15, t = min(t_first + r, p.T - 1), pp = min(pos0 + t, p.max_len - 1);
        const uint4 x = ld_cg_128(p.qkv + ((size_t)b * p.T + t) * (p.heads + 2 * p.kv_heads) * kAttnD + (size_t)h * kAttnD + c * 8);
        const uint2 cs = *reinterpret_cast<const uint2*>(p.cos_tab + (size_t)pp * 64 + c * 4), sn = *reinterpret_cast<const uint2*>(p.sin_tab + (size_t)pp * 64 + c * 4);
        sts128(qs + (uint32_t)(r * 256 + ((c ^ (r & 7)) << 4)),
               make_uint4(rope_pair(x.x, bf16_lo(cs.x), bf16_lo(sn.x)), rope_pair(x.y, bf16_hi(cs.x), bf16_hi(sn.x)),
                          rope_pair(x.z, bf16_lo(cs.y), bf16_lo(sn.y)), rope_pair(x.w, bf16_hi(cs.y), bf16_hi(sn.y))));
    }
    __syncwarp();
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
        const int r = (lane & 7) + (((lane >> 3) & 1) << 3), c = ks * 2 + (lane >> 4);
        ldmatrix_x4(qs + (uint32_t)(r * 256 + ((c ^ (r & 7)) << 4)), qa[ks]);
    }
    const int tr[2] = {t_first + g, t_first + g + 8};              // this lane's rows of the fragments
    __syncthreads();                                               // the buffer may be filled
    // this lane's rows of 16 keys for ldmatrix: the swizzle takes the row's low bits, which are the lane's
    const uint32_t k_lane = (uint32_t)(((lane & 7) + ((lane >> 4) << 3)) * 256 + ((((lane >> 3) & 1) ^ (lane & 7)) << 4));
    const uint32_t v_lane = (uint32_t)((lane & 15) * 256 + (((lane >> 4) ^ (lane & 7)) << 4));
    float o[16][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;

#pragma unroll 1
    for (int tile = rank, buf = 0; tile < tiles; tile += S, buf ^= 1) {
        const uint32_t kt = base + buf * 2 * kPfTile, vt = kt + kPfTile;
        if (tile + S < tiles) {
            fetch(tile + S, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            cp_async_wait_all();
        }
        __syncthreads();
        // ---- scores: 16 rows x 64 keys
        float s[8][4];
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {                       // 16 keys: two n-tiles x the two halves of k
                uint32_t kb[4];
                ldmatrix_x4(kt + (k_lane ^ (ks * 32)) + jj * 4096, kb);
                mma_bf16_full(s[2 * jj], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kb[0], kb[1]);
                mma_bf16_full(s[2 * jj + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kb[2], kb[3]);
            }
        // ---- online softmax; rows g (elements 0, 1) and g + 8 (2, 3)
        if ((tile + 1) * kPfKeys > pos0 + t_first + 1) {           // some row does not see all of the tile
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (tile * kPfKeys + 8 * j + 2 * q + (e & 1) > pos0 + tr[e >> 1]) s[j][e] = -INFINITY;
        }
        float mx[2] = {m[0], m[1]};                                // (of the unscaled scores)
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2));
        }
        // m, to which sum and output are relative, follows the maximum (and leaves -inf, by the NaN).  Following it only when it has
        // grown by 2^8 took 2 % less time, but the largest probabilities, no longer just below one, then round at twice the step:
        // 200 tokens behind 1000 were 2.31e-3 from float64 instead of 2.19e-3
        const bool grown = !(mx[0] - m[0] <= 0.f) || !(mx[1] - m[1] <= 0.f);
        if (__any_sync(0xffffffffu, grown)) {
            float r[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                // (S = 1: key 0 is visible to every row, so mx is finite from the first tile on; a half may see no key of a tile)
                if (S > 1 && mx[e] == -INFINITY) mx[e] = -1.0e38f;
                r[e] = ex2_approx((m[e] - mx[e]) * p.scale_log2);
                m[e] = mx[e], l[e] *= r[e];
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j][0] *= r[0], o[j][1] *= r[0], o[j][2] *= r[1], o[j][3] *= r[1];
        }
        const float ms[2] = {m[0] * p.scale_log2, m[1] * p.scale_log2};
        uint32_t pa[4][4];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[j][e] = ex2_approx(s[j][e] * p.scale_log2 - ms[e >> 1]), l[e >> 1] += s[j][e];
            pa[j >> 1][2 * (j & 1)] = bf16_pack(s[j][0], s[j][1]);
            pa[j >> 1][2 * (j & 1) + 1] = bf16_pack(s[j][2], s[j][3]);
        }
        // ---- values: 16 rows x 128 dimensions
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {                       // 16 dimensions: two n-tiles x the two halves of k
                uint32_t vb[4];
                ldmatrix_x4_trans(vt + (v_lane ^ (jj * 32)) + ks * 4096, vb);
                mma_bf16_full(o[2 * jj], pa[ks][0], pa[ks][1], pa[ks][2], pa[ks][3], vb[0], vb[1]);
                mma_bf16_full(o[2 * jj + 1], pa[ks][0], pa[ks][1], pa[ks][2], pa[ks][3], vb[2], vb[3]);
            }
        __syncthreads();                                           // the buffer may be filled again
    }
    if (S > 1) {
        cluster_arrive();
        cluster_wait();                                            // both CTAs have read their last tile
        const uint32_t slot = base + (warp & 1) * 8704 + lane * 16;
        if ((warp >> 1) != rank) {                                 // sent to the CTA that finishes this head
            const uint32_t dst = map_to_rank(slot, rank ^ 1);
#pragma unroll
            for (int j = 0; j < 16; ++j)
                st_cluster_v4(dst + j * 512, __float_as_int(o[j][0]), __float_as_int(o[j][1]), __float_as_int(o[j][2]), __float_as_int(o[j][3]));
            st_cluster_v4(dst + 16 * 512, __float_as_int(m[0]), __float_as_int(m[1]), __float_as_int(l[0]), __float_as_int(l[1]));
        }
        cluster_arrive();
        cluster_wait();                                            // nothing remote is touched after this
        if ((warp >> 1) != rank) return;
        const uint4 st = lds128(slot + 16 * 512);
        float wa[2], wb[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float m2 = __uint_as_float(e ? st.y : st.x), top = fmaxf(m[e], m2);   // (finite: one half saw key 0)
            wa[e] = ex2_approx((m[e] - top) * p.scale_log2), wb[e] = ex2_approx((m2 - top) * p.scale_log2);
            l[e] = wa[e] * l[e] + wb[e] * __uint_as_float(e ? st.w : st.z);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const uint4 v = lds128(slot + j * 512);
            o[j][0] = wa[0] * o[j][0] + wb[0] * __uint_as_float(v.x), o[j][1] = wa[0] * o[j][1] + wb[0] * __uint_as_float(v.y);
            o[j][2] = wa[1] * o[j][2] + wb[1] * __uint_as_float(v.z), o[j][3] = wa[1] * o[j][3] + wb[1] * __uint_as_float(v.w);
        }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 1);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 2);
        if (tr[e] >= p.T) continue;
        const float inv = 1.f / l[e];
        __nv_bfloat16* dst = p.out + ((size_t)b * p.T + tr[e]) * p.heads * kAttnD + (size_t)h * kAttnD + 2 * q;
#pragma unroll
        for (int j = 0; j < 16; ++j) *reinterpret_cast<uint32_t*>(dst + 8 * j) = bf16_pack(o[j][2 * e] * inv, o[j][2 * e + 1] * inv);
    }
}

}  // namespace tsp
