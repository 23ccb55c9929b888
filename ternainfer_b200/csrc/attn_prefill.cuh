// Attention glue of a prompt for sm_100a: RoPE on adjacent pairs, key / value append and causal attention of T new tokens per
// sequence over its cache (the prompt half of model.py:205-243 of Gu-J/TernaInfer).
//
// Two launches.  rope_append_kernel rotates the new keys and writes keys and values into the cache.
// attn_prefill_kernel is flash attention on mma.sync for grouped-query heads: a CTA takes 16 positions of the four query heads
// that share a key / value head - one head per warp -, so a tile of 64 keys and values is fetched once for 64 query rows.  The
// query is rotated in the registers of its A fragments (a register holds an adjacent pair).  Tiles arrive by
// cp.async, double-buffered, in an XOR-swizzled layout that ldmatrix reads without bank conflicts; three CTAs per SM.
// Probabilities are rounded to bf16 for the second product, everything else accumulates in fp32.
// flash_attn's kv-cache kernel, which rotates and appends inside every CTA, took 89 us for 2 prompts of 613 tokens (20 / 5 heads),
// the two launches take 40 us (36 of them the second).  What bounds it: the issue of mma.sync, and the CTAs of the last rows.
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

// grid: (groups of 16 positions, longest first; groups of four query heads; sequences)
__global__ void __launch_bounds__(128, 3) attn_prefill_kernel(const AttnPrefillParams p) {
    extern __shared__ __align__(128) uint8_t smem[];               // [2 buffers][keys | values]
    const uint32_t base = smem_u32(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int qg = (int)gridDim.x - 1 - (int)blockIdx.x;           // the longest rows start first
    const int h = blockIdx.y * 4 + warp, hk = h / (p.heads / p.kv_heads), b = blockIdx.z;
    griddep_launch_dependents();
    griddep_wait();
    const long long pos0_ll = *p.pos;
    const int pos0 = (int)max(0ll, min(pos0_ll, (long long)p.max_len - 1));
    const int t_first = qg * 16, t_last = min(t_first + 15, p.T - 1);
    const int n_keys = min(pos0 + t_last + 1, p.max_len), tiles = (n_keys + kPfKeys - 1) / kPfKeys;   // keys that the last row sees
    const size_t row = (size_t)p.kv_heads * kAttnD;
    const __nv_bfloat16* kc = p.k_cache + ((size_t)b * p.max_len * p.kv_heads + hk) * kAttnD;
    const __nv_bfloat16* vc = p.v_cache + ((size_t)b * p.max_len * p.kv_heads + hk) * kAttnD;

    auto fetch = [&](int tile, int buf) {                          // 16-byte chunk c of row r sits at c ^ (r & 7)
        const uint32_t dst = base + buf * 2 * kPfTile;
#pragma unroll 4
        for (int i = tid; i < kPfKeys * 16; i += 128) {
            const int r = i >> 4, c = i & 15;
            const size_t src = (size_t)min(tile * kPfKeys + r, n_keys - 1) * row + c * 8;
            const uint32_t d = (uint32_t)(r * 256 + ((c ^ (r & 7)) << 4));
            cp_async_16(dst + d, kc + src);
            cp_async_16(dst + kPfTile + d, vc + src);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);

    // ---- query fragments: rows g and g + 8 = positions t_first + g (+ 8), rotated in place
    uint32_t qa[8][4];
    int tr[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        tr[r] = t_first + g + 8 * r;
        const int t = min(tr[r], p.T - 1), pp = min(pos0 + t, p.max_len - 1);
        const __nv_bfloat16* src = p.qkv + ((size_t)b * p.T + t) * (p.heads + 2 * p.kv_heads) * kAttnD + (size_t)h * kAttnD;
#pragma unroll
        for (int s = 0; s < 8; ++s)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int d = s * 16 + 8 * k + 2 * q;               // an adjacent pair
                const uint32_t xy = ld_cg_32(src + d);
                qa[s][r + 2 * k] = rope_pair(xy, __bfloat162float(p.cos_tab[(size_t)pp * 64 + (d >> 1)]), __bfloat162float(p.sin_tab[(size_t)pp * 64 + (d >> 1)]));
            }
    }
    float o[16][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;

#pragma unroll 1
    for (int tile = 0; tile < tiles; ++tile) {
        const uint32_t kt = base + (tile & 1) * 2 * kPfTile, vt = kt + kPfTile;
        if (tile + 1 < tiles) {
            fetch(tile + 1, (tile + 1) & 1);
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
                const int r = jj * 16 + (lane & 7) + ((lane >> 4) << 3), c = ks * 2 + ((lane >> 3) & 1);
                uint32_t kb[4];
                ldmatrix_x4(kt + (uint32_t)(r * 256 + ((c ^ (r & 7)) << 4)), kb);
                mma_bf16_full(s[2 * jj], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kb[0], kb[1]);
                mma_bf16_full(s[2 * jj + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kb[2], kb[3]);
            }
        // ---- online softmax; rows g (elements 0, 1) and g + 8 (2, 3)
        const bool edge = (tile + 1) * kPfKeys > pos0 + t_first + 1;   // some row does not see all of the tile
        float mx[2] = {m[0], m[1]};
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = tile * kPfKeys + 8 * j + 2 * q + (e & 1);
                s[j][e] = (!edge || key <= pos0 + tr[e >> 1]) ? s[j][e] * p.scale_log2 : -INFINITY;
                mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
            }
        float r[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2));
            r[e] = exp2f(m[e] - mx[e]);                            // (key 0 is visible to every row: mx is finite from the first tile on)
            m[e] = mx[e], l[e] *= r[e];
        }
        uint32_t pa[4][4];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[j][e] = exp2f(s[j][e] - mx[e >> 1]), l[e >> 1] += s[j][e];
            pa[j >> 1][2 * (j & 1)] = bf16_pack(s[j][0], s[j][1]);
            pa[j >> 1][2 * (j & 1) + 1] = bf16_pack(s[j][2], s[j][3]);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j][0] *= r[0], o[j][1] *= r[0], o[j][2] *= r[1], o[j][3] *= r[1];
        // ---- values: 16 rows x 128 dimensions
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {                       // 16 dimensions: two n-tiles x the two halves of k
                const int rr = ks * 16 + (lane & 15), c = jj * 2 + (lane >> 4);
                uint32_t vb[4];
                ldmatrix_x4_trans(vt + (uint32_t)(rr * 256 + ((c ^ (rr & 7)) << 4)), vb);
                mma_bf16_full(o[2 * jj], pa[ks][0], pa[ks][1], pa[ks][2], pa[ks][3], vb[0], vb[1]);
                mma_bf16_full(o[2 * jj + 1], pa[ks][0], pa[ks][1], pa[ks][2], pa[ks][3], vb[2], vb[3]);
            }
        __syncthreads();                                           // the buffer may be filled again
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
