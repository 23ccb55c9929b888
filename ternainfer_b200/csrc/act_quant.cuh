// Fused activation front-ends of the ternary linears for sm_100a: the work the
// reference does between two TernaSpMM calls with a chain of small library
// kernels (xformers RMSNorm, the Triton-compiled `quant_input`, `squared_relu`;
// model.py:120-123, 235-243, 277-282, 323-335 of Gu-J/TernaInfer) as ONE kernel
// per linear input:
//   norm_quant       x -> RMSNorm(x) * w -> per-token absmax int8 + scale
//   gated_norm_quant [x1 | x3] -> relu(x1)^2 * x3 -> RMSNorm * w -> int8 + scale
// One CTA per token row; the row is staged once in shared memory as bf16, so
// HBM traffic is one read of the activations and one write of int8 + scale.
// Rounding points follow the eager PyTorch evaluation of the same expressions
// (bf16 after the norm, bf16(1/amax) * 127 for the scale, bf16(x*s) before the
// round-half-even).  The fp32 sum of squares has a FIXED order, so the result is
// reproducible bit for bit by any implementation that follows it: with T
// threads, thread t adds f*f (product rounded, then sum rounded: no fused
// multiply-add) over elements (j*T + t)*8 + 0..7 for j = 0, 1, ...; the 32
// lanes of a warp combine by the xor butterfly 16, 8, 4, 2, 1; warp sums are
// added in warp order.  The RMS factor is 1 / sqrt(ss / K + eps) with IEEE
// division and square root.  T = min(1024, max(64, K/8 rounded up to 32)).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx_sm100.cuh"

namespace tsp {

constexpr int kActMaxThreads = 1024;   // one 8-element vector per thread up to K = 8192; longer rows loop

__device__ __forceinline__ float bf16_round_f(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// Maximum that keeps a NaN, as torch's does: a row that holds one gets a NaN scale.
__device__ __forceinline__ float nan_max(float a, float b) { return (b > a || b != b) ? b : a; }

__device__ __forceinline__ float block_reduce(float v, float* scratch, bool is_max) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, v, d);
        v = is_max ? nan_max(v, o) : v + o;
    }
    __syncthreads();   // scratch may still be read from the previous reduction
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float r = scratch[0];
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) r = is_max ? nan_max(r, scratch[i]) : r + scratch[i];
    return r;
}

// MODE 0: y = RMSNorm(v) * w.  MODE 1: y = v * w without the normalisation, and the row's sum
// of squares of v is written to ss_out (tensor-parallel row shards: the RMS factor needs the sum
// over all shards and is applied after the all-reduce).  MODE 2: y = v (plain quantiser).
// MODE 3: y = RMSNorm(v) * w written out as bf16 to `q` (read as bf16 [M][K]), no quantiser: the
// model's final norm in the same fixed summation order.
enum ActMode : int { ACT_RMSNORM = 0, ACT_SCALE_SUMSQ = 1, ACT_PLAIN = 2, ACT_NORM_ONLY = 3 };

// One row by one CTA.  Virtual thread vt of T owns the elements 8 vt .. 8 vt + 7 (K <= 8192, so that T covers the row); a
// thread takes vt = tid, tid + blockDim, ....  What is left of this work at decode sizes is a chain of latencies -
// load, butterfly, barrier, square root, barrier, reciprocal - and the instruction fetches of code that runs once, so
// it is kept short: copies to shared memory by cp.async (every vector of a thread in flight at once, no registers
// held), loops that are not unrolled, packed bf16 arithmetic where its single rounding is the eager one.
//   act_weight_ahead   norm weight -> L2, before the dependency wait (one thread of the grid).  A copy to shared memory there could
//                      hold values that the kernel before has not replaced yet; it saved 0.09 us per linear (30-layer
//                      decode of one sequence: 908 us, 919 with the copy behind the wait)
//   act_row_copy       the row (gated: both halves), and behind it as a group of its own the norm weight -> shared memory
//   act_row_finish     norm, maximum, int8 values through store(k0, int8 x 8) (NORM_ONLY: bf16 x 8)
// `row`: K bf16 (gated: 2K), `wrow`: K bf16, both shared addresses; `part`, `mxp`: 32 words each.  The caller may reuse them
// after its next barrier.  Returns the scale s.
__device__ __forceinline__ void act_weight_ahead(const __nv_bfloat16* w, int K) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(w)), "r"(K * 2) : "memory");
}
__device__ __forceinline__ void act_row_copy(uint32_t dst, const __nv_bfloat16* src, int K) {
#pragma unroll 1
    for (int i = threadIdx.x; i * 8 < K; i += blockDim.x) cp_async_16(dst + i * 16, src + i * 8);
}

__device__ __forceinline__ uint32_t warp_max_u32(uint32_t v) {
    uint32_t r;
    asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ float act_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float act_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t act_mul2(uint32_t a, uint32_t b) {   // bf16 products, rounded once each
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t act_pack(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// acc / s rounded to nearest, for s with 8 significant bits (a bf16) in [2^-30, 2^30] and r = 1 / s rounded.  q0 is within two units
// in the last place, the remainder is exact (fused, a few bits), and q0 + rem * r errs by 2^-22 units at most before it is rounded.
// That decides the rounding: acc is a float, so a quotient that is not itself a float differs from the middle m of two floats by
// |acc - s m| / s with acc and s m whole multiples of one unit of s m, at least 2^-10 units in the last place (and is
// never such a middle: s m would have 25 significant bits).
__device__ __forceinline__ float quotient(float acc, float s, float r) {
    const float q0 = __fmul_rn(acc, r);
    return __fmaf_rn(__fmaf_rn(-q0, s, acc), r, q0);
}
__device__ __forceinline__ float quotient_rcp(float s) {     // 0: out of range
    return fabsf(s) >= 0x1p-30f && fabsf(s) <= 0x1p30f ? __fdiv_rn(1.0f, s) : 0.f;
}

// T of the fixed order
__host__ __device__ inline int act_row_threads(int K) {
    const int t = ((K >> 3) + 31) & ~31;
    return t < 64 ? 64 : (t > kActMaxThreads ? kActMaxThreads : t);
}

// scale of a row whose largest magnitude has the bf16 pattern `top`: 127 / amax as reciprocal * 127, in bf16
__device__ __forceinline__ float act_scale(uint32_t top_bits) {
    const float top = __uint_as_float(top_bits << 16);
    const float amax = bf16_round_f(top < 1e-5f ? 1e-5f : top);
    return bf16_round_f(bf16_round_f(1.0f / amax) * 127.0f);
}
// eight bf16 values times the scale (in both halves of s2), to int8
__device__ __forceinline__ uint2 act_quant8(const uint4& a, uint32_t s2) {
    const uint32_t av[4] = {a.x, a.y, a.z, a.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t pr = act_mul2(av[i], s2);
        asm("min.bf16x2 %0, %1, %2;" : "=r"(pr) : "r"(pr), "r"(0x42FE42FEu));   // 127: only +128 can lie outside of int8
        // adding 1.5 * 2^23 leaves the value rounded half to even in the low bits
        const uint32_t lo = __float_as_uint(__fadd_rn(act_lo(pr), 12582912.f)), hi = __float_as_uint(__fadd_rn(act_hi(pr), 12582912.f));
        o[i] = __byte_perm(lo, hi, 0x0040);
    }
    return make_uint2(__byte_perm(o[0], o[1], 0x5410), __byte_perm(o[2], o[3], 0x5410));
}

template <bool GATED, int MODE, typename Store>
__device__ __forceinline__ float act_row_finish(uint32_t row, uint32_t wrow, float eps, int K, int T, float* part, uint32_t* mxp,
                                                float* ss_out, Store store) {
    const int tid = threadIdx.x, lane = tid & 31, nthreads = blockDim.x, vwarps = T >> 5;
    if (MODE == ACT_PLAIN) cp_async_wait_all();
    else cp_async_wait_but_last();                     // the row is there, the norm weight may still be on its way
    // (a thread reads only vectors that it copied itself, so no barrier follows the wait)
    float rstd = 1.f;
    if (MODE != ACT_PLAIN) {
#pragma unroll 1
        for (int vt = tid; vt < T; vt += nthreads) {
            float ss = 0.f;
            if (vt * 8 < K) {
                uint4 a = lds128(row + vt * 16);
                uint32_t* av = reinterpret_cast<uint32_t*>(&a);
                if (GATED) {
                    const uint4 b = lds128(row + K * 2 + vt * 16);
                    const uint32_t bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {   // relu(x1) ** 2, bf16; * x3, bf16
                        uint32_t r;
                        asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(av[i]), "r"(0u));
                        av[i] = act_mul2(act_mul2(r, r), bv[i]);
                    }
                    sts128(row + vt * 16, a);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float lo = act_lo(av[i]), hi = act_hi(av[i]);
                    ss = __fadd_rn(ss, __fmul_rn(lo, lo));
                    ss = __fadd_rn(ss, __fmul_rn(hi, hi));
                }
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
            if (lane == 0) part[vt >> 5] = ss;
        }
        __syncthreads();
        float sum = part[0];
#pragma unroll 4
        for (int i = 1; i < vwarps; ++i) sum += part[i];
        if (MODE == ACT_SCALE_SUMSQ && tid == 0) *ss_out = sum;
        if (MODE != ACT_SCALE_SUMSQ) rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)K), eps)));
        cp_async_wait_all();
    }
#pragma unroll 1
    for (int vt = tid; vt < T; vt += nthreads) {
        uint32_t mx = 0;
        if (vt * 8 < K) {
            uint4 a = lds128(row + vt * 16);
            uint32_t* av = reinterpret_cast<uint32_t*>(&a);
            if (MODE != ACT_PLAIN) {
                const uint4 w = lds128(wrow + vt * 16);
                const uint32_t wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float lo = MODE == ACT_SCALE_SUMSQ ? act_lo(av[i]) : __fmul_rn(act_lo(av[i]), rstd);
                    const float hi = MODE == ACT_SCALE_SUMSQ ? act_hi(av[i]) : __fmul_rn(act_hi(av[i]), rstd);
                    av[i] = act_pack(__fmul_rn(lo, act_lo(wv[i])), __fmul_rn(hi, act_hi(wv[i])));
                }
                if (MODE == ACT_NORM_ONLY) store(vt * 8, a);
                else sts128(row + vt * 16, a);
            }
            // magnitudes: their bit patterns order like the values, NaN above all
#pragma unroll
            for (int i = 0; i < 4; ++i) mx = max(mx, max(av[i] & 0x7FFFu, (av[i] >> 16) & 0x7FFFu));
        }
        if (MODE != ACT_NORM_ONLY) {
            mx = warp_max_u32(mx);
            if (lane == 0) mxp[vt >> 5] = mx;
        }
    }
    if (MODE == ACT_NORM_ONLY) return 0.f;
    __syncthreads();
    const float s = act_scale(warp_max_u32(lane < vwarps ? mxp[lane] : 0u));
    const uint32_t s2 = (__float_as_uint(s) >> 16) * 0x10001u;
#pragma unroll 1
    for (int vt = tid; vt * 8 < K; vt += nthreads) {
        const uint2 v = act_quant8(lds128(row + vt * 16), s2);
        store(vt * 8, make_uint4(v.x, v.y, 0u, 0u));
    }
    return s;
}

// Up to R rows at a time by one CTA, VK vectors of each row per thread, all in registers: the front-end inside a linear's
// kernel (w2_small.cuh), where every CTA does the same rows and the chain of latencies is all there is.  Every load is asked for
// at once, the rows' butterflies run side by side, and with several rows their scalar parts (sum, square root, reciprocals)
// go to a warp each.  `part`, `mxp`: R x 32 words, `rstd_s`: R words; `scl`: scale and its quotient_rcp per row, [0 .. R) and [32 .. ).
template <bool GATED, int MODE, int VK, int R, typename Store>
__device__ __forceinline__ void act_rows(const __nv_bfloat16* x, const __nv_bfloat16* w, float eps, int K, int rows, float* part, uint32_t* mxp,
                                         float* rstd_s, float* scl, Store store) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = blockDim.x;
    const int T = act_row_threads(K), vwarps = T >> 5;
    const size_t ld = GATED ? 2 * (size_t)K : (size_t)K;
    uint4 a[R * VK], b[GATED ? R * VK : 1], wv[VK];
#pragma unroll
    for (int i = 0; i < R * VK; ++i) {
        const int r = i / VK, k0 = (tid + (i % VK) * n) * 8;
        const bool in = k0 < K && r < rows;
        a[i] = in ? ld_cg_128(x + r * ld + k0) : make_uint4(0, 0, 0, 0);
        if (GATED) b[i] = in ? ld_cg_128(x + r * ld + K + k0) : make_uint4(0, 0, 0, 0);
    }
    if (MODE != ACT_PLAIN) {
#pragma unroll
        for (int j = 0; j < VK; ++j) wv[j] = (tid + j * n) * 8 < K ? ld_cg_128(w + (tid + j * n) * 8) : make_uint4(0, 0, 0, 0);
    }
    float rstd = 1.f;
    if (MODE != ACT_PLAIN) {
        float ss[R * VK];
#pragma unroll
        for (int i = 0; i < R * VK; ++i) {
            uint32_t* av = reinterpret_cast<uint32_t*>(&a[i]);
            if (GATED) {
                const uint32_t* bv = reinterpret_cast<const uint32_t*>(&b[i]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {       // relu(x1) ** 2, bf16; * x3, bf16
                    uint32_t r;
                    asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(av[e]), "r"(0u));
                    av[e] = act_mul2(act_mul2(r, r), bv[e]);
                }
            }
            ss[i] = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float lo = act_lo(av[e]), hi = act_hi(av[e]);
                ss[i] = __fadd_rn(ss[i], __fmul_rn(lo, lo));
                ss[i] = __fadd_rn(ss[i], __fmul_rn(hi, hi));
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
#pragma unroll
            for (int i = 0; i < R * VK; ++i) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], d);
#pragma unroll
        for (int i = 0; i < R * VK; ++i) {
            const int vw = warp + (i % VK) * (n >> 5);
            if (lane == i && vw < vwarps) part[(i / VK) * 32 + vw] = ss[i];
        }
        __syncthreads();
        if (R == 1 || warp < rows) {                   // (at least four warps: rows beyond them below)
#pragma unroll 1
            for (int r = R == 1 ? 0 : warp; r < (R == 1 ? 1 : rows); r += n >> 5) {
                float4 p4[VK == 1 ? 3 : 8];
#pragma unroll
                for (int i = 0; i < (VK == 1 ? 3 : 8); ++i)
                    if (4 * i < vwarps) p4[i] = *reinterpret_cast<const float4*>(part + r * 32 + 4 * i);
                float sum = p4[0].x;
#pragma unroll
                for (int i = 0; i < (VK == 1 ? 3 : 8); ++i) {
                    if (i > 0 && 4 * i < vwarps) sum += p4[i].x;
                    if (4 * i + 1 < vwarps) sum += p4[i].y;
                    if (4 * i + 2 < vwarps) sum += p4[i].z;
                    if (4 * i + 3 < vwarps) sum += p4[i].w;
                }
                rstd = __frcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)K), eps)));
                if (R > 1 && lane == 0) rstd_s[r] = rstd;
            }
        }
        if (R > 1) __syncthreads();
    }
    uint32_t mx[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        mx[r] = 0;
        if (R > 1 && MODE != ACT_PLAIN) rstd = rstd_s[r];
#pragma unroll
        for (int j = 0; j < VK; ++j) {
            uint32_t* av = reinterpret_cast<uint32_t*>(&a[r * VK + j]);
            if (MODE != ACT_PLAIN) {
                const uint32_t* wj = reinterpret_cast<const uint32_t*>(&wv[j]);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    av[e] = act_pack(__fmul_rn(__fmul_rn(act_lo(av[e]), rstd), act_lo(wj[e])), __fmul_rn(__fmul_rn(act_hi(av[e]), rstd), act_hi(wj[e])));
            }
            // magnitudes: their bit patterns order like the values, NaN above all (of vectors beyond the row: zeros, or 0 * rstd)
            if ((tid + j * n) * 8 < K) {
#pragma unroll
                for (int e = 0; e < 4; ++e) asm("max.u16x2 %0, %0, %1;" : "+r"(mx[r]) : "r"(av[e] & 0x7FFF7FFFu));
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t m = warp_max_u32(max(mx[r] & 0xFFFFu, mx[r] >> 16));
        if (lane == r) mxp[r * 32 + warp] = m;
    }
    __syncthreads();
    float s = 0.f;
    if (R == 1) {
        s = act_scale(warp_max_u32(lane < (n >> 5) ? mxp[lane] : 0u));
        if (tid == 0) scl[0] = s;
        if (tid == 32) scl[32] = quotient_rcp(s);
    } else {
#pragma unroll 1
        for (int r = warp; r < rows; r += n >> 5) {
            s = act_scale(warp_max_u32(lane < (n >> 5) ? mxp[r * 32 + lane] : 0u));
            if (lane == 0) scl[r] = s;
            if (lane == 1) scl[32 + r] = quotient_rcp(s);
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (R > 1) s = scl[min(r, rows - 1)];
        const uint32_t s2 = (__float_as_uint(s) >> 16) * 0x10001u;
#pragma unroll
        for (int j = 0; j < VK; ++j)
            if ((tid + j * n) * 8 < K && r < rows) store(r, (tid + j * n) * 8, act_quant8(a[r * VK + j], s2));
    }
}

// Rows of at most 8192 elements: one CTA per row, T threads for few rows (a chain of latencies), T / 4 for many gated rows
// (more rows in flight per SM: 1226 rows of 6912 17.3 -> 11.5 us; held in registers, as below, 11.4 us alone and 13.0 us between
// the linears of a prompt).  Dynamic shared memory: the row (gated: both halves) and the norm weight.  x: [M][ld] bf16 (GATED: the
// row holds [x1 (K) | x3 (K)], ld = 2K), w: [K] bf16 norm weight, q: [M][K] int8, s_out: [M] bf16, ss_out: [M] fp32 (MODE 1).
template <bool GATED, int MODE>
__global__ void __launch_bounds__(kActMaxThreads) norm_quant_row_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                        float eps, int K, int8_t* __restrict__ q,
                                                                        __nv_bfloat16* __restrict__ s_out, float* __restrict__ ss_out) {
    extern __shared__ __align__(16) uint8_t act_smem[];
    __shared__ float part[32];
    __shared__ uint32_t mxp[32];
    griddep_launch_dependents();
    const int t = blockIdx.x, tid = threadIdx.x;
    const uint32_t row = smem_u32(act_smem), wrow = row + K * (GATED ? 4 : 2);
    if (MODE != ACT_PLAIN && (t | tid) == 0) act_weight_ahead(w, K);
    griddep_wait();   // the activations come from the previous kernel
    const __nv_bfloat16* xr = x + (size_t)t * (GATED ? 2 * K : K);
    act_row_copy(row, xr, K);
    if (GATED) act_row_copy(row + K * 2, xr + K, K);
    cp_async_commit();
    if (MODE != ACT_PLAIN) act_row_copy(wrow, w, K);
    cp_async_commit();
    const float s = act_row_finish<GATED, MODE>(row, wrow, eps, K, act_row_threads(K), part, mxp, MODE == ACT_SCALE_SUMSQ ? ss_out + t : nullptr,
                                                [&](int k0, const uint4& v) {
        if (MODE == ACT_NORM_ONLY) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(q) + (size_t)t * K + k0) = v;
        else *reinterpret_cast<uint2*>(q + (size_t)t * K + k0) = make_uint2(v.x, v.y);
    });
    if (MODE != ACT_NORM_ONLY && tid == 0) s_out[t] = __float2bfloat16_rn(s);
}

// The same rows ungated, many of them (two per SM and more): what bounds them is no longer the chain but the instructions, so a
// CTA of T / 4 threads keeps its row in registers, four vectors per thread, the butterflies of the four virtual warps side by
// side and one maximum per warp.  Measured between the linears of a prompt, 1226 rows of 2560: 7.8 us through shared
// memory, 5.2 here (9.4 MB: 1.4 us at the copy rate; what is left is the row's chain, one wave of CTAs long).
template <int MODE>
__global__ void __launch_bounds__(kActMaxThreads / 4, 3) norm_quant_rows_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                             float eps, int K, int8_t* __restrict__ q,
                                                                             __nv_bfloat16* __restrict__ s_out, float* __restrict__ ss_out) {
    constexpr int V = 4;
    __shared__ __align__(16) float part[kActMaxThreads / 32];
    __shared__ uint32_t mxp[kActMaxThreads / V / 32];
    griddep_launch_dependents();
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, n = blockDim.x;
    const int vwarps = act_row_threads(K) >> 5;
    uint4 a[V], wv[V];
    griddep_wait();                                    // the activations come from the previous kernel
    const __nv_bfloat16* xr = x + (size_t)t * K;
#pragma unroll
    for (int j = 0; j < V; ++j) a[j] = (tid + j * n) * 8 < K ? ld_cg_128(xr + (tid + j * n) * 8) : make_uint4(0, 0, 0, 0);
    float rstd = 1.f;
    if (MODE != ACT_PLAIN) {
        float ss[V];
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const uint32_t av[4] = {a[j].x, a[j].y, a[j].z, a[j].w};
            ss[j] = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float lo = act_lo(av[i]), hi = act_hi(av[i]);
                ss[j] = __fadd_rn(ss[j], __fmul_rn(lo, lo));
                ss[j] = __fadd_rn(ss[j], __fmul_rn(hi, hi));
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
#pragma unroll
            for (int j = 0; j < V; ++j) ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], d);
#pragma unroll
        for (int j = 0; j < V; ++j)
            if (lane == j) part[(tid + j * n) >> 5] = ss[j];   // (at most 32 virtual warps: V * n <= 1024)
#pragma unroll
        for (int j = 0; j < V; ++j)                    // (asked for this late to spare registers)
            if ((tid + j * n) * 8 < K) wv[j] = *reinterpret_cast<const uint4*>(w + (tid + j * n) * 8);
        __syncthreads();
        float sum = part[0];
#pragma unroll 4
        for (int i = 1; i < vwarps; ++i) sum += part[i];
        if (MODE == ACT_SCALE_SUMSQ && tid == 0) ss_out[t] = sum;
        if (MODE != ACT_SCALE_SUMSQ) rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)K), eps)));
    }
    uint32_t mx = 0;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        if ((tid + j * n) * 8 >= K) continue;
        uint32_t* av = reinterpret_cast<uint32_t*>(&a[j]);
        if (MODE != ACT_PLAIN) {
            const uint32_t wj[4] = {wv[j].x, wv[j].y, wv[j].z, wv[j].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float lo = MODE == ACT_SCALE_SUMSQ ? act_lo(av[i]) : __fmul_rn(act_lo(av[i]), rstd);
                const float hi = MODE == ACT_SCALE_SUMSQ ? act_hi(av[i]) : __fmul_rn(act_hi(av[i]), rstd);
                av[i] = act_pack(__fmul_rn(lo, act_lo(wj[i])), __fmul_rn(hi, act_hi(wj[i])));
            }
            if (MODE == ACT_NORM_ONLY) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(q) + (size_t)t * K + (tid + j * n) * 8) = a[j];
        }
        // magnitudes: their bit patterns order like the values, NaN above all
#pragma unroll
        for (int i = 0; i < 4; ++i) asm("max.u16x2 %0, %0, %1;" : "+r"(mx) : "r"(av[i] & 0x7FFF7FFFu));
    }
    if (MODE == ACT_NORM_ONLY) return;
    mx = warp_max_u32(max(mx & 0xFFFFu, mx >> 16));
    if (lane == 0) mxp[tid >> 5] = mx;
    __syncthreads();
    const float s = act_scale(warp_max_u32(lane < (n >> 5) ? mxp[lane] : 0u));
    const uint32_t s2 = (__float_as_uint(s) >> 16) * 0x10001u;
#pragma unroll
    for (int j = 0; j < V; ++j)
        if ((tid + j * n) * 8 < K) *reinterpret_cast<uint2*>(q + (size_t)t * K + (tid + j * n) * 8) = act_quant8(a[j], s2);
    if (tid == 0) s_out[t] = __float2bfloat16_rn(s);
}

// ---- elementwise kernels of the unfused glue: each replaces a chain of torch operators by one launch with the same
// roundings -----------------------------------------------------------------------------------------------------------
// RoPE on adjacent pairs in fp32 (products and difference rounded separately): x [B][T][H][128] with `ld` elements between
// two tokens, cos / sin fp32 [T][64] (the same for every sequence), out contiguous.  One thread per 8 elements.
__global__ void __launch_bounds__(256) rope_kernel(const __nv_bfloat16* __restrict__ x, long long ld, const float* __restrict__ cos_t,
                                                  const float* __restrict__ sin_t, __nv_bfloat16* __restrict__ out, int T, int H,
                                                  long long items) {
    griddep_launch_dependents();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    griddep_wait();
    if (i >= items) return;
    const int c = (int)(i & 15), h = (int)((i >> 4) % H);
    const long long bt = (i >> 4) / H;
    const int t = (int)(bt % T);
    const uint4 v = ld_cg_128(x + bt * ld + h * 128 + c * 8);
    const float4 cs = *reinterpret_cast<const float4*>(cos_t + (size_t)t * 64 + c * 4), sn = *reinterpret_cast<const float4*>(sin_t + (size_t)t * 64 + c * 4);
    const uint32_t a[4] = {v.x, v.y, v.z, v.w};
    const float cc[4] = {cs.x, cs.y, cs.z, cs.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float p = act_lo(a[e]), q = act_hi(a[e]);
        o[e] = act_pack(__fsub_rn(__fmul_rn(p, cc[e]), __fmul_rn(q, ss[e])), __fadd_rn(__fmul_rn(p, ss[e]), __fmul_rn(q, cc[e])));
    }
    *reinterpret_cast<uint4*>(out + i * 8) = make_uint4(o[0], o[1], o[2], o[3]);
}

// relu(x1) ** 2 * x3 of rows [x1 (K) | x3 (K)], bf16 after every step.
__global__ void __launch_bounds__(256) relu2_gate_kernel(const __nv_bfloat16* __restrict__ x13, __nv_bfloat16* __restrict__ out, int K8, long long items) {
    griddep_launch_dependents();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    griddep_wait();
    if (i >= items) return;
    const long long t = i / K8, c = i - t * K8;
    const uint4 a = ld_cg_128(x13 + (t * 2 * K8 + c) * 8), b = ld_cg_128(x13 + ((t * 2 + 1) * K8 + c) * 8);
    const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        uint32_t r;
        asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(av[e]), "r"(0u));
        o[e] = act_mul2(act_mul2(r, r), bv[e]);
    }
    *reinterpret_cast<uint4*>(out + i * 8) = make_uint4(o[0], o[1], o[2], o[3]);
}

// bf16 -> fp32.  Four values per lane and access, so that a warp's store covers whole lines (eight per lane: half a sector at a
// time), four accesses in flight, from the end: the last values of what the kernel before wrote are still in L2.
// 1226 x 128256 logits: 200 -> 160 us (144 at the copy rate).
__global__ void __launch_bounds__(256) bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ y, long long n) {
    constexpr int U = 4;
    griddep_launch_dependents();
    griddep_wait();
    const long long n4 = n >> 2, chunks = (n4 + U * 256 - 1) / (U * 256);
    for (long long c = chunks - 1 - blockIdx.x; c >= 0; c -= gridDim.x) {
        const long long i0 = c * (U * 256) + threadIdx.x;
        uint2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * 256 < n4) v[u] = __ldcg(reinterpret_cast<const uint2*>(x) + i0 + u * 256);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * 256 < n4)
                __stcs(reinterpret_cast<float4*>(y) + i0 + u * 256, make_float4(act_lo(v[u].x), act_hi(v[u].x), act_lo(v[u].y), act_hi(v[u].y)));
    }
    const long long rest = n4 * 4 + threadIdx.x;
    if (blockIdx.x == 0 && rest < n) y[rest] = __bfloat162float(x[rest]);
}

// Longer rows, staged in shared memory: same arguments, dynamic shared memory K bf16.
template <bool GATED, int MODE>
__global__ void __launch_bounds__(kActMaxThreads) norm_quant_kernel(const __nv_bfloat16* __restrict__ x,
                                                                  const __nv_bfloat16* __restrict__ w, float eps,
                                                                  int K, int8_t* __restrict__ q,
                                                                  __nv_bfloat16* __restrict__ s_out,
                                                                  float* __restrict__ ss_out) {
    extern __shared__ __align__(16) uint8_t act_smem[];
    __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(act_smem);
    __shared__ float scratch[kActMaxThreads / 32];
    griddep_launch_dependents();
    griddep_wait();   // the activations come from the previous kernel
    const int t = blockIdx.x, tid = threadIdx.x;
    const __nv_bfloat16* xr = x + (size_t)t * (GATED ? 2 * K : K);

    // pass 1: stage the row (after the gate, if any) and its sum of squares
    float ss = 0.f;
    for (int k0 = tid * 8; k0 < K; k0 += blockDim.x * 8) {
        const uint4 a = *reinterpret_cast<const uint4*>(xr + k0);
        const __nv_bfloat16* av = reinterpret_cast<const __nv_bfloat16*>(&a);
        __align__(16) __nv_bfloat16 v[8];
        if (GATED) {
            const uint4 b = *reinterpret_cast<const uint4*>(xr + K + k0);
            const __nv_bfloat16* bv = reinterpret_cast<const __nv_bfloat16*>(&b);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float r = fmaxf(__bfloat162float(av[i]), 0.f);
                const float sq = bf16_round_f(r * r);                       // relu(x1) ** 2, bf16
                v[i] = __float2bfloat16_rn(sq * __bfloat162float(bv[i]));   // * x3, bf16
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = av[i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float f = __bfloat162float(v[i]);
            ss = __fadd_rn(ss, __fmul_rn(f, f));
        }
        *reinterpret_cast<uint4*>(row + k0) = *reinterpret_cast<const uint4*>(v);
    }
    float rstd = 1.f;
    if (MODE != ACT_PLAIN) {
        ss = block_reduce(ss, scratch, false);
        if (MODE == ACT_RMSNORM || MODE == ACT_NORM_ONLY) rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
        if (MODE == ACT_SCALE_SUMSQ && tid == 0) ss_out[t] = ss;
    }

    // pass 2: normalise, apply the weight, round to bf16, absmax
    float amax = 0.f;
    for (int k0 = tid * 8; k0 < K; k0 += blockDim.x * 8) {
        uint4 a = *reinterpret_cast<const uint4*>(row + k0);
        __nv_bfloat16* av = reinterpret_cast<__nv_bfloat16*>(&a);
        if (MODE != ACT_PLAIN) {
            const uint4 wv = *reinterpret_cast<const uint4*>(w + k0);
            const __nv_bfloat16* ww = reinterpret_cast<const __nv_bfloat16*>(&wv);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float y = __fmul_rn((MODE == ACT_RMSNORM || MODE == ACT_NORM_ONLY) ? __fmul_rn(__bfloat162float(av[i]), rstd) : __bfloat162float(av[i]),
                                          __bfloat162float(ww[i]));
                av[i] = __float2bfloat16_rn(y);
            }
            if (MODE == ACT_NORM_ONLY) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(q) + (size_t)t * K + k0) = a;
            else *reinterpret_cast<uint4*>(row + k0) = a;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = nan_max(amax, fabsf(__bfloat162float(av[i])));
    }
    if (MODE == ACT_NORM_ONLY) return;
    amax = block_reduce(amax, scratch, true);
    amax = bf16_round_f(amax < 1e-5f ? 1e-5f : amax);
    const float s = bf16_round_f(bf16_round_f(1.0f / amax) * 127.0f);   // 127 / amax as reciprocal * 127, in bf16
    if (tid == 0) s_out[t] = __float2bfloat16_rn(s);

    // pass 3: quantise
    for (int k0 = tid * 16; k0 < K; k0 += blockDim.x * 16) {
        __align__(16) int8_t o[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float p = bf16_round_f(__bfloat162float(row[k0 + i]) * s);
            o[i] = (int8_t)max(min(__float2int_rn(p), 127), -128);
        }
        *reinterpret_cast<uint4*>(q + (size_t)t * K + k0) = *reinterpret_cast<const uint4*>(o);
    }
}

// Tail of a row-parallel linear after the all-reduce: buf holds the summed fp32 partial outputs
// [M][N] followed by the summed per-token sums of squares [M];
// out = bf16(buf[t][n] * rsqrt(ss[t] / full_width + eps) * ws) (+ residual, rounded again).
__global__ void __launch_bounds__(256) tp_finish_kernel(const float* __restrict__ buf, const __nv_bfloat16* ws,
                                                        float eps, int full_width, int M, int N,
                                                        const __nv_bfloat16* residual, __nv_bfloat16* out) {
    griddep_launch_dependents();
    griddep_wait();
    const float w = __bfloat162float(ws[0]);
    const long long total = (long long)M * N;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(i / N);
        const float rstd = rsqrtf(buf[total + t] / (float)full_width + eps);
        __nv_bfloat16 v = __float2bfloat16_rn((buf[i] * rstd) * w);
        if (residual) v = __float2bfloat16_rn(__bfloat162float(residual[i]) + __bfloat162float(v));
        out[i] = v;
    }
}


// ---------------------------------------------------------------------------------------------
// Row-parallel tail with the all-reduce fused in (one process per GPU, peer memory over NVLink),
// as a reduce-scatter followed by an all-gather inside ONE launch per rank.
// Every rank's fp32 partial outputs [M*N] and partial sums of squares [M] sit in a buffer that
// all ranks have mapped (symmetric memory), and so does every rank's bf16 output [M*N].
//   1. block 0 tells every peer "my partials of this call are complete" by a system-scope atomic
//      increment of this rank's counter in the peer's flag array (the partials were written by
//      the previous kernel of the stream, so they are complete when this kernel starts);
//   2. every block waits until all peers' counters in the LOCAL flag array have reached this
//      call's number (runs so far + 1) - a spin bounded by `limit_ns` of the global timer;
//   3. rank r owns the r-th slice of the M*N outputs: its blocks pull that slice of all ranks'
//      partials with plain 16-byte loads (own from local memory, the others over NVLink; no
//      multicast), add them in rank order, apply rsqrt(sum_sq/width + eps) * ws (+ residual) and
//      push the finished bf16 values into EVERY rank's output buffer with plain peer stores.
//      Per rank (T-1)/T * (4 + 2) * M*N bytes cross NVLink instead of (T-1) * 4 * M*N for
//      "every rank pulls everything"; each output element is computed once, so all ranks hold
//      bit-identical activations;
//   4. the last block of the rank to finish signals "my slice has been pushed and I have read
//      your partials" to every peer (second counter set), waits (bounded) for the same signal
//      from all peers and advances the local run counter.  When the kernel ends, this rank's
//      output is complete AND no peer still reads this rank's partial buffer, so the buffers of
//      a call site may be reused by the very next call: no ordering rule is left to the caller.
// When a wait runs out the kernel reports ST_WAIT_TIMEOUT through `status`, fills its own output
// with bf16 NaN (a missed peer shows up downstream instead of as stale data) and returns.
struct TpPeers {
    const float* buf[8];      // partial buffers of ranks 0..world-1 (this rank's own pointer included)
    unsigned int* flag[8];    // flag arrays of ranks 0..world-1: flag[r][j] = "partials ready" calls signalled by
                              // rank j, flag[r][8 + j] = "slice pushed" calls signalled by rank j
    __nv_bfloat16* out[8];    // output buffers of ranks 0..world-1
};

// Bounded wait until *f (system scope) has reached `expected`.
__device__ __forceinline__ bool wait_counter_sys(const volatile unsigned int* f, unsigned int expected,
                                                 unsigned long long limit_ns) {
    const unsigned long long t_start = global_timer_ns();
    for (unsigned int it = 0; it < (1u << 26); ++it) {   // wall-time limit below; the count is a second fence
        unsigned int v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
        if ((int)(v - expected) >= 0) return true;
        if (it > 64) {
            __nanosleep(200);
            if (global_timer_ns() - t_start > limit_ns) return false;
        }
    }
    return false;
}

__global__ void __launch_bounds__(256) tp_allreduce_finish_kernel(const TpPeers peers, int rank, int world,
                                                                  unsigned int* runs, unsigned int* done_blocks,
                                                                  const __nv_bfloat16* ws, float eps, int full_width,
                                                                  int M, int N, const __nv_bfloat16* residual,
                                                                  int* status, unsigned long long limit_ns) {
    __shared__ unsigned int expected_s;
    __shared__ int failed_s;
    __shared__ int last_s;
    griddep_launch_dependents();
    griddep_wait();            // the partials come from the previous kernel of the stream
    const int tid = threadIdx.x;
    if (tid == 0) {
        expected_s = *reinterpret_cast<volatile unsigned int*>(runs) + 1u;
        failed_s = 0;
    }
    if (blockIdx.x == 0 && tid < world && tid != rank) {
        __threadfence_system();
        atomicAdd_system(peers.flag[tid] + rank, 1u);
    }
    __syncthreads();
    const unsigned int expected = expected_s;
    if (tid < world && tid != rank && !wait_counter_sys(peers.flag[rank] + tid, expected, limit_ns)) failed_s = 1;
    __syncthreads();
    const bool failed = failed_s != 0;
    __nv_bfloat16* out = peers.out[rank];
    const long long total = (long long)M * N;          // N is a multiple of 4
    const long long vecs = total >> 2;

    if (!failed) {
        const float w = __bfloat162float(ws[0]);
        const long long v0 = vecs * rank / world, v1 = vecs * (rank + 1) / world;   // this rank's slice
        for (long long vi = v0 + (long long)blockIdx.x * blockDim.x + tid; vi < v1; vi += (long long)gridDim.x * blockDim.x) {
            const long long i = vi << 2;
            const int t = (int)(i / N);
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            float ss = 0.f;
            for (int r = 0; r < world; ++r) {
                float4 v;
                float q;
                asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                             : "l"(peers.buf[r] + i));
                asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(q) : "l"(peers.buf[r] + total + t));
                acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
                ss += q;
            }
            const float rstd = rsqrtf(ss / (float)full_width + eps);
            const float y[4] = {acc.x, acc.y, acc.z, acc.w};
            __align__(8) __nv_bfloat16 o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[e] = __float2bfloat16_rn((y[e] * rstd) * w);
                if (residual) o[e] = __float2bfloat16_rn(__bfloat162float(residual[i + e]) + __bfloat162float(o[e]));
            }
            const uint2 packed = *reinterpret_cast<const uint2*>(o);
            for (int r = 0; r < world; ++r) *reinterpret_cast<uint2*>(peers.out[r] + i) = packed;   // all-gather by push
        }
    } else {
        if (tid == 0) atomicExch(status, 4 /* ST_WAIT_TIMEOUT */);
        for (long long vi = (long long)blockIdx.x * blockDim.x + tid; vi < vecs; vi += (long long)gridDim.x * blockDim.x)
            *reinterpret_cast<uint2*>(out + (vi << 2)) = make_uint2(0x7FC07FC0u, 0x7FC07FC0u);
    }

    // the last block of this rank to get here closes the call
    __threadfence_system();    // this thread's pushes are visible system-wide before the block is counted
    __syncthreads();
    if (tid == 0) {
        const unsigned int prev = atomicAdd(done_blocks, 1u);
        last_s = prev == gridDim.x - 1;
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence_system();
    if (tid < world && tid != rank) {
        bool ok = true;
        if (!failed) {
            atomicAdd_system(peers.flag[tid] + 8 + rank, 1u);       // my slice sits in your output; I am done with your partials
            ok = wait_counter_sys(peers.flag[rank] + 8 + tid, expected, limit_ns);
        }
        if (!ok) failed_s = 2;
    }
    __syncthreads();
    if (failed_s == 2) {
        // a peer's slice never arrived: the whole output is suspect
        if (tid == 0) atomicExch(status, 4 /* ST_WAIT_TIMEOUT */);
        for (long long vi = tid; vi < vecs; vi += blockDim.x)
            *reinterpret_cast<uint2*>(out + (vi << 2)) = make_uint2(0x7FC07FC0u, 0x7FC07FC0u);
    }
    if (tid == 0) {
        *done_blocks = 0u;
        *reinterpret_cast<volatile unsigned int*>(runs) = expected;
        __threadfence();
    }
}

}  // namespace tsp
