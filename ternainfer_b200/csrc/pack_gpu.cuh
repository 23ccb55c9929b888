// Weight packer on the GPU for sm_100a: int8 ternary [N][K] -> the four packed arrays (format: packer_host.cu).
//
// One warp per 64x64 tile: lane (g, q) reads the 16 consecutive k of its eight rows with 16-byte loads, which are its four
// bitmap words.  Three launches: bitmaps, per-tile counts and quarter offsets; a scan of the padded counts; the sign words (the
// weights are read again - the sign stream's place is not known before the scan).  Bound by reading the weights, and for one
// layer by launches and the host's wait for the size of the sign stream: 3840 x 2560 took 1.07 ms as torch
// operators with 64-bit temporaries and two boolean-index synchronisations, 0.05 ms as these kernels called from Python, 0.033 ms
// from the native call site, which reads the size as soon as the scan has written it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tsp {

constexpr int kPackWarps = 8;

// Bit e: byte e of x is not zero / is negative.
__device__ __forceinline__ uint32_t pack_nonzero4(uint32_t x) { return ((__vcmpne4(x, 0u) & 0x01010101u) * 0x01020408u) >> 24; }
__device__ __forceinline__ uint32_t pack_negative4(uint32_t x) { return (((x >> 7) & 0x01010101u) * 0x01020408u) >> 24; }

// The lane's four bitmap words (and with SIGNS the words that mark the negative ones) of a tile.
template <bool SIGNS>
__device__ __forceinline__ void pack_words(const int8_t* tile, int K, int lane, uint32_t (&nz)[4], uint32_t (&neg)[4]) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        nz[r] = neg[r] = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(tile + (size_t)(16 * r + 8 * h + g) * K + 16 * q));
            const uint32_t b[4] = {v.x, v.y, v.z, v.w};   // k 4j .. 4j+3: nibble 2j + h
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                nz[r] |= (pack_nonzero4(b[j]) & 15u) << (8 * j + 4 * h);
                if (SIGNS) neg[r] |= (pack_negative4(b[j]) & 15u) << (8 * j + 4 * h);
            }
        }
    }
}

// The bits of x at the set bits of m, moved to the low end in order (H. S. Warren, Hacker's Delight, 7-4): in step i the bits move by
// 2^i whose number of clear bits of m below them has bit i set; parallel prefix by exclusive or finds these.  (A loop over the
// set bits runs as long as the lane with most: sign words of 3840 x 2560 10.0 us, 6.6 so.)
__device__ __forceinline__ uint32_t pack_compress(uint32_t x, uint32_t m) {
    uint32_t below = ~m << 1;
    x &= m;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        uint32_t odd = below ^ (below << 1);
        odd ^= odd << 2, odd ^= odd << 4, odd ^= odd << 8, odd ^= odd << 16;
        const uint32_t mv = odd & m, t = x & mv;
        m = (m ^ mv) | (mv >> (1 << i));
        x = (x ^ t) | (t >> (1 << i));
        below &= ~odd;
    }
    return x;
}

// Inclusive prefix over the warp.
__device__ __forceinline__ int warp_inclusive(int v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

// bitmap, quarter offsets, and tile_off[t + 1] = non-zeros of tile t rounded up to 32
__global__ void __launch_bounds__(kPackWarps * 32) pack_bitmap_kernel(const int8_t* __restrict__ w, int N, int K, uint4* __restrict__ bitmap,
                                                                     int* __restrict__ tile_off, uint16_t* __restrict__ quarters) {
    const int lane = threadIdx.x & 31, KT = K >> 6;
    const long long t = (long long)blockIdx.x * kPackWarps + (threadIdx.x >> 5);
    if (t >= (long long)(N >> 6) * KT) return;
    const long long rt = t / KT;
    uint32_t nz[4], neg[4];
    pack_words<false>(w + (size_t)rt * 64 * K + (size_t)(t - rt * KT) * 64, K, lane, nz, neg);
    bitmap[t * 32 + lane] = make_uint4(nz[0], nz[1], nz[2], nz[3]);
    const int incl = warp_inclusive(__popc(nz[0]) + __popc(nz[1]) + __popc(nz[2]) + __popc(nz[3]), lane);
    if ((lane & 7) == 7) {
        if (lane < 31) quarters[t * 3 + (lane >> 3)] = (uint16_t)incl;
        else tile_off[t + 1] = (incl + 31) & ~31;
    }
}

// tile_off[1 ..] -> inclusive sums, tile_off[0] = 0; one block.  *total (pinned host memory): the sum.
__global__ void __launch_bounds__(1024) pack_scan_kernel(int* __restrict__ tile_off, long long tiles, long long* total) {
    __shared__ int part[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    long long carry = 0;
    if (tid == 0) tile_off[0] = 0;
    for (long long base = 0; base < tiles; base += 4096) {   // four consecutive counts per thread
        int v[4], sum = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const long long t = base + tid * 4 + i;
            v[i] = t < tiles ? tile_off[t + 1] : 0;
            sum += v[i];
        }
        const int incl = warp_inclusive(sum, lane);
        __syncthreads();
        if (lane == 31) part[warp] = incl;
        __syncthreads();
        const int parts = warp_inclusive(part[lane], lane);   // every warp: prefix over the warps
        const int before = warp ? __shfl_sync(0xffffffffu, parts, warp - 1) : 0, all = __shfl_sync(0xffffffffu, parts, 31);
        long long at = carry + before + incl - sum;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const long long t = base + tid * 4 + i;
            at += v[i];
            if (t < tiles) tile_off[t + 1] = (int)at;
        }
        carry += all;
    }
    if (tid == 0) {
        *reinterpret_cast<volatile long long*>(total) = carry;
        __threadfence_system();
    }
}

// sign words of every tile; the four words behind the last tile are cleared
__global__ void __launch_bounds__(kPackWarps * 32) pack_signs_kernel(const int8_t* __restrict__ w, int N, int K, const int* __restrict__ tile_off,
                                                                    uint32_t* __restrict__ signs) {
    __shared__ uint32_t bits[kPackWarps][132];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, KT = K >> 6;
    const long long t = (long long)blockIdx.x * kPackWarps + warp, tiles = (long long)(N >> 6) * KT;
    if (t >= tiles) return;
    const long long rt = t / KT;
    uint32_t nz[4], neg[4], *out = bits[warp];
    for (int i = lane; i < 132; i += 32) out[i] = 0;
    pack_words<true>(w + (size_t)rt * 64 * K + (size_t)(t - rt * KT) * 64, K, lane, nz, neg);
    const int total = __popc(nz[0]) + __popc(nz[1]) + __popc(nz[2]) + __popc(nz[3]);
    int pos = warp_inclusive(total, lane) - total;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t packed = pack_compress(neg[r], nz[r]);
        const int n = __popc(nz[r]), sh = pos & 31;
        if (packed) {
            atomicOr(&out[pos >> 5], packed << sh);
            if (sh + n > 32) atomicOr(&out[(pos >> 5) + 1], packed >> (32 - sh));
        }
        pos += n;
    }
    __syncwarp();
    const int first = tile_off[t] >> 5, words = (tile_off[t + 1] >> 5) - first;
    for (int i = lane; i < words; i += 32) signs[first + i] = out[i];
    if (t == tiles - 1 && lane < 4) signs[first + words + lane] = 0;
}

}  // namespace tsp
