// libternaspmm.so for NVIDIA B200 (sm_100a): the extern "C" surface declared
// in include/ternaspmm.h and the host-side launch logic behind it.
//
// The entry points mirror kernels/TernaSpMM.cu of Gu-J/TernaInfer (same names,
// argument order and meaning); everything behind them is new.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <limits.h>
#include <stdlib.h>
#include <math.h>

#include <algorithm>
#include <vector>

#define TERNASPMM_TYPES_ONLY   // the item struct of the work lists; the prototypes use plain-C stand-in types
#include "ternaspmm.h"

#include "act_quant.cuh"
#include "attn_decode.cuh"
#include "attn_prefill.cuh"
#include "dense_pair.cuh"
#include "dense_prefill.cuh"
#include "lm_head.cuh"
#include "mma_rate_probe.cuh"
#include "pack_gpu.cuh"
#include "spmm_large_m.cuh"
#include "spmm_list.cuh"
#include "spmm_small_m.cuh"
#include "w2_pair.cuh"
#include "w2_small.cuh"

namespace tsp {

__device__ int g_status_word = 0;

static int* status_device_ptr() {
    // One address per device; looked up once per device, outside any capture.
    static int* ptrs[64] = {nullptr};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!ptrs[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_status_word) != cudaSuccess) return nullptr;
        ptrs[dev] = static_cast<int*>(p);
    }
    return ptrs[dev];
}

static thread_local int t_host_status = ST_OK;

static int device_sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!sms[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        sms[dev] = v;
    }
    return sms[dev];
}

// Launch-shape knobs.  The product reads ONE environment variable, TERNASPMM_PDL=0 (launch without
// programmatic dependent launch).  The others exist only in tuning builds (-DTSP_TUNING):
//   TERNASPMM_FAT=0              small-batch kernel: never use the one-CTA-per-SM shape
//   TERNASPMM_STAGE=0            small-batch kernel: no shared-memory slot for a warp's second tile
//   TERNASPMM_RPC2=0             small-batch kernel: never put two row tiles into one fat CTA
//   TERNASPMM_FORCE_S / _FORCE_W small-batch kernel: this K split and this many warps per CTA
//   TERNASPMM_CTAS_PER_SM_X10    small-batch kernel, thin shape: about that many CTAs per SM (x10)
//   TERNASPMM_MAX_WARPS          small-batch kernel, thin shape: cap on warps per CTA
//   TERNASPMM_CLUSTER_COST_X10   small-batch kernel, thin shape: price of a K split in tenths of a tile time
//   TERNASPMM_LARGE_MIN_M        smallest token count sent to the tcgen05 kernel (default 33)
//   TERNASPMM_LARGE_SPLIT=0      tcgen05 kernel without its cluster K split
//   TERNASPMM_LIST_WARPS         work-list kernel at 8 tokens: 20 (default), 24 or 28 warps per CTA
struct Tuning {
    int ctas_x10 = 0, max_warps = 0, pdl = 1, large_min_m = 33, large_split = 1, cluster_cost_x10 = 0, fat = 1,
        force_s = 0, force_w = 0, stage = 1, rpc2 = 1, list_warps = 20;
    Tuning() {
        if (const char* e = getenv("TERNASPMM_PDL")) pdl = atoi(e) != 0;
#ifdef TSP_TUNING
        if (const char* e = getenv("TERNASPMM_CTAS_PER_SM_X10")) ctas_x10 = atoi(e);
        if (const char* e = getenv("TERNASPMM_MAX_WARPS")) max_warps = atoi(e);
        if (const char* e = getenv("TERNASPMM_LARGE_MIN_M")) large_min_m = atoi(e) > 0 ? atoi(e) : large_min_m;
        if (const char* e = getenv("TERNASPMM_LARGE_SPLIT")) large_split = atoi(e) != 0;
        if (const char* e = getenv("TERNASPMM_CLUSTER_COST_X10")) cluster_cost_x10 = atoi(e);
        if (const char* e = getenv("TERNASPMM_FAT")) fat = atoi(e);
        if (const char* e = getenv("TERNASPMM_STAGE")) stage = atoi(e) != 0;
        if (const char* e = getenv("TERNASPMM_RPC2")) rpc2 = atoi(e) != 0;
        if (const char* e = getenv("TERNASPMM_FORCE_S")) force_s = atoi(e);
        if (const char* e = getenv("TERNASPMM_FORCE_W")) force_w = atoi(e);
        if (const char* e = getenv("TERNASPMM_LIST_WARPS")) list_warps = atoi(e);
#endif
    }
};
static const Tuning& tuning() {
    static Tuning t;
    return t;
}

// Shape of the most recent launch made on this thread (test hook, see ternaspmm_last_launch_shape).
struct LaunchEcho {
    int kernel = 0, tokens_per_pass = 0, splits = 0, warps = 0, row_tiles_per_cta = 0, ctas = 0;
};
static thread_local LaunchEcho t_echo;

// Limit of the device-side waits on a peer (fused tensor-parallel tail), in nanoseconds of the GPU's
// global timer; changed with ternaspmm_set_wait_limit_ms.
static unsigned long long g_wait_limit_ns = 1000ull * 1000 * 1000;

struct LaunchShape {
    int splits, warps;
    int rpc = 1;   // row tiles per CTA (fat shape only)
};

// K split (= cluster size, at most 8) and warps per CTA.  Take the smallest
// number of tiles per warp for which every CTA is resident at once (one wave:
// `warp_slots` warps and at most 2 CTAs per SM at this kernel's register and
// shared-memory budget), and for that the smallest cluster.
// TERNASPMM_CTAS_PER_SM_X10 > 0 overrides with "about that many CTAs per SM".
static LaunchShape choose_shape(int RT, int KT, int token_blocks, int max_warps, int warp_slots) {
    const int sms = device_sm_count();
    const long long rows = (long long)RT * token_blocks;
    const int max_w = tuning().max_warps > 0 && tuning().max_warps < max_warps ? tuning().max_warps : max_warps;
    const int max_s = KT > 1 ? (KT / 2 < 8 ? KT / 2 : 8) : 1;
    if (tuning().force_s > 0 && tuning().force_w > 0) return {tuning().force_s, tuning().force_w};
    if (tuning().ctas_x10 > 0) {
        const long long target = (long long)tuning().ctas_x10 * sms / 10;
        int s = (int)((target + rows - 1) / rows);
        s = s > max_s ? max_s : (s < 1 ? 1 : s);
        const int nt = (KT + s - 1) / s;
        return {s, nt < 2 ? 2 : (nt > max_w ? max_w : nt)};
    }
    // cost of a candidate in tenths of a tile time: tiles per warp, plus the cluster reduction when K is split
    LaunchShape best = {0, 0};
    long long best_cost = -1;
    for (int tpw = 1; tpw <= KT; ++tpw)
        for (int s = 1; s <= max_s; ++s) {
            const int nt = (KT + s - 1) / s;
            int w = (nt + tpw - 1) / tpw;
            if (w > max_w) continue;
            if (w < 2) w = 2;
            int per_sm = warp_slots / w;
            per_sm = per_sm > 2 ? 2 : per_sm;
            if (per_sm < 1 || rows * s > (long long)sms * per_sm) continue;
            const long long cost = 10ll * tpw + (s > 1 ? tuning().cluster_cost_x10 : 0);
            if (best_cost < 0 || cost < best_cost) best = {s, w}, best_cost = cost;
        }
    if (best_cost >= 0) return best;
    // more than one wave whatever we do: no K split, full CTAs
    return {1, KT < 2 ? 2 : (KT > max_w ? max_w : KT)};
}

// "Fat" shape: one CTA per SM with as many warps as the register file allows.  Measured on the
// BitNet-2B layers (QKV at 8 tokens: 5.3 -> 3.4 us), a launch whose row tiles fit the SMs once is
// fastest without any K split as long as a warp gets at most 2 (3 for 32-token blocks) tiles, and
// otherwise with the smallest split that gets there while the clusters still fit the chip in one
// wave; more CTAs than SMs (two thin CTAs per SM, each building its own tables) are slower.  A fat
// launch also leaves SMs free, on which the next launch of the stream starts its prologue at once
// (down projection inside the layer sweep: +4 % on the whole sweep against the thin shape).
// Returns splits = 0 when the thin shape should be used instead.
static LaunchShape choose_fat(int RT, int KT, int token_blocks, int max_warps, int mt) {
    const int sms = device_sm_count();
    const long long rows = (long long)RT * token_blocks;
    if (!tuning().fat) return {0, 0};
    // more row tiles than SMs, but at most twice as many: two row tiles per CTA, half of the warps each
    if (rows > sms && token_blocks == 1 && RT % 2 == 0 && RT / 2 <= sms && tuning().rpc2)
        return {1, max_warps & ~1, 2};
    if (rows > sms) return {0, 0};
    const int max_s = KT > 1 ? (KT / 2 < 8 ? KT / 2 : 8) : 1;
    const int limit = mt >= 4 ? 3 : 2;
    int pick = 0;
    for (int s = 1; s <= max_s && rows * s <= sms; ++s) {
        const int nt = (KT + s - 1) / s;
        pick = s;                                            // the largest feasible split if none reaches the limit
        if ((nt + max_warps - 1) / max_warps <= limit) break;
    }
    if (pick == 0) return {0, 0};
    const int nt = (KT + pick - 1) / pick;
    return {pick, nt < 2 ? 2 : (nt > max_warps ? max_warps : nt)};
}

template <int MT, int MAXW, int MINB>
static cudaError_t launch_small_m(SpmmParams& p, int token_blocks, int warp_slots, cudaStream_t stream,
                                  LaunchShape preset = {0, 0}) {
    using L = SmallMSmem<MT, MINB == 1 ? 2 : 1>;
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    auto kern = spmm_small_m_kernel<MT, MAXW, MINB>;
    const LaunchShape shape = preset.splits > 0 ? preset : choose_shape(p.N / 64, p.K / 64, token_blocks, MAXW, warp_slots);
    p.splits = shape.splits;
    const int warps = shape.warps;
    // one CTA per SM (MINB == 1) leaves room for a 4 KB slot per warp: second tiles are decoded before the wait
    // (only the warps that have a second tile need one: the first nt - warps of them)
    const int nt = (p.K / 64 + shape.splits - 1) / shape.splits;
    p.rpc = shape.rpc;
    const int wpr = warps / shape.rpc;   // warps that share a row tile
    const int slots = (MINB == 1 && tuning().stage && nt > wpr) ? (shape.rpc == 2 ? warps : std::min(warps, nt - warps)) : 0;
    p.stage_second = slots > 0 ? 1 : 0;
    const int smem_bytes = L::total + slots * 4096;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             L::total + (MINB == 1 ? MAXW * 4096 : 0));
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    const int RT = p.N / 64;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.splits, RT / shape.rpc, token_blocks);
    cfg.blockDim = dim3(warps * 32, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // Programmatic dependent launch: this kernel may start while the previous
    // kernel of the stream still runs; it prefetches its (immutable) weights
    // and waits (griddepcontrol.wait) before touching activations or outputs.
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 2 : 1;
    t_echo = {MINB == 1 ? 1 : 2, MT * 8, p.splits, warps, shape.rpc, (int)(cfg.gridDim.x * cfg.gridDim.y * cfg.gridDim.z)};
    return cudaLaunchKernelEx(&cfg, kern, p);
}

// 2-D tensor map over the activations x[M][K] (int8): tiles of NT tokens x
// 128 k, 128-byte swizzle, out-of-range rows and columns read as zero.
static thread_local int t_inject_encode_failure = 0;   // test hook: the next encode on this thread reports failure

// (also used for the dense weight matrix W[N][K]: rows = N, box = 128 rows)
static bool encode_x_map(CUtensorMap* map, const void* x, int M, int K, int NT) {
    if (t_inject_encode_failure) {
        t_inject_encode_failure = 0;
        return false;
    }
    typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || !ptr)
            return false;
        fn = reinterpret_cast<EncodeFn>(ptr);
    }
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)K};
    const cuuint32_t box[2] = {(cuuint32_t)kLgKStep, (cuuint32_t)NT};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(x), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NT, bool DENSE = false>
static cudaError_t launch_large_m(const SpmmParams& p_in, cudaStream_t stream, const int8_t* dense_w = nullptr) {
    using L = LargeMSmem<NT, DENSE>;
    static bool attr_done[64] = {false};
    static int max_clusters[64][4] = {};   // co-resident clusters of 2 / 4 / 8 CTAs (index log2), 0 = not asked yet
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    auto kern = spmm_large_m_kernel<NT, DENSE>;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    SpmmParams p = p_in;
    CUtensorMap map, wmap;
    if (!encode_x_map(&map, p.x, p.M, p.K, NT)) return cudaErrorInvalidValue;   // reported as status 3, nothing is launched
    if (DENSE) {
        if (!encode_x_map(&wmap, dense_w, p.N, p.K, 128)) return cudaErrorInvalidValue;
    } else {
        wmap = map;   // unused by the kernel
    }
    const long long tiles = (long long)((p.N + 127) / 128) * ((p.M + NT - 1) / NT);
    const int sms = device_sm_count(), KS = (p.K + kLgKStep - 1) / kLgKStep;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(L::threads, 1, 1);
    cfg.dynamicSmemBytes = L::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 2 : 1;
    // K split over a cluster when the tiles alone would leave more than half of the SMs idle:
    // the largest cluster of 2/4/8 CTAs that still fits the chip in one wave with >= 2 k-steps per CTA.
    p.splits = 1;
    if (!DENSE && tiles * 2 <= sms && tuning().large_split) {   // (the dense variant has no K split: its callers pick shapes that fill the chip)
        for (int lg = 3; lg >= 1; --lg) {
            const int S = 1 << lg;
            if (tiles * S > sms || KS < 2 * S || NT / S < 16) continue;
            if (max_clusters[dev][lg] == 0) {
                cfg.gridDim = dim3((unsigned)(tiles * S), 1, 1);
                attr[0].val.clusterDim.x = S;
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
                    cudaGetLastError();
                    n = 0;
                }
                max_clusters[dev][lg] = n > 0 ? n : -1;
            }
            if (max_clusters[dev][lg] >= tiles) {
                p.splits = S;
                break;
            }
        }
    }
    attr[0].val.clusterDim.x = p.splits;
    // persistent: one CTA per SM walks over the tiles (with a K split: one tile per cluster)
    cfg.gridDim = dim3(p.splits > 1 ? (unsigned)(tiles * p.splits) : (unsigned)std::min<long long>(tiles, sms), 1, 1);
    t_echo = {DENSE ? 6 : 3, NT, p.splits, L::threads / 32, 2, (int)cfg.gridDim.x};
    return cudaLaunchKernelEx(&cfg, kern, p, map, wmap);
}

// Dense tcgen05 GEMM on CTA pairs (dense_pair.cuh): 256 weight rows x 256 tokens per cluster of two CTAs.
static cudaError_t launch_dense_pair(const SpmmParams& p_in, cudaStream_t stream, const int8_t* dense_w) {
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    auto kern = spmm_dense_pair_kernel;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem::total);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    SpmmParams p = p_in;
    p.splits = 1;
    CUtensorMap map, wmap;   // each CTA of a pair loads 128 tokens and 128 weight rows per stage
    if (!encode_x_map(&map, p.x, p.M, p.K, 128) || !encode_x_map(&wmap, dense_w, p.N, p.K, 128))
        return cudaErrorInvalidValue;   // reported as status 3, nothing is launched
    const long long tiles = (long long)((p.N + kPairRows - 1) / kPairRows) * ((p.M + kPairNT - 1) / kPairNT);
    const int pairs = (int)std::min<long long>(tiles, device_sm_count() / 2);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(PairSmem::threads, 1, 1);
    cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
    cfg.dynamicSmemBytes = PairSmem::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 2 : 1;
    t_echo = {7, kPairNT, 2, PairSmem::threads / 32, 4, (int)cfg.gridDim.x};
    return cudaLaunchKernelEx(&cfg, kern, p, map, wmap);
}

// Scale-segment boundaries of a call (see ws_group): explicit ones, or the reference's rules.
static void set_segments(SpmmParams& p, const int* seg_bounds) {
    if (seg_bounds) {
        for (int i = 0; i < 3; ++i) p.seg_b[i] = (i + 1 < p.ws_num) ? seg_bounds[i] : INT_MAX;
        p.seg_gran = 1;
        return;
    }
    const bool prefill = p.epilogue == EPI_PREFILL;
    p.seg_gran = prefill ? 128 : 8;
    if (p.N == 3840 && (prefill || p.ws_num == 3)) {
        p.seg_b[0] = 2560, p.seg_b[1] = 3200, p.seg_b[2] = INT_MAX;
    } else {
        const int gw = p.ws_num > 0 ? p.N / p.ws_num : p.N;
        p.seg_b[0] = gw, p.seg_b[1] = 2 * gw, p.seg_b[2] = 3 * gw;
    }
}

static void run_spmm(int8_t* x, uint64_t* bitmap, int* tile_off, uint16_t* quarter_off, uint32_t* signs, void* out,
                     __nv_bfloat16* s, __nv_bfloat16* ws, int ws_num, int M, int N, int K, int epilogue,
                     cudaStream_t stream, const int* seg_bounds = nullptr, const __nv_bfloat16* residual = nullptr) {
    t_host_status = ST_OK;
    if (M < 1 || N < 64 || K < 64 || (N % 64) || (K % 64) ||
        (epilogue != EPI_RAW_I32 && epilogue != EPI_F32_DIV && (ws_num < 1 || ws_num > 4))) {
        fprintf(stderr, "ternaspmm: unsupported shape M=%d N=%d K=%d ws_num=%d (need M>=1, N%%64==0, K%%64==0, 1<=ws_num<=4)\n",
                M, N, K, ws_num);
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!x || !bitmap || !tile_off || !quarter_off || !signs || !out || ((epilogue == EPI_DECODE || epilogue == EPI_PREFILL) && (!s || !ws)) || (epilogue == EPI_F32_DIV && !s) ||
        (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(bitmap) & 15) ||
        (reinterpret_cast<uintptr_t>(signs) & 15)) {
        fprintf(stderr, "ternaspmm: null or misaligned pointer (x, bitmap and sign_words must be 16-byte aligned)\n");
        t_host_status = ST_BAD_POINTER;
        return;
    }
    SpmmParams p;
    p.x = x;
    p.bitmap = reinterpret_cast<const uint32_t*>(bitmap);
    p.tile_off = tile_off;
    p.quarter_off = quarter_off;
    p.signs = signs;
    p.out = out;
    p.s = s;
    p.ws = ws;
    p.residual = residual;
    p.ws_num = ws_num;
    p.M = M;
    p.N = N;
    p.K = K;
    p.epilogue = epilogue;
    set_segments(p, seg_bounds);
    p.status = status_device_ptr();
    if (!p.status) {
        t_host_status = ST_LAUNCH;
        return;
    }
    cudaError_t e;
    // Kernel choice.  Up to 32 tokens: the small-batch kernel.  Above that the
    // tcgen05 kernel (with its cluster K split when the 128-row tiles alone
    // would occupy less than half of the SMs), except for small narrow weights
    // at up to 64 tokens, where the small-batch kernel run over two blocks of
    // 32 tokens is still a little faster (measured on the BitNet-2B shapes).
    const bool narrow = M <= 64 && (N + 127) / 128 < device_sm_count() / 2 && (long long)N * K <= (32ll << 20);
    if (M >= tuning().large_min_m && !(narrow && tuning().large_min_m == 33)) {
        p.splits = 1;
        e = M <= 64 ? launch_large_m<64>(p, stream) : (M <= 128 ? launch_large_m<128>(p, stream) : launch_large_m<256>(p, stream));
    } else {
        // thin: up to two CTAs per SM; fat: one CTA per SM with twice the warps (see choose_fat)
        const int RT = N / 64, KT = K / 64;
        if (M <= 8) {
            LaunchShape fat = choose_fat(RT, KT, 1, 28, 1);
            if (tuning().force_s > 0 && tuning().force_w > 14) fat = {tuning().force_s, tuning().force_w};   // tuning runs
            e = fat.splits ? launch_small_m<1, 28, 1>(p, 1, 28, stream, fat) : launch_small_m<1, 14, 2>(p, 1, 28, stream);
        } else if (M <= 16) {
            const LaunchShape fat = choose_fat(RT, KT, 1, 20, 2);
            e = fat.splits ? launch_small_m<2, 20, 1>(p, 1, 20, stream, fat) : launch_small_m<2, 10, 2>(p, 1, 20, stream);
        } else {
            const int tb = (M + 31) / 32;
            const LaunchShape fat = choose_fat(RT, KT, tb, 16, 4);
            e = fat.splits ? launch_small_m<4, 16, 1>(p, tb, 16, stream, fat) : launch_small_m<4, 8, 2>(p, tb, 16, stream);
        }
    }
    if (e != cudaSuccess) {
        fprintf(stderr, "ternaspmm: launch failed: %s\n", cudaGetErrorString(e));
        t_host_status = ST_LAUNCH;
    }
}

__global__ void sleep_kernel(double us) {
    if (threadIdx.x == 0) {
        unsigned long long t0, t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        if (us > 1e6) us = 1e6;  // never wait longer than a second
        const unsigned long long want = (unsigned long long)(us * 1e3);
        for (unsigned it = 0; it < (1u << 28); ++it) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            if (t1 - t0 >= want) break;
            __nanosleep(200);
        }
    }
    __syncwarp();
}

}  // namespace tsp

using namespace tsp;

extern "C" void checkLastCudaError(int line) {
    cudaError_t error = cudaGetLastError();
    if (error != cudaSuccess) {
        printf("Last Cuda Error Detected at line: %d, Error: %s.\n", line, cudaGetErrorString(error));
        exit(EXIT_FAILURE);
    }
}

extern "C" void bitlinear_TernaSpMM(int8_t* x, uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets,
                                    uint32_t* sign_words, __nv_bfloat16* out, __nv_bfloat16* s, __nv_bfloat16* ws,
                                    int ws_num, int M, int N, int K, int /*split_k*/, int32_t* /*workspace*/,
                                    cudaStream_t stream) {
    run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K,
             M <= 64 ? EPI_DECODE : EPI_PREFILL, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void bitlinear_TernaSpMM_decode(int8_t* x, uint64_t* bitmap, int* tile_offsets,
                                           uint16_t* quarter_offsets, uint32_t* sign_words, __nv_bfloat16* out,
                                           __nv_bfloat16* s, __nv_bfloat16* ws, int ws_num, int M, int N, int K,
                                           int /*split_k*/, int32_t* /*workspace*/, cudaStream_t stream) {
    run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K, EPI_DECODE, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void bitlinear_TernaSpMM_prefill(int8_t* x, uint64_t* bitmap, int* tile_offsets,
                                            uint16_t* quarter_offsets, uint32_t* sign_words, __nv_bfloat16* out,
                                            __nv_bfloat16* s, __nv_bfloat16* ws, int ws_num, int M, int N, int K,
                                            int /*split_k*/, int32_t* /*workspace*/, cudaStream_t stream) {
    run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K, EPI_PREFILL, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void bitlinear_TernaSpMM_residual(int8_t* x, uint64_t* bitmap, int* tile_offsets,
                                            uint16_t* quarter_offsets, uint32_t* sign_words, __nv_bfloat16* out,
                                            __nv_bfloat16* s, __nv_bfloat16* ws, int ws_num, int M, int N, int K,
                                            __nv_bfloat16* residual, cudaStream_t stream) {
    run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K,
             M <= 64 ? EPI_DECODE : EPI_PREFILL, stream, nullptr, residual);
    checkLastCudaError(__LINE__);
}

// Large-batch path through a dense workspace: decompress once, then the tensor-core kernel with both
// operands by TMA.  Returns false when the shape is one the on-chip path serves better.
static bool dense_prefill_pays(int M, int N, int K, long long workspace_bytes) {
    // Measured on the BitNet-2B layers (one call, microseconds, on chip / through the workspace):
    //   tokens           256          384          512          1024         2048         4096
    //   3840 x 2560   14.9 / 17.0  18.7 / 17.2  18.9 / 17.7  20.5 / 18.0  32.9 / 24.4  59.0 / 37.8
    //   13824 x 2560  20.3 / 21.6  31.5 / 27.1  32.0 / 28.0  46.7 / 36.1  87.3 / 58.5  168 / 107
    //   2560 x 6912   18.0 / 27.5  26.4 / 27.9  26.7 / 28.4  36.4 / 29.0  62.8 / 45.1  91.5 / 61.9
    // The on-chip kernel decodes every weight tile once per 256 tokens, so from the second token tile on
    // decoding once into the workspace wins; deep, narrow layers (few output tiles, a long K loop) need
    // more tokens, because on chip they split K over a cluster and the pair kernel does not.
    (void)N;
    if (workspace_bytes < (long long)N * K) return false;
    return M >= 384 && (K <= 4096 || M >= 1024);
}

static cudaError_t launch_decompress(const SpmmParams& p, int8_t* dense, cudaStream_t stream) {
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    const int smem_bytes = kLut2Bytes + kLutBytes + 2048 + 256;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(decompress_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    const long long tiles = (long long)(p.N / 64) * (p.K / 64);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min<long long>(device_sm_count(), (tiles + kDecompressWarps - 1) / kDecompressWarps), 1, 1);
    cfg.blockDim = dim3(kDecompressWarps * 32, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, decompress_kernel, p, dense);
}

extern "C" void bitlinear_TernaSpMM_ws(int8_t* x, uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets,
                                       uint32_t* sign_words, __nv_bfloat16* out, __nv_bfloat16* s, __nv_bfloat16* ws,
                                       int ws_num, int M, int N, int K, __nv_bfloat16* residual, void* workspace,
                                       long long workspace_bytes, int path, cudaStream_t stream) {
    const int epilogue = M <= 64 ? EPI_DECODE : EPI_PREFILL;
    const bool dense = path == 2 || (path == 0 && workspace && !(reinterpret_cast<uintptr_t>(workspace) & 127) &&
                                    dense_prefill_pays(M, N, K, workspace_bytes));   // (a workspace that cannot be used is not an error)
    if (!dense) {
        run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K, epilogue, stream, nullptr,
                 residual);
        checkLastCudaError(__LINE__);
        return;
    }
    t_host_status = ST_OK;
    if (M < 1 || N < 64 || K < 64 || (N % 64) || (K % 64) || ws_num < 1 || ws_num > 4) {
        fprintf(stderr, "ternaspmm: unsupported shape M=%d N=%d K=%d ws_num=%d\n", M, N, K, ws_num);
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!x || !bitmap || !tile_offsets || !quarter_offsets || !sign_words || !out || !s || !ws || !workspace ||
        workspace_bytes < (long long)N * K || (reinterpret_cast<uintptr_t>(x) & 15) ||
        (reinterpret_cast<uintptr_t>(bitmap) & 15) || (reinterpret_cast<uintptr_t>(sign_words) & 15) ||
        (reinterpret_cast<uintptr_t>(workspace) & 127)) {
        fprintf(stderr, "ternaspmm: bitlinear_TernaSpMM_ws: null or misaligned pointer, or a workspace below N*K bytes "
                        "(workspace: 128-byte aligned)\n");
        t_host_status = ST_BAD_POINTER;
        return;
    }
    SpmmParams p = {};
    p.x = x, p.bitmap = reinterpret_cast<const uint32_t*>(bitmap), p.tile_off = tile_offsets, p.quarter_off = quarter_offsets;
    p.signs = sign_words, p.out = out, p.s = s, p.ws = ws, p.residual = residual;
    p.ws_num = ws_num, p.M = M, p.N = N, p.K = K, p.epilogue = epilogue, p.splits = 1;
    set_segments(p, nullptr);
    p.status = status_device_ptr();
    if (!p.status) {
        t_host_status = ST_LAUNCH;
        return;
    }
    int8_t* dense_w = static_cast<int8_t*>(workspace);
    cudaError_t e = cudaSuccess;
#ifdef TSP_TUNING
    static const int tune_nt = getenv("TERNASPMM_DENSE_NT") ? atoi(getenv("TERNASPMM_DENSE_NT")) : 0;
    static const int tune_skip = getenv("TERNASPMM_DENSE_SKIP_DECOMPRESS") ? atoi(getenv("TERNASPMM_DENSE_SKIP_DECOMPRESS")) : 0;
    if (!tune_skip) e = launch_decompress(p, dense_w, stream);
    static const int tune_pair = getenv("TERNASPMM_DENSE_PAIR") ? atoi(getenv("TERNASPMM_DENSE_PAIR")) : 1;
    if (e == cudaSuccess)
        e = (M <= 128 || tune_nt == 128) ? launch_large_m<128, true>(p, stream, dense_w)
            : (tune_pair ? launch_dense_pair(p, stream, dense_w) : launch_large_m<256, true>(p, stream, dense_w));
#else
    e = launch_decompress(p, dense_w, stream);
    if (e == cudaSuccess)
        e = M <= 128 ? launch_large_m<128, true>(p, stream, dense_w) : launch_dense_pair(p, stream, dense_w);
#endif
    if (e != cudaSuccess) {
        fprintf(stderr, "ternaspmm: launch failed: %s\n", cudaGetErrorString(e));
        t_host_status = ST_LAUNCH;
    }
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_accumulate_i32(int8_t* x, uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets,
                                         uint32_t* sign_words, int32_t* out, int M, int N, int K,
                                         cudaStream_t stream) {
    run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, nullptr, nullptr, 1, M, N, K, EPI_RAW_I32,
             stream);
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_linear_segments(int8_t* x, uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets,
                                         uint32_t* sign_words, __nv_bfloat16* out, __nv_bfloat16* s,
                                         __nv_bfloat16* ws, int ws_num, int M, int N, int K, int seg1, int seg2,
                                         int seg3, int prefill_form, cudaStream_t stream) {
    const int b[3] = {seg1, seg2, seg3};
    const int epi = prefill_form < 0 ? (M <= 64 ? EPI_DECODE : EPI_PREFILL) : (prefill_form ? EPI_PREFILL : EPI_DECODE);
    run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K, epi, stream, b);
    checkLastCudaError(__LINE__);
}

// The tcgen05 kernels release the next launch before they allocate tensor memory, and tcgen05.alloc waits without a limit.  So the CTAs
// that shared memory lets onto one SM must never ask for more columns than it has: a later launch that took them first would wait for
// an earlier one that waits for the columns.
struct TmemUse { int smem, columns; };
constexpr TmemUse kTmemUse[] = {{LargeMSmem<64>::total, 2 * 64}, {LargeMSmem<128>::total, 2 * 128}, {LargeMSmem<256>::total, 2 * 256},
                                {LargeMSmem<128, true>::total, 2 * 128}, {LargeMSmem<256, true>::total, 2 * 256}, {PairSmem::total, 2 * kPairNT},
                                {W2PairSmem::total, 512}, {kTileMinSmem, kTileCols}};
constexpr int most_tmem_columns(int smem) {          // of CTAs of these kernels that fit this much shared memory, 1 KB each for the system
    int most = 0;
    for (const TmemUse& k : kTmemUse)
        if (k.smem + 1024 <= smem) most = std::max(most, k.columns + most_tmem_columns(smem - k.smem - 1024));
    return most;
}
static_assert(most_tmem_columns(228 * 1024) <= 512, "CTAs that fit an SM side by side would compete for tensor memory");

// ---- linears on two-bit weights (w2_small.cuh) -----------------------------------------------------
constexpr int kW2MaxSmem = 227 * 1024;
// Whether the mma.sync kernel runs a call on int8 activations: up to 4 tokens, up to 8 where a CTA has three strips at most, and activations that
// leave shared memory for a ring - from five tokens on, where an SM has more than one strip, a small part of it, so that the next launch's CTA or
// a front-end's finds room.  A narrow layer's tiles pay for the exchange between K slices, and a call of them for a tensor map and a search on the
// host.  us per call in a stream of such calls, mma.sync / tensor-memory tiles, at 5 and 8 tokens: 2560 x 2560 2.5 / 3.2, 2.7 / 3.2, 2560 x 6912 3.8 / 4.3,
// 4.1 / 4.4, 5120 x 5120 4.1 / 4.8, 4.6 / 4.9, 1280 x 8192 at 8 3.5 / 4.4; eager module calls of 2560 x 2560 at 5 8.9 / 9.4.  Not with longer rows (behind a norm
// 2560 x 10240 at 8 12.6 / 10.2; but 2560 x 6912 at 8 inside the 30-layer model, where other kernels stand between: 1123 us a token, 1142 with tiles),
// nor where K is short (2560 x 256 2.2 / 2.3, 2.4 / 2.3; 6912 x 1024 behind the quantiser at 8 25 % more), nor on wider layers: alone they are even
// (13824 x 2560 5.1 / 5.2, 5.2 / 5.1), but between other kernels the tiles' expansion is done when those end (that model at batch 8 with gate-up by
// mma.sync 1164).
static bool w2_small_takes(int M, int N, int K) {
    const int strips = N / 16, sms = device_sm_count();
    const long long bytes = (long long)M * (K + 64);
    return bytes <= 120 * 1024 && (M <= 4 || (M <= 8 && K >= 640 && strips <= (K > 1024 ? 3 : 2) * sms && (strips <= sms || bytes <= 56 * 1024)));
}

template <int MW, int RG, int FE, int VK, int VR>
static cudaError_t launch_w2_strips(W2Params& p, cudaStream_t stream) {
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    auto kern = w2_small_kernel<MW, RG, FE, VK, VR>;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kW2MaxSmem);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    const int K = p.e.K, KP = w2_pairs(K), tokens = p.e.M;
    // CTAs: one per SM (fewer when there are fewer strips), so that every SM gets the same share within a strip
    // (at most 40 strips each: the kernel's item index arithmetic)
    const int strips = p.e.N / 16, ctas = std::min(strips, std::max(device_sm_count(), (strips + 39) / 40));
    const int R = (strips + ctas - 1) / ctas;
    p.strips_q = strips / ctas, p.strips_r = strips % ctas;
    const int W = w2_warps(K, MW);
    p.pairs_q = KP / W, p.pairs_r = KP % W;
    const int per = (KP + W - 1) / W;
    // ring: all of the CTA's weights when they fit 64 KB (two launches' prefetches fit an SM side by side), otherwise two
    // slots or more with copies of up to 4 KB (the copy engine takes about 60 cycles for each, whatever its size: 57344 x 8192
    // at 4 tokens 70 us with copies of 0.5 KB, 41 with 1 KB, 32.5 with 2 or 3 KB, 37 with 2.5, which cuts a share of 3.5 unevenly)
    const bool res = p.e.residual != nullptr;
    const int groups = (R + RG - 1) / RG, unit = W * RG * 512, room = kW2MaxSmem - w2_smem(R, tokens, K, W, 0, 0, res).total;
    if (room < unit) return cudaErrorInvalidValue;
    p.chunk_pairs = per, p.slots = groups;
    if (groups > kW2MaxSlots || groups * per * unit > std::min(64 * 1024, room)) {
        p.chunk_pairs = std::max(1, std::min(std::min(per, 8), room / 2 / unit));
        const int chunks = groups * ((per + p.chunk_pairs - 1) / p.chunk_pairs);
        p.slots = std::min(std::min(chunks, kW2MaxSlots), room / (p.chunk_pairs * unit));
    }
    p.smem = w2_smem(R, tokens, K, W, p.slots, RG * p.chunk_pairs * 512, res);
    if (p.smem.total > kW2MaxSmem) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(W * 32, 1, 1);
    cfg.dynamicSmemBytes = p.smem.total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    t_echo = {8, 8, 1, W, R, (int)cfg.gridDim.x};
    return cudaLaunchKernelEx(&cfg, kern, p);
}

// Strips at a time: three, whose chains overlap, where that wastes little of a CTA's last group - it has three, or six and more - and
// their share of K leaves room for the ring (not 8192 x 28672: 26.9 us at 1 token, one at a time 20.7); one otherwise.  One / three at a time, mean over
// the quantised entry and the front-ends, separate or inside, at 1 to 4 tokens: three strips 5120 x 5120 1.02 to 1.08, 6912 x 4096 1.09 to 1.13; four 8192 x 2560
// 0.90 to 0.92, 8192 x 6912 0.93 to 0.95; five 10240 x 2048 0.93 to 0.98, 10240 x 6912 0.96 to 0.99; six 13824 x 2560 1.04 to 1.06, 13824 x 4096 1.14 to 1.19; seven
// 14336 x 8192 11.4 / 9.0 us.
template <int FE, int VK, int VR>
static cudaError_t launch_w2_small(W2Params& p, cudaStream_t stream) {
    const int sms = device_sm_count(), R = (p.e.N / 16 + sms - 1) / sms;
    return p.e.K > 8192 || R <= 2 || R == 4 || R == 5 ? launch_w2_strips<kW2Warps, 1, FE, VK, VR>(p, stream) : launch_w2_strips<kW2Warps, 3, FE, VK, VR>(p, stream);
}
// Twice the warps, a strip at a time, shorten a strip's chain, but leave no place beside them: the next launch's CTAs wait for this one's, and
// these for a front-end's, 1 to 2 us once per launch.  Where a CTA has up to five strips, whose chains are most of the call, that pays from 8192
// columns on; more strips, which ten warps take three at a time, from 12288 on - or from 8192 where there are many of them and four tokens,
// whose sums cost the ten warps 10 % more than one token's and the twenty nothing.  us per call, ten / twenty warps, in a stream of such calls (and behind
// the quantiser), at 1 and 4 tokens: 2560 x 8192 3.8 / 3.5 (5.7 / 5.1), 4.0 / 3.7 (6.1 / 5.3), 10240 x 8192 7.2 / 7.2 (8.6 / 8.2), 7.5 / 7.9 (9.5 / 9.2), 14336 x 8192 9.6 /
// 13.6 (12.1 / 13.8), 11.4 / 13.4 (14.1 / 14.3), 14336 x 10240 13.1 / 15.0 (16.1 / 16.0), 13.0 / 14.1 (16.8 / 17.6), 28672 x 8192 17.0 / 19.0 (18.9 / 19.1), 18.7 / 19.1
// (21.2 / 20.4), 57344 x 8192 30.1 / 33.3 (32.6 / 33.8), 33.3 / 33.2 (36.6 / 34.6), 28672 x 12288 24.4 / 23.6 (28.6 / 25.3), 26.3 / 22.5 (32.3 / 27.6), 14336 x 16384 16.9 /
// 13.9 (21.1 / 18.3), 17.4 / 15.3 (24.5 / 22.5); shorter K 57344 x 7680 at 4 28.3 / 34.5 (31.7 / 36.0).
static cudaError_t launch_w2_int8(W2Params& p, cudaStream_t stream) {
    const int strips = p.e.N / 16, sms = device_sm_count();
    const bool twice = p.e.K >= (strips <= 5 * sms || (strips > 8 * sms && p.e.M > 3) ? 8192 : 12288);
    return twice ? launch_w2_strips<kW2MaxWarps, 1, W2_INT8, 1, 1>(p, stream) : launch_w2_small<W2_INT8, 1, 1>(p, stream);
}
template <int FE>
static cudaError_t launch_w2_fused(W2Params& p, cudaStream_t stream) {
    // Vectors of a row per thread, and rows at a time.  (The loops for three vectors cost a thread that has one 0.3 us a row: gated 2560 x 2560
    // at 1 / 4 tokens 3.5 / 8.0 with them and a row at a time, 3.1 / 4.2 so.)
    const int vk = (act_row_threads(p.e.K) / 32 + w2_warps(p.e.K) - 1) / w2_warps(p.e.K), M = p.e.M;
    if (vk > 1) return vk > 3 ? launch_w2_small<FE, 4, 1>(p, stream) : launch_w2_small<FE, 3, 1>(p, stream);
    return M == 1 ? launch_w2_small<FE, 1, 1>(p, stream) : launch_w2_small<FE, 1, 4>(p, stream);
}

static cudaError_t launch_w2_tile(const W2Params& p, const W2TilePlan& plan, cudaStream_t stream) {
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    auto kern = w2_tile_kernel;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kW2MaxSmem / 2 - 1024);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    const int M = p.e.M, tiles = (p.e.N + kTileRows - 1) / kTileRows, S = plan.splits, blocks = (M + plan.nt - 1) / plan.nt;
    W2TileParams pp = {p.e, p.w, plan.nt, 0, 0};
    pp.stages = std::min({kTileMaxStages, (kTileCols - pp.nt) / 64, 64 * 1024 / (pp.nt * 256)});
    pp.slots = pp.nt > 64 ? 2 : kTileSlots;
    const int smem = 1024 + W2TileSmem::ring + pp.slots * kTileSlotBytes + pp.stages * pp.nt * 256;
    CUtensorMap map;
    if (!encode_x_map(&map, p.e.x, M, p.e.K, pp.nt)) return cudaErrorInvalidValue;   // reported as status 3, nothing is launched
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kTileThreads, 1, 1);
    cfg.gridDim = dim3(S, tiles, blocks);
    cfg.dynamicSmemBytes = std::max(smem, kTileMinSmem);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 2 : 1;
    t_echo = {9, pp.nt, S, kTileThreads / 32, 1, S * tiles * blocks};
    return cudaLaunchKernelEx(&cfg, kern, pp, map);
}

static cudaError_t launch_w2_pair(const W2Params& p, int nt, cudaStream_t stream) {
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    auto kern = w2_pair_kernel;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, W2PairSmem::total);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    const int pairs = device_sm_count() / 2, RB = (p.e.N + kPairRows - 1) / kPairRows;
    W2PairParams pp = {p.e, p.w, nt, 0, 0, 0, 0};
    w2_pair_plan(pp);
    CUtensorMap map;   // each CTA of a pair loads half of the tile's tokens per stage
    if (!encode_x_map(&map, p.e.x, p.e.M, p.e.K, pp.nt / 2)) return cudaErrorInvalidValue;   // reported as status 3, nothing is launched
    const long long tiles = (long long)RB * ((p.e.M + pp.nt - 1) / pp.nt);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kW2PairThreads, 1, 1);
    cfg.gridDim = dim3((unsigned)(2 * std::min<long long>(tiles, pairs)), 1, 1);
    cfg.dynamicSmemBytes = W2PairSmem::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 2 : 1;
    t_echo = {7, pp.nt, 2, kW2PairThreads / 32, 4, (int)cfg.gridDim.x};
    return cudaLaunchKernelEx(&cfg, kern, pp, map);
}

// Whether a call that has both forms of the weight in hand should take the two-bit one.  It always should, deep and narrow
// layers included (us per call, two-bit / packed: 2560 x 6912 at 48 tokens 5.4 / 13.4, at 128 6.9 / 15.7, at 256 8.6 / 17.9, 1024 x 16384 at
// 333 10.0 / 25.2).
extern "C" int ternaspmm_w2_pays(int, int, int) { return 1; }

__global__ void stream_fence_kernel() {}

// Bytes of a weight's two-bit layout.
extern "C" long long ternaspmm_w2_bytes(int N, int K) { return N < 16 || K < 64 ? 0 : (long long)(N / 16) * w2_pairs(K) * 512; }

extern "C" void ternaspmm_w2_relayout(uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets, uint32_t* sign_words,
                                      int N, int K, void* w2, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (N < 64 || K < 64 || (N % 64) || (K % 64)) {
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!bitmap || !tile_offsets || !quarter_offsets || !sign_words || !w2 || (reinterpret_cast<uintptr_t>(bitmap) & 15) ||
        (reinterpret_cast<uintptr_t>(w2) & 15)) {
        t_host_status = ST_BAD_POINTER;
        return;
    }
    SpmmParams p = {};
    p.bitmap = reinterpret_cast<const uint32_t*>(bitmap), p.tile_off = tile_offsets, p.quarter_off = quarter_offsets;
    p.signs = sign_words, p.N = N, p.K = K;
    const long long tiles = (long long)(N / 64) * (K / 64);
    relayout_w2_kernel<<<(unsigned)((tiles + 7) / 8), 256, 0, stream>>>(p, static_cast<uint8_t*>(w2));
    // A linear that follows reads w2 ahead of its dependency wait, as early as the kernel before it lets it.  This one begins in
    // plain stream order, when the layout is complete and visible, and every later kernel of the stream begins after it.
    stream_fence_kernel<<<1, 32, 0, stream>>>();
    checkLastCudaError(__LINE__);
}

// Rows that a front-end inside the kernel takes: a thread holds at most four eight-element vectors of a row.
extern "C" int ternaspmm_w2_fused_rows(int K) { return K < 64 || K > 8 * kActMaxThreads ? 0 : kW2MaxRows; }

extern "C" void ternaspmm_w2_linear(void* x, int front_end, __nv_bfloat16* norm_weight, float eps, void* w2, __nv_bfloat16* out,
                                    __nv_bfloat16* s, __nv_bfloat16* ws, int ws_num, int M, int N, int K, int seg1, int seg2,
                                    int seg3, int prefill_form, __nv_bfloat16* residual, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (M < 1 || N < 64 || K < 64 || (N % 64) || (K % 64) || K >= (1 << 18) || ws_num < 1 || ws_num > 4 || front_end < W2_INT8 ||
        front_end > W2_GATED || (front_end != W2_INT8 && M > ternaspmm_w2_fused_rows(K))) {
        fprintf(stderr, "ternaspmm: w2_linear: unsupported shape M=%d N=%d K=%d ws_num=%d front_end=%d\n", M, N, K, ws_num, front_end);
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!x || !w2 || !out || !ws || (front_end == W2_INT8 && !s) || (front_end >= W2_NORM && !norm_weight) ||
        (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w2) & 15) || (reinterpret_cast<uintptr_t>(norm_weight) & 15)) {
        fprintf(stderr, "ternaspmm: w2_linear: null or misaligned pointer (x, w2, norm_weight: 16 bytes)\n");
        t_host_status = ST_BAD_POINTER;
        return;
    }
    W2Params p = {};
    p.e.x = static_cast<const int8_t*>(x), p.xb = static_cast<const __nv_bfloat16*>(x);
    p.norm_w = norm_weight, p.eps = eps, p.w = static_cast<const uint8_t*>(w2);
    p.e.out = out, p.e.s = s, p.e.ws = ws, p.e.residual = residual, p.e.ws_num = ws_num, p.e.M = M, p.e.N = N, p.e.K = K;
    p.e.epilogue = prefill_form < 0 ? (M <= 64 ? EPI_DECODE : EPI_PREFILL) : (prefill_form ? EPI_PREFILL : EPI_DECODE);
    const int seg[3] = {seg1, seg2, seg3};
    set_segments(p.e, seg1 | seg2 | seg3 ? seg : nullptr);
    p.e.status = status_device_ptr();
    if (!p.e.status) {
        t_host_status = ST_LAUNCH;
        return;
    }
    cudaError_t e;
    if (front_end == W2_PLAIN) e = launch_w2_fused<W2_PLAIN>(p, stream);
    else if (front_end == W2_NORM) e = launch_w2_fused<W2_NORM>(p, stream);
    else if (front_end == W2_GATED) e = launch_w2_fused<W2_GATED>(p, stream);
    else if (w2_small_takes(M, N, K)) e = launch_w2_int8(p, stream);
    else {
        const W2TilePlan tile = w2_tile_plan(M, N, K, device_sm_count());
        const W2PairPlan pair = w2_pair_plan_tile(M, N, K, device_sm_count() / 2);
        e = tile.us <= pair.us ? launch_w2_tile(p, tile, stream) : launch_w2_pair(p, pair.nt, stream);
    }
    if (e != cudaSuccess) {
        fprintf(stderr, "ternaspmm: launch failed: %s\n", cudaGetErrorString(e));
        t_host_status = ST_LAUNCH;
    }
    checkLastCudaError(__LINE__);
}

// ---- attention glue of a decode step (attn_decode.cuh) ---------------------------------------------
template <int GQ, bool BY_HEAD>
static cudaError_t launch_attn_decode(const AttnParams& p, int batch, cudaStream_t stream) {
    auto kern = attn_decode_kernel<GQ, BY_HEAD>;
    // CTAs per key / value head: a power of two up to the portable cluster size, so that all are resident at once (three per SM)
    int S = 8;
    while (S > 1 && (long long)batch * p.kv_heads * S > 3ll * device_sm_count()) S >>= 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S, p.kv_heads, batch);
    cfg.blockDim = dim3(kAttnWarps * 32, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // Not a programmatic dependent of the linear before it: launched early, its CTAs take the places that are left beside that
    // linear's, unevenly and some of them late (30-layer model, per layer: 7.6 us instead of 5.8 at batch 1 and 600 tokens,
    // 16.1 instead of 10.5 at batch 8 and 1100).  The kernel after it is one of this kernel's.
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

template <bool BY_HEAD>
static int run_attn_decode(__nv_bfloat16* qkv, __nv_bfloat16* k_cache, __nv_bfloat16* v_cache, const void* cos_row, const void* sin_row,
                           long long* pos, __nv_bfloat16* out, int batch, int heads, int kv_heads, int head_dim, int max_len,
                           cudaStream_t stream) {
    t_host_status = ST_OK;
    const int gq = kv_heads > 0 && heads % kv_heads == 0 ? heads / kv_heads : 0;
    if (batch < 1 || batch > 65535 || kv_heads < 1 || kv_heads > 65535 || max_len < 1 || head_dim != kAttnD || (gq != 4 && gq != 8)) {
        t_host_status = ST_BAD_SHAPE;
        return t_host_status;
    }
    const uintptr_t bits = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache);
    if (!qkv || !k_cache || !v_cache || !cos_row || !sin_row || !pos || !out || (bits & 15)) {
        t_host_status = ST_BAD_POINTER;
        return t_host_status;
    }
    AttnParams p = {qkv, k_cache, v_cache, cos_row, sin_row, pos, out, heads, kv_heads, max_len, 1.4426950408889634f / sqrtf((float)head_dim),
                    BY_HEAD ? status_device_ptr() : nullptr};
    if (BY_HEAD && !p.status) {
        t_host_status = ST_LAUNCH;
        return t_host_status;
    }
    if ((gq == 4 ? launch_attn_decode<4, BY_HEAD>(p, batch, stream) : launch_attn_decode<8, BY_HEAD>(p, batch, stream)) != cudaSuccess)
        t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
    return t_host_status;
}

extern "C" int ternaspmm_attn_decode(__nv_bfloat16* qkv, __nv_bfloat16* k_cache, __nv_bfloat16* v_cache, __nv_bfloat16* cos_row,
                                     __nv_bfloat16* sin_row, long long* pos, __nv_bfloat16* out, int batch, int heads, int kv_heads,
                                     int head_dim, int max_len, cudaStream_t stream) {
    return run_attn_decode<false>(qkv, k_cache, v_cache, cos_row, sin_row, pos, out, batch, heads, kv_heads, head_dim, max_len, stream);
}

extern "C" int ternaspmm_attn_decode_by_head(__nv_bfloat16* qkv, __nv_bfloat16* k_cache, __nv_bfloat16* v_cache, float* cos_row, float* sin_row,
                                             long long* pos, __nv_bfloat16* out, int batch, int heads, int kv_heads, int head_dim,
                                             int max_len, cudaStream_t stream) {
    return run_attn_decode<true>(qkv, k_cache, v_cache, cos_row, sin_row, pos, out, batch, heads, kv_heads, head_dim, max_len, stream);
}

extern "C" int ternaspmm_attn_prefill(__nv_bfloat16* qkv, __nv_bfloat16* k_cache, __nv_bfloat16* v_cache, __nv_bfloat16* cos_tab,
                                      __nv_bfloat16* sin_tab, long long* pos, __nv_bfloat16* out, int batch, int tokens, int heads,
                                      int kv_heads, int head_dim, int max_len, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (batch < 1 || batch > 65535 || tokens < 1 || kv_heads < 1 || heads % kv_heads || (heads / kv_heads) % 4 || heads > 4 * 65535 ||
        max_len < 1 || head_dim != kAttnD) {
        t_host_status = ST_BAD_SHAPE;
        return t_host_status;
    }
    const uintptr_t bits = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
                           reinterpret_cast<uintptr_t>(cos_tab) | reinterpret_cast<uintptr_t>(sin_tab);
    if (!qkv || !k_cache || !v_cache || !cos_tab || !sin_tab || !pos || !out || (bits & 15)) {
        t_host_status = ST_BAD_POINTER;
        return t_host_status;
    }
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(attn_prefill_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kPfTile) != cudaSuccess ||
            cudaFuncSetAttribute(attn_prefill_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kPfTile) != cudaSuccess) {
            t_host_status = ST_LAUNCH;
            return t_host_status;
        }
        attr_done[dev] = true;
    }
    const AttnPrefillParams p = {qkv, k_cache, v_cache, cos_tab, sin_tab, pos, out, tokens, heads, kv_heads, max_len,
                                 1.4426950408889634f / sqrtf((float)head_dim)};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    cfg.stream = stream;
    const long long items = (long long)batch * tokens * kv_heads * 16;
    cfg.gridDim = dim3((unsigned)((items + 255) / 256), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cudaError_t e = cudaLaunchKernelEx(&cfg, rope_append_kernel, p, items);
    const int heads_x_batch = heads / 4 * batch, items_a = (tokens + 15) / 16 * heads_x_batch, key_tiles = (tokens + 63) / 64;
    // Two CTAs per item where the chain of the longest rows outlasts an SM's share of the work: few items, the more the longer they
    // are (one prompt of 1024 tokens, 320 items: 30 us instead of 37; of 2048, 640 items: 82 instead of 76; two of 613, 390
    // items of up to 10 tiles: 30 instead of 27; four of 100, 140 items of two tiles: 10.3 instead of 9.3)
    const bool split = key_tiles >= 3 && items_a <= device_sm_count() + 12 * key_tiles;
    cfg.gridDim = dim3(split ? 2 * items_a : items_a, 1, 1);
    cfg.blockDim = dim3(128, 1, 1);
    cfg.dynamicSmemBytes = 4 * kPfTile;
    // (not a programmatic dependent: launched early its CTAs spread unevenly, one prompt of 1024 tokens 57 us instead of 47)
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = split ? 1 : 0;
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, split ? attn_prefill_kernel<2> : attn_prefill_kernel<1>, p, heads_x_batch);
    if (e != cudaSuccess) t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
    return t_host_status;
}

static void run_norm_quant(bool gated, int mode, __nv_bfloat16* x, __nv_bfloat16* w, float eps, int M, int K,
                           int8_t* q, __nv_bfloat16* s_out, float* ss_out, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (M < 1 || K < 16 || (K % 16) || K > 56 * 1024) {
        fprintf(stderr, "ternaspmm: norm_quant needs M>=1 and K a multiple of 16 up to 57344 (got M=%d K=%d)\n", M, K);
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!x || (mode != ACT_PLAIN && !w) || !q || (!s_out && mode != ACT_NORM_ONLY) || (mode == ACT_SCALE_SUMSQ && !ss_out) ||
        (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) ||
        (reinterpret_cast<uintptr_t>(q) & 15)) {
        fprintf(stderr, "ternaspmm: norm_quant: null or misaligned pointer\n");
        t_host_status = ST_BAD_POINTER;
        return;
    }
    typedef void (*Kern)(const __nv_bfloat16*, const __nv_bfloat16*, float, int, int8_t*, __nv_bfloat16*, float*);
    static const Kern by_row[5] = {norm_quant_row_kernel<false, ACT_RMSNORM>, norm_quant_row_kernel<false, ACT_SCALE_SUMSQ>,
                                    norm_quant_row_kernel<false, ACT_PLAIN>, norm_quant_row_kernel<false, ACT_NORM_ONLY>, nullptr};
    static const Kern long_row[5] = {norm_quant_kernel<false, ACT_RMSNORM>, norm_quant_kernel<false, ACT_SCALE_SUMSQ>,
                                    norm_quant_kernel<false, ACT_PLAIN>, norm_quant_kernel<false, ACT_NORM_ONLY>, nullptr};
    static const Kern many_rows[5] = {norm_quant_rows_kernel<ACT_RMSNORM>, norm_quant_rows_kernel<ACT_SCALE_SUMSQ>,
                                      norm_quant_rows_kernel<ACT_PLAIN>, norm_quant_rows_kernel<ACT_NORM_ONLY>, nullptr};
    const bool short_row = K <= 8 * kActMaxThreads;   // one eight-element vector per thread
    // two rows per SM and more: fewer threads per row (below that a row's own chain of latencies is longer with them)
    const bool many = short_row && M >= 2 * device_sm_count(), in_regs = many && !gated;
    Kern kern = in_regs ? many_rows[mode] : short_row ? by_row[mode] : long_row[mode];
    if (gated) {
        if (mode == ACT_RMSNORM) kern = short_row ? norm_quant_row_kernel<true, ACT_RMSNORM> : norm_quant_kernel<true, ACT_RMSNORM>;
        else kern = short_row ? norm_quant_row_kernel<true, ACT_SCALE_SUMSQ> : norm_quant_kernel<true, ACT_SCALE_SUMSQ>;
    }
    static bool attr_done[2][64][8] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    const int slot = (gated ? 4 : 0) + mode;
    if (!in_regs && !attr_done[short_row][dev][slot]) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * 56 * 1024);
        attr_done[short_row][dev][slot] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(M, 1, 1);
    const int T = act_row_threads(K);   // one vector per thread; for many rows four
    cfg.blockDim = dim3(many ? std::max(64, (T / 4 + 31) / 32 * 32) : T, 1, 1);
    cfg.dynamicSmemBytes = in_regs ? 0 : short_row ? (size_t)K * (gated ? 6 : (mode == ACT_PLAIN ? 2 : 4)) : (size_t)K * 2;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kern, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, eps, K, q, s_out, ss_out) !=
        cudaSuccess)
        t_host_status = ST_LAUNCH;
}

extern "C" void ternaspmm_rmsnorm_quant(__nv_bfloat16* x, __nv_bfloat16* norm_weight, float eps, int M, int K,
                                       int8_t* q, __nv_bfloat16* s_out, cudaStream_t stream) {
    run_norm_quant(false, ACT_RMSNORM, x, norm_weight, eps, M, K, q, s_out, nullptr, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_relu2_gate_rmsnorm_quant(__nv_bfloat16* x13, __nv_bfloat16* norm_weight, float eps, int M,
                                                  int K, int8_t* q, __nv_bfloat16* s_out, cudaStream_t stream) {
    run_norm_quant(true, ACT_RMSNORM, x13, norm_weight, eps, M, K, q, s_out, nullptr, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_rmsnorm(__nv_bfloat16* x, __nv_bfloat16* norm_weight, float eps, int M, int K, __nv_bfloat16* y,
                                  cudaStream_t stream) {
    run_norm_quant(false, ACT_NORM_ONLY, x, norm_weight, eps, M, K, reinterpret_cast<int8_t*>(y), nullptr, nullptr, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_quant(__nv_bfloat16* x, int M, int K, int8_t* q, __nv_bfloat16* s_out, cudaStream_t stream) {
    run_norm_quant(false, ACT_PLAIN, x, nullptr, 0.f, M, K, q, s_out, nullptr, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_scale_quant_sumsq(__nv_bfloat16* x, __nv_bfloat16* weight, int gated, int M, int K,
                                           int8_t* q, __nv_bfloat16* s_out, float* ss_out, cudaStream_t stream) {
    run_norm_quant(gated != 0, ACT_SCALE_SUMSQ, x, weight, 0.f, M, K, q, s_out, ss_out, stream);
    checkLastCudaError(__LINE__);
}

static cudaLaunchConfig_t elementwise_launch(long long items, cudaStream_t stream, cudaLaunchAttribute* attr) {
    attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr->val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((items + 255) / 256), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    return cfg;
}

extern "C" void ternaspmm_rope(__nv_bfloat16* x, long long ld, float* cos_t, float* sin_t, __nv_bfloat16* out, int batch, int tokens, int heads,
                               cudaStream_t stream) {
    t_host_status = ST_OK;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(cos_t) |
                           reinterpret_cast<uintptr_t>(sin_t);
    if (!x || !out || !cos_t || !sin_t || (bits & 15) || (ld & 7) || batch < 1 || tokens < 1 || heads < 1) {
        t_host_status = ST_BAD_POINTER;
        return;
    }
    const long long items = (long long)batch * tokens * heads * 16;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = elementwise_launch(items, stream, &attr);
    if (cudaLaunchKernelEx(&cfg, rope_kernel, (const __nv_bfloat16*)x, ld, (const float*)cos_t, (const float*)sin_t, out, tokens, heads, items) != cudaSuccess)
        t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_relu2_gate(__nv_bfloat16* x13, __nv_bfloat16* out, int M, int K, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (!x13 || !out || ((reinterpret_cast<uintptr_t>(x13) | reinterpret_cast<uintptr_t>(out)) & 15) || M < 1 || K < 8 || (K & 7)) {
        t_host_status = ST_BAD_POINTER;
        return;
    }
    const long long items = (long long)M * (K / 8);
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = elementwise_launch(items, stream, &attr);
    if (cudaLaunchKernelEx(&cfg, relu2_gate_kernel, (const __nv_bfloat16*)x13, out, K / 8, items) != cudaSuccess) t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_bf16_to_f32(__nv_bfloat16* x, float* y, long long n, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (!x || !y || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) || n < 1) {
        t_host_status = ST_BAD_POINTER;
        return;
    }
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = elementwise_launch(std::min<long long>((n + 15) / 16, 256ll * 8 * device_sm_count()), stream, &attr);
    if (cudaLaunchKernelEx(&cfg, bf16_to_f32_kernel, (const __nv_bfloat16*)x, y, n) != cudaSuccess) t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_partial_f32(int8_t* x, uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets,
                                     uint32_t* sign_words, float* out, __nv_bfloat16* s, int M, int N, int K,
                                     cudaStream_t stream) {
    run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, nullptr, 1, M, N, K, EPI_F32_DIV, stream);
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_tp_finish(float* buf, __nv_bfloat16* ws, float eps, int full_width, int M, int N,
                                   __nv_bfloat16* residual, __nv_bfloat16* out, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (!buf || !ws || !out || M < 1 || N < 1) {
        t_host_status = ST_BAD_POINTER;
        return;
    }
    const long long total = (long long)M * N;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 4 * device_sm_count()) blocks = 4 * device_sm_count();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, tp_finish_kernel, (const float*)buf, (const __nv_bfloat16*)ws, eps, full_width, M, N,
                           (const __nv_bfloat16*)residual, out) != cudaSuccess)
        t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_tp_allreduce_finish(float** bufs, unsigned int** flags, __nv_bfloat16** outs, int rank,
                                             int world, unsigned int* counters, __nv_bfloat16* ws, float eps,
                                             int full_width, int M, int N, __nv_bfloat16* residual,
                                             cudaStream_t stream) {
    t_host_status = ST_OK;
    if (!bufs || !flags || !outs || !counters || !ws || world < 1 || world > 8 || rank < 0 || rank >= world || M < 1 ||
        N < 4 || (N % 4)) {
        fprintf(stderr, "ternaspmm: tp_allreduce_finish: bad arguments (world 1..8, N a multiple of 4)\n");
        t_host_status = ST_BAD_POINTER;
        return;
    }
    TpPeers peers = {};
    for (int r = 0; r < world; ++r) {
        if (!bufs[r] || !flags[r] || !outs[r]) {
            t_host_status = ST_BAD_POINTER;
            return;
        }
        peers.buf[r] = bufs[r];
        peers.flag[r] = flags[r];
        peers.out[r] = outs[r];
    }
    int* status = status_device_ptr();
    if (!status) {
        t_host_status = ST_LAUNCH;
        return;
    }
    // this rank finishes 1/world of the outputs: one 4-element vector per thread, at most two blocks per SM
    const long long vecs = ((long long)M * N / 4 + world - 1) / world;
    int blocks = (int)std::max<long long>(1, std::min<long long>((vecs + 255) / 256, 2ll * device_sm_count()));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, tp_allreduce_finish_kernel, peers, rank, world, counters, counters + 1,
                           (const __nv_bfloat16*)ws, eps, full_width, M, N, (const __nv_bfloat16*)residual,
                           status, g_wait_limit_ns) != cudaSuccess)
        t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
}

// ---- packer on the GPU (pack_gpu.cuh) --------------------------------------------------------------
extern "C" long long ternaspmm_pack_gpu_layout(const int8_t* W, int N, int K, uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets,
                                               cudaStream_t stream) {
    t_host_status = ST_OK;
    if (N < 64 || K < 64 || (N % 64) || (K % 64)) {
        t_host_status = ST_BAD_SHAPE;
        return -1;
    }
    if (!W || !bitmap || !tile_offsets || !quarter_offsets || (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(bitmap) & 15)) {
        t_host_status = ST_BAD_POINTER;
        return -1;
    }
    static thread_local long long* total = nullptr;   // pinned, written by the scan kernel; one per thread, kept
    if (!total && cudaHostAlloc(reinterpret_cast<void**>(&total), sizeof(*total), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
        total = nullptr;
        cudaGetLastError();
        t_host_status = ST_LAUNCH;
        return -1;
    }
    volatile long long* const result = total;
    *result = -1;
    const long long tiles = (long long)(N / 64) * (K / 64);
    const unsigned blocks = (unsigned)((tiles + kPackWarps - 1) / kPackWarps);
    pack_bitmap_kernel<<<blocks, kPackWarps * 32, 0, stream>>>(W, N, K, reinterpret_cast<uint4*>(bitmap), tile_offsets, quarter_offsets);
    pack_scan_kernel<<<1, 1024, 0, stream>>>(tile_offsets, tiles, total);
    // The number is here a few microseconds before the stream is idle; the stream is asked now and then whether it still runs.
    for (int i = 1; *result < 0; ++i) {
        if (i & 4095) continue;
        const cudaError_t e = cudaStreamQuery(stream);
        if (e != cudaErrorNotReady && (e != cudaSuccess || *result < 0)) {
            t_host_status = ST_LAUNCH;
            checkLastCudaError(__LINE__);
            return -1;
        }
    }
    if (*result >= (1ll << 31)) {   // offsets are 32-bit
        t_host_status = ST_BAD_SHAPE;
        return -1;
    }
    return *result / 32;
}

extern "C" void ternaspmm_pack_gpu_signs(const int8_t* W, int N, int K, const int* tile_offsets, uint32_t* sign_words, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (N < 64 || K < 64 || (N % 64) || (K % 64)) {
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!W || !tile_offsets || !sign_words || (reinterpret_cast<uintptr_t>(W) & 15)) {
        t_host_status = ST_BAD_POINTER;
        return;
    }
    const long long tiles = (long long)(N / 64) * (K / 64);
    pack_signs_kernel<<<(unsigned)((tiles + kPackWarps - 1) / kPackWarps), kPackWarps * 32, 0, stream>>>(W, N, K, tile_offsets, sign_words);
    checkLastCudaError(__LINE__);
}

// ---- work lists ----------------------------------------------------------------------------------
struct ternaspmm_list {
    void* device_table;
    void* scratch;
    int entries, mt;
};

static size_t list_scratch_bytes() { return sizeof(ListScratch) + (size_t)device_sm_count() * kListAreaInts * 4; }

// Validates the items and turns them into device entries.  Returns false on a bad item.
static bool list_entries(const ternaspmm_list_item* items, int n, std::vector<ListItem>& out, int& max_m) {
    max_m = 0;
    long long tiles = 0;
    if (n > kListMaxItems) {
        fprintf(stderr, "ternaspmm: a list holds at most %d items (got %d)\n", kListMaxItems, n);
        t_host_status = ST_BAD_SHAPE;
        return false;
    }
    for (int i = 0; i < n; ++i) {
        const ternaspmm_list_item& u = items[i];
        if (u.M < 1 || u.M > 16 || u.N < 64 || u.K < 64 || (u.N % 64) || (u.K % 64) || u.K / 64 > 4095 || u.N / 64 > 4095 ||
            u.ws_num < 1 || u.ws_num > 4) {
            fprintf(stderr, "ternaspmm: list item %d: unsupported shape M=%d N=%d K=%d ws_num=%d (need 1<=M<=16, N%%64==0, "
                            "K%%64==0, N and K below 262144)\n", i, u.M, u.N, u.K, u.ws_num);
            t_host_status = ST_BAD_SHAPE;
            return false;
        }
        if (!u.x || !u.bitmap || !u.tile_offsets || !u.quarter_offsets || !u.sign_words || !u.out || !u.s || !u.ws ||
            (reinterpret_cast<uintptr_t>(u.x) & 15) || (reinterpret_cast<uintptr_t>(u.bitmap) & 15) ||
            (reinterpret_cast<uintptr_t>(u.sign_words) & 15)) {
            fprintf(stderr, "ternaspmm: list item %d: null or misaligned pointer\n", i);
            t_host_status = ST_BAD_POINTER;
            return false;
        }
        const int epi = u.prefill_form < 0 ? (u.M <= 64 ? EPI_DECODE : EPI_PREFILL) : (u.prefill_form ? EPI_PREFILL : EPI_DECODE);
        ListItem e = {};
        e.x = u.x, e.bitmap = reinterpret_cast<const uint32_t*>(u.bitmap), e.tile_off = u.tile_offsets;
        e.quarter_off = u.quarter_offsets, e.signs = u.sign_words;
        e.out = reinterpret_cast<__nv_bfloat16*>(u.out), e.residual = reinterpret_cast<const __nv_bfloat16*>(u.residual);
        e.s = reinterpret_cast<const __nv_bfloat16*>(u.s), e.ws = reinterpret_cast<const __nv_bfloat16*>(u.ws);
        e.M = u.M, e.N = u.N, e.K = u.K, e.ld_out = u.N, e.ws_num = u.ws_num, e.epilogue = epi;
        if (u.seg1 || u.seg2 || u.seg3) {   // explicit boundaries
            const int b[3] = {u.seg1, u.seg2, u.seg3};
            for (int k = 0; k < 3; ++k) e.seg_b[k] = (k + 1 < u.ws_num) ? b[k] : INT_MAX;
            e.seg_gran = 1;
        } else {                            // the reference's rules (see ws_group in spmm_small_m.cuh)
            const bool prefill = epi == EPI_PREFILL;
            e.seg_gran = prefill ? 128 : 8;
            if (u.N == 3840 && (prefill || u.ws_num == 3)) {
                e.seg_b[0] = 2560, e.seg_b[1] = 3200, e.seg_b[2] = INT_MAX;
            } else {
                const int gw = u.N / u.ws_num;
                e.seg_b[0] = gw, e.seg_b[1] = 2 * gw, e.seg_b[2] = 3 * gw;
            }
        }
        e.tile_base = tiles;
        tiles += (long long)(u.N / 64) * (u.K / 64);
        out.push_back(e);
        max_m = std::max(max_m, u.M);
    }
    if (tiles / std::max(1, device_sm_count()) > (1ll << 30)) {
        t_host_status = ST_BAD_SHAPE;
        return false;
    }
    return true;
}

extern "C" int ternaspmm_list_plan(const ternaspmm_list_item* items, int n_items, long long* table_bytes,
                                   long long* scratch_bytes) {
    t_host_status = ST_OK;
    std::vector<ListItem> e;
    int max_m;
    if (!items || n_items < 1 || !list_entries(items, n_items, e, max_m)) {
        if (t_host_status == ST_OK) t_host_status = ST_BAD_POINTER;
        return -1;
    }
    if (table_bytes) *table_bytes = (long long)e.size() * sizeof(ListItem);
    if (scratch_bytes) *scratch_bytes = (long long)list_scratch_bytes();
    return (int)e.size();
}

extern "C" ternaspmm_list* ternaspmm_list_create(const ternaspmm_list_item* items, int n_items, void* device_table,
                                                 void* scratch, cudaStream_t stream) {
    t_host_status = ST_OK;
    std::vector<ListItem> e;
    int max_m;
    if (!items || n_items < 1 || !device_table || !scratch || (reinterpret_cast<uintptr_t>(device_table) & 15) ||
        (reinterpret_cast<uintptr_t>(scratch) & 15)) {
        t_host_status = ST_BAD_POINTER;
        return nullptr;
    }
    if (!list_entries(items, n_items, e, max_m)) return nullptr;
    if (cudaMemcpyAsync(device_table, e.data(), e.size() * sizeof(ListItem), cudaMemcpyHostToDevice, stream) != cudaSuccess ||
        cudaMemsetAsync(scratch, 0, list_scratch_bytes(), stream) != cudaSuccess || cudaStreamSynchronize(stream) != cudaSuccess) {
        t_host_status = ST_LAUNCH;
        return nullptr;
    }
    ternaspmm_list* l = static_cast<ternaspmm_list*>(malloc(sizeof(ternaspmm_list)));
    if (!l) return nullptr;
    l->device_table = device_table, l->scratch = scratch, l->entries = (int)e.size();
    l->mt = max_m <= 8 ? 1 : 2;
    return l;
}

extern "C" void ternaspmm_list_destroy(ternaspmm_list* l) { free(l); }

template <int MT, int W>
static cudaError_t launch_list(const ternaspmm_list* l, int* status, cudaStream_t stream) {
    using L = ListSmem<MT>;
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    auto kern = spmm_list_kernel<MT, W>;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(device_sm_count(), kListMaxCtas), 1, 1);       // one persistent CTA per SM
    cfg.blockDim = dim3(W * 32, 1, 1);                  // W - 1 decoder warps and one epilogue warp
    cfg.dynamicSmemBytes = L::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    t_echo = {5, MT * 8, 1, W, 0, (int)cfg.gridDim.x};
    return cudaLaunchKernelEx(&cfg, kern, static_cast<const ListItem*>(l->device_table), l->entries,
                              static_cast<uint8_t*>(l->scratch), status);
}

extern "C" void ternaspmm_list_run(ternaspmm_list* l, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (!l) {
        t_host_status = ST_BAD_POINTER;
        return;
    }
    int* status = status_device_ptr();
    if (!status) {
        t_host_status = ST_LAUNCH;
        return;
    }
#ifdef TSP_TUNING
    if (const char* ab = getenv("TERNASPMM_LIST_ABLATE")) {
        const int v = atoi(ab);
        cudaMemcpyToSymbol(g_list_ablate, &v, sizeof(int));
    }
#endif
    cudaError_t e;
    if (l->mt == 2) e = launch_list<2, 16>(l, status, stream);
    else if (tuning().list_warps == 24) e = launch_list<1, 24>(l, status, stream);
    else if (tuning().list_warps == 28) e = launch_list<1, 28>(l, status, stream);
    else e = launch_list<1, 20>(l, status, stream);   // 96 registers per thread, no spills: measured faster than 24 or 28 warps with spills
    if (e != cudaSuccess) {
        fprintf(stderr, "ternaspmm: list launch failed: %s\n", cudaGetErrorString(e));
        t_host_status = ST_LAUNCH;
    }
    checkLastCudaError(__LINE__);
}

extern "C" long long ternaspmm_lm_head_scratch_bytes(void) { return (long long)kHeadScratchBytes; }

extern "C" void ternaspmm_lm_head_argmax(__nv_bfloat16* h, __nv_bfloat16* embedding, int M, int V, int K, float* logits,
                                        long long* argmax, int round_bf16, void* scratch, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (M < 1 || M > 8 || V < 1 || K < 32 || (K % 32) || K > 12288) {
        fprintf(stderr, "ternaspmm: lm_head_argmax needs 1 <= M <= 8, V >= 1, K a multiple of 32 up to 12288 (got M=%d V=%d K=%d)\n",
                M, V, K);
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!h || !embedding || (!logits && !argmax) || (argmax && !scratch) || (reinterpret_cast<uintptr_t>(h) & 15) ||
        (reinterpret_cast<uintptr_t>(embedding) & 15) || (reinterpret_cast<uintptr_t>(scratch) & 15)) {
        fprintf(stderr, "ternaspmm: lm_head_argmax: null or misaligned pointer (h, embedding, scratch: 16 bytes)\n");
        t_host_status = ST_BAD_POINTER;
        return;
    }
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(lm_head_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * (12288 * 2 + 64)) != cudaSuccess ||
            cudaFuncSetAttribute(lm_head_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * (12288 * 2 + 64)) != cudaSuccess) {
            t_host_status = ST_LAUNCH;
            return;
        }
        attr_done[dev] = true;
    }
    HeadParams p;
    p.h = h, p.emb = embedding, p.logits = logits, p.argmax = argmax;
    p.counter = reinterpret_cast<unsigned int*>(scratch);
    p.cand = reinterpret_cast<HeadCandidate*>(reinterpret_cast<uint8_t*>(scratch) + 16);
    p.M = M, p.V = V, p.K = K, p.round_bf16 = round_bf16;
    const int groups = (V + 7) / 8, R = head_rows(V, device_sm_count());
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(std::min(device_sm_count(), groups), kHeadMaxCtas), 1, 1);
    cfg.blockDim = dim3(kHeadWarps * 32, 1, 1);
    cfg.dynamicSmemBytes = 8 * (K * 2 + 64);
    cfg.stream = stream;
    // No programmatic dependent launch for this kernel: it wants every SM for itself from the first cycle.
    // Launched early behind a kernel that releases its dependents at once (the library's norm kernel), its
    // CTAs compete for SMs with the still unplaced CTAs of the linears before it: measured on the 30-layer
    // model, the decoded token took 5 % longer.  In stream order it starts a few microseconds later and
    // runs on an empty chip.
    t_echo = {4, 8, 1, kHeadWarps, 0, (int)cfg.gridDim.x};
    if (cudaLaunchKernelEx(&cfg, R == 8 ? lm_head_kernel<8> : lm_head_kernel<16>, p) != cudaSuccess) t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
}

// ---- output head without any caller-provided scratch memory -------------------------------------
// Some callers of this library cannot hand it scratch memory at all: an operator plugged into a
// serving runtime that owns every byte of device memory through its own arena and forbids its
// operators to call cudaMalloc; a control loop for which the device-wide synchronisation hidden in
// cudaMalloc / cudaFree is unacceptable; code that runs while a stream is being captured, where an
// allocation is an error.  For them the arg-max candidates and the arrival counter of the head
// kernel live in the array below, which is part of the library's image: every GPU that loads the
// library holds these 16 KB until the process exits.
constexpr int kHeadStaticCtas = 256;   // candidate slots: the launch uses min(SMs, row groups, this many) CTAs
static __device__ __align__(256) unsigned char g_head_static_scratch[16 + sizeof(HeadCandidate) * 8 * kHeadStaticCtas];

// Device address of the array above on the current device.  The array's NAME is only a host-side
// handle here - passing it to a kernel would hand the GPU a host address - so the real address is
// asked for once per device, with that device current, and the answer is kept.
static void* head_static_scratch_ptr() {
    static void* ptrs[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!ptrs[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_head_static_scratch) != cudaSuccess || !p) {
            cudaGetLastError();
            return nullptr;
        }
        ptrs[dev] = p;
    }
    return ptrs[dev];
}

extern "C" void ternaspmm_lm_head_argmax_noalloc(__nv_bfloat16* h, __nv_bfloat16* embedding, int M, int V, int K,
                                                float* logits, long long* argmax, int round_bf16, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (M < 1 || M > 8 || V < 1 || K < 32 || (K % 32) || K > 12288) {
        fprintf(stderr, "ternaspmm: lm_head_argmax_noalloc: the built-in scratch area holds candidates for at most 8 rows; "
                        "needs 1 <= M <= 8, V >= 1, K a multiple of 32 up to 12288 (got M=%d V=%d K=%d)\n", M, V, K);
        t_host_status = ST_BAD_SHAPE;
        return;
    }
    if (!h || !embedding || (!logits && !argmax) || (reinterpret_cast<uintptr_t>(h) & 15) ||
        (reinterpret_cast<uintptr_t>(embedding) & 15)) {
        fprintf(stderr, "ternaspmm: lm_head_argmax_noalloc: null or misaligned pointer (h, embedding: 16 bytes)\n");
        t_host_status = ST_BAD_POINTER;
        return;
    }
    void* scratch = head_static_scratch_ptr();   // the first call on a device looks the address up
    if (!scratch) {
        fprintf(stderr, "ternaspmm: lm_head_argmax_noalloc: cannot resolve the built-in scratch area on this device\n");
        t_host_status = ST_LAUNCH;
        return;
    }
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(lm_head_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * (12288 * 2 + 64)) != cudaSuccess ||
            cudaFuncSetAttribute(lm_head_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * (12288 * 2 + 64)) != cudaSuccess) {
            t_host_status = ST_LAUNCH;
            return;
        }
        attr_done[dev] = true;
    }
    // every call shares the area and finds the previous call's candidates in it; only the arrival
    // counter has to start at zero, and it is cleared here rather than trusted
    if (cudaMemsetAsync(scratch, 0, 16, stream) != cudaSuccess) {
        t_host_status = ST_LAUNCH;
        return;
    }
    HeadParams p;
    p.h = h, p.emb = embedding, p.logits = logits, p.argmax = argmax;
    p.counter = reinterpret_cast<unsigned int*>(scratch);
    p.cand = reinterpret_cast<HeadCandidate*>(reinterpret_cast<uint8_t*>(scratch) + 16);
    p.M = M, p.V = V, p.K = K, p.round_bf16 = round_bf16;
    const int groups = (V + 7) / 8, R = head_rows(V, device_sm_count());
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(std::min(device_sm_count(), groups), kHeadStaticCtas), 1, 1);
    cfg.blockDim = dim3(kHeadWarps * 32, 1, 1);
    cfg.dynamicSmemBytes = 8 * (K * 2 + 64);
    cfg.stream = stream;
    if (cudaLaunchKernelEx(&cfg, R == 8 ? lm_head_kernel<8> : lm_head_kernel<16>, p) != cudaSuccess) t_host_status = ST_LAUNCH;
    checkLastCudaError(__LINE__);
}

extern "C" void ternaspmm_debug_inject_host_failure(int kind) {
    if (kind == 1) t_inject_encode_failure = 1;
}

extern "C" int ternaspmm_last_status(void);

// Measurement hook (see mma_rate_probe.cuh): int8 tensor-core operations per second that this GPU issues
// from shared-memory operands, over all SMs; 0 on failure.  Synchronises the stream.
extern "C" double ternaspmm_debug_int8_mma_rate(int iters, cudaStream_t stream) {
    t_host_status = ST_OK;
    if (iters < 64) iters = 64;
    iters = (iters + 63) / 64 * 64;
    int* status = status_device_ptr();
    const int smem_bytes = 1024 + 1024 + kLgAStage + 256 * kLgKStep;
    if (!status || cudaFuncSetAttribute(int8_mma_rate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) {
        t_host_status = ST_LAUNCH;
        return 0.0;
    }
    const int sms = device_sm_count();
    cudaEvent_t e0, e1;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return 0.0;
    int8_mma_rate_kernel<<<sms, 128, smem_bytes, stream>>>(64, status);   // warm-up
    cudaEventRecord(e0, stream);
    int8_mma_rate_kernel<<<sms, 128, smem_bytes, stream>>>(iters, status);
    cudaEventRecord(e1, stream);
    float ms = 0.f;
    const bool ok = cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess && ms > 0.f;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (!ok || ternaspmm_last_status() != 0) return 0.0;
    return 2.0 * 128 * 256 * 32 * 4.0 * iters * sms / (ms * 1e-3);
}

extern "C" void ternaspmm_set_wait_limit_ms(int ms) {
    if (ms < 1) ms = 1;
    if (ms > 10000) ms = 10000;
    g_wait_limit_ns = (unsigned long long)ms * 1000ull * 1000ull;
}

extern "C" void ternaspmm_last_launch_shape(int* out6) {
    if (!out6) return;
    out6[0] = t_echo.kernel, out6[1] = t_echo.tokens_per_pass, out6[2] = t_echo.splits, out6[3] = t_echo.warps;
    out6[4] = t_echo.row_tiles_per_cta, out6[5] = t_echo.ctas;
}

extern "C" int ternaspmm_last_status(void) {
    if (t_host_status != ST_OK) return t_host_status;
    int v = 0;
    int* d = status_device_ptr();
    if (!d) return ST_LAUNCH;
    if (cudaMemcpy(&v, d, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return ST_LAUNCH;
    if (v != 0) {
        int zero = 0;
        cudaMemcpy(d, &zero, sizeof(int), cudaMemcpyHostToDevice);
    }
    return v;
}

extern "C" void bitlinear_TernaSpMM_benchmark(int mode, int warmup_iters, int bench_iters, int8_t* x,
                                              uint64_t* bitmap, int* tile_offsets, uint16_t* quarter_offsets,
                                              uint32_t* sign_words, __nv_bfloat16* out, __nv_bfloat16* s,
                                              __nv_bfloat16* ws, int ws_num, int M, int N, int K, int split_k,
                                              int32_t* workspace, cudaStream_t stream) {
    if (mode < 0 || mode > 2) mode = 0;
    const int epilogue = mode == 1 ? EPI_PREFILL : (mode == 2 ? EPI_DECODE : (M <= 64 ? EPI_DECODE : EPI_PREFILL));
    (void)split_k;
    (void)workspace;
    for (int i = 0; i < warmup_iters; ++i)
        run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K, epilogue, stream);
    cudaStreamSynchronize(stream);
    checkLastCudaError(__LINE__);
    cudaEvent_t start, stop;
    cudaEventCreate(&start);
    cudaEventCreate(&stop);
    cudaEventRecord(start, stream);
    for (int i = 0; i < bench_iters; ++i)
        run_spmm(x, bitmap, tile_offsets, quarter_offsets, sign_words, out, s, ws, ws_num, M, N, K, epilogue, stream);
    cudaEventRecord(stop, stream);
    cudaEventSynchronize(stop);
    checkLastCudaError(__LINE__);
    float total_ms = 0.f;
    cudaEventElapsedTime(&total_ms, start, stop);
    const float avg_us = bench_iters > 0 ? total_ms / bench_iters * 1000.0f : 0.f;
    printf("Shape(M=%d, N=%d, K=%d): %.2f us (avg over %d iters, warmup=%d)\n", M, N, K, avg_us, bench_iters,
           warmup_iters);
    cudaEventDestroy(start);
    cudaEventDestroy(stop);
}

#ifdef TSP_PHASE_TIMERS
// Tuning builds only: copy the per-CTA phase timestamps of the last launch.
extern "C" int ternaspmm_debug_read_phases(unsigned long long* dst, int ctas) {
    if (ctas > 4096) ctas = 4096;
    return (int)cudaMemcpyFromSymbol(dst, g_phase_log, sizeof(unsigned long long) * ctas * kPhaseSlots);
}
#endif

extern "C" void gpu_sleep(double sleep_us, cudaStream_t stream) { sleep_kernel<<<1, 32, 0, stream>>>(sleep_us); }
