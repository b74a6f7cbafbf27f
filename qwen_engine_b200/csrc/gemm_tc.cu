// M-token W4A16 contraction on the 5th-generation tensor cores (tcgen05 / TMEM), sm_100a: PTX wrappers, tensor maps, dispatch.
// The kernels: gemm_tc_stream.cuh (weight streaming with K split), gemm_tc_pair.cuh (CTA pairs, prefill).
//
// Replaces the reference's wmma prefill GEMMs (src/kernels/gemm_prefill.cu:319-610).
// Arithmetic is the reference's: weights dequantised to fp16 as (q - 8) * scale with one fp16
// rounding (include/quant_primitives.cuh:92-115), fp16 x fp16 products exact, fp32 accumulation,
// epilogue fp16(acc) [+ fp16 residual add] / SwiGLU on the fp32 accumulators
// (gemm_prefill.cu:257-275, 572-605).
//
// Formulation of both: D[n][m] = sum_k W[n][k] * X[m][k] with the WEIGHT rows on the 128-wide M side of the MMA and the
// tokens on its N side.  Every mbarrier wait is bounded: on expiry the kernel raises an abort flag, all roles leave their
// loops, TMEM is freed and the kernel returns; the host can read the count of such events with w4a16_debug_counter(0).
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "gemm_smallm.cuh"
#include "w4a16_common.cuh"
#include "w4a16_internal.hpp"

namespace w4 {

__device__ unsigned int g_tc_wait_timeouts = 0;

namespace {

constexpr int kTileRows = 128;          // weight rows per CTA (UMMA M)
constexpr int kBK = 64;                 // fp16 elements per k-block: one 128-byte swizzle row
constexpr unsigned kWaitLimit = 1u << 22;

// ---- PTX wrappers ------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// The same for a phase that stores of other CTAs of the cluster complete: what they wrote is read behind it.
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Non-blocking test of a phase (try_wait may park the thread for a while when the phase is still open).
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false if the barrier did not flip within the limit or another role gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_test_wait(bar, parity)) return true;   // already complete: no need to park the thread
    for (unsigned it = 0; it < kWaitLimit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (it > 2048) __nanosleep(64);
    }
    *abort_flag = 1;
    atomicAdd(&g_tc_wait_timeouts, 1u);
    return false;
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Cluster-wide barrier (all threads of all CTAs of the cluster) and stores into another CTA's shared memory.
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map_shared(uint32_t local_addr, uint32_t cta_rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(cta_rank));
    return remote;
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16 consecutive 32-bit columns of this thread's tensor-memory lane, from registers.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major tile, 128-byte swizzle, rows 128 B apart, 8-row groups
// 1024 B apart (stride byte offset), descriptor version 1 (sm_100).  `addr` may be advanced by
// 32 B per 16-element K slice inside the 128-byte swizzle row.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);   // start address, 16-byte units
    d |= static_cast<uint64_t>(1) << 16;                  // leading byte offset (unused with swizzle)
    d |= static_cast<uint64_t>(1024 >> 4) << 32;          // stride byte offset
    d |= static_cast<uint64_t>(1) << 46;                  // version
    d |= static_cast<uint64_t>(2) << 61;                  // SWIZZLE_128B
    return d;
}
// Instruction descriptor: D fp32, A/B fp16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t make_idesc(int n) {
    return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(kTileRows >> 4) << 24);
}

// One lane polls the barrier for its warp (512 threads polling would keep the mbarrier unit busy and
// delay the single MMA-issuing thread); __syncwarp then orders the other lanes' reads after it.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int lane) {
    int ok = 1;
    if (lane == 0) ok = mbar_wait(bar, parity, abort_flag) ? 1 : 0;
    __syncwarp();
    return __shfl_sync(0xFFFFFFFFu, ok, 0) != 0;
}

#include "gemm_tc_stream.cuh"
#include "gemm_tc_pair.cuh"

// ---- host side ----------------------------------------------------------------------------

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// A driver call wants a context current in the calling thread; the runtime binds the device's only with the thread's first
// call that needs it, and for a host thread whose first call is a launch of this file that would be the launch itself.
// True where there was none and now is; a context that the host made current itself stays.
bool bind_context() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    CUcontext ctx = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) return false;
    if (reinterpret_cast<CUresult (*)(CUcontext*)>(p)(&ctx) != CUDA_SUCCESS || ctx != nullptr) return false;
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess;
}

// A tensor map, encoded anew for each launch: 64 ns.  (Kept by address and shape in a table of 256 they took the host longer to find:
// four launches of a layer at 47 tokens 11.8 us with 28 layers and 12.3 with 80, so 11.6 and 11.5.)
bool encode_2d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t inner, uint64_t outer,
               uint64_t row_bytes, uint32_t box_inner, uint32_t box_outer,
               CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    auto encode = [&] {
        return fn(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    return encode() || (bind_context() && encode());
}

}  // namespace

int gemm_tc_set_attributes() {
    cudaError_t e = cudaSuccess;
    auto raise_pair = [&e](auto* kernel) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    };
    raise_pair(gemm_w4a16_tc_stream_kernel<kPlain>);
    raise_pair(gemm_w4a16_tc_stream_kernel<kQkv>);
    raise_pair(gemm_w4a16_tc_stream_kernel<kSwiglu>);
    raise_pair(gemm_w4a16_tc_pair_kernel<kPlain, kStoreValues>);
    raise_pair(gemm_w4a16_tc_pair_kernel<kPlain, kStoreWords>);
    raise_pair(gemm_w4a16_tc_pair_kernel<kPlain, kStoreWordsPeers>);
    raise_pair(gemm_w4a16_tc_pair_kernel<kQkv, kStoreValues>);
    raise_pair(gemm_w4a16_tc_pair_kernel<kQkv, kStoreWords>);
    raise_pair(gemm_w4a16_tc_pair_kernel<kSwiglu, kStoreWords>);
    return static_cast<int>(e);
}

// Can the tensor-core kernel take this problem?  (alignment for TMA, tile-aligned QKV tensors)
bool gemm_tc_supported(const GemmArgs& g) {
    if (encode_tiled_fn() == nullptr) return false;
    const int nt = g.mode == kQkv ? 3 : 1;
    for (int t = 0; t < nt; ++t) {
        if (reinterpret_cast<uintptr_t>(g.qweight[t]) % 16) return false;
        if (g.mode == kQkv && g.rows[t] % kTileRows) return false;
    }
    return reinterpret_cast<uintptr_t>(g.x) % 16 == 0;
}

namespace {
// The streaming kernel's cut of a shape: token tiles and K slices, two steps each at least, within one CTA per SM where that is
// possible, by the time it is estimated to take, in cycles of 1.9 GHz.  The constants are fitted to 2200 timed cuts of 14
// shapes (512 x 512 to 17920 x 1536 and 1536 x 8960) at 4 to 1024 tokens, launches one behind another (the cut they choose is on
// average 1.2 % slower than the best one).  The first steps hide behind the launch; a step is 400 of
// dequantisation, 650 beyond what the token slots hold, or 6 a token of its tile's way from L2; 35 a token of the tile for the
// epilogue; the exchange of a K split 1100 and 66 a token sent; CTAs on more than half of the SMs keep the next launch's from
// starting early; a further wave costs its launch again.
double stream_cost(int T, int split, int steps, int ctas, int sm_count) {
    const int per = (steps + split - 1) / split, waves = (ctas + sm_count - 1) / sm_count;
    const double work = std::max(0, std::min(per, 12) - 2) * std::max(400.0, 6.0 * T) + std::max(0, per - 12) * std::max(650.0, 6.0 * T) + 35.0 * T / split;
    const double exchange = split > 1 ? 1100.0 + 66.0 * T * (split - 1) / split : 0.0;
    const double crowd = 3100.0 * std::min(1.0, std::max(0.0, 2.0 * ctas / sm_count - 1.0));
    return 4700.0 + waves * work + exchange + crowd + 3200.0 * (waves - 1);
}
template <int MODE>
StreamPlan stream_plan(int M, int K, int tiles, int sm_count) {
    static PlanCache<StreamPlan> plans;
    return plans.get(plan_key(MODE, M, K, tiles), [&] {
        const int steps = K / kGroup;
        StreamPlan best;
        const int ts_min = (M + 127) / 128, ts_max = (M + 15) / 16;
        for (int ts = ts_min; ts <= ts_max; ++ts) {
            const int T = ((M + ts - 1) / ts + 15) & ~15;
            if (ts > ts_min && static_cast<long long>(tiles) * ts > sm_count) break;
            if (ts > ts_min && (M + T - 1) / T != ts) continue;
            for (int split = std::max(1, std::min({kStMaxSplit, sm_count / (tiles * ts), steps / 2})); split >= 1; --split) {
                const double cost = stream_cost(T, split, steps, tiles * ts * split, sm_count);
                if (best.smem != 0 && cost >= best.cost) continue;
                StreamPlan p;
                if (!plan_stream(T, split, steps, &p)) continue;
                if (split > 1 && max_active_clusters(reinterpret_cast<const void*>(gemm_w4a16_tc_stream_kernel<MODE>), kStThreads, p.smem, split) < tiles * ts) continue;
                best = p;
                best.cost = cost;
            }
        }
        return best;
    });
}
StreamPlan stream_plan(const GemmArgs& g, int tiles, int sm_count) {
    switch (g.mode) {
        case kPlain: return stream_plan<kPlain>(g.M, g.K, tiles, sm_count);
        case kQkv: return stream_plan<kQkv>(g.M, g.K, tiles, sm_count);
        default: return stream_plan<kSwiglu>(g.M, g.K, tiles, sm_count);
    }
}
// What both kernels' arguments have in common.
template <typename Args>
int fill_args(const GemmArgs& g, Args* a, int* total_tiles) {
    const int nt = g.mode == kQkv ? 3 : 1;
    *total_tiles = 0;
    for (int t = 0; t < 3; ++t) {
        a->scales[t] = g.scales[t];
        a->out[t] = g.out[t];
        a->rows[t] = t < nt ? g.rows[t] : 0;
        a->tiles[t] = (a->rows[t] + kTileRows - 1) / kTileRows;
        *total_tiles += a->tiles[t];
        a->out_ld[t] = g.mode == kSwiglu ? g.rows[0] / 2 : a->rows[t];
        if (g.mode == kPlain && t == 0 && g.ldc > 0) a->out_ld[0] = g.ldc;
    }
    a->residual = g.residual;
    a->M = g.M;
    a->K = g.K;
    a->num_peers = g.mode == kPlain ? g.num_peers : 0;
    for (int p = 0; p < 7; ++p) a->peer_out[p] = p < a->num_peers ? g.peer_out[p] : nullptr;
    for (int t = 0; t < nt; ++t) {
        if (!encode_2d(&a->tmap_w[t], CU_TENSOR_MAP_DATA_TYPE_UINT8, g.qweight[t], static_cast<uint64_t>(g.K / 2),
                       static_cast<uint64_t>(g.rows[t]), static_cast<uint64_t>(g.K / 2), 64, kTileRows, CU_TENSOR_MAP_SWIZZLE_64B))
            return W4A16_ERR_INVALID_ARG;
    }
    for (int t = nt; t < 3; ++t) a->tmap_w[t] = a->tmap_w[0];
    return 0;
}
int stream_launch(const GemmArgs& g, const StreamPlan& plan, cudaStream_t stream) {
    StreamArgs a;
    int tiles = 0;
    if (int e = fill_args(g, &a, &tiles)) return e;
    a.p = plan;
    if (!encode_2d(&a.tmap_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.x, static_cast<uint64_t>(g.K), static_cast<uint64_t>(g.M),
                   static_cast<uint64_t>(g.K) * 2, kBK, static_cast<uint32_t>(plan.T)))
        return W4A16_ERR_INVALID_ARG;
    auto launch = [&](auto* kernel) {
        return static_cast<int>(launch_kernel_cluster(kernel, dim3(tiles, (g.M + plan.T - 1) / plan.T, plan.ksplit), dim3(kStThreads), plan.smem, stream,
                                                      pdl_enabled(), dim3(1, 1, static_cast<unsigned>(plan.ksplit)), a));
    };
    switch (g.mode) {
        case kPlain: return launch(gemm_w4a16_tc_stream_kernel<kPlain>);
        case kQkv: return launch(gemm_w4a16_tc_stream_kernel<kQkv>);
        default: return launch(gemm_w4a16_tc_stream_kernel<kSwiglu>);
    }
}
int pair_launch(const GemmArgs& g, int sm_count, cudaStream_t stream) {
    PairArgs a;
    int tiles = 0;
    if (int e = fill_args(g, &a, &tiles)) return e;
    const int n_pairs = (tiles + 1) / 2, pairs = std::max(1, sm_count / 2);
    const int T = pair_token_tile(g.M, n_pairs, g.K / kGroup, pairs, nullptr);
    a.halves = T > kPairAccCols ? 2 : 1;
    a.n_half = T / a.halves;
    // Two rows of an output as one word: even strides and rows, 4-byte aligned.
    auto word = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 4 == 0; };
    bool words = word(a.residual);
    for (int p = 0; p < a.num_peers; ++p) words = words && word(a.peer_out[p]);
    for (int t = 0; t < (g.mode == kQkv ? 3 : 1); ++t) words = words && a.out_ld[t] % 2 == 0 && a.rows[t] % 2 == 0 && word(a.out[t]);
    // weight matrices that do not stay in L2 next to the tokens and outputs: panels of 4 token tiles (28672 x 8192 at 4096
    // tokens, passes back to back: 1543 us in panels of 1, 1460 in panels of 4); smaller ones: row tiles fastest
    a.panel = static_cast<size_t>(tiles) * kTileRows * (g.K / 2) > (48u << 20) ? 4 : 1;
    if (!encode_2d(&a.tmap_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.x, static_cast<uint64_t>(g.K), static_cast<uint64_t>(g.M),
                   static_cast<uint64_t>(g.K) * 2, kBK, static_cast<uint32_t>(a.n_half / 2)))
        return W4A16_ERR_INVALID_ARG;
    // persistent: one pair per two SMs, each walking the pair tiles p, p + P, ...
    const int grid = 2 * std::min(pairs, n_pairs * ((g.M + T - 1) / T));
    const size_t smem = tc_pair_smem_bytes(g.mode, T);
    auto launch = [&](auto* kernel) {
        return static_cast<int>(launch_kernel_cluster(kernel, dim3(grid), dim3(kPairThreads), smem, stream, pdl_enabled(), dim3(2, 1, 1), a));
    };
    switch (g.mode) {
        case kPlain:
            if (!words) return launch(gemm_w4a16_tc_pair_kernel<kPlain, kStoreValues>);
            return a.num_peers > 0 ? launch(gemm_w4a16_tc_pair_kernel<kPlain, kStoreWordsPeers>) : launch(gemm_w4a16_tc_pair_kernel<kPlain, kStoreWords>);
        case kQkv: return words ? launch(gemm_w4a16_tc_pair_kernel<kQkv, kStoreWords>) : launch(gemm_w4a16_tc_pair_kernel<kQkv, kStoreValues>);
        default: return launch(gemm_w4a16_tc_pair_kernel<kSwiglu, kStoreWords>);
    }
}
}  // namespace

// Up to 256 tokens the streaming kernel (more CTAs, K split), above that whichever of the two is estimated to be faster: thin
// matrices stay with the streaming kernel up to about 1024 tokens (streaming / pairs, us, at 1024: QKV 8.4 / 10.7, O 9.3 / 11.1,
// down 25.0 / 31.8), gate_up goes to pairs at once (23.1 / 20.0 at 300, 32.3 / 24.8 at 450).  W4A16_OPT_GEMM_FORM = 1 / 2 asks for one of them.
int gemm_tc_launch(const GemmArgs& g, int sm_count, cudaStream_t stream) {
    const int form = option(W4A16_OPT_GEMM_FORM);
    if (form != 2) {
        int tiles = 0;
        for (int t = 0; t < (g.mode == kQkv ? 3 : 1); ++t) tiles += (g.rows[t] + kTileRows - 1) / kTileRows;
        const StreamPlan plan = stream_plan(g, tiles, sm_count);
        double pairs_cost = 0;
        if (form == 0 && g.M > 256) pair_token_tile(g.M, (tiles + 1) / 2, g.K / kGroup, std::max(1, sm_count / 2), &pairs_cost);
        if (plan.smem != 0 && (form == 1 || g.M <= 256 || plan.cost < pairs_cost)) return stream_launch(g, plan, stream);
    }
    return pair_launch(g, sm_count, stream);
}

int gemm_tc_timeouts(unsigned int* out) {
    return static_cast<int>(cudaMemcpyFromSymbol(out, g_tc_wait_timeouts, sizeof(unsigned int)));
}

}  // namespace w4
