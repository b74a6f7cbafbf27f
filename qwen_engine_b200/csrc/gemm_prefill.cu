// Host dispatch of the M-token W4A16 contraction (small-M decode batches and prefill).
#include <algorithm>

#include "gemm_dispatch.hpp"
#include "gemm_smallm.cuh"
#include "gemm_smallm_mma.cuh"
#include "w4a16_internal.hpp"

namespace w4 {
namespace {

template <int MODE>
cudaError_t launch_smallm(const SmallMArgs& a, int mt, dim3 grid, dim3 block, cudaStream_t stream) {
    const bool pdl = pdl_enabled();
    switch (mt) {
        case 1: return launch_kernel(gemm_smallm_kernel<MODE, 1>, grid, block, 0, stream, pdl, a);
        case 2: return launch_kernel(gemm_smallm_kernel<MODE, 2>, grid, block, 0, stream, pdl, a);
        default: return launch_kernel(gemm_smallm_kernel<MODE, 4>, grid, block, 0, stream, pdl, a);
    }
}

// ---- few-token form (gemm_smallm_v2_kernel) ----
template <int MODE, int U, int MT>
cudaError_t launch_v2_one(const SmallMArgs& a, const SmallMPlan& p, dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    return launch_kernel(gemm_smallm_v2_kernel<MODE, U, MT>, grid, block, smem, stream, pdl_enabled(), a, p);
}
template <int MODE>
cudaError_t launch_v2(const SmallMArgs& a, const SmallMPlan& p, int U, int mt, dim3 grid, dim3 block, size_t smem,
                      cudaStream_t stream) {
    if (U == 4) {
        if (mt == 1) return launch_v2_one<MODE, 4, 1>(a, p, grid, block, smem, stream);
        if (mt == 2) return launch_v2_one<MODE, 4, 2>(a, p, grid, block, smem, stream);
        return launch_v2_one<MODE, 4, 4>(a, p, grid, block, smem, stream);
    }
    if (mt == 1) return launch_v2_one<MODE, 8, 1>(a, p, grid, block, smem, stream);
    if (mt == 2) return launch_v2_one<MODE, 8, 2>(a, p, grid, block, smem, stream);
    return launch_v2_one<MODE, 8, 4>(a, p, grid, block, smem, stream);
}
template <int MODE, int U, int MT>
cudaError_t raise_v2() {
    return cudaFuncSetAttribute(gemm_smallm_v2_kernel<MODE, U, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
}
template <int MODE>
cudaError_t raise_v2_mode() {
    cudaError_t e = raise_v2<MODE, 4, 1>();
    if (e == cudaSuccess) e = raise_v2<MODE, 4, 2>();
    if (e == cudaSuccess) e = raise_v2<MODE, 4, 4>();
    if (e == cudaSuccess) e = raise_v2<MODE, 8, 1>();
    if (e == cudaSuccess) e = raise_v2<MODE, 8, 2>();
    if (e == cudaSuccess) e = raise_v2<MODE, 8, 4>();
    return e;
}

// CTA shape of the few-token form: as the decode GEMV's -- enough CTAs for every SM, all sub-warps busy,
// the K range of a sub-warp at most 8 steps deep, and the whole grid resident (16 warps per SM at the
// kernel's 128 registers).  Returns false when a K slice would be deeper than 8 steps.
bool plan_v2(const GemmArgs& g, int units, int sm_count, SmallMPlan* out, int* U) {
    const int steps = g.K / kStepElems;
    const int target = (sm_count * 13 + 9) / 10;
    int upc = 32;
    while (upc > 4 && (units + upc - 1) / upc < target) upc /= 2;
    if (g.mode == kQkv)
        while (upc > 1 && (g.rows[0] % upc || g.rows[1] % upc)) upc /= 2;
    int cap = std::min(std::max(1, 32 / upc), steps);
    int per = (steps + cap - 1) / cap;
    int ksplit = (steps + per - 1) / per;
    const int grid = (units + upc - 1) / upc;
    while (ksplit > 1 && per < 8) {
        const int warps = (upc * ksplit * kSubwarp + 31) / 32;
        if (grid <= (16 / warps) * sm_count) break;
        per = (steps + (ksplit - 1) - 1) / (ksplit - 1);
        ksplit = (steps + per - 1) / per;
    }
    if (per > 8) return false;
    out->units_per_cta = upc;
    out->ksplit = ksplit;
    out->steps_per_split = per;
    *U = per <= 4 ? 4 : 8;
    return true;
}

// ---- few-token mma.sync form (gemm_smallm_mma_kernel) ----
constexpr size_t kMmaMaxSmem = 200 * 1024;
using MmaKernel = void (*)(const SmallMArgs, const SmallMmaPlan);
template <int MODE>
MmaKernel mma_kernel_nt(int NT) {
    return NT == 1 ? gemm_smallm_mma_kernel<MODE, 1> : gemm_smallm_mma_kernel<MODE, 2>;
}
MmaKernel mma_kernel(int mode, int NT) {
    return mode == kPlain ? mma_kernel_nt<kPlain>(NT) : mode == kQkv ? mma_kernel_nt<kQkv>(NT) : mma_kernel_nt<kSwiglu>(NT);
}
cudaError_t raise_mma() {
    for (int mode : {static_cast<int>(kPlain), static_cast<int>(kQkv), static_cast<int>(kSwiglu)})
        for (int NT : {1, 2}) {
            cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(mma_kernel(mode, NT)), cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaMaxSmem);
            if (e != cudaSuccess) return e;
            // the same carve-out for every kernel of a layer: CTAs of two launches share an SM only if they agree on it
            e = cudaFuncSetAttribute(reinterpret_cast<const void*>(mma_kernel(mode, NT)), cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

struct MmaLaunch {
    SmallMmaPlan plan{};
    int NT = 0, grid = 0, block = 0;
    size_t smem = 0;
    bool ok = false;
};
// How the rows and K are cut: the cheapest of all cuts that keep the whole grid resident (16 warps per SM) by an estimate in
// cycles: per warp and step 34 + 3 NT issue slots or 16 NT tensor-core cycles, whichever is more, and 300 of latency per
// step of the chain; the staging of a CTA's tokens at 25 bytes a cycle; 900 for an exchange over a cluster, 1200 more where
// the clusters would fill nearly every SM (the GPCs' sizes are not multiples of theirs, so the last ones wait: down at 4
// tokens 6.0 us as 24 clusters of 6, 5.0 as 24 of 5); 500 per further CTA on an SM (they stand in the way of the
// next launch's); the owner's addition of the slices.
MmaLaunch plan_mma(int mode, int units, int M, int K, int sm_count) {
    MmaLaunch best;
    const int uw = mode == kSwiglu ? 8 : 16, groups = units / uw, G = K / kGroup;
    if (M > 16) return best;
    const int NT = M <= 8 ? 1 : 2;
    double best_cost = 0;
    for (int rg : {1, 2, 4, 8})
        for (int ks : {1, 2, 4, 8, 16}) {
            const int warps = rg * ks;
            if (warps > 16) continue;
            for (int S = 1; S <= kMmaMaxCluster; ++S) {
                const int slices = ks * S, per = (G + slices - 1) / slices;
                if (slices > G || per > 16) continue;
                const int blocks = (groups + rg - 1) / rg, ctas = blocks * S, per_sm = (ctas + sm_count - 1) / sm_count;
                if (per_sm * warps > 16) continue;
                const int cta_steps = std::min(G, ks * per), own = (rg + S - 1) / S;
                MmaLaunch c;
                c.plan.row_groups = rg; c.plan.kslices = ks; c.plan.cluster = S; c.plan.steps = per;
                c.plan.x_pitch = cta_steps * 256 + 64;
                c.plan.x_offset = warps * per * kMmaSlot;
                c.plan.part_offset = c.plan.x_offset + M * c.plan.x_pitch;
                c.smem = static_cast<size_t>(c.plan.part_offset) + static_cast<size_t>(own) * slices * NT * 512;
                if (c.smem * per_sm > kMmaMaxSmem) continue;
                const double cost = static_cast<double>(per_sm) * warps * per * std::max(34.0 + 3 * NT, 16.0 * NT) + 300.0 * per +
                                    static_cast<double>(per_sm) * M * cta_steps * 256 / 25 + 12.0 * slices * ((own * NT + warps - 1) / warps) +
                                    (S == 1 ? 0.0 : ctas > 0.85 * per_sm * sm_count ? 2100.0 : 900.0) + 500.0 * (per_sm - 1);
                if (best.ok && cost >= best_cost) continue;
                c.NT = NT; c.grid = ctas; c.block = 32 * warps; c.ok = true;
                if (S > 1 && max_active_clusters(reinterpret_cast<const void*>(mma_kernel(mode, NT)), c.block, c.smem, S) < blocks) continue;
                best = c;
                best_cost = cost;
            }
        }
    return best;
}

}  // namespace

int gemm_set_attributes() {
    cudaError_t e = raise_v2_mode<kPlain>();
    if (e == cudaSuccess) e = raise_v2_mode<kQkv>();
    if (e == cudaSuccess) e = raise_v2_mode<kSwiglu>();
    if (e == cudaSuccess) e = raise_mma();
    if (e != cudaSuccess) return static_cast<int>(e);
    return gemm_tc_set_attributes();
}

int gemm_mma_timeouts(unsigned int* out) {
    return static_cast<int>(cudaMemcpyFromSymbol(out, g_mma_wait_timeouts, sizeof(unsigned int)));
}

int gemm_launch(GemmArgs g, cudaStream_t stream) {
    const DeviceInfo* dev = nullptr;
    if (int st = ensure_device_ready(&dev)) return st;

    SmallMArgs a;
    a.g = g;
    const int total_rows = g.rows[0] + (g.mode == kQkv ? g.rows[1] + g.rows[2] : 0);
    a.units = (g.mode == kSwiglu) ? total_rows / 2 : total_rows;
    if (g.mode == kQkv) {
        a.out_ld[0] = g.rows[0]; a.out_ld[1] = g.rows[1]; a.out_ld[2] = g.rows[2];
    } else {
        a.out_ld[0] = (g.mode == kPlain && g.ldc > 0) ? g.ldc : a.units; a.out_ld[1] = a.out_ld[2] = 0;
    }
    const bool tc = gemm_tc_supported(g);
    auto form_of = [&](bool mma) {
        return gemm_form(g, dev->sm_count, tc, mma, option(W4A16_OPT_GEMM_MIN_TOKENS_TENSOR_CORE), option(W4A16_OPT_GEMM_MMA_MAX_TOKENS));
    };
    GemmForm form = form_of(gemm_mma_supported(g));
    if (form == GemmForm::kMma) {
        static PlanCache<MmaLaunch> plans;
        const MmaLaunch m = plans.get(plan_key(g.mode, g.M, g.K, a.units), [&] { return plan_mma(g.mode, a.units, g.M, g.K, dev->sm_count); });
        if (m.ok)
            return static_cast<int>(launch_kernel_cluster(mma_kernel(g.mode, m.NT), dim3(m.grid), dim3(m.block), m.smem, stream, pdl_enabled(),
                                                          dim3(static_cast<unsigned>(m.plan.cluster), 1, 1), a, m.plan));
        form = form_of(false);
    }
    if (form == GemmForm::kTc) return gemm_tc_launch(g, dev->sm_count, stream);
    if (g.num_peers > 0) return W4A16_ERR_SHAPE;   // peer stores exist in the tensor-core form only

    // few tokens, 16-byte aligned tensors: the form that streams like the decode GEMV
    SmallMPlan plan;
    int U = 8;
    if (gemm_aligned16(g) && plan_v2(g, a.units, dev->sm_count, &plan, &U)) {
        const int R = g.mode == kSwiglu ? 2 : 1;
        // tokens per pass: as many as the shared-memory budget of a CTA (about a third of an SM) allows
        int mt = g.M >= 4 ? 4 : (g.M >= 2 ? 2 : 1);
        auto smem_for = [&](int t) {
            return (static_cast<size_t>(t) * smallm_x_stride(g.K) + static_cast<size_t>(plan.ksplit) * plan.units_per_cta * R * t) * sizeof(float);
        };
        if (g.mode == kSwiglu && U == 8) mt = std::min(mt, 2);   // row pairs with 8 loads each: the registers are full
        while (mt > 1 && smem_for(mt) > 72 * 1024) mt /= 2;
        if (smem_for(mt) <= 160 * 1024) {
            const int threads = plan.units_per_cta * plan.ksplit * kSubwarp;
            const dim3 grid2((a.units + plan.units_per_cta - 1) / plan.units_per_cta), block2((threads + 31) / 32 * 32);
            cudaError_t e2;
            switch (g.mode) {
                case kPlain: e2 = launch_v2<kPlain>(a, plan, U, mt, grid2, block2, smem_for(mt), stream); break;
                case kQkv: e2 = launch_v2<kQkv>(a, plan, U, mt, grid2, block2, smem_for(mt), stream); break;
                default: e2 = launch_v2<kSwiglu>(a, plan, U, mt, grid2, block2, smem_for(mt), stream); break;
            }
            return static_cast<int>(e2);
        }
    }
    int upc = 32;
    const int target = (dev->sm_count * 13 + 9) / 10;
    while (upc > 4 && (a.units + upc - 1) / upc < target) upc /= 2;
    if (g.mode == kQkv)
        while (upc > 1 && (g.rows[0] % upc || g.rows[1] % upc)) upc /= 2;
    a.units_per_cta = upc;
    const int mt = g.M >= 4 ? 4 : (g.M >= 2 ? 2 : 1);
    const dim3 grid((a.units + upc - 1) / upc), block(std::max(32, upc * kSubwarp));
    cudaError_t e;
    switch (g.mode) {
        case kPlain: e = launch_smallm<kPlain>(a, mt, grid, block, stream); break;
        case kQkv: e = launch_smallm<kQkv>(a, mt, grid, block, stream); break;
        default: e = launch_smallm<kSwiglu>(a, mt, grid, block, stream); break;
    }
    return static_cast<int>(e);
}

}  // namespace w4
