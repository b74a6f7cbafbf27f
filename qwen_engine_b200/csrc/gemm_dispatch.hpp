// Which form of the M-token contraction a call takes: a rule on its sizes, types and alignment alone.
#pragma once

#include <algorithm>

#include "w4a16_internal.hpp"

namespace w4 {

enum class GemmForm {
    kMma,    // weight streaming on mma.sync (gemm_smallm_mma.cuh)
    kTc,     // the tcgen05 kernels (gemm_tc.cu)
    kCuda,   // CUDA cores (gemm_smallm.cuh)
};

inline bool gemm_aligned16(const GemmArgs& g) {
    bool ok = reinterpret_cast<uintptr_t>(g.x) % 16 == 0;
    for (int t = 0; t < (g.mode == kQkv ? 3 : 1); ++t) ok = ok && reinterpret_cast<uintptr_t>(g.qweight[t]) % 16 == 0;
    return ok;
}

// Can the mma.sync form address this problem?  Rows in whole groups of 16 (a group of QKV rows from one tensor), scales in aligned
// pairs.  (Whether a cut of it fits is the planner's to say.)
inline bool gemm_mma_supported(const GemmArgs& g) {
    bool ok = gemm_aligned16(g) && g.num_peers == 0;
    for (int t = 0; t < (g.mode == kQkv ? 3 : 1); ++t)
        ok = ok && g.rows[t] % 16 == 0 && reinterpret_cast<uintptr_t>(g.scales[t]) % 4 == 0;
    return ok;
}

// `tc`, `mma`: the tcgen05 kernels and the mma.sync form can take the call.  `min_opt`, `mma_opt`: the options
// MIN_TOKENS_TENSOR_CORE and MMA_MAX_TOKENS.
inline GemmForm gemm_form(const GemmArgs& g, int sm_count, bool tc, bool mma, int min_opt, int mma_opt) {
    const int rows = g.rows[0] + (g.mode == kQkv ? g.rows[1] + g.rows[2] : 0);
    const size_t weights = static_cast<size_t>(rows) * g.K;

    // The tcgen05 kernel pads the token count to its smallest tile (16), so for shapes that the mma form below refuses the CUDA-core
    // form (the decode GEMV's memory behaviour with fp16 arithmetic) is the faster one at the fewest tokens: up to 3 on the narrow
    // K <= 4096 shapes (QKV, O), one where K > 4096 (the few-token form stages only two tokens per pass there) or where the matrix
    // gives every SM a CTA of its own.  CUDA cores / tcgen05, us: down 10.6 / 5.6 and gate_up 8.2 / 6.3 at 2 tokens, 8192 x 8192
    // 80 / 13 at 2, O 5.4 / 3.7 and QKV 4.4 / 3.8 at 4 (3.6 / 3.8 at 2).  The CUDA-core forms also take what TMA cannot address.
    const int tc_min_m = min_opt > 0 ? min_opt : (g.K > 4096 || rows >= 64 * sm_count ? 2 : 4);
    tc = tc && (g.M >= tc_min_m || g.num_peers > 0);     // (stores to peers exist in the tcgen05 kernels only)

    // A few tokens: the weight-streaming kernel with the warp-level MMA (no fixed tcgen05 costs).  Where tcgen05 takes the call
    // too, by what a layer takes, since CTAs of two launches share an SM in the mma form and one launch chained with itself says
    // little about that.  28 layers with weights of their own in a graph, us a layer, everything on mma / as the lines have it / mma
    // never:
    //   1536 / 8960   at 4 tokens 18.2 / 18.3 / 18.8, at 6 22.1 / 18.5 / 18.8 (from there on gate_up and down, 138 and 113 KB of shared
    //                 memory, no longer share an SM), at 9 22.5 / 19.0 / 19.0, at 16 24.1 / 19.4 / 19.2
    //   2048 / 8960   (gate_up 35 Mi weights) at 2 / 3 tokens 24.1 / 23.9, 24.5 / 24.2, at 5 24.6 / 24.5 / 21.4
    //   2048 / 6144   at 4 tokens 22.1 / 22.2 / 19.8, at 6 22.0 / 19.3 / 19.9, at 9 24.7 / 20.0 / 19.9
    //   1024 / 4096   at 6 tokens the lines leave it on mma: 12.8 to 13.9 against 14.8; at 9 14.9 / 15.1 / 14.9
    // (so a layer of 2048 would be better off whole on tcgen05 from 4 tokens, which no line by one matrix's size says.)
    // The smallest matrices keep mma to 16 tokens: 2048 x 512 at 9 2.9 / 3.5 chained with itself.  Where tcgen05 does not take it, up to 16 tokens whatever the size: mma / CUDA cores, us, 9216 x 4096 at 2 / 3 tokens
    // 8.2 / 37 and 8.3 / 58 (SWIGLU 8.1 / 11.3 and 8.2 / 20.4), QKV of 24 + 2 x 5 heads of 64 on K = 1536 at 9 / 16 4.4 / 10.9 and
    // 4.6 / 14.3, of 64 + 2 x 9 on K = 4096 at 6 / 16 7.5 / 30 and 9.2 / 71.
    const int mma_max_m = mma_opt > 0 ? mma_opt : !tc || weights <= 2u << 20 ? 16 : weights <= 10u << 20 ? 8 : weights <= 32u << 20 ? 5 : 1;
    if (mma && g.M >= std::max(2, min_opt) && g.M <= std::min(mma_max_m, 16)) return GemmForm::kMma;
    return tc ? GemmForm::kTc : GemmForm::kCuda;
}

}  // namespace w4
