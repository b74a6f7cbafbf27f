// Few-token W4A16 contraction (decode batches of 2 to 5 tokens; to 8 or 16 on small matrices and where tcgen05 does not take
// the call) as a weight-streaming kernel whose inner product runs on the warp-level tensor-core instruction mma.sync.m16n8k16
// (fp16 x fp16 -> fp32).
//
// Why not tcgen05 here: at these token counts a launch is latency, and one on tcgen05 carries tensor-memory allocation,
// TMA round trips, commits and barrier hand-overs whatever the token count.  Here a launch is: weights into registers
// (before the wait for the previous kernel), tokens into shared memory, one barrier, MMAs, one exchange of partial sums.
//
// What bounds it: the chain above, and the dequantisation's ALU work.  So K is split until every SM has warps and no lane
// has more than a few 16-byte weight loads, over the warps of a CTA and over a cluster of CTAs, and a CTA stages only ITS
// K range of the tokens (staging all of K in every CTA was 72 KB per CTA at 4 tokens of K = 8960).  The weights go to
// shared memory, each lane copying what it will multiply itself (cp.async, no barrier): with weights in registers the loop
// over the steps had to be unrolled, and its 40 KB of code, executed once per launch, took longer to fetch than to run
// (gate_up at 4 tokens: 3 us of a launch).  The partial sums of all slices go straight to the CTA that finishes their
// rows, as 16-byte asynchronous stores counted on its mbarrier: the reduction over warps and over CTAs is one step.
//
// Arithmetic: the reference's prefill GEMM (src/kernels/gemm_prefill.cu:100-150): fp16 weights (q - 8) * scale with
// one rounding, fp16 activations, fp32 accumulation; epilogue as gemm_prefill.cu:257-275, 572-605.
//
// Mapping.  A warp owns 16 MMA rows and a slice of K in steps of 128: lane (g = lane / 4, t = lane % 4) loads, per step,
// the 16 bytes [32 t, 32 t + 32) of rows g and g + 8.  PLAIN / QKV: MMA row r is output row base + r.  SWIGLU: MMA row g
// is the gate row of pair base + g and row g + 8 its up row, so a lane ends with gate and up of the same output.
// The k index inside an MMA is free as long as A and B agree: MMA j (0..7) of a step takes, from each lane's piece,
// elements 4 j .. 4 j + 3 (k slots 2t, 2t+1 <- 4j, 4j+1; slots 2t+8, 2t+9 <- 4j+2, 4j+3).  The 16-byte chunk of a token that
// holds elements 8 m .. 8 m + 7 of lane t's piece is staged at position 4 m + t of its 256-byte step, and token rows are
// 64 bytes off a multiple of 128: the B operands of two MMAs are one 16-byte load without bank conflicts.
#pragma once

#include "gemm_smallm.cuh"

namespace w4 {

struct SmallMmaPlan {
    int row_groups;         // groups of 16 MMA rows per CTA
    int kslices;            // K slices per CTA (one warp per group and slice)
    int cluster;            // CTAs that share the rows of a CTA
    int steps;              // 128-element steps per slice at most
    int x_pitch;            // bytes of a staged token row
    int x_offset, part_offset;   // shared memory: weights and scales at 0, then the tokens, then the partial sums
};
constexpr int kMmaMaxCluster = 8;
constexpr int kMmaSlot = 1024 + 64;      // shared memory of one warp and step: weights, scale pairs

__device__ __forceinline__ void mma_m16n8k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ unsigned int g_mma_wait_timeouts = 0;

// Bounded wait for the stores of the cluster's CTAs that are counted on `bar`.
__device__ __forceinline__ bool wait_for_peers(uint32_t bar) {
    uint32_t ok = 0;
    for (unsigned it = 0; it < (1u << 22) && ok == 0; ++it)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar) : "memory");
    return ok != 0;
}

template <int MODE, int NT>
__global__ void __launch_bounds__(512, NT == 1 ? 2 : 1) gemm_smallm_mma_kernel(const SmallMArgs a, const SmallMmaPlan p) {
    constexpr int UW = (MODE == kSwiglu) ? 8 : 16;   // outputs per warp
    extern __shared__ __align__(128) uint8_t s_raw[];
    __shared__ __align__(8) uint64_t s_bar;
    const int K = a.g.K, M = a.g.M, G = K / kGroup;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int S = p.cluster, rank = static_cast<int>(blockIdx.x) % S, block = static_cast<int>(blockIdx.x) / S;
    const int ug = warp % p.row_groups, ks = warp / p.row_groups;
    const int unit0 = (block * p.row_groups + ug) * UW;    // first output of this warp
    const int slices = S * p.kslices, per = G / slices, rest = G - per * slices;
    auto slice_begin = [&](int sl) { return sl * per + min(sl, rest); };
    const int cta_begin = slice_begin(rank * p.kslices), cta_steps = slice_begin((rank + 1) * p.kslices) - cta_begin;
    const int slice = rank * p.kslices + ks, s_begin = slice_begin(slice), nst = per + (slice < rest ? 1 : 0);
    uint8_t* s_w = s_raw + static_cast<size_t>(warp) * p.steps * kMmaSlot;    // this warp: per step 2 x 32 lanes x 16 bytes, then 2 x 8 scale pairs
    uint8_t* s_x = s_raw + p.x_offset;
    uint8_t* s_part = s_raw + p.part_offset;        // [own group][slice][n][lane] x 16 bytes
    const int own_groups = rank < p.row_groups ? (p.row_groups - rank + S - 1) / S : 0;   // groups rank, rank + S, ...
    const uint32_t bar = static_cast<uint32_t>(__cvta_generic_to_shared(&s_bar));

    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(own_groups * slices * NT * 512) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    // the two weight rows of this lane (MMA rows g and g + 8) and where their outputs go
    const int words = K / 8;
    const uint32_t* wrow[2] = {nullptr, nullptr};
    const __half* srow[2] = {nullptr, nullptr};
    const bool active = unit0 < a.units;
    if (active) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            int tns = 0, local = MODE == kSwiglu ? 2 * (unit0 + g) + r : unit0 + g + 8 * r;
            if constexpr (MODE == kQkv) {
                if (local >= a.g.rows[0]) { local -= a.g.rows[0]; tns = 1; }
                if (tns == 1 && local >= a.g.rows[1]) { local -= a.g.rows[1]; tns = 2; }
            }
            wrow[r] = a.g.qweight[tns] + static_cast<size_t>(local) * words + s_begin * 16 + t * 4;
            srow[r] = a.g.scales[tns] + static_cast<size_t>(local) * G + s_begin;
        }
    }
    // Weights and scales into this lane's own slots, in two copy groups of half the steps each.  A scale comes as the aligned pair it is in
    // (K / 128 is even, the host checks the base): through registers it would hold up everything behind it.
    if (active) {
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(s_w)) + lane * 16;
        const uint32_t sdst = static_cast<uint32_t>(__cvta_generic_to_shared(s_w)) + 1024 + t * 32 + g * 4;
        const __half* ssrc = t == 0 ? srow[0] : srow[1];
#pragma unroll 1
        for (int u = 0; u < nst; ++u) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + u * kMmaSlot + r * 512), "l"(wrow[r] + u * 16) : "memory");
            if (t < 2) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sdst + u * kMmaSlot), "l"(ssrc + ((s_begin + u) & ~1) - s_begin) : "memory");
            if (u == (nst - 1) / 2) asm volatile("cp.async.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __syncthreads();        // the barrier exists
    if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    pdl_release_dependents();
    pdl_wait_prior_grids();

    // tokens of this CTA's K range, through registers (their copies must not queue behind the weights' groups)
    {
        constexpr int kBatch = 4;
        const int row_chunks = cta_steps * 16, total = M * row_chunks;
        const __half* x0 = a.g.x + static_cast<size_t>(cta_begin) * kGroup;
#pragma unroll 1
        for (int base = tid; base < total; base += kBatch * blockDim.x) {
            uint4 v[kBatch];
            int at[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int idx = base + i * blockDim.x;
                const int tok = idx / row_chunks, c = idx - tok * row_chunks;
                at[i] = tok * p.x_pitch + (c >> 4) * 256 + ((c & 3) * 4 + ((c >> 2) & 3)) * 16;
                if (idx < total) v[i] = *reinterpret_cast<const uint4*>(x0 + static_cast<size_t>(tok) * K + c * 8);
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i)
                if (base + i * static_cast<int>(blockDim.x) < total) *reinterpret_cast<uint4*>(s_x + at[i]) = v[i];
        }
    }
    __syncthreads();

    // (rows of tokens past M hold whatever the memory held: they only reach accumulator columns that nobody stores)
    float d[NT][2][4];      // even and odd MMAs apart: consecutive ones do not wait for each other
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i) d[n][c][i] = 0.0f;
    const uint8_t* x_lane[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n)    // (rows past M are read from an earlier row: the memory behind may not exist)
        x_lane[n] = s_x + min(n * 8 + g, M - 1) * p.x_pitch + (s_begin - cta_begin) * 256 + t * 16;
    const __half2 k10 = __float2half2_rn(1024.0f), m8 = __float2half2_rn(-8.0f);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();        // the scales were copied by other lanes of the warp
#pragma unroll 1
    for (int u = 0; active && u < nst; ++u) {
        if (u == (nst - 1) / 2 + 1) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();
        }
        const uint8_t* slot = s_w + u * kMmaSlot;
        const uint4 w0 = *reinterpret_cast<const uint4*>(slot + lane * 16), w1 = *reinterpret_cast<const uint4*>(slot + 512 + lane * 16);
        const int odd = ((s_begin + u) & 1) * 2;
        const __half sc0 = *reinterpret_cast<const __half*>(slot + 1024 + g * 4 + odd), sc1 = *reinterpret_cast<const __half*>(slot + 1056 + g * 4 + odd);
        const __half2 s0 = __half2half2(sc0), s1 = __half2half2(sc1);
        const bool small = __all_sync(0xFFFFFFFFu, __habs(sc0) < __float2half_rn(0.0624f) && __habs(sc1) < __float2half_rn(0.0624f));
        const __half2 s0_20 = __hmul2(__hmul2(s0, k10), k10), s1_20 = __hmul2(__hmul2(s1, k10), k10);
        const __half2 s0_m8 = __hmul2(s0, m8), s1_m8 = __hmul2(s1, m8);
        uint4 b[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int m = 0; m < 4; ++m) b[n][m] = *reinterpret_cast<const uint4*>(x_lane[n] + u * 256 + m * 64);
        auto multiply = [&](auto&& dequant) {
#pragma unroll
            for (int m = 0; m < 4; ++m) {                 // one packed word of each row = two MMAs
                uint32_t h0[4], h1[4];
                dequant(m == 0 ? w0.x : m == 1 ? w0.y : m == 2 ? w0.z : w0.w, s0, s0_20, s0_m8, h0);
                dequant(m == 0 ? w1.x : m == 1 ? w1.y : m == 2 ? w1.z : w1.w, s1, s1_20, s1_m8, h1);
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    mma_m16n8k16(d[n][0], h0[0], h1[0], h0[1], h1[1], b[n][m].x, b[n][m].y);
                    mma_m16n8k16(d[n][1], h0[2], h1[2], h0[3], h1[3], b[n][m].z, b[n][m].w);
                }
            }
        };
        // (one branch per step, so that the words of a step can overlap)
        if (small) multiply([](uint32_t w, __half2, __half2 s20, __half2 sm8, uint32_t* h) { dequant_word_small_scale(w, s20, sm8, h); });
        else multiply([](uint32_t w, __half2 s, __half2, __half2, uint32_t* h) { dequant_word_fp16(w, s, reinterpret_cast<__half2(&)[4]>(*h)); });
    }

    // partial sums to the CTA that finishes this row group
    if (S > 1) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // the peers have started
        const int owner = ug % S, lg = ug / S;
        const uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(s_part)) + static_cast<uint32_t>(((lg * slices + slice) * NT * 32 + lane) * 16);
        uint32_t dst, rbar;
        // (s_part lies at the same offset in every CTA: M and the pitch are the same)
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(local), "r"(owner));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbar) : "r"(bar), "r"(owner));
#pragma unroll
        for (int n = 0; n < NT; ++n)
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];"
                         ::"r"(dst + n * 512), "r"(rbar), "r"(__float_as_uint(d[n][0][0] + d[n][1][0])), "r"(__float_as_uint(d[n][0][1] + d[n][1][1])),
                           "r"(__float_as_uint(d[n][0][2] + d[n][1][2])), "r"(__float_as_uint(d[n][0][3] + d[n][1][3])) : "memory");
    } else {
        // no cluster: plain stores and a block barrier (asynchronous stores want a cluster launch)
        float4* dst = reinterpret_cast<float4*>(s_part) + (ug * slices + slice) * NT * 32 + lane;
#pragma unroll
        for (int n = 0; n < NT; ++n)
            dst[n * 32] = make_float4(d[n][0][0] + d[n][1][0], d[n][0][1] + d[n][1][1], d[n][0][2] + d[n][1][2], d[n][0][3] + d[n][1][3]);
        __syncthreads();
    }
    // The owner: one warp per group and token tile adds the slices in order.
    for (int wk = warp; wk < own_groups * NT; wk += static_cast<int>(blockDim.x >> 5)) {
        const int lg = wk / NT, n = wk - lg * NT;
        const int unit = (block * p.row_groups + rank + lg * S) * UW;
        const bool on = unit < a.units;
        int tns = 0, local = unit + g;
        if constexpr (MODE == kQkv) {       // the 16 rows of a group come from one tensor (host check)
            if (local >= a.g.rows[0]) { local -= a.g.rows[0]; tns = 1; }
            if (tns == 1 && local >= a.g.rows[1]) { local -= a.g.rows[1]; tns = 2; }
        }
        const int ld = a.out_ld[tns];
        const int tok = n * 8 + 2 * t;
        __half res[4];
        if constexpr (MODE == kPlain) {
            if (a.g.residual != nullptr) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (on && tok + (i & 1) < M) res[i] = a.g.residual[static_cast<size_t>(tok + (i & 1)) * ld + local + 8 * (i >> 1)];
            }
        }
        int have = S == 1;
        if (S > 1 && lane == 0) {
            have = wait_for_peers(bar) ? 1 : 0;
            if (!have) {
                atomicAdd(&g_mma_wait_timeouts, 1u);
                wait_for_peers(bar);     // what is still on its way into this CTA's memory has to land before it goes (bounded too)
            }
        }
        __syncwarp();            // the peers' stores before the reads of all lanes: a shuffle orders no memory
        have = __shfl_sync(0xFFFFFFFFu, have, 0);
        if (!have) break;
        float y[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const uint8_t* src = s_part + static_cast<size_t>((lg * slices * NT + n) * 32 + lane) * 16;
#pragma unroll 4
        for (int sl = 0; sl < slices; ++sl) {
            const float4 v = *reinterpret_cast<const float4*>(src + static_cast<size_t>(sl) * NT * 512);
            y[0] += v.x; y[1] += v.y; y[2] += v.z; y[3] += v.w;
        }
        __half* out = a.g.out[tns] + static_cast<size_t>(tok) * ld + local;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (on && tok + i < M) {
                if constexpr (MODE == kSwiglu) {
                    out[static_cast<size_t>(i) * ld] = __float2half_rn((y[i] / (1.0f + expf(-y[i]))) * y[2 + i]);
                } else {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        __half h = __float2half_rn(y[2 * r + i]);
                        if constexpr (MODE == kPlain) {
                            if (a.g.residual != nullptr) h = __hadd(h, res[2 * r + i]);
                        }
                        out[static_cast<size_t>(i) * ld + 8 * r] = h;
                    }
                }
            }
        }
    }
}

}  // namespace w4
