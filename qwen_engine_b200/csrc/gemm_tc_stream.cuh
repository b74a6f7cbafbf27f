// Batched-decode W4A16 contraction on tcgen05 (from a few tokens, by size, to 256; thin matrices above) as a weight-streaming
// kernel.  Included by gemm_tc.cu behind the PTX wrappers.
//
// What bounds it: at these token counts a launch reads 1-14 MB of packed weights (0.2-2 us of HBM time) and the rest is
// latency -- the launch boundary, the dequantisation, the token tile's way from L2, the hand-overs between roles, the
// K-split exchange.  So what does not depend on the previous kernel is done before the wait for it (barriers, group scales,
// the ring of weights, the first steps' dequantisation), hand-overs are few (one barrier wait per 128 k in each role), and
// tokens and K are split over CTAs where the row tiles alone leave SMs idle.
//
// D[n][m] = sum_k W[n][k] X[m][k], 128 weight rows on the M side of the MMA, T tokens on its N side, in steps of 128 k (one
// quantisation group).  A (dequantised weights) goes from registers to tensor memory, a thread owning a weight row = a TMEM
// lane; B (tokens) comes from shared memory.  With A in tensor memory an MMA of 16..64 tokens takes 12..32 cycles against
// 40..48 with A in shared memory (measured in a loop), provided the issuing thread is chosen by elect.sync: behind a
// `lane == 0` branch every operand is moved to a uniform register first and each MMA costs 67.
//
//   warps 0..15 : dequantise, four warps a step (steps s % 4), then the epilogue
//   warp 16     : allocates tensor memory; one thread issues the MMAs of the even steps (8 per step) behind ONE barrier per slot
//                 that counts the dequantising warps and the token tile's bytes; warp 19 the same for the odd steps, which have an
//                 accumulator of their own
//   warp 17     : one thread loads packed weights by TMA, 128 rows x 128 k (8 KB) per ring slot
//   warp 18     : one thread loads tokens by TMA, T x 128 k per slot
//
// The loading threads are chosen by elect.sync too, and each ring has one of its own: as one `lane == 0` thread that looked
// after both rings a step took them 430 cycles, and with every other part of the kernel taken out a launch was hardly faster
// (gate_up at 47 tokens 8.6 us, 5.7 without data, dequantisation, MMAs or epilogue).  Every token slot that fits is asked for at
// once.  One layer of 1536 / 8960 at 47 tokens: QKV 6.0 -> 4.7, O 5.6 -> 4.3, gate_up 8.5 -> 6.7, down 8.4 -> 6.4 us a launch (as
// the kernel is now 4.3, 4.3, 6.1 and 6.5).
//
// Tensor memory: even and odd steps go into accumulators of their own: half as many additions per fp32 sum, which at
// K = 8192 is the difference between 2.7 and 2 fp16 steps of error.  A slots of 64 columns follow: six up to 64 tokens,
// four above.
//
// K split: every CTA of a cluster finishes its own share of the tokens.  Partials travel as 16-byte asynchronous stores
// into the owner's shared memory which count themselves on the owner's mbarrier, so the exchange needs no cluster barrier
// behind it; the one that makes sure that the peers have started is passed before the main loop.  A CTA sends T x 512 bytes
// at about 18 bytes a cycle, which is why the planner prefers a smaller token tile to a deeper K split.
constexpr int kStGroups = 4;                     // groups of four dequantising warps = 128 rows
constexpr int kStDqWarps = 4 * kStGroups, kStDqThreads = kStDqWarps * 32;
constexpr int kStWeightWarp = kStDqWarps + 1, kStTokenWarp = kStDqWarps + 2;      // the others behind the dequantising ones issue MMAs
constexpr int kStIssuers = 2;
constexpr int kStThreads = kStDqThreads + (2 + kStIssuers) * 32;
constexpr int kStRawBytes = kTileRows * 64;      // 128 rows x 128 k of packed nibbles
constexpr int kStMaxRaw = 24, kStMaxSlots = 12;  // ring slots at most
constexpr int kStACols = kGroup / 2;             // 128 k of fp16 = 64 columns
constexpr int kStMaxSplit = 8;                   // portable cluster size

// How a launch is cut.
struct StreamPlan {
    int T;                // tokens of a CTA's tile
    int ksplit;           // cluster size along grid z
    int steps_each;       // steps of every slice; the first K / 128 - ksplit * steps_each have one more
    int tpr;              // tokens a CTA of the cluster finishes (multiple of 4)
    int raw_slots;        // multiple of 4: a slot always belongs to the same group of dequantising warps (parity waits)
    int a_slots;          // A slots in tensor memory, at least `groups` (the MMAs complete in order, so a group is never two uses ahead)
    int slots;            // token slots, and barriers of a step; at least a_slots.  Both even: an issuing thread has its own slots
    int x_mem;            // token slots that have memory: `slots`, or the steps of a short K range
    int part_offset;      // K split: byte offset of the partials in shared memory; 0 = on top of the rings
    int acc2_col, a_col;  // second accumulator; first column of the A slots
    size_t smem = 0;      // 0: does not fit
    double cost = 0;      // estimated cycles
};
struct StreamArgs {
    CUtensorMap tmap_w[3];
    CUtensorMap tmap_x;
    const __half* scales[3];
    __half* out[3];
    int rows[3];
    int out_ld[3];
    int tiles[3];
    const __half* residual;
    int M, K;
    StreamPlan p;
    __half* peer_out[7];  // PLAIN: the output block's place in other GPUs' matrices
    int num_peers;
};

// One thread of the (converged) warp, in a form the compiler knows to be warp-uniform.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// D[tmem] (+)= A[tmem] * B[smem]^T, one CTA.
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// 16 bytes into a CTA of the cluster; the bytes are counted on the barrier there once they have landed.
__device__ __forceinline__ void st_async_16(uint32_t cluster_addr, uint32_t cluster_bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];"
                 ::"r"(cluster_addr), "r"(cluster_bar), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Bounded wait that does not look at the abort flag.
__device__ __forceinline__ bool wait_regardless(uint32_t bar, uint32_t parity, unsigned limit) {
    for (unsigned it = 0; it < limit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// 8 token columns of this thread's weight row, both accumulators added.
__device__ __forceinline__ void stream_load_acc(uint32_t taddr, int acc2_col, float (&v)[8]) {
    uint32_t x[8], y[8];
    tmem_ld8(taddr, x);
    tmem_ld8(taddr + static_cast<uint32_t>(acc2_col), y);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(x[j]) + __uint_as_float(y[j]);
}

// gate / (1 + e^-gate) * up.  The quotient: by the approximate reciprocal (1 ulp), then one correction by its residual, Newton's
// step for a quotient, which leaves little but the last rounding.  The divisor is a sixteenth (and up with it): the reciprocal of
// one above 2^126, gates of -87.4 to -88.7, would be flushed to zero, and an infinite up then made NaN of it.  No correction where
// there is nothing to correct or no residual (NaN, with an infinite gate or divisor): the quotient itself is right there, the sign
// of a zero included.  Compared with an IEEE division for every gate of 2^-48 to 2^124 (sums of fp16 products lie in between), of
// both signs, zeros and infinities: the same bits.  Its checks and branch cost gate_up at 300 / 512 / 1024 tokens 22.0 / 26.1 / 44.0
// us, so 20.4 / 24.9 / 42.7, and with the sixteenth 1 % more.
__device__ __forceinline__ float swiglu_f32(float gate, float up) {
    const float d = fmaf(0.0625f, expf(-gate), 0.0625f);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = gate * r, rest = fmaf(-q, d, gate);
    return (fabsf(rest) > 0.0f ? fmaf(rest, r, q) : q) * (0.0625f * up);
}

// NV tokens m0 .. m0 + NV - 1 of weight row n (acc) to the output.  All lanes of a warp call it with consecutive rows and
// the same tokens.  SWIGLU: rows 2i / 2i + 1 are gate and up of one output; the lane pair exchanges one value per two
// tokens, then the even lane finishes the first token and the odd lane the second.
template <int MODE, int NV>
__device__ __forceinline__ void stream_store(const StreamArgs& a, int t, int n, bool row_ok, int m0, const float (&acc)[NV], const __half (&res)[NV]) {
    const size_t ld = static_cast<size_t>(a.out_ld[t]);
    if constexpr (MODE == kSwiglu) {
        const int odd = n & 1;
        __half* out = a.out[t] + static_cast<size_t>(m0 + odd) * ld + (n >> 1);
#pragma unroll
        for (int q = 0; q < NV; q += 2) {
            const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? acc[q] : acc[q + 1], 1);
            // (the operands are chosen, not the result: a choice between two calls ran both, gate_up at 47 / 115 tokens 6.8 -> 6.1 / 9.9 -> 8.5 us)
            const float y = swiglu_f32(odd ? other : acc[q], odd ? acc[q + 1] : other);
            if (row_ok && m0 + q + odd < a.M) *out = __float2half_rn(y);
            out += 2 * ld;
        }
    } else {
        __half* out = a.out[t] + static_cast<size_t>(m0) * ld + n;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            if (row_ok && m0 + q < a.M) {
                __half y = __float2half_rn(acc[q]);
                if constexpr (MODE == kPlain) {
                    if (a.residual != nullptr) y = __hadd(y, res[q]);
                }
                *out = y;
                if constexpr (MODE == kPlain) {
                    for (int p = 0; p < a.num_peers; ++p) a.peer_out[p][static_cast<size_t>(m0 + q) * ld + n] = y;
                }
            }
            out += ld;
        }
    }
}
template <int MODE, int NV>
__device__ __forceinline__ void stream_load_residual(const StreamArgs& a, int t, int n, bool row_ok, int m0, __half (&res)[NV]) {
#pragma unroll
    for (int q = 0; q < NV; ++q) res[q] = __half(0.0f);
    if constexpr (MODE == kPlain) {
        if (a.residual != nullptr) {
#pragma unroll
            for (int q = 0; q < NV; ++q)
                if (row_ok && m0 + q < a.M) res[q] = a.residual[static_cast<size_t>(m0 + q) * a.out_ld[t] + n];
        }
    }
}

// All lanes look at the barrier; only if it is still open one lane polls for the warp.
__device__ __forceinline__ bool group_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int lane) {
    if (__all_sync(0xFFFFFFFFu, mbar_test_wait(bar, parity))) return true;
    return warp_wait(bar, parity, abort_flag, lane);
}

template <int MODE>
__global__ void __launch_bounds__(kStThreads, 1) gemm_w4a16_tc_stream_kernel(const __grid_constant__ StreamArgs a) {
    extern __shared__ uint8_t smem_raw_base[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw_base) + 1023) & ~uintptr_t(1023));
    const int T = a.p.T, NS = a.p.slots, NA = a.p.a_slots, SR = a.p.raw_slots, K = a.K;
    const int x_box = T * 128, x_bytes = 2 * x_box;      // a step's tokens: two boxes of 64 k
    uint8_t* s_x = smem;
    uint8_t* s_raw = s_x + a.p.x_mem * x_bytes;
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(s_raw + SR * kStRawBytes);
    const uint32_t bar0 = smem_u32(s_bar);
    auto raw_full = [&](int i) { return bar0 + 8u * i; };
    auto raw_empty = [&](int i) { return bar0 + 8u * (kStMaxRaw + i); };
    auto full = [&](int i) { return bar0 + 8u * (2 * kStMaxRaw + i); };          // weights dequantised and tokens landed
    auto empty = [&](int i) { return bar0 + 8u * (2 * kStMaxRaw + kStMaxSlots + i); };
    constexpr int kBars = 2 * kStMaxRaw + 2 * kStMaxSlots + 2;
    const uint32_t accum_full = bar0 + 8u * (kBars - 2), part_full = bar0 + 8u * (kBars - 1);
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(s_bar + kBars);
    volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
    int* s_issued = reinterpret_cast<int*>(s_tmem + 2);          // steps whose weights were asked for

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int t = 0, tile = blockIdx.x;
    if constexpr (MODE == kQkv) {
        if (tile >= a.tiles[0]) { tile -= a.tiles[0]; t = 1; }
        if (t == 1 && tile >= a.tiles[1]) { tile -= a.tiles[1]; t = 2; }
    }
    const int n0 = tile * kTileRows, rows_t = a.rows[t], m0 = blockIdx.y * T;
    // K range: whole steps, spread over the cluster as evenly as they go
    const int ksplit = a.p.ksplit, krank = static_cast<int>(blockIdx.z);
    const int G = K / kGroup, per = a.p.steps_each, rest = G - per * ksplit;
    const int st0 = krank * per + min(krank, rest), nst = per + (krank < rest ? 1 : 0);

    const int r = (warp & 3) * 32 + lane, group = warp >> 2;      // dequantising warps: weight row = TMEM lane, first step
    // Scales of this thread's next two steps, straight into registers: the first loads, since behind the weight stream they would arrive
    // last.  (Through shared memory they cost a division per value, a block barrier and 0.4 us of a launch's start.)
    const bool row_ok = n0 + r < rows_t;
    const unsigned short* scale_row = reinterpret_cast<const unsigned short*>(a.scales[t]) + (row_ok ? static_cast<size_t>(n0 + r) * G + st0 : 0);
    auto load_scale = [&](int s) -> unsigned short {
        unsigned short v = 0;
        if (row_ok && s < nst) v = __ldg(scale_row + s);
        return v;
    };
    unsigned short sc_a = 0, sc_b = 0;
    if (warp < kStDqWarps) {
        sc_a = load_scale(group);
        sc_b = load_scale(group + kStGroups);
    } else if (warp == kStWeightWarp) {
        // barriers (three a lane, without a branch), then the ring of packed weights
#pragma unroll
        for (int i = lane; i < (kBars + 31) / 32 * 32; i += 32) {
            const int count = i < kStMaxRaw ? 1 : i < 2 * kStMaxRaw ? 4 : i < 2 * kStMaxRaw + kStMaxSlots ? 4 + 1 : i == kBars - 2 ? kStIssuers : 1;
            if (i < kBars) mbar_init(bar0 + 8u * i, count);
        }
        if (lane == (kBars - 1) % 32) {
            const int mine = max(0, min(a.p.tpr, T - krank * a.p.tpr));
            if (ksplit > 1) mbar_arrive_expect_tx(part_full, static_cast<uint32_t>(ksplit * mine * kTileRows * 4));
            *s_abort = 0;
            *s_issued = min(SR, nst);
        }
        fence_barrier_init();
        fence_proxy_async_smem();
        __syncwarp();
        // (only announced: this warp goes on to the weights)
        asm volatile("bar.arrive 2, %0;" ::"n"(kStThreads) : "memory");
        if (elect_one()) {
            const int first = min(SR, nst);
#pragma unroll 1
            for (int i = 0; i < first; ++i) {
                mbar_arrive_expect_tx(raw_full(i), kStRawBytes);
                tma_load_2d(smem_u32(s_raw + i * kStRawBytes), &a.tmap_w[t], (st0 + i) * 64, n0, raw_full(i));
            }
        }
        __syncwarp();
    } else if (warp == kStTokenWarp) {
        if (elect_one()) tma_prefetch_desc(&a.tmap_x);
    } else if (warp == kStTokenWarp + 1) {
        if (elect_one()) tma_prefetch_desc(&a.tmap_w[t]);
    } else {
        // Blocks while a CTA of the previous launch on this SM holds it; the next launch may only follow once every CTA of
        // this one has its share, or a CTA of the next could take it first and wait for this launch with it.
        tmem_alloc(smem_u32(s_tmem), 512);
        tmem_relinquish();
        pdl_release_dependents();
    }
    tc_fence_before();
    if (warp != kStWeightWarp) asm volatile("bar.sync 2, %0;" ::"n"(kStThreads) : "memory");
    tc_fence_after();
    const bool own_part = a.p.part_offset != 0;      // partials in memory of their own: they may come while the rings are in use
    // (one warp has something to publish, the barriers; a release here would make the others wait for their scales: 0.7 us)
    if (ksplit > 1 && own_part) {
        if (warp == kStWeightWarp) cluster_arrive();
        else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    }

    if (warp < kStDqWarps) {
        const uint32_t tmem_base = *s_tmem;
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const int swz = (r >> 1) & 3;            // 64-byte swizzle: 16-byte chunk index xor row pair
        const uint8_t* raw_lane = s_raw + r * 64;
        bool ok = true;
        int rs = group;                          // ring slot of this group's next step
        uint32_t rph = 0;
        int slot = group, aslot = group;         // the step's barrier and its A slot
        int wslot = group + NS - NA;             // barrier of the step that had the A slot before, and the parity it completes
        uint32_t eph = 1;
        if (rs >= SR) { rs -= SR; rph ^= 1; }    // (SR is a multiple of 4: never for the first step)
        for (int s = group; s < nst; s += kStGroups) {
            const __half sc1 = __ushort_as_half(sc_a);
            sc_a = sc_b;
            sc_b = load_scale(s + 2 * kStGroups);
            ok = group_wait(raw_full(rs), rph, s_abort, lane);
            if (!ok) break;
            const uint8_t* raw_row = raw_lane + rs * kStRawBytes;
            // A quarter of the step (16 columns) is in registers as fp16 before the slot is free; the rest is stored as it comes.  With
            // the whole step in registers first one layer takes 19.5 / 20.8 / 23.0 / 30.0 us at 9 / 17 / 47 / 115 tokens, with none of it
            // 18.9 / 20.2 / 22.3 / 30.4, so 19.0 / 20.3 / 22.3 / 30.2.
            const __half2 sc2 = __half2half2(sc1), k10 = __float2half2_rn(1024.0f);
            const __half2 s20 = __hmul2(__hmul2(sc2, k10), k10), m8s = __hmul2(sc2, __float2half2_rn(-8.0f));
            const uint32_t a_lane = lane_base + static_cast<uint32_t>(a.p.a_col + aslot * kStACols);
            auto slot_free = [&]() -> bool {
                ok = group_wait(empty(wslot), eph, s_abort, lane);
                tc_fence_after();
                return ok;
            };
            if (__all_sync(0xFFFFFFFFu, __habs(sc1) < __float2half_rn(0.0624f))) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 w = *reinterpret_cast<const uint4*>(raw_row + ((c ^ swz) << 4));
                    uint32_t o[16];
                    dequant_word_small_scale(w.x, s20, m8s, o);
                    dequant_word_small_scale(w.y, s20, m8s, o + 4);
                    dequant_word_small_scale(w.z, s20, m8s, o + 8);
                    dequant_word_small_scale(w.w, s20, m8s, o + 12);
                    if (c == 0 && !slot_free()) break;
                    tmem_st16(a_lane + 16u * c, o);
                }
            } else if (slot_free()) {
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    const uint4 w = *reinterpret_cast<const uint4*>(raw_row + ((c ^ swz) << 4));
                    uint32_t o[16];
                    dequant_word_fp16(w.x, sc2, reinterpret_cast<__half2(&)[4]>(o[0]));
                    dequant_word_fp16(w.y, sc2, reinterpret_cast<__half2(&)[4]>(o[4]));
                    dequant_word_fp16(w.z, sc2, reinterpret_cast<__half2(&)[4]>(o[8]));
                    dequant_word_fp16(w.w, sc2, reinterpret_cast<__half2(&)[4]>(o[12]));
                    tmem_st16(a_lane + 16u * c, o);
                }
            }
            if (!ok) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(raw_empty(rs));
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(full(slot));
            rs += kStGroups;
            if (rs >= SR) { rs -= SR; rph ^= 1; }
            slot += kStGroups;
            if (slot >= NS) slot -= NS;
            aslot += kStGroups;
            if (aslot >= NA) aslot -= NA;
            wslot += kStGroups;
            if (wslot >= NS) { wslot -= NS; eph ^= 1; }
        }
        // ---------------- epilogue: thread = weight row, registers = tokens ----------------
        pdl_wait_prior_grids();                  // the previous kernels' reads of the outputs and writes of the residual
        const int n = n0 + r;
        if (ksplit == 1) {
            // eight tokens a round (a loop, not unrolled: this code runs once and its instructions have to be fetched)
            __half res[8];
            stream_load_residual<MODE>(a, t, n, row_ok, m0 + group * 8, res);
            if (ok) ok = warp_wait(accum_full, 0, s_abort, lane);
            tc_fence_after();
            if (ok) {
#pragma unroll 1
                for (int c0 = group * 8; c0 < T; c0 += 8 * kStGroups) {
                    float acc[8];
                    stream_load_acc(lane_base + static_cast<uint32_t>(c0), a.p.acc2_col, acc);
                    stream_store<MODE>(a, t, n, row_ok, m0 + c0, acc, res);
                    if (c0 + 8 * kStGroups < T) stream_load_residual<MODE>(a, t, n, row_ok, m0 + c0 + 8 * kStGroups, res);
                }
            }
        } else {
            // Tokens [rank * tpr, (rank + 1) * tpr) are finished by that rank; partials land at [source][token / 4][row][4].
            // They are sent whatever the waits returned: a peer that waits for them must not be left alone.
            const int tpr = a.p.tpr;
            uint8_t* s_part = smem + a.p.part_offset;
            __half res[4];
            stream_load_residual<MODE>(a, t, n, row_ok && group * 4 < tpr, m0 + krank * tpr + group * 4, res);
            if (ok) ok = warp_wait(accum_full, 0, s_abort, lane);
            tc_fence_after();
            if (!own_part) cluster_arrive();     // this CTA's rings are free
            cluster_wait();
            const uint32_t part0 = smem_u32(s_part) + static_cast<uint32_t>(krank * (tpr / 4) * kTileRows + r) * 16u;
#pragma unroll 1
            for (int c0 = group * 8; c0 < T; c0 += 8 * kStGroups) {
                float v[8];
                stream_load_acc(lane_base + static_cast<uint32_t>(c0), a.p.acc2_col, v);
#pragma unroll
                for (int q = 0; q < 8; q += 4) {
                    const int owner = (c0 + q) / tpr, k = c0 + q - owner * tpr;
                    st_async_16(cluster_map_shared(part0 + static_cast<uint32_t>((k >> 2) * kTileRows) * 16u, static_cast<uint32_t>(owner)),
                                cluster_map_shared(part_full, static_cast<uint32_t>(owner)), __float_as_uint(v[q]), __float_as_uint(v[q + 1]),
                                __float_as_uint(v[q + 2]), __float_as_uint(v[q + 3]));
                }
            }
            bool have = false;
            if (lane == 0)
                for (unsigned it = 0; it < 4 * kWaitLimit && !have; ++it) have = mbar_try_wait_cluster(part_full, 0);
            __syncwarp();                        // the peers' stores before the reads of all lanes: a shuffle orders no memory
            have = __shfl_sync(0xFFFFFFFFu, have ? 1 : 0, 0) != 0;
            if (!have && lane == 0) { *s_abort = 1; atomicAdd(&g_tc_wait_timeouts, 1u); }
            if (have) {
#pragma unroll 1
                for (int k = group * 4; k < tpr; k += 4 * kStGroups) {
                    const int m = krank * tpr + k;
                    if (m >= T) break;
                    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int s = 0; s < kStMaxSplit; ++s) {
                        if (s < ksplit) {
                            const float4 p = *reinterpret_cast<const float4*>(s_part + static_cast<size_t>((s * (tpr / 4) + (k >> 2)) * kTileRows + r) * 16);
                            acc[0] += p.x; acc[1] += p.y; acc[2] += p.z; acc[3] += p.w;
                        }
                    }
                    stream_store<MODE>(a, t, n, row_ok, m0 + m, acc, res);
                    if (k + 4 * kStGroups < tpr) stream_load_residual<MODE>(a, t, n, row_ok, m0 + m + 4 * kStGroups, res);
                }
            }
        }
    } else {
        if (warp != kStWeightWarp && warp != kStTokenWarp) {
            // ---------------- MMA issue: one thread, or one each for the even and the odd steps ----------------
            const uint32_t tmem_base = *s_tmem;
            if (elect_one()) {
                const int first = warp == kStDqWarps ? 0 : 1;
                const uint32_t idesc = make_idesc(T);
                const uint64_t b_desc0 = make_smem_desc(smem_u32(s_x));
                const uint32_t b_step = static_cast<uint32_t>(x_bytes) >> 4, b_half = static_cast<uint32_t>(x_box) >> 4;
                int slot = first, aslot = first;
                uint32_t ph = 0;
                bool ready = mbar_test_wait(full(slot), 0);
                for (int s = first; s < nst; s += kStIssuers) {
                    if (!ready && !mbar_wait(full(slot), ph, s_abort)) break;
                    tc_fence_after();
                    const uint32_t bar_empty = empty(slot);
                    const uint64_t b0 = b_desc0 + static_cast<uint32_t>(slot) * b_step;
                    const uint32_t a0 = tmem_base + static_cast<uint32_t>(a.p.a_col + aslot * kStACols);
                    aslot += kStIssuers;
                    if (aslot >= NA) aslot -= NA;
                    slot += kStIssuers;
                    if (slot >= NS) { slot -= NS; ph ^= 1; }
                    ready = mbar_test_wait(full(slot), ph);      // the answer arrives while the MMAs below are issued
                    const uint32_t tmem_d = tmem_base + ((s & 1) != 0 ? static_cast<uint32_t>(a.p.acc2_col) : 0u);
#pragma unroll
                    for (int ks = 0; ks < kGroup / 16; ++ks)
                        tc_mma_f16_ts(tmem_d, a0 + 8u * ks, b0 + (ks >= 4 ? b_half : 0u) + static_cast<uint32_t>(2 * (ks & 3)), idesc,
                                      (ks != 0 || s >= 2) ? 1u : 0u);
                    tc_commit(bar_empty);
                }
                tc_commit(accum_full);   // also after a wait that ran out: nothing may be in flight at the end
            }
        } else if (warp == kStWeightWarp) {
            // ---------------- packed weights, as the ring empties ----------------
            if (elect_one()) {
                int i = min(SR, nst), slot = 0;
                uint32_t ph = 0;
#pragma unroll 1
                for (; i < nst; ++i) {
                    if (!mbar_wait(raw_empty(slot), ph, s_abort)) break;
                    mbar_arrive_expect_tx(raw_full(slot), kStRawBytes);
                    tma_load_2d(smem_u32(s_raw + slot * kStRawBytes), &a.tmap_w[t], (st0 + i) * 64, n0, raw_full(slot));
                    if (++slot == SR) { slot = 0; ph ^= 1; }
                }
                *s_issued = i;
            }
        } else if (elect_one()) {
            // ---------------- tokens, as soon as the previous kernel is through ----------------
            int i = 0, slot = 0;
            uint32_t ph = 1;
            pdl_wait_prior_grids();
#pragma unroll 1
            for (; i < nst; ++i) {
                if (i >= NS && !mbar_wait(empty(slot), ph, s_abort)) break;
                const uint32_t dst = smem_u32(s_x + slot * x_bytes), bar = full(slot);
                mbar_arrive_expect_tx(bar, static_cast<uint32_t>(x_bytes));
                tma_load_2d(dst, &a.tmap_x, (st0 + i) * kGroup, m0, bar);
                tma_load_2d(dst + x_box, &a.tmap_x, (st0 + i) * kGroup + kBK, m0, bar);
                if (++slot == NS) { slot = 0; ph ^= 1; }
            }
        }
        __syncwarp();
        if (ksplit > 1) {
            if (!own_part) cluster_arrive();
            cluster_wait();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*s_abort) {          // a bounded wait ran out: what is in flight has to land before the memory goes (bounded too)
        if (tid == 0) {
            for (int i = 0; i < min(SR, *s_issued); ++i) wait_regardless(raw_full(i), static_cast<uint32_t>((*s_issued - 1 - i) / SR) & 1u, kWaitLimit);
            wait_regardless(accum_full, 0, kWaitLimit);
            __nanosleep(100000);     // token copies whose slot never filled up have no barrier phase of their own to wait for
        }
        __syncthreads();
    }
    if (warp == kStDqWarps) tmem_dealloc(*s_tmem, 512);
}

// ---- host side of the streaming form ----
// Ring sizes for token tiles of T and the `all_steps` steps of K split `ksplit` ways.  False where it does not fit.
bool plan_stream(int T, int ksplit, int all_steps, StreamPlan* a) {
    const int steps = (all_steps + ksplit - 1) / ksplit;
    a->T = T;
    a->ksplit = ksplit;
    a->steps_each = all_steps / ksplit;
    a->acc2_col = T <= 64 ? 64 : 128;
    a->a_col = 2 * a->acc2_col;
    a->a_slots = T <= 64 ? 6 : 4;
    a->tpr = ((T + a->ksplit - 1) / a->ksplit + 3) & ~3;
    const size_t part_bytes = a->ksplit > 1 ? static_cast<size_t>(a->ksplit) * a->tpr * kTileRows * 4 : 0;
    const size_t budget = 226 * 1024;
    const size_t fixed = 1024 + (2 * kStMaxRaw + 2 * kStMaxSlots + 2) * 8 + 16;
    // As many token slots as fit beside a whole ring of weights: every slot that does not have to be waited for is asked for at once.
    const int all_raw = std::min(kStMaxRaw, (steps + kStGroups - 1) / kStGroups * kStGroups);
    a->slots = std::max(a->a_slots, std::min(kStMaxSlots, (steps + 1) & ~1));
    while (a->slots > a->a_slots && fixed + part_bytes + 128 + static_cast<size_t>(a->slots) * T * 256 + static_cast<size_t>(all_raw) * kStRawBytes > budget) a->slots -= 2;
    for (; a->slots >= kStGroups; a->slots -= 2) {
        a->a_slots = std::min(a->a_slots, a->slots);
        a->x_mem = std::min(a->slots, steps);
        const size_t x_bytes = static_cast<size_t>(a->x_mem) * T * 256;
        for (int own = part_bytes ? 1 : 0; own >= 0; --own) {
            const size_t extra = own ? part_bytes + 128 : 0;
            int raw = all_raw;
            while (raw > kStGroups && fixed + extra + x_bytes + static_cast<size_t>(raw) * kStRawBytes > budget) raw -= kStGroups;
            const size_t ring = x_bytes + static_cast<size_t>(raw) * kStRawBytes;
            if (fixed + extra + ring > budget) continue;
            if (!own && ring < part_bytes) continue;     // the partials go on top of the rings
            a->raw_slots = raw;
            const size_t used = (fixed - 1024 + ring + 127) / 128 * 128;
            a->part_offset = own ? static_cast<int>(used) : 0;
            // At least half an SM, so that no SM ever holds two of these CTAs: each takes all columns of tensor memory, and the
            // second would sit in its allocation.  (Today the registers rule that out already.)
            a->smem = std::max<size_t>(1024 + used + (own ? part_bytes : 0), 116 * 1024);
            return true;
        }
    }
    return false;
}
