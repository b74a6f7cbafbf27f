// Prefill W4A16 contraction on CTA pairs (tcgen05.mma.cta_group::2).  Included by gemm_tc.cu behind the PTX wrappers.
//
// Two CTAs of a cluster -- two SMs -- share a tile of 256 weight rows x T tokens: each dequantises ITS 128 weight rows
// (the A operand, M = 256 split over the pair) into its tensor memory and loads ITS T / 2 tokens (half of the B operand)
// into its shared memory; one thread of the leading CTA issues the MMAs, which accumulate into both CTAs' tensor memory.
// A does not pass through shared memory: with it there the operand reads alone exceed what shared memory delivers beside
// the loads (measured on a one-CTA form: 0.57 of the bf16 peak).  Steps are 128 k, one quantisation group.
//
// What bounds it: the tensor pipe on long K (28672 x 8192), the work around a tile on short K (K = 1536 gives 12 steps per
// tile).  So the epilogue has warps of its own, and tensor memory holds two accumulators of up to 128 token columns: a tile
// of up to 128 tokens uses one of them in turn with the next tile's, a larger one both as its two halves.  The epilogue
// takes a half into registers (SWIGLU: the second one into shared memory) and gives it back at once, and the MMAs of the next
// tile's first half run ahead meanwhile.
// The rest of tensor memory are four A slots of one step.  Arrivals on the leader's barriers carry no cluster-scope release:
// with one the peer's dequantising warps waited for their own prefetched loads at every step (1400 cycles a step, 930 of
// them for nothing).
//
//   warps 0..7  : dequantise; group g = warp / 4 takes the steps g, g + 2, ...  A quarter of a step is in registers as fp16
//                 before its slot is free, the rest is stored as it comes.  (The whole step in registers took 88 of them, by
//                 setmaxnreg, and spilled; with 72 for every warp and no spills gate_up at 300 / 1024 / 4096 tokens
//                 23.8 -> 22.4, 48.2 -> 47.1, 184 -> 179 us, 8192 x 8192 at 1024 104 -> 102.)
//   warps 8..23 : epilogue, 128 rows of a finished accumulator (four warps per 32 rows, a quarter of the tokens each)
//   warp 24     : tensor memory; in the leading CTA one thread issues the MMAs
//   warp 25     : TMA of the packed weights, 128 rows x 128 k per slot (private ring, before the wait for the previous kernel)
//   warp 26     : TMA of this CTA's half of the token tile, T / 2 x 128 k per slot
//
// Synchronisation: one "full" barrier per slot in the leader counts the dequantising warps of both CTAs and the bytes
// of both token halves; one "done" barrier per slot in both CTAs (tcgen05.commit with a CTA mask) frees the A slot and
// the token slot.  Two "accumulator full" barriers in both CTAs, two "accumulator empty" ones in the leader.
constexpr int kPairGroups = 2;
constexpr int kPairDqWarps = 4 * kPairGroups, kPairEpiWarps = 16;
constexpr int kPairThreads = (kPairDqWarps + kPairEpiWarps + 3) * 32;
constexpr int kPairAccCols = 128;            // one accumulator
constexpr int kPairACol = 2 * kPairAccCols, kPairACols = kGroup / 2;   // A slots behind the two accumulators
constexpr int kPairSlots = 4;                // A and token slots; a multiple of the groups (parity waits)
constexpr int kPairMaxRaw = 8;               // packed weights; likewise
constexpr int kPairRawBytes = kTileRows * 64;
constexpr int kPairParkBytes = kPairEpiWarps * 32 * (kPairAccCols / 4) * 4;    // an accumulator in shared memory
// SWIGLU parks the second accumulator of a tile (see the epilogue); its 64 KB are taken from the ring of packed weights.
constexpr bool pair_parks(int mode) { return mode == kSwiglu; }
constexpr int pair_raw_slots(int mode) { return pair_parks(mode) ? 4 : kPairMaxRaw; }

struct PairArgs {
    CUtensorMap tmap_w[3];
    CUtensorMap tmap_x;
    const __half* scales[3];
    __half* out[3];
    int rows[3];
    int out_ld[3];
    int tiles[3];
    const __half* residual;
    int M, K;
    int halves, n_half;      // accumulators of a tile and tokens of each: T = halves * n_half
    int panel;               // token tiles per panel of the tile order
    __half* peer_out[7];     // PLAIN: the output block's place in other GPUs' matrices
    int num_peers;
};

__device__ __forceinline__ uint32_t cluster_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Arrival on a barrier of the other CTA.  What it announces lies in tensor memory, ordered by the tcgen05 fences and waits
// on both sides.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(leader_bar)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// arrives on the barrier at this shared-memory offset in both CTAs of the pair once the MMAs issued so far are done
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
// Instruction descriptor of the pair: D fp32, A/B fp16, both K-major, M = 256 (128 rows per CTA), N = n.
__device__ __forceinline__ uint32_t make_idesc_pair(int n) {
    return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24);
}
// D[tmem] (+)= A[tmem] * B[smem]^T over the CTA pair.
__device__ __forceinline__ void tc_mma_f16_pair_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                                   uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Which 128-row tile of which tensor, and which tokens, a pair tile index stands for (this CTA's half).
struct PairTile {
    int t, n0, m0;
};
__device__ __forceinline__ PairTile pair_tile(const PairArgs& a, int pt, int n_pairs, int rank, bool qkv) {
    PairTile r;
    // Tile order: panels of a.panel token tiles; inside a panel the token tile runs fastest.  With a panel of 4 the
    // tiles in flight at one time (one per CTA pair) cover 4 token tiles x about 18 row-tile pairs, and both the
    // token slabs and the packed weight rows are re-used out of L2; a panel of 1 (row tiles fastest) shares one
    // token slab among all tiles in flight but streams the whole weight matrix once per token tile, which is
    // right only while the matrix stays in L2 (the host picks).
    const int T = a.halves * a.n_half;
    const int m_tiles = (a.M + T - 1) / T;
    const int per_panel = a.panel * n_pairs;
    const int panel = pt / per_panel;
    const int q = pt - panel * per_panel;
    const int w = min(a.panel, m_tiles - panel * a.panel);
    const int m_idx = panel * a.panel + q % w;
    int tile = 2 * (q / w) + rank;      // consecutive 128-row tiles form a pair; an odd last one is paired with rows past the end
    r.t = 0;
    if (qkv) {
        if (tile >= a.tiles[0]) { tile -= a.tiles[0]; r.t = 1; }
        if (r.t == 1 && tile >= a.tiles[1]) { tile -= a.tiles[1]; r.t = 2; }
    }
    r.n0 = tile * kTileRows;
    r.m0 = m_idx * T;
    return r;
}

// Eight tokens of a weight row.  All lanes of a warp call it with consecutive rows and the same tokens.  The even lane of a
// pair finishes the first token of two, the odd lane the second: SWIGLU has its gate in the even and its up in the odd row,
// the others hold both rows of a token.  `take(q, even_row, odd_row)` gets token pair q.
template <typename F>
__device__ __forceinline__ void pair_exchange8(int odd, const uint32_t (&v)[8], F&& take) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float a = __uint_as_float(v[2 * q]), b = __uint_as_float(v[2 * q + 1]);
        const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? a : b, 1);
        take(q, odd ? other : a, odd ? b : other);
    }
}

// STORE (the host picks): kStoreWords where both rows of an output lie in one aligned word, kStoreWordsPeers the same with
// copies to peer GPUs (a warp's store is two runs of 64 bytes, which travel as such), kStoreValues value by value.
enum PairStore { kStoreValues = 0, kStoreWords = 1, kStoreWordsPeers = 2 };
template <int MODE, int STORE>
__global__ void __launch_bounds__(kPairThreads, 1) gemm_w4a16_tc_pair_kernel(const __grid_constant__ PairArgs a) {
    constexpr bool WORDS = STORE != kStoreValues, PARK = pair_parks(MODE);
    constexpr int kRawSlots = pair_raw_slots(MODE);
    constexpr int kEpi0 = kPairDqWarps, kMmaWarp = kEpi0 + kPairEpiWarps, kRawWarp = kMmaWarp + 1;
    extern __shared__ uint8_t smem_raw_base[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw_base) + 1023) & ~uintptr_t(1023));
    const int H = a.halves, NH = a.n_half, T = H * NH, K = a.K, G = K / kGroup;
    const int b_box = (NH / 2) * 128, b_bytes = 2 * H * b_box;      // [accumulator][64 k]: half of each accumulator's tokens
    uint8_t* s_b = smem;
    uint8_t* s_raw = s_b + kPairSlots * b_bytes;
    uint8_t* s_park = s_raw + kRawSlots * kPairRawBytes;
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(s_park + (PARK && H == 2 ? kPairParkBytes : 0));
    const uint32_t bar0 = smem_u32(s_bar);
    auto raw_full = [&](int i) { return bar0 + 8u * i; };
    auto raw_empty = [&](int i) { return bar0 + 8u * (kPairMaxRaw + i); };
    auto full = [&](int i) { return bar0 + 8u * (2 * kPairMaxRaw + i); };
    auto done = [&](int i) { return bar0 + 8u * (2 * kPairMaxRaw + kPairSlots + i); };
    auto acc_full = [&](int i) { return bar0 + 8u * (2 * kPairMaxRaw + 2 * kPairSlots + i); };
    auto acc_empty = [&](int i) { return bar0 + 8u * (2 * kPairMaxRaw + 2 * kPairSlots + 2 + i); };
    constexpr int kBars = 2 * kPairMaxRaw + 2 * kPairSlots + 4;
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(s_bar + kBars);
    volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
    volatile int* s_epi_ok = reinterpret_cast<volatile int*>(s_tmem + 2);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = static_cast<int>(cluster_cta_rank());
    const bool leader = rank == 0;
    const int pair_id = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    const int n_pairs = (a.tiles[0] + a.tiles[1] + a.tiles[2] + 1) / 2;
    const int total_pt = n_pairs * ((a.M + T - 1) / T);

    if (warp == kRawWarp) {
        if (lane < kPairMaxRaw) { mbar_init(raw_full(lane), 1); mbar_init(raw_empty(lane), 4); }
        // full: four dequantising warps of each CTA and the leader's expect_tx arrival
        if (lane < kPairSlots) { mbar_init(full(lane), 2 * 4 + 1); mbar_init(done(lane), 1); }
        if (lane < 2) { mbar_init(acc_full(lane), 1); mbar_init(acc_empty(lane), 2 * kPairEpiWarps); }
        if (lane == 0) { *s_abort = 0; tma_prefetch_desc(&a.tmap_x); tma_prefetch_desc(&a.tmap_w[0]); }
        fence_barrier_init();
        fence_proxy_async_smem();
        __syncwarp();
    }
    if (warp == kMmaWarp) {          // the same warp in both CTAs, the same shared-memory offset for the result
        tmem_alloc_pair(smem_u32(s_tmem), 512);
        tmem_relinquish_pair();
        pdl_release_dependents();    // not before: a CTA of the next launch must not take this one's tensor memory
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();              // the peer's barriers exist before anything arrives on them from here
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem;

    if (warp < kPairDqWarps) {
        // ================= dequantise: thread = weight row = tensor-memory lane =================
        const int r = (warp & 3) * 32 + lane, g = warp >> 2;
        const int swz = (r >> 1) & 3;            // 64-byte swizzle: 16-byte chunk index xor row pair
        const uint32_t a_lane = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(kPairACol);
        const uint32_t leader_full0 = cluster_map_shared(full(0), 0);
        bool ok = true;
        // The walk over (tile, step) pairs is one sequence: a group's next step after a tile's last one lies in the next tile.
        const int my_tiles = pair_id < total_pt ? (total_pt - pair_id + num_pairs - 1) / num_pairs : 0;
        const int total = my_tiles * G;
        int rs = g, slot = g;                    // ring positions of this group's next step
        uint32_t rph = 0, dph = 1;               // parities: raw slot filled; slot freed by its previous use
        int it = 0, st = g;                      // tile iteration and step in it
        const __half* sc_row = nullptr;          // scales of this thread's row; null past the tensor
        auto row_of = [&](int iteration) {
            const PairTile pt = pair_tile(a, pair_id + iteration * num_pairs, n_pairs, rank, MODE == kQkv);
            const int row = pt.n0 + r;
            sc_row = row < a.rows[pt.t] ? a.scales[pt.t] + static_cast<size_t>(row) * G : nullptr;
        };
        auto settle = [&]() {                    // (it, st) back into range after st moved on
            while (st >= G) {
                st -= G;
                if (++it < my_tiles) row_of(it);
            }
        };
        if (my_tiles > 0) row_of(0);
        settle();
        auto load_scale = [&]() -> __half { return sc_row != nullptr ? __ldg(sc_row + st) : __half(0.0f); };
        __half sc_next = g < total ? load_scale() : __half(0.0f);
        for (int i = g; i < total; i += kPairGroups) {
            const __half sc = sc_next;
            st += kPairGroups;
            settle();
            if (i + kPairGroups < total) sc_next = load_scale();     // the next step's, one visit ahead
            ok = group_wait(raw_full(rs), rph, s_abort, lane);
            if (!ok) break;
            const uint8_t* raw_row = s_raw + rs * kPairRawBytes + r * 64;
            const __half2 sc2 = __half2half2(sc), k10 = __float2half2_rn(1024.0f);
            const __half2 s20 = __hmul2(__hmul2(sc2, k10), k10), m8s = __hmul2(sc2, __float2half2_rn(-8.0f));
            const uint32_t a_slot = a_lane + static_cast<uint32_t>(slot * kPairACols);
            auto slot_free = [&]() -> bool {
                ok = group_wait(done(slot), dph, s_abort, lane);
                tc_fence_after();
                return ok;
            };
            if (__all_sync(0xFFFFFFFFu, __habs(sc) < __float2half_rn(0.0624f))) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 w = *reinterpret_cast<const uint4*>(raw_row + ((c ^ swz) << 4));
                    uint32_t o[16];
                    dequant_word_small_scale(w.x, s20, m8s, o);
                    dequant_word_small_scale(w.y, s20, m8s, o + 4);
                    dequant_word_small_scale(w.z, s20, m8s, o + 8);
                    dequant_word_small_scale(w.w, s20, m8s, o + 12);
                    if (c == 0 && !slot_free()) break;
                    tmem_st16(a_slot + 16u * c, o);
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
                    tmem_st16(a_slot + 16u * c, o);
                }
            }
            if (!ok) break;
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(raw_empty(rs));
                if (leader) mbar_arrive(full(slot));
                else mbar_arrive_remote(leader_full0 + 8u * slot);
            }
            rs += kPairGroups;
            if (rs >= kRawSlots) { rs -= kRawSlots; rph ^= 1; }
            slot += kPairGroups;
            if (slot >= kPairSlots) { slot -= kPairSlots; dph ^= 1; }
        }
    } else if (warp < kMmaWarp) {
        // ================= epilogue: thread = weight row, registers = tokens =================
        const int part = (warp - kEpi0) >> 2, r = (warp & 3) * 32 + lane, odd = lane & 1;
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(8 * part);
        const uint32_t leader_empty0 = cluster_map_shared(acc_empty(0), 0);
        constexpr int kMaxGroups = kPairAccCols / 32;          // this warp's groups of eight tokens: part, part + 4, ...
        const int n_groups = (NH / 8 - part + 3) / 4;
        const bool add = MODE == kPlain && a.residual != nullptr;
        bool ok = true;
        int buf = 0;
        uint32_t ph = 0;
        pdl_wait_prior_grids();                  // the previous kernels' reads of the outputs and writes of the residual
        for (int pt_i = pair_id; pt_i < total_pt && ok; pt_i += num_pairs) {
            const PairTile pt = pair_tile(a, pt_i, n_pairs, rank, MODE == kQkv);
            const int ne = (pt.n0 + r) & ~1, rows = a.rows[pt.t];
            const size_t ld = static_cast<size_t>(a.out_ld[pt.t]);
            // One warp polls, the others wait at a block barrier: sixteen polling warps slow the dequantising ones down.
            // Its answer goes through one word per buffer, rewritten only after everybody has read it.
            auto wait_full = [&]() -> bool {
                if (warp == kEpi0) {
                    ok = group_wait(acc_full(buf), ph, s_abort, lane);
                    if (lane == 0) s_epi_ok[buf] = ok ? 1 : 0;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(kPairEpiWarps * 32) : "memory");
                ok = s_epi_ok[buf] != 0;
                if (ok) tc_fence_after();
                return ok;
            };
            auto give_back = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (leader) mbar_arrive(acc_empty(buf));
                    else mbar_arrive_remote(leader_empty0 + 8u * buf);
                }
                buf ^= 1;
                if (buf == 0) ph ^= 1;
            };
            // This warp's columns of an accumulator into registers, then it goes back: the next tile's MMAs need it.
            uint32_t v[kMaxGroups][8];
            auto take = [&]() -> bool {
                if (!wait_full()) return false;
#pragma unroll
                for (int i = 0; i < kMaxGroups; ++i)
                    if (i < n_groups) tmem_ld8(lane_base + static_cast<uint32_t>(buf * kPairAccCols + 32 * i), v[i]);
                tmem_ld_wait();
                give_back();
                return true;
            };
            // SWIGLU: the arithmetic on the first accumulator takes longer than the MMAs can run ahead without the second, so that one is
            // parked in shared memory and goes back too (each thread has its own words there, nobody waits for anybody).  gate_up at
            // 1024 / 4096 tokens 47.0 -> 43.5 / 177 -> 160 us; the others, whose epilogue is short, lose by it (O at 4096 tokens 22 -> 26).
            [[maybe_unused]] uint4* park = reinterpret_cast<uint4*>(s_park) + (tid - kEpi0 * 32);
            if constexpr (PARK) {
                if (!take()) break;
                if (H == 2) {
                    if (!wait_full()) break;
#pragma unroll
                    for (int i = 0; i < kMaxGroups; ++i) {
                        if (i < n_groups) {
                            uint32_t u[8];
                            tmem_ld8(lane_base + static_cast<uint32_t>(buf * kPairAccCols + 32 * i), u);
                            tmem_ld_wait();
                            park[(2 * i) * kPairEpiWarps * 32] = make_uint4(u[0], u[1], u[2], u[3]);
                            park[(2 * i + 1) * kPairEpiWarps * 32] = make_uint4(u[4], u[5], u[6], u[7]);
                        }
                    }
                    give_back();
                }
            }
#pragma unroll 1
            for (int h = 0; h < H; ++h) {
                // this lane's first token, its place in the output, and how many tokens are left from there (it has 0, 2, 4, .. of them)
                const int m0 = pt.m0 + h * NH + 8 * part + odd;
                const size_t off = static_cast<size_t>(m0) * ld + (MODE == kSwiglu ? ne >> 1 : ne);
                const int left = ne < rows ? a.M - m0 : 0;
                // the residual of the first group while the tensor core is still at it
                __half2 res[4];
                auto load_res = [&](int i) {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (32 * i + 2 * q < left) res[q] = *reinterpret_cast<const __half2*>(a.residual + off + static_cast<size_t>(32 * i + 2 * q) * ld);
                };
                if (WORDS && add) load_res(0);
                if constexpr (!PARK) {
                    if (!take()) break;
                } else if (h == 1) {
#pragma unroll
                    for (int i = 0; i < kMaxGroups; ++i) {
                        if (i < n_groups) {
                            const uint4 x = park[(2 * i) * kPairEpiWarps * 32], y = park[(2 * i + 1) * kPairEpiWarps * 32];
                            v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
                            v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
                        }
                    }
                }
                __half* out = a.out[pt.t] + off;
#pragma unroll
                for (int i = 0; i < kMaxGroups; ++i) {
                    if (i < n_groups) {
                        pair_exchange8(odd, v[i], [&](int q, float even_row, float odd_row) {
                            const bool on = 32 * i + 2 * q < left;
                            if constexpr (MODE == kSwiglu) {
                                const __half y = __float2half_rn(swiglu_f32(even_row, odd_row));
                                if (on) *out = y;
                            } else if constexpr (WORDS) {
                                __half2 y = __floats2half2_rn(even_row, odd_row);
                                if (add) y = __hadd2(y, res[q]);
                                if (on) {
                                    *reinterpret_cast<__half2*>(out) = y;
                                    if constexpr (STORE == kStoreWordsPeers) {
                                        for (int p = 0; p < a.num_peers; ++p) *reinterpret_cast<__half2*>(a.peer_out[p] + (out - a.out[pt.t])) = y;
                                    }
                                }
                            } else if (on) {
                                const size_t o = static_cast<size_t>(out - a.out[pt.t]);
                                for (int k = 0; k < (ne + 1 < rows ? 2 : 1); ++k) {
                                    __half y = __float2half_rn(k == 0 ? even_row : odd_row);
                                    if constexpr (MODE == kPlain) {
                                        if (add) y = __hadd(y, a.residual[o + k]);
                                        for (int p = 0; p < a.num_peers; ++p) a.peer_out[p][o + k] = y;
                                    }
                                    out[k] = y;
                                }
                            }
                            out += 2 * ld;
                        });
                        out += 24 * ld;          // the groups of the other three warps
                        if (WORDS && add && i + 1 < n_groups) load_res(i + 1);
                    }
                }
            }
        }
    } else if (warp == kMmaWarp) {
        // ================= MMA issue: one thread of the leading CTA =================
        if (leader && elect_one()) {
            const uint32_t idesc = make_idesc_pair(NH);
            const uint64_t b_desc0 = make_smem_desc(smem_u32(s_b));
            const uint32_t b_step = static_cast<uint32_t>(b_bytes) >> 4, b_boxd = static_cast<uint32_t>(b_box) >> 4;
            int slot = 0, buf = 0;
            uint32_t ph = 0, eph = 1;            // eph: parity that frees an accumulator (fresh barriers pass)
            bool ok = true;
            // the eight MMAs of one step into one accumulator
            auto issue = [&](int sl, int half, int buffer, bool fresh) {
                const uint32_t a_tmem = tmem_base + static_cast<uint32_t>(kPairACol + sl * kPairACols);
                const uint64_t b_desc = b_desc0 + static_cast<uint32_t>(sl) * b_step + static_cast<uint32_t>(half) * 2u * b_boxd;
                const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(buffer * kPairAccCols);
#pragma unroll
                for (int ks = 0; ks < kGroup / 16; ++ks)
                    tc_mma_f16_pair_ts(tmem_d, a_tmem + 8u * ks, b_desc + (ks >= 4 ? b_boxd : 0u) + static_cast<uint32_t>(2 * (ks & 3)), idesc,
                                       (ks != 0 || !fresh) ? 1u : 0u);
            };
            auto advance = [&](int& sl, uint32_t& p) {
                if (++sl == kPairSlots) { sl = 0; p ^= 1; }
            };
            bool ready = mbar_test_wait(full(0), 0);
            for (int pt_i = pair_id; pt_i < total_pt && ok; pt_i += num_pairs) {
                if (!mbar_wait(acc_empty(buf), eph, s_abort)) break;
                tc_fence_after();
                int st = 0;
                bool first_half_committed = false;
                if (H == 2) {
                    // the first half runs ahead while the epilogue still has the second
                    int ahead = 0, sl = slot;
                    uint32_t p = ph;
                    const int most = min(kPairSlots, G);
                    while (ahead < most && !mbar_test_wait(acc_empty(1), eph)) {
                        if (!mbar_wait(full(sl), p, s_abort)) { ok = false; break; }
                        tc_fence_after();
                        issue(sl, 0, 0, ahead == 0);
                        advance(sl, p);
                        ++ahead;
                    }
                    if (!ok || !mbar_wait(acc_empty(1), eph, s_abort)) break;
                    tc_fence_after();
                    for (; st < ahead; ++st) {
                        issue(slot, 1, 1, st == 0);
                        tc_commit_pair(done(slot));
                        advance(slot, ph);
                    }
                    if (ahead > 0) ready = st < G && mbar_test_wait(full(slot), ph);
                }
                for (; st < G; ++st) {
                    if (!ready && !mbar_wait(full(slot), ph, s_abort)) { ok = false; break; }
                    tc_fence_after();
                    const int sl = slot;
                    advance(slot, ph);
                    ready = mbar_test_wait(full(slot), ph);      // the answer arrives while the MMAs below are issued
                    issue(sl, 0, H == 2 ? 0 : buf, st == 0);
                    if (H == 2) {
                        if (st == G - 1) { tc_commit_pair(acc_full(0)); first_half_committed = true; }
                        issue(sl, 1, 1, st == 0);
                    }
                    tc_commit_pair(done(sl));
                }
                if (!ok) break;
                if (H == 2) {
                    if (!first_half_committed) tc_commit_pair(acc_full(0));   // (all of a short tile was issued ahead)
                    tc_commit_pair(acc_full(1));
                    eph ^= 1;
                } else {
                    tc_commit_pair(acc_full(buf));
                    buf ^= 1;
                    if (buf == 0) eph ^= 1;
                }
            }
        }
        __syncwarp();
    } else if (warp == kRawWarp) {
        // ================= TMA: raw packed weights of this CTA's 128 rows (private ring) =================
        if (elect_one()) {
            int rs = 0;
            uint32_t rph = 1;
            bool ok = true;
            for (int pt_i = pair_id; pt_i < total_pt && ok; pt_i += num_pairs) {
                const PairTile pt = pair_tile(a, pt_i, n_pairs, rank, MODE == kQkv);
                for (int s = 0; s < G; ++s) {
                    if (!mbar_wait(raw_empty(rs), rph, s_abort)) { ok = false; break; }
                    mbar_arrive_expect_tx(raw_full(rs), kPairRawBytes);
                    tma_load_2d(smem_u32(s_raw + rs * kPairRawBytes), &a.tmap_w[pt.t], s * 64, pt.n0, raw_full(rs));
                    if (++rs == kRawSlots) { rs = 0; rph ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == kRawWarp + 1) {
        // ================= TMA: this CTA's half of the token tile; bytes counted on the LEADER's barrier =================
        if (elect_one()) {
            int slot = 0;
            uint32_t dph = 1;
            bool ok = true;
            const uint32_t leader_full0 = cluster_map_shared(full(0), 0);
            pdl_wait_prior_grids();
            for (int pt_i = pair_id; pt_i < total_pt && ok; pt_i += num_pairs) {
                const PairTile pt = pair_tile(a, pt_i, n_pairs, rank, MODE == kQkv);
                for (int s = 0; s < G; ++s) {
                    if (!mbar_wait(done(slot), dph, s_abort)) { ok = false; break; }
                    if (leader) mbar_arrive_expect_tx(full(slot), static_cast<uint32_t>(2 * b_bytes));
                    uint32_t dst = smem_u32(s_b + slot * b_bytes);
                    for (int h = 0; h < H; ++h)
                        for (int kk = 0; kk < 2; ++kk, dst += b_box)
                            tma_load_2d_pair(dst, &a.tmap_x, s * kGroup + kk * kBK, pt.m0 + h * NH + rank * (NH / 2), leader_full0 + 8u * slot);
                    if (++slot == kPairSlots) { slot = 0; dph ^= 1; }
                }
            }
        }
        __syncwarp();
    }

    // Neither CTA may leave (or free its tensor memory) while the other's instructions can still touch its
    // shared memory, barriers or accumulators.
    tc_fence_before();
    __syncthreads();
    if (*s_abort) __nanosleep(500000);      // a bounded wait ran out: what is in flight lands before the memory goes
    cluster_sync_all();
    if (warp == kMmaWarp) tmem_dealloc_pair(tmem_base, 512);
}

// ---- host side ----
size_t tc_pair_smem_bytes(int mode, int T) {
    return 1024 + static_cast<size_t>(kPairSlots) * T * 128 + static_cast<size_t>(pair_raw_slots(mode)) * kPairRawBytes +
           (pair_parks(mode) && T > kPairAccCols ? kPairParkBytes : 0) +
           (2 * kPairMaxRaw + 2 * kPairSlots + 4) * 8 + 16;
}
// Estimated cycles of a launch with token tiles of T, from measurements on B200: a step takes 4 T of MMA or 1100 of
// dequantisation, whichever is more; a tile of two accumulators waits 2500 for the second one to be drained; the first fill,
// the exchange at the start and the last tile's epilogue are not overlapped.  (Constants of the kernel's first form.  A fit to the
// present one, 4.4 T, 780 and 1900, is closer to the times but picks worse tiles: gate_up at 4096 tokens 183 -> 199 us, QKV 24 -> 29.)
double pair_cost(int M, int n_pairs, int steps, int pairs, int T) {
    const int tiles = n_pairs * ((M + T - 1) / T), rounds = (tiles + pairs - 1) / pairs;
    return rounds * (steps * std::max(4.0 * T, 1100.0) + (T > kPairAccCols ? 2500.0 : 0.0)) + 9000.0 + 25.0 * T;
}
// The token tile for `n_pairs` pairs of row tiles on `pairs` pairs of SMs: one accumulator of 16..128 or two of 80..128.
int pair_token_tile(int M, int n_pairs, int steps, int pairs, double* estimate) {
    int best = 16;
    double best_cost = 0;
    for (int T = 16; T <= 2 * kPairAccCols; T += T < kPairAccCols ? 16 : 32) {
        const double cost = pair_cost(M, n_pairs, steps, pairs, T);
        if (best_cost == 0 || cost < best_cost) { best = T; best_cost = cost; }
    }
    if (estimate != nullptr) *estimate = best_cost;
    return best;
}
