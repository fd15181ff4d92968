// Fused linear layer y = act(x · Wᵀ + bias) for sm_100a, large problems: CTA PAIRS on 256 x 256 tiles.
//
// linear.cuh gives every SM its own 128 x 256 tile: per 64-wide k-block an SM pulls 16 KB of x and
// 32 KB of W through shared memory for 512 tensor-core cycles, and neighbouring SMs load the same W
// tile again from L2 (ncu on [8192,4096]x[11008,4096]: 2.7x the algorithmic DRAM bytes, tensor pipe
// 79 % busy). Here two CTAs of a cluster (two neighbouring SMs) share one 256 x 256 output tile and
// issue `tcgen05.mma.cta_group::2`: each CTA stages its own 128 rows of x and only HALF of the W tile
// (128 of its 256 rows), the tensor cores of both SMs read both halves, and each CTA ends up with its
// 128 rows of the result in its own tensor memory. Per SM and k-block that is 32 KB through shared
// memory instead of 48 KB, and every W byte is fetched once per pair instead of once per SM.
//
// Roles per CTA (576 threads): warp 0 TMA producer, warp 1 tcgen05 issuer (only the pair's leader —
// cluster rank 0 — issues; the other CTA's warp 1 only allocates tensor memory), warps 2..17
// epilogue: warp w reads the tensor-memory lanes of quadrant w % 4 (its 32 rows) and the 64 (narrow tile: 48) columns
// (w - 2) / 4 of the CTA's 128 x 256 accumulator. Sixteen warps, because with a short K loop the
// epilogue is the longer of the two pipelines: clock stamps at K = 768 showed eight warps needing
// 7500-9000 cycles per tile (tensor-memory reads, conversion and stores each saturate their unit in
// turn, all warps in the same phase) against 6144 tensor-pipe cycles of the main loop. Barriers:
//   full[s]    in the LEADER's shared memory: the leader's producer arrives with the byte count of all
//              four copies of a stage; both CTAs' TMA copies complete on it (the second CTA addresses
//              it through the cluster's shared window);
//   empty[s]   in each CTA: `tcgen05.commit` of the leader, multicast to both CTAs;
//   tfull[a]   in each CTA: accumulator a complete (multicast commit);
//   tempty[a]  in the leader: all 32 epilogue warps of the pair have read accumulator a (a warp
//              arrives as soon as the last of its columns are in registers: ahead of the conversion and store of its only box of 48,
//              or of the second of its two boxes of 32; behind the second one's store [4096, 256] x [8192, 256] took 23.4 us, 22.3 so).
// Accumulators are double-buffered (2 x 256 columns = all of tensor memory), the ring has six stages.
// Every bulk copy has one destination CTA: the pair's sharing happens inside the tensor-core instruction.
#pragma once
#include <type_traits>

#include "linear.cuh"
#include "rope.cuh"

namespace kb {

constexpr int kPairBN = 256;          // columns of the pair's widest tile (the kernel is also built for 192)
#ifndef KB_PAIR_STAGES
#define KB_PAIR_STAGES 6
#endif
constexpr int kPairStages = KB_PAIR_STAGES;
constexpr int kPairABytes = kGemmBM * kGemmBK * 2;     // 16 KB: this CTA's 128 rows of x
constexpr int kPairEpilogueWarps = 16;
constexpr int kPairThreads = (2 + kPairEpilogueWarps) * 32;
// Output staging of the epilogue: 32 rows x kStoreCols columns of 16-bit results per epilogue warp, the box of one
// bulk tensor store. 256-column tiles: a warp's 64 columns go in two boxes of 32 (64-byte rows, 64-byte swizzle: piece c of
// row r sits at c ^ ((r >> 1) & 3)), so that six stages still fit beside them. 192: all 48 columns in one box
// (96-byte rows, no swizzle), and a stage needs 28 KB only.
template <int BN>
struct PairCfg {
    static_assert(BN == 256 || BN == 192, "tile width of the pair kernel");
    static constexpr int kHalfN = BN / 2;                                   // W rows staged by each CTA
    static constexpr int kStageBytes = kPairABytes + kHalfN * kGemmBK * 2;  // bytes one CTA's copies put into a stage
    static constexpr int kWarpCols = BN / 4;                                // accumulator columns of an epilogue warp
    static constexpr int kStoreCols = BN == 256 ? 32 : 48;
    static constexpr int kOutWarpBytes = 32 * kStoreCols * 2;
    static constexpr int kSmemBytes = kPairStages * kStageBytes + kPairEpilogueWarps * kOutWarpBytes + 256 + 1024;
    static_assert(kStageBytes % 1024 == 0 && kOutWarpBytes % 1024 == 0, "swizzled buffers begin at multiples of 1024 bytes");
    static_assert(kSmemBytes <= 227 * 1024 - 64, "shared memory of the pair kernel");
};
constexpr uint32_t kPairTmemCols = 512;
// The address, in the cluster's shared window, of the leader's (rank 0) copy of one of this CTA's own
// shared-memory locations: both CTAs lay out their shared memory identically.
__device__ __forceinline__ uint32_t in_leader(uint32_t own_smem_addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(own_smem_addr), "r"(0u));
    return r;
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    cluster_arrive();
    cluster_wait();
}
// Arrive on a barrier of the pair's other CTA. CTA-scope release (the default): what the arrival
// orders are this warp's tensor-memory reads, which tcgen05.wait::ld and the tcgen05 fence before it
// have completed — no global data is handed over. A cluster-scope release also waits for the warp's
// earlier global stores to be acknowledged, which showed as 3.3 stall cycles per issued instruction.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA tile load whose completion is counted on a barrier that may live in the pair's other CTA.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem of both CTAs] (+)= A[smem of both CTAs] * B[smem of both CTAs]: M = 256 (128 rows per CTA)
__device__ __forceinline__ void tc_mma_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive (once all MMAs issued so far have completed) on the barrier at this offset in BOTH CTAs.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}

// Optional clock stamps for tuning (compiled in with -DKB_GEMM_TRACE only): per CTA and for its first
// eight tiles, clock64 of: 0 issuer starts waiting for the accumulator, 1 has it, 2 has issued the
// tile's last MMA; 3 epilogue warp 2 starts waiting for the accumulator, 4 has it, 5 is done with it; 8 its
// columns are in registers, 9 its first box is in shared memory. Event 7 of tile 0 is the CTA's start.
#ifdef KB_GEMM_TRACE
__device__ long long g_gemm_trace[148 * 8 * 16];
#define KB_GTRACE(tile, ev)                                                                   \
    do {                                                                                      \
        if (blockIdx.x < 148 && (tile) < 8) g_gemm_trace[(blockIdx.x * 8 + (tile)) * 16 + (ev)] = clock64(); \
    } while (0)
#else
#define KB_GTRACE(tile, ev) do { } while (0)
#endif

// BN: columns of the pair's tile, 256 or 192. Each CTA stages BN / 2 rows of W per stage (32 or 28 KB a stage),
// the accumulators sit at tensor-memory columns 0 and 256 whatever BN, and an epilogue warp owns BN / 4 columns. The narrower
// tile leaves less undone where the wide one does not fill its rounds: [1800, 768] x [3072, 768] is 96 wide tiles on 74 pairs, two rounds
// and 13.5 us, or 128 narrow ones, two cheaper rounds and 12.5; one-round problems have the cheaper round, too. (Where both take several rounds
// there is little between them: [8192, 768] x [3072, 768], 6 or 7 rounds, 34.9 us both.)
// ROPE: a stacked q/k/v projection whose results are rotated (q, k) on their way out and whose k and v go to the cache, [B, H, max_seq, D].
// Saves the kernel behind it its pass over the projection's result (402 MB per layer at 8192 rows of [12288, 4096], 74 us).
struct PairRope {
    CUtensorMap k, v;  // the caches; q goes by tmap_y
    RopeDev r;
};
struct NoRope {};
// Eight bias values. SLICE: a bias that does not lie at a whole 16 bytes, value by value. It has kernels of its own: behind a branch here,
// also one that is not taken, the loads of a box are waited for at once (2115 rows of [1440, 360] 8.2 us, 8.8 with the branch).
// With the threads storing for themselves, as for rows of y at odd places, such calls took 12.6 to 41 us for 8.8 to 25.
template <typename T, bool SLICE>
__device__ __forceinline__ uint4 bias_8(const T* p) {
    if (!SLICE) return __ldg(reinterpret_cast<const uint4*>(p));
    const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = (uint32_t)__ldg(h + 2 * i) | ((uint32_t)__ldg(h + 2 * i + 1) << 16);
    return make_uint4(w[0], w[1], w[2], w[3]);
}
template <typename T, int BN, bool ROPE = false, bool SLICE = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
linear_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                   const __grid_constant__ CUtensorMap tmap_y, int staged, const T* __restrict__ bias, T* __restrict__ y, T* __restrict__ act_inputs, int M, int N, int K,
                   int64_t y_row_stride, int activation, const __grid_constant__ std::conditional_t<ROPE, PairRope, NoRope> rope) {
    constexpr int STAGES = kPairStages;
    using Cfg = PairCfg<BN>;
    static_assert(!ROPE || BN == 256, "the rotary epilogue takes boxes of 32 columns, inside a head");
    constexpr int kStageBytes = Cfg::kStageBytes;
    constexpr int CW = Cfg::kWarpCols;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* out_stage = smem + STAGES * kStageBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + kPairEpilogueWarps * Cfg::kOutWarpBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();  // 0 = the pair's leader
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

    // A wait that expired earlier leaves the status word set: such a launch does no work. Both CTAs
    // of a pair must take the same decision (they allocate tensor memory together), so the leader's
    // reading counts for both: it is exchanged through the cluster barrier below. It may be too early
    // (status_word()); the epilogue looks again before it stores.
    __shared__ int s_skip, s_expired;
    if (threadIdx.x == 0) {
        KB_GTRACE(0, 7);
        s_skip = status_word();
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 2 * kPairEpilogueWarps);  // the epilogue warps of both CTAs
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmap_x);
        tma_prefetch_desc(&tmap_w);
        if (staged) tma_prefetch_desc(&tmap_y);
    }
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers exist before anybody signals across the pair
    // the leader's decision, read from its shared memory through the cluster window
    int skip;
    {
        const uint32_t leader_skip = in_leader(smem_u32(&s_skip));
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(skip) : "r"(leader_skip) : "memory");
    }
    if (skip == 0) {
        if (warp == 1) {
            tmem_alloc_pair(smem_u32(tmem_slot), kPairTmemCols);
            tmem_relinquish_pair();
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }
    const uint32_t tmem_base = (skip == 0) ? *tmem_slot : 0u;
    // Launched with programmatic dependent launch: barriers, tensor memory and descriptors are set up while the
    // kernel ahead drains (a 30 us GEMM of an encoder spent 2-3 us of it on them). Nothing of global memory
    // but the status word has been touched so far.
    pdl_wait();

    const int num_m = (M + 2 * kGemmBM - 1) / (2 * kGemmBM);  // 256-row tiles
    const int num_n = (N + BN - 1) / BN;
    const int num_tiles = num_m * num_n;
    const int num_k = (K + kGemmBK - 1) / kGemmBK;

    if (skip == 0 && warp == 0) {
        // ------------------------------------------------------------------ TMA producer (both CTAs)
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = pair; t < num_tiles && ok; t += num_pairs) {
                int m_idx, n_idx;
                tile_coords(t, num_m, num_n, m_idx, n_idx);
                const int row0 = m_idx * 2 * kGemmBM + (int)rank * kGemmBM;    // this CTA's rows of x
                const int wrow0 = n_idx * BN + (int)rank * Cfg::kHalfN;    // this CTA's rows of W
                for (int kb = 0; kb < num_k; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1, abort_flag, 110)) { ok = false; break; }
                    // the leader's barrier counts the bytes of both CTAs' copies of this stage
                    if (rank == 0) mbar_arrive_expect_tx(full_bar(stage), 2 * kStageBytes);
                    const uint32_t a_dst = smem_base + stage * kStageBytes;
                    const uint32_t leader_full = in_leader(full_bar(stage));
                    tma_load_2d_pair(a_dst, &tmap_x, leader_full, kb * kGemmBK, row0);
                    tma_load_2d_pair(a_dst + kPairABytes, &tmap_w, leader_full, kb * kGemmBK, wrow0);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
            pdl_launch_dependents();  // every load is on its way: what is left are the last tile's products and its epilogue
            if (!ok) {
                for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies in flight land
            }
        }
    } else if (skip == 0 && warp == 1) {
        // ------------------------------------------------------------------ tcgen05 issuer (leader only)
        if (rank == 0 && elect_one()) {
            constexpr uint32_t idesc = make_idesc_f16(Elem<T>::kIsBf16, 2 * kGemmBM, BN, 0, 0);
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool ok = true;
            int ti = 0;
            for (int t = pair; t < num_tiles && ok; t += num_pairs, ++ti) {
                KB_GTRACE(ti, 0);
                if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1, abort_flag, 210)) { ok = false; break; }
                KB_GTRACE(ti, 1);
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * kPairBN);
                for (int kb = 0; kb < num_k; ++kb) {
                    if (!mbar_wait(full_bar(stage), phase, abort_flag, 211)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_base + stage * kStageBytes;
                    const uint64_t a_desc = make_smem_desc_sw128(a_addr, 16, 1024);
                    const uint64_t b_desc = make_smem_desc_sw128(a_addr + kPairABytes, 16, 1024);
#pragma unroll
                    for (int k = 0; k < kGemmBK / 16; ++k)
                        tc_mma_ss_pair(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit_pair(empty_bar(stage));  // frees this stage in both CTAs
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                tc_commit_pair(tfull_bar(acc));  // both CTAs' epilogues may read accumulator `acc`
                KB_GTRACE(ti, 2);
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
        }
    } else if (skip == 0) {
        // ------------------------------------------------------------------ epilogue (both CTAs)
        const int q = warp & 3;                 // TMEM lane quadrant this warp may access
        const int c_begin = ((warp - 2) >> 2) * CW;  // the warp's CW columns of the tile
        const uint32_t leader_tempty[2] = {in_leader(tempty_bar(0)), in_leader(tempty_bar(1))};
        uint8_t* mine = out_stage + (warp - 2) * Cfg::kOutWarpBytes;
        const bool gated = CW == 64 && activation == KB_ACT_SWIGLU;  // (192-column tiles are not chosen for it; forced, they store value by value)
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        int ti = 0;
        if (threadIdx.x == 64) s_expired = status_word();
        named_barrier(1, kPairEpilogueWarps * 32);
        const int m_end = s_expired == 0 ? M : 0;  // rows that may be stored
        int m_idx, n_idx;
        tile_coords(pair, num_m, num_n, m_idx, n_idx);
        for (int t = pair; t < num_tiles && ok; t += num_pairs, ++ti) {
            const int n0 = n_idx * BN;
            const int row_base = m_idx * 2 * kGemmBM + (int)rank * kGemmBM + q * 32;  // the warp's first row
            // The bias of the warp's first box, asked for ahead of the accumulator (loads between the conversions of a box stalled
            // every 16 columns: 2300 cycles for 48 columns without an activation). Every lane reads the same 16 bytes.
            constexpr int kPieces = Cfg::kStoreCols / 8;  // 16-byte pieces of a staged row
            uint4 bias_w[kPieces];
            auto load_bias = [&](int c) {
#pragma unroll
                for (int v = 0; v < kPieces; ++v) {
                    const int col = n0 + c_begin + c + v * 8;
                    bias_w[v] = staged && bias != nullptr && col < N ? bias_8<T, SLICE>(bias + col) : make_uint4(0u, 0u, 0u, 0u);
                }
            };
            load_bias(0);
            if (warp == 2 && lane == 0) KB_GTRACE(ti, 3);
            if (!mbar_wait(tfull_bar(acc), acc_phase, abort_flag, 310)) { ok = false; break; }
            if (warp == 2 && lane == 0) KB_GTRACE(ti, 4);
            tc_fence_after();
            if (staged) {
                // Whole boxes of results go through shared memory to bulk tensor stores, one per warp: what a warp's
                // own stores cost (a thousand cycles per 16 columns with all sixteen warps at it, 6000 to 7500 per tile, where a
                // main loop of twelve k-blocks takes 4600 to 6100) the copy engine does while the warps convert: 1500 to 2500
                // cycles, 3500 to 4500 with a GELU. [8192, 768] x [2304, 768] 26.4 -> 24.0 us, x [3072, 768] with GELU 36.8 -> 33.6,
                // [4000, 512] x [3000, 512] 16.3 -> 13.9 (clocks at the power cap for the first two).
                // (256 columns: a box's 32 at a time. All 64 at once and the bias do not fit in 96 registers.)
                constexpr int SC = Cfg::kStoreCols;
                uint32_t r2[SC];
                const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * kPairBN + c_begin);
                tmem_ld_32x32(t_addr, *reinterpret_cast<uint32_t(*)[32]>(&r2[0]));
                if (SC == 48) tmem_ld_32x16(t_addr + 32, *reinterpret_cast<uint32_t(*)[16]>(&r2[SC - 16]));
                tmem_ld_wait();
                auto release = [&] {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(leader_tempty[acc]);
                };
                if (SC == CW) release();
                if (warp == 2 && lane == 0) KB_GTRACE(ti, 8);
                // z = accumulator + bias of the 16 columns from c on (of a box; their bias is in bias_w[c / 8] and the one behind it)
                auto add_bias = [&](int c, float (&z)[16]) {
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        const uint4 w = bias_w[c / 8 + g];
                        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float2 b2 = Elem<T>::unpack2(ww[i]);
                            z[g * 8 + 2 * i] = __uint_as_float(r2[c + g * 8 + 2 * i]) + b2.x;
                            z[g * 8 + 2 * i + 1] = __uint_as_float(r2[c + g * 8 + 2 * i + 1]) + b2.y;
                        }
                    }
                };
                uint32_t o[kPieces * 4];
#pragma unroll
                for (int bx = 0; bx < CW / SC; ++bx) {
                    if (gated) {
                        // blocks of eight gate and eight up columns: the 64 accumulator columns make one box of 32
#pragma unroll
                        for (int c = 0; c < SC; c += 16) {
                            float z[16];
                            add_bias(c, z);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                o[(bx * SC + c) / 4 % (kPieces * 4) + i] = Elem<T>::pack2(act_silu(z[2 * i]) * z[8 + 2 * i], act_silu(z[2 * i + 1]) * z[8 + 2 * i + 1]);
                        }
                    } else if constexpr (ROPE) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = Elem<T>::pack2(__uint_as_float(r2[2 * i]), __uint_as_float(r2[2 * i + 1]));
                    } else {
#pragma unroll
                        for (int c = 0; c < SC; c += 16) {
                            float z[16];
                            add_bias(c, z);
                            apply_activation<16>(z, activation);
#pragma unroll
                            for (int i = 0; i < 8; ++i) o[c / 2 + i] = Elem<T>::pack2(z[2 * i], z[2 * i + 1]);
                        }
                    }
                    if (bx + 1 < CW / SC) {
                        load_bias((bx + 1) * SC);
                        tmem_ld_32x32(t_addr + (uint32_t)((bx + 1) * SC), *reinterpret_cast<uint32_t(*)[32]>(&r2[0]));
                    }
                    const int ycol = gated ? (n0 + c_begin) / 2 : n0 + c_begin + bx * SC;
                    if (gated && bx + 1 < CW / SC) {  // (half of the box only)
                        tmem_ld_wait();
                        if (bx + 2 == CW / SC) release();
                        continue;
                    }
                    int part = 0, b0 = 0, head = 0, d0 = 0;  // ROPE: q, k or v; the first row's sequence; head and its first column
                    long long pos0 = 0;                      // the first row's position
                    bool box = true;                         // the rows go out as one box
                    if constexpr (ROPE) {
                        const RopeDev& rp = rope.r;
                        const int hd = rp.H * rp.D;
                        part = ycol / hd;
                        head = (ycol % hd) / rp.D;
                        d0 = (ycol % hd) % rp.D;
                        b0 = row_base / rp.S;
                        const long long first = rp.pos_dev ? *rp.pos_dev : rp.pos_host;
                        pos0 = first + (row_base - b0 * rp.S);
                        const int row = row_base + lane, b = row / rp.S;
                        const long long pos = first + (row - b * rp.S);
                        const bool inside = pos >= 0 && pos < rp.max_seq;
                        if (part < 2) {
                            const int64_t at = (inside ? pos : 0) * (rp.D / 2) + d0 / 2;
#pragma unroll
                            for (int v = 0; v < 4; ++v) {
                                const float4 c4 = __ldg(reinterpret_cast<const float4*>(rp.cos_t + at) + v), s4 = __ldg(reinterpret_cast<const float4*>(rp.sin_t + at) + v);
                                const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const float2 t2 = rope_pair(Elem<T>::unpack2(o[v * 4 + i]), cs[i], ss[i]);
                                    o[v * 4 + i] = Elem<T>::pack2(t2.x, t2.y);
                                }
                            }
                        }
                        // Stored one by one: rows of k and v that lie in two sequences, or beyond the last one, and boxes with a position
                        // outside the cache, whose rows (those of q too) stay as they are, as in rope_kv_write_kernel. Positions are compared
                        // in 64 bits; those of a whole box fit the copy's 32-bit coordinate.
                        box = __all_sync(0xffffffffu, inside || row >= M) && (part == 0 || (row_base + 31 < M && (row_base + 31) / rp.S == b0));
                        if (!box && row < m_end && inside && ycol < N) {
                            T* dst = part == 0 ? reinterpret_cast<T*>(rp.q_out) + (int64_t)row * hd + ycol
                                               : reinterpret_cast<T*>(part == 1 ? rp.k_cache : rp.v_cache) + (((int64_t)b * rp.H + head) * rp.max_seq + pos) * rp.D + d0;
#pragma unroll
                            for (int v = 0; v < 4; ++v) reinterpret_cast<uint4*>(dst)[v] = make_uint4(o[v * 4], o[v * 4 + 1], o[v * 4 + 2], o[v * 4 + 3]);
                        }
                    }
                    if (lane == 0) bulk_wait_read();  // the box before this one has left the buffer
                    __syncwarp();
                    if (SC == 32) {
#pragma unroll
                        for (int v = 0; v < kPieces; ++v)
                            *reinterpret_cast<uint4*>(mine + lane * 64 + ((v ^ ((lane >> 1) & 3)) * 16)) =
                                make_uint4(o[v * 4], o[v * 4 + 1], o[v * 4 + 2], o[v * 4 + 3]);
                    } else {
                        // rows of 96 bytes: lanes l and l + 4 meet in the same banks, so every other four lanes take their pieces in
                        // pairs the other way round
                        const bool swap = (lane & 4) != 0;
#pragma unroll
                        for (int v = 0; v < kPieces; ++v) {
                            uint4 w;
                            w.x = swap ? o[(v ^ 1) * 4 + 0] : o[v * 4 + 0];
                            w.y = swap ? o[(v ^ 1) * 4 + 1] : o[v * 4 + 1];
                            w.z = swap ? o[(v ^ 1) * 4 + 2] : o[v * 4 + 2];
                            w.w = swap ? o[(v ^ 1) * 4 + 3] : o[v * 4 + 3];
                            *reinterpret_cast<uint4*>(mine + lane * 96 + (swap ? v ^ 1 : v) * 16) = w;
                        }
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (warp == 2 && lane == 0 && bx == 0) KB_GTRACE(ti, 9);
                    if (lane == 0 && row_base < m_end && ycol < (gated ? N / 2 : N)) {
                        if constexpr (ROPE) {
                            if (part == 0 && box) tma_store_2d(&tmap_y, smem_u32(mine), ycol, row_base);
                            else if (box) tma_store_4d(part == 1 ? &rope.k : &rope.v, smem_u32(mine), d0, (int)pos0, head, b0);
                        } else {
                            tma_store_2d(&tmap_y, smem_u32(mine), ycol, row_base);
                        }
                        bulk_commit();
                    }
                    if (bx + 1 < CW / SC) {
                        tmem_ld_wait();
                        if (bx + 2 == CW / SC) release();  // the last box is in registers
                    }
                }
                if (t + num_pairs < num_tiles) tile_coords(t + num_pairs, num_m, num_n, m_idx, n_idx);
            } else {
                const int row = row_base + lane;
                T* y_row = y + (int64_t)row * y_row_stride;
                T* a_row = act_inputs ? act_inputs + (int64_t)row * y_row_stride : nullptr;
#pragma unroll 1
                // (a 32-column chunk at a time: with 48 columns per warp, warps pair up on chunks — the
                // even warp of a pair of column groups takes the chunk that straddles them)
                for (int c0 = (c_begin / 32) * 32; c0 < c_begin + CW; c0 += 32) {
                    if (n0 + c0 >= N) break;
                    if (c0 < c_begin || c0 + 32 > c_begin + CW) {
                        if ((((warp - 2) >> 2) & 1) != 0) continue;  // the straddling chunk belongs to the even group
                    }
                    uint32_t r[32];
                    tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * kPairBN + c0), r);
                    tmem_ld_wait();
                    float accv[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) accv[j] = __uint_as_float(r[j]);
                    if (activation == KB_ACT_SWIGLU) epilogue_chunk_swiglu<T>(accv, bias, y_row, n0 + c0, N, row < m_end);
                    else epilogue_chunk<T>(accv, bias, y_row, a_row, n0 + c0, N, row < m_end, activation);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_tempty[acc]);  // counted in the leader, whose issuer reuses the accumulator
                if (t + num_pairs < num_tiles) tile_coords(t + num_pairs, num_m, num_n, m_idx, n_idx);
            }
            if (warp == 2 && lane == 0) KB_GTRACE(ti, 5);
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
        if (staged && lane == 0) bulk_wait_all();
    }

    // Teardown: every role of both CTAs falls through to here, also after an abandoned wait. Neither
    // CTA may retire while the other can still signal its barriers or use its tensor memory.
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (skip == 0 && warp == 1) {
        __syncwarp();
        tmem_dealloc_pair(tmem_base, kPairTmemCols);
    }
}

static int g_linear_pair = 1;  // test hook (kb_debug_linear_pair): 0 = never use the pair kernel, 192 / 256 = force that tile width

// Whether the rows of y do not allow stores of 16 bytes.
static bool linear_stores_values(const kb_linear_params& p) { return p.y_row_stride % 8 != 0 || (((uintptr_t)p.y) & 15) != 0; }

// Whether results leave through bulk tensor stores: rows of y at whole 16 bytes, no pre-activation output, whole pieces of eight
// columns of y and bias (wherever the bias begins); the gated form needs the 64 accumulator columns per warp of the wide tile.
static bool linear_pair_staged(const kb_linear_params& p, int bn) {
    if (p.act_inputs != nullptr || linear_stores_values(p) || p.y_row_stride <= 0) return false;
    return p.activation == KB_ACT_SWIGLU ? bn == 256 && p.N % 16 == 0 : p.N % 8 == 0;
}

// What a GEMM kernel whose CTAs stay for several tiles costs, in us: a fixed part, more of it when there is one round of tiles only,
// whose first operands and epilogue nothing hides; per round the k-blocks of 64, each the dearer the more SMs pull on L2 at once, and
// the part of an epilogue that the next tile does not hide, with what a GELU's exponential adds to it, what a gated epilogue, which
// stores half, takes off, and what threads that store for themselves add, by 16 bytes a row or value by value; more of it for rows of x
// and W that are no multiple of 128 bytes. Fitted to 12 400 problems of 129 to 8192 rows (ratios of the kernels' times inside each problem).
struct GemmCost {
    double fixed, one_round, block, busy_block, epilogue, gelu, gated, ragged, ragged_epilogue, rows, values;
};
static double gemm_us(const GemmCost& c, const kb_linear_params& p, int64_t tiles, int64_t slots, bool by_rows) {
    const int64_t rounds = (tiles + slots - 1) / slots;
    const double busy = (double)tiles / (double)(rounds * slots), num_k = (double)((p.K + kGemmBK - 1) / kGemmBK);
    const bool ragged = p.K % kGemmBK != 0;
    const double block = (c.block + c.busy_block * busy * busy * busy) * (ragged ? 1.0 + c.ragged : 1.0);
    const double act = p.activation == KB_ACT_GELU ? c.gelu : p.activation == KB_ACT_SWIGLU ? c.gated : 0.0;
    const double stores = linear_stores_values(p) ? c.values : by_rows ? c.rows : 0.0;
    const double us = c.fixed + (rounds == 1 ? c.one_round : 0.0) + (double)rounds * (num_k * block + c.epilogue + act + (ragged ? c.ragged_epilogue : 0.0) + stores);
    const double hbm = c.fixed + (double)p.N * (double)p.K * 2.0 / 6.8e6;  // W once from memory
    return us > hbm ? us : hbm;
}

// Estimated time in us of the pair kernel with tiles of 256 x `bn`.
static double linear_pair_us(const kb_linear_params& p, int bn) {
    static constexpr GemmCost kNarrow{3.3, 1.04, 0.244, 0.068, 0.60, 0.70, 0.0, 0.10, 0.45, 3.5, 23.0};
    static constexpr GemmCost kWide{3.3, 1.25, 0.311, 0.100, 0.64, 0.70, 0.0, 0.05, 0.40, 5.5, 31.0};
    const int64_t pairs = gemm_sms() / 2 > 0 ? gemm_sms() / 2 : 1;
    return gemm_us(bn == 192 ? kNarrow : kWide, p, ((p.M + 255) / 256) * ((p.N + bn - 1) / bn), pairs, !linear_pair_staged(p, bn));
}

// Tile width (192 or 256 columns), and the estimate that goes with it.
static int linear_pair_tile_width(const kb_linear_params& p, double* us) {
    const double wide = linear_pair_us(p, 256), narrow = linear_pair_us(p, 192);
    const int bn = g_linear_pair == 192 || g_linear_pair == 256 ? g_linear_pair : p.activation != KB_ACT_SWIGLU && narrow < wide ? 192 : 256;
    *us = bn == 192 ? narrow : wide;
    return bn;
}

template <typename T, int BN, bool ROPE = false, bool SLICE = false>
static int launch_linear_pair_tb(const kb_linear_params& p, cudaStream_t stream, const RopeDev* rope = nullptr) {
    using Cfg = PairCfg<BN>;
    auto kernel = linear_pair_kernel<T, BN, ROPE, SLICE>;
    std::conditional_t<ROPE, PairRope, NoRope> rp;
    if constexpr (ROPE) {
        rp.r = *rope;
        const uint64_t dims[4] = {(uint64_t)rope->D, (uint64_t)rope->max_seq, (uint64_t)rope->H, (uint64_t)rope->B};
        const uint64_t row = (uint64_t)rope->D * 2, strides[4] = {0, row, row * rope->max_seq, row * rope->max_seq * rope->H};
        const uint32_t box[4] = {32, 32, 1, 1};
        int st = encode_tmap_16bit(&rp.k, rope->k_cache, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (st == KB_OK) st = encode_tmap_16bit(&rp.v, rope->v_cache, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (st != KB_OK) return st;
    }
    CUtensorMap tmap_x, tmap_w, tmap_y;
    {
        const uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)p.M};
        const uint64_t strides[2] = {0, (uint64_t)p.x_row_stride * 2};
        const uint32_t box[2] = {kGemmBK, kGemmBM};
        int st = encode_tmap_16bit(&tmap_x, p.x, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (st != KB_OK) return st;
    }
    {
        const uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)p.N};
        const uint64_t strides[2] = {0, (uint64_t)p.K * 2};
        const uint32_t box[2] = {kGemmBK, BN / 2};
        int st = encode_tmap_16bit(&tmap_w, p.w, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (st != KB_OK) return st;
    }
    int staged = ROPE || linear_pair_staged(p, BN) ? 1 : 0;
    if (staged) {
        const int64_t cols = p.activation == KB_ACT_SWIGLU ? p.N / 2 : ROPE ? p.N / 3 : p.N;  // (ROPE: q alone)
        const uint64_t dims[2] = {(uint64_t)cols, (uint64_t)p.M};
        const uint64_t strides[2] = {0, (uint64_t)(ROPE ? cols : p.y_row_stride) * 2};
        const uint32_t box[2] = {(uint32_t)Cfg::kStoreCols, 32};
        const int st = encode_tmap_16bit(&tmap_y, ROPE ? rope->q_out : p.y, 2, dims, strides, box, BN == 256 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
                                         CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (st != KB_OK) {
            if (ROPE) return st;
            staged = 0;  // (rows of y further apart than a tensor map takes)
        }
    }
    if (!staged) tmap_y = tmap_x;  // (not used)
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // pairs that can be resident at once, per device (the grid is persistent: one pair per slot)
    static std::atomic<int> max_pairs[64] = {};  // (set after the attribute; two threads that ask at once get the same answer)
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return KB_ERR_LAUNCH;
    int resident = max_pairs[dev].load(std::memory_order_acquire);
    if (resident == 0) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess)
            return KB_ERR_LAUNCH;
        cfg.gridDim = dim3(2 * (unsigned)(sm_count() / 2));
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            return KB_ERR_LAUNCH;
        }
        resident = n < sm_count() / 2 ? n : sm_count() / 2;
        max_pairs[dev].store(resident, std::memory_order_release);
    }
    const int64_t tiles = ((p.M + 255) / 256) * ((p.N + BN - 1) / BN);
    int pairs = (int)(tiles < resident ? tiles : resident);
    if (pairs > gemm_sms() / 2) pairs = gemm_sms() / 2;  // a caller-set limit leaves SMs to a concurrent collective
    cfg.gridDim = dim3(2 * (unsigned)pairs);
    cfg.numAttrs = g_use_pdl ? 2u : 1u;
    if (cudaLaunchKernelEx(&cfg, kernel, tmap_x, tmap_w, tmap_y, staged, (const T*)p.bias, (T*)p.y, (T*)p.act_inputs, (int)p.M,
                           (int)p.N, (int)p.K, p.y_row_stride, p.activation, rp) != cudaSuccess)
        return KB_ERR_LAUNCH;
    return cudaGetLastError() == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

// Whether this kernel's rotary epilogue can take the place of the launch behind the projection: heads of whole boxes of 32 columns, stored
// at whole 16 bytes. (The streaming kernel of a decode step keeps the launch behind it: with pairs of rows as its unit and the rotation in
// its epilogue a step of eight layers took 1031 us, 1019 without, since decode attention's first K and V arrive behind that launch.)
static bool linear_pair_rope(const kb_linear_params& p, const RopeDev& r) {
    return p.activation == KB_ACT_NONE && p.bias == nullptr && p.act_inputs == nullptr && p.N == 3 * (int64_t)r.H * r.D &&
           p.M == (int64_t)r.B * r.S && r.D % 32 == 0 && (int64_t)r.H * r.max_seq * r.D < ((int64_t)1 << 38) && ((((uintptr_t)r.q_out) | ((uintptr_t)r.k_cache) | ((uintptr_t)r.v_cache)) & 15) == 0;
}

template <typename T>
static int launch_linear_pair_t(const kb_linear_params& p, cudaStream_t stream, int bn, const RopeDev* rope = nullptr) {
    if (rope != nullptr) return launch_linear_pair_tb<T, 256, true>(p, stream, rope);
    if ((((uintptr_t)p.bias) & 15) != 0 && linear_pair_staged(p, bn))
        return bn == 192 ? launch_linear_pair_tb<T, 192, false, true>(p, stream) : launch_linear_pair_tb<T, 256, false, true>(p, stream);
    return bn == 192 ? launch_linear_pair_tb<T, 192>(p, stream) : launch_linear_pair_tb<T, 256>(p, stream);
}

}  // namespace kb
