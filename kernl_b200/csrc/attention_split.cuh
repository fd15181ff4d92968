// Fused attention forward for sm_100a, head dimension 64, "split-row" variant.
//
// One 128-row query tile per CTA, two CTAs per SM, keys in blocks of 64, K/V through a 4-stage TMA
// ring, one tcgen05 issuer warp, and EIGHT softmax warps: every query row is shared by two
// threads of different warps, one owning key columns
// [0,32) of each block, the other [32,64). The two halves never talk to each other inside the key
// loop: each keeps its own running maximum and row sum, writes its own half of P, and its P·V goes
// into its own accumulator in TMEM (O_a from the keys of the first halves, O_b from the second
// halves; two K=32 tcgen05.mma chains instead of one K=64 chain, the same tensor-core work). The
// halves are merged once, in the epilogue: O = (w_a·O_a + w_b·O_b) / (w_a·l_a + w_b·l_b) with
// w_x = 2^(m_x - max(m_a, m_b)).
//
// Why: a softmax warp's block is a serial chain of fixed latencies (barrier poll, TMEM load, the
// dependent maximum reduction, special-function-unit results, TMEM store, hand-off) that one warp
// cannot overlap with itself, and with one row per thread there are only two such warps per SM
// sub-partition. Clock stamps taken inside the kernel showed a block taking ~2200 cycles of which
// the special-function unit was busy for 512. Four warps per sub-partition overlap those chains.
//
// Two independent CTAs on an SM also hide each other's fixed costs (set-up, first loads from DRAM, epilogue, exit), and
// the second wave starts per tile: one CTA of two tiles that shares K/V was 2 % (B8 H12 S4096) to 20 % (B64 H12 S512) slower.
//
// Warps (384 threads): 0..7 softmax (0..3 first halves, 4..7 second halves), 8 TMA producer, 9 tcgen05 issuer, 10..11 mask
// loaders (MODE 3). TMEM columns (256 of 512): S ring slot s at 64·s (s = 0,1; 64 fp32 columns; P of the
// first half overwrites columns [0,16), P of the second half columns [32,48) of the same slot),
// O_a at 128, O_b at 192.
#pragma once
#include "attention.cuh"

namespace kb {

struct SplitShape {
    static constexpr int kThreads = 384;
    static constexpr int kAuxWarp = 8;  // first non-softmax warp: TMA producer; the issuer follows
    static constexpr int kRegsLaunch = 80;  // 65536 / (2 x 384), rounded down to 8
    static constexpr int kRegsHigh = 96;
    static constexpr int kRegsLow = 48;
    static_assert(2 * kRegsHigh + kRegsLow <= 3 * kRegsLaunch, "setmaxnreg totals exceed the CTA's register pool");
    static_assert(kRegsHigh % 8 == 0 && kRegsLow % 8 == 0, "setmaxnreg wants multiples of 8");
};
static int g_split_tiles = 0;  // test hook: 1 = this kernel whatever the size of the launch
static int g_attn_persistent = -1;  // test hook: -1 = dispatcher's choice, 0 = one CTA per tile, 1 = persistent CTAs

__device__ __forceinline__ void tma_prefetch_l2_4d(const CUtensorMap* map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}

template <int MODE>
struct AttnSplitCfg {
    // MODE 3: mask tiles of 128 rows x 64 keys through two slots of shared memory, for which the
    // K/V ring gives up a stage (two CTAs per SM). A row is staged as the nine 16-byte chunks that hold its
    // 128 bytes wherever they start.
    static constexpr bool kMaskRing = MODE == 3;
    static constexpr int kMaskRowBytes = 9 * 16;
    static constexpr int kMaskSlotBytes = kMaskRing ? kAttnBlock * kMaskRowBytes : 0;
    static constexpr int kKvStages = kMaskRing ? 3 : 4;
    static constexpr int kQTileBytes = kAttnBlock * 64 * 2;
    static constexpr int kKvBytes = kBlkN * 64 * 2;
    static constexpr int kTilesBytes = kQTileBytes + 2 * kKvStages * kKvBytes;
    static constexpr int kBarBytes = 1024;
    static constexpr int kXchBytes = 2 * kAttnBlock * 8;  // [half][row] (m, l)
    // MODE 1 keeps the whole row-broadcast mask of its (batch, head) in shared memory, as fp32 in the
    // log2 domain, staged by all threads during set-up; longer rows are read like per-row masks (MODE 2)
    static constexpr int kMaskMaxN = 8192;
    static constexpr int kMaskLoads = (kMaskMaxN + SplitShape::kThreads - 1) / SplitShape::kThreads;  // per thread
    static constexpr int kSmemBase = kTilesBytes + kBarBytes + kXchBytes + 2 * kMaskSlotBytes + 1024;
    static constexpr int kSmemMax = kSmemBase + (MODE == 1 ? kMaskMaxN * 4 : 0);
    static_assert(!kMaskRing || 2 * (kSmemMax + 1024) <= 227 * 1024, "two CTAs per SM");
};

// A staged mask row begins at byte `lead` of its nine chunks, where `lead` is its address modulo 16, so that every
// aligned chunk of global memory is a chunk here. How much of chunk `c` belongs to the row, from the chunk's first byte on,
// for a row of `len` bytes (an even number, at most 128). What a chunk holds ahead of its row is not looked at.
__host__ __device__ constexpr int mask_chunk_bytes(int lead, int c, int len) {
    const int n = lead + len - 16 * c;
    return n < 0 ? 0 : n < 16 ? n : 16;
}
constexpr bool mask_chunks_cover_a_row() {
    for (int lead = 0; lead < 16; lead += 2)
        for (int len = 2; len <= 2 * kBlkN; len += 2) {
            int end = 0;
            for (int c = 0; c < 9; ++c) {
                const int n = mask_chunk_bytes(lead, c, len);
                if (n > 0 && (end != 16 * c || n > 16)) return false;
                if (n > 0) end = 16 * c + n;
            }
            if (end != lead + len) return false;
        }
    return true;
}
static_assert(mask_chunks_cover_a_row(), "the chunks of a staged mask row end with the row");

// Adds sixteen mask values of a staged row to scores, in score units: s += max(mask, lowest) * inv_scale, two
// values per instruction. `src` is the 16-byte chunk in which the row's 32 bytes begin, `shift` (0..7
// elements) where in it: rows of a mask whose length is no multiple of eight all start differently.
// (Read ahead of the wait for the scores instead, the sixteen words cost more in spilled registers than
// their latency: 12.6 -> 16.1 us at [3, 12, 333, 64].)
__device__ __forceinline__ void add_staged_mask(const AttnDev& p, const uint8_t* src, int shift, float inv_scale, uint32_t* sr) {
    uint32_t w[12];
    const uint4* v = reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (i == 2 && p.mask_vec) break;
        const uint4 q = v[i];
        w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
    }
    if (!p.mask_vec) {
#pragma unroll
        for (int i = 0; i < 10; ++i) w[i] = (shift & 4) ? w[i + 2] : w[i];
#pragma unroll
        for (int i = 0; i < 9; ++i) w[i] = (shift & 2) ? w[i + 1] : w[i];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], (uint32_t)(shift & 1) * 16u);
    }
    const float2 inv2 = make_float2(inv_scale, inv_scale);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float2 f;
        uint32_t m;
        if (p.mask_dtype == KB_F16) {
            asm("max.f16x2 %0, %1, %2;" : "=r"(m) : "r"(w[i]), "r"(0xfbfffbffu));  // the lowest finite value, twice
            f = Elem<__half>::unpack2(m);
        } else {
            asm("max.bf16x2 %0, %1, %2;" : "=r"(m) : "r"(w[i]), "r"(0xff7fff7fu));
            f = Elem<__nv_bfloat16>::unpack2(m);
        }
        const float2 x = __ffma2_rn(f, inv2, make_float2(__uint_as_float(sr[2 * i]), __uint_as_float(sr[2 * i + 1])));
        sr[2 * i] = __float_as_uint(x.x);
        sr[2 * i + 1] = __float_as_uint(x.y);
    }
}

// MODE 0, 1: as in attention.cuh. MODE 2: no positive scale, or a mask of which every softmax thread reads its own row: 32-bit
// values, values apart, rows of more than kMaskMaxN keys. MODE 3: per-row masks of 16-bit values side by side, staged by two
// loader warps. (A kernel each: with both in one, the general masks shared the registers and the smaller K/V ring of the staged
// ones. fp32 masks at [2, 12, 512, 64] 23.0 -> 16.8 us, staged ones at [8, 12, 512, 64] 31.0 -> 29.0.) EDGE (MODE 3): the mask begins or ends inside a 16-byte chunk, and copies of whole chunks would read outside it.
template <typename T, int MODE, bool EDGE = false>
__global__ void __launch_bounds__(SplitShape::kThreads, 2)
attention_split_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const AttnDev p) {
    using Cfg = AttnSplitCfg<MODE>;
    using Shape = SplitShape;
    constexpr int kThreads = Shape::kThreads;
    constexpr int W0 = Shape::kAuxWarp;
    constexpr int D = 64;
    constexpr int KVS = Cfg::kKvStages;
    constexpr int QTILE = Cfg::kQTileBytes;
    constexpr int KVB = Cfg::kKvBytes;
    constexpr int NB = 2;
    constexpr uint32_t kTmemCols = 256;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t q_smem = smem_u32(smem);
    const uint32_t k_smem = q_smem + QTILE;
    const uint32_t v_smem = k_smem + KVS * KVB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kTilesBytes);
    const uint32_t bar_base = smem_u32(bars);
    // q_full | o_final | p_full, s_full, pv_done [2] each | ep[4] | k_full, k_empty, v_full, v_empty [KVS] each | m_full, m_empty [2]
    const uint32_t q_full = bar_base, o_final = bar_base + 8u;
    auto p_full = [&](int bf) { return bar_base + 8u * (2 + bf); };
    auto s_full = [&](int bf) { return bar_base + 8u * (4 + bf); };
    auto pv_done = [&](int bf) { return bar_base + 8u * (6 + bf); };
    auto ep_bar = [&](int q) { return bar_base + 8u * (8 + q); };
    constexpr int kKvBar = 12;
    auto k_full = [&](int s) { return bar_base + 8u * (kKvBar + s); };
    auto k_empty = [&](int s) { return bar_base + 8u * (kKvBar + KVS + s); };
    auto v_full = [&](int s) { return bar_base + 8u * (kKvBar + 2 * KVS + s); };
    auto v_empty = [&](int s) { return bar_base + 8u * (kKvBar + 3 * KVS + s); };
    auto m_full = [&](int sl) { return bar_base + 8u * (kKvBar + 4 * KVS + sl); };
    auto m_empty = [&](int sl) { return bar_base + 8u * (kKvBar + 4 * KVS + 2 + sl); };
    constexpr int kNumBars = kKvBar + 4 * KVS + 4;
    static_assert(kNumBars * 8 + 32 <= Cfg::kBarBytes, "barrier area too small");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint32_t* act_bits = tmem_slot + 4;  // MODE 1: which key blocks have at least one unmasked key
    float2* xch = reinterpret_cast<float2*>(smem + Cfg::kTilesBytes + Cfg::kBarBytes);
    float* mask_smem = reinterpret_cast<float*>(smem + Cfg::kTilesBytes + Cfg::kBarBytes + Cfg::kXchBytes);  // MODE 1: [N rounded up to 64]
    uint8_t* mask_ring = reinterpret_cast<uint8_t*>(mask_smem);  // MODE 3: two slots of kMaskSlotBytes

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ int s_expired;  // the issuer reads the status word behind pdl_wait()
    {
        __shared__ int s_skip;
        if (threadIdx.x == 0) s_skip = status_word();  // (the epilogue looks again before it stores)
        if (MODE == 1 && threadIdx.x < 4) act_bits[threadIdx.x] = 0u;
        __syncthreads();
        if (s_skip != 0) {
            pdl_wait();
            return;
        }
    }

    const int BH = p.B * p.H;
    int bh, mt;  // (batch, head) and query tile
    attn_work_item(p, BH, (int)blockIdx.x, bh, mt);
    const int b = bh / p.H, h = bh % p.H;
    const int hk = h / p.kv_group;  // K/V head of this query head
    const int num_n_blocks = (p.N + kBlkN - 1) / kBlkN;
    const int max_blk = p.is_causal ? min(num_n_blocks, (mt + 1) * (kAttnBlock / kBlkN)) : num_n_blocks;

    // Set-up is spread over three warps so that the first loads are in flight as early as possible:
    // the TMA warp initialises the barriers its loads complete on and issues both Q tiles and the
    // first ring of K/V blocks at once; warp 0 initialises the other barriers, one per lane; warp 17
    // allocates TMEM. Everybody else meets them at the barrier below.
    // MODE 1 does not know which key blocks it will visit before the mask has been looked at: it
    // only pulls the first ring of K/V blocks into L2 and issues the real loads after the set-up barrier.
    const int first_kv = (MODE == 1) ? 0 : min(KVS, max_blk);
    if (warp == W0) {
        if (lane == 0) {
            tma_prefetch_desc(&tmap_q);
            tma_prefetch_desc(&tmap_k);
            tma_prefetch_desc(&tmap_v);
            mbar_init(q_full, 1);
            for (int s = 0; s < KVS; ++s) {
                mbar_init(k_full(s), 1);
                mbar_init(k_empty(s), 1);
                mbar_init(v_full(s), 1);
                mbar_init(v_empty(s), 1);
            }
            fence_mbar_init();
            pdl_wait();  // q/k/v may be the output of the kernel before this one
            mbar_arrive_expect_tx(q_full, QTILE);
            tma_load_4d(q_smem, &tmap_q, q_full, 0, mt * kAttnBlock, h, b);
            if (MODE == 1) {
                for (int j = 0; j < min(KVS, max_blk); ++j) {
                    tma_prefetch_l2_4d(&tmap_k, 0, j * kBlkN, hk, b);
                    tma_prefetch_l2_4d(&tmap_v, 0, j * kBlkN, hk, b);
                }
            }
            if (first_kv > 0) {  // K_0 right behind Q: the first Q·Kᵀ needs just these two
                mbar_arrive_expect_tx(k_full(0), KVB);
                tma_load_4d(k_smem, &tmap_k, k_full(0), 0, 0, hk, b);
            }
            for (int j = 0; j < first_kv; ++j) {
                if (j > 0) {
                    mbar_arrive_expect_tx(k_full(j), KVB);
                    tma_load_4d(k_smem + j * KVB, &tmap_k, k_full(j), 0, j * kBlkN, hk, b);
                }
                mbar_arrive_expect_tx(v_full(j), KVB);
                tma_load_4d(v_smem + j * KVB, &tmap_v, v_full(j), 0, j * kBlkN, hk, b);
            }
        }
    } else if (warp == 0) {
        if (lane == 0) mbar_init(o_final, 2);  // the last product, and the issuer itself, for s_expired
        if (lane < 2) {
            mbar_init(p_full(lane), 8);
            mbar_init(s_full(lane), 1);
            mbar_init(pv_done(lane), 1);
        }
        if (lane < 4) mbar_init(ep_bar(lane), 2);
        if (Cfg::kMaskRing && lane < 2) {
            mbar_init(m_full(lane), EDGE ? 128 : 64);  // the threads of the two loader warps: their copies (and their own stores)
            mbar_init(m_empty(lane), 8);
        }
        if (lane == 0) *abort_flag = 0;
        fence_mbar_init();
    } else if (warp == W0 + 1) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    // Launched with programmatic dependent launch: everything above (barriers, TMEM, descriptors)
    // may run while the previous kernel of the stream drains; nothing of global memory is touched
    // before this point.
    pdl_wait();
    if (MODE == 1) {
        // every thread stages its share of the mask row: clamped, in the log2 domain, -inf beyond N
        const float mlow = mask_lowest(p.mask_dtype);
        const int64_t moff = (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1];
        const int ncols = max_blk * kBlkN;
        float vals[Cfg::kMaskLoads];
#pragma unroll
        for (int e = 0; e < Cfg::kMaskLoads; ++e) {
            const int col = e * kThreads + (int)threadIdx.x;
            vals[e] = (col < p.N && col < ncols) ? mask_load(p.mask, moff + (int64_t)col * p.mask_strides[3], p.mask_dtype) : -INFINITY;
        }
#pragma unroll
        for (int e = 0; e < Cfg::kMaskLoads; ++e) {
            const int col = e * kThreads + (int)threadIdx.x;  // a warp covers half of one key block
            if (e * kThreads < ncols) {
                const bool inside = col < p.N && col < ncols;
                const float v = inside ? fmaxf(vals[e], mlow) * kLog2e : -INFINITY;
                if (col < ncols) mask_smem[col] = v;
                const bool live = __any_sync(0xffffffffu, inside && v > kSkipBelow);
                if (live && lane == 0) atomicOr(&act_bits[col >> 11], 1u << ((col >> 6) & 31));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // the key blocks this CTA visits: all of them, or (MODE 1) those with an unmasked key
    uint32_t act[4] = {0u, 0u, 0u, 0u};
    int visits = max_blk;
    if (MODE == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) act[i] = act_bits[i];
        // Causal rows see a prefix of the keys, which may consist of masked keys only even when the
        // row as a whole has live ones: no skipping then.
        if ((act[0] | act[1] | act[2] | act[3]) == 0u || p.is_causal) {
#pragma unroll
            for (int i = 0; i < 4; ++i) act[i] = 0xffffffffu;
        }
        visits = bits_count_below(act, max_blk);
    }
    auto next_blk = [&](int from) { return MODE == 1 ? bits_next(act, from) : from; };

    if (warp >= W0) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Shape::kRegsLow));
      if (warp == W0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            bool ok = true;
            int jb = next_blk(first_kv);
            for (int i = first_kv; i < visits && ok; ++i) {  // (MODE 0/2: the first ring was issued during set-up)
                const int s = i % KVS;
                const uint32_t ph = (uint32_t)((i / KVS) & 1);
                if (!mbar_wait(k_empty(s), ph ^ 1, abort_flag, 600)) { ok = false; break; }
                mbar_arrive_expect_tx(k_full(s), KVB);
                tma_load_4d(k_smem + s * KVB, &tmap_k, k_full(s), 0, jb * kBlkN, hk, b);
                if (!mbar_wait(v_empty(s), ph ^ 1, abort_flag, 601)) { ok = false; break; }
                mbar_arrive_expect_tx(v_full(s), KVB);
                tma_load_4d(v_smem + s * KVB, &tmap_v, v_full(s), 0, jb * kBlkN, hk, b);
                jb = next_blk(jb + 1);
            }
            if (!ok) {
                for (int i = 0; i < 64; ++i) __nanosleep(2000);
            }
        }
      } else if (warp == W0 + 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            s_expired = status_word();
            constexpr uint32_t idesc_qk = make_idesc_f16(Elem<T>::kIsBf16, 128, kBlkN, 0, 0);
            constexpr uint32_t idesc_pv = make_idesc_f16(Elem<T>::kIsBf16, 128, D, 0, 1);
            constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
            const uint32_t q_lo = (q_smem & 0x3FFFF) >> 4;
            const uint32_t k_lo = (k_smem & 0x3FFFF) >> 4;
            const uint32_t v_lo = (v_smem & 0x3FFFF) >> 4;
            auto desc = [&](uint32_t lo) { return ((uint64_t)desc_hi << 32) | (uint64_t)lo; };
            auto issue_qk = [&](int j) {  // S[j & 1] = Q · K_jᵀ
                const uint32_t b_lo = k_lo + (uint32_t)((j % KVS) * (KVB >> 4));
                const uint32_t d_tmem = tmem_base + (uint32_t)((j & 1) * kBlkN);
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    tc_mma_ss(d_tmem, desc(q_lo + (uint32_t)((ks * 32) >> 4)), desc(b_lo + (uint32_t)((ks * 32) >> 4)), idesc_qk,
                              ks > 0 ? 1u : 0u);
            };
            auto issue_pv = [&](int j) {  // O_a += P_j[:, 0:32] · V_j[0:32, :],  O_b += P_j[:, 32:64] · V_j[32:64, :]
                const uint32_t b_lo = v_lo + (uint32_t)((j % KVS) * (KVB >> 4));
                const uint32_t s_tmem = tmem_base + (uint32_t)((j & 1) * kBlkN);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {
                        tc_mma_ts(tmem_base + (uint32_t)(128 + hf * 64), s_tmem + (uint32_t)(hf * 32 + ks * 8),
                                  desc(b_lo + (uint32_t)((hf * 2 + ks) * (2048 >> 4))), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
                    }
                }
            };
            // j counts visited blocks (ring positions), not key-block numbers
            bool ok = mbar_wait(q_full, 0, abort_flag, 610);
            for (int jj = 0; jj < NB && jj < visits && ok; ++jj) {
                if (!mbar_wait(k_full(jj % KVS), (uint32_t)((jj / KVS) & 1), abort_flag, 611)) { ok = false; break; }
                tc_fence_after();
                issue_qk(jj);
                tc_commit(s_full(jj & 1));
                tc_commit(k_empty(jj % KVS));
            }
            for (int j = 0; j < visits && ok; ++j) {
                const int s = j % KVS;
                if (!mbar_wait(v_full(s), (uint32_t)((j / KVS) & 1), abort_flag, 612)) { ok = false; break; }
                const int j2 = j + NB;
                if (j2 < visits) {
                    if (!mbar_wait(k_full(j2 % KVS), (uint32_t)((j2 / KVS) & 1), abort_flag, 613)) { ok = false; break; }
                }
                if (!mbar_wait(p_full(j & 1), (uint32_t)((j >> 1) & 1), abort_flag, 614)) { ok = false; break; }
                tc_fence_after();
                issue_pv(j);
                tc_commit(pv_done(j & 1));
                if (j2 < visits) {
                    issue_qk(j2);  // into the slot that P_j has just been read from (in-order execution)
                    tc_commit(s_full(j & 1));
                }
                if (j + 1 == visits) {
                    mbar_arrive(o_final);
                    tc_commit(o_final);
                }
                tc_commit(v_empty(s));
                if (j2 < visits) tc_commit(k_empty(j2 % KVS));
            }
        }
      } else if (Cfg::kMaskRing && warp >= W0 + 2) {
        // ------------------------------------------------------------------ mask loaders (two warps)
        // Eight threads in a row read neighbouring chunks of one mask row. (Every softmax thread fetching its own
        // row touched 32 cache lines per instruction: a block with a mask took twice as long as one without.)
        // Thread (r0, ch) of 7 x 9 takes chunk ch of rows r0, r0 + 7, ...: pointers advance by a constant. Nothing outside
        // the mask, from its first value to its last, is read: whole chunks lie inside it where it begins and ends with
        // one, and else (EDGE) a copy ends with its row and the chunk in which the mask begins is taken value by value.
        // (EDGE copies are a little slower; rows read byte for byte, with their heads word by word, took 15.7 us at
        // [3, 12, 333, 64] where EDGE takes 12.0.)
        const int lt = (int)threadIdx.x - (W0 + 2) * 32;
        const int r0 = lt / 9, ch = lt % 9;
        const int rows = lt < 63 ? min(kAttnBlock, p.M - mt * kAttnBlock) : 0;
        const int64_t step = 14 * p.mask_strides[2];
        const uint8_t* base = reinterpret_cast<const uint8_t*>(p.mask) +
                              2 * ((int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1] + (int64_t)(mt * kAttnBlock + r0) * p.mask_strides[2]);
        const uint32_t dst0 = smem_u32(mask_ring) + (uint32_t)(r0 * Cfg::kMaskRowBytes + ch * 16);
        for (int j = 0; j < visits; ++j) {
            if (!mbar_wait(m_empty(j & 1), (uint32_t)(((j >> 1) & 1) ^ 1), abort_flag, 640)) break;
            const uint32_t dst = dst0 + (uint32_t)((j & 1) * Cfg::kMaskSlotBytes);
            const uint8_t* first = base + j * (kBlkN * 2);
            const int bytes = 2 * min(kBlkN, p.N - j * kBlkN) - ch * 16;  // of the row, from chunk ch of an aligned row on
            if (!EDGE) {
#pragma unroll
                for (int it = 0; it < (kAttnBlock + 6) / 7; ++it) {
                    const uint32_t lead = (uint32_t)(uintptr_t)first & 15u;
                    // a chunk is fetched if it holds a value of the row; what else it holds is not looked at
                    if (it * 7 + r0 < rows && (int)(0u - lead) < bytes)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)(it * 7 * Cfg::kMaskRowBytes)), "l"(first - lead + ch * 16) : "memory");
                    first += step;
                }
            } else if (j > 0 || p.mask_lead == 0) {
                const int len = 2 * min(kBlkN, p.N - j * kBlkN);
#pragma unroll
                for (int it = 0; it < (kAttnBlock + 6) / 7; ++it) {
                    const int lead = (int)((uintptr_t)first & 15u), n = mask_chunk_bytes(lead, ch, len);
                    if (it * 7 + r0 < rows && n > 0)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(it * 7 * Cfg::kMaskRowBytes)), "l"(first - lead + ch * 16), "r"(n) : "memory");
                    first += step;
                }
            } else {
                // rows that begin in the same chunk as the mask itself: value by value up to the next one
                const int len = 2 * min(kBlkN, p.N);
#pragma unroll 1
                for (int r = r0; r < rows; r += 7, first += step) {
                    const int lead = (int)((uintptr_t)first & 15u), n = mask_chunk_bytes(lead, ch, len);
                    const uint32_t to = dst + (uint32_t)((r - r0) * Cfg::kMaskRowBytes);
                    if (n > 0 && first - lead + ch * 16 >= reinterpret_cast<const uint8_t*>(p.mask))
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(first - lead + ch * 16), "r"(n) : "memory");
                    else
                        for (int e = lead; e < n; e += 2)
                            asm volatile("st.shared.u16 [%0], %1;" ::"r"(to + (uint32_t)e), "h"(__ldg(reinterpret_cast<const uint16_t*>(first - lead + e))) : "memory");
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(m_full(j & 1)) : "memory");
            if (EDGE) mbar_arrive(m_full(j & 1));  // for the values that the thread has stored itself
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
      }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Shape::kRegsHigh));
        // ------------------------------------------------------------------ softmax warps
        const int hf = (warp >> 2) & 1;  // which 32 key columns of every block
        const int q = warp & 3;          // TMEM lane quarter = 32 query rows
        // (always so; without the test the compiler arranges the key loop of MODE 1 otherwise: [2, 12, 8192, 64] 864 -> 923 us)
        if (visits > 0) {
            const int nb = visits;
            const int r_in_tile = q * 32 + lane;
            const int row = mt * kAttnBlock + r_in_tile;
            const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
            const uint32_t o_own = lane_addr + (uint32_t)(128 + hf * 64);
            const float c = p.scale_log2;
            const float mlow = mask_lowest(p.mask_dtype);
            const int64_t mask_row_off =
                (MODE >= 2 && p.mask != nullptr)
                    ? (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1] + (int64_t)min(row, p.M - 1) * p.mask_strides[2]
                    : 0;
            // where this row starts in its staged chunks, in elements
            const int mask_shift = (int)(((uintptr_t)p.mask + 2 * (uintptr_t)mask_row_off) >> 1) & 7;
            // MODE 0 and staged masks: scores stay in their own units, the exponent is (s - m) * c; else log2 domain
            const float unit = (MODE == 0 || MODE == 3) ? c : 1.0f;
            const float inv_scale = kLog2e / c;
            float m_ref = -INFINITY;
            float l = 0.f;
            bool ok = true;
            int jb = next_blk(0);  // key-block number of visit j
            for (int j = 0; j < nb; ++j, jb = next_blk(jb + 1)) {
                const int bf = j & 1;
                const uint32_t ph = (uint32_t)((j >> 1) & 1);
                const uint32_t s_addr = lane_addr + (uint32_t)(bf * kBlkN + hf * 32);
                if (!mbar_wait(s_full(bf), ph, abort_flag, 630)) { ok = false; break; }
                tc_fence_after();
                uint32_t sr[32];
                tmem_ld_32x32(s_addr, sr);
                tmem_ld_wait();

                const int col0 = jb * kBlkN + hf * 32;
                if (MODE == 1) {
                    const float4* ms = reinterpret_cast<const float4*>(mask_smem + col0);
#pragma unroll
                    for (int v4 = 0; v4 < 8; ++v4) {
                        const float4 a = ms[v4];
                        sr[v4 * 4 + 0] = __float_as_uint(fmaf(__uint_as_float(sr[v4 * 4 + 0]), c, a.x));
                        sr[v4 * 4 + 1] = __float_as_uint(fmaf(__uint_as_float(sr[v4 * 4 + 1]), c, a.y));
                        sr[v4 * 4 + 2] = __float_as_uint(fmaf(__uint_as_float(sr[v4 * 4 + 2]), c, a.z));
                        sr[v4 * 4 + 3] = __float_as_uint(fmaf(__uint_as_float(sr[v4 * 4 + 3]), c, a.w));
                    }
                } else if (MODE == 3) {
                    if (!mbar_wait(m_full(bf), ph, abort_flag, 641)) { ok = false; break; }
                    const uint8_t* src = mask_ring + bf * Cfg::kMaskSlotBytes + r_in_tile * Cfg::kMaskRowBytes + hf * 64;
                    add_staged_mask(p, src, mask_shift, inv_scale, sr);
                    add_staged_mask(p, src + 32, mask_shift, inv_scale, sr + 16);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(m_empty(bf));
                } else if (MODE == 2) {
                    if (p.mask == nullptr) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) sr[i] = __float_as_uint(__uint_as_float(sr[i]) * c);
                    } else {
#pragma unroll
                        for (int hc = 0; hc < 2; ++hc) {
                            const int colc = col0 + hc * 16;
                            float mvals[16];
                            mask_values(p, mask_row_off, colc, mvals);
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                uint32_t& sv = sr[hc * 16 + i];
                                sv = __float_as_uint(fmaf(fmaxf(mvals[i], mlow), kLog2e, __uint_as_float(sv) * c));
                            }
                        }
                    }
                }
                const bool causal_edge = p.is_causal && col0 + 31 > mt * kAttnBlock;
                if ((MODE != 1 && col0 + 32 > p.N) || causal_edge) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int col = col0 + i;
                        if (col >= p.N || (p.is_causal && col > row)) sr[i] = __float_as_uint(-INFINITY);
                    }
                }
                float m4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) m4[i] = fmaxf(__uint_as_float(sr[2 * i]), __uint_as_float(sr[2 * i + 1]));
#pragma unroll
                for (int i = 4; i < 16; ++i) m4[i & 3] = fmax3(m4[i & 3], __uint_as_float(sr[2 * i]), __uint_as_float(sr[2 * i + 1]));
                const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
                float m_new = fmaxf(m_ref, mx);
                if (m_new == -INFINITY) m_new = 0.f;
                const bool grow = (m_new - m_ref) * unit > kLazyThreshold;
                float alpha = 1.0f;
                if (grow) {
                    alpha = (m_ref == -INFINITY) ? 0.f : fast_exp2((m_ref - m_new) * unit);
                    m_ref = m_new;
                    l *= alpha;
                }
                if (j > 0 && __any_sync(0xffffffffu, grow)) {
                    // This half's accumulator must be quiescent before it is rescaled: P·V of block j-1
                    // complete, the ((j-1)>>1)-th completion of the barrier of parity (j-1)&1. S_j
                    // being ready implies P·V of block j-2 (hence j-3) complete, i.e. every earlier
                    // completion of this barrier, so the parity cannot be mistaken for an older phase.
                    if (!mbar_wait(pv_done((j - 1) & 1), (uint32_t)(((j - 1) >> 1) & 1), abort_flag, 650)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int dch = 0; dch < D / 16; ++dch) {
                        uint32_t orr[16];
                        tmem_ld_32x16(o_own + dch * 16, orr);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * alpha);
                        tmem_st_32x16(o_own + dch * 16, orr);
                    }
                }
                const float neg_ref = -m_ref * unit;
                const float2 unit2 = make_float2(unit, unit);
                const float2 neg2 = make_float2(neg_ref, neg_ref);
                float2 lp[2] = {{0.f, 0.f}, {0.f, 0.f}};
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 a = __ffma2_rn(make_float2(__uint_as_float(sr[2 * i]), __uint_as_float(sr[2 * i + 1])), unit2, neg2);
                    float2 e;
                    // (all on the special-function unit: with 16 softmax warps the issue slots are what is short here,
                    // and a quarter of the pairs on the FMA pipe was 3 % slower at [8, 12, 4096, 64])
                    e.x = fast_exp2(a.x);
                    e.y = fast_exp2(a.y);
                    lp[i & 1] = __fadd2_rn(lp[i & 1], e);
                    pk[i] = Elem<T>::pack2(e.x, e.y);
                }
                tmem_st_32x16(s_addr, pk);
                {
                    const float2 st = __fadd2_rn(lp[0], lp[1]);
                    l += st.x + st.y;
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full(bf));
            }
            // The key loop is over: a dependent kernel's CTAs may take the slots that free up from
            // here on and set themselves up (they read nothing before this grid has completed). The
            // first caller in a CTA counts; no thread calls it earlier, so a dependent never
            // competes with CTAs of this launch that have not started yet.
            pdl_launch_dependents();
            // ---- epilogue: merge the two halves of every row, O / l -> global
            // (m, l) of this half to the partner warp (same rows, other half) through shared memory
            // a half that never saw a finite score (all of its columns beyond N) must not set the scale
            const float m_own = (l > 0.f) ? m_ref * unit : -INFINITY;
            xch[hf * kAttnBlock + r_in_tile] = make_float2(m_own, l);
            __syncwarp();
            if (lane == 0) mbar_arrive(ep_bar(q));
            if (ok && mbar_wait(ep_bar(q), 0, abort_flag, 660) && mbar_wait(o_final, 0, abort_flag, 670)) {
                tc_fence_after();
                const int m_end = s_expired == 0 ? p.M : 0;  // rows that may be stored
                const float2 other = xch[(hf ^ 1) * kAttnBlock + r_in_tile];
                float m_all = fmaxf(m_own, other.x);
                if (m_all == -INFINITY) m_all = 0.f;
                const float w_own = fast_exp2(m_own - m_all), w_oth = fast_exp2(other.x - m_all);
                const float inv_l = 1.0f / (w_own * l + w_oth * other.y);
                const float wa = (hf == 0 ? w_own : w_oth) * inv_l;  // weight of O_a
                const float wb = (hf == 0 ? w_oth : w_own) * inv_l;  // weight of O_b
                // this warp writes output columns [32·hf, 32·hf + 32) of its 32 rows
                uint32_t oa[32], ob[32];
                tmem_ld_32x32(lane_addr + (uint32_t)(128 + hf * 32), oa);
                tmem_ld_32x32(lane_addr + (uint32_t)(192 + hf * 32), ob);
                tmem_ld_wait();
                T* o_row = reinterpret_cast<T*>(p.o) + (int64_t)b * p.o_strides[0] + (int64_t)h * p.o_strides[1] +
                           (int64_t)row * p.o_strides[2];
                const bool vec = p.o_strides[3] == 1 && ((((uintptr_t)o_row) & 15) == 0);
                if (row < m_end) {
                    float val[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) val[i] = fmaf(__uint_as_float(oa[i]), wa, __uint_as_float(ob[i]) * wb);
                    if (hf * 32 + 32 <= p.d_out) attn_store_32<T, false>(o_row, hf * 32, p.o_strides[3], vec, val, p.d_out);
                    else attn_store_32<T, true>(o_row, hf * 32, p.o_strides[3], vec, val, p.d_out);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == W0 + 1) {
        __syncwarp();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// Whether the rows of a per-row mask are staged: 16-bit values side by side, the first one at the lowest address.
static bool mask_is_staged(const kb_attn_params& p) {
    return p.mask != nullptr && p.mask_dtype != KB_F32 && p.mask_strides[3] == 1 && p.sm_scale > 0.f && p.mask_strides[0] >= 0 &&
           p.mask_strides[1] >= 0 && p.mask_strides[2] >= 0;
}
// Whether a mask whose rows are staged begins or ends inside a 16-byte chunk.
static bool mask_has_edges(const kb_attn_params& p) {
    const int64_t last = (p.B - 1) * p.mask_strides[0] + (p.H - 1) * p.mask_strides[1] + (p.M - 1) * p.mask_strides[2] + p.N;  // values from the first on
    return ((((uintptr_t)p.mask) | ((uintptr_t)p.mask + 2 * (uintptr_t)last)) & 15) != 0;
}

template <typename T, int MODE, bool EDGE = false>
static int launch_attention_split_tm(const kb_attn_params& p, cudaStream_t stream) {
    using Cfg = AttnSplitCfg<MODE>;
    using Shape = SplitShape;
    CUtensorMap tq, tk, tv;
    const int64_t kv_group = p.kv_group > 1 ? p.kv_group : 1;
    if (p.H % kv_group != 0) return KB_ERR_BAD_ARG;
    auto enc = [&](CUtensorMap* out, const void* ptr, int64_t rows, const int64_t* st, uint32_t box_rows, int64_t heads) -> int {
        if (st[3] != 1) return KB_ERR_UNSUPPORTED;
        const uint64_t dims[4] = {(uint64_t)p.D, (uint64_t)rows, (uint64_t)heads, (uint64_t)p.B};  // the box reaches to 64: zero fill
        auto fix = [](int64_t extent, int64_t stride) -> uint64_t { return (extent == 1) ? 16u : (uint64_t)stride * 2u; };
        const uint64_t strides[4] = {0, fix(rows, st[2]), fix(heads, st[1]), fix(p.B, st[0])};
        const uint32_t box[4] = {64, box_rows, 1, 1};
        return encode_tmap_16bit(out, ptr, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    };
    int st = enc(&tq, p.q, p.M, p.q_strides, kAttnBlock, p.H);
    if (st != KB_OK) return st;
    st = enc(&tk, p.k, p.N, p.k_strides, kBlkN, p.H / kv_group);
    if (st != KB_OK) return st;
    st = enc(&tv, p.v, p.N, p.v_strides, kBlkN, p.H / kv_group);
    if (st != KB_OK) return st;

    AttnDev d;
    d.o_bulk = 0;
    d.o = p.o;
    d.mask = p.mask;
    for (int i = 0; i < 4; ++i) {
        d.o_strides[i] = p.o_strides[i];
        d.mask_strides[i] = p.mask ? p.mask_strides[i] : 0;
    }
    d.B = (int)p.B; d.H = (int)p.H; d.M = (int)p.M; d.N = (int)p.N;
    d.scale_log2 = p.sm_scale * kLog2e;
    d.is_causal = p.is_causal ? 1 : 0;
    d.mask_dtype = p.mask ? p.mask_dtype : KB_F32;
    d.mask_vec = 0;
    if (p.mask != nullptr && p.mask_strides[3] == 1 && (((uintptr_t)p.mask) & 15) == 0) {
        const int64_t per16 = (p.mask_dtype == KB_F32) ? 4 : 8;
        d.mask_vec = (p.mask_strides[0] % per16 == 0 && p.mask_strides[1] % per16 == 0 && p.mask_strides[2] % per16 == 0) ? 1 : 0;
    }
    d.mask_lead = p.mask != nullptr ? (int)((uintptr_t)p.mask & 15) : 0;
    const int num_m_tiles = (int)((p.M + kAttnBlock - 1) / kAttnBlock);
    d.num_pairs = num_m_tiles;  // work items per (batch, head)
    d.head_group = attn_head_group(p.B * p.H, p.N, p.D);
    d.kv_group = (int)kv_group;
    d.d_out = (int)p.D;
    static std::atomic<int> regs_ok{0};  // 0 = not checked, 1 = usable, -1 = register allocation does not fit
    if (regs_ok == 0) {
        // setmaxnreg.inc blocks until the CTA's pool holds the registers: refuse to launch a build
        // whose launch allocation is smaller than the redistribution assumes.
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, attention_split_kernel<T, MODE, EDGE>) != cudaSuccess) return KB_ERR_LAUNCH;
        regs_ok = (fa.numRegs < Shape::kRegsLaunch) ? -1 : 1;
    }
    if (regs_ok < 0) return KB_ERR_UNSUPPORTED;
    static PerDeviceOnce attr_once;
    if (!attr_once.run([] {
            return cudaFuncSetAttribute(attention_split_kernel<T, MODE, EDGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemMax) == cudaSuccess;
        }))
        return KB_ERR_LAUNCH;
    const int64_t grid = (int64_t)d.num_pairs * p.B * p.H;
    if (grid > 0x7fffffff) return KB_ERR_UNSUPPORTED;
    const int num_n_blocks = (int)((p.N + kBlkN - 1) / kBlkN);
    const size_t smem_bytes = (size_t)Cfg::kSmemBase + (MODE == 1 ? (size_t)num_n_blocks * kBlkN * 4 : 0);
    if (launch_pdl(attention_split_kernel<T, MODE, EDGE>, (unsigned)grid, (unsigned)Shape::kThreads, smem_bytes, stream, tq,
                   tk, tv, d) != cudaSuccess)
        return KB_ERR_LAUNCH;
    return cudaGetLastError() == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

// The persistent form of this kernel (attention_persist.cuh) takes the launches it is made for.
static bool attention_persist_applicable(const kb_attn_params& p, int mode);
template <typename T, int MODE>
static int launch_attention_persist_tm(const kb_attn_params& p, cudaStream_t stream, unsigned int* queue);

template <typename T>
static int launch_attention_split_t(const kb_attn_params& p, cudaStream_t stream) {
    const int mode = (p.mask == nullptr && p.sm_scale > 0.f) ? 0
                     : (p.mask != nullptr && p.mask_strides[2] == 0 && p.N <= AttnSplitCfg<1>::kMaskMaxN) ? 1
                     : (p.mask_strides[2] != 0 && mask_is_staged(p)) ? 3 : 2;
    unsigned int* queue = g_split_tiles == 0 && attention_persist_applicable(p, mode) ? attention_queue_slot(stream) : nullptr;
    if (queue != nullptr) {
        if (mode == 0) return launch_attention_persist_tm<T, 0>(p, stream, queue);
        if (mode == 1) return launch_attention_persist_tm<T, 1>(p, stream, queue);
        return launch_attention_persist_tm<T, 2>(p, stream, queue);
    }
    if (mode == 0) return launch_attention_split_tm<T, 0>(p, stream);
    if (mode == 1) return launch_attention_split_tm<T, 1>(p, stream);
    if (mode == 2) return launch_attention_split_tm<T, 2>(p, stream);
    return mask_has_edges(p) ? launch_attention_split_tm<T, 3, true>(p, stream) : launch_attention_split_tm<T, 3>(p, stream);
}

static int launch_attention_split(const kb_attn_params& p, cudaStream_t stream) {
    if (p.D > 64 || p.D % 8 != 0) return KB_ERR_UNSUPPORTED;
    if (p.dtype == KB_F16) return launch_attention_split_t<__half>(p, stream);
    if (p.dtype == KB_BF16) return launch_attention_split_t<__nv_bfloat16>(p, stream);
    return KB_ERR_UNSUPPORTED;
}

}  // namespace kb
