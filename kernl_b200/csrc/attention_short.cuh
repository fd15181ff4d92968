// Fused attention forward for short key ranges, on mma.sync: O = softmax(sm_scale·Q·Kᵀ + mask [causal]) · V.
//
// Bound: fixed costs and latencies. A query tile that meets two or three key blocks spends most of its
// time in the tcgen05 kernels outside the products — barriers and tensor memory set up and handed over,
// scores travelling TMEM -> registers -> TMEM, an epilogue that waits for the last product: 4-6 us per
// tile against about 1 us per key block. Here scores, probabilities and the accumulator never leave
// the registers of the warp that owns the rows, a CTA is 64 query rows on four warps with 41 KB of
// shared memory (D = 64), four to five CTAs hide each other's latencies on an SM, and a tile costs little more
// than its loads. The price is the rate of the products (mma.sync is about a third of tcgen05), so long
// key ranges stay with the other kernels; attention_short_applicable() draws the line.
//
//   warp w      query rows [16 w, 16 w + 16) of the tile; q in registers as mma.sync.m16n8k16 operands
//   per block   64 keys: K and V through two buffers of asynchronous 16-byte copies (rows padded to an
//               odd number of 16-byte chunks: ldmatrix without bank conflicts), one barrier per block
//   epilogue    rows through shared memory, stored as whole 16-byte pieces
//
// Same semantics as the other kernels (attention.cuh): scale before mask, masks clamped to the lowest
// finite value of their type, causal = keep col <= row, P rounded to the input type, fp32 statistics;
// key blocks whose row-broadcast mask is minus infinity throughout are not visited (attention_split.cuh).
#pragma once
#include "attention_split.cuh"

namespace kb {

constexpr int kShortThreads = 128;
constexpr int kShortRows = 64;      // query rows per CTA
constexpr int kShortKeys = 64;      // keys per block
constexpr int kShortMaskCols = 4096;  // longest row-broadcast mask kept in shared memory

struct AttnShortDev {
    AttnDev a;
    const void* q; const void* k; const void* v;
    int64_t q_strides[3], k_strides[3], v_strides[3];
    int trigger_early;  // the whole launch is resident at once: a dependent launch takes nothing from it
};

template <int D>
struct ShortCfg {
    static constexpr int kChunks = D / 8;                  // 16-byte chunks of a row
    static constexpr int kRowBytes = (kChunks | 1) * 16;   // odd number of chunks (D / 8 is even)
    static constexpr int kTileBytes = 64 * kRowBytes;      // q, or a K or V block
    static constexpr int kSmemBytes = 5 * kTileBytes;      // q + two buffers of K and V; MODE 1: + the mask row
    static constexpr int ctas(int mode) { return D == 64 ? (mode == 2 ? 3 : 4) : 2; }
};

template <typename T, int D, int MODE>
__global__ void __launch_bounds__(kShortThreads, ShortCfg<D>::ctas(MODE))
attention_short_kernel(const AttnShortDev s) {
    using Cfg = ShortCfg<D>;
    constexpr int CH = Cfg::kChunks, ROWB = Cfg::kRowBytes;
    const AttnDev& p = s.a;
    extern __shared__ __align__(128) uint8_t short_smem[];
    __shared__ uint32_t live_bits[4];
    float* mask_s = reinterpret_cast<float*>(short_smem + Cfg::kSmemBytes);
    const uint32_t q_s = smem_u32(short_smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;

    const int tiles = (p.M + kShortRows - 1) / kShortRows, BH = p.B * p.H;
    // head-major, so that the tiles of a head share its K/V in L2; causal: the late, longer tiles first
    const int bh = p.is_causal ? (int)blockIdx.x % BH : (int)blockIdx.x / tiles;
    const int tile = p.is_causal ? tiles - 1 - (int)blockIdx.x / BH : (int)blockIdx.x % tiles;
    const int b = bh / p.H, h = bh % p.H, hk = h / p.kv_group;
    const int row0 = tile * kShortRows;
    const int all_blocks = (p.N + kShortKeys - 1) / kShortKeys;
    const int n_blocks = p.is_causal ? min(all_blocks, tile + 1) : all_blocks;
    const T* qp = reinterpret_cast<const T*>(s.q) + (int64_t)b * s.q_strides[0] + (int64_t)h * s.q_strides[1];
    const T* kp = reinterpret_cast<const T*>(s.k) + (int64_t)b * s.k_strides[0] + (int64_t)hk * s.k_strides[1];
    const T* vp = reinterpret_cast<const T*>(s.v) + (int64_t)b * s.v_strides[0] + (int64_t)hk * s.v_strides[1];
    // 64 rows from `r0` on; rows beyond `n` and columns beyond the caller's head dimension are zero-filled
    auto load_rows = [&](uint32_t dst, const T* base, int64_t stride, int r0, int n) {
#pragma unroll
        for (int it = 0; it < 64 * CH / kShortThreads; ++it) {
            const int idx = it * kShortThreads + tid, r = idx / CH, j = idx % CH;
            const bool in = r0 + r < n && j * 8 < p.d_out;
            const T* src = in ? base + (int64_t)(r0 + r) * stride + j * 8 : base;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(r * ROWB + j * 16)), "l"(src), "r"(in ? 16 : 0) : "memory");
        }
    };
    auto load_block = [&](int i, int jb) {  // key block jb, the i-th that is visited
        const uint32_t dst = q_s + (uint32_t)((1 + 2 * (i & 1)) * Cfg::kTileBytes);
        load_rows(dst, kp, s.k_strides[2], jb * kShortKeys, p.N);
        load_rows(dst + Cfg::kTileBytes, vp, s.v_strides[2], jb * kShortKeys, p.N);
    };

    if (MODE == 1 && tid < 4) live_bits[tid] = 0u;
    pdl_wait();
    if (s.trigger_early) pdl_launch_dependents();
    // set by a wait that expired in an earlier launch: nothing is stored then (looked at in the end, off the path of the loads)
    const int skip = status_word();
    load_rows(q_s, qp, s.q_strides[2], row0, p.M);
    asm volatile("cp.async.commit_group;" ::: "memory");
    uint32_t act[4] = {0u, 0u, 0u, 0u};
    int nb = n_blocks;
    if (MODE == 1) {
        __syncthreads();
        const float mlow = mask_lowest(p.mask_dtype);
        const int64_t moff = (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1];
        for (int c0 = 0; c0 < n_blocks * kShortKeys; c0 += kShortThreads) {
            const int col = c0 + tid;
            const bool inside = col < p.N && col < n_blocks * kShortKeys;
            const float v = inside ? fmaxf(mask_load(p.mask, moff + (int64_t)col * p.mask_strides[3], p.mask_dtype), mlow) * kLog2e : -INFINITY;
            if (col < n_blocks * kShortKeys) mask_s[col] = v;
            if (__any_sync(0xffffffffu, inside && v > kSkipBelow) && lane == 0) atomicOr(&live_bits[col >> 11], 1u << ((col >> 6) & 31));
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) act[i] = live_bits[i];
        // nothing is skipped when everything is masked, nor for causal rows, which may see masked keys only
        if ((act[0] | act[1] | act[2] | act[3]) == 0u || p.is_causal) {
#pragma unroll
            for (int i = 0; i < 4; ++i) act[i] = 0xffffffffu;
        }
        nb = bits_count_below(act, n_blocks);
    }
    auto next_blk = [&](int from) { return MODE == 1 ? bits_next(act, from) : from; };
    int jb = next_blk(0);
    load_block(0, jb);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    uint32_t qf[D / 16][4];
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
        ldmatrix_x4(q_s + (uint32_t)((warp * 16 + (lane & 15)) * ROWB + (ks * 2 + (lane >> 4)) * 16), qf[ks]);

    float o[D / 8][4];
#pragma unroll
    for (int nt = 0; nt < D / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[nt][e] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    const float scale = p.scale_log2, unit = MODE == 0 ? scale : 1.0f;  // MODE 0 takes the maximum of raw scores
    const float mlow = mask_lowest(p.mask_dtype);
    const int row[2] = {row0 + warp * 16 + g, row0 + warp * 16 + g + 8};
    int64_t mask_row[2] = {0, 0};
    if (MODE == 2 && p.mask != nullptr) {
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
            mask_row[hh] = (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1] + (int64_t)min(row[hh], p.M - 1) * p.mask_strides[2];
    }

    for (int i = 0; i < nb; ++i) {
        const int key0 = jb * kShortKeys;
        jb = next_blk(jb + 1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the block has arrived for everybody, and everybody is done with the other buffer
        if (i + 1 < nb) load_block(i + 1, jb);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const uint32_t k_s = q_s + (uint32_t)((1 + 2 * (i & 1)) * Cfg::kTileBytes), v_s = k_s + Cfg::kTileBytes;
        float x[8][4];  // scores: tile nt = keys key0 + 8 nt + {2c, 2c + 1}, rows g (0, 1) and g + 8 (2, 3)
        if (MODE == 2 && p.mask != nullptr) {  // requested ahead of the products
            if (p.mask_vec == 2 && key0 + kShortKeys <= p.N) {  // 16-bit pairs
#pragma unroll
                for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint16_t*>(p.mask) + mask_row[hh] + key0 + nt * 8 + 2 * c));
                        const float2 f = p.mask_dtype == KB_F16 ? Elem<__half>::unpack2(w) : Elem<__nv_bfloat16>::unpack2(w);
                        x[nt][2 * hh] = f.x;
                        x[nt][2 * hh + 1] = f.y;
                    }
            } else {
                auto grab = [&](const auto* base) {  // all loads before the first conversion
                    auto raw = [&](int nt, int e) {
                        const int key = key0 + nt * 8 + 2 * c + (e & 1);
                        return key < p.N ? __ldg(base + mask_row[e >> 1] + (int64_t)key * p.mask_strides[3]) : decltype(__ldg(base))(0.f);
                    };
                    decltype(__ldg(base)) v[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = raw(i >> 2, i & 3);
#pragma unroll
                    for (int i = 0; i < 32; ++i) x[i >> 2][i & 3] = (float)v[i];
                };
                if (p.mask_dtype == KB_F16) grab(reinterpret_cast<const __half*>(p.mask));
                else if (p.mask_dtype == KB_BF16) grab(reinterpret_cast<const __nv_bfloat16*>(p.mask));
                else grab(reinterpret_cast<const float*>(p.mask));
            }
        }
        float sc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; nt += 2) {
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[nt][e] = sc[nt + 1][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                uint32_t kf[4];  // (tile nt: d lo, d hi), (tile nt + 1: d lo, d hi)
                ldmatrix_x4(k_s + (uint32_t)((nt * 8 + (lane & 7) + (lane >> 4) * 8) * ROWB + (ks * 2 + ((lane >> 3) & 1)) * 16), kf);
                mma_16816<T>(sc[nt], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], kf[0], kf[1]);
                mma_16816<T>(sc[nt + 1], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], kf[2], kf[3]);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            if (MODE == 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) x[nt][e] = sc[nt][e];
            } else if (MODE == 1) {
                const float2 mk = *reinterpret_cast<const float2*>(mask_s + key0 + nt * 8 + 2 * c);
#pragma unroll
                for (int e = 0; e < 4; ++e) x[nt][e] = fmaf(sc[nt][e], scale, (e & 1) ? mk.y : mk.x);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    x[nt][e] = p.mask != nullptr ? fmaf(fmaxf(x[nt][e], mlow), kLog2e, sc[nt][e] * scale) : sc[nt][e] * scale;
            }
        }
        if ((MODE != 1 && key0 + kShortKeys > p.N) || (p.is_causal && key0 + kShortKeys - 1 > row0 + warp * 16)) {
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int key = key0 + nt * 8 + 2 * c + (e & 1);
                    if (key >= p.N || (p.is_causal && key > row[e >> 1])) x[nt][e] = -INFINITY;
                }
        }
        float alpha[2], neg[2];
        bool moved = false;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            float mx = fmaxf(x[0][2 * hh], x[0][2 * hh + 1]);
#pragma unroll
            for (int nt = 1; nt < 8; ++nt) mx = fmax3(mx, x[nt][2 * hh], x[nt][2 * hh + 1]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            float m_new = fmaxf(m_run[hh], mx);
            if (m_new == -INFINITY) m_new = 0.f;
            alpha[hh] = m_run[hh] == -INFINITY ? 0.f : fast_exp2((m_run[hh] - m_new) * unit);
            moved |= m_new != m_run[hh];
            m_run[hh] = m_new;
            neg[hh] = -m_new * unit;
        }
        if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) l_run[hh] *= alpha[hh];
#pragma unroll
            for (int nt = 0; nt < D / 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[nt][e] *= alpha[e >> 1];
        }
        uint32_t pf[8][2];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const float2 a = __ffma2_rn(make_float2(x[nt][2 * hh], x[nt][2 * hh + 1]), make_float2(unit, unit), make_float2(neg[hh], neg[hh]));
                const float e0 = fast_exp2(a.x), e1 = fast_exp2(a.y);
                l_run[hh] += e0 + e1;
                pf[nt][hh] = Elem<T>::pack2(e0, e1);
            }
#pragma unroll
        for (int kb = 0; kb < kShortKeys / 16; ++kb)
#pragma unroll
            for (int nt = 0; nt < D / 8; nt += 2) {
                uint32_t vf[4];
                ldmatrix_x4_trans(v_s + (uint32_t)((kb * 16 + (lane & 15)) * ROWB + (nt + (lane >> 4)) * 16), vf);
                mma_16816<T>(o[nt], pf[2 * kb][0], pf[2 * kb][1], pf[2 * kb + 1][0], pf[2 * kb + 1][1], vf[0], vf[1]);
                mma_16816<T>(o[nt + 1], pf[2 * kb][0], pf[2 * kb][1], pf[2 * kb + 1][0], pf[2 * kb + 1][1], vf[2], vf[3]);
            }
    }
    if (!s.trigger_early) pdl_launch_dependents();
    // rows of a warp are its own: q is in registers, so its part of the q tile takes the result
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        float l = l_run[hh];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        const float inv = 1.0f / l;
#pragma unroll
        for (int nt = 0; nt < D / 8; ++nt)
            *reinterpret_cast<uint32_t*>(short_smem + (warp * 16 + g + 8 * hh) * ROWB + nt * 16 + c * 4) =
                Elem<T>::pack2(o[nt][2 * hh] * inv, o[nt][2 * hh + 1] * inv);
    }
    __syncwarp();
    T* op = reinterpret_cast<T*>(p.o) + (int64_t)b * p.o_strides[0] + (int64_t)h * p.o_strides[1];
#pragma unroll
    for (int it = 0; it < 16 * CH / 32; ++it) {
        const int idx = it * 32 + lane, r = warp * 16 + idx / CH, j = idx % CH;
        if (skip == 0 && row0 + r < p.M && j * 8 < p.d_out)
            *reinterpret_cast<uint4*>(op + (int64_t)(row0 + r) * p.o_strides[2] + j * 8) = *reinterpret_cast<const uint4*>(short_smem + r * ROWB + j * 16);
    }
}

static int g_attn_short = -1;  // test hook: -1 = the rule below, 0 = never, 1 = wherever the layout allows

static bool attention_short_layout(const kb_attn_params& p) {
    auto rows_ok = [](const void* base, const int64_t* st) {
        return st[3] == 1 && st[0] % 8 == 0 && st[1] % 8 == 0 && st[2] % 8 == 0 && (((uintptr_t)base) & 15) == 0;
    };
    const bool row_mask = p.mask != nullptr && p.mask_strides[2] == 0;
    return p.D % 8 == 0 && p.D <= 128 && rows_ok(p.q, p.q_strides) && rows_ok(p.k, p.k_strides) && rows_ok(p.v, p.v_strides) &&
           rows_ok(p.o, p.o_strides) && (!row_mask || p.N <= kShortMaskCols);
}

// Which kernel is faster, from times measured over 16 to 800 keys, 1 to 200 sequences of 12 and 16 heads (ns).
// A launch takes the latency of one tile (a fixed part and one per key block) and, for every tile beyond
// one per SM, what a tile costs when the GPU is full (the same two parts). Per tile of 64 rows, this
// kernel: 3.5 + 4 per 64-key block (D = 64), 7 + 8 (80), 6 + 12 (128). Per tile of 128 rows, the kernels
// for D = 64: 8 + 4.3 per block, with a row mask 17.5 + 4.3, with a full mask 11 + 7. Per pair of tiles of
// 128 rows, attention.cuh: 57 (one tile: 35) + 13 per 128-key block, more with masks, 28 (12) + 13 without a mask, where
// its CTAs stay ([64, 32, 130, 80] causal 97 us, 117 here).
static bool attention_short_applicable(const kb_attn_params& p) {
    if (g_attn_short == 0 || !attention_short_layout(p)) return false;
    if (g_attn_short == 1) return true;
    if (g_split_tiles != 0 || g_attn_persistent != -1) return false;  // a test asks for one of those kernels
    const double sms = sm_count();
    const double bh = (double)p.B * (double)p.H;
    const bool row_mask = p.mask != nullptr && p.mask_strides[2] == 0, full_mask = p.mask != nullptr && !row_mask;
    const double blocks = (double)((p.N + 63) / 64);
    // blocks that are multiplied on average: half of a causal square; two thirds behind a padding mask
    const double live = p.is_causal ? (blocks + 1) / 2 : row_mask && blocks > 1 ? 0.33 + 0.67 * blocks : blocks;
    auto estimate = [&](double tiles, double latency, double per_tile) { return latency + (tiles > sms ? (tiles - sms) * per_tile : 0.0); };
    const double tiles64 = bh * (double)((p.M + 63) / 64), tiles128 = bh * (double)((p.M + 127) / 128);
    const double fa = full_mask ? 2.5 : 0.0, fb = full_mask ? (p.D <= 64 ? 1.5 : 1.3) : 1.0;  // a full mask is read value by value here
    if (p.D <= 64) {
        // where the persistent kernel runs, the two are within a few per cent of each other except for one key block
        if (tiles128 > 2 * sms && p.N > 64) return false;
        const double mine = estimate(tiles64, 2000.0 + 1000.0 * (full_mask ? 1.7 : 1.0) * live, 3.5 + fa + 4.0 * fb * live);
        const double other = estimate(tiles128, 2600.0 + (row_mask ? 2200.0 : 0.0) + (full_mask ? 1500.0 : 720.0) * live,
                                      (row_mask ? 17.5 : full_mask ? 11.0 : 8.0) + (full_mask ? 7.0 : 4.3) * live);
        return mine < other;
    }
    const bool d80 = p.D <= 80;
    // a causal launch takes as long as its last tile, which meets all blocks; from a tile per SM on, two share an SM
    const double lat = 2300.0 + (d80 ? 1080.0 : 1650.0) * fb * (p.is_causal ? blocks : live);
    const double spread = estimate(tiles64, lat, (d80 ? 7.0 : 6.0) + 2 * fa + (d80 ? 8.0 : 12.0) * fb * live);
    const double mine = tiles64 > sms && spread < 1.45 * lat ? 1.45 * lat : spread;
    const double pairs = bh * (double)((p.M + 255) / 256), b128 = (double)((p.N + 127) / 128);
    const double live128 = p.is_causal ? (b128 + 1) / 2 : row_mask && b128 > 1 ? 0.33 + 0.67 * b128 : b128;
    const bool ragged = full_mask && (p.mask_strides[2] % 8 != 0 || p.mask_strides[3] != 1);
    const double slow = ragged ? 2.6 : full_mask ? 1.8 : row_mask ? 1.15 : 1.0;  // masks cost that kernel's softmax warps
    const bool stays = p.mask == nullptr && p.sm_scale > 0.f;  // its CTAs take several pairs each
    const double per_pair = stays ? (p.M > 128 ? 28.0 : 12.0) : (p.M > 128 ? 57.0 : 35.0) * (full_mask ? 1.5 : 1.0);
    const double other = estimate(pairs, (3000.0 + 2950.0 * live128) * slow, per_pair + 13.0 * live128 * slow);
    return mine < other;
}

template <typename T, int D, int MODE>
static int launch_attention_short_t(const kb_attn_params& p, cudaStream_t stream) {
    using Cfg = ShortCfg<D>;
    const int tiles = (int)((p.M + kShortRows - 1) / kShortRows);
    const int64_t grid = (int64_t)tiles * p.B * p.H;
    if (grid > 0x7fffffff) return KB_ERR_UNSUPPORTED;
    AttnShortDev s = {};
    s.q = p.q; s.k = p.k; s.v = p.v;
    for (int i = 0; i < 3; ++i) {
        s.q_strides[i] = p.q_strides[i];
        s.k_strides[i] = p.k_strides[i];
        s.v_strides[i] = p.v_strides[i];
    }
    AttnDev& d = s.a;
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
    // 2: rows of a per-row mask can be read as pairs of 16-bit values
    d.mask_vec = (p.mask != nullptr && p.mask_dtype != KB_F32 && p.mask_strides[3] == 1 && (((uintptr_t)p.mask) & 3) == 0 && p.mask_strides[0] % 2 == 0 &&
                  p.mask_strides[1] % 2 == 0 && p.mask_strides[2] % 2 == 0) ? 2 : 0;
    d.kv_group = p.kv_group > 1 ? (int)p.kv_group : 1;
    if (p.H % d.kv_group != 0) return KB_ERR_BAD_ARG;
    d.d_out = (int)p.D;
    s.trigger_early = grid <= (int64_t)sm_count() * Cfg::ctas(MODE) ? 1 : 0;
    static PerDeviceOnce attr_once;
    if (!attr_once.run([] {
            return cudaFuncSetAttribute(attention_short_kernel<T, D, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        Cfg::kSmemBytes + (MODE == 1 ? kShortMaskCols * 4 : 0)) == cudaSuccess;
        }))
        return KB_ERR_LAUNCH;
    const size_t smem = (size_t)Cfg::kSmemBytes + (MODE == 1 ? (size_t)((p.N + 63) / 64) * 64 * 4 : 0);
    if (launch_pdl(attention_short_kernel<T, D, MODE>, (unsigned)grid, kShortThreads, smem, stream, s) != cudaSuccess) return KB_ERR_LAUNCH;
    return cudaGetLastError() == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

template <typename T, int D>
static int launch_attention_short_d(const kb_attn_params& p, cudaStream_t stream) {
    if (p.mask == nullptr && p.sm_scale > 0.f) return launch_attention_short_t<T, D, 0>(p, stream);
    if (p.mask != nullptr && p.mask_strides[2] == 0) return launch_attention_short_t<T, D, 1>(p, stream);
    return launch_attention_short_t<T, D, 2>(p, stream);
}

static int launch_attention_short(const kb_attn_params& p, cudaStream_t stream) {
    if (p.dtype == KB_F16)
        return p.D <= 64 ? launch_attention_short_d<__half, 64>(p, stream) : p.D <= 80 ? launch_attention_short_d<__half, 80>(p, stream)
                                                                                      : launch_attention_short_d<__half, 128>(p, stream);
    return p.D <= 64 ? launch_attention_short_d<__nv_bfloat16, 64>(p, stream) : p.D <= 80 ? launch_attention_short_d<__nv_bfloat16, 80>(p, stream)
                                                                                         : launch_attention_short_d<__nv_bfloat16, 128>(p, stream);
}

// The fused-attention entry: short key ranges -> the kernel above; head dimensions up to 64 -> the split-row
// kernels, up to 128 -> attention.cuh (multiples of 8; the missing columns of the last two are zeros).
static int launch_attention(const kb_attn_params& p, cudaStream_t stream) {
    if (p.N <= 0) return KB_ERR_UNSUPPORTED;
    if (p.M > 0x7fffffff || p.N > 0x7fffffff || p.B * p.H > 0x7fffffff) return KB_ERR_UNSUPPORTED;
    if (p.D % 8 != 0 || p.D > 128) return KB_ERR_UNSUPPORTED;
    if (attention_short_applicable(p)) return launch_attention_short(p, stream);
    if (p.D <= 64) return launch_attention_split(p, stream);
    return launch_attention128(p, stream);
}

}  // namespace kb
