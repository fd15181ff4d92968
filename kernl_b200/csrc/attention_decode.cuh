// Decode-shape ("skinny") attention for sm_100a: few query rows against many keys, bound by streaming
// K and V from HBM once.
//   attn_decode_group_kernel  the common layout: one CTA per K/V head and key share, the query heads of
//                             a group as the rows of mma.sync, shares merged inside a cluster
//   attn_decode_part1/2       any strides and head dimensions: one key per thread, partial results of
//                             chunks (m, l, acc[D]) in fp32 scratch, merged by the second kernel
// Same maths as src/kernl/implementations/attention_skinny.py:58-366 of the reference (which keeps
// its partial outputs in fp16; fp32 here). Additive masks and the causal flag are honoured in-kernel.
#pragma once
#include "common.cuh"
#include "attention.cuh"

namespace kb {

constexpr int kDecThreads = 128;
constexpr int kDecMaxSplits = 256;
constexpr int kDecMaxD = 256;
constexpr int kDecMaxShares = 16;  // the largest cluster (above eight with the non-portable size allowed)

struct DecDev {
    const void* q; const void* k; const void* v; void* o; const void* mask;
    int64_t q_strides[4], k_strides[4], v_strides[4], o_strides[4], mask_strides[4];
    int B, H, M, N, D;
    float scale_log2;
    int is_causal, mask_dtype;
    int num_splits, chunk;  // chunk = keys per split, multiple of 128
    int kv_group;           // query heads per K/V head, >= 1
    const long long* kv_len_dev;  // optional: number of keys that exist (device side), else N
    float* scratch;         // [B*H, M, num_splits, D+2]
};

// Keys per CTA: 128 when there are few (batch x head x row) problems, so that the key dimension
// supplies the parallelism; doubled (up to 1024) while the launch still has about one full wave of
// CTAs (16 per SM). Longer chunks amortise a CTA's fixed phases (q load, three barriers per 128 keys,
// the final cross-warp sum) and leave fewer partial results for the second kernel to merge.
static void decode_split(int64_t N, int64_t problems, int* num_splits, int* chunk) {
    int64_t c = 128;
    while ((N + c - 1) / c > kDecMaxSplits) c *= 2;
    const int64_t want = 2000;
    while (c < 1024 && problems * ((N + 2 * c - 1) / (2 * c)) >= want) c *= 2;
    *chunk = (int)c;
    *num_splits = (int)((N + c - 1) / c);
    if (*num_splits < 1) *num_splits = 1;
}

static int64_t decode_scratch_bytes(int64_t B, int64_t H, int64_t M, int64_t N, int64_t D) {
    if (B < 0 || H < 0 || M < 0 || N < 0 || D <= 0) return -1;
    int splits, chunk;
    decode_split(N, B * H * M, &splits, &chunk);
    return B * H * M * (int64_t)splits * (D + 2) * (int64_t)sizeof(float);
}

// Keys that exist: all N, or the device-side count of a partly filled cache.
__device__ __forceinline__ int decode_live_keys(const DecDev& p) {
    if (p.kv_len_dev == nullptr) return p.N;
    const long long n = *reinterpret_cast<const volatile long long*>(p.kv_len_dev);
    return n < 0 ? 0 : (n < (long long)p.N ? (int)n : p.N);
}

template <typename T>
__global__ void __launch_bounds__(kDecThreads)
attn_decode_part1_kernel(const DecDev p) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float q_s[kDecMaxD];
    __shared__ float sc_s[kDecThreads];
    __shared__ float red_s[kDecThreads / 32];
    const int split = blockIdx.x, row = blockIdx.y, bh = blockIdx.z;
    const int b = bh / p.H, h = bh % p.H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = p.D;

    const T* qp = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_strides[0] + (int64_t)h * p.q_strides[1] +
                  (int64_t)row * p.q_strides[2];
    for (int d = tid; d < D; d += kDecThreads) q_s[d] = Elem<T>::to_f32(qp[(int64_t)d * p.q_strides[3]]) * p.scale_log2;
    __syncthreads();

    const int hk = h / p.kv_group;
    const T* kbase = reinterpret_cast<const T*>(p.k) + (int64_t)b * p.k_strides[0] + (int64_t)hk * p.k_strides[1];
    const T* vbase = reinterpret_cast<const T*>(p.v) + (int64_t)b * p.v_strides[0] + (int64_t)hk * p.v_strides[1];
    const bool k_vec = p.k_strides[3] == 1 && (p.k_strides[2] % 8) == 0 && (((uintptr_t)kbase) & 15) == 0 && (D % 8) == 0;
    const float mlow = mask_lowest(p.mask_dtype);
    const int64_t mask_off = p.mask ? (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1] +
                                          (int64_t)row * p.mask_strides[2]
                                    : 0;

    float m_run = -INFINITY, l_run = 0.f;
    float acc[kDecMaxD / kDecThreads];
#pragma unroll
    for (int i = 0; i < kDecMaxD / kDecThreads; ++i) acc[i] = 0.f;

    const int key_begin = split * p.chunk;
    const int key_end = min(decode_live_keys(p), key_begin + p.chunk);  // a chunk beyond the live keys scores nothing: (m, l) = (-inf, 0)
    for (int k0 = key_begin; k0 < key_end; k0 += kDecThreads) {
        // ---- one key per thread: score in the log2 domain
        const int key = k0 + tid;
        float s = -INFINITY;
        if (key < key_end && !(p.is_causal && key > row)) {
            const T* kr = kbase + (int64_t)key * p.k_strides[2];
            float dot = 0.f;
            if (k_vec) {
                for (int d = 0; d < D; d += 8) {
                    const uint4 w = __ldg(reinterpret_cast<const uint4*>(kr + d));
                    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = Elem<T>::unpack2(ww[i]);
                        dot = fmaf(f.x, q_s[d + 2 * i], dot);
                        dot = fmaf(f.y, q_s[d + 2 * i + 1], dot);
                    }
                }
            } else {
                for (int d = 0; d < D; ++d) dot = fmaf(Elem<T>::to_f32(kr[(int64_t)d * p.k_strides[3]]), q_s[d], dot);
            }
            s = dot;
            if (p.mask) {
                float mv = mask_load(p.mask, mask_off + (int64_t)key * p.mask_strides[3], p.mask_dtype);
                s = fmaf(fmaxf(mv, mlow), kLog2e, s);
            }
        }
        // ---- block maximum
        float mx = s;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) red_s[warp] = mx;
        __syncthreads();
        mx = fmaxf(fmaxf(red_s[0], red_s[1]), fmaxf(red_s[2], red_s[3]));
        __syncthreads();
        float m_new = fmaxf(m_run, mx);
        if (m_new == -INFINITY) m_new = 0.f;
        const float alpha = (m_run == -INFINITY) ? 0.f : fast_exp2(m_run - m_new);
        const float pe = fast_exp2(s - m_new);
        // P is rounded to the input dtype before P·V, as the reference does (attention_skinny.py:262).
        sc_s[tid] = Elem<T>::to_f32(Elem<T>::from_f32(pe));
        float ps = pe;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
        if (lane == 0) red_s[warp] = ps;
        __syncthreads();
        l_run = l_run * alpha + (red_s[0] + red_s[1] + red_s[2] + red_s[3]);
        m_run = m_new;
        // ---- P·V: thread d accumulates output dimension d over the block's keys
        const int nk = min(kDecThreads, key_end - k0);
#pragma unroll
        for (int i = 0; i < kDecMaxD / kDecThreads; ++i) {
            const int d = tid + i * kDecThreads;
            if (d < D) {
                float a = acc[i] * alpha;
                const T* vp = vbase + (int64_t)k0 * p.v_strides[2] + (int64_t)d * p.v_strides[3];
                for (int kk = 0; kk < nk; ++kk) a = fmaf(sc_s[kk], Elem<T>::to_f32(vp[(int64_t)kk * p.v_strides[2]]), a);
                acc[i] = a;
            }
        }
        __syncthreads();
    }
    float* out = p.scratch + (((int64_t)bh * p.M + row) * p.num_splits + split) * (D + 2);
    if (tid == 0) { out[0] = m_run; out[1] = l_run; }
#pragma unroll
    for (int i = 0; i < kDecMaxD / kDecThreads; ++i) {
        const int d = tid + i * kDecThreads;
        if (d < D) out[2 + d] = acc[i];
    }
}

// Split-KV kernel for the common layout (unit stride on the head dimension, 16-byte aligned rows,
// D = 64, 128 or 256). Bound: streaming K and V from HBM once.
//   * One CTA of four warps takes one K/V head of one sequence, one query row, and one contiguous
//     share of the keys. The query heads of a group (grouped-query attention) are the ROWS of the
//     tensor-core operand, so a group reads its K/V once; with one CTA per query head a group of four
//     read them four times (batch 16, 32 heads over 8, 3000 keys, D = 128: 137 us; the K/V alone
//     take 30 us at the copy bandwidth).
//   * The warps never meet inside the key loop. A warp owns every fourth piece of 16 (D = 64: 32) keys,
//     stages it with asynchronous 16-byte copies in a ring of its own, and keeps its own running
//     maximum, sum and accumulator; no barrier, only its own copy groups. Two CTAs of three stages
//     keep up to 128 KB in flight per SM (D = 128), which is what the copy bandwidth needs here.
//   * q·kᵀ and P·V are mma.sync.m16n8k16: K rows [key][d] are the "col" operand as they lie, V goes
//     through ldmatrix.trans. mma.sync on purpose: at most 16 rows exist and the kernel is bound by
//     memory; what counts is that a byte costs few instructions (130 per warp and 8 KB of K/V).
//   * The key shares of one problem form a cluster (up to sixteen CTAs) and meet in distributed
//     shared memory: every CTA adds up its slice of the output over the cluster. No scratch, no
//     second launch (which alone was 3-9 us). The share is computed from the live key count on the device, so
//     a half-filled cache is spread over all CTAs as evenly as a full one.
template <int D>
struct DecTile {
    static constexpr int kKeys = D == 64 ? 32 : 16;   // keys per piece
    static constexpr int kStages = 3;
    static constexpr int kRowChunks = D / 8;          // 16-byte chunks per row
    static constexpr int kTileBytes = kKeys * D * 2;  // K or V of one piece
    static constexpr int kWarpBytes = kStages * 2 * kTileBytes;
    static constexpr int kSmemBytes = (kDecThreads / 32) * kWarpBytes;
    // partial results of the CTA's warps [warp][row][D] and of the CTA [row][D], in the ring's memory
    static_assert(((kDecThreads / 32) + 1) * 16 * D * 4 <= kSmemBytes, "the partial results do not fit the ring");
};

__device__ __forceinline__ float ld_cluster_f32(uint32_t own_addr, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(own_addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// Grid: x = key share (the cluster dimension), y = query row, z = (sequence, K/V head, group of up to
// ROWS of its query heads). ROWS = 8: rows 8..15 of the operand are zero and never looked at.
template <typename T, int D, int ROWS>
__global__ void __launch_bounds__(kDecThreads, D == 256 ? 1 : 2)
attn_decode_group_kernel(const DecDev p, const int head_groups) {
    using Tile = DecTile<D>;
    constexpr int KEYS = Tile::kKeys, NT = KEYS / 8, WARPS = kDecThreads / 32, RH = ROWS / 8;
    extern __shared__ __align__(128) uint8_t dec_smem[];
    __shared__ float2 ml_warp[WARPS][16];  // (maximum, sum) of a warp
    __shared__ float2 ml_cta[16];          // ... of the CTA, read by the whole cluster
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, c = lane & 3;
    const int row = blockIdx.y;
    const int hg = (int)blockIdx.z % head_groups, bk = (int)blockIdx.z / head_groups;
    const int kv_heads = p.H / p.kv_group;
    const int b = bk / kv_heads, hk = bk % kv_heads;
    const int h0 = hk * p.kv_group + hg * ROWS;
    const int rows = min(ROWS, p.kv_group - hg * ROWS);
    const T* kbase = reinterpret_cast<const T*>(p.k) + (int64_t)b * p.k_strides[0] + (int64_t)hk * p.k_strides[1];
    const T* vbase = reinterpret_cast<const T*>(p.v) + (int64_t)b * p.v_strides[0] + (int64_t)hk * p.v_strides[1];

    // this CTA's keys: an equal share of the live ones, in whole rounds of the four warps
    int key_begin, key_end;
    auto take_share = [&]() {
        const int live = decode_live_keys(p);
        const int round = WARPS * KEYS;
        const int share = ((live + p.num_splits - 1) / p.num_splits + round - 1) / round * round;
        key_begin = min(live, (int)blockIdx.x * share);
        key_end = min(live, key_begin + share);
    };
    // Before the wait for the kernel ahead (which may have written q, the newest key and the count) nothing
    // is read, but the first pieces are asked for in L2: by the count as it is now, which is a hint.
    take_share();
    {
        constexpr int LINES = D * 2 / 128;  // 128-byte lines of a key
        for (int i = tid; i < (Tile::kStages - 1) * WARPS * KEYS * LINES; i += kDecThreads) {
            const int key = key_begin + i / LINES;
            if (key < key_end) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(kbase + (int64_t)key * p.k_strides[2] + (i % LINES) * 64));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(vbase + (int64_t)key * p.v_strides[2] + (i % LINES) * 64));
            }
        }
    }
    pdl_wait();
    pdl_launch_dependents();
    take_share();
    const int pieces = (key_end - key_begin + KEYS - 1) / KEYS;
    const int mine = pieces > warp ? (pieces - warp + WARPS - 1) / WARPS : 0;
    const uint32_t ring = smem_u32(dec_smem) + (uint32_t)(warp * Tile::kWarpBytes);
    // chunk j (16 bytes) of row r sits at r * kRowChunks + (j ^ (r & 7)): eight rows of one chunk column lie
    // in eight different bank groups, for the copies as for ldmatrix
    auto stage = [&](int i) {  // piece i of this warp -> ring slot i % kStages
        const int k0 = key_begin + (warp + i * WARPS) * KEYS;
        const uint32_t dst0 = ring + (uint32_t)((i % Tile::kStages) * 2 * Tile::kTileBytes);
#pragma unroll
        for (int it = 0; it < KEYS * Tile::kRowChunks / 32; ++it) {
            const int idx = it * 32 + lane;
            const int r = idx / Tile::kRowChunks, j = idx % Tile::kRowChunks;
            const bool in = k0 + r < key_end;
            const int key = in ? k0 + r : k0;
            const uint32_t dst = dst0 + (uint32_t)((r * Tile::kRowChunks + (j ^ (r & 7))) * 16);
            const int n = in ? 16 : 0;  // beyond the share: zero fill, nothing is read
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(kbase + (int64_t)key * p.k_strides[2] + j * 8), "r"(n) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + Tile::kTileBytes), "l"(vbase + (int64_t)key * p.v_strides[2] + j * 8), "r"(n) : "memory");
        }
    };
#pragma unroll
    for (int i = 0; i < Tile::kStages - 1; ++i) {
        if (i < mine) stage(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    // q: rows of the A operand, (row g, k 2c..) / (row g, k 2c + 8..) and the same of row g + 8
    uint32_t qf[D / 16][2 * RH];
#pragma unroll
    for (int hh = 0; hh < RH; ++hh) {
        const bool ok = g + 8 * hh < rows;
        const T* qp = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_strides[0] + (int64_t)(h0 + (ok ? g + 8 * hh : 0)) * p.q_strides[1] +
                      (int64_t)row * p.q_strides[2];
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                qf[ks][e * RH + hh] = ok ? __ldg(reinterpret_cast<const uint32_t*>(qp + ks * 16 + e * 8 + 2 * c)) : 0u;
    }
    const float mlow = mask_lowest(p.mask_dtype);
    int64_t mask_off[RH];
#pragma unroll
    for (int hh = 0; hh < RH; ++hh)
        mask_off[hh] = p.mask == nullptr ? 0 : (int64_t)b * p.mask_strides[0] + (int64_t)(h0 + min(g + 8 * hh, rows - 1)) * p.mask_strides[1] +
                                                 (int64_t)row * p.mask_strides[2];

    float o[D / 8][4];
#pragma unroll
    for (int nt = 0; nt < D / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[nt][e] = 0.f;
    float m_run[RH], l_run[RH];
#pragma unroll
    for (int hh = 0; hh < RH; ++hh) { m_run[hh] = -INFINITY; l_run[hh] = 0.f; }

    // Mask values of a piece, as raw bits, one piece ahead: no load is waited for where it is issued. (Fetched and
    // converted one after the other for the piece at hand, they were the critical path of a masked call: 115 us
    // instead of 101 before this kernel at [8, 12, 7075, 128] with a bias.)
    uint32_t mask_next[RH][NT][2];
    auto fetch_mask = [&](int i) {
        if (p.mask == nullptr) return;
        const int k0 = key_begin + (warp + i * WARPS) * KEYS;
        auto fetch = [&](const auto* base) {
#pragma unroll
            for (int hh = 0; hh < RH; ++hh)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int key = k0 + nt * 8 + 2 * c + e;
                        mask_next[hh][nt][e] = (key < key_end && g + 8 * hh < rows) ? __ldg(base + mask_off[hh] + (int64_t)key * p.mask_strides[3]) : 0u;
                    }
        };
        if (p.mask_dtype == KB_F32) fetch(reinterpret_cast<const uint32_t*>(p.mask));
        else fetch(reinterpret_cast<const uint16_t*>(p.mask));
    };
    auto mask_value = [&](uint32_t bits) {
        if (p.mask_dtype == KB_F32) return __uint_as_float(bits);
        const uint16_t h = (uint16_t)bits;
        return p.mask_dtype == KB_F16 ? __half2float(__ushort_as_half(h)) : __uint_as_float((uint32_t)h << 16);
    };
    if (mine > 0) fetch_mask(0);
    for (int i = 0; i < mine; ++i) {
        __syncwarp();  // the slot that is refilled next has been read by all lanes
        if (i + Tile::kStages - 1 < mine) stage(i + Tile::kStages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const int k0 = key_begin + (warp + i * WARPS) * KEYS;
        uint32_t mv[RH][NT][2];
#pragma unroll
        for (int hh = 0; hh < RH; ++hh)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) mv[hh][nt][e] = mask_next[hh][nt][e];
        if (i + 1 < mine) fetch_mask(i + 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(Tile::kStages - 1) : "memory");
        __syncwarp();
        const uint32_t kt = ring + (uint32_t)((i % Tile::kStages) * 2 * Tile::kTileBytes), vt = kt + Tile::kTileBytes;
        // ---- scores: column tile nt = keys k0 + 8 nt ..
        float s[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[nt][e] = 0.f;
            const int r = nt * 8 + (lane & 7);
#pragma unroll
            for (int ks = 0; ks < D / 16; ks += 2) {
                uint32_t kf[4];  // d 16 ks + 8 (lane / 8) ..
                ldmatrix_x4(kt + (uint32_t)((r * Tile::kRowChunks + ((ks * 2 + (lane >> 3)) ^ (r & 7))) * 16), kf);
                mma_16816<T>(s[nt], qf[ks][0], RH == 2 ? qf[ks][1] : 0u, qf[ks][RH], RH == 2 ? qf[ks][2 * RH - 1] : 0u, kf[0], kf[1]);
                mma_16816<T>(s[nt], qf[ks + 1][0], RH == 2 ? qf[ks + 1][1] : 0u, qf[ks + 1][RH], RH == 2 ? qf[ks + 1][2 * RH - 1] : 0u, kf[2], kf[3]);
            }
        }
        // ---- online softmax of the warp's own keys (a row is spread over four lanes)
        uint32_t pf[NT][RH];
        float alpha[RH];
        bool moved = false;
#pragma unroll
        for (int hh = 0; hh < RH; ++hh) {
            float mx = -INFINITY;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int key = k0 + nt * 8 + 2 * c + e;
                    float x = s[nt][hh * 2 + e] * p.scale_log2;
                    if (p.mask != nullptr) x = fmaf(fmaxf(mask_value(mv[hh][nt][e]), mlow), kLog2e, x);
                    if (key >= key_end || (p.is_causal && key > row)) x = -INFINITY;
                    s[nt][hh * 2 + e] = x;
                    mx = fmaxf(mx, x);
                }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            float m_new = fmaxf(m_run[hh], mx);
            if (m_new == -INFINITY) m_new = 0.f;
            alpha[hh] = m_run[hh] == -INFINITY ? 0.f : fast_exp2(m_run[hh] - m_new);
            moved |= m_new != m_run[hh];
            m_run[hh] = m_new;
            float sum = 0.f;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const float e0 = fast_exp2(s[nt][hh * 2] - m_new), e1 = fast_exp2(s[nt][hh * 2 + 1] - m_new);
                sum += e0 + e1;
                pf[nt][hh] = Elem<T>::pack2(e0, e1);  // rounded to the input type, as the reference does (attention_skinny.py:262)
            }
            l_run[hh] = l_run[hh] * alpha[hh] + sum;
        }
        if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
            for (int nt = 0; nt < D / 8; ++nt)
#pragma unroll
                for (int e = 0; e < 2 * RH; ++e) o[nt][e] *= alpha[e >> 1];
        }
        // ---- O += P · V: the score fragments are the A operand of the next product
#pragma unroll
        for (int kb = 0; kb < KEYS / 16; ++kb) {
            const int r = kb * 16 + (lane & 15);
#pragma unroll
            for (int nt = 0; nt < D / 8; nt += 2) {
                uint32_t vf[4];  // keys 0-7, 8-15 of the columns of nt, then of nt + 1
                ldmatrix_x4_trans(vt + (uint32_t)((r * Tile::kRowChunks + ((nt + (lane >> 4)) ^ (r & 7))) * 16), vf);
                const uint32_t a1 = RH == 2 ? pf[2 * kb][RH - 1] : 0u, a3 = RH == 2 ? pf[2 * kb + 1][RH - 1] : 0u;
                mma_16816<T>(o[nt], pf[2 * kb][0], a1, pf[2 * kb + 1][0], a3, vf[0], vf[1]);
                mma_16816<T>(o[nt + 1], pf[2 * kb][0], a1, pf[2 * kb + 1][0], a3, vf[2], vf[3]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    // ---- merge the four warps, then the cluster
#pragma unroll
    for (int hh = 0; hh < RH; ++hh) {
        l_run[hh] += __shfl_xor_sync(0xffffffffu, l_run[hh], 1);
        l_run[hh] += __shfl_xor_sync(0xffffffffu, l_run[hh], 2);
        // a warp that saw no key it may attend to (sum zero) must not set the scale
        if (c == 0) ml_warp[warp][g + 8 * hh] = make_float2(l_run[hh] > 0.f ? m_run[hh] : -INFINITY, l_run[hh]);
    }
    __syncthreads();  // every warp is done with its ring: the partial results go there
    float* part = reinterpret_cast<float*>(dec_smem);       // [warp][row][D]
    float* cta = part + WARPS * ROWS * D;                   // [row][D]
#pragma unroll
    for (int hh = 0; hh < RH; ++hh)
        if (g + 8 * hh < rows)
#pragma unroll
            for (int nt = 0; nt < D / 8; ++nt)
                *reinterpret_cast<float2*>(part + (warp * ROWS + g + 8 * hh) * D + nt * 8 + 2 * c) = make_float2(o[nt][2 * hh], o[nt][2 * hh + 1]);
    __syncthreads();
    const int n_out = rows * D;
    for (int e = tid; e < n_out; e += kDecThreads) {
        const int r = e / D;
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) m = fmaxf(m, ml_warp[w][r].x);
        const float ref = m == -INFINITY ? 0.f : m;
        float acc = 0.f, l = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float sc = fast_exp2(ml_warp[w][r].x - ref);
            l = fmaf(ml_warp[w][r].y, sc, l);
            acc = fmaf(part[(w * ROWS + r) * D + e % D], sc, acc);
        }
        cta[e] = acc;
        if (e % D == 0) ml_cta[r] = make_float2(m, l);
    }
    cluster_sync_all();  // (a cluster of one: a CTA barrier)
    const uint32_t ml_addr = smem_u32(ml_cta), cta_addr = smem_u32(cta);
    for (int e = (int)blockIdx.x * kDecThreads + tid; e < n_out; e += p.num_splits * kDecThreads) {
        const int r = e / D, d = e % D;
        float m = -INFINITY;
        for (int q = 0; q < p.num_splits; ++q) m = fmaxf(m, ld_cluster_f32(ml_addr + 8u * r, q));
        const float ref = m == -INFINITY ? 0.f : m;
        float acc = 0.f, l = 0.f;
        for (int q = 0; q < p.num_splits; ++q) {
            const float sc = fast_exp2(ld_cluster_f32(ml_addr + 8u * r, q) - ref);
            l = fmaf(ld_cluster_f32(ml_addr + 8u * r + 4u, q), sc, l);
            acc = fmaf(ld_cluster_f32(cta_addr + 4u * e, q), sc, acc);
        }
        T* op = reinterpret_cast<T*>(p.o) + (int64_t)b * p.o_strides[0] + (int64_t)(h0 + r) * p.o_strides[1] + (int64_t)row * p.o_strides[2];
        op[(int64_t)d * p.o_strides[3]] = Elem<T>::from_f32(acc / l);
    }
    cluster_sync_all();  // nobody leaves while its shared memory may still be read
}

template <typename T>
__global__ void __launch_bounds__(kDecThreads)
attn_decode_part2_kernel(const DecDev p) {
    pdl_wait();
    pdl_launch_dependents();
    const int row = blockIdx.x, bh = blockIdx.y;
    const int b = bh / p.H, h = bh % p.H;
    const int D = p.D;
    const float* in = p.scratch + ((int64_t)bh * p.M + row) * p.num_splits * (D + 2);
    float m_tot = -INFINITY;
    for (int s = 0; s < p.num_splits; ++s) m_tot = fmaxf(m_tot, in[(int64_t)s * (D + 2)]);
    float l_tot = 0.f;
    for (int s = 0; s < p.num_splits; ++s) {
        const float ms = in[(int64_t)s * (D + 2)];
        if (ms != -INFINITY) l_tot += in[(int64_t)s * (D + 2) + 1] * fast_exp2(ms - m_tot);
    }
    T* op = reinterpret_cast<T*>(p.o) + (int64_t)b * p.o_strides[0] + (int64_t)h * p.o_strides[1] +
            (int64_t)row * p.o_strides[2];
    for (int d = threadIdx.x; d < D; d += kDecThreads) {
        float a = 0.f;
        for (int s = 0; s < p.num_splits; ++s) {
            const float ms = in[(int64_t)s * (D + 2)];
            if (ms != -INFINITY) a += in[(int64_t)s * (D + 2) + 2 + d] * fast_exp2(ms - m_tot);
        }
        op[(int64_t)d * p.o_strides[3]] = Elem<T>::from_f32(a / l_tot);
    }
}

template <typename T, int D, int ROWS>
static int launch_decode_group_r(DecDev d, cudaStream_t stream) {
    auto* kernel = attn_decode_group_kernel<T, D, ROWS>;
    const int head_groups = (d.kv_group + ROWS - 1) / ROWS;
    const unsigned problems = (unsigned)(d.B * (d.H / d.kv_group) * head_groups);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kDecThreads);
    cfg.dynamicSmemBytes = DecTile<D>::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    // Clusters that are resident at once, by size: a cluster stays inside one GPC, so that sizes which do not
    // divide a GPC's CTA slots leave some of them empty (asked once per device).
    static std::mutex mu;
    static int resident[64][kDecMaxShares + 1] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return KB_ERR_NO_DEVICE;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (resident[dev][1] == 0) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DecTile<D>::kSmemBytes) != cudaSuccess ||
                cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
                return KB_ERR_LAUNCH;
            cfg.numAttrs = 1;
            for (int s = kDecMaxShares; s >= 1; --s) {
                int n = 0;
                cfg.gridDim = dim3((unsigned)s);
                attr[0].val.clusterDim.x = (unsigned)s;
                if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
                    cudaGetLastError();
                    n = s > 8 ? 0 : 1;  // (not every device takes the large ones)
                }
                resident[dev][s] = n;
            }
        }
    }
    // Key shares per problem (the cluster size). A wave of clusters costs the bytes of one share plus a fixed
    // part — first copies from DRAM, q, the merge: about 2.5 us, which at a CTA slot's part of the copy
    // bandwidth is 56 KB — so shares are cut until one wave is full and no further.
    const int64_t units = (int64_t)problems * d.M, round = (kDecThreads / 32) * DecTile<D>::kKeys;
    double best_cost = 1e300;
    d.num_splits = 1;
    for (int s = 1; s <= kDecMaxShares && (s - 1) * round < d.N; ++s) {
        if (resident[dev][s] == 0) continue;
        const int64_t share = ((d.N + s - 1) / s + round - 1) / round * round;
        const double cost = (double)((units + resident[dev][s] - 1) / resident[dev][s]) * ((double)share * D * 4.0 + 56.0 * 1024.0);
        if (cost < best_cost) {
            best_cost = cost;
            d.num_splits = s;
        }
    }
    cfg.gridDim = dim3((unsigned)d.num_splits, (unsigned)d.M, problems);
    attr[0].val.clusterDim.x = (unsigned)d.num_splits;
    cfg.numAttrs = g_use_pdl ? 2u : 1u;
    return cudaLaunchKernelEx(&cfg, kernel, d, head_groups) == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

template <typename T>
static int launch_decode_group(const DecDev& d, cudaStream_t stream) {
    const bool wide = d.kv_group > 8;  // sixteen operand rows only where a group fills more than eight
    if (d.D == 64) return wide ? launch_decode_group_r<T, 64, 16>(d, stream) : launch_decode_group_r<T, 64, 8>(d, stream);
    if (d.D == 128) return wide ? launch_decode_group_r<T, 128, 16>(d, stream) : launch_decode_group_r<T, 128, 8>(d, stream);
    return wide ? launch_decode_group_r<T, 256, 16>(d, stream) : launch_decode_group_r<T, 256, 8>(d, stream);
}

static int launch_attention_decode(const kb_attn_params& p, void* scratch, int64_t scratch_bytes, cudaStream_t stream) {
    if (p.N <= 0 || p.D > kDecMaxD) return KB_ERR_UNSUPPORTED;
    if (p.M > 65535 || p.B * p.H > 65535) return KB_ERR_UNSUPPORTED;
    DecDev d;
    d.q = p.q; d.k = p.k; d.v = p.v; d.o = p.o; d.mask = p.mask;
    for (int i = 0; i < 4; ++i) {
        d.q_strides[i] = p.q_strides[i]; d.k_strides[i] = p.k_strides[i]; d.v_strides[i] = p.v_strides[i];
        d.o_strides[i] = p.o_strides[i]; d.mask_strides[i] = p.mask ? p.mask_strides[i] : 0;
    }
    d.B = (int)p.B; d.H = (int)p.H; d.M = (int)p.M; d.N = (int)p.N; d.D = (int)p.D;
    d.scale_log2 = p.sm_scale * kLog2e;
    d.is_causal = p.is_causal ? 1 : 0;
    d.mask_dtype = p.mask ? p.mask_dtype : KB_F32;
    d.kv_group = p.kv_group > 1 ? p.kv_group : 1;
    if (p.H % d.kv_group != 0) return KB_ERR_BAD_ARG;
    d.kv_len_dev = reinterpret_cast<const long long*>(p.kv_len_dev);
    const bool vec_ok = (p.D == 64 || p.D == 128 || p.D == 256) && p.q_strides[3] == 1 && p.k_strides[3] == 1 &&
                        p.v_strides[3] == 1 && (p.k_strides[2] % 8) == 0 && (p.v_strides[2] % 8) == 0 &&
                        (p.k_strides[1] % 8) == 0 && (p.v_strides[1] % 8) == 0 && (p.k_strides[0] % 8) == 0 &&
                        (p.v_strides[0] % 8) == 0 && (((uintptr_t)p.k) & 15) == 0 && (((uintptr_t)p.v) & 15) == 0 &&
                        (((uintptr_t)p.q) & 15) == 0 && (p.q_strides[0] % 8) == 0 && (p.q_strides[1] % 8) == 0 &&
                        (p.q_strides[2] % 8) == 0;
    if (vec_ok) return p.dtype == KB_F16 ? launch_decode_group<__half>(d, stream) : launch_decode_group<__nv_bfloat16>(d, stream);
    // any other layout: chunks through scratch and a second kernel
    if (scratch == nullptr || scratch_bytes < decode_scratch_bytes(p.B, p.H, p.M, p.N, p.D)) return KB_ERR_BAD_ARG;
    d.scratch = reinterpret_cast<float*>(scratch);
    decode_split(p.N, p.B * p.H * p.M, &d.num_splits, &d.chunk);
    const dim3 g1((unsigned)d.num_splits, (unsigned)p.M, (unsigned)(p.B * p.H));
    const dim3 g2((unsigned)p.M, (unsigned)(p.B * p.H));
    if (p.dtype == KB_F16) {
        launch_pdl(attn_decode_part1_kernel<__half>, g1, kDecThreads, 0, stream, d);
        launch_pdl(attn_decode_part2_kernel<__half>, g2, kDecThreads, 0, stream, d);
    } else {
        launch_pdl(attn_decode_part1_kernel<__nv_bfloat16>, g1, kDecThreads, 0, stream, d);
        launch_pdl(attn_decode_part2_kernel<__nv_bfloat16>, g2, kDecThreads, 0, stream, d);
    }
    return cudaGetLastError() == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

}  // namespace kb
