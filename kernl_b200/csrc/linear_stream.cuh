// Linear layer for few rows: y = act(x · Wᵀ + bias), the decode-step shape, and small problems of some more.
//
// With a handful of rows the op is a single pass over W from HBM (2·N·K bytes; x is a few dozen KB and
// lives in L2), so what matters is how many bytes every SM keeps in flight, without a break, and how
// little fixed cost a launch carries — not the tensor-core generation. The tcgen05 GEMM pays for tensor
// maps, a TMEM allocation, a 128-row tile of which 8 rows are real, and a second kernel to finish its
// split-K sums. Here:
//   * W is the row operand of mma.sync.m16n8k16 (16 weight rows x 8 rows of x): up to eight rows of x
//     cost one instruction per 16 x 16 block of W;
//   * every CTA (two per SM) takes an equal share of the rows of W, whatever their number: 11008 rows
//     are 37 or 38 for each of 296 CTAs. It walks them in tiles of at most 48 rows. With tiles of a fixed
//     16 rows the same matrix was 2.3 rounds, run as 3;
//   * the four warps of a CTA split K in interleaved pieces of 64 elements. Each warp stages its pieces
//     — W rows and the same columns of x — with asynchronous 16-byte copies in a ring of its own: no
//     barrier in the main loop, no register holds a byte in flight, and the ring runs on into the next
//     tile while the four partial tiles meet in shared memory;
//   * before it waits for the kernel that produces x, a CTA asks for its first pieces of W in L2 only
//     (W itself may be that kernel's output, so nothing of it is read before the wait).
// Dividing tiles between CTAs to even out the rounds (partial sums through the workspace, the last CTA
// finishes) was tried: the fence, the counter and the second read cost 3 us at the end of every launch.
// The kernel before this one held 8 loads per thread in registers and drained them once per
// 1024 columns, in rounds of one 16-row tile per CTA: [16, 4096] x [11008, 4096] took 23.4 us (3.9 TB/s).
// Same contract as the reference's linear_layer (src/kernl/implementations/linear_layer.py:213-282).
#pragma once
#include "linear.cuh"

namespace kb {

constexpr int kStreamThreads = 128;
constexpr int kStreamWarps = kStreamThreads / 32;
constexpr int kStreamK = 64;  // elements of K per piece: 128-byte rows in shared memory
constexpr int kStreamMaxM = 32;  // rows of x per CTA; more rows are further CTAs (grid.y) over the same W
constexpr int kStreamSmemBytes = 112 * 1024;  // rings and partial tiles of a CTA: two CTAs per SM

constexpr int stream_red_nx(int nx) { return nx > 2 ? 2 : nx; }  // 8-row tiles of x whose partial sums meet at a time
constexpr int stream_red_bytes(int rmax, int nx) { return kStreamWarps * stream_red_nx(nx) * 8 * (rmax + 1) * 4; }

// RMAX: most rows of W per tile (a multiple of 8), NX: 8-row tiles of x.
template <int RMAX, int NX>
struct StreamCfg {
    static constexpr int kTiles16 = (RMAX + 15) / 16;  // 16-row operand tiles; rows beyond the tile's hold anything
    static constexpr int kWBytes = RMAX * kStreamK * 2;
    static constexpr int kStageBytes = kWBytes + NX * 8 * kStreamK * 2;
    static constexpr int kRedNx = stream_red_nx(NX);
    static constexpr int kRedRow = RMAX + 1;  // partial tile of a warp: [x row][W row], rows padded
    static constexpr int kFit = (kStreamSmemBytes - stream_red_bytes(RMAX, NX)) / (kStreamWarps * kStageBytes);
    static constexpr int kStages = kFit > 10 ? 10 : kFit;
    static constexpr int kSmemBytes = kStreamWarps * kStages * kStageBytes + stream_red_bytes(RMAX, NX);
    static_assert(kStages >= 3, "a warp needs two pieces in flight");
};

// `lines`: what is shared out among the CTAs — rows of W, or pairs of a gate and an up row (gated
// epilogue: pair o is rows 16 (o / 8) + o % 8 and eight further). `tiles`: tiles per CTA.
template <typename T, int RMAX, int NX>
__global__ void __launch_bounds__(kStreamThreads, 2)
linear_stream_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias, T* __restrict__ y,
                     T* __restrict__ act_inputs, int M, int lines, int K, int64_t x_row_stride, int64_t y_row_stride,
                     int activation, int tiles) {
    using Cfg = StreamCfg<RMAX, NX>;
    constexpr int STAGES = Cfg::kStages, MT = Cfg::kTiles16, RNX = Cfg::kRedNx;
    extern __shared__ __align__(128) uint8_t stream_smem[];
    {
        const int m0 = (int)blockIdx.y * kStreamMaxM;
        x += m0 * x_row_stride;
        y += m0 * y_row_stride;
        if (act_inputs != nullptr) act_inputs += m0 * y_row_stride;
        M = min(M - m0, kStreamMaxM);
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, c = lane & 3;
    const uint32_t ring = smem_u32(stream_smem) + (uint32_t)(warp * STAGES * Cfg::kStageBytes);
    float* red = reinterpret_cast<float*>(stream_smem + kStreamWarps * STAGES * Cfg::kStageBytes);
    const bool gated = activation == KB_ACT_SWIGLU;

    const int pieces = (K + kStreamK - 1) / kStreamK;
    const int mine = pieces > warp ? (pieces - warp + kStreamWarps - 1) / kStreamWarps : 0;  // this warp's pieces of a tile
    // every CTA starts elsewhere in K, so that the CTAs do not walk the memory channels in step (1-4 %)
    const int start = mine > 0 ? (int)(blockIdx.x * 5u) % mine : 0;
    const int cta_begin = (int)((int64_t)blockIdx.x * lines / gridDim.x);
    const int cta_lines = (int)((int64_t)(blockIdx.x + 1) * lines / gridDim.x) - cta_begin;
    auto tile_begin = [&](int t) { return cta_begin + t * cta_lines / tiles; };
    // row r of the tile that covers lines [l0, l0 + n): the gate rows of its pairs, then their up rows
    auto w_row = [&](int l0, int n, int r) {
        if (!gated) return l0 + r;
        const int o = l0 + (r < n ? r : r - n);
        return (o >> 3) * 16 + (o & 7) + (r < n ? 0 : 8);
    };

    if (mine > 0) {
        const int l0 = tile_begin(0), n = tile_begin(1) - l0, rows = gated ? 2 * n : n;
        for (int i = lane; i < rows * min(mine, STAGES - 1); i += 32)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (int64_t)w_row(l0, n, i % rows) * K + (warp + (start + i / rows) % mine * kStreamWarps) * kStreamK));
    }
    pdl_wait();
    pdl_launch_dependents();

    // a 16-byte chunk j of row r sits at r * 128 + (j ^ (r & 7)) * 16: conflict-free for ldmatrix. A lane copies
    // chunk lj of every fourth row; its row pointers change only with the tile, so that a piece costs two
    // instructions per copy (a warp has some 700 cycles per piece before it falls behind the memory).
    const int lr = lane >> 3, lj = lane & 7;
    const T* wp[RMAX / 4];
    const T* xp[NX * 2];
    int in_tile = 0, in_piece = 0, in_slot = 0, in_rows = 0;
    auto enter_tile = [&]() {
        const int l0 = tile_begin(in_tile), n = tile_begin(in_tile + 1) - l0;
        in_rows = gated ? 2 * n : n;
#pragma unroll
        for (int it = 0; it < RMAX / 4; ++it) wp[it] = w + (int64_t)w_row(l0, n, it * 4 + lr) * K + lj * 8;
    };
#pragma unroll
    for (int it = 0; it < NX * 2; ++it) xp[it] = x + (int64_t)(it * 4 + lr) * x_row_stride + lj * 8;
    if (mine > 0) enter_tile();
    auto issue = [&]() {
        if (mine > 0 && in_tile < tiles) {
            const int turn = in_piece + start, k = (warp + (turn < mine ? turn : turn - mine) * kStreamWarps) * kStreamK;
            const int n_copy = k + lj * 8 < K ? 16 : 0;  // K is a multiple of 8; nothing is read beyond it
            const int ks = n_copy ? k : -lj * 8;
            const uint32_t dst = ring + (uint32_t)(in_slot * Cfg::kStageBytes);
#pragma unroll
            for (int it = 0; it < RMAX / 4; ++it) {
                const int r = it * 4 + lr;  // rows beyond the tile are not copied: their results are not used
                if (r < in_rows)
                    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(r * 128 + ((lj ^ (r & 7)) * 16))),
                                 "l"(wp[it] + ks), "r"(n_copy) : "memory");
            }
#pragma unroll
            for (int it = 0; it < NX * 2; ++it) {
                const int r = it * 4 + lr;
                if (r < M)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(Cfg::kWBytes + r * 128 + ((lj ^ (r & 7)) * 16))),
                                 "l"(xp[it] + ks), "r"(n_copy) : "memory");
            }
            if (++in_slot == STAGES) in_slot = 0;
            if (++in_piece == mine) {
                in_piece = 0;
                if (++in_tile < tiles) enter_tile();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = 0; i < STAGES - 1; ++i) issue();

    int slot = 0;
    for (int tile = 0; tile < tiles; ++tile) {
        const int l0 = tile_begin(tile), n_lines = tile_begin(tile + 1) - l0;
        constexpr int LH = (RMAX + 31) / 32;
        float bias_r[LH], bias_up[LH];
#pragma unroll
        for (int h = 0; h < LH; ++h) {
            const int r = h * 32 + lane;
            bias_r[h] = bias_up[h] = 0.f;
            if (bias != nullptr && r < n_lines) {
                bias_r[h] = Elem<T>::to_f32(__ldg(bias + w_row(l0, n_lines, r)));
                if (gated) bias_up[h] = Elem<T>::to_f32(__ldg(bias + w_row(l0, n_lines, n_lines + r)));
            }
        }
        float acc[2][MT][NX][4];  // two chains: a product waits for the one before the last
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nx = 0; nx < NX; ++nx)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[0][mt][nx][e] = acc[1][mt][nx][e] = 0.f;
        for (int i = 0; i < mine; ++i) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncwarp();  // every lane's copies of this piece are visible, and the slot before it has been read
            const uint32_t st = ring + (uint32_t)(slot * Cfg::kStageBytes), sx = st + Cfg::kWBytes;
            if (++slot == STAGES) slot = 0;
            uint32_t xf[NX][8], wf[kStreamK / 16][MT][4];
#pragma unroll
            for (int nx = 0; nx < NX; ++nx) {
                const int r = nx * 8 + (lane & 7);
                uint32_t f[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    ldmatrix_x4(sx + (uint32_t)(r * 128 + (((h * 4 + (lane >> 3)) ^ (r & 7)) * 16)), f);
#pragma unroll
                    for (int e = 0; e < 4; ++e) xf[nx][h * 4 + e] = f[e];
                }
            }
#pragma unroll
            for (int ks = 0; ks < kStreamK / 16; ++ks)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const int r = mt * 16 + (lane & 15);
                    ldmatrix_x4(st + (uint32_t)(r * 128 + (((ks * 2 + (lane >> 4)) ^ (r & 7)) * 16)), wf[ks][mt]);
                }
            issue();  // while the fragments arrive
#pragma unroll
            for (int ks = 0; ks < kStreamK / 16; ++ks)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nx = 0; nx < NX; ++nx)
                        mma_16816<T>(acc[ks & 1][mt][nx], wf[ks][mt][0], wf[ks][mt][1], wf[ks][mt][2], wf[ks][mt][3], xf[nx][ks * 2], xf[nx][ks * 2 + 1]);
        }
        // c0, c1 -> (W row g, x rows 2c, 2c + 1); c2, c3 -> (W row g + 8, same)
        // The sums of the four warps, 16 rows of x at a time. A lane keeps to its lines of the tile and a warp to its
        // rows of x: no division, and bias is in registers since the tile began.
#pragma unroll
        for (int nx0 = 0; nx0 < NX; nx0 += RNX) {
            if (nx0 * 8 >= M) break;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nx = 0; nx < RNX; ++nx)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int r = mt * 16 + g + 8 * (e >> 1);
                        if (r < RMAX)
                            red[(warp * RNX * 8 + nx * 8 + 2 * c + (e & 1)) * Cfg::kRedRow + r] = acc[0][mt][nx0 + nx][e] + acc[1][mt][nx0 + nx][e];
                    }
            __syncthreads();
            auto sum = [&](int m, int r) {
                float z = 0.f;
#pragma unroll
                for (int wi = 0; wi < kStreamWarps; ++wi) z += red[(wi * RNX * 8 + m) * Cfg::kRedRow + r];
                return z;
            };
            const int m_live = min(M - nx0 * 8, RNX * 8);
#pragma unroll
            for (int h = 0; h < LH; ++h) {
                const int r = h * 32 + lane;
                if (r >= n_lines) break;
                for (int m = warp; m < m_live; m += kStreamWarps) {
                    const int64_t out = (int64_t)(nx0 * 8 + m) * y_row_stride + l0 + r;
                    float z = sum(m, r) + bias_r[h];
                    if (gated) {
                        y[out] = Elem<T>::from_f32(act_silu(z) * (sum(m, n_lines + r) + bias_up[h]));
                        continue;
                    }
                    if (act_inputs != nullptr) act_inputs[out] = Elem<T>::from_f32(z);
                    switch (activation) {
                        case KB_ACT_TANH: z = act_tanh(z); break;
                        case KB_ACT_GELU: z = act_gelu(z); break;
                        case KB_ACT_FAST_GELU: z = act_fast_gelu(z); break;
                        case KB_ACT_RELU: z = fmaxf(z, 0.f); break;
                        case KB_ACT_SILU: z = act_silu(z); break;
                        default: break;
                    }
                    y[out] = Elem<T>::from_f32(z);
                }
            }
            __syncthreads();  // the partial sums are rewritten by the next pass
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <typename T, int RMAX, int NX>
static int launch_linear_stream(const kb_linear_params& p, cudaStream_t stream, int64_t lines, int64_t ctas, int tiles) {
    using Cfg = StreamCfg<RMAX, NX>;
    static PerDeviceOnce attr_once;
    if (!attr_once.run([] {
            return cudaFuncSetAttribute(linear_stream_kernel<T, RMAX, NX>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) == cudaSuccess;
        }))
        return KB_ERR_LAUNCH;
    launch_pdl(linear_stream_kernel<T, RMAX, NX>, dim3((unsigned)ctas, (unsigned)((p.M + kStreamMaxM - 1) / kStreamMaxM)), kStreamThreads, Cfg::kSmemBytes, stream, (const T*)p.x, (const T*)p.w,
               (const T*)p.bias, (T*)p.y, (T*)p.act_inputs, (int)p.M, (int)lines, (int)p.K, p.x_row_stride, p.y_row_stride, p.activation, tiles);
    return cudaGetLastError() == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

// Rows of W that a CTA keeps in flight with tiles of r rows: all stages but the one being read.
template <int NX>
static int stream_rows_in_flight(int r) {
    if (r <= 8) return (StreamCfg<8, NX>::kStages - 1) * r;
    if (r <= 16) return (StreamCfg<16, NX>::kStages - 1) * r;
    if (r <= 24) return (StreamCfg<24, NX>::kStages - 1) * r;
    if (r <= 32) return (StreamCfg<32, NX>::kStages - 1) * r;
    if constexpr (NX < 4) {
        if (r <= 40) return (StreamCfg<40, NX>::kStages - 1) * r;
        return (StreamCfg<48, NX>::kStages - 1) * r;
    }
    return 0;
}

struct StreamPlan {
    int64_t ctas;  // per 32 rows of x
    int tiles, rows;
    double us;     // above 16 rows: estimated time
};

// Up to 16 rows: W is what counts. Two CTAs per SM, fewer where that would leave a CTA less than eight rows
// (a whole mma.sync operand half); tiles per CTA: the fewer the better (a tile costs a cross-warp sum, about as
// long as four pieces of a warp), as long as the tile's rows keep the ring full: below about 112 rows in
// flight per CTA the copies are bound by latency.
template <int NX>
static StreamPlan stream_plan_w(const kb_linear_params& p, int64_t lines, int per_line) {
    StreamPlan best{2 * (int64_t)sm_count(), 1, 0, 0.0};
    if (lines * per_line < best.ctas * 8) best.ctas = (lines * per_line + 7) / 8;
    const int64_t share = (lines + best.ctas - 1) / best.ctas * per_line;  // most rows of a CTA
    double best_cost = 1e300;
    const int max_rows = 48;
    for (int64_t t = (share + max_rows - 1) / max_rows; t <= share && t <= (share + 7) / 8 + 1; ++t) {
        const int rows = (int)((share / per_line + t - 1) / t) * per_line;
        if (rows > max_rows) continue;
        const double fill = stream_rows_in_flight<NX>(rows) / 112.0;
        const double cost = (double)share * p.K / (fill < 1.0 ? fill : 1.0) + (double)t * 16 * kStreamK * rows;
        if (cost < best_cost) {
            best_cost = cost;
            best.tiles = (int)t;
            best.rows = rows;
        }
    }
    return best;
}

// Above 16 rows: CTAs of 32 rows of x and `rows` of W, one tile each. A CTA pulls its rows through half an SM's
// port to L2 (59 bytes per ns) and multiplies them at half an SM's mma.sync rate (0.49 products per ps); the
// rest is fitted to times over 20 to 384 rows and W from 500 x 1000 to 4096 x 4096.
static StreamPlan stream_plan_x(const kb_linear_params& p) {
    const int per_line = p.activation == KB_ACT_SWIGLU ? 2 : 1;
    const int64_t slots = 2 * (int64_t)sm_count(), groups = (p.M + kStreamMaxM - 1) / kStreamMaxM;
    StreamPlan best{1, 1, 0, 1e300};
    for (int rows = 8 * per_line; rows <= 32; rows += 8 * per_line) {
        const int64_t ctas = (p.N + rows - 1) / rows;
        const double load = (double)p.K * 2.0 * (rows + kStreamMaxM) / 59e3;
        const double math = (double)((rows + 15) / 16 * 16) * kStreamMaxM * (double)p.K / 486e3;
        // (rows of W that are no multiple of 128 bytes: 6.6 us for the 5.0 this gives without at 128 rows of [500, 1000])
        const double us = 2.4 + (p.K % kStreamK != 0 ? 1.8 : 1.2) * (double)((ctas * groups + slots - 1) / slots) * (load + 0.5 * math + 0.3);
        if (us < best.us) best = StreamPlan{ctas, 1, rows, us};
    }
    const double hbm = (double)p.N * (double)p.K * 2.0 / 5.0e6;  // (with x in every ring, W does not come faster)
    if (best.us < 2.4 + hbm) best.us = 2.4 + hbm;
    return best;
}

static bool stream_layout(const kb_linear_params& p) {
    return p.M >= 1 && p.K % 8 == 0 && p.x_row_stride % 8 == 0 && (((uintptr_t)p.x) & 15) == 0 && (((uintptr_t)p.w) & 15) == 0 &&
           p.N <= (int64_t)0x7fffffff / 2 && p.K <= 0x7fffffff;
}

template <typename T, int NX>
static int launch_linear_stream_n(const kb_linear_params& p, cudaStream_t stream) {
    const int per_line = p.activation == KB_ACT_SWIGLU ? 2 : 1;
    const int64_t lines = p.N / per_line;
    const StreamPlan plan = NX == 4 ? stream_plan_x(p) : stream_plan_w<NX>(p, lines, per_line);
    if (plan.rows <= 8) return launch_linear_stream<T, 8, NX>(p, stream, lines, plan.ctas, plan.tiles);
    if (plan.rows <= 16) return launch_linear_stream<T, 16, NX>(p, stream, lines, plan.ctas, plan.tiles);
    if (plan.rows <= 24) return launch_linear_stream<T, 24, NX>(p, stream, lines, plan.ctas, plan.tiles);
    if constexpr (NX < 4) {
        if (plan.rows > 40) return launch_linear_stream<T, 48, NX>(p, stream, lines, plan.ctas, plan.tiles);
        if (plan.rows > 32) return launch_linear_stream<T, 40, NX>(p, stream, lines, plan.ctas, plan.tiles);
    }
    return launch_linear_stream<T, 32, NX>(p, stream, lines, plan.ctas, plan.tiles);
}

template <typename T>
static int launch_linear_stream_t(const kb_linear_params& p, cudaStream_t stream) {
    if (p.M <= 8) return launch_linear_stream_n<T, 1>(p, stream);
    if (p.M <= 16) return launch_linear_stream_n<T, 2>(p, stream);
    return launch_linear_stream_n<T, 4>(p, stream);
}

}  // namespace kb
