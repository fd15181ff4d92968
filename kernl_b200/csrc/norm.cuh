// LayerNorm / RMSNorm forward for sm_100a. HBM-bound: x is read once and y written once.
//
// Fast path: one, four or eight warps per row, the whole row held in registers as 128-bit vectors (8 elements of
// a 16-bit type per load), statistics by warp shuffles in fp32 in one sweep over the registers
// (shifted sums, no second trip to memory). Algorithmic traffic per row is 2*cols*2 bytes.
// Generic path: arbitrary strides / column counts, one warp per row, re-reads the row (served by
// L1/L2) — correctness path for the strided cases the reference accepts
// (src/kernl/implementations/layer_norm.py:321-324).
#pragma once
#include "common.cuh"

namespace kb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint4 ld_stream_16B(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ void st_stream_16B(void* p, uint4 v) {
    asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w)
                 : "memory");
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

constexpr int kNormMaxCols = 16384;  // longest row that is held in registers

// WPR warps share one row: 1 for many short rows, 4 (the whole CTA) for rows of more than 1024 columns and for
// few rows, 8 above 4096 columns. A lane owns CHUNKS = ceil(cols / (256 WPR)) vectors of 8 elements, at most four
// on every path that matters: with one warp per row a row of 4096 columns took 150 registers per thread
// and left twelve warps on an SM, all of them loading, then all computing, then all storing:
// [16384, 4096] bf16 add + RMSNorm 120.9 us (4.4 TB/s), with four warps per row 89.2 us (6.0 TB/s).
// Vector c of lane l of warp w covers columns ((c*WPR + w)*32 + l)*8 .. +8. cols must be a multiple of 8.
// CHAIN (RMSNorm of 1025 to 4096 columns, more than 1024 rows): the warps own consecutive parts of the row and pass each
// lane's sum of squares on from warp to warp, so that the row is summed in the order of one warp walking it, the order a
// decoder's prefill at these widths has always had: another one moves its hidden states by roundings, and near-ties of
// its greedy tokens with them. Nothing more is promised: the same row in a launch of up to 1024 rows, longer rows
// (eight warps) and LayerNorm add up their warps' sums pairwise. The hand-over is
// hidden behind the other CTAs of the SM.
// EARLY (up to 64 rows of 1025 to 4096 columns: the norms of a decode step): gamma, beta and the residual are asked for in L2 ahead of the
// wait; behind it they would queue behind the weights that the next GEMM asks for (8 rows of 4096: 5.2 -> 3.8 us between the ends of the
// two kernels, a step of eight layers 1034 -> 1019). A decode step of four layers without and with it: 16 rows 475 and 467 us, 32 548 and 538,
// 64 649 and 642, 96 760 and 753, 128 852 and 847, 192 and 256 rows no difference. With hundreds of rows it is a second pass over the residual:
// LayerNorm of [500, 3000] 4.0 us without, 4.4 with it, of [2430, 2368] 9.9 and 12.0. Rows of 8192 (eight warps): no difference at 8 and 64 rows.
template <typename T, int CHUNKS, bool RMS, int WPR = 1, bool CHAIN = false, bool EARLY = false>
__global__ void __launch_bounds__(WPR == 8 ? 256 : 128)
norm_fwd_rowwarp_kernel(const T* __restrict__ x, T* __restrict__ y, const T* __restrict__ gamma,
                        const T* __restrict__ beta, float* __restrict__ mean_out,
                        float* __restrict__ rstd_out, int64_t rows, int cols, int64_t x_row_stride,
                        int64_t y_row_stride, float eps, const T* __restrict__ residual,
                        T* __restrict__ sum_out) {
    __shared__ float red_s[2][8];
    __shared__ float chain_s[CHAIN ? 32 : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wir = warp % WPR;  // this warp's position inside its row
    const int64_t row = WPR == 1 ? (int64_t)blockIdx.x * 4 + warp : (int64_t)blockIdx.x;
#define KB_NORM_COL(c) (((CHAIN ? wir * CHUNKS + (c) : (c) * WPR + wir) * 32 + lane) * 8)
    if (EARLY && (lane & 7) == 0) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const int col = KB_NORM_COL(c);
            if (col < cols) {
                prefetch_l2(gamma + col);
                if (!RMS && beta != nullptr) prefetch_l2(beta + col);
                if (residual != nullptr) prefetch_l2(residual + row * (int64_t)cols + col);
            }
        }
    }
    pdl_wait();
    pdl_launch_dependents();
    if (row >= rows) return;  // (WPR > 1: the whole CTA leaves together)
    const T* xr = x + row * x_row_stride;
    T* yr = y + row * y_row_stride;

    uint4 v[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        const int col = KB_NORM_COL(c);
        if (col < cols) v[c] = ld_stream_16B(xr + col);
        else v[c] = make_uint4(0, 0, 0, 0);
    }
    // Short rows: fetch gamma/beta now, next to the row itself, instead of after the statistics, where
    // their (L1/L2) latency would sit at the end of a warp that has nothing left to overlap it with.
    // Not for a LayerNorm of several warps per row: gamma and beta then cost 32 registers a thread and a third of
    // the warps on an SM ([16384, 4096] with a residual: 109.7 us early, 86.7 us late).
    constexpr bool kEarlyAffine = CHUNKS <= 4 && (RMS || WPR == 1);
    uint4 gv[kEarlyAffine ? CHUNKS : 1], bv[kEarlyAffine ? CHUNKS : 1];
    if (kEarlyAffine) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const int col = KB_NORM_COL(c);
            gv[c] = make_uint4(0, 0, 0, 0);
            bv[c] = make_uint4(0, 0, 0, 0);
            if (col < cols) {
                gv[c] = *reinterpret_cast<const uint4*>(gamma + col);
                if (!RMS && beta != nullptr) bv[c] = *reinterpret_cast<const uint4*>(beta + col);
            }
        }
    }
    if (residual != nullptr) {
        // pre-norm residual stream: s = x + residual (rounded to the 16-bit type, as a separate add
        // kernel would store it), written out once if it is asked for, and normalised from the registers
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const int col = KB_NORM_COL(c);
            if (col < cols) {
                const uint4 r = ld_stream_16B(residual + row * (int64_t)cols + col);
                const uint32_t xw[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
                const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
                uint32_t sw[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 a = Elem<T>::unpack2(xw[i]), b = Elem<T>::unpack2(rw[i]);
                    sw[i] = Elem<T>::pack2(a.x + b.x, a.y + b.y);
                }
                v[c] = make_uint4(sw[0], sw[1], sw[2], sw[3]);
                if (sum_out != nullptr) st_stream_16B(sum_out + row * (int64_t)cols + col, v[c]);
            }
        }
    }

    const float inv_n = 1.0f / (float)cols;
    float mean = 0.f, rstd;
    {
        // One sweep over the registers. LayerNorm accumulates sum(x-K) and sum((x-K)^2) with K = the
        // warp's first element: shifting by a value of the row itself keeps the subtraction
        // E[(x-K)^2] - E[x-K]^2 well conditioned even when |mean| >> std (rows like -20 +- 0.5).
        float shift = 0.f;
        if (!RMS) shift = __shfl_sync(0xffffffffu, Elem<T>::unpack2(v[0].x).x, 0);
        // (two values per instruction: at 4096 columns a third of the issue slots went into this sweep and the
        // last one, and a LayerNorm row took a quarter longer than an RMSNorm row)
        // (RMSNorm keeps one scalar chain per lane: it needs half the instructions, and its order is kept, see CHAIN)
        float s1 = 0.f, s2 = 0.f;
        auto add_squares = [&]() {
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                if (KB_NORM_COL(c) < cols) {
                    const uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = Elem<T>::unpack2(w[i]);
                        s2 = fmaf(f.x, f.x, fmaf(f.y, f.y, s2));
                    }
                }
            }
        };
        if (CHAIN) {
#pragma unroll
            for (int w = 0; w < WPR; ++w) {
                if (wir == w) {
                    if (w > 0) s2 = chain_s[lane];
                    add_squares();
                    chain_s[lane] = s2;
                }
                __syncthreads();
            }
            s2 = chain_s[lane];
        } else if (RMS) {
            add_squares();
        } else {
            float2 p1 = make_float2(0.f, 0.f), p2 = make_float2(0.f, 0.f);
            const float2 neg_shift = make_float2(-shift, -shift);
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                if (KB_NORM_COL(c) < cols) {
                    const uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __fadd2_rn(Elem<T>::unpack2(w[i]), neg_shift);
                        p1 = __fadd2_rn(p1, f);
                        p2 = __ffma2_rn(f, f, p2);
                    }
                }
            }
            s1 = p1.x + p1.y;
            s2 = p2.x + p2.y;
        }
        s2 = warp_sum(s2);
        if (!RMS) s1 = warp_sum(s1);
        if (WPR > 1 && RMS && !CHAIN) {
            if (lane == 0) red_s[1][warp] = s2;
            __syncthreads();
            s2 = (red_s[1][0] + red_s[1][1]) + (red_s[1][2] + red_s[1][3]);
            if (WPR == 8) s2 += (red_s[1][4] + red_s[1][5]) + (red_s[1][6] + red_s[1][7]);
            s2 *= inv_n;
        } else if (WPR > 1 && !RMS) {
            // the warps of a row meet: their means and squared deviations, whose combination needs no common shift
            auto columns_of = [&](int w) {
                int n = 0;
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c) n += min(256, max(0, cols - (c * WPR + w) * 256));
                return (float)n;
            };
            if (lane == 0) {
                const float n = columns_of(warp), d = n > 0.f ? s1 / n : 0.f;
                red_s[0][warp] = shift + d;
                red_s[1][warp] = fmaxf(s2 - s1 * d, 0.f);
            }
            __syncthreads();
            float total = 0.f, m2 = 0.f;
#pragma unroll
            for (int w = 0; w < WPR; ++w) total = fmaf(columns_of(w), red_s[0][w], total);
            mean = total * inv_n;
#pragma unroll
            for (int w = 0; w < WPR; ++w) {
                const float d = red_s[0][w] - mean;
                m2 = fmaf(columns_of(w) * d, d, m2 + red_s[1][w]);
            }
            s2 = m2 * inv_n;
        } else {
            s2 *= inv_n;
            if (!RMS) {
                const float d = s1 * inv_n;
                mean = shift + d;
                s2 = fmaxf(s2 - d * d, 0.f);
            }
        }
        rstd = rsqrtf(s2 + eps);
    }
    if (lane == 0 && wir == 0) {
        if (mean_out) mean_out[row] = mean;
        if (rstd_out) rstd_out[row] = rstd;
    }

    const float2 rstd2 = make_float2(rstd, rstd), neg_mean = make_float2(-mean, -mean);
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        const int col = KB_NORM_COL(c);
        if (col < cols) {
            uint4 g, b = make_uint4(0, 0, 0, 0);
            if (kEarlyAffine) {
                g = gv[c];
                b = bv[c];
            } else {
                g = *reinterpret_cast<const uint4*>(gamma + col);
                if (!RMS && beta != nullptr) b = *reinterpret_cast<const uint4*>(beta + col);
            }
            const uint32_t xw[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
            const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
            const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
            uint32_t ow[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 xf = Elem<T>::unpack2(xw[i]);
                const float2 gf = Elem<T>::unpack2(gw[i]);
                float2 o = RMS ? __fmul2_rn(xf, rstd2) : __fmul2_rn(__fadd2_rn(xf, neg_mean), rstd2);
                o = RMS ? __fmul2_rn(o, gf) : __ffma2_rn(o, gf, Elem<T>::unpack2(bw[i]));
                ow[i] = Elem<T>::pack2(o.x, o.y);
            }
            st_stream_16B(yr + col, make_uint4(ow[0], ow[1], ow[2], ow[3]));
        }
    }
}

// Generic strided path: one warp per row, three sweeps over the row.
template <typename T, bool RMS>
__global__ void __launch_bounds__(128)
norm_fwd_generic_kernel(const T* __restrict__ x, T* __restrict__ y, const T* __restrict__ gamma,
                        const T* __restrict__ beta, float* __restrict__ mean_out,
                        float* __restrict__ rstd_out, int64_t rows, int64_t cols,
                        int64_t x_row_stride, int64_t x_col_stride, int64_t y_row_stride,
                        int64_t y_col_stride, float eps) {
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (row >= rows) return;
    const T* xr = x + row * x_row_stride;
    T* yr = y + row * y_row_stride;
    const float inv_n = 1.0f / (float)cols;
    float mean = 0.f;
    if (!RMS) {
        float s = 0.f;
        for (int64_t c = lane; c < cols; c += 32) s += Elem<T>::to_f32(xr[c * x_col_stride]);
        mean = warp_sum(s) * inv_n;
    }
    float s2 = 0.f;
    for (int64_t c = lane; c < cols; c += 32) {
        const float d = Elem<T>::to_f32(xr[c * x_col_stride]) - mean;
        s2 += d * d;
    }
    const float rstd = rsqrtf(warp_sum(s2) * inv_n + eps);
    if (lane == 0) {
        if (mean_out) mean_out[row] = mean;
        if (rstd_out) rstd_out[row] = rstd;
    }
    for (int64_t c = lane; c < cols; c += 32) {
        const float xv = Elem<T>::to_f32(xr[c * x_col_stride]);
        const float g = Elem<T>::to_f32(gamma[c]);
        const float b = (!RMS && beta != nullptr) ? Elem<T>::to_f32(beta[c]) : 0.f;
        yr[c * y_col_stride] = Elem<T>::from_f32((xv - mean) * rstd * g + b);
    }
}

template <typename T, bool RMS>
static int launch_norm_t(const kb_norm_params& p, cudaStream_t stream) {
    const T* x = (const T*)p.x;
    T* y = (T*)p.y;
    const T* g = (const T*)p.gamma;
    const T* b = (const T*)p.beta;
    constexpr int kWarps = 4;
    const unsigned grid = (unsigned)((p.rows + kWarps - 1) / kWarps);
    const bool vec_ok = p.x_col_stride == 1 && p.y_col_stride == 1 && (p.cols % 8) == 0 &&
                        (p.x_row_stride % 8) == 0 && (p.y_row_stride % 8) == 0 &&
                        ((uintptr_t)p.x % 16) == 0 && ((uintptr_t)p.y % 16) == 0 &&
                        ((uintptr_t)p.gamma % 16) == 0 &&
                        (p.beta == nullptr || ((uintptr_t)p.beta % 16) == 0) && p.cols <= kNormMaxCols;
#define KB_NORM_LAUNCH(C, W, ...)                                                                 \
    return launch_pdl(norm_fwd_rowwarp_kernel<T, C, RMS, W, ##__VA_ARGS__>, W == 1 ? grid : (unsigned)p.rows, W == 8 ? 256 : 128, 0, stream, \
                      x, y, g, b, p.mean, p.rstd, p.rows, (int)p.cols, p.x_row_stride, p.y_row_stride, p.eps,                  \
                      (const T*)p.residual, (T*)p.sum_out) == cudaSuccess ? KB_OK : KB_ERR_LAUNCH
    if (vec_ok && p.cols > 4096) {
        if (p.cols <= 3 * 2048) KB_NORM_LAUNCH(3, 8);
        if (p.cols <= 4 * 2048) KB_NORM_LAUNCH(4, 8);
        KB_NORM_LAUNCH(8, 8);
    }
    if (vec_ok && p.rows <= 64 && p.cols > 1024) {
        if (p.cols <= 2 * 1024) KB_NORM_LAUNCH(2, 4, false, true);
        if (p.cols <= 3 * 1024) KB_NORM_LAUNCH(3, 4, false, true);
        KB_NORM_LAUNCH(4, 4, false, true);
    }
    if (vec_ok && p.rows <= 1024) {
        if (p.cols <= 1024) KB_NORM_LAUNCH(1, 4);
        if (p.cols <= 2 * 1024) KB_NORM_LAUNCH(2, 4);
        if (p.cols <= 3 * 1024) KB_NORM_LAUNCH(3, 4);
        KB_NORM_LAUNCH(4, 4);
    }
    if (vec_ok && p.cols > 1024) {
        if (p.cols <= 2 * 1024) KB_NORM_LAUNCH(2, 4, RMS);
        if (p.cols <= 3 * 1024) KB_NORM_LAUNCH(3, 4, RMS);
        KB_NORM_LAUNCH(4, 4, RMS);
    }
    if (vec_ok) {
        if (p.cols <= 256) KB_NORM_LAUNCH(1, 1);
        if (p.cols <= 2 * 256) KB_NORM_LAUNCH(2, 1);
        if (p.cols <= 3 * 256) KB_NORM_LAUNCH(3, 1);
        KB_NORM_LAUNCH(4, 1);
    }
#undef KB_NORM_LAUNCH
    if (p.residual != nullptr) return KB_ERR_UNSUPPORTED;  // the fused add needs the vector layout
    return launch_pdl(norm_fwd_generic_kernel<T, RMS>, grid, kWarps * 32, 0, stream, x, y, g, b, p.mean, p.rstd, p.rows,
                      p.cols, p.x_row_stride, p.x_col_stride, p.y_row_stride, p.y_col_stride, p.eps) == cudaSuccess
               ? KB_OK : KB_ERR_LAUNCH;
}

static int launch_norm(const kb_norm_params& p, cudaStream_t stream) {
    if (p.dtype == KB_F16)
        return p.is_rms ? launch_norm_t<__half, true>(p, stream) : launch_norm_t<__half, false>(p, stream);
    if (p.dtype == KB_BF16)
        return p.is_rms ? launch_norm_t<__nv_bfloat16, true>(p, stream)
                        : launch_norm_t<__nv_bfloat16, false>(p, stream);
    return KB_ERR_UNSUPPORTED;
}

}  // namespace kb
