// Linear layer for up to about a thousand rows: one output tile per cluster, its K range divided among the
// cluster's CTAs. y = act(x · Wᵀ + bias).
//
// Bound: latency (a projection of BERT-base over 128 tokens moves 1-5 MB and takes 0.1 us of tensor time)
// and, for a large W, HBM. What such a launch pays for is the bytes each SM has to pull through its own
// port to L2 (a 128 x 32 tile over K = 768 pulled 245 KB, 2 us, on 24 of 148 SMs) and the passes around the
// products. So:
//   * W is the M = 128 operand of tcgen05.mma, x the N = 32, 64 or 128 one: a few rows waste no tensor
//     memory or shared memory on absent ones, and a tile of 128 x 128 reads the least per product;
//   * the K range of a tile goes to `splits` CTAs (one cluster, up to sixteen), so that every SM takes part
//     and each pulls little. The fp32 partial tiles meet in distributed shared memory: every CTA writes each
//     row of its part to the CTA that adds that row up, which applies bias and activation and stores it. (Reading
//     the others' parts instead waits for the cluster's memory twice per four values: 3700 to 6100 cycles, and a third barrier
//     before anybody may leave: [128, 3072] x [768, 3072] 6.9 us, 6.4 this way, [512, 3072] x [768, 3072] 10.2 and 9.5.) No workspace, no
//     atomics, no second launch (the split-K this replaces took 2.6 us for its finishing kernel alone and
//     added in no fixed order);
//   * two CTAs share an SM; barriers, tensor memory and descriptors are set up, and the first W tiles asked
//     for in L2, while the kernel ahead drains (programmatic dependent launch).
// Warps: 0 TMA producer, 1 tcgen05 issuer, 2..5 tensor memory -> shared memory; all six add and store.
#pragma once
#include "linear.cuh"
#include "linear_pair.cuh"
#include "linear_stream.cuh"

namespace kb {

constexpr int kClThreads = 192;
constexpr int kClMaxSplits = 16;

template <int NB>
struct ClCfg {  // NB: rows of x per tile
    static constexpr int kWBytes = 128 * kGemmBK * 2;
    static constexpr int kStageBytes = kWBytes + NB * kGemmBK * 2;
    static constexpr int kStages = NB == 128 ? 3 : NB == 64 ? 4 : 5;
    static constexpr int kSmemBytes = kStages * kStageBytes + 256 + 1024;
    static_assert((NB + kClMaxSplits - 1) * 128 * 4 <= kStages * kStageBytes, "the parts to be added up reuse the stages");
    static_assert(2 * (kSmemBytes + 1024) <= 227 * 1024, "two CTAs per SM");
};

// Into the shared memory of the cluster's CTA `rank`, at the place that has the address `own_addr` here.
__device__ __forceinline__ void st_cluster_f32(uint32_t own_addr, uint32_t rank, uint32_t v) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(own_addr), "r"(rank));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

template <typename T, int NB>
__global__ void __launch_bounds__(kClThreads, 2)
linear_cluster_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const T* __restrict__ bias,
                      T* __restrict__ y, T* __restrict__ act_inputs, int M, int N, int K, int64_t y_row_stride, int activation, int splits) {
    using Cfg = ClCfg<NB>;
    constexpr int STAGES = Cfg::kStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::kStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t smem_base = smem_u32(smem), bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    const uint32_t done_bar = bar_base + 8u * (2 * STAGES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % splits, tile = (int)blockIdx.x / splits;
    const int num_m = (M + NB - 1) / NB;
    const int m0 = (tile % num_m) * NB, n0 = (tile / num_m) * 128;  // the row tiles of one W tile are neighbours
    const int num_k = (K + kGemmBK - 1) / kGemmBK;
    const int kb0 = rank * num_k / splits, kb1 = (rank + 1) * num_k / splits;  // never empty: splits <= num_k

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmap_w);
        tma_prefetch_desc(&tmap_x);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(done_bar, 1);
        *abort_flag = 0;
        fence_mbar_init();
        // only a hint to L2: W may be the output of the kernel ahead, so nothing of it is read before the wait
        for (int kb = kb0; kb < min(kb1, kb0 + STAGES); ++kb) tma_prefetch_l2_2d(&tmap_w, kb * kGemmBK, n0);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), NB);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents();
    // set by a wait that expired in an earlier launch: nothing is stored then (looked at in the end, so that the
    // CTAs of a cluster, which may read it at different times, take the same way through its barriers)
    const int skip = status_word();

    // A thread adds up the same four columns in every row (its step is a multiple of a row's groups): their bias is asked for here, and
    // turned into fp32 where it is added: done here, that held the producer up until it had come (17 to 24 rows of [1024, 4096]: 0.3 us).
    const bool gated = activation == KB_ACT_SWIGLU;
    const int quads = gated ? 16 : 32;  // groups of four output columns of a tile row
    static_assert(kClThreads % 32 == 0, "whole rows of groups");
    unsigned short bias_lo[4], bias_up[4];
    {
        const unsigned short* b = reinterpret_cast<const unsigned short*>(bias);
        const int g = (int)threadIdx.x % quads, nl = n0 + (gated ? (g >> 1) * 16 + (g & 1) * 4 : g * 4);
        const int b_end = bias != nullptr ? N : 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            bias_lo[e] = nl + e < b_end ? __ldg(b + nl + e) : (unsigned short)0;
            bias_up[e] = gated && nl + 8 + e < b_end ? __ldg(b + nl + 8 + e) : (unsigned short)0;
        }
    }
    const int rows = min(NB, M - m0);            // rows of x in this tile: row m is added up by rank m % splits
    const int own = (NB + splits - 1) / splits;  // most rows of a rank
    bool complete = false;                       // an epilogue warp: this CTA's products are
    if (warp == 0) {
        if (elect_one()) {
            bool ok = true;
            for (int kb = kb0; kb < kb1 && ok; ++kb) {
                const int i = kb - kb0, s = i % STAGES;
                if (!mbar_wait(empty_bar(s), (uint32_t)((i / STAGES) & 1) ^ 1u, abort_flag, 130)) { ok = false; break; }
                mbar_arrive_expect_tx(full_bar(s), Cfg::kStageBytes);
                const uint32_t dst = smem_base + s * Cfg::kStageBytes;
                tma_load_2d(dst, &tmap_w, full_bar(s), kb * kGemmBK, n0);
                tma_load_2d(dst + Cfg::kWBytes, &tmap_x, full_bar(s), kb * kGemmBK, m0);
            }
            if (!ok) {
                for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies in flight land
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc_f16(Elem<T>::kIsBf16, 128, NB, 0, 0);
            bool ok = true;
            for (int kb = kb0; kb < kb1; ++kb) {
                const int i = kb - kb0, s = i % STAGES;
                if (!mbar_wait(full_bar(s), (uint32_t)((i / STAGES) & 1), abort_flag, 230)) { ok = false; break; }
                tc_fence_after();
                const uint32_t a_addr = smem_base + s * Cfg::kStageBytes;
                const uint64_t a_desc = make_smem_desc_sw128(a_addr, 16, 1024);
                const uint64_t b_desc = make_smem_desc_sw128(a_addr + Cfg::kWBytes, 16, 1024);
#pragma unroll
                for (int k = 0; k < kGemmBK / 16; ++k) tc_mma_ss(tmem_base, a_desc + 2 * k, b_desc + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                tc_commit(empty_bar(s));
            }
            if (ok) tc_commit(done_bar);
        }
    } else {
        complete = __all_sync(0xffffffffu, mbar_wait(done_bar, 0, abort_flag, 330));
    }
    // Once every CTA's products are complete the stages are free in all of them: the rows' parts go there, [rank][row / splits][W row].
    __syncwarp();
    cluster_arrive();
    const int q = warp & 3;  // tensor-memory quadrant: 32 rows of W
    const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16);
    uint32_t r[32];
    if (complete) {
        tc_fence_after();
        tmem_ld_32x32(t_addr, r);
        tmem_ld_wait();
    }
    __syncwarp();
    cluster_wait();
    if (complete) {
        const uint32_t to = smem_base + (uint32_t)((rank * own * 128 + q * 32 + lane) * 4);
        int owner = 0, at = 0;
#pragma unroll 1
        for (int c0 = 0; c0 < rows; c0 += 32) {
            if (c0 > 0) {
                tmem_ld_32x32(t_addr + (uint32_t)c0, r);
                tmem_ld_wait();
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (c0 + j < rows) st_cluster_f32(to + (uint32_t)(at * 512), (uint32_t)owner, r[j]);
                if (++owner == splits) { owner = 0; ++at; }
            }
        }
        tc_fence_before();
    }
    __syncwarp();
    cluster_sync_all();  // (nobody reads or writes another CTA's memory behind this)

    // ---- this CTA's rows of the tile: four outputs per thread, summed in rank order
    const int total = rows > rank ? (rows - rank + splits - 1) / splits * quads : 0;
    for (int i = (int)threadIdx.x; i < total; i += kClThreads) {
        const int at = i / quads, m = at * splits + rank, q = i % quads;
        // gated: W rows in blocks of eight gate and eight up rows; outputs 8 j .. from gate rows 16 j .., up rows 16 j + 8 ..
        const int nl = gated ? (q >> 1) * 16 + (q & 1) * 4 : q * 4;
        auto sum4 = [&](int n_local, const unsigned short (&b4)[4], float (&z)[4]) {
            const float* part = reinterpret_cast<const float*>(smem) + at * 128 + n_local;
            z[0] = z[1] = z[2] = z[3] = 0.f;
            for (int s = 0; s < splits; s += 4) {  // four loads on their way before the first is added
                float4 f[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) f[e] = *reinterpret_cast<const float4*>(part + min(s + e, splits - 1) * own * 128);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (s + e < splits) { z[0] += f[e].x; z[1] += f[e].y; z[2] += f[e].z; z[3] += f[e].w; }
            }
            if (bias != nullptr) {
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const float2 b2 = Elem<T>::unpack2((uint32_t)b4[e] | ((uint32_t)b4[e + 1] << 16));
                    z[e] += b2.x;
                    z[e + 1] += b2.y;
                }
            }
        };
        if (n0 + nl >= N) continue;
        float z[4];
        sum4(nl, bias_lo, z);
        const int64_t row = (int64_t)(m0 + m) * y_row_stride;
        int n_out = n0 + nl, left = N - n_out;
        if (gated) {
            float up[4];
            sum4(nl + 8, bias_up, up);
#pragma unroll
            for (int e = 0; e < 4; ++e) z[e] = act_silu(z[e]) * up[e];
            n_out = (n0 >> 1) + (q >> 1) * 8 + (q & 1) * 4;
            left = 4;
        } else {
            if (act_inputs != nullptr && skip == 0)
                for (int e = 0; e < 4 && e < left; ++e) act_inputs[row + n_out + e] = Elem<T>::from_f32(z[e]);
            apply_activation(z, activation);
        }
        if (skip != 0) continue;
        T* dst = y + row + n_out;
        if (left >= 4 && (((uintptr_t)dst) & 7) == 0) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(Elem<T>::pack2(z[0], z[1]), Elem<T>::pack2(z[2], z[3]));
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (e < left) dst[e] = Elem<T>::from_f32(z[e]);
        }
    }
    __syncwarp();
    if (warp == 1) tmem_dealloc(tmem_base, NB);
}

// Clusters that are resident at once on the current device, by size (asked once per device; null: no device).
// A plain pointer to the table: a plan looks at all sizes of three kernels, and a lock and a device query for
// each of them were 2.5 us of host time per call.
template <typename T, int NB>
static const int* linear_cluster_resident() {
    static int resident[64][kClMaxSplits + 1] = {};
    static std::atomic<bool> known[64] = {};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (known[dev].load(std::memory_order_acquire)) return resident[dev];
    std::lock_guard<std::mutex> lock(mu);
    if (!known[dev].load(std::memory_order_relaxed)) {
        auto* kernel = linear_cluster_kernel<T, NB>;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ClCfg<NB>::kSmemBytes) != cudaSuccess ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return nullptr;
        cudaLaunchConfig_t cfg = {};
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = ClCfg<NB>::kSmemBytes;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        for (int s = kClMaxSplits; s >= 1; --s) {
            int n = 0;
            cfg.gridDim = dim3((unsigned)s);
            attr[0].val.clusterDim.x = (unsigned)s;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
                cudaGetLastError();
                n = s > 8 ? 0 : 1;  // (not every device takes the large ones)
            }
            resident[dev][s] = n;
        }
        known[dev].store(true, std::memory_order_release);
    }
    return resident[dev];
}

template <typename T, int NB>
static int launch_linear_cluster(const kb_linear_params& p, cudaStream_t stream, int splits) {
    const int* table = linear_cluster_resident<T, NB>();  // (also sets the kernel's attributes)
    if (table == nullptr || table[splits] == 0) return KB_ERR_LAUNCH;
    CUtensorMap tmap_w, tmap_x;
    {
        const uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)p.N};
        const uint64_t strides[2] = {0, (uint64_t)p.K * 2};
        const uint32_t box[2] = {kGemmBK, 128};
        const int st = encode_tmap_16bit(&tmap_w, p.w, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (st != KB_OK) return st;
    }
    {
        const uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)p.M};
        const uint64_t strides[2] = {0, (uint64_t)p.x_row_stride * 2};
        const uint32_t box[2] = {kGemmBK, NB};
        const int st = encode_tmap_16bit(&tmap_x, p.x, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (st != KB_OK) return st;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(((p.M + NB - 1) / NB) * ((p.N + 127) / 128) * splits));
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = ClCfg<NB>::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_use_pdl ? 2u : 1u;
    return cudaLaunchKernelEx(&cfg, linear_cluster_kernel<T, NB>, tmap_w, tmap_x, (const T*)p.bias, (T*)p.y, (T*)p.act_inputs, (int)p.M, (int)p.N,
                              (int)p.K, p.y_row_stride, p.activation, splits) == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

template <typename T>
static int launch_linear_cluster_n(const kb_linear_params& p, cudaStream_t stream, int nb, int splits) {
    if (nb == 32) return launch_linear_cluster<T, 32>(p, stream, splits);
    if (nb == 64) return launch_linear_cluster<T, 64>(p, stream, splits);
    return launch_linear_cluster<T, 128>(p, stream, splits);
}


// ---- which kernel a problem goes to
//
// Estimates in us, fitted to times of the kernels (graphs of calls with cold W). Above 128 rows, at 1170 problems that the fit has not
// seen (129 to 8192 rows, K and N from 256 to 11008, every activation): the chosen kernel is 0.5 % slower than the fastest one on
// average, at 6 % of them by more than 3 %, at 1.5 % by more than 10. (Estimates fitted to some thirty problems, before the kernels' epilogues
// changed, and bent towards the new ones since: 1.6 % on average, 13 % and 7 %; 3 % of the problems were slower than with the earlier kernels
// and their own estimates, [129, 256] x [11008, 256] by 32 %, [2000, 8192] x [1024, 8192] by 22.) Up to 128 rows an SM pulls about
// 118 bytes per ns through its port to L2, shared by its CTAs; W comes from HBM at 6.5 bytes per ps at best.
struct ClusterPlan {
    int nb, splits;
    double us;
};
template <typename T>
static ClusterPlan linear_cluster_plan(const kb_linear_params& p) {
    ClusterPlan best{0, 0, 1e300};
    const int64_t num_k = (p.K + kGemmBK - 1) / kGemmBK, num_n = (p.N + 127) / 128;
    const double w_bytes = (double)p.N * (double)p.K * 2.0, hbm = w_bytes / 6.5e6;
    for (int nb : {32, 64, 128}) {
        if (nb == 32 ? p.M > 256 : nb == 64 ? p.M <= 32 : p.M <= 64) continue;
        const int64_t tiles = ((p.M + nb - 1) / nb) * num_n;
        const int* table = nb == 32 ? linear_cluster_resident<T, 32>() : nb == 64 ? linear_cluster_resident<T, 64>() : linear_cluster_resident<T, 128>();
        if (table == nullptr) continue;
        // Powers of two: they pack the GPU's clusters of SMs and divide the sums of the epilogue, which take four partial
        // tiles at a time, evenly. (Five CTAs per tile at 512 rows of [768, 3072]: 13.1 us, four: 10.7.)
        for (int s = 1; s <= kClMaxSplits && s <= num_k; s *= 2) {
            const int resident = table[s];
            if (resident == 0) continue;
            const double waves = (double)((tiles + resident - 1) / resident);
            // two CTAs meet on an SM before every SM has one: clusters do not fill all of them
            const bool shared_sm = (tiles < resident ? tiles : resident) * s > sm_count() * 7 / 8;
            const double rows = (double)(p.M < nb ? p.M : nb);
            const double load = (double)((num_k + s - 1) / s) * (16384.0 + rows * 128.0) / (shared_sm ? 85e3 : 100e3);
            const double body = waves * load > hbm ? waves * load : hbm;
            const double sums = 0.0203 * rows * (double)((s + 3) / 4 * 4) / (double)s * (shared_sm ? 2.0 : 1.0);
            const double us = 3.9 + (w_bytes > 8e6 ? 2.0 : 0.0) + body + waves * sums;
            if (us < best.us) best = ClusterPlan{nb, s, us};
        }
    }
    return best;
}
static double linear_single_us(const kb_linear_params& p) {
    const int bn = plan_linear_bn(p.M, p.N, p.K, 0);
    const int64_t tiles = ((p.M + kGemmBM - 1) / kGemmBM) * ((p.N + bn - 1) / bn);
    const double waves = (double)((tiles + gemm_sms() - 1) / gemm_sms());
    if (p.M > 128) {
        static constexpr GemmCost kTile[4] = {{2.7, 0.0, 0.146, 0.020, 0.25, 0.15, -0.2, 0.25, 0.35, 0.1, 3.5}, {2.6, 0.1, 0.159, 0.018, 1.1, 0.36, -0.75, 0.40, 0.70, 0.5, 8.3},
                                              {3.4, 0.55, 0.220, 0.025, 0.62, 0.74, -1.2, 0.38, 1.05, 1.0, 17.0}, {2.7, 1.1, 0.357, 0.090, 2.4, 1.2, -1.7, 0.26, 0.80, 2.7, 32.0}};
        return gemm_us(kTile[bn == 32 ? 0 : bn == 64 ? 1 : bn == 128 ? 2 : 3], p, tiles, gemm_sms(), p.act_inputs != nullptr);
    }
    // An SM's port gives 118 bytes per ns, narrow tiles pull faster (512 rows of [768, 3072], 32 columns: 9.9 us, 11.5 at that
    // rate), rows that are no multiple of 128 bytes take longer. An epilogue stores a column of a tile in 0.012 us by whole
    // 16-byte pieces, in 0.05 value by value. A tile of which most rows lie outside x arrives later (zero fill): 5.5 us at
    // 128 rows of [3072, 768], 6.9 at 33.
    const double load = (double)(kGemmBM + bn) * (double)p.K * 2.0 / (bn <= 64 ? 150e3 : 118e3) * (p.K % kGemmBK != 0 ? 1.8 : 1.0);
    return 2.8 + (p.M < 96 ? 1.3 : 0.0) + waves * (load + (linear_stores_values(p) ? 0.05 : 0.012) * bn);
}
template <typename T>
static int launch_linear_t(const kb_linear_params& p, cudaStream_t stream, int forced_bn, int forced_splits, const RopeDev* rope, bool* roped) {
    // `rope`: the rotary embedding and cache write that follow; *roped says that the projection's kernel has done them
    const RopeDev* in_pair = rope != nullptr && linear_pair_rope(p, *rope) ? rope : nullptr;
    if (forced_splits > 1) {
        const int num_k = (int)((p.K + kGemmBK - 1) / kGemmBK), most = num_k < kClMaxSplits ? num_k : kClMaxSplits;
        const int nb = forced_bn == 32 || forced_bn == 64 ? forced_bn : p.M <= 64 ? 32 : 128;
        return launch_linear_cluster_n<T>(p, stream, nb, forced_splits < most ? forced_splits : most);
    }
    if (forced_bn != 0) return launch_linear_single<T>(p, stream, forced_bn);
    if (stream_layout(p) && p.M <= 16) return launch_linear_stream_t<T>(p, stream);
    const double single = linear_single_us(p);
    const ClusterPlan cl = p.M <= 1024 && g_linear_pair == 1 && gemm_sms() == sm_count() ? linear_cluster_plan<T>(p) : ClusterPlan{0, 0, 1e300};
    if (p.M > 128 && p.N >= 128 && p.K >= 256 && g_linear_pair != 0) {
        double pair;
        int bn = linear_pair_tile_width(p, &pair);
        if (in_pair != nullptr && g_linear_pair == 1) {
            // The rotary epilogue has the wide tile only, and saves a launch that reads and writes the result (402 MB in 74 us at 8192 rows of
            // [12288, 4096]) for some work of its own. Where the narrow tile is faster by more than that, the launch stays: prompts of 141 and 198
            // tokens, four and three layers, 673 us for 694 and 524 for 538.
            const double wide = linear_pair_us(p, 256) + 2.0 - (double)p.M * (double)p.N * 4.0 / 5.5e6;
            if (bn == 256 || wide < pair) {
                bn = 256;
                pair = wide;
            }
        }
        if (g_linear_pair != 1 || pair < single) {
            if (pair <= cl.us) {
                const RopeDev* fused = bn == 256 ? in_pair : nullptr;
                if (fused != nullptr) *roped = true;
                return launch_linear_pair_t<T>(p, stream, bn, fused);
            }
        }
    }
    if (p.M <= 1024 && gemm_sms() == sm_count()) {
        const double stream_us = stream_layout(p) && p.M <= 512 ? stream_plan_x(p).us : 1e300;
        if (p.M <= 128) {
            // (the streaming kernel's estimate is a tenth high for few rows: 5.5 us for 5.0 at 33 rows of [3072, 768], the cluster's 5.3 for 5.4)
            if (stream_us < single && stream_us < 1.05 * cl.us) return launch_linear_stream_t<T>(p, stream);
            // (ahead by more than a trifle: where the two are close, the cluster's estimate is the less certain one)
            if (cl.us < 0.97 * single) return launch_linear_cluster_n<T>(p, stream, cl.nb, cl.splits);
        } else {
            // (here the streaming kernel's is a little low, for gated calls high, 4.3 us for 2.8 at 150 rows of [256, 360], and does not know
            // what values stored one by one cost it: 30 us at 200 rows of [8192, 512], 22 with single CTAs)
            const double likely = stream_us * (p.activation == KB_ACT_SWIGLU ? 0.9 : 1.05) + (linear_stores_values(p) ? 8e-6 * (double)p.M * (double)p.N : 0.0);
            if (likely < single && likely < 1.1 * cl.us) return launch_linear_stream_t<T>(p, stream);
            if (cl.us < single) return launch_linear_cluster_n<T>(p, stream, cl.nb, cl.splits);
        }
    }
    return launch_linear_single<T>(p, stream, 0);
}

static int launch_linear(const kb_linear_params& p, cudaStream_t stream, int forced_bn, int forced_splits, const RopeDev* rope = nullptr,
                         bool* roped = nullptr) {
    if (p.dtype == KB_F16) return launch_linear_t<__half>(p, stream, forced_bn, forced_splits, rope, roped);
    if (p.dtype == KB_BF16) return launch_linear_t<__nv_bfloat16>(p, stream, forced_bn, forced_splits, rope, roped);
    return KB_ERR_UNSUPPORTED;
}

}  // namespace kb
