// Fused attention forward for sm_100a: O = softmax(sm_scale·Q·Kᵀ + mask [causal]) · V.
//
// One CTA owns TWO query tiles of 128 rows of one (batch, head) and streams the keys/values in
// blocks of 128. Roles (384 threads = 3 warpgroups):
//   warps 0..3    softmax group of tile 0 (one query row per thread)
//   warps 4..7    softmax group of tile 1
//   warp 8        TMA producer: both Q tiles once, then the K and V blocks through two small rings
//   warp 9        tcgen05 issuer (one elected thread):  S_t = Q_t·K_jᵀ  (operands in shared memory)
//                 and  O_t += P_t·V_j  (P read from TMEM, V from shared memory, N-major)
//   warps 10..11  idle (they only give their registers away)
// The third warpgroup shrinks its register allowance (setmaxnreg) so that the softmax threads can
// hold a whole 128-wide score row in registers.
// While one group runs its exponentials, the tensor core works on the other tile (ping-pong).
// Without a mask, in launches of more pairs of query tiles than SMs (MODE 0), a CTA stays for the whole launch, one per SM: further items (pairs of query tiles) come from a
// device-side counter, the issuer starts an item's scores while the softmax warps store the one before, and every barrier's
// phase counts on over the items. A CTA per item spent 12 000 of 45 000 to 67 000 cycles on setting itself up, its first
// loads, its stores and its end (all of an SM's tensor memory and shared memory are one CTA's). [4, 32 over 8, 2048, 128]
// causal 174 -> 149 us (with the hand-over of P below), [16, 16, 512, 128] 61 -> 46, [2, 32, 4096, 128] 463 -> 440; same bits.
// A launch without a second item per SM (MODE 4) has one CTA per item and none of that.
// TMEM columns: S_0 [0,128)  S_1 [128,256)  O_0 [256,256+D)  O_1 [384,384+D); P_t (16-bit, two
// per column) overwrites the first 64 columns of S_t once the thread has its row in registers.
//
// Online softmax in the log2 domain with LAZY rescaling: the running reference maximum of a row
// only moves (and O is only rescaled in TMEM) when the true maximum has grown by more than 2^8,
// so P stays below 256 — exactly representable range for fp16/bf16 — and most iterations skip
// the O round trip. The final O is divided by the fp32 row sum.
//
// Semantics follow src/kernl/implementations/attention.py:122-435 of the reference: scale before
// mask (:345), additive mask with -inf clamped to the lowest finite value of the mask's dtype
// (:380,:516), causal = keep col <= row, top-left aligned (:347), P rounded to the input dtype
// before P·V (:424), fp32 statistics and accumulation (:290-295).
#pragma once
#include "common.cuh"

namespace kb {

constexpr int kAttnThreads = 384;
constexpr int kAttnBlock = 128;  // rows per query tile and keys per block
constexpr int kBlkN = 64;        // keys per block of the head-dimension-64 kernel (attention_split.cuh)
// Register re-balancing between the warpgroups (setmaxnreg). The CTA is launched with
// 65536 / 384 -> 168 registers per thread; the third warpgroup shrinks to attn_regs_low() and the two
// softmax warpgroups grow to attn_regs_high(). The increase waits (without bound) until the CTA's own
// pool has the registers, so the totals MUST fit the launch allocation: 2*high + low <= 3*168.
constexpr int kAttnRegsLaunch = 168;
// (The issuer and producer of the persistent form, MODE 0, keep more counters than 72 registers hold.)
__host__ __device__ constexpr int attn_regs_low(int mode) { return mode == 0 ? 104 : 72; }
__host__ __device__ constexpr int attn_regs_high(int mode) { return mode == 0 ? 200 : 216; }
static_assert(2 * attn_regs_high(0) + attn_regs_low(0) <= 3 * kAttnRegsLaunch && 2 * attn_regs_high(1) + attn_regs_low(1) <= 3 * kAttnRegsLaunch,
              "setmaxnreg totals exceed the CTA's register pool");
static_assert(attn_regs_low(0) % 8 == 0 && attn_regs_high(0) % 8 == 0 && attn_regs_low(1) % 8 == 0 && attn_regs_high(1) % 8 == 0,
              "setmaxnreg wants multiples of 8");
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLazyThreshold = 8.0f;

// Work queues of the persistent kernels. A launch has a slot and its CTAs draw tile numbers
// from slot[0]; slot[1] counts CTAs that have finished, and the last one puts both words back to
// zero, so a slot is clean again when its launch ends — also when the launch gave up on an expired
// wait. Eager launches take theirs from a ring: two would have to be in flight kAttnQueueSlots launches apart to share one.
// A captured launch comes again whenever its graph is replayed, beside the calls of other streams, so it owns its slot for as long as
// the graph, or one instantiated or cloned from it, exists. (A graph that is only used to update another's instantiation has to outlive that.)
constexpr int kAttnQueueSlots = 1024, kAttnGraphSlots = 65536;
__device__ unsigned int g_attn_queue[kAttnQueueSlots + kAttnGraphSlots][2];

struct AttnSlots {  // of one device
    std::atomic<unsigned int*> base{nullptr};  // g_attn_queue there (the symbol is a host-side handle)
    std::atomic<unsigned> next{0};             // the eager ring
    std::atomic<unsigned> from{0};             // where the next search begins
    std::atomic<int> held{0};                  // slots that graphs own
    std::atomic<uint64_t> owned[kAttnGraphSlots / 64] = {};
};
static AttnSlots g_attn_slots[64];
static int g_attn_graph_slots = kAttnGraphSlots;  // test hook (kb_debug_attention_slots)
static std::atomic<int> g_attn_last_slot{-1};     // likewise

// A free slot of the captured launches' pool, now owned; -1: none.
static int attention_own_slot(AttnSlots& d) {
    const unsigned words = (unsigned)(g_attn_graph_slots + 63) / 64, first = words > 0 ? d.from.load() % words : 0;
    for (unsigned n = 0; n < words; ++n) {
        const unsigned w = (first + n) % words;
        uint64_t seen = d.owned[w].load();
        while (~seen != 0) {
            const int bit = __builtin_ctzll(~seen);
            if ((int)(w * 64) + bit >= g_attn_graph_slots) break;
            if (d.owned[w].compare_exchange_weak(seen, seen | (1ull << bit))) {
                d.from.store(w);
                d.held.fetch_add(1);
                return (int)(w * 64) + bit;
            }
        }
    }
    return -1;
}
// The last graph that owned a slot is gone (called by CUDA on a thread of its own, after the last replay has ended).
static void CUDART_CB attention_free_slot(void* which) {
    const uintptr_t id = (uintptr_t)which - 1;
    AttnSlots& d = g_attn_slots[id / kAttnGraphSlots];
    const unsigned slot = (unsigned)(id % kAttnGraphSlots);
    d.owned[slot / 64].fetch_and(~(1ull << (slot % 64)));
    d.held.fetch_sub(1);
}

// A queue slot on the current device for a launch into `stream`. nullptr: none (as many captured launches as there are slots; the caller
// has a form that does not draw), or no device.
static unsigned int* attention_queue_slot(cudaStream_t stream) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return nullptr;
    }
    AttnSlots& d = g_attn_slots[dev];
    unsigned int* base = d.base.load(std::memory_order_acquire);
    if (base == nullptr) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_attn_queue) != cudaSuccess || ptr == nullptr) {
            cudaGetLastError();
            return nullptr;
        }
        base = reinterpret_cast<unsigned int*>(ptr);
        d.base.store(base, std::memory_order_release);
    }
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo_v2(stream, &capture, nullptr, &graph) != cudaSuccess) {  // (the legacy stream while another one is captured: the launch will say so)
        cudaGetLastError();
        capture = cudaStreamCaptureStatusNone;
    }
    if (capture == cudaStreamCaptureStatusNone) {
        const int slot = (int)(d.next.fetch_add(1) % (unsigned)kAttnQueueSlots);
        g_attn_last_slot.store(slot, std::memory_order_relaxed);
        return base + 2 * slot;
    }
    const int slot = attention_own_slot(d);
    if (slot < 0) return nullptr;
    const uintptr_t id = (uintptr_t)dev * kAttnGraphSlots + (uintptr_t)slot;
    cudaUserObject_t owner = nullptr;
    if (cudaUserObjectCreate(&owner, reinterpret_cast<void*>(id + 1), attention_free_slot, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        cudaGetLastError();
        attention_free_slot(reinterpret_cast<void*>(id + 1));
        return nullptr;
    }
    if (graph == nullptr || cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaGetLastError();
        cudaUserObjectRelease(owner, 1);  // (gives the slot back)
        return nullptr;
    }
    g_attn_last_slot.store(kAttnQueueSlots + slot, std::memory_order_relaxed);
    return base + 2 * (kAttnQueueSlots + slot);
}

struct AttnDev {
    void* o;
    const void* mask;
    int64_t o_strides[4];
    int64_t mask_strides[4];
    int B, H, M, N;
    float scale_log2;  // sm_scale * log2(e)
    int is_causal;
    int mask_dtype;
    int mask_vec;   // mask rows can be read with aligned 128-bit loads
    int mask_lead;  // the mask's address modulo 16 (head dimension 64, staged per-row masks)
    int num_pairs;  // ceil(ceil(M/128)/2)
    int o_bulk;     // persistent kernels: the result leaves through bulk tensor stores
    int head_group; // heads whose CTAs are interleaved (see attn_work_item)
    int kv_group;   // query heads per K/V head (grouped-query attention), >= 1
    int d_out;      // head dimension of the caller's tensors (a multiple of 8, at most the kernel's D): the
                    // tensor maps end there — TMA fills the columns beyond with zeros, which add nothing to
                    // q·kᵀ — and only these output columns are stored
};

// Stores 32 output columns [col0, col0 + 32) of one row. GUARD: the caller's head dimension ends
// inside or before the chunk (d_out < col0 + 32), so only whole 8-column pieces below d_out are
// written; the unguarded form is the hot path and carries no per-store condition (a guard inside the
// store loop of the head-dimension-64 kernel cost 2.7 µs of a 21 µs launch).
template <typename T, bool GUARD>
__device__ __forceinline__ void attn_store_32(T* __restrict__ o_row, int col0, int64_t col_stride, bool vec,
                                              const float (&val)[32], int d_out) {
    if (vec) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            if (GUARD && col0 + v * 8 >= d_out) continue;
            uint4 w;
            w.x = Elem<T>::pack2(val[v * 8 + 0], val[v * 8 + 1]);
            w.y = Elem<T>::pack2(val[v * 8 + 2], val[v * 8 + 3]);
            w.z = Elem<T>::pack2(val[v * 8 + 4], val[v * 8 + 5]);
            w.w = Elem<T>::pack2(val[v * 8 + 6], val[v * 8 + 7]);
            reinterpret_cast<uint4*>(o_row + col0)[v] = w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {  // (fully unrolled: val stays in registers)
            if (GUARD && col0 + i >= d_out) continue;
            o_row[(int64_t)(col0 + i) * col_stride] = Elem<T>::from_f32(val[i]);
        }
    }
}

// Work item (a CTA's number, or one drawn from a queue) -> (batch*head, query-tile pair). Heads are taken in groups of p.head_group; inside a group
// the order is pair-major with the late (causally heavier) pairs first, so the tail of a causal
// launch is made of light tiles, and consecutive CTAs are different heads of the same group. The
// group is sized on the host so that the K/V of all its heads (what the resident CTAs stream) stay
// in L2: with one group over all heads, 148 resident CTAs of a long-sequence launch streamed the
// K/V of 148 heads and DRAM read traffic was ten times the algorithmic bytes.
__device__ __forceinline__ void attn_work_item(const AttnDev& p, int BH, int idx, int& bh, int& pair) {
    const int per_group = p.num_pairs * p.head_group;
    const int g = idx / per_group;
    const int rem = idx % per_group;
    const int first = g * p.head_group;
    const int gsz = min(p.head_group, BH - first);
    pair = p.num_pairs - 1 - rem / gsz;
    bh = first + rem % gsz;
}
static int attn_head_group(int64_t BH, int64_t N, int64_t D) {
    const int64_t kv_bytes = 2 * N * D * 2;
    int64_t g = ((int64_t)32 << 20) / (kv_bytes > 0 ? kv_bytes : 1);
    if (g < 1) g = 1;
    if (g > BH) g = BH;
    return (int)g;
}

// Bulk stores want rows, heads and batches of the result at whole 16 bytes; anything else is stored by the threads.
static bool attn_bulk_out(const kb_attn_params& p) {
    const int64_t extent[3] = {p.B, p.H, p.M};
    bool whole = p.o_strides[3] == 1 && (((uintptr_t)p.o) & 15) == 0;
    for (int i = 0; i < 3; ++i) whole = whole && (extent[i] == 1 || (p.o_strides[i] > 0 && p.o_strides[i] % 8 == 0));
    return whole;
}

template <int D>
struct AttnCfg {
    static constexpr int kKvStages = 2;
    static constexpr int kTileBytes = kAttnBlock * D * 2;  // one Q tile / one K block / one V block
    static constexpr int kSmemBase = (2 + 2 * kKvStages) * kTileBytes + 512 + 1024;
    static constexpr int kMaskMaxN = 7168;  // MODE 1: the longest mask row that fits behind the tiles
    static constexpr int kMaskRingBytes = 2 * 2 * kAttnBlock * 4;  // MODE 3
    static constexpr int kOutWarpBytes = 32 * 64 * 2;  // MODE 0 and 4: 32 rows x 64 columns of results per softmax warp, a box of one bulk store
    static constexpr int kOutOffset = (2 + 2 * kKvStages) * kTileBytes + 1024;
    static constexpr int kSmemNoMask = kOutOffset + 8 * kOutWarpBytes + 1024;
    static_assert(kSmemNoMask <= 227 * 1024 - 256, "shared memory of one CTA");
    static constexpr int kSmemMax = kSmemBase + kMaskMaxN * 4;
    static_assert(kSmemMax <= 227 * 1024 - 256, "shared memory of one CTA");
};

__device__ __forceinline__ float mask_lowest(int mask_dtype) {
    if (mask_dtype == KB_F16) return -65504.0f;
    if (mask_dtype == KB_BF16) return -3.3895313892515355e38f;
    return -3.4028234663852886e38f;
}

__device__ __forceinline__ float mask_load(const void* base, int64_t off, int mask_dtype) {
    if (mask_dtype == KB_F16) return __half2float(reinterpret_cast<const __half*>(base)[off]);
    if (mask_dtype == KB_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[off]);
    return reinterpret_cast<const float*>(base)[off];
}

// NV consecutive values of one mask row from `off` on, of which the first `n` exist (the rest read as 0). The
// type is looked at once and every load is issued before the first value is used: with the type looked
// at per value, each of a row's loads waited for the one before it (one 64-key block of a mask with odd
// row strides: 3.3 us).
template <typename MT, int NV>
__device__ __forceinline__ void mask_values_t(const MT* __restrict__ row, int64_t stride, int n, float (&out)[NV]) {
    MT raw[NV];
    if (stride == 1 && n >= NV) {
#pragma unroll
        for (int i = 0; i < NV; ++i) raw[i] = __ldg(row + i);
    } else {
#pragma unroll
        for (int i = 0; i < NV; ++i) raw[i] = i < n ? __ldg(row + (int64_t)i * stride) : MT(0.f);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) out[i] = (float)raw[i];
}
template <int NV>
__device__ __forceinline__ void mask_values(const AttnDev& p, int64_t row_off, int col, float (&out)[NV]) {
    static_assert(NV % 8 == 0, "whole 128-bit loads");
    const int64_t off = row_off + (int64_t)col * p.mask_strides[3];
    if (p.mask_vec && col + NV <= p.N) {
        if (p.mask_dtype == KB_F32) {
            const float4* mp = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.mask) + off);
#pragma unroll
            for (int v4 = 0; v4 < NV / 4; ++v4) {
                const float4 f = __ldg(mp + v4);
                out[v4 * 4 + 0] = f.x; out[v4 * 4 + 1] = f.y; out[v4 * 4 + 2] = f.z; out[v4 * 4 + 3] = f.w;
            }
        } else {
            const uint4* mp = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.mask) + off);
#pragma unroll
            for (int v4 = 0; v4 < NV / 8; ++v4) {
                const uint4 w = __ldg(mp + v4);
                const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = (p.mask_dtype == KB_F16) ? Elem<__half>::unpack2(ww[i]) : Elem<__nv_bfloat16>::unpack2(ww[i]);
                    out[v4 * 8 + 2 * i] = f.x;
                    out[v4 * 8 + 2 * i + 1] = f.y;
                }
            }
        }
    } else if (p.mask_dtype == KB_F16) {
        mask_values_t(reinterpret_cast<const __half*>(p.mask) + off, p.mask_strides[3], p.N - col, out);
    } else if (p.mask_dtype == KB_BF16) {
        mask_values_t(reinterpret_cast<const __nv_bfloat16*>(p.mask) + off, p.mask_strides[3], p.N - col, out);
    } else {
        mask_values_t(reinterpret_cast<const float*>(p.mask) + off, p.mask_strides[3], p.N - col, out);
    }
}

__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Key blocks of a MODE 1 launch whose mask is "minus infinity" for every key (the padding behind a
// sequence) contribute exp(-65504 + ...) = 0 to every row and are skipped: not loaded, not multiplied,
// not exponentiated. A block is skipped only if all of its mask values are below kSkipBelow (in the
// log2 domain), far beyond where fp32 exp underflows for any score difference up to 2^14; if the
// whole row is like that (a fully padded sequence, where the mask cancels and the reference
// returns a plain softmax) nothing is skipped. At most 128 blocks (N <= 8192): a 128-bit set.
constexpr float kSkipBelow = -30000.0f * 1.4426950408889634f;
__device__ __forceinline__ int bits_next(const uint32_t (&w)[4], int from) {  // smallest set bit >= from
    int r = 1 << 20;
#pragma unroll
    for (int wi = 3; wi >= 0; --wi) {
        uint32_t m = w[wi];
        const int lo = from - wi * 32;
        if (lo >= 32) m = 0u;
        else if (lo > 0) m &= 0xffffffffu << lo;
        if (m != 0u) r = wi * 32 + __ffs((int)m) - 1;
    }
    return r;
}
__device__ __forceinline__ int bits_count_below(const uint32_t (&w)[4], int limit) {  // set bits with index < limit
    int n = 0;
#pragma unroll
    for (int wi = 0; wi < 4; ++wi) {
        const int hi = limit - wi * 32;
        uint32_t m = w[wi];
        if (hi <= 0) m = 0u;
        else if (hi < 32) m &= (1u << hi) - 1u;
        n += __popc(m);
    }
    return n;
}
// MODE 0: no mask and positive scale (maximum taken on raw scores, one FFMA + EX2 per element), CTAs that stay; MODE 4: the same, a CTA
//         per item;
// MODE 1: additive mask that is the same for every query row (padding masks): all threads stage it in
//         shared memory during set-up, already clamped, scaled by log2(e) and with -inf for columns
//         beyond N, and key blocks that are masked throughout are not visited; MODE 2: anything else (per-row masks read from global memory with
//         128-bit loads where the layout allows, non-positive scale); MODE 3: a row mask too long to be staged whole: the two
//         idle warps keep two key blocks of it in shared memory, and every block is visited ([1, 16, 8192, 128] padded
//         1265 us with every thread reading the row for itself).
template <typename T, int D, int MODE>
__global__ void __launch_bounds__(kAttnThreads, 1)
attention_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const AttnDev p,
                    const int num_items, unsigned int* const queue) {
    using Cfg = AttnCfg<D>;
    constexpr bool kNoMask = MODE == 0 || MODE == 4;
    constexpr int KVS = Cfg::kKvStages;
    constexpr int TILE = Cfg::kTileBytes;
    constexpr int CHUNK = kAttnBlock * 64 * 2;  // one 64-column (128-byte swizzled) slab of a tile
    constexpr uint32_t kTmemCols = 512;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t q_smem = smem_u32(smem);
    const uint32_t k_smem = q_smem + 2 * TILE;
    const uint32_t v_smem = k_smem + KVS * TILE;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (2 + 2 * KVS) * TILE);
    const uint32_t bar_base = smem_u32(bars);
    // barrier slots
    auto q_full = [&](int t) { return bar_base + 8u * t; };
    auto k_full = [&](int s) { return bar_base + 8u * (2 + s); };
    auto k_empty = [&](int s) { return bar_base + 8u * (2 + KVS + s); };
    auto v_full = [&](int s) { return bar_base + 8u * (2 + 2 * KVS + s); };
    auto v_empty = [&](int s) { return bar_base + 8u * (2 + 3 * KVS + s); };
    auto s_full = [&](int t) { return bar_base + 8u * (2 + 4 * KVS + t); };
    auto p_full = [&](int t, int half) { return bar_base + 8u * (8 + 4 * KVS + t * 2 + half); };  // keys [0, 64) / [64, 128) of P
    auto o_final = [&](int t) { return bar_base + 8u * (6 + 4 * KVS + t); };
    auto m_full = [&](int t, int bf) { return bar_base + 8u * (12 + 4 * KVS + t * 2 + bf); };  // MODE 3
    auto m_empty = [&](int t, int bf) { return bar_base + 8u * (16 + 4 * KVS + t * 2 + bf); };
    auto q_empty = [&](int t) { return bar_base + 8u * (20 + 4 * KVS + t); };    // the last product of an item has read Q_t
    auto o_free = [&](int t) { return bar_base + 8u * (22 + 4 * KVS + t); };     // O_t is in the softmax warps' registers
    auto item_full = [&](int s) { return bar_base + 8u * (24 + 4 * KVS + s); };  // MODE 0: drawn items
    auto item_free = [&](int s) { return bar_base + 8u * (26 + 4 * KVS + s); };
    constexpr int kNumBars = 28 + 4 * KVS;
    static_assert(kNumBars * 8 + 48 <= 512, "barrier area too small");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* mask_smem = reinterpret_cast<float*>(smem + (2 + 2 * KVS) * TILE + 512);  // MODE 1: [N rounded up to 128]; MODE 3: [tile][two blocks][128]
    uint32_t* act_bits = tmem_slot + 2;  // MODE 1: key blocks with an unmasked key
    volatile int* items = reinterpret_cast<volatile int*>(tmem_slot + 6);  // MODE 0: two slots for drawn items, -1: no more

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // A wait that expired in an earlier CTA or launch leaves the status word set: do no work until
    // the host has read (and cleared) it, so that one failure cannot cost a second per CTA. What is read here may be
    // too early (status_word()); the epilogue looks again before it stores.
    __shared__ int s_expired;
    // MODE 0: one thread of every CTA reports in when it draws no more items; the last one leaves the queue's slot clean.
    // (Reported by the producer, while the last item is computed: at the CTA's end it cost a microsecond.)
    auto report = [&] {
        if (MODE == 0) {
            __threadfence();
            if (atomicAdd(&queue[1], 1u) == gridDim.x - 1) {
                queue[0] = 0u;
                queue[1] = 0u;
                __threadfence();
            }
        }
    };
    {
        __shared__ int s_skip;
        if (threadIdx.x == 0) s_skip = status_word();
        __syncthreads();
        if (s_skip != 0) {
            pdl_wait();
            if (threadIdx.x == 0) report();
            return;
        }
    }

    // Work assignment: heavy (late) query tiles first so that causal work is balanced.
    const int BH = p.B * p.H;
    const int num_m_tiles = (p.M + kAttnBlock - 1) / kAttnBlock;
    const int num_n_blocks = (p.N + kAttnBlock - 1) / kAttnBlock;
    int b, h, mt[2], nblk[2];
    int ntl;  // live tiles of the item (1 or 2)
    auto locate = [&](int idx) {
        int bh, pair;
        attn_work_item(p, BH, idx, bh, pair);
        b = bh / p.H;
        h = bh % p.H;
        ntl = 0;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            mt[t] = pair * 2 + t;
            nblk[t] = 0;
            if (mt[t] < num_m_tiles) {
                ntl = t + 1;
                nblk[t] = p.is_causal ? min(num_n_blocks, mt[t] + 1) : num_n_blocks;
            }
        }
    };
    locate((int)blockIdx.x);
    const int max_blk = max(nblk[0], nblk[1]);

    if (threadIdx.x == 0) {
        for (int t = 0; t < 2; ++t) {
            mbar_init(q_full(t), 1);
            mbar_init(s_full(t), 1);
            mbar_init(p_full(t, 0), 4);
            mbar_init(p_full(t, 1), 4);
            for (int bf = 0; MODE == 3 && bf < 2; ++bf) {
                mbar_init(m_full(t, bf), 2);  // the loader warps
                mbar_init(m_empty(t, bf), 4);  // the tile's softmax warps
            }
            mbar_init(o_final(t), 2);  // the last product, and the issuer itself, for s_expired
            mbar_init(q_empty(t), 1);
            mbar_init(o_free(t), 4);
            mbar_init(item_full(t), 1);
            mbar_init(item_free(t), 9);  // the softmax warps and the issuer
        }
        for (int s = 0; s < KVS; ++s) {
            mbar_init(k_full(s), 1);
            mbar_init(k_empty(s), 1);
            mbar_init(v_full(s), 1);
            mbar_init(v_empty(s), 1);
        }
        *abort_flag = 0;
        for (int i = 0; i < 4; ++i) act_bits[i] = 0u;
        fence_mbar_init();
    }
    if (warp == 9) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    if (warp == 8 && lane == 0) {
        tma_prefetch_desc(&tmap_q);
        tma_prefetch_desc(&tmap_k);
        tma_prefetch_desc(&tmap_v);
        if (kNoMask && p.o_bulk) tma_prefetch_desc(&tmap_o);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Launched with programmatic dependent launch: nothing of global memory but the status word is touched above
    pdl_wait();
    if (warp == 8 && lane == 0) {
        for (int t = 0; t < ntl; ++t) {
            mbar_arrive_expect_tx(q_full(t), TILE);
            for (int c = 0; c < D / 64; ++c)
                tma_load_4d(q_smem + t * TILE + c * CHUNK, &tmap_q, q_full(t), c * 64, mt[t] * kAttnBlock, h, b);
        }
    }
    uint32_t act[4] = {0u, 0u, 0u, 0u};
    if (MODE == 1) {
        const float mlow = mask_lowest(p.mask_dtype);
        const int64_t moff = (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1];
        const int cols = max_blk * kAttnBlock;
        for (int c0 = 0; c0 < cols; c0 += kAttnThreads) {
            const int col = c0 + (int)threadIdx.x;  // a warp's 32 columns lie in one key block
            const bool inside = col < p.N && col < cols;
            const float v = inside ? fmaxf(mask_load(p.mask, moff + (int64_t)col * p.mask_strides[3], p.mask_dtype), mlow) * kLog2e : -INFINITY;
            if (col < cols) mask_smem[col] = v;
            if (__any_sync(0xffffffffu, inside && v > kSkipBelow) && lane == 0) atomicOr(&act_bits[col >> 12], 1u << ((col >> 7) & 31));
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) act[i] = act_bits[i];
        // nothing is skipped when everything is masked, nor for causal rows, which may see masked keys only
        if ((act[0] | act[1] | act[2] | act[3]) == 0u || p.is_causal) {
#pragma unroll
            for (int i = 0; i < 4; ++i) act[i] = 0xffffffffu;
        }
        nblk[0] = bits_count_below(act, nblk[0]);
        nblk[1] = bits_count_below(act, nblk[1]);
    }
    // from here on nblk counts the blocks that a tile visits; both tiles visit a prefix of the same list
    // The CTA's item number `u` + 1, as the producer has drawn it (MODE 0): false when there is none. `warp_wide`: called by a whole warp.
    auto next_item = [&](int u, bool warp_wide, bool& ok) -> bool {
        if (MODE != 0) return false;
        if (!mbar_wait(item_full(u & 1), (uint32_t)((u >> 1) & 1), abort_flag, 500)) { ok = false; return false; }
        const int idx = items[u & 1];
        if (warp_wide) __syncwarp();
        if (!warp_wide || lane == 0) mbar_arrive(item_free(u & 1));
        if (idx < 0) return false;
        locate(idx);
        return true;
    };
    auto next_blk = [&](int from) { return MODE == 1 ? bits_next(act, from) : from; };

    if (warp >= 8) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(attn_regs_low(MODE)));
      if (warp == 8) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            bool ok = true;
            int kv = 0;                 // ring position, running over the CTA's items (as every barrier's phase does)
            int seen[2] = {ntl > 0, ntl > 1};  // items in which a tile was live: their Q has been asked for
            for (int u = 0; ok; ++u) {
                const int visits = max(nblk[0], nblk[1]);
                int jb = next_blk(0);
                for (int j = 0; j < visits && ok; ++j, ++kv, jb = next_blk(jb + 1)) {
                    const int s = kv % KVS;
                    const uint32_t ph = (uint32_t)((kv / KVS) & 1);
                    if (!mbar_wait(k_empty(s), ph ^ 1, abort_flag, 100)) { ok = false; break; }
                    mbar_arrive_expect_tx(k_full(s), TILE);
                    for (int c = 0; c < D / 64; ++c)
                        tma_load_4d(k_smem + s * TILE + c * CHUNK, &tmap_k, k_full(s), c * 64,
                                    jb * kAttnBlock, h / p.kv_group, b);
                    if (!mbar_wait(v_empty(s), ph ^ 1, abort_flag, 101)) { ok = false; break; }
                    mbar_arrive_expect_tx(v_full(s), TILE);
                    for (int c = 0; c < D / 64; ++c)
                        tma_load_4d(v_smem + s * TILE + c * CHUNK, &tmap_v, v_full(s), c * 64,
                                    jb * kAttnBlock, h / p.kv_group, b);
                }
                if (MODE != 0 || !ok) break;
                // The item's last block is on its way, so the item is two blocks from its end: time to draw the next one. (A CTA
                // that is busy with a long item should not hold back one that an idle CTA could start.)
                if (u >= 2 && !mbar_wait(item_free(u & 1), (uint32_t)(((u >> 1) - 1) & 1), abort_flag, 102)) { ok = false; break; }
                const unsigned int drawn = gridDim.x + atomicAdd(&queue[0], 1u);  // (up to num_items + 2 x gridDim.x: beyond 31 bits)
                const bool more = drawn < (unsigned int)num_items;
                items[u & 1] = more ? (int)drawn : -1;
                mbar_arrive(item_full(u & 1));
                if (!more) {
                    pdl_launch_dependents();  // nothing more to draw: a dependent launch may take the SM once this item is done
                    break;
                }
                locate((int)drawn);
                for (int t = 0; t < ntl; ++t) {
                    if (seen[t] > 0 && !mbar_wait(q_empty(t), (uint32_t)((seen[t] - 1) & 1), abort_flag, 103)) { ok = false; break; }
                    ++seen[t];
                    mbar_arrive_expect_tx(q_full(t), TILE);
                    for (int c = 0; c < D / 64; ++c)
                        tma_load_4d(q_smem + t * TILE + c * CHUNK, &tmap_q, q_full(t), c * 64, mt[t] * kAttnBlock, h, b);
                }
            }
            report();
            if (!ok) {
                for (int i = 0; i < 64; ++i) __nanosleep(2000);
            }
        }
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            s_expired = status_word();
            constexpr uint32_t idesc_qk = make_idesc_f16(Elem<T>::kIsBf16, 128, 128, 0, 0);
            constexpr uint32_t idesc_pv = make_idesc_f16(Elem<T>::kIsBf16, 128, D, 0, 1);
            bool ok = true;
            // Descriptor halves that never change: high word = stride offset 1024 B, version 1, 128-byte
            // swizzle; low word = address >> 4 (+ the leading offset for the N-major V operand).
            constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
            const uint32_t q_lo = (q_smem & 0x3FFFF) >> 4;
            const uint32_t k_lo = (k_smem & 0x3FFFF) >> 4;
            // leading offset of the V operand = distance to the next 64-column slab along N
            const uint32_t v_lo = ((v_smem & 0x3FFFF) >> 4) | ((uint32_t)(CHUNK >> 4) << 16);
            auto desc = [&](uint32_t lo) { return ((uint64_t)desc_hi << 32) | (uint64_t)lo; };
            auto issue_qk = [&](int t, int s) {
                const uint32_t a_lo = q_lo + (uint32_t)(t * (TILE >> 4));
                const uint32_t b_lo = k_lo + (uint32_t)(s * (TILE >> 4));
                const uint32_t d_tmem = tmem_base + (uint32_t)(t * 128);
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint32_t off = (uint32_t)(((ks / 4) * CHUNK + (ks % 4) * 32) >> 4);
                    tc_mma_ss(d_tmem, desc(a_lo + off), desc(b_lo + off), idesc_qk, ks > 0 ? 1u : 0u);
                }
            };
            auto issue_pv = [&](int t, int s, int half, bool accumulate) {
                const uint32_t b_lo = v_lo + (uint32_t)(s * (TILE >> 4));
                const uint32_t d_tmem = tmem_base + (uint32_t)(256 + t * 128);
                const uint32_t a_tmem = tmem_base + (uint32_t)(t * 128);
#pragma unroll
                for (int k4 = 0; k4 < kAttnBlock / 32; ++k4) {
                    const int ks = half * (kAttnBlock / 32) + k4;
                    // 16 keys = 16 rows of 128 bytes = 2048 B; the second 64-wide slab of D is CHUNK bytes away
                    tc_mma_ts(d_tmem, a_tmem + (uint32_t)(ks * 8), desc(b_lo + (uint32_t)(ks * (2048 >> 4))), idesc_pv,
                              (accumulate || ks > 0) ? 1u : 0u);
                }
            };
            int kv = 0;             // ring position of the item's first block
            int cnt[2] = {0, 0};    // blocks of each tile in the items before
            int seen[2] = {0, 0};   // items before in which the tile was live
            for (int u = 0; ok; ++u) {
                const int visits = max(nblk[0], nblk[1]);
                // the first scores, while the softmax warps are still storing the item before: S_t is free, since that
                // item's last P·V has been issued ahead of this product
                if (!mbar_wait(k_full(kv % KVS), (uint32_t)((kv / KVS) & 1), abort_flag, 201)) { ok = false; break; }
                for (int t = 0; t < ntl && ok; ++t) {
                    if (!mbar_wait(q_full(t), (uint32_t)(seen[t] & 1), abort_flag, 200)) { ok = false; break; }
                    tc_fence_after();
                    issue_qk(t, kv % KVS);
                    tc_commit(s_full(t));
                    if (nblk[t] == 1) tc_commit(q_empty(t));
                }
                if (!ok) break;
                tc_commit(k_empty(kv % KVS));
                for (int j = 0; j < visits && ok; ++j) {
                    const int s = (kv + j) % KVS;
                    const uint32_t ph = (uint32_t)(((kv + j) / KVS) & 1);
                    const int s1 = (kv + j + 1) % KVS;
                    const uint32_t ph1 = (uint32_t)(((kv + j + 1) / KVS) & 1);
                    if (!mbar_wait(v_full(s), ph, abort_flag, 202)) { ok = false; break; }
                    if (j + 1 < visits) {
                        if (!mbar_wait(k_full(s1), ph1, abort_flag, 203)) { ok = false; break; }
                    }
                    for (int t = 0; t < ntl; ++t) {
                        if (j >= nblk[t]) continue;
                        const uint32_t pp = (uint32_t)((cnt[t] + j) & 1);
                        // P in halves: the first product runs while the second half's exponentials are taken
                        if (!mbar_wait(p_full(t, 0), pp, abort_flag, 204)) { ok = false; break; }
                        if (j == 0 && seen[t] > 0) {  // the item before: O_t has been read out
                            if (!mbar_wait(o_free(t), (uint32_t)((seen[t] - 1) & 1), abort_flag, 206)) { ok = false; break; }
                        }
                        tc_fence_after();
                        issue_pv(t, s, 0, j > 0);
                        if (!mbar_wait(p_full(t, 1), pp, abort_flag, 205)) { ok = false; break; }
                        tc_fence_after();
                        issue_pv(t, s, 1, true);
                        if (j + 1 < nblk[t]) {
                            issue_qk(t, s1);
                            tc_commit(s_full(t));
                            if (j + 2 == nblk[t]) tc_commit(q_empty(t));
                        } else {
                            mbar_arrive(o_final(t));
                            tc_commit(o_final(t));
                        }
                    }
                    if (!ok) break;
                    tc_commit(v_empty(s));
                    if (j + 1 < visits) tc_commit(k_empty(s1));
                }
                kv += visits;
                for (int t = 0; t < 2; ++t) {
                    cnt[t] += nblk[t];
                    seen[t] += nblk[t] > 0;
                }
                if (!ok || !next_item(u, false, ok)) break;
            }
        }
      } else if (MODE == 3) {
        // ------------------------------------------------------------------ mask loaders (warps 10, 11)
        const int li = (int)threadIdx.x - 320;  // 0 ... 63, two columns each
        const float mlow = mask_lowest(p.mask_dtype);
        const int64_t moff = (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1];
        bool ok = true;
        const int visits = max(nblk[0], nblk[1]);
        for (int j = 0; j < visits && ok; ++j) {
            float a[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = j * kAttnBlock + li + e * 64;
                a[e] = col < p.N ? fmaxf(mask_load(p.mask, moff + (int64_t)col * p.mask_strides[3], p.mask_dtype), mlow) * kLog2e : -INFINITY;
            }
            for (int t = 0; t < ntl && ok; ++t) {
                if (j >= nblk[t]) continue;
                if (!mbar_wait(m_empty(t, j & 1), (uint32_t)((j >> 1) & 1) ^ 1u, abort_flag, 400 + t)) { ok = false; break; }
                mask_smem[(t * 2 + (j & 1)) * kAttnBlock + li] = a[0];
                mask_smem[(t * 2 + (j & 1)) * kAttnBlock + li + 64] = a[1];
                __syncwarp();
                if (lane == 0) mbar_arrive(m_full(t, j & 1));
            }
        }
      }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(attn_regs_high(MODE)));
        // ------------------------------------------------------------------ softmax groups
        const int t = warp >> 2;        // tile handled by this group
        const int q = warp & 3;         // TMEM lane quadrant of this warp
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const uint32_t s_addr = lane_addr + (uint32_t)(t * 128);
        const uint32_t o_addr = lane_addr + (uint32_t)(256 + t * 128);
        const float c = p.scale_log2;
        const float mlow = mask_lowest(p.mask_dtype);
        // Without a mask the running maximum is kept in raw score units and the exponent is
        // (s - m_ref) * c; otherwise scores are first moved to the log2 domain (s*c + mask).
        const float unit = kNoMask ? c : 1.0f;
        int cnt = 0, seen = 0;  // blocks of this tile in the items before, and items in which it was live
        bool ok = true;
        for (int u = 0; ok; ++u) {
          const int m0 = t == 0 ? mt[0] : mt[1], nb = t == 0 ? nblk[0] : nblk[1];
          if (t < ntl && nb > 0) {
            const int row = m0 * kAttnBlock + q * 32 + lane;
            const int64_t mask_row_off =
                (MODE == 2 && p.mask != nullptr)
                    ? (int64_t)b * p.mask_strides[0] + (int64_t)h * p.mask_strides[1] + (int64_t)min(row, p.M - 1) * p.mask_strides[2]
                    : 0;
            float m_ref = -INFINITY;
            float l = 0.f;
            int jb = next_blk(0);
            for (int j = 0; j < nb; ++j, jb = next_blk(jb + 1)) {
                if (!mbar_wait(s_full(t), (uint32_t)((cnt + j) & 1), abort_flag, 300 + t)) { ok = false; break; }
                tc_fence_after();
                uint32_t sr[4][32];
#pragma unroll
                for (int cch = 0; cch < 4; ++cch) tmem_ld_32x32(s_addr + cch * 32, sr[cch]);
                tmem_ld_wait();

                const int col0 = jb * kAttnBlock;
                const bool causal_edge = p.is_causal && col0 + kAttnBlock - 1 > m0 * kAttnBlock;
                if (MODE == 1 || MODE == 3) {
                    if (MODE == 3 && !mbar_wait(m_full(t, j & 1), (uint32_t)((j >> 1) & 1), abort_flag, 320 + t)) { ok = false; break; }
                    const float4* ms = reinterpret_cast<const float4*>(mask_smem + (MODE == 1 ? col0 : (t * 2 + (j & 1)) * kAttnBlock));
#pragma unroll
                    for (int cch = 0; cch < 4; ++cch) {
#pragma unroll
                        for (int v4 = 0; v4 < 8; ++v4) {
                            const float4 a = ms[cch * 8 + v4];  // same address in every lane: broadcast
                            sr[cch][v4 * 4 + 0] = __float_as_uint(fmaf(__uint_as_float(sr[cch][v4 * 4 + 0]), c, a.x));
                            sr[cch][v4 * 4 + 1] = __float_as_uint(fmaf(__uint_as_float(sr[cch][v4 * 4 + 1]), c, a.y));
                            sr[cch][v4 * 4 + 2] = __float_as_uint(fmaf(__uint_as_float(sr[cch][v4 * 4 + 2]), c, a.z));
                            sr[cch][v4 * 4 + 3] = __float_as_uint(fmaf(__uint_as_float(sr[cch][v4 * 4 + 3]), c, a.w));
                        }
                    }
                    if (MODE == 3) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(m_empty(t, j & 1));
                    }
                } else if (MODE == 2) {
                    if (p.mask == nullptr) {
#pragma unroll
                        for (int cch = 0; cch < 4; ++cch) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) sr[cch][i] = __float_as_uint(__uint_as_float(sr[cch][i]) * c);
                        }
                    } else {
#pragma unroll
                        for (int hc = 0; hc < 8; ++hc) {
                            const int colc = col0 + hc * 16;
                            float mvals[16];
                            mask_values(p, mask_row_off, colc, mvals);
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                uint32_t& sv = sr[hc >> 1][(hc & 1) * 16 + i];
                                sv = __float_as_uint(fmaf(fmaxf(mvals[i], mlow), kLog2e, __uint_as_float(sv) * c));
                            }
                        }
                    }
                }
                // columns beyond N (already -inf in MODE 1 and 3) and, on the diagonal block, above the diagonal
                if ((MODE != 1 && MODE != 3 && col0 + kAttnBlock > p.N) || causal_edge) {
#pragma unroll
                    for (int cch = 0; cch < 4; ++cch) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int col = col0 + cch * 32 + i;
                            if (col >= p.N || (p.is_causal && col > row)) sr[cch][i] = __float_as_uint(-INFINITY);
                        }
                    }
                }
                // ---- row maximum (three-input max halves the instruction count)
                float mx4[4];
#pragma unroll
                for (int cch = 0; cch < 4; ++cch) {
                    float mloc = fmaxf(__uint_as_float(sr[cch][0]), __uint_as_float(sr[cch][1]));
#pragma unroll
                    for (int i = 2; i < 32; i += 2) mloc = fmax3(mloc, __uint_as_float(sr[cch][i]), __uint_as_float(sr[cch][i + 1]));
                    mx4[cch] = mloc;
                }
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                // ---- lazy rescale
                float m_new = fmaxf(m_ref, mx);
                if (m_new == -INFINITY) m_new = 0.f;  // row with nothing visible yet
                const bool grow = (m_new - m_ref) * unit > kLazyThreshold;  // also true on the first block
                float alpha = 1.0f;
                if (grow) {
                    alpha = (m_ref == -INFINITY) ? 0.f : fast_exp2((m_ref - m_new) * unit);
                    m_ref = m_new;
                    l *= alpha;
                }
                if (j > 0 && __any_sync(0xffffffffu, grow)) {
                    // S_j complete implies P·V of block j-1 complete (issued earlier, same thread), so O is quiescent.
#pragma unroll
                    for (int dch = 0; dch < D / 16; ++dch) {
                        uint32_t orr[16];
                        tmem_ld_32x16(o_addr + dch * 16, orr);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * alpha);
                        tmem_st_32x16(o_addr + dch * 16, orr);
                    }
                }
                // ---- exponentials, row sum (four independent partial sums), pack to 16 bit, write P over
                //      the first 64 columns of S
                const float neg_ref = -m_ref * unit;
                const float2 unit2 = make_float2(unit, unit), neg2 = make_float2(neg_ref, neg_ref);
                // Row sum: four scalar chains (pair i adds to chain i & 3), taken after P has been handed over. Two values
                // per instruction would save issue slots (155 us instead of 164 at [4, 32 over 8, 2048, 128] causal with a CTA per item) but
                // add in another order, and a decoder's greedy tokens should not depend on that. (A quarter to a half
                // of the exponentials on the FMA pipe was no faster: the special-function unit is half idle.)
                float lp[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int cch = 0; cch < 4; ++cch) {
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float2 a = __ffma2_rn(make_float2(__uint_as_float(sr[cch][2 * i]), __uint_as_float(sr[cch][2 * i + 1])), unit2, neg2);
                        const float e0 = fast_exp2(a.x), e1 = fast_exp2(a.y);
                        sr[cch][2 * i] = __float_as_uint(e0);
                        sr[cch][2 * i + 1] = __float_as_uint(e1);
                        pk[i] = Elem<T>::pack2(e0, e1);
                    }
                    // Without a mask the first half is handed over once the third quarter's exponentials are under way: waiting for its
                    // store right away leaves the special-function unit idle for the store's latency (4 % there). With one the
                    // values held meanwhile cost more than that ([2, 32, 3916, 128] padded 297 us as here, 309 handed over late).
                    if (!kNoMask) {
                        tmem_st_32x16(s_addr + cch * 16, pk);
                        if (cch & 1) {
                            tmem_st_wait();
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(p_full(t, cch >> 1));
                        }
                        continue;
                    }
                    if (cch >= 2) {
                        if (cch == 3) tmem_st_32x16(s_addr + cch * 16, pk);
                        tmem_st_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(p_full(t, cch - 2));
                    }
                    if (cch < 3) tmem_st_32x16(s_addr + cch * 16, pk);
                }
#pragma unroll
                for (int cch = 0; cch < 4; ++cch) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) lp[i & 3] += __uint_as_float(sr[cch][2 * i]) + __uint_as_float(sr[cch][2 * i + 1]);
                }
                l += (lp[0] + lp[1]) + (lp[2] + lp[3]);
            }
            if (MODE != 0) pdl_launch_dependents();  // the key loop is over: a dependent launch may take the slots that free up
            // ---- epilogue: O / l -> global
            if (!ok || !mbar_wait(o_final(t), (uint32_t)(seen & 1), abort_flag, 310 + t)) { ok = false; break; }
            tc_fence_after();
            const int m_end = s_expired == 0 ? p.M : 0;  // rows that may be stored
            const float inv_l = 1.0f / l;
            if (kNoMask && p.o_bulk) {
                // Boxes of 32 rows x 64 columns through shared memory to bulk stores (rows of 128 bytes, 128-byte swizzle; rows
                // beyond M and columns beyond the head dimension are left out): a thread per row stores 16 bytes to each of 32 lines
                // at a time, 2600 cycles per item in which the tile's next scores wait.
                uint8_t* mine = smem + Cfg::kOutOffset + warp * Cfg::kOutWarpBytes;
                uint32_t orr[4][32];
#pragma unroll
                for (int dch = 0; dch < 4; ++dch) tmem_ld_32x32(o_addr + dch * 32, orr[dch]);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(o_free(t));
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    if (lane == 0) bulk_wait_read();  // the box before this one has left the buffer
                    __syncwarp();
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        const uint32_t (&w)[32] = orr[hf * 2 + v / 4];
                        uint32_t o4[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            o4[i] = Elem<T>::pack2(__uint_as_float(w[(v & 3) * 8 + 2 * i]) * inv_l, __uint_as_float(w[(v & 3) * 8 + 2 * i + 1]) * inv_l);
                        *reinterpret_cast<uint4*>(mine + lane * 128 + ((v ^ (lane & 7)) * 16)) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && m0 * kAttnBlock + q * 32 < m_end) {
                        tma_store_4d(&tmap_o, smem_u32(mine), hf * 64, m0 * kAttnBlock + q * 32, h, b);
                        bulk_commit();
                    }
                }
            } else {
                T* o_row = reinterpret_cast<T*>(p.o) + (int64_t)b * p.o_strides[0] + (int64_t)h * p.o_strides[1] +
                           (int64_t)row * p.o_strides[2];
                const bool vec = p.o_strides[3] == 1 && ((((uintptr_t)o_row) & 15) == 0);
#pragma unroll
                for (int dch = 0; dch < D / 32; ++dch) {
                    uint32_t orr[32];
                    tmem_ld_32x32(o_addr + dch * 32, orr);
                    tmem_ld_wait();
                    if (row < m_end) {
                        float val[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) val[i] = __uint_as_float(orr[i]) * inv_l;
                        if (dch * 32 + 32 <= p.d_out) attn_store_32<T, false>(o_row, dch * 32, p.o_strides[3], vec, val, p.d_out);
                        else attn_store_32<T, true>(o_row, dch * 32, p.o_strides[3], vec, val, p.d_out);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(o_free(t));
            }
            cnt += nb;
            ++seen;
          }
          if (!next_item(u, true, ok)) break;
        }
        if (kNoMask && p.o_bulk && lane == 0) bulk_wait_all();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        __syncwarp();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

template <typename T, int D, int MODE>
static int launch_attention_tdm(const kb_attn_params& p, cudaStream_t stream, unsigned int* queue = nullptr) {
    using Cfg = AttnCfg<D>;
    constexpr bool kNoMask = MODE == 0 || MODE == 4;
    CUtensorMap tq, tk, tv, to;
    const int64_t kv_group = p.kv_group > 1 ? p.kv_group : 1;
    if (p.H % kv_group != 0) return KB_ERR_BAD_ARG;
    auto enc = [&](CUtensorMap* out, const void* ptr, int64_t rows, const int64_t* st, int64_t heads, int box_rows = kAttnBlock) -> int {
        if (st[3] != 1) return KB_ERR_UNSUPPORTED;
        const uint64_t dims[4] = {(uint64_t)p.D, (uint64_t)rows, (uint64_t)heads, (uint64_t)p.B};  // boxes reach to D: zero fill
        // A dimension of extent 1 may carry any stride in the caller's tensor; TMA still wants a
        // multiple of 16 bytes, and the value is never used, so substitute a harmless one.
        auto fix = [](int64_t extent, int64_t stride) -> uint64_t {
            return (extent == 1) ? 16u : (uint64_t)stride * 2u;
        };
        const uint64_t strides[4] = {0, fix(rows, st[2]), fix(heads, st[1]), fix(p.B, st[0])};
        const uint32_t box[4] = {64, (uint32_t)box_rows, 1, 1};
        return encode_tmap_16bit(out, ptr, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    };
    int st = enc(&tq, p.q, p.M, p.q_strides, p.H);
    if (st != KB_OK) return st;
    st = enc(&tk, p.k, p.N, p.k_strides, p.H / kv_group);
    if (st != KB_OK) return st;
    st = enc(&tv, p.v, p.N, p.v_strides, p.H / kv_group);
    if (st != KB_OK) return st;

    AttnDev d;
    const int num_m_tiles = (int)((p.M + kAttnBlock - 1) / kAttnBlock);
    d.num_pairs = (num_m_tiles + 1) / 2;
    const int64_t items = (int64_t)d.num_pairs * p.B * p.H;
    if (items > 0x7fffffff) return KB_ERR_UNSUPPORTED;
    d.o_bulk = kNoMask && attn_bulk_out(p) && enc(&to, p.o, p.M, p.o_strides, p.H, 32) == KB_OK ? 1 : 0;
    if (!d.o_bulk) to = tq;  // (not used)
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
        const int64_t per16 = (p.mask_dtype == KB_F32) ? 4 : 8;  // elements per 16 bytes
        d.mask_vec = (p.mask_strides[0] % per16 == 0 && p.mask_strides[1] % per16 == 0 && p.mask_strides[2] % per16 == 0) ? 1 : 0;
    }
    d.head_group = attn_head_group(p.B * p.H, p.N, p.D);
    d.kv_group = (int)kv_group;
    d.d_out = (int)p.D;

    static PerDeviceOnce attr_once;
    if (!attr_once.run([] {
            const int most = kNoMask ? Cfg::kSmemNoMask : MODE == 1 ? Cfg::kSmemMax : Cfg::kSmemBase + (MODE == 3 ? Cfg::kMaskRingBytes : 0);
            return cudaFuncSetAttribute(attention_tc_kernel<T, D, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess;
        }))
        return KB_ERR_LAUNCH;
    const int64_t grid = MODE == 0 ? gemm_sms() : items;  // a caller-set limit leaves SMs to a concurrent collective, as for the GEMMs
    const size_t smem_bytes = kNoMask ? (size_t)Cfg::kSmemNoMask : (size_t)Cfg::kSmemBase +
        (MODE == 1 ? (size_t)((p.N + kAttnBlock - 1) / kAttnBlock) * kAttnBlock * 4 : MODE == 3 ? Cfg::kMaskRingBytes : 0);
    if (launch_pdl(attention_tc_kernel<T, D, MODE>, (unsigned)grid, kAttnThreads, smem_bytes, stream, tq, tk, tv, to, d, (int)items, queue) != cudaSuccess)
        return KB_ERR_LAUNCH;
    return cudaGetLastError() == cudaSuccess ? KB_OK : KB_ERR_LAUNCH;
}

template <typename T, int D>
static int launch_attention_td(const kb_attn_params& p, cudaStream_t stream) {
    if (p.mask == nullptr && p.sm_scale > 0.f) {
        // As many CTAs as pairs of query tiles where an SM holds them at once. (Drawing, counters and registers for several items cost a launch
        // that has no second item 0.1 to 0.5 us: [4, 32, 200, 128] 9.9 -> 9.5, causal 9.75 -> 9.45, [4, 32 over 8, 130, 128] causal 9.5 -> 9.1.)
        const int64_t items = (p.M + 2 * kAttnBlock - 1) / (2 * kAttnBlock) * p.B * p.H;
        unsigned int* queue = items > gemm_sms() ? attention_queue_slot(stream) : nullptr;
        return queue == nullptr ? launch_attention_tdm<T, D, 4>(p, stream) : launch_attention_tdm<T, D, 0>(p, stream, queue);
    }
    if (p.mask != nullptr && p.mask_strides[2] == 0)
        return p.N <= AttnCfg<D>::kMaskMaxN ? launch_attention_tdm<T, D, 1>(p, stream) : launch_attention_tdm<T, D, 3>(p, stream);
    return launch_attention_tdm<T, D, 2>(p, stream);
}

static int launch_attention128(const kb_attn_params& p, cudaStream_t stream) {
    if (p.N <= 0) return KB_ERR_UNSUPPORTED;
    if (p.M > 0x7fffffff || p.N > 0x7fffffff || p.B * p.H > 0x7fffffff) return KB_ERR_UNSUPPORTED;
    // head dimensions up to 64 are served by attention_split.cuh; 72 ... 128 run here on the D = 128 kernel
    if (p.D <= 64 || p.D > 128 || p.D % 8 != 0) return KB_ERR_UNSUPPORTED;
    if (p.dtype == KB_F16) return launch_attention_td<__half, 128>(p, stream);
    if (p.dtype == KB_BF16) return launch_attention_td<__nv_bfloat16, 128>(p, stream);
    return KB_ERR_UNSUPPORTED;
}

}  // namespace kb
