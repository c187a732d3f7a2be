// Small-M (decode) W8A8 linear over PRE-PACKED weights: the HBM-roofline form.
//
// Same arithmetic as the other GEMV kernels (exact int32 sum per K-group from mma.sync.m16n8k32.s8
// with the weights as the A operand, acc = fma(float(P) * ws, xs, acc) over ascending groups, fp32
// partial tiles of a cut row tile added in ascending-K order). What changes is the weight layout.
//
// A row-major [N,K] matrix makes every 16-row tile 16 separate runs in DRAM, 256 bytes at a time per
// run; measured, that streams at about half of what a linear copy reaches. The loader therefore
// re-packs each weight once (w8a8_pack_weight) into the order in which this kernel consumes it:
//
//   block (rt, kb) = 16 rows x 256 bytes of K      rt = row tile, kb = 256-byte K block
//     [4 chunks of 64 K-bytes][2 halves][32 lanes][16 bytes]   a lane's MMA A-fragment pieces: half 0 =
//                                                   row gq, half 1 = row gq+8 (gq = lane / 4)
//     [16 rows][groups per block] fp16              the block's weight scales (32, 64 or 128 bytes)
//   blocks ordered rt-major, kb ascending, one after another with no gaps.
//
// Work split: whole 16-row tiles per CTA (tile t of T goes to CTA t * C / T), the CTA's units of 256 K-bytes
// in equal contiguous runs to its eight warps. A warp's run is then ONE contiguous byte range: the warp
// pulls it through a private ring of shared-memory stages with 1-D bulk copies (cp.async.bulk, one
// block per copy, completion on an mbarrier), reads its fragments back with conflict-free 128-bit
// shared loads, and finds the scales in the same stage — no strided access, no separate scale
// traffic, no tensor map. Rows past N are stored as zeros, so no tail handling is needed on loads.
// A row tile cut by a run boundary is always cut between warps of one CTA: its fp32 partial tiles meet in
// shared memory, and once the CTA has streamed its blocks all its threads add them up in ascending-K order. (One
// warp, the last to arrive, used to do that, with two divisions per contributor: 2300 clocks of a 6400-clock launch
// of 2560 x 4096. An earlier form still cut one global range over all warps of the grid and fixed cut tiles up
// through global scratch and L2 atomics: perfectly balanced, but two to three L2 round trips at the tail of every
// launch; measured 2 us slower per launch on the decode shapes than the at most one-tile imbalance of this form.)
//
// Launched with programmatic dependent launch: the first kStages blocks are requested before
// griddepcontrol.wait. Every mbarrier wait is bounded; on expiry the warp records an error word.
#pragma once

#include <cstdlib>

#include "sm100_ptx.cuh"
#include "w8a8_internal.h"
#include "w8a8_trace.cuh"

namespace w8a8 {
namespace gemv {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kBlockW = 16 * 256;        // weight bytes of a block
constexpr int kStagePitch = kBlockW + 128;  // room for the largest scale tail, keeps stages 128-byte aligned
// How the activations arrive (template parameter PRO):
enum { kProCodes = 0,   // int8 codes + fp32 scales made by an earlier launch (Xq, Xs)
       kProNorm = 1,    // fp16 rows: every CTA does [x + residual] -> RMSNorm -> quantiser itself, in its prologue
       kProQuant = 2 }; // fp16 rows: a warp quantises the activations of each block it consumes, in registers

// Forms of the kernel, by 8-token B tiles, group size class and tiles at once (reasons: see the consumer loop).
constexpr bool in_place(int mt, int gm, int nr) { return mt == 4 || (mt == 2 && gm != 64 && nr == 1); }
constexpr bool two_per_sm(int mt, int gm, int nr) { return mt == 1 || (mt == 2 && gm != 64 && nr == 1); }

struct GemvPackedParams {
    LinearArgs a;
    const unsigned char* packed;
    int block_bytes;  // kBlockW + 32 * groups per block
    int upt;          // units per 16-row tile
    int bpu;          // blocks per unit (1, or g / 256 when g > 256)
    unsigned U;       // units in all
    int* status;
#ifdef W8A8_TRACE
    int ablate;       // diagnostic build: bit mask of pieces of the kernel to leave out (timing experiments only)
#endif
};
#ifdef W8A8_TRACE
#define W8A8_ABLATED(bit) ((p.ablate & (bit)) != 0)
#else
#define W8A8_ABLATED(bit) false
#endif

__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The same onto zero: no registers to clear before it.
__device__ __forceinline__ void mma_s8_first(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    return static_cast<uint64_t>(__float_as_uint(a)) | (static_cast<uint64_t>(__float_as_uint(b)) << 32);
}
// Two sums of one weight row: acc = fma(float(P) * ws, xs, acc), two at a time.
__device__ __forceinline__ void promote2(float& acc0, float& acc1, int p0, int p1, uint64_t ws, uint64_t xs) {
    uint64_t acc = pack2(acc0, acc1);
    asm("{\n\t.reg .f32 lo, hi;\n\t.reg .b64 t;\n\tcvt.rn.f32.s32 lo, %1;\n\tcvt.rn.f32.s32 hi, %2;\n\tmov.b64 t, {lo, hi};\n\t"
        "mul.rn.f32x2 t, t, %3;\n\tfma.rn.f32x2 %0, t, %4, %0;\n\t}" : "+l"(acc) : "r"(p0), "r"(p1), "l"(ws), "l"(xs));
    acc0 = __uint_as_float(static_cast<uint32_t>(acc));
    acc1 = __uint_as_float(static_cast<uint32_t>(acc >> 32));
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(addr));
    return v;
}

// A row's scales of a block, one word.
template <int N>
__device__ __forceinline__ void lds_scales(uint32_t addr, __half (&s)[N]) {
    if constexpr (N == 4) {
        uint32_t v[2];
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v[0]), "=r"(v[1]) : "r"(addr));
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = __ushort_as_half(static_cast<unsigned short>(v[i >> 1] >> (16 * (i & 1))));
    } else if constexpr (N == 2) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(addr));
        s[0] = __ushort_as_half(static_cast<unsigned short>(v));
        s[1] = __ushort_as_half(static_cast<unsigned short>(v >> 16));
    } else {
        s[0] = __ushort_as_half(static_cast<unsigned short>(lds16(addr)));
    }
}

__device__ __forceinline__ uint4 ld_cg16(const __half* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

#ifdef W8A8_TAIL_TIMELINE
// Diagnostic build only: the last CTA to arrive leaves nanosecond stamps of its launch in tail_counters[128..].
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#define W8A8_STAMP(slot) do { if (threadIdx.x == 0) tl[slot] = now_ns(); } while (0)
#define W8A8_STAMP_FLUSH(counters, is_last) do { if (threadIdx.x == 0 && (is_last)) { \
    unsigned long long* o = reinterpret_cast<unsigned long long*>((counters) + 128); \
    for (int i_ = 0; i_ < 8; ++i_) o[i_] = tl[i_]; o[8] = blockIdx.x; } } while (0)
#else
#define W8A8_STAMP(slot) do {} while (0)
#define W8A8_STAMP_FLUSH(counters, is_last) do {} while (0)
#endif

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Tail, kind kTailRowNorm. Called by all 256 threads of a CTA after its last tile is stored. The CTA takes a ticket;
// the last min(M, grid) CTAs to arrive each wait (bounded) until every CTA of the grid has arrived, i.e. until the
// whole output Y = [M, N] is in L2, and then run, for the token rows they own, exactly what the kernel launched next
// would have run (rowquant_compact_kernel): x = half(x + Y) (ffn_activations.cu:41-45), RMSNorm with the
// reference's 1024-thread summation order (rms_norm.cu:23-49), the group quantiser (int8_gemm.cu:147-211).
// N % 256 == 0, 512 < N <= 4096. The last row CTA to finish puts the counters back to zero.
__device__ __forceinline__ void tail_row_norm(const LinearArgs& a, unsigned char* scratch, int* status,
                                              unsigned long long (&tl)[8]) {
    __shared__ int s_ticket, s_fail;
    __shared__ float s_red[32];
    __half* row_s = reinterpret_cast<__half*>(scratch);  // [N]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int total = gridDim.x, n_row = a.M < total ? a.M : total, first = total - n_row;
    if (tid == 0) {
        __threadfence();  // this CTA's tiles (stored by all its warps, ordered by the barrier before the call)
        s_ticket = atomicAdd(&a.tail_counters[0], 1);
        s_fail = 0;
    }
    __syncthreads();
    const int ticket = s_ticket;
    W8A8_STAMP(3);
    if (ticket < first) return;
    if (tid == 0) {
        unsigned spins = 0;
        while (ld_acquire_gpu(&a.tail_counters[0]) < total) {
            if (++spins > (1u << 22)) { atomicExch(status, 610); s_fail = 1; break; }
            if (spins > 32) __nanosleep(32);
        }
    }
    __syncthreads();
    W8A8_STAMP(4);
    const int K = a.N, T = 1024, VW = T / kThreads, pieces = K / 8;
    const int G = K / a.tail_g;
    if (!s_fail) {
        for (int row = ticket - first; row < a.M; row += n_row) {
            const size_t base = static_cast<size_t>(row) * K;
            uint4 xv[2], dv[2], wv[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {  // every load first (at most two pieces per thread)
                const int c8 = tid + i * kThreads;
                const int cc = c8 < pieces ? c8 : 0;
                wv[i] = __ldg(reinterpret_cast<const uint4*>(a.tail_norm_weight) + cc);
                xv[i] = __ldcg(reinterpret_cast<const uint4*>(a.tail_x + base) + cc);
                dv[i] = __ldcg(reinterpret_cast<const uint4*>(a.Y + base) + cc);  // written by other SMs: past L1
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int c8 = tid + i * kThreads;
                if (c8 < pieces) {
                    __half* hx = reinterpret_cast<__half*>(&xv[i]);
                    const __half* hd = reinterpret_cast<const __half*>(&dv[i]);
#pragma unroll
                    for (int e = 0; e < 8; ++e) hx[e] = __float2half(__half2float(hx[e]) + __half2float(hd[e]));
                    *reinterpret_cast<uint4*>(a.tail_x + base + c8 * 8) = xv[i];
                    reinterpret_cast<uint4*>(row_s)[c8] = xv[i];
                }
            }
            __syncthreads();
            W8A8_STAMP(5);
#pragma unroll 1
            for (int k = 0; k < VW; ++k) {  // real warp w plays the reference's warps w*VW .. w*VW + VW - 1
                float local_sum = 0.0f;
#pragma unroll 1
                for (int e = (warp * VW + k) * 32 + lane; e < K; e += T) {
                    float val = __half2float(row_s[e]);
                    local_sum += val * val;
                }
                for (int offset = 16; offset > 0; offset /= 2) local_sum += __shfl_down_sync(0xffffffffu, local_sum, offset);
                if (lane == 0) s_red[warp * VW + k] = local_sum;
            }
            __syncthreads();
            float total_sum = 0.0f;
            if (warp == 0) {
                total_sum = s_red[lane];
                for (int offset = 16; offset > 0; offset /= 2) total_sum += __shfl_down_sync(0xffffffffu, total_sum, offset);
            }
            __syncthreads();
            if (tid == 0) s_red[0] = rsqrtf(total_sum / K + a.tail_eps);
            __syncthreads();
            const float rms = s_red[0];
            const int lanes = a.tail_g / 8;  // threads per quantisation group: 8, 16 or 32
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int c8 = tid + i * kThreads;
                const bool live = c8 < pieces;  // whole warps are live or not (pieces is a multiple of 32)
                __half* hx = reinterpret_cast<__half*>(&xv[i]);
                const __half* hw = reinterpret_cast<const __half*>(&wv[i]);
                float v[8], amax = 0.0f;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float val = __half2float(hx[e]) * rms;
                    hx[e] = __float2half(val * __half2float(hw[e]));
                    v[e] = __half2float(hx[e]);
                    amax = fmaxf(amax, fabsf(v[e]));
                }
                if (live && a.tail_normed_out) *reinterpret_cast<uint4*>(a.tail_normed_out + base + c8 * 8) = xv[i];
                if (!a.tail_Xq) continue;
                for (int o = lanes / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                if (!live) continue;
                float scale = amax / 127.0f;
                if (scale < 1e-8f) scale = 1e-8f;
                if ((lane & (lanes - 1)) == 0) a.tail_Xs[static_cast<size_t>(row) * G + (c8 * 8) / a.tail_g] = scale;
                const float inv_scale = 1.0f / scale;
                uint32_t lo = 0, hi = 0;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    int q = __float2int_rn(v[e] * inv_scale);
                    q = max(-127, min(127, q));
                    if (e < 4) lo |= (static_cast<uint32_t>(q) & 0xffu) << (8 * e);
                    else hi |= (static_cast<uint32_t>(q) & 0xffu) << (8 * (e - 4));
                }
                *reinterpret_cast<uint2*>(a.tail_Xq + base + c8 * 8) = make_uint2(lo, hi);
            }
            __syncthreads();  // row_s and s_red are reused by the next row of this CTA
        }
    }
    W8A8_STAMP(6);
    W8A8_STAMP_FLUSH(a.tail_counters, ticket == total - 1);
    if (tid == 0) {
        const int done = atomicAdd(&a.tail_counters[1], 1);
        if (done == n_row - 1) {  // every row CTA is past its wait: the counters can go back to zero
            a.tail_counters[1] = 0;
            __threadfence();
            a.tail_counters[0] = 0;
        }
    }
}

// Tail, kind kTailGroupQuant: the quantiser (int8_gemm.cu:147-211) of the launch's own output for the linear that
// follows. out = Y as stored: [M, N] (16 channels per row tile) or, with the SwiGLU epilogue, [M, N/2] (8 channels
// per tile). A CTA adds the number of its tiles in each quantisation group to that group's counter; the CTA whose
// add completes a group quantises it (one warp per token row, 8 channels per lane and step) and zeroes the counter.
// Nothing waits. tail_g % 8 == 0 and a multiple of the channels per tile.
__device__ __forceinline__ void tail_group_quant(const LinearArgs& a, int ct0, int ct1, unsigned char* scratch,
                                                 unsigned long long (&tl)[8]) {
    int* s_mine = reinterpret_cast<int*>(scratch);  // [groups this CTA touches]: 1 = this CTA completes the group
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cpt = a.epilogue == W8A8_EPI_SWIGLU ? 8 : 16;      // output channels per row tile
    const int Kout = a.epilogue == W8A8_EPI_SWIGLU ? a.N / 2 : a.N;
    const int tpg = a.tail_g / cpt;                               // tiles per group
    const int tiles = (a.N + 15) / 16, G = (Kout + a.tail_g - 1) / a.tail_g;
    if (ct1 <= ct0) return;
    const int j0 = ct0 / tpg, j1 = (ct1 - 1) / tpg;
    if (tid <= j1 - j0) {
        const int j = j0 + tid;
        const int lo = max(ct0, j * tpg), hi = min(ct1, (j + 1) * tpg);
        const int in_group = min(tiles, (j + 1) * tpg) - j * tpg;
        __threadfence();  // this CTA's tiles (ordered before by the barrier before the call)
        const int old = atomicAdd(&a.tail_counters[j], hi - lo);
        const int mine = (old + (hi - lo) == in_group) ? 1 : 0;
        if (mine) {
            a.tail_counters[j] = 0;
            __threadfence();  // acquire side: the other CTAs' tiles are visible to the loads below
        }
        s_mine[tid] = mine;
    }
    __syncthreads();
    W8A8_STAMP(3);
    bool any_mine = false;
    for (int j = j0; j <= j1; ++j) any_mine |= s_mine[j - j0] != 0;
    for (int j = j0; j <= j1; ++j) {
        if (!s_mine[j - j0]) continue;
        const int c0 = j * a.tail_g, width = min(a.tail_g, Kout - c0);
        for (int row = warp; row < a.M; row += kWarps) {
            const __half* src = a.Y + static_cast<size_t>(row) * Kout + c0;
            float amax = 0.0f;
            for (int e = lane * 8; e < width; e += 256) {
                const uint4 u = __ldcg(reinterpret_cast<const uint4*>(src + e));
                const __half* h = reinterpret_cast<const __half*>(&u);
#pragma unroll
                for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(__half2float(h[i])));
            }
            for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            float scale = amax / 127.0f;
            if (scale < 1e-8f) scale = 1e-8f;
            if (lane == 0) a.tail_Xs[static_cast<size_t>(row) * G + j] = scale;
            const float inv_scale = 1.0f / scale;
            for (int e = lane * 8; e < width; e += 256) {
                const uint4 u = __ldcg(reinterpret_cast<const uint4*>(src + e));
                const __half* h = reinterpret_cast<const __half*>(&u);
                uint32_t lo = 0, hi = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    int q = __float2int_rn(__half2float(h[i]) * inv_scale);
                    q = max(-127, min(127, q));
                    if (i < 4) lo |= (static_cast<uint32_t>(q) & 0xffu) << (8 * i);
                    else hi |= (static_cast<uint32_t>(q) & 0xffu) << (8 * (i - 4));
                }
                *reinterpret_cast<uint2*>(a.tail_Xq + static_cast<size_t>(row) * Kout + c0 + e) = make_uint2(lo, hi);
            }
        }
    }
    __syncthreads();
    W8A8_STAMP(6);
    W8A8_STAMP_FLUSH(a.tail_counters, any_mine && j1 == G - 1);
    (void)any_mine;
}

// GM: 64 or 128 = the group size itself; 256 = any group size that is a multiple of 256 (a unit is then
// one whole group = g/256 blocks).
//
// PRO == kProNorm: the activations arrive as fp16 rows and every CTA forms codes and scales itself before it
// consumes its first block (whose copy is already in flight): [x + residual] -> RMSNorm with the summation
// order of the reference's 1024-thread launch (rms_norm.cu:23-49) -> group quantiser (int8_gemm.cu:147-211).
// One warp per token row (M <= 8), the row in registers from the load to the codes; only the codes and scales
// go to shared memory. This replaces a separate launch of a kernel that runs on M CTAs and leaves the rest of
// the GPU idle, and the trip of its results through L2.
// PRO == kProQuant (M <= 8, g = 64, 128 or 256): the linear without the quantiser's launch before it. A lane's B fragments of a
// block are 64 activations of one token, the four lanes of a quad hold the block's 256 of that token: a group's absmax is a
// few packed maxima and two shuffles, and the codes go from registers into the MMA. Every warp that meets a K block quantises
// it again, some 300 instructions per block, so the form is chosen where a CTA has few row tiles (see quant_form_wins).
// NR: row tiles that a warp takes through a K block together, so that the activations it reads, by then as many bytes as the weights, serve
// both (1 or 2; more than eight rows). A CTA's last tile may be alone. Which launches take two: see make_plan.
// ST: stages of a warp's ring (3; 2 for kProNorm so that two CTAs fit an SM beside the code rows).
// KI: kProNorm only, the 16-byte pieces of a row a lane holds (K <= 256 * KI): 10 for the stack's K = 2560, else 16.
// EXTRA: the call wants the group sums dumped, has a tail or sends to a tensor-parallel exchange. An instance of its own: the check
// per promote alone cost 0.1-1.1 us per launch, and the exchange's stores were half of a decode launch's code, which runs cold.
// EPI: the epilogue, or -1: the call's (one of three code paths is fetched past).
// ROWS: the weights are the row-major matrix itself. A block is then a TMA box of 16 rows x two 128-byte K blocks (128-byte
// swizzle), its scales come from the matrix's own scale array a unit ahead, and everything else is the same.
template <int MT, int GM, int NR, int PRO, int ST, int KI, int EPI, bool EXTRA, bool ROWS>
__device__ __forceinline__ void gemv_body(const GemvPackedParams& p, const CUtensorMap* map) {
    constexpr bool FUSED = PRO == kProNorm, QUANT = PRO == kProQuant;
    const int epilogue = EPI >= 0 ? EPI : p.a.epilogue;
    constexpr bool TP = EXTRA || FUSED;  // instances that can send to a tensor-parallel exchange
    constexpr int kStages = ST;
    constexpr int kPitch = ROWS ? kBlockW : kStagePitch;
    constexpr int kRingBytes = kStages * kPitch;
    static_assert(PRO == kProCodes || MT == 1, "the fused prologue handles one row per warp, the fused quantiser one token per quad");
    extern __shared__ unsigned char smem_raw[];
    W8A8_TRACE_SCOPE();
    unsigned long long tl[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    (void)tl;
    W8A8_STAMP(0);
    __shared__ __align__(8) uint64_t bars[kWarps][kStages];
    const LinearArgs& a = p.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gq = lane >> 2, c = lane & 3;
    // Which row of a tile a fragment row holds. ROWS: bits 0 and 1 swapped, so that the two rows of a quarter-warp's fragment load
    // lie four box lines apart, where the swizzle puts them in different banks (w2 at M = 8, g = 256: 8.4 -> 7.5 us).
    auto row_of = [](int q) { return ROWS ? (q & 4) | ((q & 1) << 1) | ((q >> 1) & 1) : q; };
    const int gr = row_of(gq);
    constexpr int GPU = GM == 64 ? 4 : GM == 128 ? 2 : 1;  // groups per unit

    // ---- this warp's contiguous range of units; the eight ranges of a CTA are neighbours, so that most row
    // tiles cut by a range boundary are cut between warps of ONE CTA and can be added up in shared memory ----
    __shared__ float red_s[kWarps][NR * MT * 4 * 32];  // a warp's part of the tile its run begins in (slot 0)
    __shared__ int cut_s[kWarps][3];  // per boundary between two warps' runs: the row tile it cuts (-1: none, or counted with
                                      // the boundary before it), the slot of its first contributor, its last contributor
    // Whole 16-row tiles per CTA (tile t of `tiles` goes to CTA t * C / tiles), the CTA's units in equal contiguous
    // runs to its warps (none with an empty run): a tile cut by a run boundary is always cut between warps of
    // this CTA.
    const unsigned tiles = p.U / p.upt;
    const unsigned ct0 = blockIdx.x * tiles / gridDim.x, ct1 = (blockIdx.x + 1) * tiles / gridDim.x;
    // NR = 2: a unit is two neighbouring tiles (the CTA's last one may be alone) x a unit of K, counted from the CTA's first.
    const unsigned cu0 = NR == 1 ? ct0 * p.upt : 0, n_cta = (ct1 - ct0 + NR - 1) / NR * p.upt;
    const unsigned nw_cta = n_cta < kWarps ? n_cta : kWarps;
    unsigned u0 = cu0, u1 = cu0;
    if (static_cast<unsigned>(warp) < nw_cta) {
        u0 = cu0 + warp * n_cta / nw_cta;
        u1 = cu0 + (warp + 1) * n_cta / nw_cta;
    }
    auto first_tile = [&](unsigned u) { return static_cast<int>(NR == 1 ? u / p.upt : ct0 + u / p.upt * NR); };  // of a unit
    const int T = static_cast<int>(u1 - u0) * p.bpu;  // steps: a K block of the unit's tiles
    int blocks = T;                                    // blocks of the run
    if constexpr (NR == 2) {
        const unsigned paired = (ct1 - ct0) / 2 * p.upt;  // units of two tiles, ahead of those of a lone last one
        if (u0 < paired) blocks += static_cast<int>(min(u1, paired) - u0) * p.bpu;
    }
    // The row tiles cut by run boundaries, worked out while nothing is waited for: a division costs a lone warp some forty
    // clocks, and this used to sit between a tile's last block and its store.
    if (threadIdx.x < kWarps) {
        const int w = threadIdx.x;
        auto start = [&](int i) { return cu0 + i * n_cta / nw_cta; };
        int tile = -1, slot = 0, last = 0;
        if (w + 1 < static_cast<int>(nw_cta)) {
            const unsigned b = start(w + 1), t = b / p.upt;
            if (b != t * p.upt && (w == 0 || start(w) <= t * p.upt)) {  // inside tile t, and no boundary before it is
                tile = static_cast<int>(t);
                slot = start(w) / p.upt == t ? 0 : 1;
                last = w + 1;
                while (last + 1 < static_cast<int>(nw_cta) && start(last + 1) < (t + 1) * p.upt) ++last;
            }
        }
        cut_s[w][0] = tile;
        cut_s[w][1] = slot;
        cut_s[w][2] = last;
    }

    constexpr uint32_t kAlign = ROWS ? 1024u : 128u;  // (the swizzle pattern repeats every 1024 bytes)
    const uint32_t ring = ((ptx::smem_u32(smem_raw) + kAlign - 1) & ~(kAlign - 1)) + warp * kRingBytes;
    uint64_t* bar = bars[warp];
    if (lane == 0) {
        for (int s = 0; s < kStages; ++s) ptx::mbar_init(&bar[s], 1);
        ptx::fence_barrier_init();
        ptx::fence_proxy_async();
    }
    __syncwarp();

    // producer (lane 0): the range is one contiguous run of blocks in the packed image, of boxes in the row-major matrix
    int pt = 0;
    const int k_blocks = p.upt * p.bpu;
    const unsigned char* src = ROWS ? nullptr : p.packed + static_cast<size_t>(u0) * p.bpu * p.block_bytes;
    int pkb = 0, prt = 0, pr = 0;  // ROWS, NR = 2: the next block's K block, its unit's first tile, which of the tiles
    if constexpr (ROWS || NR == 2) { prt = first_tile(u0); pkb = static_cast<int>(u0 % p.upt) * p.bpu; }
    if constexpr (!ROWS && NR == 2) src = p.packed + (static_cast<size_t>(prt) * k_blocks + pkb) * p.block_bytes;
    // Weights are read once per launch and a stack's do not fit in L2: as evict-first lines they do not push out the activations,
    // scales and cache rows that the next launches read, nor wait behind their write-back (decode step, batch 8: 1517 -> 1490 us;
    // ten fast-AR steps 1710 -> 1650). Marking a quarter of them evict-last, to find it again at the next step: 1502 and 1687.
    unsigned long long once;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
    auto issue = [&]() {  // lane 0 only
        const int slot = pt % kStages;
        if constexpr (ROWS) {
            ptx::mbar_arrive_expect_tx(&bar[slot], kBlockW);
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;"
                ::"r"(ring + slot * kPitch), "l"(map), "r"(ptx::smem_u32(&bar[slot])), "r"(0), "r"(pkb * 2), "r"((prt + pr) * 16), "l"(once)
                : "memory");
        } else {
            ptx::mbar_arrive_expect_tx(&bar[slot], p.block_bytes);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                         ::"r"(ring + slot * kPitch), "l"(NR == 1 ? src : src + static_cast<size_t>(pr * k_blocks) * p.block_bytes),
                         "r"(p.block_bytes), "r"(ptx::smem_u32(&bar[slot])), "l"(once)
                         : "memory");
        }
        ++pt;
        if constexpr (NR == 2) {
            if (pr == 0 && prt + 1 < static_cast<int>(ct1)) { pr = 1; return; }
            pr = 0;
        }
        if constexpr (!ROWS) src += p.block_bytes;
        if constexpr (ROWS || NR == 2) {
            if (++pkb == k_blocks) {  // (the image goes on with the next tile, which of two was taken along)
                pkb = 0;
                prt += NR;
                if constexpr (!ROWS) src += static_cast<size_t>(k_blocks) * p.block_bytes;
            }
        }
    };
    if (lane == 0) {
        const int pre = blocks < kStages ? blocks : kStages;
        for (int i = 0; i < pre; ++i) issue();
    }
    // The blocks behind the ring's go to L2 meanwhile, one or two per warp: a linear of few rows meets its activations late, and the
    // memory would idle once the rings are full. More of them, or any at M > 8, hold up the row kernel that this launch waits for.
    // (Decode step, batch 1: 1404 -> 1354 us with two; batch 8: 1494 -> 1472 with one, 1543 with four; batch 16: 1922 -> 1938.)
    if (MT == 1 && !ROWS && lane == 0) {
        const int more = min(T - pt, a.M <= 2 ? 2 : 1);
        if (more > 0)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(more * p.block_bytes) : "memory");
    }
    // kProNorm shared memory behind the rings: norm weight [K] fp16 | code rows [8][K + 64] | scales [8][G] fp32
    unsigned char* const fbase = smem_raw + (ring - warp * kRingBytes - ptx::smem_u32(smem_raw)) + kWarps * kRingBytes;
    if constexpr (FUSED) {  // the norm weight is a parameter too: stage it before the wait
        __half* normw_s = reinterpret_cast<__half*>(fbase);
        for (int c8 = threadIdx.x; c8 < a.K / 8; c8 += kThreads)
            reinterpret_cast<uint4*>(normw_s)[c8] = __ldg(reinterpret_cast<const uint4*>(a.norm_weight) + c8);
        __syncthreads();  // staged by all threads, read by each warp on its own after the wait
    }
    // ROWS: the scales of a lane's two rows of a unit, one aligned word each (K is a multiple of 256, so G of the unit's groups)
    __align__(8) __half wsn[NR][2][GPU];
    auto load_ws = [&](int tile, int unit) {
#pragma unroll
        for (int i = 0; i < 2 * NR; ++i) {
            const int h = i & 1;
            const __half* src_s = a.w_scale + static_cast<size_t>(min(tile * 16 + gr + 8 * i, a.N - 1)) * a.G + unit * GPU;
            if constexpr (GPU == 4) {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(src_s));
                *reinterpret_cast<uint2*>(wsn[i >> 1][h]) = v;
            } else if constexpr (GPU == 2) {
                const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(src_s));
                *reinterpret_cast<uint32_t*>(wsn[i >> 1][h]) = v;
            } else {
                wsn[i >> 1][h][0] = __ldg(src_s);
            }
        }
    };
    if constexpr (ROWS) {
        if (T > 0) load_ws(first_tile(u0), static_cast<int>(u0 % p.upt));
    }
    // Everything above touches only weights. Let the next launch begin its own prologue, then wait
    // for the kernel before this one: it produces the activations.
    ptx::pdl_launch_dependents();
    ptx::pdl_wait();
    W8A8_TRACE_WAITED();
    W8A8_STAMP(1);
    // tensor-parallel send: this exchange's epoch = the last finished one + 1 (advanced by the receive kernel)
    int tp_ep = 0;
    if (TP && a.tp.world > 0)
        tp_ep = *reinterpret_cast<const volatile int*>(a.tp.peers[a.tp.rank] + a.tp.ctl_off) + 1;

    const int8_t* xq[MT];
    const float* xsp[MT][2];
    uint32_t xq_s = 0;                    // kProNorm: this lane's code row in shared memory
    const float* xsp_s[2] = {nullptr, nullptr};
    if constexpr (FUSED) {
        const int K = a.K, pitch = K + 64;  // the pitch puts rows gq and gq+1 in different bank halves
        const __half* normw_s = reinterpret_cast<const __half*>(fbase);
        int8_t* codes_s = reinterpret_cast<int8_t*>(fbase + static_cast<size_t>(K) * 2);   // [8][pitch]
        float* scales_s = reinterpret_cast<float*>(codes_s + 8 * pitch);                    // [8][G]
        const int row = warp;
        const bool writer = blockIdx.x == 0;
        // Lane l owns the 16-byte pieces c8 = l + 32 i of its row, i.e. elements e = 8 l + j + 256 i (j < 8): these
        // are ALL the elements of the reference's virtual threads vt = 8 l + j + 256 r (r = i mod 4 < 4), which sum
        // e = vt, vt + 1024, vt + 2048, ... in that order (rms_norm.cu:23-27 with a 1024-thread block).
        constexpr int kMaxI = KI;  // K <= 256 * KI
        const int iters = K / 256;
        uint4 v[kMaxI];
        if (row < a.M) {
            // All loads are requested before anything is used or stored: a load placed after a store that might
            // alias it would wait for it.
            uint4 r[kMaxI];
#pragma unroll
            for (int i = 0; i < kMaxI; ++i) {
                v[i] = make_uint4(0u, 0u, 0u, 0u);
                r[i] = make_uint4(0u, 0u, 0u, 0u);
                if (i < iters) {
                    const size_t off = static_cast<size_t>(row) * K + (lane + 32 * i) * 8;
                    v[i] = ld_cg16(a.X + off);
                    if (a.norm_residual) r[i] = ld_cg16(a.norm_residual + off);
                }
            }
            if (a.norm_residual) {
#pragma unroll
                for (int i = 0; i < kMaxI; ++i) {
                    if (i < iters) {
                        __half* hv = reinterpret_cast<__half*>(&v[i]);
                        const __half* hr = reinterpret_cast<const __half*>(&r[i]);
#pragma unroll
                        for (int e = 0; e < 8; ++e) hv[e] = __float2half(__half2float(hv[e]) + __half2float(hr[e]));
                        if (writer && a.norm_x_out)
                            *reinterpret_cast<uint4*>(a.norm_x_out + static_cast<size_t>(row) * K + (lane + 32 * i) * 8) = v[i];
                    }
                }
            }
            W8A8_STAMP(2);
            // per virtual thread (r, j): local_sum over i = r, r + 4, r + 8, r + 12 ascending
            float ls[4][8];
#pragma unroll
            for (int r4 = 0; r4 < 4; ++r4)
#pragma unroll
                for (int j = 0; j < 8; ++j) ls[r4][j] = 0.0f;
#pragma unroll
            for (int i = 0; i < kMaxI; ++i) {
                if (i < iters) {
                    const __half* hv = reinterpret_cast<const __half*>(&v[i]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float val = __half2float(hv[j]);
                        ls[i & 3][j] += val * val;
                    }
                }
            }
            // The reference's shuffle-down tree over a virtual warp. Virtual warp (r, l / 4) is made of the
            // virtual lanes vl = 8 (l % 4) + j: offsets 16 and 8 cross real lanes (l + 2, l + 1), offsets 4, 2, 1
            // stay inside the lane's eight j. Only virtual lane 0 (l % 4 == 0, j == 0) is used afterwards, and its
            // sum takes exactly the reference's operands in the reference's order.
            float wsum[4];
#pragma unroll
            for (int r4 = 0; r4 < 4; ++r4) {
                float b8[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float local_sum = ls[r4][j];
                    local_sum += __shfl_down_sync(0xffffffffu, local_sum, 2);   // virtual offset 16
                    local_sum += __shfl_down_sync(0xffffffffu, local_sum, 1);   // virtual offset 8
                    b8[j] = local_sum;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) b8[j] += b8[j + 4];                  // virtual offset 4
                b8[0] += b8[2];                                                  // virtual offset 2
                b8[1] += b8[3];
                wsum[r4] = b8[0] + b8[1];                                        // virtual offset 1
            }
            // second tree (rms_norm.cu:36-42): lane vw takes s_red[vw]; virtual warp vw = 8 r + q lives in lane 4 q
            float total_sum = 0.0f;
#pragma unroll
            for (int r4 = 0; r4 < 4; ++r4) {
                const float t = __shfl_sync(0xffffffffu, wsum[r4], 4 * (lane & 7));
                if ((lane >> 3) == r4) total_sum = t;
            }
            for (int offset = 16; offset > 0; offset /= 2)
                total_sum += __shfl_down_sync(0xffffffffu, total_sum, offset);
            total_sum = __shfl_sync(0xffffffffu, total_sum, 0);
            const float rms = rsqrtf(total_sum / K + a.norm_eps);
            W8A8_STAMP(3);
            // normalise in registers (rounded to fp16 like rms_norm's output) and find the group maxima; a run
            // of 256 channels is one i across the warp
            constexpr int kLanesPerGroup = GM == 64 ? 8 : GM == 128 ? 16 : 32;
            const int per_group = GM == 256 ? a.g / 256 : 1;
            float gmax[kMaxI];
#pragma unroll
            for (int i = 0; i < kMaxI; ++i) {
                gmax[i] = 0.0f;
                if (i < iters) {
                    const uint4 w = reinterpret_cast<const uint4*>(normw_s)[lane + 32 * i];
                    __half* hv = reinterpret_cast<__half*>(&v[i]);
                    const __half* hw = reinterpret_cast<const __half*>(&w);
                    float m = 0.0f;
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        float val = __half2float(hv[e]) * rms;
                        hv[e] = __float2half(val * __half2float(hw[e]));
                        m = fmaxf(m, fabsf(__half2float(hv[e])));
                    }
#pragma unroll
                    for (int o = 1; o < kLanesPerGroup; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                    gmax[i] = m;
                }
            }
            W8A8_STAMP(4);
            if (GM == 256 && per_group > 1) {  // a group spans per_group consecutive runs: give each run its group's maximum
#pragma unroll
                for (int i = 1; i < kMaxI; ++i)   // forward: the last run of a group collects the maximum
                    if (i < iters && i % per_group != 0) gmax[i] = fmaxf(gmax[i], gmax[i - 1]);
#pragma unroll
                for (int i = kMaxI - 2; i >= 0; --i)  // backward: hand it to the runs before it
                    if (i + 1 < iters && (i + 1) % per_group != 0) gmax[i] = gmax[i + 1];
            }
#pragma unroll
            for (int i = 0; i < kMaxI; ++i) {
                if (i < iters) {
                    float scale = gmax[i] / 127.0f;
                    if (scale < 1e-8f) scale = 1e-8f;
                    const int j = GM == 256 ? i / per_group : i * (256 / GM) + lane / kLanesPerGroup;
                    if (lane % kLanesPerGroup == 0 && (GM != 256 || i % per_group == 0)) {
                        scales_s[row * a.G + j] = scale;
                        if (writer && a.scales_out) a.scales_out[static_cast<size_t>(row) * a.G + j] = scale;
                    }
                    const float inv_scale = 1.0f / scale;
                    const __half* hv = reinterpret_cast<const __half*>(&v[i]);
                    __align__(8) int8_t q8[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        int q = __float2int_rn(__half2float(hv[e]) * inv_scale);
                        q8[e] = static_cast<int8_t>(max(-127, min(127, q)));
                    }
                    const int c8 = lane + 32 * i;
                    *reinterpret_cast<uint2*>(codes_s + row * pitch + c8 * 8) = *reinterpret_cast<const uint2*>(q8);
                    if (writer && a.codes_out)
                        *reinterpret_cast<uint2*>(a.codes_out + static_cast<size_t>(row) * K + c8 * 8) =
                            *reinterpret_cast<const uint2*>(q8);
                }
            }
        }
        __syncthreads();  // all rows' codes and scales are in place
        W8A8_STAMP(5);
        xq_s = ptx::smem_u32(codes_s) + min(gq, a.M - 1) * pitch + c * 16;
        xsp_s[0] = scales_s + min(2 * c, a.M - 1) * a.G;
        xsp_s[1] = scales_s + min(2 * c + 1, a.M - 1) * a.G;
    } else if constexpr (!QUANT) {
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) {
            xq[nt] = a.Xq + static_cast<size_t>(min(nt * 8 + gq, a.M - 1)) * a.K + c * 16;
            xsp[nt][0] = a.Xs + static_cast<size_t>(min(nt * 8 + 2 * c, a.M - 1)) * a.G;
            xsp[nt][1] = a.Xs + static_cast<size_t>(min(nt * 8 + 2 * c + 1, a.M - 1)) * a.G;
        }
    }

    // Two integer accumulators per tile: consecutive MMAs alternate between them, so that one MMA does
    // not wait for the previous one's result (with one warp per scheduler that latency is exposed).
    // One group per four MMAs at one token tile leaves the chain bare; with more token tiles their MMAs fill it and one accumulator
    // does. The first MMA of a group starts from zero and two sums are promoted per instruction, except in the one-tile form
    // of g = 64, where clearing and scalar promotes came out ahead (ten fast-AR steps and one slow, batch 8: 1527 us, else 1546; batch 1 step 1122 and 1130).
    constexpr bool kTwoSums = GM != 64 || MT == 1, kPairs = GM != 64 || MT > 1;
    int P[NR][MT][4], Q[NR][MT][4];
    float acc[NR][MT][4];
#pragma unroll
    for (int h = 0; h < NR; ++h)
#pragma unroll
        for (int nt = 0; nt < MT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) { P[h][nt][r] = 0; Q[h][nt][r] = 0; acc[h][nt][r] = 0.0f; }

    // Stores a finished 16-row tile held in fragment layout: rows gr / gr+8, tokens 2c / 2c+1.
    auto store_tile = [&](int rt, const float (&v)[MT][4]) {
        const int rA = rt * 16 + gr;
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int tok = nt * 8 + 2 * c + e;
                if (tok >= a.M) continue;
                if (epilogue == W8A8_EPI_SWIGLU) {
                    if (rA + 8 < a.N) {
                        const float g16 = __half2float(__float2half(v[nt][e]));
                        const __half s16 = __float2half(g16 / (1.0f + expf(-g16)));
                        const float u16 = __half2float(__float2half(v[nt][2 + e]));
                        a.Y[static_cast<size_t>(tok) * (a.N / 2) + rt * 8 + gr] = __float2half(__half2float(s16) * u16);
                    }
                } else {
#pragma unroll
                    for (int hrow = 0; hrow < 2; ++hrow) {
                        const int row = rA + 8 * hrow;
                        if (row >= a.N) continue;
                        const size_t o = static_cast<size_t>(tok) * a.N + row;
                        if (TP && a.tp.world > 0) {
                            // the fp32 partial as a self-validating word {value, epoch} into slot [rank] of every rank
                            const size_t word = (static_cast<size_t>((tp_ep & 1) * a.tp.world + a.tp.rank) * a.tp.max_tokens + tok) *
                                                    a.N + row;
                            const uint2 w = make_uint2(__float_as_uint(v[nt][2 * hrow + e]), static_cast<unsigned>(tp_ep));
                            for (int r = 0; r < a.tp.world; ++r) reinterpret_cast<uint2*>(a.tp.peers[r])[word] = w;
                        }
                        if (!a.Y || W8A8_ABLATED(4)) continue;
                        __half y = __float2half(v[nt][2 * hrow + e]);
                        if (epilogue == W8A8_EPI_RESIDUAL)
                            y = __float2half(__half2float(y) + __half2float(a.residual[o]));
                        a.Y[o] = y;
                    }
                }
            }
        }
    };

    // Slot 1, a warp's part of the tile its run ends in, lies in the warp's own ring: it is written after the run's last block.
    static_assert(NR * MT * 4 * 32 * sizeof(float) <= kRingBytes, "partial tiles fit a warp's ring");
    float* const ring0 = reinterpret_cast<float*>(smem_raw + (ring - warp * kRingBytes - ptx::smem_u32(smem_raw)));
    auto slot1 = [&](int w) { return ring0 + w * (kRingBytes / 4); };
    // Called when the warp has added its last unit of row tile rt into acc. A tile that lies inside the warp's run is stored;
    // of a cut tile the fp32 partial goes to the warp's slot in shared memory (0: the tile its run begins in, 1: the tile it
    // ends in) and is added up when the whole CTA has streamed its blocks (below).
    auto finish_tile = [&](int rt0) {  // rt0: the unit's first tile
        const unsigned t_lo = (NR == 1 ? static_cast<unsigned>(rt0) : (static_cast<unsigned>(rt0) - ct0) / NR) * p.upt, t_hi = t_lo + p.upt;  // [t_lo, t_hi)
        const bool whole = (u0 <= t_lo && t_hi <= u1) || W8A8_ABLATED(8);
        float* mine = u0 < t_hi && u0 >= t_lo ? red_s[warp] : slot1(warp);
#pragma unroll
        for (int h = 0; h < NR; ++h) {
            if (whole) {
                const int rt = rt0 + h;
                if (NR == 1 || rt < static_cast<int>(ct1)) store_tile(rt, acc[h]);
            } else {
#pragma unroll
                for (int nt = 0; nt < MT; ++nt)
#pragma unroll
                    for (int r = 0; r < 4; ++r) mine[((h * MT + nt) * 4 + r) * 32 + lane] = acc[h][nt][r];
            }
#pragma unroll
            for (int nt = 0; nt < MT; ++nt)
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[h][nt][r] = 0.0f;
        }
    };

    auto promote = [&](int h, int rt, int j, __half hsa, __half hsb, const float (&xsv)[MT][2]) {
        const float fa = __half2float(hsa), fb = __half2float(hsb);
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) {
            if constexpr (kTwoSums) {
#pragma unroll
                for (int r = 0; r < 4; ++r) P[h][nt][r] += Q[h][nt][r];
            }
            if (EXTRA && a.dump) {
                const int t0 = nt * 8 + 2 * c, rA = rt * 16 + gr;
                const size_t NG = static_cast<size_t>(a.N) * a.G;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int row = rA + 8 * (r >> 1), tok = t0 + (r & 1);
                    if (row < a.N && tok < a.M) a.dump[tok * NG + static_cast<size_t>(row) * a.G + j] = P[h][nt][r];
                }
            }
            if constexpr (kPairs) {
                const uint64_t x2 = pack2(xsv[nt][0], xsv[nt][1]);
                promote2(acc[h][nt][0], acc[h][nt][1], P[h][nt][0], P[h][nt][1], pack2(fa, fa), x2);
                promote2(acc[h][nt][2], acc[h][nt][3], P[h][nt][2], P[h][nt][3], pack2(fb, fb), x2);
            } else {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    acc[h][nt][r] = __fmaf_rn(__fmul_rn(static_cast<float>(P[h][nt][r]), r < 2 ? fa : fb), xsv[nt][r & 1], acc[h][nt][r]);
            }
            if constexpr (GM == 256 || !kPairs) {
#pragma unroll
                for (int r = 0; r < 4; ++r) P[h][nt][r] = Q[h][nt][r] = 0;
            }
        }
    };

    // ---- consumer loop: one packed block (16 rows x 256 bytes of K, plus its scales) per step ----
    // Activation codes and scales are a few KB shared by the whole grid, but each warp touches a
    // given piece only once, so these reads mostly miss L1 and cost an L2 round trip. They are requested a block
    // ahead, into a second set of registers; or (kInPlace) the registers of a 64-byte chunk are refilled as soon as
    // its MMAs have been issued, a little later but in half the registers: for M > 16, and for M = 9..16 where it lets
    // two CTAs share an SM (w2 at M = 16, g = 256: 11.3 -> 9.4 us; at g = 64 the second CTA gains less than the
    // later request costs; at M <= 8 two CTAs fit either way, and a run is often just two blocks long).
    int si = 0;
    int ub = static_cast<int>(u0 % p.upt), rt0 = first_tile(u0), taken = 0;  // the unit's first tile; blocks consumed
    bool ok = true;
    constexpr bool kInPlace = (in_place(MT, GM, NR) && !FUSED) || QUANT;
    constexpr int NX = kInPlace ? 1 : 2;
    uint4 x[NX][4][MT];
    float xs[NX][GPU][MT][2];
    auto load_x = [&](int kbase, int ch, int buf) {
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) {
            if constexpr (FUSED) x[buf][ch][nt] = lds128(xq_s + kbase + ch * 64);
            else if (W8A8_ABLATED(1)) x[buf][ch][nt] = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
            else x[buf][ch][nt] = ptx::ld_result_v4(xq[nt] + kbase + ch * 64);
        }
    };
    auto load_xs = [&](int unit_b, int q, int buf) {
#pragma unroll
        for (int nt = 0; nt < MT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if constexpr (FUSED) xs[buf][q][nt][e] = xsp_s[e][unit_b * GPU + q];
                else if (W8A8_ABLATED(2)) xs[buf][q][nt][e] = 1.0f;
                else xs[buf][q][nt][e] = ptx::ld_result_f32(xsp[nt][e] + unit_b * GPU + q);
            }
    };
    // The scales of a unit at once: a word of two or four where the instance may (the host checks the address).
    constexpr bool kWideXs = GPU > 1 && PRO == kProCodes && !EXTRA && !kInPlace;
    auto load_xs_unit = [&](int unit_b, int buf) {
        if constexpr (kWideXs) {
#pragma unroll
            for (int nt = 0; nt < MT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float* s = xsp[nt][e] + unit_b * GPU;
                    __align__(16) float v[4];
                    if constexpr (GPU == 4) *reinterpret_cast<uint4*>(v) = ptx::ld_result_v4(s);
                    else *reinterpret_cast<uint2*>(v) = ptx::ld_result_v2(s);
#pragma unroll
                    for (int q = 0; q < GPU; ++q) xs[buf][q][nt][e] = v[q];
                }
        } else {
#pragma unroll
            for (int q = 0; q < GPU; ++q) load_xs(unit_b, q, buf);
        }
    };
    // kProQuant: this lane's 64 activations of a block (chunk ch: 16 from ch * 64 + c * 16 on), requested a block ahead
    uint4 raw[QUANT ? 8 : 1];
    auto load_raw = [&](int kbase) {
        const __half* src = a.X + static_cast<size_t>(min(gq, a.M - 1)) * a.K + kbase + c * 16;
#pragma unroll
        for (int i = 0; i < 8; ++i) raw[i] = ptx::ld_result_v4(src + (i >> 1) * 64 + (i & 1) * 8);
    };
    auto quantise = [&]() {  // raw -> codes in x[0], scales of tokens 2c and 2c + 1 in xs[0] (int8_gemm.cu:147-211)
        float am[GPU];
#pragma unroll
        for (int q = 0; q < GPU; ++q) {
            __half2 m2 = __float2half2_rn(0.0f);
#pragma unroll
            for (int i = q * (8 / GPU); i < (q + 1) * (8 / GPU); ++i) {
                const __half2* h = reinterpret_cast<const __half2*>(&raw[i]);
#pragma unroll
                for (int e = 0; e < 4; ++e) m2 = __hmax2(m2, __habs2(h[e]));
            }
            float m = fmaxf(__low2float(m2), __high2float(m2));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            am[q] = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
        }
        // lane c of a quad makes the scale of group c (of c % GPU), the others get it by shuffles
        float mine = am[0];
#pragma unroll
        for (int q = 1; q < GPU; ++q)
            if ((c & (GPU - 1)) == q) mine = am[q];
        float scale = mine / 127.0f;
        if (scale < 1e-8f) scale = 1e-8f;
        const float inv_mine = 1.0f / scale;
#pragma unroll
        for (int q = 0; q < GPU; ++q) {
            const float inv = GPU == 1 ? inv_mine : __shfl_sync(0xffffffffu, inv_mine, (lane & ~3) + q);
#pragma unroll
            for (int e = 0; e < 2; ++e) xs[0][q][0][e] = __shfl_sync(0xffffffffu, scale, (2 * c + e) * 4 + q);
#pragma unroll
            for (int ch = q * (4 / GPU); ch < (q + 1) * (4 / GPU); ++ch) {
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const __half2* h = reinterpret_cast<const __half2*>(&raw[2 * ch + (k >> 1)]) + 2 * (k & 1);
                    const float2 f0 = __half22float2(h[0]), f1 = __half22float2(h[1]);
                    // (no code of a group's own scale leaves [-127, 127])
                    const int q0 = __float2int_rn(f0.x * inv), q1 = __float2int_rn(f0.y * inv);
                    const int q2 = __float2int_rn(f1.x * inv), q3 = __float2int_rn(f1.y * inv);
                    uint32_t hi;
                    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(q3), "r"(q2), "r"(0));
                    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w[k]) : "r"(q1), "r"(q0), "r"(hi));
                }
                x[0][ch][0] = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    };
    if constexpr (QUANT) {
        if (T > 0) load_raw(ub * 256);
    } else if (T > 0) {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) load_x(ub * p.bpu * 256, ch, 0);
        load_xs_unit(ub, 0);
    }
    for (int t = 0; t < T; ++t) {
        // position of the next block (the same row tile or the next one: K restarts at 0)
        int nsi = si + 1, nub = ub;
        if (nsi == p.bpu) { nsi = 0; if (++nub == p.upt) nub = 0; }
        const int nkb = (nub * p.bpu + nsi) * 256;
        if constexpr (QUANT) {
            quantise();
            if (t + 1 < T) load_raw(nkb);
        }
        if (!kInPlace && t + 1 < T) {
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) load_x(nkb, ch, NX - 1);
            if (nsi == 0) load_xs_unit(nub, NX - 1);
        }
        __half sa[NR][GPU], sb[NR][GPU];
#pragma unroll
        for (int h = 0; h < NR; ++h) {
            if (NR > 1 && h > 0 && rt0 + h >= static_cast<int>(ct1)) break;  // (a lone last tile)
            const int rt = rt0 + h, nth = NR == 1 ? t : taken, slot = nth % kStages;
            if (!ptx::mbar_wait_bounded(&bar[slot], (nth / kStages) & 1)) {
                if (lane == 0) atomicExch(p.status, 600 + slot);
                ok = false;
                break;
            }
            if constexpr (NR > 1) ++taken;
            const uint32_t st = ring + slot * kPitch;
            // this block's weight scales ride behind its weights: [16 rows][GPU] fp16 (ROWS: in registers since the unit before)
            if constexpr (ROWS) {
#pragma unroll
                for (int q = 0; q < GPU; ++q) {
                    sa[h][q] = wsn[h][0][q];
                    sb[h][q] = wsn[h][1][q];
                }
                if (h == NR - 1 || rt + 1 >= static_cast<int>(ct1)) {
                    if (nsi == 0 && t + 1 < T) load_ws(nub == 0 ? rt0 + NR : rt0, nub);
                }
            } else {
                lds_scales<GPU>(st + kBlockW + gq * GPU * 2, sa[h]);
                lds_scales<GPU>(st + kBlockW + (gq + 8) * GPU * 2, sb[h]);
            }
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {  // 64-byte K chunks
                uint32_t fa, fb;
                if constexpr (ROWS) {  // box lines are ordered [row][K block]; the 16-byte piece is XOR-ed with the line's low three bits
                    const uint32_t line = static_cast<uint32_t>(gr * 2 + (ch >> 1));
                    fa = st + line * 128 + ((static_cast<uint32_t>((ch & 1) * 4 + c) ^ (line & 7u)) << 4);
                    fb = fa + 16 * 128;
                } else {
                    fa = st + ch * 1024 + lane * 16;
                    fb = fa + 512;
                }
                const uint4 wa = lds128(fa), wb = lds128(fb);
                const bool opens = kPairs && (GM == 64 || (GM == 128 && (ch & 1) == 0));  // a group
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    const uint4 xv = x[0][ch][nt];
                    if (opens) mma_s8_first(P[h][nt], wa.x, wb.x, wa.y, wb.y, xv.x, xv.y);
                    else mma_s8(P[h][nt], wa.x, wb.x, wa.y, wb.y, xv.x, xv.y);
                }
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    const uint4 xv = x[0][ch][nt];
                    if (!kTwoSums) mma_s8(P[h][nt], wa.z, wb.z, wa.w, wb.w, xv.z, xv.w);
                    else if (opens) mma_s8_first(Q[h][nt], wa.z, wb.z, wa.w, wb.w, xv.z, xv.w);
                    else mma_s8(Q[h][nt], wa.z, wb.z, wa.w, wb.w, xv.z, xv.w);
                }
                const bool last_use = h == NR - 1 || rt + 1 >= static_cast<int>(ct1);
                if (kInPlace && !QUANT && last_use) load_x(nkb, ch, 0);  // (after the range's last block: a block of the same rows, read for nothing)
                if (GM == 64) {
                    promote(h, rt, ub * 4 + ch, sa[h][ch % GPU], sb[h][ch % GPU], xs[0][ch % GPU]);
                    if (kInPlace && !QUANT && last_use) load_xs(nub, ch % GPU, 0);
                }
                if (GM == 128 && (ch & 1)) {
                    promote(h, rt, ub * 2 + (ch >> 1), sa[h][(ch >> 1) % GPU], sb[h][(ch >> 1) % GPU], xs[0][(ch >> 1) % GPU]);
                    if (kInPlace && !QUANT && last_use) load_xs(nub, (ch >> 1) % GPU, 0);
                }
            }
            // The block's bytes are in registers: the slot may be refilled.
            __syncwarp();
            // The fence orders the reads of the slot before the copy that overwrites it. Without it the compiler may sink the
            // scales' loads down to their use in the promote, past the copy: it did in the M = 9..16 form (128 registers), and
            // a group's promote then took the next block's scales now and then.
            if (lane == 0 && pt < blocks) {
                ptx::fence_proxy_async();
                issue();
            }
            if (GM == 256 && NR > 1 && si + 1 == p.bpu) promote(h, rt, ub, sa[h][0], sb[h][0], xs[0][0]);
        }
        if (!ok) break;
#ifdef W8A8_TAIL_TIMELINE
        if (t == 0) W8A8_STAMP(6);
#endif
        if (++si == p.bpu) {
            si = 0;
            if (GM == 256 && NR == 1) promote(0, rt0, ub, sa[0][0], sb[0][0], xs[0][0]);
            if (GM == 256 && kInPlace && !QUANT) load_xs(nub, 0, 0);
            // one call site for the tile end: the row tile is complete, or the range ends inside it
            ++ub;
            if (ub == p.upt || t + 1 == T) {
                finish_tile(rt0);
                if (ub == p.upt) { ub = 0; rt0 += NR; }
            }
            if (!kInPlace) {
#pragma unroll
                for (int q = 0; q < GPU; ++q)
#pragma unroll
                    for (int nt = 0; nt < MT; ++nt) { xs[0][q][nt][0] = xs[NX - 1][q][nt][0]; xs[0][q][nt][1] = xs[NX - 1][q][nt][1]; }
            }
        }
        if (!kInPlace) {
#pragma unroll
            for (int ch = 0; ch < 4; ++ch)
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) x[0][ch][nt] = x[NX - 1][ch][nt];
        }
    }
    if (!ok) {
        // Leave only once every requested block has landed (or a second bounded wait ran out): a TMA write
        // must not arrive in shared memory that already belongs to another CTA.
        pt = __shfl_sync(0xffffffffu, pt, 0);
        for (int s = 0; s < kStages; ++s)
            if (pt > s) ptx::mbar_wait_bounded(&bar[s], ((pt - 1 - s) / kStages) & 1, 1u << 16);
    }
    // ---- cut tiles: all warps add the partials up, in ascending-K order, a token's pair of rows per item ----
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < (kWarps - 1) * NR * MT * 64; i += kThreads) {
        const int w = i / (NR * MT * 64), rg_cut = cut_s[w][0];
        if (rg_cut < 0) continue;
        const int f = i % (NR * MT * 64), hn = f >> 6, e = (f >> 5) & 1, fl = f & 31, last = cut_s[w][2];  // hn: tile x token tile
        const int nt = hn % MT, rt_cut = NR == 1 ? rg_cut : static_cast<int>(ct0) + rg_cut * NR + hn / MT;
        if (NR > 1 && rt_cut >= static_cast<int>(ct1)) continue;
        const float* src = (cut_s[w][1] ? slot1(w) : red_s[w]) + (hn * 4 + e) * 32 + fl;
        float v[2] = {0.0f + src[0], 0.0f + src[64]};
#pragma unroll 1
        for (int ww = w + 1; ww <= last; ++ww) {
            const float* more = red_s[ww] + (hn * 4 + e) * 32 + fl;
            v[0] += more[0];
            v[1] += more[64];
        }
        const int tok = nt * 8 + 2 * (fl & 3) + e, rA = rt_cut * 16 + row_of(fl >> 2);
        if (tok >= a.M) continue;
        if (epilogue == W8A8_EPI_SWIGLU) {
            if (rA + 8 < a.N) {
                const float g16 = __half2float(__float2half(v[0]));
                const __half s16 = __float2half(g16 / (1.0f + expf(-g16)));
                const float u16 = __half2float(__float2half(v[1]));
                a.Y[static_cast<size_t>(tok) * (a.N / 2) + rt_cut * 8 + row_of(fl >> 2)] = __float2half(__half2float(s16) * u16);
            }
            continue;
        }
#pragma unroll 1
        for (int row = rA; row <= rA + 8 && row < a.N; row += 8) {
            const size_t o = static_cast<size_t>(tok) * a.N + row;
            const float val = row == rA ? v[0] : v[1];
            if (TP && a.tp.world > 0) {
                const size_t word = (static_cast<size_t>((tp_ep & 1) * a.tp.world + a.tp.rank) * a.tp.max_tokens + tok) * a.N + row;
                const uint2 wd = make_uint2(__float_as_uint(val), static_cast<unsigned>(tp_ep));
                for (int r = 0; r < a.tp.world; ++r) reinterpret_cast<uint2*>(a.tp.peers[r])[word] = wd;
            }
            if (!a.Y || W8A8_ABLATED(4)) continue;
            __half y = __float2half(val);
            if (epilogue == W8A8_EPI_RESIDUAL) y = __float2half(__half2float(y) + __half2float(a.residual[o]));
            a.Y[o] = y;
        }
    }
#ifdef W8A8_TAIL_TIMELINE
    if (a.tail_kind == kTailNone && a.tail_counters) {
        W8A8_STAMP(7);
        W8A8_STAMP_FLUSH(a.tail_counters, blockIdx.x == gridDim.x - 1);
    }
#endif
    if constexpr (EXTRA && PRO == kProCodes && MT == 1) {
        if (a.tail_kind != kTailNone) {
            // every copy this CTA asked for has been consumed: the rings are free to serve as the tail's scratch
            W8A8_STAMP(7);  // this thread's own warp is done
            __syncthreads();
            W8A8_STAMP(2);
            unsigned char* scratch = smem_raw + (ring - warp * kRingBytes - ptx::smem_u32(smem_raw));
            if (a.tail_kind == kTailRowNorm) tail_row_norm(a, scratch, p.status, tl);
            else tail_group_quant(a, static_cast<int>(ct0), static_cast<int>(ct1), scratch, tl);
        }
    }
#ifdef W8A8_TRACE
    __syncthreads();  // diagnostic build: the record's end is the CTA's end, not warp 0's
    W8A8_TRACE_END(10u + PRO + 4u * a.tail_kind, static_cast<unsigned>(a.N));
#endif
}

// How a linear is cut over CTAs and warps.
struct Plan {
    int MT, GM, NR, upt, bpu, block_bytes, tiles, ctas, pro;
    long long U;
};
bool make_plan(const LinearArgs& a, Plan& pl, bool rows, int sms);
// The plain instances read the activation scales of a unit as one word; a call whose scales are not aligned for that runs EXTRA.
inline bool plain_instance(const LinearArgs& a) {
    return !a.dump && a.tail_kind == kTailNone && a.tp.world == 0 && (reinterpret_cast<uintptr_t>(a.Xs) & (a.g == 64 ? 15u : a.g == 128 ? 7u : 3u)) == 0;
}
void fill_params(const LinearArgs& a, const Plan& pl, int* status, GemvPackedParams& p);

}  // namespace gemv
}  // namespace w8a8
