// Decode-step neighbours of the linear layer inside one transformer layer:
//   (1) split the fused qkv row, per-head RMSNorm of q and k, interleaved-pair RoPE, and the write
//       of k / v into the paged cache — one launch instead of the reference's three device copies,
//       two rms_norm launches, rope_qk and 2 x n_kv cudaMemcpyAsync per layer
//       (src/engine/dual_ar_engine.cc:585-628, src/kernels/rope.cu:9-65);
//   (2) single-query paged attention over 16-token blocks with GQA
//       (src/kernels/paged_attention.cu:13-110), one CTA cluster per (sequence, kv head) so that the
//       four query heads of a group share every K/V byte, the context split over the cluster and over
//       warps, partial softmax states merged through (distributed) shared memory; the epilogue can
//       emit the o-projection's int8 codes and scales directly.
// Both follow the reference's fp16 rounding points; (1) also follows its summation order, so q, k and
// the cache contents are bit-identical to the reference chain. (2) sums in a different order than
// the reference's one-warp-per-head loop and is compared at a tolerance.
#include "sm100_ptx.cuh"
#include "w8a8_internal.h"
#include "w8a8_trace.cuh"

namespace w8a8 {
namespace {

constexpr int kHeadDim = 128;
constexpr int kBlockTokens = 16;

struct RopeParams {
    const __half* qkv;        // [B, (n_q + 2 n_kv) * 128]
    const __half* q_norm_w;   // [128] or null (no qk-norm: the fast AR)
    const __half* k_norm_w;
    float eps;
    const float* freqs;       // [64]
    const int* positions;     // [B] position of the new token
    const int* block_table;   // [B, max_blocks]
    int max_blocks;
    __half* k_cache;
    __half* v_cache;          // [blocks, n_layers, n_kv, 16, 128]
    int layer, n_layers, n_q, n_kv;
    __half* q_out;            // [B, n_q, 128]
};

// One warp per (sequence, head). Lane i holds elements i, 32+i, 64+i, 96+i: the four 32-element
// runs are the four "warps" of the reference's 128-thread rms_norm launch, so four shuffle-down
// trees followed by (p0+p2)+(p1+p3) reproduce its sum bit for bit (rms_norm.cu:23-49).
__global__ void __launch_bounds__(128) qknorm_rope_kvwrite_kernel(const RopeParams p) {
    ptx::pdl_launch_dependents();
    const int b = blockIdx.x;
    const int head = blockIdx.y * 4 + (threadIdx.x >> 5);  // 0..n_q-1 q, then k heads, then v heads
    const int lane = threadIdx.x & 31;
    const int total_heads = p.n_q + 2 * p.n_kv;
    if (head >= total_heads) return;
    const __half* src = p.qkv + (static_cast<size_t>(b) * total_heads + head) * kHeadDim;
    const bool is_q = head < p.n_q, is_k = !is_q && head < p.n_q + p.n_kv;
    // parameters (norm weights, rotation frequencies) are requested before the wait for the qkv projection
    const __half* w = is_q ? p.q_norm_w : (is_k ? p.k_norm_w : nullptr);
    __half wv[4];
    float fr[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        wv[v] = w ? w[v * 32 + lane] : __float2half(1.0f);
        fr[v] = p.freqs[(v * 32 + lane) >> 1];
    }
    ptx::pdl_wait();
    const int pos = p.positions[b];
    __half h[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) h[v] = src[v * 32 + lane];
    // the cache slot of the new token: a second dependent load, started now rather than after the arithmetic
    int phys = 0;
    if (!is_q) phys = p.block_table[static_cast<size_t>(b) * p.max_blocks + pos / kBlockTokens];

    if (is_q || is_k) {
        if (w) {
            float part[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                float val = __half2float(h[v]);
                float local_sum = 0.0f;
                local_sum += val * val;
                for (int offset = 16; offset > 0; offset /= 2)
                    local_sum += __shfl_down_sync(0xffffffffu, local_sum, offset);
                part[v] = __shfl_sync(0xffffffffu, local_sum, 0);
            }
            // the reference's second tree over its four warp partials (lanes 4..31 hold 0.0f)
            float total_sum = (part[0] + part[2]) + (part[1] + part[3]);
            const float rms = rsqrtf(total_sum / kHeadDim + p.eps);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                float val = __half2float(h[v]) * rms;
                h[v] = __float2half(val * __half2float(wv[v]));
            }
        }
        // RoPE on interleaved pairs (2i, 2i+1): neighbours in the same run (rope.cu:36-45)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const float freq = fr[v];
            float angle = freq * static_cast<float>(pos);
            float cos_a = cosf(angle), sin_a = sinf(angle);
            const float mine = __half2float(h[v]);
            const float other = __shfl_xor_sync(0xffffffffu, mine, 1);
            float q0 = (lane & 1) ? other : mine, q1 = (lane & 1) ? mine : other;
            h[v] = (lane & 1) ? __float2half(q0 * sin_a + q1 * cos_a) : __float2half(q0 * cos_a - q1 * sin_a);
        }
    }
    if (is_q) {
        __half* dst = p.q_out + (static_cast<size_t>(b) * p.n_q + head) * kHeadDim;
#pragma unroll
        for (int v = 0; v < 4; ++v) dst[v * 32 + lane] = h[v];
    } else {
        const int kvh = is_k ? head - p.n_q : head - p.n_q - p.n_kv;
        if (phys < 0) return;
        __half* cache = is_k ? p.k_cache : p.v_cache;
        __half* dst = cache + ((((static_cast<size_t>(phys) * p.n_layers + p.layer) * p.n_kv + kvh) * kBlockTokens) +
                               pos % kBlockTokens) * kHeadDim;
#pragma unroll
        for (int v = 0; v < 4; ++v) dst[v * 32 + lane] = h[v];
    }
}

// ---------------------------------------------------------------------------------------------
struct AttnParams {
    const __half* q;          // [B, n_q, 128]
    const __half* k_cache;
    const __half* v_cache;
    const int* block_table;
    const int* seq_lens;
    int max_blocks;
    int n_q, n_kv, layer, n_layers;
    float sm_scale;
    __half* out;              // [B, n_q, 128] or null
    int8_t* Xq;               // [B, n_q*128] or null: codes of `out` for the following linear
    float* Xs;                // [B, n_q*128/g]
    int g;
    int S;                    // context slices = cluster size
    // fused prologue (ROPE form): q, k, v of the new token come from the qkv projection's output
    const __half* qkv;        // [B, (n_q + 2 n_kv) * 128]
    const __half* q_norm_w;   // [128] or null
    const __half* k_norm_w;
    float eps;
    const float* freqs;       // [64]
    const int* positions;     // [B]
    __half* k_cache_w;        // the caches again, writable
    __half* v_cache_w;
    int* status;              // error word for bounded waits that ran out
    bool ahead;               // ROPE form: all it reads but qkv may be read before the dependency wait (see the kernel)
};

#ifndef W8A8_ATTN_WARPS
#define W8A8_ATTN_WARPS 8
#endif
#ifndef W8A8_ATTN_RING
#define W8A8_ATTN_RING 24
#endif
constexpr int kAttnWarps = W8A8_ATTN_WARPS;      // consumer warps
constexpr int kAttnThreads = (kAttnWarps + 1) * 32;  // + one producer warp
constexpr int kQPerKv = 4;                       // query heads per kv head handled by one CTA
constexpr int kBoxBytes = kBlockTokens * 128;    // a TMA box: 16 token rows x 128 bytes (64 dims), 128-byte swizzle
constexpr int kBlkBytes = 2 * kBoxBytes;         // one 16-token block of K (or of V): dims 0..63, then dims 64..127
constexpr int kStageBytes = 2 * kBlkBytes;       // K block, then V block
// Stages of the CTA's ring, 8 KB each: three blocks per consumer warp on their way before the query arrives, as many as fit.
// A multiple of the consumer warps: a stage then belongs to one warp, and that warp alone waits for its phases (a warp that
// meets a stage for the first time in its second phase would take "phase -1 is complete" for its block).
constexpr int kRing = W8A8_ATTN_RING;
static_assert(kRing % kAttnWarps == 0, "a stage belongs to one consumer warp");

// Byte offset, inside a K or V block in shared memory, of the 16-byte chunk that holds dims [8 c16, 8 c16 + 8) of
// token row r: the box of its 64-dim half, the row's 128 bytes, the chunk XOR-ed with the row (what the tensor
// map's 128-byte swizzle does, and what makes eight rows of one chunk column fall into eight different bank groups).
__device__ __forceinline__ uint32_t kv_chunk(int r, int c16) {
    return (c16 >> 3) * kBoxBytes + r * 128 + (((c16 & 7) ^ (r & 7)) << 4);
}


// Cosine and sine of the 64 rotation angles, two per lane (pairs lane and lane + 32). They depend on the position alone, so they
// are made before the dependency wait, and in a rolled loop: sixteen inlined evaluations per head (one per element) were some
// 700 instructions that a launch runs once, cold.
struct RopeAngles {
    float c[2], s[2];
    __device__ __forceinline__ void make(const float* freqs, int pos, int lane) {
        const float f[2] = {freqs[lane], freqs[lane + 32]};
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            const float angle = (i ? f[1] : f[0]) * static_cast<float>(pos);
            const float ca = cosf(angle), sa = sinf(angle);
            if (i) { c[1] = ca; s[1] = sa; } else { c[0] = ca; s[0] = sa; }
        }
    }
};

// One warp, one head of the new token: per-head RMSNorm in the reference's order (rms_norm.cu:23-49 with a
// 128-thread block) and interleaved-pair RoPE (rope.cu:36-45) — the arithmetic of qknorm_rope_kvwrite_kernel.
// h: elements lane, 32+lane, 64+lane, 96+lane; w: norm weights of the same elements. (A butterfly leaves in every lane the sum
// that the reference's shuffle-down tree leaves in lane 0: the same pairs, and addition commutes.)
__device__ __forceinline__ void head_norm_rope(__half (&h)[4], bool with_norm, const __half (&w)[4], float eps,
                                               const RopeAngles& rot, int lane) {
    if (with_norm) {
        float part[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            float val = __half2float(h[v]);
            part[v] = 0.0f;
            part[v] += val * val;
        }
#pragma unroll
        for (int offset = 16; offset > 0; offset /= 2)
#pragma unroll
            for (int v = 0; v < 4; ++v) part[v] += __shfl_xor_sync(0xffffffffu, part[v], offset);
        float total_sum = (part[0] + part[2]) + (part[1] + part[3]);
        const float rms = rsqrtf(total_sum / kHeadDim + eps);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            float val = __half2float(h[v]) * rms;
            h[v] = __float2half(val * __half2float(w[v]));
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {  // element 32 v + lane belongs to pair 16 v + lane / 2
        const int from = ((v & 1) << 4) + (lane >> 1);
        const float cos_a = __shfl_sync(0xffffffffu, rot.c[v >> 1], from), sin_a = __shfl_sync(0xffffffffu, rot.s[v >> 1], from);
        const float mine = __half2float(h[v]);
        const float other = __shfl_xor_sync(0xffffffffu, mine, 1);
        float q0 = (lane & 1) ? other : mine, q1 = (lane & 1) ? mine : other;
        h[v] = (lane & 1) ? __float2half(q0 * sin_a + q1 * cos_a) : __float2half(q0 * cos_a - q1 * sin_a);
    }
}

// D(16x8, fp32) += A(16x16 fp16, rows 8..15 zero) x B(16x8 fp16). Only rows 0..7 of D are kept.
__device__ __forceinline__ void mma_top_rows(float& d0, float& d1, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
    float j2, j3;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d0), "=f"(d1), "=f"(j2), "=f"(j3)
        : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(d0), "f"(d1), "f"(0.0f), "f"(0.0f));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void consumer_barrier() {  // the eight consumer warps only
    asm volatile("bar.sync 1, %0;" ::"n"(kAttnWarps * 32) : "memory");
}

// grid (S, n_kv, B), cluster (S,1,1); eight consumer warps and one producer warp per CTA.
//
// The K and V of one (sequence, kv head) are 4 KB blocks scattered over the paged cache. The producer warp brings them
// into a ring of shared-memory stages with TMA (cp.async.bulk.tensor.2d over the cache seen as rows of 256 bytes,
// two 16 x 128-byte boxes per block, 128-byte swizzle, completion counted on the stage's mbarrier; single 256-byte
// row copies were tried first and are bound by the copy engine's request rate), so no registers are tied up by bytes in
// flight. 16-token blocks are dealt round-robin, first over the cluster's CTAs, then over the consumer
// warps; a consumer waits for its block, computes on it from shared memory (ldmatrix into mma.sync.m16n8k16 with
// fp32 accumulation: scores = Q K^T with the four query heads of the group as rows 0..3 of the tile, then
// out += P V with P rounded to fp16 and the softmax denominator summed from the same rounded values) and hands the
// stage back. Partial softmax states are merged over the warps in shared memory and over the cluster through
// distributed shared memory; the epilogue can emit the o-projection's int8 codes and scales directly.
//
// ROPE form: the launch also does what qknorm_rope_kvwrite_kernel does. Consumer warps 0..3 norm and rotate the four
// query heads into shared memory; warps 4 and 5 do the same for the new k and v rows, which go to shared memory and,
// in the CTA that owns the block the new token joins, to the cache. That block is read from the cache like any other
// (possibly before the new rows are there) and the new rows are put over it in shared memory.
//
// What may be read before the dependency wait. The kernels ahead on the stream that are launched early let their dependents
// start at their first instruction, so this kernel can be running while several of them still are, a cache write or an
// update of the positions among them; the wait covers them all, an earlier read none. By default the kernel therefore
// waits before it reads anything, and lets its own dependents start after that: once any kernel behind it runs, all
// that was ahead of it is complete. Such a kernel is what `ahead` rests on (ROPE form only): the caller says that the
// positions, lengths, block table and cached rows were complete before it, and the ring is filled and the rotation angles
// are made while the projection ahead still runs (decode step at batch 8 / 1 and fast-AR frame with every layer waiting 1455 / 1260 /
// 1577 us, with the first layer waiting and the others ahead 1421 / 1252 / 1560).
#ifdef W8A8_TRACE
// Diagnostic build only: nanosecond stamps of the phases of CTA (0, 0, 0), written by consumer thread 0, kept from
// the last launch; read out by w8a8_trace_read_attn_phases.
__device__ unsigned long long g_attn_phase[8];
#define ATTN_PHASE(i)                                                                     \
    do {                                                                                  \
        if (threadIdx.x == 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) g_attn_phase[i] = w8a8::trace::now(); \
    } while (0)
#else
#define ATTN_PHASE(i) do {} while (0)
#endif

constexpr int kMaxSlices = 8;
struct __align__(16) SliceState {
    float acc[kQPerKv][kHeadDim];
    float m[kQPerKv], l[kQPerKv];
};
// Four-byte and eight-byte stores into the shared memory of the cluster's CTA 0 (at the same offset as `local` here).
__device__ __forceinline__ uint32_t in_cta0(const void* local) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(ptx::smem_u32(local)));
    return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster2(uint32_t addr, float a, float b) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <bool ROPE>
__global__ void __maxnreg__(128) paged_attention_decode_kernel(const __grid_constant__ CUtensorMap map_k,
                                                               const __grid_constant__ CUtensorMap map_v,
                                                               const AttnParams p) {
    extern __shared__ unsigned char attn_smem[];
    __shared__ __align__(8) uint64_t full_bar[kRing], empty_bar[kRing];
    __shared__ __align__(16) __half q_s[kQPerKv][kHeadDim];
    __shared__ __align__(16) __half kv_new_s[2][kHeadDim];
    __shared__ float red_m[kAttnWarps][kQPerKv], red_l[kAttnWarps][kQPerKv];
    __shared__ float red_acc[kAttnWarps][kQPerKv][kHeadDim];
    __shared__ SliceState slice_s[kMaxSlices - 1];  // in CTA 0 of the cluster: the partial states of context slices 1, 2, ...
    __shared__ float amax_s[kAttnWarps];
    __shared__ int s_fail;
    W8A8_TRACE_SCOPE();
    ATTN_PHASE(0);
    const bool ahead = ROPE && p.ahead;
    if (ahead) ptx::pdl_launch_dependents();

    const int s = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z, S = p.S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t ring = (ptx::smem_u32(attn_smem) + 1023u) & ~1023u;  // the swizzle pattern repeats every 1024 bytes
    if (threadIdx.x < kRing) {
        if (threadIdx.x == 0) {
            ptx::prefetch_tensormap(&map_k);
            ptx::prefetch_tensormap(&map_v);
            s_fail = 0;
        }
        ptx::mbar_init(&full_bar[threadIdx.x], 1);
        ptx::mbar_init(&empty_bar[threadIdx.x], 1);
        ptx::fence_barrier_init();
        ptx::fence_proxy_async();
    }
    if (!ahead) {
        ptx::pdl_wait();
        ptx::pdl_launch_dependents();
    }
    __syncthreads();  // the only whole-CTA barrier: from here on the producer warp runs by itself
    if (S > 1) cluster_arrive();  // (waited for before anything is written to another CTA: that CTA has started then)

    // The producer asks for the first 32 block numbers without waiting for the sequence length (the read is bounded by the
    // table's width), so that the two reads are one round trip, not two.
    int phys_first = 0;
    if (warp == kAttnWarps) {
        const int bi = s + lane * S;
        phys_first = bi < p.max_blocks ? p.block_table[static_cast<size_t>(b) * p.max_blocks + bi] : 0;
    }
    const int seq_len = p.seq_lens[b];
    const int n_blocks = (seq_len + kBlockTokens - 1) / kBlockTokens;
    const int n_local = s < n_blocks ? (n_blocks - s + S - 1) / S : 0;  // blocks s, s + S, s + 2 S, ...
    const int heads_here = p.n_q / p.n_kv;                                // == kQPerKv (checked on the host)

    if (warp == kAttnWarps) {
        // ------------------------------ producer ------------------------------
        // Eight blocks per round, four lanes per block (one TMA box each): a single lane issuing every copy of the
        // CTA one after the other costs more than the copies take.
        int phys_mine = phys_first;
        bool failed = false;
        for (int li0 = 0; li0 < n_local && !failed; li0 += 8) {
            if ((li0 & 31) == 0 && li0 > 0) {  // the physical numbers of the next 32 local blocks, one per lane
                const int bi = s + (li0 + lane) * S;
                phys_mine = (bi < n_blocks && bi < p.max_blocks) ? p.block_table[static_cast<size_t>(b) * p.max_blocks + bi] : 0;
            }
            const int li = li0 + (lane >> 2), box = lane & 3;
            const int phys = __shfl_sync(0xffffffffu, phys_mine, li & 31);
            const int bi = s + li * S, st = li % kRing;
            const bool live = li < n_local;
            if (live && li >= kRing && !ptx::mbar_wait_bounded(&empty_bar[st], ((li / kRing) - 1) & 1)) {
                if (box == 0) { atomicExch(p.status, 800 + st); s_fail = 1; }
                failed = true;
            }
            failed = __any_sync(0xffffffffu, failed);
            if (failed) break;
            if (live && box == 0) ptx::mbar_arrive_expect_tx(&full_bar[st], kStageBytes);
            __syncwarp();
            if (live) {  // box 0: K dims 0..63, 1: K dims 64..127, 2: V dims 0..63, 3: V dims 64..127
                const int y = ((phys < 0 ? 0 : phys) * p.n_layers + p.layer) * p.n_kv * kBlockTokens + kvh * kBlockTokens;
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                    ::"r"(ring + st * kStageBytes + box * kBoxBytes), "l"(box < 2 ? &map_k : &map_v),
                      "r"(ptx::smem_u32(&full_bar[st])), "r"((box & 1) * 128), "r"(y)
                    : "memory");
            }
        }
        ptx::pdl_wait();
    } else {
        // ------------------------------ consumers ------------------------------
        int pos = 0;
        bool owner = false;
        RopeAngles rot;
        if constexpr (ROPE) {
            pos = p.positions[b];
            rot.make(p.freqs, pos, lane);
            owner = ((pos / kBlockTokens) % S) == s;  // this CTA attends over the block the new token joins
        }
        const int new_bi = pos / kBlockTokens;
        if constexpr (ROPE) {
            // With `ahead` the first pass is a rehearsal on zeros, before the dependency wait: cold code costs about six clocks an instruction
            // (step at batch 8: 1554 -> 1536 us). Rehearsing the block loop and the merges as well takes longer than the wait
            // it hides in (1517 -> 1756 us).
#pragma unroll 1
            for (int pass = ahead ? 0 : 1; pass < 2; ++pass) {
            const bool real = pass == 1;
            if (real) {
                ptx::pdl_wait();
                W8A8_TRACE_WAITED();
                ATTN_PHASE(1);
            }
            // six head rows of the new token: the group's four query heads, then its k and its v; a warp per row
            const int total_heads = p.n_q + 2 * p.n_kv;
            for (int h = warp; h < kQPerKv + 2; h += kAttnWarps) {
                const bool role_q = h < kQPerKv, is_k = h == kQPerKv, is_v = h == kQPerKv + 1;
                const __half* norm_w = role_q ? p.q_norm_w : p.k_norm_w;
                const __half* src = p.qkv + (static_cast<size_t>(b) * total_heads +
                                             (role_q ? kvh * heads_here + h : p.n_q + (is_k ? 0 : p.n_kv) + kvh)) * kHeadDim;
                __half hq[4], wq[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    hq[v] = __float2half(0.0f);
                    if (real) hq[v] = src[v * 32 + lane];
                    wq[v] = (norm_w && !is_v) ? norm_w[v * 32 + lane] : __float2half(1.0f);
                }
                if (!is_v) head_norm_rope(hq, norm_w != nullptr, wq, p.eps, rot, lane);
                if (role_q) {
#pragma unroll
                    for (int v = 0; v < 4; ++v) q_s[h][v * 32 + lane] = hq[v];
                } else {
#pragma unroll
                    for (int v = 0; v < 4; ++v) kv_new_s[is_v ? 1 : 0][v * 32 + lane] = hq[v];
                    if (owner && real) {
                        const int phys = p.block_table[static_cast<size_t>(b) * p.max_blocks + new_bi];
                        if (phys >= 0) {
                            __half* dst = (is_k ? p.k_cache_w : p.v_cache_w) +
                                          ((((static_cast<size_t>(phys) * p.n_layers + p.layer) * p.n_kv + kvh) * kBlockTokens) +
                                           pos % kBlockTokens) * kHeadDim;
#pragma unroll
                            for (int v = 0; v < 4; ++v) dst[v * 32 + lane] = hq[v];
                        }
                    }
                }
            }
            }
            consumer_barrier();  // q and the new k / v rows are in shared memory
        }
        // q of head g (rows 4..15 of the tile are zero): A fragments of the eight 16-dim steps
        uint32_t qa[8][2];
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            qa[kk][0] = 0u;
            qa[kk][1] = 0u;
            if (g < kQPerKv) {
                if constexpr (ROPE) {
                    qa[kk][0] = *reinterpret_cast<const uint32_t*>(&q_s[g][16 * kk + 2 * t]);
                    qa[kk][1] = *reinterpret_cast<const uint32_t*>(&q_s[g][16 * kk + 8 + 2 * t]);
                } else {
                    const __half* qrow = p.q + (static_cast<size_t>(b) * p.n_q + kvh * heads_here + g) * kHeadDim;
                    qa[kk][0] = *reinterpret_cast<const uint32_t*>(qrow + 16 * kk + 2 * t);
                    qa[kk][1] = *reinterpret_cast<const uint32_t*>(qrow + 16 * kk + 8 + 2 * t);
                }
            }
        }

        ATTN_PHASE(2);  // q (and the new k / v rows) are ready
        float m_run = -1e30f, l_run = 0.0f;
        float o[16][2];  // head g, dims 8 n + 2 t, 8 n + 2 t + 1
#pragma unroll
        for (int n = 0; n < 16; ++n) { o[n][0] = 0.0f; o[n][1] = 0.0f; }

        for (int li = warp; li < n_local; li += kAttnWarps) {
            const int st = li % kRing, bi = s + li * S;
            if (!ptx::mbar_wait_bounded(&full_bar[st], (li / kRing) & 1)) {
                if (lane == 0) { atomicExch(p.status, 810 + st); s_fail = 1; }
                break;
            }
            if (li == warp) ATTN_PHASE(3);  // the warp's first block is in shared memory
            const uint32_t ks = ring + st * kStageBytes, vs = ks + kBlkBytes;
            const int tokens = min(kBlockTokens, seq_len - bi * kBlockTokens);
            if (ROPE && bi == new_bi) {  // the new token's rows over whatever the cache held there (lane: 4 dims)
                const int r = pos % kBlockTokens;
                const uint2 kn = reinterpret_cast<const uint2*>(kv_new_s[0])[lane], vn = reinterpret_cast<const uint2*>(kv_new_s[1])[lane];
                const uint32_t off = kv_chunk(r, lane >> 1) + (lane & 1) * 8;
                asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(ks + off), "r"(kn.x), "r"(kn.y) : "memory");
                asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(vs + off), "r"(vn.x), "r"(vn.y) : "memory");
            }
            // V rows past the sequence's end: their weights are exactly zero, but whatever lies there (it may not be
            // a number) must not meet the multiply. (K rows past the end only feed scores that are replaced below.)
#pragma unroll 1
            for (int r = tokens; r < kBlockTokens; ++r)
                asm volatile("st.shared.v2.u32 [%0], {%1,%1};" ::"r"(vs + (lane >> 4) * kBoxBytes + r * 128 + (lane & 15) * 8), "r"(0u)
                             : "memory");
            __syncwarp();
            // scores: two tiles of 8 tokens x eight steps of 16 dims
            float sc[2][2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                sc[j][0] = 0.0f; sc[j][1] = 0.0f;
#pragma unroll
                for (int k2 = 0; k2 < 4; ++k2) {  // matrices: dims 32 k2 + 8 (lane >> 3) of tokens 8 j + (lane & 7)
                    uint32_t r4[4];
                    ldmatrix_x4(r4, ks + kv_chunk(8 * j + (lane & 7), 4 * k2 + (lane >> 3)));
                    mma_top_rows(sc[j][0], sc[j][1], qa[2 * k2][0], qa[2 * k2][1], r4[0], r4[1]);
                    mma_top_rows(sc[j][0], sc[j][1], qa[2 * k2 + 1][0], qa[2 * k2 + 1][1], r4[2], r4[3]);
                }
            }
            float mx = -1e30f;
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int tok = j * 8 + 2 * t + e;
                    sc[j][e] = tok < tokens ? sc[j][e] * p.sm_scale : -1e30f;
                    mx = fmaxf(mx, sc[j][e]);
                }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float new_m = fmaxf(m_run, mx);
            const float corr = __expf(m_run - new_m);
            m_run = new_m;
            const __half2 p0 = __floats2half2_rn(__expf(sc[0][0] - new_m), __expf(sc[0][1] - new_m));
            const __half2 p1 = __floats2half2_rn(__expf(sc[1][0] - new_m), __expf(sc[1][1] - new_m));
            const float2 f0 = __half22float2(p0), f1 = __half22float2(p1);
            l_run = l_run * corr + ((f0.x + f0.y) + (f1.x + f1.y));
            const uint32_t pa0 = *reinterpret_cast<const uint32_t*>(&p0), pa2 = *reinterpret_cast<const uint32_t*>(&p1);
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {  // matrices (transposed): tokens 8 (m & 1) + (lane & 7), dims 16 n2 + 8 (m >> 1)
                uint32_t r4[4];
                const int m = lane >> 3;
                ldmatrix_x4_trans(r4, vs + kv_chunk(8 * (m & 1) + (lane & 7), 2 * n2 + (m >> 1)));
                o[2 * n2][0] *= corr; o[2 * n2][1] *= corr;
                o[2 * n2 + 1][0] *= corr; o[2 * n2 + 1][1] *= corr;
                mma_top_rows(o[2 * n2][0], o[2 * n2][1], pa0, pa2, r4[0], r4[1]);
                mma_top_rows(o[2 * n2 + 1][0], o[2 * n2 + 1][1], pa0, pa2, r4[2], r4[3]);
            }
            // the stage goes back to the producer; the writes above (the new rows) are ordered before its next copy
            ptx::fence_proxy_async();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&empty_bar[st]);
        }
        ATTN_PHASE(4);  // the warp's blocks are done
        // the four lanes of a quad hold the same head: their partial denominators add up
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
        if (g < kQPerKv) {
            if (t == 0) { red_m[warp][g] = m_run; red_l[warp][g] = l_run; }
#pragma unroll
            for (int n = 0; n < 16; ++n) {
                red_acc[warp][g][8 * n + 2 * t] = o[n][0];
                red_acc[warp][g][8 * n + 2 * t + 1] = o[n][1];
            }
        }
        consumer_barrier();
    }
    // ---- merge the warps (thread -> head, 2 dims) and hand the slice's state to CTA 0 of the cluster. Everything is pushed: CTA 0
    // then reads its own shared memory, and one cluster barrier is enough. (Pulled by CTA 0, every value was a round trip
    // through the cluster, eight deep at eight slices, and the others had to be kept alive with a second barrier.) ----
    ATTN_PHASE(5);
    __syncwarp();
    if (S > 1) cluster_wait();  // (every thread, the producer warp included: CTA 0 has started)
    const int hh = (warp & 7) >> 1, d0 = (warp & 1) * 64 + 2 * lane;
    float m = -1e30f, l = 0.0f, a[2] = {0.0f, 0.0f};  // of this CTA's slice, then (CTA 0) of all
    if (warp < kAttnWarps) {
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) m = fmaxf(m, red_m[w][hh]);
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) {
            const float scw = __expf(red_m[w][hh] - m);
            const float2 v2 = *reinterpret_cast<const float2*>(&red_acc[w][hh][d0]);
            l += red_l[w][hh] * scw;
            a[0] += v2.x * scw;
            a[1] += v2.y * scw;
        }
        if (s > 0) {
            SliceState& mine = slice_s[s - 1];
            st_cluster2(in_cta0(&mine.acc[hh][d0]), a[0], a[1]);
            if (d0 == 0) { st_cluster(in_cta0(&mine.m[hh]), m); st_cluster(in_cta0(&mine.l[hh]), l); }
        }
    }
    if (S > 1) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    ATTN_PHASE(6);  // every CTA of the cluster has its partial state in CTA 0
    // ---- CTA 0 of the cluster merges the S context slices, writes the 4 heads and quantises them for the o-projection ----
    if (s == 0 && warp < kAttnWarps) {
        if (S > 1) {
            const float m_own = m;
            for (int r = 0; r < S - 1; ++r) m = fmaxf(m, slice_s[r].m[hh]);
            const float own = __expf(m_own - m);
            l *= own;
            a[0] *= own;
            a[1] *= own;
            for (int r = 0; r < S - 1; ++r) {
                const float scr = __expf(slice_s[r].m[hh] - m);
                const float2 v2 = *reinterpret_cast<const float2*>(&slice_s[r].acc[hh][d0]);
                l += slice_s[r].l[hh] * scr;
                a[0] += v2.x * scr;
                a[1] += v2.y * scr;
            }
        }
        const float inv = seq_len > 0 ? 1.0f / l : 0.0f;  // empty sequence -> zeros (paged_attention.cu:44-50)
        const __half2 o2 = __floats2half2_rn(seq_len > 0 ? a[0] * inv : 0.0f, seq_len > 0 ? a[1] * inv : 0.0f);
        const int K = p.n_q * kHeadDim, ch = kvh * heads_here * kHeadDim + hh * kHeadDim + d0;  // this thread's first channel
        const size_t oo = static_cast<size_t>(b) * K + ch;
        if (p.out) *reinterpret_cast<__half2*>(p.out + oo) = o2;
        if (p.Xq) {  // int8_gemm.cu:147-211; a group is g / 2 threads (g divides 512: a power of two)
            const float2 f = __half22float2(o2);
            float amax = fmaxf(fabsf(f.x), fabsf(f.y));
            const int span = p.g / 2 < 32 ? p.g / 2 : 32;
            for (int off = span / 2; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            if (p.g > 64) {  // two, four or eight warps to a group
                if (lane == 0) amax_s[warp] = amax;
                consumer_barrier();
                const int wpg = p.g / 64, w0 = warp & ~(wpg - 1);
#pragma unroll 1
                for (int w = 0; w < wpg; ++w) amax = fmaxf(amax, amax_s[w0 + w]);
            }
            float am[2] = {amax, amax};
            if (p.g == 1) { am[0] = fabsf(f.x); am[1] = fabsf(f.y); }
            const int lg = 31 - __clz(p.g);
            int q[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float scale = am[e] / 127.0f;
                if (scale < 1e-8f) scale = 1e-8f;
                if (((ch + e) & (p.g - 1)) == 0) p.Xs[static_cast<size_t>(b) * (K >> lg) + ((ch + e) >> lg)] = scale;
                const float inv_scale = 1.0f / scale;
                q[e] = max(-127, min(127, __float2int_rn((e ? f.y : f.x) * inv_scale)));
            }
            p.Xq[oo] = static_cast<int8_t>(q[0]);
            p.Xq[oo + 1] = static_cast<int8_t>(q[1]);
        }
    }
    if (s_fail) {  // a bounded wait ran out: give copies that may still be in flight time to land before the CTA goes
#pragma unroll 1  // (unrolled copies of the runtime loops were a quarter of the kernel's code, which runs cold)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    ATTN_PHASE(7);
    W8A8_TRACE_END(4u);
}

}  // namespace

int launch_qknorm_rope_kvwrite(const __half* qkv, const __half* q_norm_w, const __half* k_norm_w, float eps,
                               const float* freqs, const int* positions, const int* block_table, int max_blocks,
                               __half* k_cache, __half* v_cache, int layer, int n_layers, int B, int n_q, int n_kv,
                               __half* q_out, cudaStream_t stream) {
    if (B == 0) return W8A8_OK;
    RopeParams p = {qkv, q_norm_w, k_norm_w, eps, freqs, positions, block_table, max_blocks, k_cache, v_cache,
                    layer, n_layers, n_q, n_kv, q_out};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(B, (n_q + 2 * n_kv + 3) / 4, 1);
    cfg.blockDim = dim3(128, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled(kPdlAttn) ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, qknorm_rope_kvwrite_kernel, p);
    if (e != cudaSuccess) return fail(W8A8_ERR_CUDA, "qknorm_rope_kvwrite launch: %s", cudaGetErrorString(e));
    return W8A8_OK;
}

// Context slices per (sequence, kv head) pair: the count that costs least for the longest sequence the block table can hold (the host knows
// the table's width, not the lengths: a wide table gets the slices of a long context). In 10 ns, fitted to a decode layer's time over 8, 4, 2
// and 1 kv heads, batches of 1 to 16 and 8 to 128 blocks, by the choices it makes:
//   15 a block of the slice           70 a round of its eight warps      300 if there is a second slice, whose state has to be merged
//   38 a slice                        160 if not all CTAs find a free SM while the projection ahead, of 48 row tiles a kv head, still runs
// Only counts whose clusters run at once, each in one GPC (room[S] of them): sixteen clusters of eight take two rounds (36 blocks 40.4 us, with three 35.8).
// It loses 0.2, 0.3, 0.7 and 0.7 % of a layer against the best count at 8, 4, 2 and 1 kv heads, 4 % at most (table widths just past a
// round). us a layer: 8 kv heads, 17 blocks, batch 1 34.3 with eight and 32.6 with one, batch 5 37.0 with two and 34.6; 45 blocks, batch 1 34.9 with
// eight and 33.0 with three, batch 3 36.9 with three and 36.6 with four; 128 blocks, batch 5 46.0 with two and 41.8 with three; 2 kv heads,
// batch 1, 25 blocks 24.7 with one and 23.4 with four.
int attention_slices(int batch, int n_kv, int blocks, int sms, const int* room) {
    const int pairs = batch * n_kv, free_sms = sms - 48 * n_kv > sms / 6 ? sms - 48 * n_kv : sms / 6;
    int best = 1;
    long best_cost = 0;
    for (int S = 1; S <= kMaxSlices; ++S) {
        if (S == 5 || S == 7 || (S > 1 && pairs > room[S])) continue;
        const long mine = (blocks + S - 1) / S, rounds = (mine + kAttnWarps - 1) / kAttnWarps;
        const long cost = 15 * mine + 70 * rounds + (S > 1 ? 300 : 0) + 38 * S + (pairs * S > free_sms ? 160 : 0);
        if (S == 1 || cost < best_cost) { best = S; best_cost = cost; }
    }
    return best;
}

namespace {
constexpr int kAttnSmem = kRing * kStageBytes + 1024;
SmemAttribute attn_attribute[2];

// Clusters of 2 .. 8 CTAs of the attention that the current device runs at once; asked for once per device.
void cluster_room(int (&room)[kMaxSlices + 1]) {
    static std::atomic<int> known[64][kMaxSlices + 1];  // plus one
    int dev = 0;
    const bool named = cudaGetDevice(&dev) == cudaSuccess && dev < 64;
    for (int S = 2; S <= kMaxSlices; ++S) {
        int n = named ? known[dev][S].load(std::memory_order_relaxed) - 1 : -1;
        if (n < 0) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(S, 1, 1);
            cfg.blockDim = dim3(kAttnThreads, 1, 1);
            cfg.dynamicSmemBytes = kAttnSmem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = S;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (attn_attribute[1](reinterpret_cast<const void*>(paged_attention_decode_kernel<true>), kAttnSmem) != cudaSuccess ||
                cudaOccupancyMaxActiveClusters(&n, paged_attention_decode_kernel<true>, &cfg) != cudaSuccess) {
                cudaGetLastError();
                n = 0;
            } else if (named) {
                known[dev][S].store(n + 1, std::memory_order_relaxed);
            }
        }
        room[S] = n;
    }
}

int launch_attention(const AttnParams& base, int B, int splits, cudaStream_t stream);
}

int launch_paged_attention_decode(const __half* q, const __half* k_cache, const __half* v_cache,
                                  const int* block_table, const int* seq_lens, int B, int n_q, int n_kv,
                                  int max_blocks, float sm_scale, int layer, int n_layers, __half* out, int g,
                                  int8_t* Xq, float* Xs, int splits, int* status, cudaStream_t stream) {
    AttnParams p = {};
    p.status = status;
    p.q = q; p.k_cache = k_cache; p.v_cache = v_cache; p.block_table = block_table; p.seq_lens = seq_lens;
    p.max_blocks = max_blocks; p.n_q = n_q; p.n_kv = n_kv; p.layer = layer; p.n_layers = n_layers; p.sm_scale = sm_scale;
    p.out = out; p.Xq = Xq; p.Xs = Xs; p.g = g;
    return launch_attention(p, B, splits, stream);
}

int launch_qkv_attention_decode(const __half* qkv, const __half* q_norm_w, const __half* k_norm_w, float eps,
                                const float* freqs, const int* positions, __half* k_cache, __half* v_cache,
                                const int* block_table, const int* seq_lens, int B, int n_q, int n_kv, int max_blocks,
                                float sm_scale, int layer, int n_layers, __half* out, int g, int8_t* Xq, float* Xs,
                                int splits, bool ahead, int* status, cudaStream_t stream) {
    AttnParams p = {};
    p.status = status;
    p.ahead = ahead;
    p.k_cache = k_cache; p.v_cache = v_cache; p.block_table = block_table; p.seq_lens = seq_lens;
    p.max_blocks = max_blocks; p.n_q = n_q; p.n_kv = n_kv; p.layer = layer; p.n_layers = n_layers; p.sm_scale = sm_scale;
    p.out = out; p.Xq = Xq; p.Xs = Xs; p.g = g;
    p.qkv = qkv; p.q_norm_w = q_norm_w; p.k_norm_w = k_norm_w; p.eps = eps; p.freqs = freqs; p.positions = positions;
    p.k_cache_w = k_cache; p.v_cache_w = v_cache;
    return launch_attention(p, B, splits, stream);
}

namespace {
int launch_attention(const AttnParams& base, int B, int splits, cudaStream_t stream) {
    const int n_q = base.n_q, n_kv = base.n_kv, g = base.g;
    const int8_t* Xq = base.Xq;
    if (B == 0) return W8A8_OK;
    if (n_kv <= 0 || n_q != n_kv * kQPerKv)
        return fail(W8A8_ERR_UNSUPPORTED, "paged attention here handles 4 query heads per kv head (got %d / %d)", n_q, n_kv);
    if (Xq && (g <= 0 || (kQPerKv * kHeadDim) % g != 0))
        return fail(W8A8_ERR_UNSUPPORTED, "fused output quantisation needs a group size dividing 512 (got %d)", g);
    if (splits <= 0) {
        int room[kMaxSlices + 1];
        cluster_room(room);
        splits = attention_slices(B, n_kv, base.max_blocks, device_sms(), room);
    }
    if (splits > kMaxSlices) splits = kMaxSlices;
    AttnParams p = base;
    p.S = splits;
    // The caches as rows of 256 bytes (one token of one head); a box is 16 rows x 128 bytes. The row count only bounds
    // the coordinates the kernel may ask for: the physical block numbers come from the caller's block table.
    CUtensorMap map_k, map_v;
    int rc = make_tensor_map_2d_u8(&map_k, p.k_cache, kHeadDim * 2, uint64_t(1) << 30, kHeadDim * 2, 128, kBlockTokens, 1);
    if (rc) return rc;
    rc = make_tensor_map_2d_u8(&map_v, p.v_cache, kHeadDim * 2, uint64_t(1) << 30, kHeadDim * 2, 128, kBlockTokens, 1);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, n_kv, B);
    cfg.blockDim = dim3(kAttnThreads, 1, 1);
    cfg.dynamicSmemBytes = kAttnSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled(kPdlAttn) ? 2 : 1;
    const cudaError_t e = p.qkv ? launch_with_smem(attn_attribute[1], kAttnSmem, cfg, paged_attention_decode_kernel<true>, map_k, map_v, p)
                                : launch_with_smem(attn_attribute[0], kAttnSmem, cfg, paged_attention_decode_kernel<false>, map_k, map_v, p);
    if (e != cudaSuccess) return fail(W8A8_ERR_CUDA, "paged_attention_decode launch: %s", cudaGetErrorString(e));
    return W8A8_OK;
}
}  // namespace

}  // namespace w8a8

W8A8_TRACE_READER(attn)
#ifdef W8A8_TRACE
extern "C" __attribute__((visibility("default"))) int w8a8_trace_read_attn_phases(unsigned long long* out8) {
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    return cudaMemcpyFromSymbol(out8, w8a8::g_attn_phase, 8 * sizeof(unsigned long long)) == cudaSuccess ? 8 : -1;
}
#endif
