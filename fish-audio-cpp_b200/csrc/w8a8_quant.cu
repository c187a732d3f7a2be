// Row kernels: residual add -> RMSNorm -> activation quantiser, any subset, one launch.
//
// One CTA owns one token row and keeps it in shared memory from the first load
// to the last store, so the chain
//     residual_add (ffn_activations.cu:41-45) -> rms_norm (rms_norm.cu:10-58)
//     -> quantize_activation_groups_kernel (int8_gemm.cu:147-211)
// costs one read of the row instead of three round trips through HBM. Every
// value that the reference would have rounded to fp16 on its way through global
// memory is rounded to fp16 here too, so the int8 codes and the fp32 scales are
// bit-identical to those of the unfused reference chain.
#include <cstdlib>

#include "sm100_ptx.cuh"
#include "w8a8_internal.h"
#include "w8a8_trace.cuh"

namespace w8a8 {
namespace {

constexpr int kWarp = 32;

struct RowQuantParams {
    const __half* x_in;
    __half* x_out;            // where x_in + residual goes (null: not stored)
    const __half* residual;   // null: no add
    const __half* norm_weight;  // null: no norm
    float eps;
    const __half* smooth_inv;
    const __half* act_scale;  // static scales [G] or null
    __half* normed_out;       // null: not stored
    int8_t* Xq;               // null: no quantisation (plain rms_norm)
    float* Xs;
    int K, g, G;
    int per_token;
    int vec_ok;               // K % 8 == 0 and all fp16 pointers 16-byte aligned
    int first_pass;           // 0: the compact kernel runs a rehearsal before its dependency wait (see rehearses)
};

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = kWarp / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Eight int8 codes (int8_gemm.cu:201-210), packed two at a time by the saturating pack instruction. A scale made from the
// group's own maximum gives no code below -127, so only a static scale (STATIC) needs the lower clamp. (At prefill sizes the
// row kernels are bound by instructions as much as by bytes; shifts and masks per code were half of them.)
__device__ __forceinline__ uint2 codes8(const float (&v)[8], float inv_scale, bool is_static) {
    int q[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) q[e] = __float2int_rn(v[e] * inv_scale);
    if (is_static) {
#pragma unroll
        for (int e = 0; e < 8; ++e) q[e] = max(-127, q[e]);
    }
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w[h]) : "r"(q[4 * h + 3]), "r"(q[4 * h + 2]), "r"(0));
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w[h]) : "r"(q[4 * h + 1]), "r"(q[4 * h]), "r"(w[h]));
    }
    return make_uint2(w[0], w[1]);
}

__global__ void __launch_bounds__(1024) rowquant_kernel(const RowQuantParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* row = reinterpret_cast<__half*>(smem_raw);
    float* gscale = reinterpret_cast<float*>(smem_raw + ((static_cast<size_t>(p.K) * 2 + 15) & ~size_t(15)));
    __shared__ float s_red[kWarp];

    const int tid = threadIdx.x;
    const int T = blockDim.x;
    const int K = p.K;
    const size_t base = static_cast<size_t>(blockIdx.x) * K;
    // Let the next kernel in the stream start its own prologue; wait for the one before this.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- stage the row (+ residual add, rounded to fp16 like residual_add_kernel) ----
    if (p.vec_ok) {
        const uint4* src = reinterpret_cast<const uint4*>(p.x_in + base);
        const uint4* res = p.residual ? reinterpret_cast<const uint4*>(p.residual + base) : nullptr;
        uint4* dst = p.x_out ? reinterpret_cast<uint4*>(p.x_out + base) : nullptr;
        for (int v = tid; v < K / 8; v += T) {
            uint4 u = src[v];
            if (res) {
                uint4 r = res[v];
                __half2* uh = reinterpret_cast<__half2*>(&u);
                const __half2* rh = reinterpret_cast<const __half2*>(&r);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float2 a = __half22float2(uh[i]), b = __half22float2(rh[i]);
                    uh[i] = __halves2half2(__float2half(a.x + b.x), __float2half(a.y + b.y));
                }
                if (dst) dst[v] = u;
            }
            reinterpret_cast<uint4*>(row)[v] = u;
        }
    } else {
        for (int i = tid; i < K; i += T) {
            __half h = p.x_in[base + i];
            if (p.residual) {
                h = __float2half(__half2float(h) + __half2float(p.residual[base + i]));
                if (p.x_out) p.x_out[base + i] = h;
            }
            row[i] = h;
        }
    }
    __syncthreads();

    // ---- RMSNorm, with the reference's summation order (rms_norm.cu:23-49): thread t sums
    // elements t, t+T, ...; shuffle-down tree inside each warp; shuffle-down tree over warps. ----
    if (p.norm_weight) {
        float local_sum = 0.0f;
        for (int i = tid; i < K; i += T) {
            float val = __half2float(row[i]);
            local_sum += val * val;
        }
        for (int offset = kWarp / 2; offset > 0; offset /= 2)
            local_sum += __shfl_down_sync(0xffffffffu, local_sum, offset);
        if ((tid & (kWarp - 1)) == 0) s_red[tid / kWarp] = local_sum;
        __syncthreads();
        float total_sum = 0.0f;
        int num_warps = (T + kWarp - 1) / kWarp;
        if (tid < num_warps) total_sum = s_red[tid];
        for (int offset = kWarp / 2; offset > 0; offset /= 2)
            total_sum += __shfl_down_sync(0xffffffffu, total_sum, offset);
        __syncthreads();
        if (tid == 0) s_red[0] = rsqrtf(total_sum / K + p.eps);
        __syncthreads();
        const float rms = s_red[0];
        for (int i = tid; i < K; i += T) {
            float val = __half2float(row[i]) * rms;
            __half o = __float2half(val * __half2float(p.norm_weight[i]));
            row[i] = o;
            if (p.normed_out) p.normed_out[base + i] = o;
        }
        __syncthreads();
    }
    if (!p.Xq) return;

    // ---- scales: one warp per group; absmax is order-free (int8_gemm.cu:177-199) ----
    const int lane = tid & (kWarp - 1), warp = tid / kWarp, nwarps = T / kWarp;
    const int g = p.g, G = p.G;
    if (p.act_scale) {
        for (int j = tid; j < G; j += T) {
            float s = __half2float(p.act_scale[j]);
            gscale[j] = s < 1e-8f ? 1e-8f : s;
        }
    } else {
        for (int j = warp; j < G; j += nwarps) {
            int start = j * g, end = min(start + g, K);
            float m = 0.0f;
            for (int k = start + lane; k < end; k += kWarp) {
                float v = __half2float(row[k]);
                if (p.smooth_inv) v *= __half2float(p.smooth_inv[k]);
                m = fmaxf(m, fabsf(v));
            }
            m = warp_max(m);
            if (lane == 0) gscale[j] = m;  // absmax for now
        }
        __syncthreads();
        if (p.per_token) {
            float m = 0.0f;
            for (int j = tid; j < G; j += T) m = fmaxf(m, gscale[j]);
            m = warp_max(m);
            if (lane == 0) s_red[warp] = m;
            __syncthreads();
            m = 0.0f;
            for (int w = 0; w < nwarps; ++w) m = fmaxf(m, s_red[w]);
            __syncthreads();
            for (int j = tid; j < G; j += T) gscale[j] = m;
            __syncthreads();
        }
        for (int j = tid; j < G; j += T) {
            float s = gscale[j] / 127.0f;
            gscale[j] = s < 1e-8f ? 1e-8f : s;
        }
    }
    __syncthreads();
    for (int j = tid; j < G; j += T) p.Xs[static_cast<size_t>(blockIdx.x) * G + j] = gscale[j];

    // ---- codes (int8_gemm.cu:201-210) ----
    int8_t* q_row = p.Xq + base;
    if ((K & 3) == 0 && (g & 3) == 0) {
        for (int w4 = tid; w4 < K / 4; w4 += T) {
            const int k0 = w4 * 4;
            const float inv_scale = 1.0f / gscale[k0 / g];
            uint32_t packed = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v = __half2float(row[k0 + i]);
                if (p.smooth_inv) v *= __half2float(p.smooth_inv[k0 + i]);
                int q = __float2int_rn(v * inv_scale);
                q = max(-127, min(127, q));
                packed |= (static_cast<uint32_t>(q) & 0xffu) << (8 * i);
            }
            reinterpret_cast<uint32_t*>(q_row)[w4] = packed;
        }
    } else {
        for (int k = tid; k < K; k += T) {
            const float inv_scale = 1.0f / gscale[k / g];
            float v = __half2float(row[k]);
            if (p.smooth_inv) v *= __half2float(p.smooth_inv[k]);
            int q = __float2int_rn(v * inv_scale);
            q = max(-127, min(127, q));
            q_row[k] = static_cast<int8_t>(q);
        }
    }
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Register-resident form of the fused row kernel for rows of at most 4 x blockDim elements (the decode
// case: K = 2560 with 1024 threads). Same arithmetic and the same summation order as rowquant_kernel —
// thread t owns elements t, t+T, t+2T, ... exactly like the reference's rms_norm launch — but nothing is
// staged in shared memory and only three block barriers separate the first load from the last store;
// at 8 rows per launch the kernel's length is a latency chain, not a bandwidth figure. Needs g % 32 == 0
// so that the 32 lanes of a warp always sit in one quantisation group.
constexpr int kFastElems = 4;
__global__ void __launch_bounds__(1024) rowquant_fast_kernel(const RowQuantParams p) {
    __shared__ float s_red[kWarp];
    __shared__ unsigned s_gmax[160];  // absmax per group as float bits (non-negative floats order like uints)
    const int tid = threadIdx.x, T = blockDim.x, K = p.K, g = p.g, G = p.G;
    const int lane = tid & (kWarp - 1), warp = tid / kWarp;
    const size_t base = static_cast<size_t>(blockIdx.x) * K;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // the norm weight and the smoothing vector are parameters, not results of the kernel before this one
    __half nw[kFastElems], sm[kFastElems];
#pragma unroll
    for (int i = 0; i < kFastElems; ++i) {
        const int e = tid + i * T;
        if (e < K) {
            if (p.norm_weight) nw[i] = p.norm_weight[e];
            if (p.smooth_inv) sm[i] = p.smooth_inv[e];
        }
    }
    for (int j = tid; j < G; j += T) s_gmax[j] = 0u;
    asm volatile("griddepcontrol.wait;" ::: "memory");

    __half h[kFastElems], res[kFastElems];
    float local_sum = 0.0f;
    // every load is requested before the first store: x_out may be x_in, so a load placed after a store
    // would have to wait for it, one memory round trip per element
#pragma unroll
    for (int i = 0; i < kFastElems; ++i) {
        const int e = tid + i * T;
        if (e < K) {
            h[i] = p.x_in[base + e];
            if (p.residual) res[i] = p.residual[base + e];
        }
    }
#pragma unroll
    for (int i = 0; i < kFastElems; ++i) {
        const int e = tid + i * T;
        if (e < K) {
            __half v = h[i];
            if (p.residual) {
                v = __float2half(__half2float(v) + __half2float(res[i]));
                if (p.x_out) p.x_out[base + e] = v;
            }
            h[i] = v;
            float val = __half2float(v);
            local_sum += val * val;
        }
    }
    if (p.norm_weight) {
        for (int offset = kWarp / 2; offset > 0; offset /= 2)
            local_sum += __shfl_down_sync(0xffffffffu, local_sum, offset);
        if (lane == 0) s_red[warp] = local_sum;
        __syncthreads();
        float total_sum = 0.0f;
        const int num_warps = (T + kWarp - 1) / kWarp;
        if (tid < num_warps) total_sum = s_red[tid];
        if (warp == 0) {
            for (int offset = kWarp / 2; offset > 0; offset /= 2)
                total_sum += __shfl_down_sync(0xffffffffu, total_sum, offset);
        }
        __syncthreads();
        if (tid == 0) s_red[0] = rsqrtf(total_sum / K + p.eps);
        __syncthreads();
        const float rms = s_red[0];
#pragma unroll
        for (int i = 0; i < kFastElems; ++i) {
            const int e = tid + i * T;
            if (e < K) {
                float val = __half2float(h[i]) * rms;
                h[i] = __float2half(val * __half2float(nw[i]));
                if (p.normed_out) p.normed_out[base + e] = h[i];
            }
        }
    }
    if (!p.Xq) return;
    float v[kFastElems];
#pragma unroll
    for (int i = 0; i < kFastElems; ++i) {
        const int e = tid + i * T;
        v[i] = 0.0f;
        if (e < K) {
            v[i] = __half2float(h[i]);
            if (p.smooth_inv) v[i] *= __half2float(sm[i]);
        }
    }
    if (!p.act_scale) {
#pragma unroll
        for (int i = 0; i < kFastElems; ++i) {
            const int e0 = warp * kWarp + i * T;  // first element of this warp's run
            if (e0 < K) {
                float m = warp_max(fabsf(v[i]));
                if (lane == 0) atomicMax(&s_gmax[p.per_token ? 0 : e0 / g], __float_as_uint(m));
            }
        }
    }
    __syncthreads();
    for (int j = tid; j < G; j += T) {
        float sc = p.act_scale ? __half2float(p.act_scale[j]) : __uint_as_float(s_gmax[p.per_token ? 0 : j]) / 127.0f;
        if (sc < 1e-8f) sc = 1e-8f;
        p.Xs[static_cast<size_t>(blockIdx.x) * G + j] = sc;
    }
#pragma unroll
    for (int i = 0; i < kFastElems; ++i) {
        const int e = tid + i * T;
        if (e < K) {
            const int j = e / g;
            float sc = p.act_scale ? __half2float(p.act_scale[j]) : __uint_as_float(s_gmax[p.per_token ? 0 : j]) / 127.0f;
            if (sc < 1e-8f) sc = 1e-8f;
            const float inv_scale = 1.0f / sc;
            int q = __float2int_rn(v[i] * inv_scale);
            q = max(-127, min(127, q));
            p.Xq[base + e] = static_cast<int8_t>(q);
        }
    }
}

// residual add + RMSNorm + group quantiser of one token row by 128 threads, for the decode step; K a multiple of 256 up to
// 4096, g in {64, 128, 256}. At 8 rows a launch is a latency chain: what counts is its length. Thread t owns the 16-byte
// pieces t + 128 i, i.e. elements 8 t + j + 1024 i (j < 8): ALL the elements of the reference's virtual threads 8 t + j of its
// 1024-thread launch (rms_norm.cu:23-27), in its order of addition. (For K <= 512 the reference launches fewer threads; the
// virtual threads past K then add zeros, which changes no sum.) Its shuffle-down tree over a virtual warp (virtual lanes
// 8 (l % 4) + j) crosses real lanes twice and stays inside a thread three times; the 32 sums go through shared memory, one
// barrier, and every warp runs the second tree (rms_norm.cu:36-42) itself. (Before: the row staged in shared memory by 256
// threads, rounds of serial sums and five-step trees, five barriers.)
// The first pass is a rehearsal on the norm weights, with nothing stored, while the kernel before this one still runs: code
// that runs for the first time after another kernel costs about six clocks an instruction, warm code a fifth of that,
// and a launch of this kernel runs its code once. (Decode step, batch 8: 1726 -> 1700 us together with the quantiser's.
// The same in the linear's CTAs made the step slower. Which launches rehearse: see rehearses.)
template <int GM>
__global__ void __launch_bounds__(128) rowquant_compact_kernel(const __grid_constant__ RowQuantParams p) {
    constexpr int LANES = GM / 8, kPieces = 4;
    __shared__ float s_red[2][32];
    const int tid = threadIdx.x, lane = tid & 31, K = p.K, pieces = K / 8, row = blockIdx.x;
    const size_t base = static_cast<size_t>(row) * K;
    W8A8_TRACE_SCOPE();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    uint4 wv[kPieces];
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
        const int c8 = tid + i * 128;
        wv[i] = __ldg(reinterpret_cast<const uint4*>(p.norm_weight) + (c8 < pieces ? c8 : 0));
    }
    const __half* res = p.residual ? p.residual : p.x_in;
#pragma unroll 1
    for (int pass = p.first_pass; pass < 2; ++pass) {
        const bool real = pass == 1;
        if (real) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            W8A8_TRACE_WAITED();
        }
        uint4 xv[kPieces], dv[kPieces];
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {  // every load first
            const int c8 = tid + i * 128;
            xv[i] = dv[i] = wv[i];
            if (real && c8 < pieces) {
                xv[i] = *reinterpret_cast<const uint4*>(p.x_in + base + c8 * 8);
                dv[i] = *reinterpret_cast<const uint4*>(res + base + c8 * 8);
            }
        }
        float ls[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) ls[j] = 0.0f;
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int c8 = tid + i * 128;
            if (c8 < pieces) {
                __half* hx = reinterpret_cast<__half*>(&xv[i]);
                if (p.residual) {
                    const __half* hd = reinterpret_cast<const __half*>(&dv[i]);
#pragma unroll
                    for (int e = 0; e < 8; ++e) hx[e] = __float2half(__half2float(hx[e]) + __half2float(hd[e]));
                    if (real && p.x_out) *reinterpret_cast<uint4*>(p.x_out + base + c8 * 8) = xv[i];
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float val = __half2float(hx[j]);
                    ls[j] += val * val;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ls[j] += __shfl_down_sync(0xffffffffu, ls[j], 2);  // virtual offset 16
#pragma unroll
        for (int j = 0; j < 8; ++j) ls[j] += __shfl_down_sync(0xffffffffu, ls[j], 1);  // virtual offset 8
#pragma unroll
        for (int j = 0; j < 4; ++j) ls[j] += ls[j + 4];
        ls[0] += ls[2];
        ls[1] += ls[3];
        if ((lane & 3) == 0) s_red[pass][tid >> 2] = ls[0] + ls[1];
        __syncthreads();
        float total_sum = s_red[pass][lane];
#pragma unroll
        for (int offset = 16; offset > 0; offset /= 2) total_sum += __shfl_xor_sync(0xffffffffu, total_sum, offset);
        const float rms = rsqrtf(total_sum / K + p.eps);
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int c8 = tid + i * 128;
            if (c8 >= pieces) break;  // (whole warps: pieces is a multiple of 32)
            __half* hx = reinterpret_cast<__half*>(&xv[i]);
            const __half* hw = reinterpret_cast<const __half*>(&wv[i]);
            float v[8], amax = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float val = __half2float(hx[e]) * rms;
                hx[e] = __float2half(val * __half2float(hw[e]));
                v[e] = __half2float(hx[e]);
                amax = fmaxf(amax, fabsf(v[e]));
            }
            if (real && p.normed_out) *reinterpret_cast<uint4*>(p.normed_out + base + c8 * 8) = xv[i];
            if (!p.Xq) continue;
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            float scale = amax / 127.0f;
            if (scale < 1e-8f) scale = 1e-8f;
            if (real && (lane & (LANES - 1)) == 0) p.Xs[static_cast<size_t>(row) * p.G + (c8 * 8) / GM] = scale;
            const uint2 cd = codes8(v, 1.0f / scale, false);
            if (real) *reinterpret_cast<uint2*>(p.Xq + base + c8 * 8) = cd;
        }
    }
    W8A8_TRACE_END(2u);
}

// [residual add] -> RMSNorm -> [group quantiser] for many rows (prefill): a WARP per row, the row in registers from the
// load to the codes, no shared memory and no barrier; K a multiple of 256, 512 < K <= 256 * KI, g in {64, 128, 256}.
// Lane l owns the 16-byte pieces l + 32 i of its row, i.e. elements e = 8 l + j + 256 i (j < 8): these are ALL the elements
// of the reference's virtual threads vt = 8 l + j + 256 (i mod 4) of its 1024-thread launch (rms_norm.cu:23-27), which sum
// e = vt, vt + 1024, ... in that order, so its sum of squares can be taken in exactly the reference's order.
// A row kernel at these sizes is bandwidth: what counts is loads in flight. A CTA per row (rowquant_compact_kernel) has
// two 16-byte loads per thread and four barriers: 8192 x 2560 took 40 us (1.6 TB/s); ten per lane and no barrier: 19 us.
template <int GM, int KI>
__global__ void __launch_bounds__(128, KI > 10 ? 4 : 5) rownorm_warp_kernel(const RowQuantParams p, int M) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31, row = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= M) return;
    const int K = p.K, iters = K / 256;
    const size_t base = static_cast<size_t>(row) * K;
    const __half* res = KI <= 10 && p.residual ? p.residual + base : nullptr;  // (wider rows with a residual: a CTA per row)
    uint4 v[KI];
#pragma unroll
    for (int i = 0; i < KI; ++i)
        if (i < iters) v[i] = reinterpret_cast<const uint4*>(p.x_in + base)[lane + 32 * i];
    if (res) {
#pragma unroll
        for (int i0 = 0; i0 < KI; i0 += 5) {  // five residual pieces in flight at a time
            uint4 r[5];
#pragma unroll
            for (int i = 0; i < 5; ++i)
                if (i0 + i < KI && i0 + i < iters) r[i] = reinterpret_cast<const uint4*>(res)[lane + 32 * (i0 + i)];
#pragma unroll
            for (int i = 0; i < 5; ++i)
                if (i0 + i < KI && i0 + i < iters) {
                    __half* hv = reinterpret_cast<__half*>(&v[i0 + i < KI ? i0 + i : 0]);
                    const __half* hr = reinterpret_cast<const __half*>(&r[i]);
#pragma unroll
                    for (int e = 0; e < 8; ++e) hv[e] = __float2half(__half2float(hv[e]) + __half2float(hr[e]));
                }
        }
        if (p.x_out) {  // (may be x_in: every load of the row is above)
#pragma unroll
            for (int i = 0; i < KI; ++i)
                if (i < iters) reinterpret_cast<uint4*>(p.x_out + base)[lane + 32 * i] = v[i];
        }
    }
    float ls[4][8];  // per virtual thread (r, j): its elements i = r, r + 4, r + 8, ... ascending
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int j = 0; j < 8; ++j) ls[r][j] = 0.0f;
#pragma unroll
    for (int i = 0; i < KI; ++i)
        if (i < iters) {
            const __half* hv = reinterpret_cast<const __half*>(&v[i]);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float val = __half2float(hv[j]);
                ls[i & 3][j] += val * val;
            }
        }
    // The reference's shuffle-down tree over a virtual warp: virtual warp (r, l / 4) is made of the virtual lanes
    // 8 (l % 4) + j; offsets 16 and 8 cross real lanes (l + 2, l + 1), offsets 4, 2, 1 stay inside the lane's eight j. Only
    // virtual lane 0 is used afterwards, and it takes exactly the reference's operands in the reference's order.
    float wsum[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float b8[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float local_sum = ls[r][j];
            local_sum += __shfl_down_sync(0xffffffffu, local_sum, 2);
            local_sum += __shfl_down_sync(0xffffffffu, local_sum, 1);
            b8[j] = local_sum;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) b8[j] += b8[j + 4];
        b8[0] += b8[2];
        b8[1] += b8[3];
        wsum[r] = b8[0] + b8[1];
    }
    // second tree (rms_norm.cu:36-42): lane w takes the sum of virtual warp w = 8 r + q, which lives in lane 4 q
    float total_sum = 0.0f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float t = __shfl_sync(0xffffffffu, wsum[r], 4 * (lane & 7));
        if ((lane >> 3) == r) total_sum = t;
    }
    for (int offset = 16; offset > 0; offset /= 2) total_sum += __shfl_down_sync(0xffffffffu, total_sum, offset);
    total_sum = __shfl_sync(0xffffffffu, total_sum, 0);
    const float rms = rsqrtf(total_sum / K + p.eps);
    constexpr int LANES = GM / 8;
#pragma unroll
    for (int i = 0; i < KI; ++i)
        if (i < iters) {
            const int c8 = lane + 32 * i;
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(p.norm_weight) + c8);
            __half* hv = reinterpret_cast<__half*>(&v[i]);
            const __half* hw = reinterpret_cast<const __half*>(&w);
            float f[8], amax = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float val = __half2float(hv[e]) * rms;
                hv[e] = __float2half(val * __half2float(hw[e]));
                f[e] = __half2float(hv[e]);
                amax = fmaxf(amax, fabsf(f[e]));
            }
            if (p.normed_out) reinterpret_cast<uint4*>(p.normed_out + base)[c8] = v[i];
            if (p.Xq) {
#pragma unroll
                for (int o = LANES / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                float scale = amax / 127.0f;
                if (scale < 1e-8f) scale = 1e-8f;
                if ((lane & (LANES - 1)) == 0) p.Xs[static_cast<size_t>(row) * p.G + (c8 * 8) / GM] = scale;
                *reinterpret_cast<uint2*>(p.Xq + base + c8 * 8) = codes8(f, 1.0f / scale, false);
            }
        }
}

// The quantiser alone (int8_gemm.cu:147-211) for g in {64, 128, 256}, K a multiple of g: no shared memory, no block
// barrier. A thread owns 8 consecutive activations (one 128-bit load), the g/8 threads of a group find the absmax with
// shuffles, and each thread stores its 8 codes as one 64-bit word. The groups of all rows lie one after another ([M, K] and
// [M, G] are contiguous and K is a multiple of g), so the whole matrix is one flat run of pieces. At decode sizes it is a
// few KB, and what counts is the length of the dependency chain (one load, log2(g/8) shuffles, one divide, one store): one
// piece per thread (U = 1). At prefill sizes it is bandwidth: four loads in flight per thread (8192 x 9728: 86 -> 37 us, 6.5 TB/s).
// Twelve CTAs of that form fit an SM with 40 registers a thread; compiled to 44 it ran at eleven (8192 x 9728 36.5 -> 38.4 us). Only the
// outputs are __restrict__: loads may move past stores, and are still not taken for constant.
template <int LANES, int U>  // LANES: threads per group = g / 8
__global__ void __launch_bounds__(128, U == 1 ? 1 : 12) groupquant_kernel(const __half* X, const __half* smooth_inv, const __half* act_scale,
                                                         int8_t* __restrict__ Xq, float* __restrict__ Xs, unsigned pieces, unsigned K8, int first_pass) {
    W8A8_TRACE_SCOPE();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll 1
    for (int pass = U == 1 ? first_pass : 1; pass < 2; ++pass) {
    const bool real = pass == 1;
    if (real) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        W8A8_TRACE_WAITED();
    }
    const unsigned p0 = blockIdx.x * (128u * U) + threadIdx.x;
    // Neither smoothing nor static scales are read by the rehearsal: they may be results of the launch ahead. With one piece per
    // thread they are asked for with the activations: after those had arrived it was a second memory latency (8 x 9728: 2.5 -> 2.1 us).
    uint4 u[U], su = make_uint4(0, 0, 0, 0);
    float st = 0.0f;
#pragma unroll
    for (int k = 0; k < U; ++k)  // (a whole group is live or not: pieces is a multiple of LANES)
        u[k] = real && p0 + k * 128u < pieces ? ptx::ld_result_v4(reinterpret_cast<const uint4*>(X) + p0 + k * 128u) : make_uint4(0, 0, 0, 0);
    auto load_vectors = [&](unsigned pc) {
        const unsigned c8 = pc % K8;  // piece inside its row
        if (smooth_inv) su = *(reinterpret_cast<const uint4*>(smooth_inv) + c8);
        if (act_scale) st = __half2float(act_scale[c8 / LANES]);
    };
    const bool vectors = real && (smooth_inv || act_scale);
    if (U == 1 && vectors) load_vectors(p0);
#pragma unroll
    for (int k = 0; k < U; ++k) {
        const unsigned pc = p0 + k * 128u;
        const bool live = pc < pieces;
        const __half* h = reinterpret_cast<const __half*>(&u[k]);
        float v[8], amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __half2float(h[i]);
        if (U != 1 && vectors) load_vectors(pc);
        if (smooth_inv) {
            const __half* sh = reinterpret_cast<const __half*>(&su);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] *= __half2float(sh[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (!live) continue;
        float scale = act_scale ? st : amax / 127.0f;
        if (scale < 1e-8f) scale = 1e-8f;
        if (real && (threadIdx.x & (LANES - 1)) == 0) Xs[pc / LANES] = scale;
        const uint2 cd = codes8(v, 1.0f / scale, act_scale != nullptr);
        if (real) *reinterpret_cast<uint2*>(Xq + static_cast<size_t>(pc) * 8) = cd;
    }
    }
    W8A8_TRACE_END(3u);
}

template <typename... Params, typename... Args>
int launch_row_kernel(const char* what, void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t stream,
                      Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled(kPdlRow) ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) return fail(W8A8_ERR_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
    return W8A8_OK;
}

// A rehearsal pays where the kernel ahead lets this one start early and is still busy: behind the decode linears, up to 32 rows. The
// GEMM lets nothing start before its end, so behind it, as behind other kernels, the rehearsal is time added, once per CTA
// (quantiser at 600 x 4096 3.8 us without and 4.7 with, at 150 x 2560 2.3 and 2.7; row kernel at 600 x 2560 6.6 and 6.9).
bool rehearses(int rows) { return rows <= 32; }

template <int LANES>
int launch_groupquant(const __half* X, const __half* smooth_inv, const __half* act_scale, int8_t* Xq, float* Xs,
                      unsigned pieces, unsigned K8, int first_pass, cudaStream_t stream) {
    // four pieces per thread once the single-piece form would fill every SM with more than two rounds of threads
    if (pieces > static_cast<unsigned>(device_sms()) * 2048u * 2u)
        return launch_row_kernel("groupquant", groupquant_kernel<LANES, 4>, (pieces + 511) / 512, 128, 0, stream, X, smooth_inv,
                                 act_scale, Xq, Xs, pieces, K8, first_pass);
    return launch_row_kernel("groupquant", groupquant_kernel<LANES, 1>, (pieces + 127) / 128, 128, 0, stream, X, smooth_inv, act_scale,
                             Xq, Xs, pieces, K8, first_pass);
}

template <int GM>
int launch_rownorm_warp(const RowQuantParams& p, int M, cudaStream_t stream) {
    const unsigned blocks = (M + 3) / 4;
    if (p.K <= 2560) return launch_row_kernel("rownorm_warp", rownorm_warp_kernel<GM, 10>, blocks, 128, 0, stream, p, M);
    return launch_row_kernel("rownorm_warp", rownorm_warp_kernel<GM, 16>, blocks, 128, 0, stream, p, M);
}

}  // namespace

int launch_rowquant(const __half* x_in, __half* x_out, const __half* residual,
                    const __half* norm_weight, float eps, const __half* smooth_inv,
                    const __half* act_scale, int M, int K, int g, int act_mode, __half* normed_out,
                    int8_t* Xq, float* Xs, cudaStream_t stream) {
    if (M == 0) return W8A8_OK;
    {   // the quantiser alone, common group sizes: the barrier-free kernel (pieces are counted in 32 bits)
        const int gn = norm_group(K, g);
        if (!residual && !norm_weight && !normed_out && Xq && act_mode == W8A8_ACT_PER_TOKEN_GROUP &&
            (gn == 64 || gn == 128 || gn == 256) && K % gn == 0 && static_cast<long long>(M) * K / 8 < (1ll << 31) && aligned16(x_in) &&
            (reinterpret_cast<uintptr_t>(Xq) & 7u) == 0 && (!smooth_inv || aligned16(smooth_inv))) {
            const unsigned pieces = static_cast<unsigned>(static_cast<long long>(M) * K / 8), K8 = static_cast<unsigned>(K / 8);
            const int first = rehearses(M) ? 0 : 1;
            if (gn == 64) return launch_groupquant<8>(x_in, smooth_inv, act_scale, Xq, Xs, pieces, K8, first, stream);
            if (gn == 128) return launch_groupquant<16>(x_in, smooth_inv, act_scale, Xq, Xs, pieces, K8, first, stream);
            return launch_groupquant<32>(x_in, smooth_inv, act_scale, Xq, Xs, pieces, K8, first, stream);
        }
    }
    RowQuantParams p;
    p.x_in = x_in;
    p.x_out = x_out;
    p.residual = residual;
    p.norm_weight = norm_weight;
    p.eps = eps;
    p.smooth_inv = smooth_inv;
    p.act_scale = act_scale;
    p.normed_out = normed_out;
    p.Xq = Xq;
    p.Xs = Xs;
    p.K = K;
    p.g = norm_group(K, g);
    p.G = num_groups(K, g);
    p.per_token = act_mode == W8A8_ACT_PER_TOKEN;
    p.first_pass = rehearses(M) ? 0 : 1;
    p.vec_ok = (K % 8 == 0) && aligned16(x_in) && (!residual || aligned16(residual)) &&
               (!x_out || aligned16(x_out));
    // The norm must run with the reference's block size to reproduce its summation order:
    // min(1024, next_pow2(dim)), rms_norm.cu:69-70.
    int threads = 256;
    if (norm_weight) {
        threads = 1;
        while (threads < K && threads < 1024) threads <<= 1;
        if (threads < 32) threads = 32;  // shuffles need whole warps; lanes past K add 0.0f
    } else if (K >= 4096) {
        threads = 512;
    }
    static const bool compact_ok = [] {
        const char* v = std::getenv("W8A8_ROW_COMPACT");
        return v ? (*v && *v != '0') : true;
    }();
    // (without codes to make, the group size does not matter)
    const int gm = Xq ? p.g : 256;
    if (compact_ok && norm_weight && threads >= 256 && K % 256 == 0 && K <= 4096 && !smooth_inv && !act_scale && (!p.per_token || !Xq) &&
        (gm == 64 || gm == 128 || gm == 256) && p.vec_ok && aligned16(norm_weight) &&
        (!normed_out || aligned16(normed_out)) && (!Xq || (reinterpret_cast<uintptr_t>(Xq) & 7u) == 0)) {
        // A CTA per row has the shorter chain, a warp per row more bytes in flight. CTA / warp, us: 1185 x 2560 5.8 / 7.6, 1700 6.9 /
        // 7.8, 2048 8.4 / 7.9, 8192 31.8 / 21.2; 1185 x 1024 4.3 / 4.6, 1400 4.8 / 4.7. Past 2560 columns a warp per row fits an SM
        // sixteen times, and a second wave has to be worth it: 2368 x 4096 11.5 / 10.7, 2500 12.7 / 18.9, 4001 19.4 / 21.5, 8192 38.6 /
        // 36.5; with a residual it never is (sixteen loads, then four rounds of the residual): 1185 x 4096 7.8 / 13.4, 8192 47 / 69.
        const int sms = device_sms();
        const bool warp_per_row = threads == 1024 && M > sms * (K <= 1024 ? 9 : 13) &&
                                  (K <= 2560 || (!residual && (M <= sms * 16 || M > sms * 40)));
        if (warp_per_row)
            return gm == 64 ? launch_rownorm_warp<64>(p, M, stream) : gm == 128 ? launch_rownorm_warp<128>(p, M, stream)
                                                                                : launch_rownorm_warp<256>(p, M, stream);
        return launch_row_kernel("rowquant_compact", gm == 64    ? rowquant_compact_kernel<64>
                                                     : gm == 128 ? rowquant_compact_kernel<128>
                                                                 : rowquant_compact_kernel<256>, M, 128, 0, stream, p);
    }
    if (norm_weight && threads >= 32 && K <= kFastElems * threads && p.g % 32 == 0 && p.G <= 160)
        return launch_row_kernel("rowquant_fast", rowquant_fast_kernel, M, threads, 0, stream, p);
    size_t smem = ((static_cast<size_t>(K) * 2 + 15) & ~size_t(15)) + static_cast<size_t>(p.G) * 4;
    if (smem > 200 * 1024) return fail(W8A8_ERR_UNSUPPORTED, "row of K=%d does not fit shared memory", K);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(rowquant_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(smem));
        if (e != cudaSuccess) return fail(W8A8_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    }
    return launch_row_kernel("rowquant", rowquant_kernel, M, threads, smem, stream, p);
}

}  // namespace w8a8

W8A8_TRACE_READER(quant)
