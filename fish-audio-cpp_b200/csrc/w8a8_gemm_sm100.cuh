// Large-M (prefill) W8A8 linear on the 5th-generation tensor cores: TMA -> shared memory -> tcgen05.mma kind::i8 ->
// int32 accumulators in tensor memory -> fp32 promote per K-group -> fp16. Kernel template; instantiated per group size
// by w8a8_gemm_sm100_g*.cu, chosen and launched by w8a8_gemm_sm100.cu.
//
// Replaces, for tokens > 32, the reference's loop of one cuBLAS int8 GEMM per K-group plus an accumulate pass over the
// whole [tokens, rows] matrix per group and a cast pass (int8_gemm.cu:423-505): here a K-group's exact int32 sums never
// leave the SM.
//
// Roles of the operands: the WEIGHTS are the MMA's A operand (128 weight rows = the 128 tensor-memory lanes of a CTA),
// the TOKENS are B (BT columns), so that the token width BT of a tile can be fitted to the problem (32 ... 256): short
// prompts get narrow tiles and with them enough CTAs, long ones get wide tiles and fewer operand bytes. The warps:
//   warp 0       producer: TMA loads of 128 weight rows and BT token rows, 128 bytes of K each (both matrices are
//                row-major with K contiguous, i.e. already the K-major operand; TMA applies the 128-byte swizzle)
//   warp 1       MMA issuer: four tcgen05.mma (K = 32) per stage; every K-group accumulates into its own BT-column slice
//                of tensor memory (two or four slices), starting with "overwrite"
//   warps 2, 3   stage the scales of four K-groups at a time in a ring of their own
//   warps 4 ...  epilogue, eight or sixteen warps, each 32 weight rows x a part of the tokens. For every K-group
//                acc = fma(float(P) * ws, xs, acc), groups ascending -- the arithmetic and order of
//                accumulate_group_kernel (int8_gemm.cu:213-234) -- in fp32 registers, then the fp16 store
// One persistent CTA (or CTA pair) per SM (pair of SMs) walks over the tiles; all rings keep running across tiles, so
// the store of a tile overlaps the MMAs of the next.
//
// PAIR: the two CTAs of a cluster share 256 weight rows x BT tokens: each loads its own 128 weight rows and HALF of the
// tokens, the leader issues tcgen05.mma.cta_group::2 (M = 256) and each CTA ends with the sums of its own rows. A third
// fewer operand bytes per MAC through L2 and through each SM's shared-memory port. No load is multicast: each CTA issues
// plain TMA loads into its own shared memory, completing on the leader's mbarrier.
//
// What bounds it (measured with operands resident, no loads, no epilogue): an MMA of 128 x 256 x 32 takes 128 clocks, so
// the issuing warp has 512 clocks per stage of four. Run by a single lane, with stage index, parities and descriptors in
// registers, that warp needed 800-880 clocks per stage WHATEVER the tile (each instruction of a lone warp costs its full
// latency, and descriptors computed in divergent code are moved to uniform registers one by one): the tensor pipe ran at
// 0.6 of its rate. Hence: the whole warp runs the loop and one elected lane issues; the loop is unrolled over the stages
// so that stage, accumulator slice and descriptor offsets are immediates; group sizes 64 / 128 / 256 are template cases.
// The promote is the other side, and at g = 64 the bound: per sum one int -> fp32 conversion (64 a clock and SM), half a
// packed multiply and half a packed FMA, about 3 clocks per warp and scheduler, 770 clocks per group of a 128 x 256 tile
// against 256 of MMAs; with tensor-memory and shared loads 870-900 (measured alone). So the sums are read in the layout of
// an mma.sync accumulator (16x256b): a lane then holds 4 weight rows x 2 tokens of every 16 x 8 block and needs one
// 8-byte read of activation scales per eight sums. With a thread per row (32x32b) it was a 16-byte read per four, and a
// 16-byte read costs 8 clocks per scheduler even when all lanes read the same address: the promote took twice as long.
// The other exact conversions (integer add into the mantissa of 1.5 * 2^23, the bias taken out by a subtract or inside
// the multiply) measured 15-25 % slower than the conversion instruction: they compete with the FMAs for their pipe.
//
// Measured, M x N x K = 8192 x 19456 x 2560: g = 256 591 us -> 346 us (1381 -> 2360 TOPS), g = 64 1511 us -> 898 us
// (540 -> 909 TOPS), against the form before (tokens as A, one lane issuing, a thread per token row).
//
// Every mbarrier wait is bounded; a wait that runs out records an error word, and the CTA still frees its tensor memory
// before it returns.
#pragma once

#include "sm100_ptx.cuh"
#include "w8a8_internal.h"
#include "w8a8_swiglu.cuh"

namespace w8a8 {
namespace gemm {

constexpr int BR = 128, BK = 128;            // weight rows per CTA; bytes of K per stage
constexpr int kScGroups = 4, kScRing = 4;    // K-groups per chunk of scales, chunks in the ring
constexpr uint32_t kSpin = 1u << 21;

struct GemmParams {
    LinearArgs a;
    int* status;
    int tiles_m, tiles_total;
    int splits, split_kb;  // SPLIT: CTAs that share a tile's K, and the stages each of them takes (the last one what is left)
    int tma_store;  // output rows are multiples of 16 bytes and aligned: the tile leaves by TMA
};

// Registers per thread of the 640-thread form that moves some between its warpgroups: at launch, in warpgroup 0, in the others.
constexpr int kLaunchRegs = 96, kLowRegs = 56, kHighRegs = 104;
static_assert(128 * (kLaunchRegs - kLowRegs) >= 512 * (kHighRegs - kLaunchRegs), "setmaxnreg sums must balance");

template <int BT, bool PAIR>
struct Config {
    static constexpr int kRowsB = PAIR ? BT / 2 : BT;                 // token rows this CTA loads
    static constexpr int kStageBytes = (BR + kRowsB) * BK;
    static constexpr int kPanelBytes = BT * 128;                      // BT tokens x 64 fp16 columns, 128-byte swizzle
    static constexpr int kOutBytes = 2 * kPanelBytes;
    static constexpr int kScSlot = kScGroups * (BT + BR) * 4;         // activation scales [4][BT], weight scales [4][128]
    static constexpr int kScBytes = kScRing * kScSlot;
    static constexpr int kRoom = 226 * 1024 - 1024 - kOutBytes - kScBytes;
    static constexpr int kStages = kRoom / kStageBytes >= 8 ? 8 : 4;  // a multiple of four (see the issuer)
    static constexpr int kSmem = kStages * kStageBytes + kOutBytes + kScBytes + 1024;
    // Epilogue warps: four per part of the tokens (one per 32 weight rows). Four warps per scheduler on the wide tiles: with
    // two, half of the issue slots stay empty (g = 64, 8192 x 19456 x 2560: 1012 us with eight warps, 900 with sixteen).
    static constexpr int kParts = BT >= 128 ? 4 : 2;
    static constexpr int kEpiWarps = 4 * kParts, kThreads = 128 + kEpiWarps * 32;
    // The widest tile needs more registers in sixteen epilogue warps than 640 threads can have each: warpgroup 0 gives some up.
    static constexpr bool kMoveRegs = BT > 192;
    static constexpr int kAcc = BT <= 128 ? 4 : 2;                    // accumulator slices
    static constexpr int kTmemCols = kAcc * BT <= 128 ? 128 : kAcc * BT <= 256 ? 256 : 512;
    static_assert(kStages * kStageBytes <= kRoom, "stages do not fit");
    static_assert(BT % 32 == 0 && BT <= 256, "token width");
};

// ---- tcgen05 wrappers ----
template <bool PAIR>
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t cols) {
    if constexpr (PAIR) {  // one warp of EACH CTA of the pair, with the same warp index
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(smem_dst)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(smem_dst)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <bool PAIR>
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc),
                     "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc),
                     "r"(accumulate) : "memory");
}
// Completion of the MMAs this thread has issued so far, signalled on an mbarrier; for a pair on the mbarrier at the same
// shared-memory offset in BOTH CTAs (an arrive, not a load: nothing is copied).
template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    if constexpr (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                         ptx::smem_u32(bar)), "h"(static_cast<uint16_t>(3)) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ptx::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16 lanes x 8 columns per .x1, in the layout of an mma.sync accumulator: registers 4i .. 4i + 3 of a lane are
// (row lane / 4, columns 8i + 2 (lane % 4) and + 1), then the same columns of row lane / 4 + 8.
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The address, in the cluster's shared-memory window, of `local` in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool elect_one() {  // true in one lane of the (converged) warp
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) {  // whole warp; bounded
    if (ptx::mbar_try_wait(bar, parity)) return true;
    return ptx::mbar_wait_bounded(bar, parity, kSpin);
}
template <int THREADS>
__device__ __forceinline__ void epi_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }
// The same barrier; true in every epilogue thread if it was passed true by any (they leave the tile loop together).
template <int THREADS>
__device__ __forceinline__ bool epi_barrier_any(bool v) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
                 : "=r"(r) : "r"(static_cast<uint32_t>(v)), "n"(THREADS) : "memory");
    return r != 0;
}

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    return static_cast<uint64_t>(__float_as_uint(a)) | (static_cast<uint64_t>(__float_as_uint(b)) << 32);
}
__device__ __forceinline__ float lo2(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float hi2(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
// Two sums of one weight row: acc = fma(float(P) * ws, xs, acc).
__device__ __forceinline__ void promote2(uint64_t& acc, uint32_t p0, uint32_t p1, uint64_t ws, uint64_t xs) {
    asm("{\n\t.reg .f32 lo, hi;\n\t.reg .b64 t;\n\t"
        "cvt.rn.f32.s32 lo, %1;\n\tcvt.rn.f32.s32 hi, %2;\n\tmov.b64 t, {lo, hi};\n\t"
        "mul.rn.f32x2 t, t, %3;\n\tfma.rn.f32x2 %0, t, %4, %0;\n\t}"
        : "+l"(acc) : "r"(p0), "r"(p1), "l"(ws), "l"(xs));
}
__device__ __forceinline__ uint64_t lds64(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float lds32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
// Four 8 x 8 fp16 matrices held as accumulator fragments, stored TRANSPOSED: lane l gives the address of the 16-byte row
// l % 8 of matrix l / 8.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint32_t half2_bits(uint64_t v) {
    const __half2 h = __floats2half2_rn(lo2(v), hi2(v));
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t swiglu2_bits(uint64_t gate, uint64_t up) {
    const __half2 h = swiglu2(__floats2half2_rn(lo2(gate), hi2(gate)), __floats2half2_rn(lo2(up), hi2(up)));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Shared-memory operand descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
    return static_cast<uint64_t>((saddr & 0x3ffffu) >> 4) | (1ull << 16) /* leading offset (unused) */ |
           (static_cast<uint64_t>(1024 >> 4) << 32) /* stride between 8-row groups */ | (1ull << 46) /* version */ |
           (2ull << 61) /* SWIZZLE_128B */;
}

// GM: the group size when it is 64, 128 or 256; 0 = any multiple of 32 (plain loops), and whenever the group sums are asked
// for as well.
//
// SPLIT: few tiles and a long K. The CTAs of a cluster take one tile, each a run of its K-groups; at the end the first CTA reads
// the others' fp32 sums from their shared memory and adds them in ascending-K order. Narrow tiles are a serial chain of some
// 430-650 clocks per K-group, whatever the number of CTAs (tokens x rows x K, g = 64: 150 x 2560 x 9728 34.8 -> 27.0 us, 64 x
// 2560 x 9728 34.8 -> 17.9, 150 x 2560 x 4096 19.3 -> 16.4).
template <int BT, bool PAIR, int GM, bool SPLIT>
__global__ void __launch_bounds__(Config<BT, PAIR>::kThreads, 1)
gemm_i8_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
               const __grid_constant__ CUtensorMap map_y, const GemmParams p) {
    using C = Config<BT, PAIR>;
    constexpr int S = C::kStages, kEpiWarps = C::kEpiWarps, kEpiThreads = kEpiWarps * 32;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[S], empty_bar[S], acc_full[C::kAcc], acc_empty[C::kAcc], sc_full[kScRing], sc_empty[kScRing];
    __shared__ uint32_t tmem_base_s;
    __shared__ int failed_s;

    const LinearArgs& a = p.a;
    // (through a shuffle, so that the compiler knows it is the same in all lanes and keeps what follows from it in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t tiles = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t out_stage = tiles + S * C::kStageBytes, sc_ring = out_stage + C::kOutBytes;
    static_assert(!SPLIT || (!PAIR && GM != 0), "a split tile is one CTA's, of whole K-groups");
    const int srank = SPLIT ? static_cast<int>(cluster_rank()) : 0;
    const int kb0 = SPLIT ? srank * p.split_kb : 0;
    const int num_kb = SPLIT ? min(p.split_kb, a.K / BK - kb0) : a.K / BK;
    const int G = a.G, g_first = SPLIT ? kb0 * BK / GM : 0, g_end = SPLIT ? g_first + num_kb * BK / GM : G;  // this CTA's K-groups
    const uint32_t crank = PAIR ? cluster_rank() : 0u;
    const int walker = SPLIT ? static_cast<int>(blockIdx.x) / p.splits : PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
    const int walkers = SPLIT ? p.tiles_total : PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
    auto tile_m0 = [&](int tile) { return (tile % p.tiles_m) * BT; };
    auto tile_n0 = [&](int tile) { return (tile / p.tiles_m) * (PAIR ? 2 * BR : BR) + static_cast<int>(crank) * BR; };
    int my_tiles = 0;
    if (walker < p.tiles_total) my_tiles = (p.tiles_total - walker + walkers - 1) / walkers;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { ptx::mbar_init(&full_bar[s], 1); ptx::mbar_init(&empty_bar[s], 1); }
        for (int s = 0; s < C::kAcc; ++s) {
            ptx::mbar_init(&acc_full[s], 1);
            ptx::mbar_init(&acc_empty[s], PAIR ? 2 * kEpiWarps : kEpiWarps);
        }
        for (int s = 0; s < kScRing; ++s) { ptx::mbar_init(&sc_full[s], 128); ptx::mbar_init(&sc_empty[s], kEpiWarps); }
        failed_s = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async();
    }
    if (warp == 1) tmem_alloc<PAIR>(&tmem_base_s, C::kTmemCols);
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();  // the peer's barriers are initialised before anything signals them
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    // The activation codes come from the kernel before this one (the row quantiser).
    ptx::pdl_wait();

    if (warp < 4) {
        if constexpr (C::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLowRegs) : "memory");
        if (warp == 0) {
            // ---------------- producer ----------------
            const bool leader = elect_one();
            // a pair's loads complete on the LEADER's barrier, which alone expects the bytes of both CTAs
            const uint32_t full0 = PAIR ? map_to_rank(ptx::smem_u32(&full_bar[0]), 0) : ptx::smem_u32(&full_bar[0]);
            int tile = walker, kx = kb0 * BK, left = my_tiles * num_kb;
            int m0 = tile_m0(tile) + (PAIR ? static_cast<int>(crank) * C::kRowsB : 0), n0 = tile_n0(tile);
            uint32_t parity = 1;
            bool ok = true;
            while (left > 0 && ok) {
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    if (s >= left) break;
                    if (!wait(&empty_bar[s], parity)) {
                        if (leader) atomicExch(p.status, 200 + s);
                        ok = false;
                        break;
                    }
                    if (leader) {
                        const uint32_t dst = tiles + s * C::kStageBytes, bar = full0 + s * 8;
                        if (PAIR) {
                            if (crank == 0) ptx::mbar_arrive_expect_tx(&full_bar[s], 2 * C::kStageBytes);
                            asm volatile(
                                "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                                ::"r"(dst), "l"(&map_w), "r"(bar), "r"(kx), "r"(n0) : "memory");
                            asm volatile(
                                "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                                ::"r"(dst + BR * BK), "l"(&map_x), "r"(bar), "r"(kx), "r"(m0) : "memory");
                        } else {
                            ptx::mbar_arrive_expect_tx(&full_bar[s], C::kStageBytes);
                            asm volatile(
                                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                                ::"r"(dst), "l"(&map_w), "r"(bar), "r"(kx), "r"(n0) : "memory");
                            asm volatile(
                                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                                ::"r"(dst + BR * BK), "l"(&map_x), "r"(bar), "r"(kx), "r"(m0) : "memory");
                        }
                    }
                    kx += BK;
                    if (kx == a.K) {
                        kx = 0;
                        tile += walkers;
                        m0 = tile_m0(tile) + (PAIR ? static_cast<int>(crank) * C::kRowsB : 0);
                        n0 = tile_n0(tile);
                    }
                }
                left -= S;
                parity ^= 1u;
            }
        } else if (warp == 1) {
            // ---------------- MMA issuer (of a pair, the leader alone) ----------------
            if (crank == 0) {
                constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) /* int8 x int8 -> int32, both K-major */ |
                                           (static_cast<uint32_t>(BT >> 3) << 17) | (static_cast<uint32_t>((PAIR ? 2 * BR : BR) >> 4) << 24);
                const bool leader = elect_one();
                const uint64_t desc0 = smem_desc(tiles);
                int left = my_tiles * num_kb;
                uint32_t parity = 0, acc_parity = 1;
                int code = 0;  // what ran out, if anything
                int q_in_group = 0, as_any = 0;
                const int mpg = a.g / 32;
                while (left > 0 && code == 0) {
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        if (s >= left) break;
                        const uint64_t da = desc0 + static_cast<uint64_t>((s * C::kStageBytes) >> 4);
                        const uint64_t db = da + static_cast<uint64_t>((BR * BK) >> 4);
                        // (a step of 32 bytes along K inside the 128-byte swizzled row: +2 in the descriptor's address field)
                        if constexpr (GM != 0) {
                            // the groups of this stage: half a group, one, or two
                            constexpr int kPerStage = GM == 64 ? 2 : 1, kMmas = 4 / kPerStage, kLoopGroups = S * 128 / GM;
                            const bool first = GM != 256 || s % 2 == 0, last = GM != 256 || s % 2 == 1;
                            if (!wait(&full_bar[s], parity)) { code = 300 + s; break; }
#pragma unroll
                            for (int h = 0; h < kPerStage; ++h) {
                                const int lg = GM == 256 ? s / 2 : s * kPerStage + h;                  // group inside this turn of the ring
                                const int as = kLoopGroups >= C::kAcc ? lg % C::kAcc : lg + as_any;     // its accumulator slice
                                if (first) {
                                    if (!wait(&acc_empty[as], acc_parity)) { code = 400 + as; break; }
                                    tc_fence_after();
                                }
                                if (leader) {
#pragma unroll
                                    for (int sub = h * kMmas; sub < (h + 1) * kMmas; ++sub)
                                        mma_i8<PAIR>(tmem_base + as * BT, da + 2 * sub, db + 2 * sub, idesc, (first && sub == h * kMmas) ? 0u : 1u);
                                    if (last) tc_commit<PAIR>(&acc_full[as]);  // the K-group's sums are complete
                                }
                                if (kLoopGroups >= C::kAcc && last && lg % C::kAcc == C::kAcc - 1) acc_parity ^= 1u;
                            }
                            if (code) break;
                            if (leader) tc_commit<PAIR>(&empty_bar[s]);  // the stage may be refilled once these MMAs retire
                            if (kLoopGroups < C::kAcc && s == S - 1 && (as_any = kLoopGroups - as_any) == 0) acc_parity ^= 1u;
                        } else {
                            if (!wait(&full_bar[s], parity)) { code = 300 + s; break; }
                            // (Rolled up, the four MMAs of a stage took the issuing warp longer than they take: one scale per channel,
                            // 4096 x 19456 x 2560 309 -> 204 us, groups of 512 342 -> 234.)
#pragma unroll
                            for (int sub = 0; sub < 4; ++sub) {
                                if (q_in_group == 0) {
                                    if (!wait(&acc_empty[as_any], acc_parity)) { code = 400 + as_any; break; }
                                    tc_fence_after();
                                }
                                if (leader) mma_i8<PAIR>(tmem_base + as_any * BT, da + 2 * sub, db + 2 * sub, idesc, q_in_group != 0 ? 1u : 0u);
                                if (++q_in_group == mpg) {
                                    if (leader) tc_commit<PAIR>(&acc_full[as_any]);
                                    q_in_group = 0;
                                    if (++as_any == C::kAcc) { as_any = 0; acc_parity ^= 1u; }
                                }
                            }
                            if (code) break;
                            if (leader) tc_commit<PAIR>(&empty_bar[s]);
                        }
                    }
                    left -= S;
                    parity ^= 1u;
                }
                if (code && leader) atomicExch(p.status, code);
            }
        } else {
            // ---------------- scales, four groups per chunk: activation scales [4][BT], weight scales [4][128], fp32 ----------------
            const int t64 = threadIdx.x - 64;
            int slot = 0;
            uint32_t parity = 1;
            bool ok = true;
            for (int tile = walker; tile < p.tiles_total && ok; tile += walkers) {
                const int m0 = tile_m0(tile), n0 = tile_n0(tile);
                if (a.epilogue == W8A8_EPI_RESIDUAL && srank == 0) {  // the tile's residual rows to L2, long before its end needs them
                    for (int i = t64; i < 2 * BT; i += 64) {
                        const int t = m0 + (i >> 1), col = n0 + (i & 1) * 64;
                        if (t < a.M && col < a.N)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.residual + static_cast<size_t>(t) * a.N + col));
                    }
                }
                const __half* ws0 = a.w_scale + static_cast<size_t>(min(n0 + t64, a.N - 1)) * G;
                const __half* ws1 = a.w_scale + static_cast<size_t>(min(n0 + 64 + t64, a.N - 1)) * G;
                for (int j0 = g_first; j0 < g_end; j0 += kScGroups) {
                    const int nj = min(kScGroups, g_end - j0);
                    __half w[2][kScGroups];  // on their way while the slot is waited for
#pragma unroll
                    for (int q = 0; q < kScGroups; ++q) {
                        w[0][q] = ws0[min(j0 + q, G - 1)];
                        w[1][q] = ws1[min(j0 + q, G - 1)];
                    }
                    if (!wait(&sc_empty[slot], parity)) {
                        atomicExch(p.status, 600 + slot);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = sc_ring + slot * C::kScSlot;
                    for (int t = t64; t < BT; t += 64) {
                        const float* src = a.Xs + static_cast<size_t>(min(m0 + t, a.M - 1)) * G + j0;
#pragma unroll
                        for (int q = 0; q < kScGroups; ++q)
                            if (q < nj) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + (q * BT + t) * 4), "l"(src + q) : "memory");
                    }
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(ptx::smem_u32(&sc_full[slot])) : "memory");
#pragma unroll
                    for (int q = 0; q < kScGroups; ++q) {
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + (kScGroups * BT + q * BR + t64) * 4), "f"(__half2float(w[0][q])) : "memory");
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + (kScGroups * BT + q * BR + 64 + t64) * 4), "f"(__half2float(w[1][q])) : "memory");
                    }
                    ptx::mbar_arrive(&sc_full[slot]);
                    if (++slot == kScRing) { slot = 0; parity ^= 1u; }
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncwarp();
        if constexpr (SPLIT) cluster_sync_all();  // (the epilogue's meeting below)
    } else {
        if constexpr (C::kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kHighRegs) : "memory");
        // ---------------- epilogue: each warp 32 weight rows x a part of the tokens ----------------
        // A lane holds four weight rows (16 h + 8 e + lane / 4) and, of every eight tokens, two neighbouring ones.
        constexpr int HC = BT / C::kParts;              // tokens per warp
        constexpr int CH = 16;                          // tokens per step
        constexpr int NCH = HC / CH, OCT = HC / 8;
        const int quad = warp & 3;                      // the tensor-memory lane quadrant this warp may read
        const int part = (warp - 4) >> 2;               // which part of the tokens
        const int et = (warp - 4) * 32 + lane;
        int as = 0, slot = 0;
        uint32_t acc_parity = 0, sc_parity = 0;
        bool ok = true;
        const uint32_t acc_empty0 = PAIR ? map_to_rank(ptx::smem_u32(&acc_empty[0]), 0) : ptx::smem_u32(&acc_empty[0]);
        const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + part * HC;
        for (int tile = walker; tile < p.tiles_total; tile += walkers) {
            const int m0 = tile_m0(tile), n0 = tile_n0(tile);
            uint64_t acc[2][2][OCT];                    // [h][e][eight tokens]: two neighbouring tokens, packed
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int o = 0; o < OCT; ++o) acc[h][e][o] = 0ull;
            // (A second buffer of sums, filled while the first is promoted, and a look-ahead into the next group were measured: no
            // gain with four warps per scheduler, and a loss where the tensor pipe is the slower side.)
            uint32_t r[2][CH / 2];
            auto load_sums = [&](uint32_t taddr) {
                tmem_ld(taddr, r[0]);
                tmem_ld(taddr + (16u << 16), r[1]);
            };
#pragma unroll 1
            for (int j0 = g_first; j0 < g_end && ok; j0 += kScGroups) {
                if (!wait(&sc_full[slot], sc_parity)) {
                    if (lane == 0) atomicExch(p.status, 700 + slot);
                    ok = false;
                    break;
                }
                uint32_t xs_addr = sc_ring + slot * C::kScSlot + (part * HC + 2 * (lane & 3)) * 4;
                uint32_t ws_addr = sc_ring + slot * C::kScSlot + (kScGroups * BT + quad * 32 + (lane >> 2)) * 4;
                const int j1 = min(j0 + kScGroups, g_end);
#pragma unroll 1
                for (int j = j0; j < j1; ++j) {
                    uint64_t w2[2][2];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float w = lds32(ws_addr + (16 * h + 8 * e) * 4);
                            w2[h][e] = pack2(w, w);
                        }
                    const uint32_t taddr = taddr0 + as * BT;
                    if (!wait(&acc_full[as], acc_parity)) {
                        if (lane == 0) atomicExch(p.status, 500 + as);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    load_sums(taddr);
#pragma unroll
                    for (int ci = 0; ci < NCH; ++ci) {
                        uint64_t x2[CH / 8];
#pragma unroll
                        for (int o = 0; o < CH / 8; ++o) x2[o] = lds64(xs_addr + (ci * CH + 8 * o) * 4);
                        tmem_ld_wait();
                        if (ci + 1 == NCH) {
                            // The group's last sums are in registers: the slice may be overwritten while they are promoted.
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) {
                                if (PAIR && crank != 0) mbar_arrive_cluster(acc_empty0 + as * 8);
                                else ptx::mbar_arrive(&acc_empty[as]);
                            }
                            if (++as == C::kAcc) { as = 0; acc_parity ^= 1u; }
                        }
#pragma unroll
                        for (int o = 0; o < CH / 8; ++o)
#pragma unroll
                            for (int h = 0; h < 2; ++h)
#pragma unroll
                                for (int e = 0; e < 2; ++e)
                                    promote2(acc[h][e][ci * (CH / 8) + o], r[h][4 * o + 2 * e], r[h][4 * o + 2 * e + 1], w2[h][e], x2[o]);
                        if constexpr (GM == 0) {
                            if (a.dump) {
#pragma unroll
                                for (int o = 0; o < CH / 8; ++o)
#pragma unroll
                                    for (int i = 0; i < 8; ++i) {
                                        const int n = n0 + quad * 32 + 16 * (i >> 2) + 8 * ((i >> 1) & 1) + (lane >> 2);
                                        const int m = m0 + part * HC + ci * CH + 8 * o + 2 * (lane & 3) + (i & 1);
                                        if (m < a.M && n < a.N)
                                            a.dump[(static_cast<size_t>(m) * a.N + n) * G + j] = static_cast<int>(r[i >> 2][4 * o + (i & 3)]);
                                    }
                            }
                        }
                        if (ci + 1 < NCH) load_sums(taddr + (ci + 1) * CH);
                    }
                    xs_addr += BT * 4;
                    ws_addr += BR * 4;
                }
                // the chunk's scales are used up
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sc_empty[slot]);
                if (++slot == kScRing) { slot = 0; sc_parity ^= 1u; }
            }
            if constexpr (SPLIT) {
                // Every stage of this CTA's ring has been loaded and multiplied: its memory holds the sums now. One tile per CTA.
                static_assert(4 * OCT * kEpiThreads * 8 <= S * C::kStageBytes, "the sums fit the ring");
                const uint32_t mine = tiles + et * 8;
                if (srank > 0) {
#pragma unroll
                    for (int i = 0; i < 4 * OCT; ++i)
                        asm volatile("st.shared.b64 [%0], %1;" ::"r"(mine + i * kEpiThreads * 8), "l"(acc[i / (2 * OCT)][i / OCT % 2][i % OCT]) : "memory");
                }
                __syncwarp();
                cluster_sync_all();
                if (srank > 0) {
                    if (epi_barrier_any<kEpiThreads>(!ok)) failed_s = 1;
                    break;
                }
                for (int c = 1; c < p.splits; ++c) {
                    const uint32_t theirs = map_to_rank(mine, c);
                    uint64_t v[4 * OCT];
#pragma unroll
                    for (int i = 0; i < 4 * OCT; ++i)
                        asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(v[i]) : "r"(theirs + i * kEpiThreads * 8) : "memory");
#pragma unroll
                    for (int i = 0; i < 4 * OCT; ++i) {
                        uint64_t& mine_i = acc[i / (2 * OCT)][i / OCT % 2][i % OCT];
                        mine_i = pack2(lo2(mine_i) + lo2(v[i]), hi2(mine_i) + hi2(v[i]));
                    }
                }
            }
            // ---- the tile as fp16 in shared memory: panels of [BT tokens][64 columns], 128-byte rows, swizzled ----
            if (et == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the tile before has left it
            if (epi_barrier_any<kEpiThreads>(!ok)) {
                failed_s = 1;
                break;
            }
            const bool swiglu = a.epilogue == W8A8_EPI_SWIGLU;
            if (swiglu) {
                // Rows come in blocks of 8 gate rows (e = 0) and the 8 up rows of the same channels (e = 1).
                const int t = part * HC + ((lane >> 1) & 8) + (lane & 7), chunk = quad * 2 + ((lane >> 3) & 1);
                const uint32_t dst = out_stage + t * 128 + ((chunk ^ (lane & 7)) << 4);
#pragma unroll
                for (int o = 0; o < OCT; o += 2)
                    stmatrix_x4_trans(dst + o * 8 * 128, swiglu2_bits(acc[0][0][o], acc[0][1][o]), swiglu2_bits(acc[1][0][o], acc[1][1][o]),
                                      swiglu2_bits(acc[0][0][o + 1], acc[0][1][o + 1]), swiglu2_bits(acc[1][0][o + 1], acc[1][1][o + 1]));
            } else {
                const int t = part * HC + (lane & 7), chunk = (quad & 1) * 4 + (lane >> 3);
                const uint32_t dst = out_stage + (quad >> 1) * C::kPanelBytes + t * 128 + ((chunk ^ (lane & 7)) << 4);
#pragma unroll
                for (int o = 0; o < OCT; ++o)
                    stmatrix_x4_trans(dst + o * 8 * 128, half2_bits(acc[0][0][o]), half2_bits(acc[0][1][o]), half2_bits(acc[1][0][o]),
                                      half2_bits(acc[1][1][o]));
            }
            const int ycols = swiglu ? a.N / 2 : a.N, y0 = swiglu ? n0 / 2 : n0;   // first output column of this CTA
            const int width = min(swiglu ? BR / 2 : BR, ycols - y0);                // columns it owns (<= 0: none)
            if (p.tma_store && a.epilogue != W8A8_EPI_RESIDUAL) {
                ptx::fence_proxy_async();
                epi_barrier<kEpiThreads>();
                if (et == 0) {
                    for (int pnl = 0; pnl * 64 < width; ++pnl)  // (a box that starts inside the tensor is clipped at its edges)
                        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                                     ::"l"(&map_y), "r"(out_stage + pnl * C::kPanelBytes), "r"((y0 + pnl * 64) * 2), "r"(m0) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else {
                epi_barrier<kEpiThreads>();
                const int tokens = min(BT, a.M - m0);
                if (p.tma_store) {  // residual: 16-byte pieces, sixteen threads per token row
                    const int piece = et & 15, rt = et >> 4;
                    if (piece * 8 < width) {
                        // Up to four rows at a time: their reads are memory latencies, one after the other eight to a tile of 256
                        // tokens. (All of them at once, or four in the forms for any group size, spill registers in the loop above.)
                        constexpr int kRowStep = kEpiThreads / 16;
                        constexpr int kRows = GM == 0 ? 2 : BT % (4 * kRowStep) == 0 ? 4 : BT % (3 * kRowStep) == 0 ? 3 : 2;
                        static_assert(BT % (kRows * kRowStep) == 0, "whole rounds");
                        const size_t o0 = static_cast<size_t>(m0) * ycols + y0 + piece * 8;
#pragma unroll 1
                        for (int t0 = rt; t0 < tokens; t0 += kRows * kRowStep) {
                            uint4 rv[kRows];
#pragma unroll
                            for (int i = 0; i < kRows; ++i) {
                                const int t = t0 + i * kRowStep < tokens ? t0 + i * kRowStep : t0;
                                rv[i] = *reinterpret_cast<const uint4*>(a.residual + o0 + static_cast<size_t>(t) * ycols);
                            }
#pragma unroll
                            for (int i = 0; i < kRows; ++i) {
                                const int t = t0 + i * kRowStep;
                                if (t >= tokens) break;
                                uint4 v;
                                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                                             : "r"(out_stage + (piece >> 3) * C::kPanelBytes + t * 128 + (((piece & 7) ^ (t & 7)) << 4)));
                                __half2* hv = reinterpret_cast<__half2*>(&v);
                                const __half2* hr = reinterpret_cast<const __half2*>(&rv[i]);
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const float2 x = __half22float2(hv[k]), y = __half22float2(hr[k]);
                                    hv[k] = __floats2half2_rn(x.x + y.x, x.y + y.y);
                                }
                                *reinterpret_cast<uint4*>(a.Y + o0 + static_cast<size_t>(t) * ycols) = v;
                            }
                        }
                    }
                } else {  // any row pitch: element by element
                    const int col = et & 127;
                    if (col < width) {
                        for (int t = et >> 7; t < tokens; t += C::kParts) {
                            const size_t o = static_cast<size_t>(m0 + t) * ycols + y0 + col;
                            uint16_t b;
                            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(b)
                                         : "r"(out_stage + (col >> 6) * C::kPanelBytes + t * 128 + ((((col & 63) >> 3) ^ (t & 7)) << 4) + (col & 7) * 2));
                            __half y = __ushort_as_half(b);
                            if (a.epilogue == W8A8_EPI_RESIDUAL) y = __float2half(__half2float(y) + __half2float(a.residual[o]));
                            a.Y[o] = y;
                        }
                    }
                }
            }
        }
        // the last tile's store must have read shared memory before the CTA gives it up
        if (et == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    // ---- teardown: everyone meets, then the allocating warp frees the tensor memory ----
    tc_fence_before();
    __syncthreads();
    if (failed_s)  // a bounded wait ran out: give copies and MMAs that may still be in flight time to land
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    if constexpr (PAIR || SPLIT) cluster_sync_all();  // (SPLIT: the others' sums have been read); nothing of the peer still signals this CTA's barriers or uses its tensor memory
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<PAIR>(tmem_base, C::kTmemCols);
    }
}

using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const GemmParams);
struct FormState {
    SmemAttribute attribute;
    std::atomic<int> registers{0};  // per thread, as compiled (0: not asked for yet)
};
// A tile form: its kernel and what the launch needs to know about it. stage_ns, group_ns: what a tile takes per 128 bytes of
// K and per K-group, fitted to one shape, 8192 x 19456 x 2560 at g = 256 and g = 64 (the two overlap; their sum is what was
// measured). There is no term for a chain's start or a tile's end (conversion, residual, store): at 2048 and 8192 tokens the
// predicted times of w2 lie 10-25 % below measured ones, so forms that differ by a few per cent are not told apart.
struct Form {
    int bt;
    bool pair, split;
    Kernel kernel;
    int threads, smem;
    bool move_regs;
    float stage_ns, group_ns;
    FormState* state;
};
template <int BT, bool PAIR, int GM, bool SPLIT>
inline FormState form_state;
template <int BT, bool PAIR, int GM, bool SPLIT = false>
Form form(float stage_ns, float group_ns) {
    return Form{BT, PAIR, SPLIT, gemm_i8_kernel<BT, PAIR, GM, SPLIT>, Config<BT, PAIR>::kThreads, Config<BT, PAIR>::kSmem, Config<BT, PAIR>::kMoveRegs, stage_ns, group_ns,
                &form_state<BT, PAIR, GM, SPLIT>};
}
template <int GM>
const Form* all_forms(int* count) {
    static const Form table[] = {form<32, false, GM>(148, 157), form<64, false, GM>(136, 196), form<96, false, GM>(106, 300),
                                 form<128, false, GM>(135, 330), form<192, true, GM>(215, 440), form<256, true, GM>(247, 557),
                                 form<32, false, GM, true>(148, 157), form<64, false, GM, true>(136, 196), form<96, false, GM, true>(106, 300),
                                 form<128, false, GM, true>(135, 330)};
    *count = static_cast<int>(sizeof(table) / sizeof(table[0]));
    return table;
}
const Form* forms_g64(int* count);
const Form* forms_g128(int* count);
const Form* forms_g256(int* count);
const Form* forms_any(int* count);

}  // namespace gemm
}  // namespace w8a8
