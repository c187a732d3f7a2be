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
//                of tensor memory (two to sixteen), starting with "overwrite" or, at g = 64, with a bias (below)
//   warps 2, 3   stage the scales of eight (four) K-groups at a time in a ring of their own
//   warps 4 ...  epilogue, eight to sixteen warps, each 32 weight rows x a part of the tokens. For every K-group
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
// The promote is the other side, and the bound in most forms. Stamps of the clock in an epilogue warp, taken before the units, the chunks of eight
// groups and the wide reads of scales (they cost some 10 % themselves, and have not been taken again), showed 1216, 1424 and 1451 clocks per
// K-group of a 128 x 256 tile at groups of 64, 128 and 256, of which 224-358 were waits for the MMAs, against 384 (with the bias), 512 and 1024
// of MMAs. The counters of the present forms at 2048 x 19456 x 2560: tensor pipe 59 % busy at g = 256 (256 wide), 35 % at g = 64 (128 wide), a
// third of that the bias; issue slots 53 and 50 %. In trial programs of sixteen such warps alone, clocks per warp and scheduler for two sums (the programs are not kept):
//   * two conversions, a packed multiply and a packed FMA 4.3 by themselves, 6.9-7.2 with the tensor-memory and shared-memory reads around
//     them, as if conversions and those reads shared a way into the registers; two packed FMAs without conversions 5.1-5.6 with the
//     reads. Hence the BIAS at g = 64 (promote2): each group's accumulator starts from a constant, made by one more MMA of a
//     constant operand with itself, that makes every sum positive; as bits it then is an fp32 number, and the multiply that had to
//     follow the conversion takes the bias out again, exactly. At g = 128 it would take two more MMAs per four, and at g = 256 the tensor pipe
//     is the next bound.
//   * the integer conversions (add into the mantissa of 1.5 * 2^23) 15-25 % slower than the conversion instruction.
//   * the sums are read in the layout of an mma.sync accumulator (16x256b): a lane then holds 4 weight rows x 2 tokens of every 16 x 8
//     block and reads the activation scales of sixteen sums, four tokens, with 16 bytes. (32x32b, a thread per row, is three times as
//     fast out of tensor memory but needs a 16-byte read per four sums: 1.3-2 times as long in all, most while the MMAs read shared
//     memory.)
// Some 270 clocks of a hand-over do not depend on the tile's width: two waits, the arrive, the loop, each of them the end of what the
// compiler can mix. Hence UNITS: up to 128 tokens, issuer and epilogue hand one another as many K-groups as two slots of tensor
// memory hold, up to two, four or eight, and the loop over a chunk of scales is unrolled where that measured faster. us back to back, one
// (g = 128, 256) or two (g = 64) groups per unit in a rolled loop, and now: g = 64 150 x 19456 x 2560, 32 wide 37.8 -> 30.1, 613 x 19456 x
// 2560, 64 wide 101.8 -> 88.6, 2048 x 6144 x 2560, 96 wide 82.9 -> 73.1; g = 128 32 wide 28.2 -> 21.7, 64 wide 68.1 -> 56.7, 96 wide 60.0 -> 52.8; g = 256
// 32 wide 20.9 -> 20.2 (96 and 128 wide lose a sixth by units of two: there the MMAs of a unit take longer than its promote hides).
// A tile's K, or its run of a split, is padded to whole units, so that slots and columns stay immediates of the issuer: loads past
// K bring zeros, those past a run the next run's operands, and the scales of the groups that only fill a unit are zero, which adds
// 0 to sums that are never -0. (700 x 2560 x 2816, g = 256, 64 wide: 11 groups as 12, 11.0 us and 11.7. A short K pays most: 150 x 2560 x 1280,
// g = 128, ten groups as twelve, 5.1 us with single groups and 5.5; 267 x 3680 x 384, g = 64, six as eight, 4.9 and 5.9.)
//
// Back to back, us, without the bias, the units, the 16-byte scale reads and the cheaper SwiGLU, and as it is (M x N x K; the long ones under the power cap):
//   8192 x 19456 x 2560 with SwiGLU, g = 64 967 -> 799 (844 -> 1021 TOPS); g = 128 617 -> 531; g = 256 447 -> 369 (1827 -> 2211 TOPS)
//   g = 64 2048 x 2560 x 9728 154 -> 90;  613 x 2560 x 9728 52.8 -> 32.8;  150 x 19456 x 2560 with SwiGLU 52.6 -> 29.4
//   4001 x 6144 x 2560, g = 128 95.2 -> 77.8; g = 256 66.9 -> 55.6
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
constexpr uint32_t kSpin = 1u << 21;

struct GemmParams {
    LinearArgs a;
    int* status;
    int inner, tiles_total;  // tiles along the side that is walked first; in all
    int splits, split_kb;  // SPLIT: CTAs that share a tile's K, and the stages each of them takes (the last one what is left)
    int tma_store;  // output rows are multiples of 16 bytes and aligned: the tile leaves by TMA
};

// g = 64: the sums come out of the MMAs with kBias added, by a first MMA of a constant operand with itself.
constexpr int kBiasByte = 184, kBias = kBiasByte * kBiasByte * 32, kConstBytes = BR * 32;
static_assert(kBias > 128 * 128 * 64 && kBias + 128 * 128 * 64 < (1 << 23) && kBias % (1 << 11) == 0 && (kBias >> 11) < (1 << 13),
              "sums above zero and below 2^23; 11 bits of a weight scale times the bias are exact in fp32");

template <int BT, bool PAIR, int GM, bool SPLIT>
struct Config {
    static constexpr bool kBiased = GM == 64 && BT >= 64;  // (32 wide the MMA lengthens the chain: 2560 x 4096 13.3 and 14.8 us)
    static constexpr int kRowsB = PAIR ? BT / 2 : BT;                 // token rows this CTA loads
    static constexpr int kStageBytes = (BR + kRowsB) * BK;
    static constexpr int kPanelBytes = BT * 128;                      // BT tokens x 64 fp16 columns, 128-byte swizzle
    static constexpr int kOutBytes = 2 * kPanelBytes;
    // K-groups per chunk of scales, chunks in the ring. An epilogue warp spends some 240 clocks where one chunk ends and the next begins: its
    // arrive, a wait, new addresses, and between them nothing to mix the promote with. With twelve groups in three chunks of four, us
    // back to back: 4096 x 19456 x 2560 g = 64, 256 wide 395 and now 387, 192 wide 429 and 421, g = 128, 256 wide 281 and 275; 2048 x 6144 x
    // 2560 g = 64, 96 wide 86.8 and 82.9; 150 x 19456 x 2560 g = 64, 32 wide 40.2 and 37.8. (Sixteen in two chunks of eight have room in every form; chunks
    // of sixteen in the narrower ones lose stages of operands for them: 613 x 2560 x 9728 g = 256, 64 wide 29.2 and 42.7.)
    // Narrow tiles at g = 256 take four at a time after all: they start when a chunk's scales are there, and a chunk of eight is most of a short K
    // (us, eight and four: 64 wide, 33 x 9728 x 2560 8.19 and 8.05, 150 x 6144 x 2560 7.35 and 7.14; 32 wide, 100 x 19456 x 2560 18.1 and 17.9). Wider tiles at g = 256 lose
    // by it, 192 and 256 wide up to 2 %.
    static constexpr int kScGroups = GM == 256 && BT <= 64 ? 4 : 8, kScRing = 16 / kScGroups;
    static constexpr int kScSlot = kScGroups * (BT + BR) * 4;         // activation scales [kScGroups][BT], weight scales [kScGroups][128]
    static constexpr int kScBytes = kScRing * kScSlot;
    static constexpr int kConst = kBiased ? kConstBytes : 0;
    static constexpr int kRoom = 226 * 1024 - 1024 - kOutBytes - kScBytes - kConst;
    static constexpr int kStages = kRoom / kStageBytes >= 8 ? 8 : 4;  // a multiple of four (see the issuer)
    static constexpr int kSmem = kStages * kStageBytes + kOutBytes + kScBytes + kConst + 1024;
    // Epilogue warps: four per part of the tokens (one per 32 weight rows). More warps hide more of one another's waits, fewer have the
    // registers to mix more of the promote with the reads; measured form by form. g = 64, 96 wide, 2048 x 6144 x 2560: three parts 70.5 us,
    // two 79.4; 192 wide, 4096 x 19456 x 2560: four 390, three 404, two 393. g = 128, 128 wide, 2048 x 6144 x 2560: two, in steps of 32 tokens, 44.3, four 46.4;
    // 192 wide, 4001 x 2560 x 9728: four 124.6, three 130, two 136. g = 256, 256 wide, 4096 x 19456 x 2560: two 160, four 165; 128 wide, 2048 x
    // 6144 x 2560: two, in steps of 32, 35.4, four 36.7.
    static constexpr int kParts = GM == 64 ? (BT == 192 ? 4 : BT == 96 ? 3 : 2) : GM == 128 ? (BT >= 192 ? 4 : 2) : GM == 256 ? (BT == 192 ? 4 : 2) : 4;
    // With two parts at 128 and 256 tokens a thread stores twice as much as with four: all reads of a residual tile at once, and rows that leave element
    // by element eight or sixteen tokens at a time. us, one read after another and now: g = 256, 256 wide 5299 x 1836 x 9728 with a residual
    // 247 and 124, 7730 x 9728 x 1280 with a residual 155 and 137, 7071 x 7721 x 9984 615 and 562; g = 128, 128 wide 943 x 19456 x 896 with a
    // residual 47.8 and 41.9. (The narrower tiles as they are: unrolled, they lose more by code placement than that store is.)
    static constexpr bool kFewStore = kParts == 2 && BT >= 128 && GM >= 128;
    static constexpr int kStep = (GM == 64 && BT == 256) || (GM >= 128 && BT == 128) ? 32 : 16;  // tokens per step of the promote
    static constexpr int kEpiWarps = 4 * kParts, kThreads = 128 + kEpiWarps * 32;
    // The widest tile needs more registers in its epilogue warps than all threads can have: warpgroup 0 gives some up.
    static constexpr bool kMoveRegs = BT > 192;
    // Registers per thread of the form that moves some: at launch, in warpgroup 0, in the others.
    static constexpr int kLaunchRegs = kParts == 2 ? 168 : 96, kLowRegs = kParts == 2 ? 40 : 56, kHighRegs = kParts == 2 ? 232 : 104;
    static_assert(128 * (kLaunchRegs - kLowRegs) >= kEpiWarps * 32 * (kHighRegs - kLaunchRegs), "setmaxnreg sums must balance");
    // K-groups per unit (see above), the stages that a unit takes, units per turn of the epilogue's loop. A split at g = 256 takes one: two pad a run of
    // nineteen groups (33 x 2560 x 9728, 32 wide, two CTAs 11.08 us, with one 10.91).
    static constexpr int kUnit = GM == 64 ? (BT == 32 ? 8 : BT == 64 ? 4 : BT <= 128 ? 2 : 1) : GM == 128 ? (BT <= 64 ? 4 : BT <= 128 ? 2 : 1) : GM == 256 && BT <= 64 && !SPLIT ? 2 : 1;
    static constexpr int kUnitKb = kUnit * GM > BK ? kUnit * GM / BK : 1;
    static constexpr int kUnroll = GM == 64 ? (BT >= 192 || BT == 32 ? 1 : BT == 64 ? 2 : 4) : GM == 128 ? (BT >= 192 || BT == 64 ? 1 : BT == 96 ? 4 : 2) : 1;
    // No more of them than a turn of the ring fills, so that the issuer knows each at compile time.
    static constexpr int kTurn = GM == 0 ? 4 : kStages * BK / GM / kUnit;  // units per turn of the ring
    static constexpr int kSlotsRoom = 4 * kUnit * BT <= 512 ? 4 : 2, kSlots = kSlotsRoom < kTurn ? kSlotsRoom : kTurn;
    static constexpr int kAcc = kUnit * kSlots;                       // accumulator slices
    // Where the arrive by a branch is the faster one: 256 wide, g = 64, 4096 x 19456 x 2560 384 us and 392 with arrive_lane0; 128 wide,
    // g = 256, 2048 x 6144 x 2560 38.1 and 38.8.
    static constexpr bool kBranchArrive = (GM == 64 && BT == 256) || (GM == 256 && BT == 128);
    // The weight scales a chunk ahead (see the scales' warps): 256 wide, g = 64, 4096 x 19456 x 2560 380 us and 390 without; any group
    // size, 4096 x 19456 x 2560 with one group 267 and 273. Elsewhere it costs what it holds registers for: g = 64, 64 wide, 150 x 6144 x
    // 2560 12.2 and 11.4.
    // A chunk's scales in reads of 16 or 8 bytes, and activation scales through registers. As reads of two bytes and copies of four, a lane a row, a chunk
    // takes 1300 to 3000 cycles of the load unit, as long as the tile takes to compute it, and where rows of scales are a power of two
    // apart (K = 4096) the lines that eight such reads share have left L1 between them. us before and after, g = 64: 150 x 2560 x 4096, 64 wide 18.3 and 13.6;
    // 150 x 19456 x 2560, 96 wide 30.5 and 28.9; 613 x 2560 x 9728, 96 wide 37.7 and 33.4; 4001 x 2560 x 9728, 192 wide 205 and 194; g = 128 2048 x
    // 2560 x 4096, 128 wide 40.8 and 37.5. The widest form: registers are short there (weight scales only, g = 128; at g = 64 a chunk ahead is better,
    // 4096 x 19456 x 2560 403 us and 410). A split at g = 128 starts its runs off those boundaries; at g = 256, with few scales, 2560 x 9728 in narrow tiles lost 1 to 4 %.
    static constexpr bool kWideScales = GM == 64 ? BT <= 192 : GM == 128 && !SPLIT, kWideX = kWideScales && BT <= 192;
    static constexpr bool kScalesAhead = GM == 0 || (GM == 64 && BT == 256);
    static constexpr int kBatch = GM == 64 && BT <= 64 ? 2 : 1;  // steps whose sums are requested together
    static constexpr int kTmemCols = kAcc * BT <= 128 ? 128 : kAcc * BT <= 256 ? 256 : 512;
    static_assert(kSlots >= 2 && kTurn % kSlots == 0, "one unit's sums are formed while another's are promoted");
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
// Lane 0 arrives, by a predicate: a branch would end the block of instructions in which the compiler mixes the promote with the reads.
// (For the hand-over of sums: reading them and waiting for them is the warp's as one, so no lane is behind.) us with a branch and without,
// 4096 x 19456 x 2560: 192 wide, g = 64 418 and 390, g = 128 307 and 286, g = 256 213 and 207; 256 wide, g = 128 244 and 238.
template <bool CLUSTER>
__device__ __forceinline__ void arrive_lane0(uint32_t addr, int lane) {
    if constexpr (CLUSTER) asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cluster.b64 _, [%0];\n\t}" ::"r"(addr), "r"(lane) : "memory");
    else asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(addr), "r"(lane) : "memory");
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
// The same where the sums carry kBias: as bits, P + kBias is the fp32 number (P + kBias) * 2^-149, so one FMA converts, takes the
// bias out and multiplies, with one rounding, that of float(P) * ws: ws comes times 2^111, bias is -kBias * 2^-149 times that, and
// acc is 2^-38 times the sum.
__device__ __forceinline__ void promote2(uint64_t& acc, uint32_t p0, uint32_t p1, uint64_t ws, uint64_t bias, uint64_t xs) {
    asm("{\n\t.reg .b64 t;\n\tmov.b64 t, {%1, %2};\n\tfma.rn.f32x2 t, t, %3, %4;\n\tfma.rn.f32x2 %0, t, %5, %0;\n\t}"
        : "+l"(acc) : "r"(p0), "r"(p1), "l"(ws), "l"(bias), "l"(xs));
}
__device__ __forceinline__ void mul2(uint64_t& v, uint64_t f) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(f)); }
// Where the scales of token t and of weight row n lie in their [groups][BT] and [groups][128] of shared memory: what a lane reads for
// sixteen tokens (two neighbouring ones of either eight), or for its four weight rows, is one 16-byte piece. Such a read, its
// address shared by the lanes of a row or column, takes shared memory as long as one of 8 bytes (two clocks, twice that while the
// MMAs read their operands), of which there would be two, or four of 4 bytes.
__device__ __forceinline__ int xs_slot(int t) { return (t & ~15) | ((t & 6) << 1) | ((t >> 2) & 2) | (t & 1); }
__device__ __forceinline__ int ws_slot(int n) { return (n & ~31) | ((n & 7) << 2) | ((n >> 3) & 3); }
__device__ __forceinline__ void lds_2x64(uint32_t addr, uint64_t& a, uint64_t& b) {
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ void lds_4x32(uint32_t addr, float (&v)[4]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(addr));
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

// With the bias (promote2), an infinite weight scale gives infinity less infinity. The output columns of such weight rows, in the
// tile that lies in shared memory, are formed anew, from the operands: signed infinities and NaN as float(P) * ws has them. Slow, and
// only run for a tile that has met an infinite scale (one such row: 4001 x 6144 x 2560 997 us with a search of every row by every
// thread in every tile that followed, 171 now, 116 without such a row). First which rows those are, a thread per row, into rows[4]:
__device__ __forceinline__ void find_infinite_rows(const LinearArgs& a, uint32_t* rows, int n0, int et) {
    bool any = false;
    if (et < BR && n0 + et < a.N)
        for (int j = 0; j < a.G; ++j) any |= isinf(__half2float(a.w_scale[static_cast<size_t>(n0 + et) * a.G + j]));
    const uint32_t word = __ballot_sync(0xffffffffu, any);
    if (et < BR && (et & 31) == 0) rows[et >> 5] = word;
}
template <class C>
__device__ __forceinline__ void infinite_rows(const LinearArgs& a, const uint32_t* rows, uint32_t out_stage, int m0, int n0, int tokens, bool swiglu, int et) {
    auto sum = [&](int n, int m) {
        const int4* w = reinterpret_cast<const int4*>(a.W + static_cast<size_t>(n) * a.K);
        const int4* x = reinterpret_cast<const int4*>(a.Xq + static_cast<size_t>(m) * a.K);
        float acc = 0.0f;
#pragma unroll 1
        for (int j = 0; j < a.G; ++j) {
            int p = 0;
#pragma unroll 1
            for (int k = j * (a.g / 16); k < (j + 1) * (a.g / 16); ++k) {
                const int4 wv = w[k], xv = x[k];
                p = __dp4a(wv.x, xv.x, __dp4a(wv.y, xv.y, __dp4a(wv.z, xv.z, __dp4a(wv.w, xv.w, p))));
            }
            acc = fmaf(static_cast<float>(p) * __half2float(a.w_scale[static_cast<size_t>(n) * a.G + j]), a.Xs[static_cast<size_t>(m) * a.G + j], acc);
        }
        return acc;
    };
#pragma unroll 1
    for (int row = 0; row < BR; ++row) {
        if (swiglu && (row & 8)) continue;  // (taken with its gate row)
        if (!(rows[row >> 5] >> (row & 31) & (swiglu ? 0x101u : 1u))) continue;
        const int n = n0 + row;
        const int col = swiglu ? (row >> 4) * 8 + (row & 7) : row;
#pragma unroll 1
        for (int t = et; t < tokens; t += C::kEpiWarps * 32) {
            __half y = __float2half(sum(n, m0 + t));
            if (swiglu) y = __low2half(swiglu2(__half2half2(y), __half2half2(__float2half(sum(n + 8, m0 + t)))));
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(out_stage + (col >> 6) * C::kPanelBytes + t * 128 +
                                                         ((((col & 63) >> 3) ^ (t & 7)) << 4) + (col & 7) * 2), "h"(__half_as_ushort(y)) : "memory");
        }
    }
}

// GM: the group size when it is 64, 128 or 256; 0 = any multiple of 32 (plain loops), and whenever the group sums are asked
// for as well.
//
// SPLIT: few tiles and a long K. The CTAs of a cluster take one tile, each a run of its K-groups; at the end the first CTA reads
// the others' fp32 sums from their shared memory and adds them in ascending-K order. Narrow tiles are a serial chain of K-groups,
// whatever the number of CTAs (tokens x rows x K, the best form without a split and with one: g = 64, 33 x 2560 x 9728 25.0 and 16.4 us,
// 150 x 2560 x 9728 25.2 and 23.5, 33 x 2560 x 4096 14.3 and 11.2; g = 256, 64 x 2560 x 9728 14.5 and 11.2).
//
// ROWS_FIRST: which side of the tiles is walked first (see walk_rows_first). An instance of its own: chosen in the kernel, by a parameter, it
// cost the pairs of 192 tokens at g = 64 up to 3 % wherever it was not taken (code placement: 4001 x 6144 x 2560 121.7 and 126.6 us).
template <int BT, bool PAIR, int GM, bool SPLIT, bool ROWS_FIRST>
__global__ void __launch_bounds__(Config<BT, PAIR, GM, SPLIT>::kThreads, 1)
gemm_i8_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
               const __grid_constant__ CUtensorMap map_y, const GemmParams p) {
    using C = Config<BT, PAIR, GM, SPLIT>;
    constexpr int S = C::kStages, kEpiWarps = C::kEpiWarps, kEpiThreads = kEpiWarps * 32, kScGroups = C::kScGroups;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[S], empty_bar[S], acc_full[C::kSlots], acc_empty[C::kSlots], sc_full[C::kScRing], sc_empty[C::kScRing];
    __shared__ uint32_t tmem_base_s;
    __shared__ int failed_s;
    // kBiased: infinite_s[i % kMarks] is i + 1 if a weight scale of this CTA's i-th tile is infinite (the scales' warps are up to kScRing
    // chunks, so as many tiles, ahead of the epilogue); the same, as all epilogue threads are to see it at a tile's end
    constexpr int kMarks = C::kScRing + 1;
    __shared__ int infinite_s[kMarks], infinite_tile_s;
    __shared__ uint32_t infinite_rows_s[BR / 32];

    const LinearArgs& a = p.a;
    // (through a shuffle, so that the compiler knows it is the same in all lanes and keeps what follows from it in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t tiles = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t out_stage = tiles + S * C::kStageBytes, sc_ring = out_stage + C::kOutBytes, const_tile = sc_ring + C::kScBytes;
    static_assert(!SPLIT || (!PAIR && GM != 0), "a split tile is one CTA's, of whole K-groups");
    const int srank = SPLIT ? static_cast<int>(cluster_rank()) : 0;
    const int kb0 = SPLIT ? srank * p.split_kb : 0;
    const int real_kb = SPLIT ? min(p.split_kb, a.K / BK - kb0) : a.K / BK, num_kb = (real_kb + C::kUnitKb - 1) / C::kUnitKb * C::kUnitKb;
    // this CTA's K-groups, and where they end with those that only fill the last unit
    const int G = a.G, g_first = SPLIT ? kb0 * BK / GM : 0, g_end = SPLIT ? g_first + real_kb * BK / GM : G;
    const int g_pad = GM == 0 ? G : g_first + num_kb * BK / (GM == 0 ? 1 : GM);
    const uint32_t crank = PAIR ? cluster_rank() : 0u;
    const int walker = SPLIT ? static_cast<int>(blockIdx.x) / p.splits : PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
    const int walkers = SPLIT ? p.tiles_total : PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
    auto tile_m0 = [&](int tile) { return (ROWS_FIRST ? tile / p.inner : tile % p.inner) * BT; };
    auto tile_n0 = [&](int tile) { return (ROWS_FIRST ? tile % p.inner : tile / p.inner) * (PAIR ? 2 * BR : BR) + static_cast<int>(crank) * BR; };
    int my_tiles = 0;
    if (walker < p.tiles_total) my_tiles = (p.tiles_total - walker + walkers - 1) / walkers;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { ptx::mbar_init(&full_bar[s], 1); ptx::mbar_init(&empty_bar[s], 1); }
        for (int s = 0; s < C::kSlots; ++s) {
            ptx::mbar_init(&acc_full[s], 1);
            ptx::mbar_init(&acc_empty[s], PAIR ? 2 * kEpiWarps : kEpiWarps);
        }
        for (int s = 0; s < C::kScRing; ++s) { ptx::mbar_init(&sc_full[s], 128); ptx::mbar_init(&sc_empty[s], kEpiWarps); }
        failed_s = 0;
        for (int i = 0; i < kMarks; ++i) infinite_s[i] = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async();
    }
    if constexpr (C::kBiased) {  // (the operand of the first MMA of every K-group: the same byte everywhere, so its layout is any)
        for (int i = threadIdx.x; i < kConstBytes / 4; i += C::kThreads)
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(const_tile + i * 4), "r"(kBiasByte * 0x01010101u) : "memory");
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
        if constexpr (C::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kLowRegs) : "memory");
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
                    if (kx == (kb0 + num_kb) * BK) {
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
                // uint8 x uint8; rows of 32 bytes in groups of eight, 32-byte swizzle
                constexpr uint32_t bias_idesc = idesc & ~((7u << 7) | (7u << 10));
                const uint64_t bias_desc = static_cast<uint64_t>((const_tile & 0x3ffffu) >> 4) | (1ull << 16) |
                                           (static_cast<uint64_t>(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
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
                            constexpr int kPerStage = GM == 64 ? 2 : 1, kMmas = 4 / kPerStage;
                            const bool first = GM != 256 || s % 2 == 0, last = GM != 256 || s % 2 == 1;
                            if (!wait(&full_bar[s], parity)) { code = 300 + s; break; }
#pragma unroll
                            for (int h = 0; h < kPerStage; ++h) {
                                // A turn of the ring is whole rounds of the slots. The lanes of this warp may be apart here, some past a
                                // wait that others are still in: what the leader issues must not be a register that moves with the loop.
                                static_assert(S * 128 / GM % C::kUnit == 0 && C::kTurn % C::kSlots == 0, "rounds of the slots");
                                const int lg = GM == 256 ? s / 2 : s * kPerStage + h, lu = lg / C::kUnit;  // group and unit inside this turn
                                const int as = lu % C::kSlots;
                                const bool opens = first && lg % C::kUnit == 0, closes = last && lg % C::kUnit == C::kUnit - 1;
                                if (opens) {
                                    if (!wait(&acc_empty[as], acc_parity)) { code = 400 + as; break; }
                                    tc_fence_after();
                                }
                                if (leader) {
                                    const uint32_t to = tmem_base + (as * C::kUnit + lg % C::kUnit) * BT;
                                    if (C::kBiased && first) mma_i8<PAIR>(to, bias_desc, bias_desc, bias_idesc, 0u);
#pragma unroll
                                    for (int sub = h * kMmas; sub < (h + 1) * kMmas; ++sub)
                                        mma_i8<PAIR>(to, da + 2 * sub, db + 2 * sub, idesc, (!C::kBiased && first && sub == h * kMmas) ? 0u : 1u);
                                    if (closes) tc_commit<PAIR>(&acc_full[as]);  // the unit's sums are complete
                                }
                                if (closes && as == C::kSlots - 1) acc_parity ^= 1u;
                            }
                            if (code) break;
                            if (leader) tc_commit<PAIR>(&empty_bar[s]);  // the stage may be refilled once these MMAs retire
                        } else {
                            // Slot and place in the group run in registers here, so the lanes of the warp stay together: they agree on every
                            // wait, and none moves on before the leader has issued.
                            if (!__all_sync(0xffffffffu, wait(&full_bar[s], parity))) { code = 300 + s; break; }
                            // (Rolled up, the four MMAs of a stage took the issuing warp longer than they take: one scale per channel,
                            // 4096 x 19456 x 2560 309 -> 204 us, groups of 512 342 -> 234.)
#pragma unroll
                            for (int sub = 0; sub < 4; ++sub) {
                                if (q_in_group == 0) {
                                    if (!__all_sync(0xffffffffu, wait(&acc_empty[as_any], acc_parity))) { code = 400 + as_any; break; }
                                    tc_fence_after();
                                }
                                if (leader) mma_i8<PAIR>(tmem_base + as_any * BT, da + 2 * sub, db + 2 * sub, idesc, q_in_group != 0 ? 1u : 0u);
                                __syncwarp();
                                if (++q_in_group == mpg) {
                                    if (leader) tc_commit<PAIR>(&acc_full[as_any]);
                                    __syncwarp();
                                    q_in_group = 0;
                                    if (++as_any == C::kSlots) { as_any = 0; acc_parity ^= 1u; }
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
            // ---------------- scales, a chunk at a time: activation scales [kScGroups][BT], weight scales [kScGroups][128], fp32 ----------------
            const int t64 = threadIdx.x - 64;
            constexpr float kScale = C::kBiased ? 0x1p111f : 1.0f;  // (see promote2)
            int slot = 0;
            uint32_t parity = 1;
            bool ok = true;
            // kScalesAhead: the weight scales are read a chunk ahead, as a read takes as long as a narrow tile takes for a chunk.
            __half w[2][kScGroups];
            auto w_row = [&](int n) { return a.w_scale + static_cast<size_t>(min(n + t64, a.N - 1)) * G; };
            auto load_w = [&](const __half* ws0, const __half* ws1, int j0) {
#pragma unroll
                for (int q = 0; q < kScGroups; ++q) {
                    w[0][q] = ws0[min(j0 + q, G - 1)];
                    w[1][q] = ws1[min(j0 + q, G - 1)];
                }
            };
            auto load_w_ahead = [&](int tile, int j0) {
                if (j0 >= g_pad) { tile += walkers; j0 = g_first; }
                if (tile >= p.tiles_total) return;
                const int n0 = tile_n0(tile);
                load_w(w_row(n0), w_row(n0 + 64), j0);
            };
            // kWideScales: by 16 or 8 bytes where the address, the row's length and the run's start are multiples of that.
            uint32_t wv[2][kScGroups / 2];
            constexpr int XQ = BT == 32 ? kScGroups / 2 : kScGroups, XT = (BT + 63) / 64;  // activation scales per thread and token (32 tokens: half of them), tokens per thread
            float xv[XT][XQ];
            const int xt = BT == 32 ? t64 % 32 : t64, xq0 = BT == 32 ? t64 / 32 * XQ : 0;
            const unsigned w_at = static_cast<unsigned>(reinterpret_cast<unsigned long long>(a.w_scale)) | (2u * G) | (2u * g_first);
            const unsigned x_at = static_cast<unsigned>(reinterpret_cast<unsigned long long>(a.Xs)) | (4u * G) | (4u * g_first);
            const bool w16 = (w_at & 15) == 0, w8 = (w_at & 7) == 0, x16 = C::kWideX && (x_at & 15) == 0;
            auto load_wide = [&](const __half* ws0, const __half* ws1, int m0, int j0) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const __half* row = h ? ws1 : ws0;
                    if (w16) {
                        const uint4 v = *reinterpret_cast<const uint4*>(row + j0);
                        wv[h][0] = v.x; wv[h][1] = v.y; wv[h][2] = v.z; wv[h][3] = v.w;
                    } else if (w8) {
                        const uint2 v = *reinterpret_cast<const uint2*>(row + j0), u = *reinterpret_cast<const uint2*>(row + min(j0 + 4, G - 4));
                        wv[h][0] = v.x; wv[h][1] = v.y; wv[h][2] = u.x; wv[h][3] = u.y;
                    } else {
                        const unsigned short* r = reinterpret_cast<const unsigned short*>(row);
#pragma unroll
                        for (int i = 0; i < kScGroups / 2; ++i)
                            wv[h][i] = r[min(j0 + 2 * i, G - 1)] | static_cast<uint32_t>(r[min(j0 + 2 * i + 1, G - 1)]) << 16;
                    }
                }
                if (x16) {
#pragma unroll
                    for (int k = 0; k < XT; ++k) {
                        const float* xs = a.Xs + static_cast<size_t>(min(m0 + xt + 64 * k, a.M - 1)) * G;
#pragma unroll
                        for (int i = 0; i < XQ; i += 4) {
                            const float4 v = *reinterpret_cast<const float4*>(xs + min(j0 + xq0 + i, G - 4));
                            xv[k][i] = v.x; xv[k][i + 1] = v.y; xv[k][i + 2] = v.z; xv[k][i + 3] = v.w;
                        }
                    }
                }
            };
            if constexpr (C::kScalesAhead) load_w_ahead(walker, g_first);
            int ith = 0;
            for (int tile = walker; tile < p.tiles_total && ok; tile += walkers, ++ith) {
                const int m0 = tile_m0(tile), n0 = tile_n0(tile);
                if (a.epilogue == W8A8_EPI_RESIDUAL && srank == 0) {  // the tile's residual rows to L2, long before its end needs them
                    for (int i = t64; i < 2 * BT; i += 64) {
                        const int t = m0 + (i >> 1), col = n0 + (i & 1) * 64;
                        if (t < a.M && col < a.N)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.residual + static_cast<size_t>(t) * a.N + col));
                    }
                }
                // (Once a tile: formed anew for every chunk they cost the tiles of 192 tokens 1 %, a call of one wave up to 2 %.)
                const __half* ws0 = w_row(n0);
                const __half* ws1 = w_row(n0 + 64);
                for (int j0 = g_first; j0 < g_pad; j0 += kScGroups) {
                    const int nj = min(kScGroups, g_end - j0);
                    if constexpr (C::kWideScales) load_wide(ws0, ws1, m0, j0);
                    else if constexpr (!C::kScalesAhead) load_w(ws0, ws1, j0);  // on their way while the slot is waited for
                    if (!wait(&sc_empty[slot], parity)) {
                        atomicExch(p.status, 600 + slot);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = sc_ring + slot * C::kScSlot;
                    if (x16) {
#pragma unroll
                        for (int k = 0; k < XT; ++k) {
                            if (BT % 64 != 0 && BT > 64 && xt + 64 * k >= BT) break;
#pragma unroll
                            for (int q = 0; q < XQ; ++q)
                                asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + ((xq0 + q) * BT + xs_slot(xt + 64 * k)) * 4), "f"(xq0 + q < nj ? xv[k][q] : 0.0f) : "memory");
                        }
                    }
                    for (int t = x16 ? BT : t64; t < BT; t += 64) {
                        const float* src = a.Xs + static_cast<size_t>(min(m0 + t, a.M - 1)) * G + j0;
#pragma unroll
                        for (int q = 0; q < kScGroups; ++q) {
                            const uint32_t to = dst + (q * BT + xs_slot(t)) * 4;
                            if (q < nj) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(src + q) : "memory");
                            else if (C::kUnit > 1 && j0 + q < g_pad) asm volatile("st.shared.f32 [%0], %1;" ::"r"(to), "f"(0.0f) : "memory");
                        }
                    }
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(ptx::smem_u32(&sc_full[slot])) : "memory");
#pragma unroll
                    for (int q = 0; q < kScGroups; ++q) {
                        const bool real = C::kUnit == 1 || q < nj;
                        if constexpr (C::kWideScales) {
                            w[0][q] = __ushort_as_half(static_cast<unsigned short>(wv[0][q >> 1] >> (16 * (q & 1))));
                            w[1][q] = __ushort_as_half(static_cast<unsigned short>(wv[1][q >> 1] >> (16 * (q & 1))));
                        }
                        const float w0 = real ? __half2float(w[0][q]) : 0.0f, w1 = real ? __half2float(w[1][q]) : 0.0f;
                        if (C::kBiased && (isinf(w0) || isinf(w1))) infinite_s[ith % kMarks] = ith + 1;
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + (kScGroups * BT + q * BR + ws_slot(t64)) * 4), "f"(w0 * kScale) : "memory");
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + (kScGroups * BT + q * BR + 64 + ws_slot(t64)) * 4), "f"(w1 * kScale) : "memory");
                    }
                    ptx::mbar_arrive(&sc_full[slot]);
                    if constexpr (C::kScalesAhead) load_w_ahead(tile, j0 + kScGroups);
                    if (++slot == C::kScRing) { slot = 0; parity ^= 1u; }
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncwarp();
        if constexpr (SPLIT) cluster_sync_all();  // (the epilogue's meeting below)
    } else {
        if constexpr (C::kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kHighRegs) : "memory");
        // ---------------- epilogue: each warp 32 weight rows x a part of the tokens ----------------
        // A lane holds four weight rows (16 h + 8 e + lane / 4) and, of every eight tokens, two neighbouring ones.
        constexpr int HC = BT / C::kParts;              // tokens per warp
        constexpr int CH = C::kStep;                    // tokens per step
        constexpr int NCH = HC / CH, OCT = HC / 8;
        const int quad = warp & 3;                      // the tensor-memory lane quadrant this warp may read
        const int part = (warp - 4) >> 2;               // which part of the tokens
        const int et = (warp - 4) * 32 + lane;
        constexpr int U = C::kUnit;
        constexpr int STEPS = U * NCH, BATCH = C::kBatch;
        static_assert(STEPS % BATCH == 0 && kScGroups % U == 0, "whole batches, whole units in a chunk of scales");
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
            // (A second buffer of sums, filled while the first is promoted, within a group or from one to the next: no gain.)
            uint32_t r[BATCH][2][CH / 2];
#pragma unroll 1
            for (int j0 = g_first; j0 < g_pad && ok; j0 += kScGroups) {
                if (!wait(&sc_full[slot], sc_parity)) {
                    if (lane == 0) atomicExch(p.status, 700 + slot);
                    ok = false;
                    break;
                }
                uint32_t xs_addr = sc_ring + slot * C::kScSlot + (part * HC + 4 * (lane & 3)) * 4;
                uint32_t ws_addr = sc_ring + slot * C::kScSlot + (kScGroups * BT + quad * 32 + 4 * (lane >> 2)) * 4;
                const int j1 = min(j0 + kScGroups, g_pad);
#pragma unroll C::kUnroll
                for (int j = j0; j < j1; j += U) {
                    const uint32_t taddr = taddr0 + as * (U * BT);
                    float w4[BATCH][4];
                    uint64_t w2[2][2], b2[2][2];
                    auto take_scales = [&](const float (&w)[4]) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            w2[i / 2][i % 2] = pack2(w[i], w[i]);
                            if constexpr (C::kBiased) {
                                const float bias = w[i] * -__int_as_float(kBias);
                                b2[i / 2][i % 2] = pack2(bias, bias);
                            }
                        }
                    };
                    // One group per unit: made ready before the wait; behind it they cost every group (g = 128, M x N x K 2048 x 2560 x
                    // 9728, 128 wide 92.8 -> 88.6 us, 4001 x 2560 x 9728, 192 wide 152.5 -> 149.6). Not so in the forms for any group size
                    // (2048 x 6144 x 2560, g = 32 208 -> 204 us behind it).
                    constexpr bool kBefore = U == 1 && GM != 0;
                    if constexpr (U == 1) lds_4x32(ws_addr, w4[0]);
                    if constexpr (kBefore) take_scales(w4[0]);
                    if (!wait(&acc_full[as], acc_parity)) {
                        if (lane == 0) atomicExch(p.status, 500 + as);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    auto load_sums = [&](int q0) {  // the sums of the steps from q0
#pragma unroll
                        for (int b = 0; b < BATCH; ++b)
#pragma unroll
                            for (int c = 0; c < CH; c += 16) {
                                const uint32_t from = taddr + (q0 + b) / NCH * BT + (q0 + b) % NCH * CH + c;
                                tmem_ld(from, *reinterpret_cast<uint32_t(*)[8]>(&r[b][0][c / 2]));
                                tmem_ld(from + (16u << 16), *reinterpret_cast<uint32_t(*)[8]>(&r[b][1][c / 2]));
                            }
                    };
                    load_sums(0);
#pragma unroll
                    for (int q0 = 0; q0 < STEPS; q0 += BATCH) {
                        uint64_t x2[BATCH][CH / 8];
#pragma unroll
                        for (int b = 0; b < BATCH; ++b)
#pragma unroll
                            for (int o = 0; o < CH / 8; o += 2)
                                lds_2x64(xs_addr + ((q0 + b) / NCH * BT + (q0 + b) % NCH * CH + 8 * o) * 4, x2[b][o], x2[b][o + 1]);
                        if constexpr (U > 1) {
#pragma unroll
                            for (int b = 0; b < BATCH; ++b)
                                if ((q0 + b) % NCH == 0) lds_4x32(ws_addr + (q0 + b) / NCH * BR * 4, w4[b]);
                        }
                        tmem_ld_wait();
                        if (q0 + BATCH == STEPS) {
                            // The unit's last sums are in registers: its slices may be overwritten while they are promoted.
                            tc_fence_before();
                            if constexpr (C::kBranchArrive) {
                                __syncwarp();
                                if (lane == 0) {
                                    if (PAIR && crank != 0) mbar_arrive_cluster(acc_empty0 + as * 8);
                                    else ptx::mbar_arrive(&acc_empty[as]);
                                }
                            } else {
                                arrive_lane0<PAIR>(acc_empty0 + as * 8, lane);
                            }
                        }
#pragma unroll
                        for (int b = 0; b < BATCH; ++b) {
                            const int ci = (q0 + b) % NCH;
                            if (!kBefore && ci == 0) take_scales(w4[b]);
#pragma unroll
                            for (int o = 0; o < CH / 8; ++o)
#pragma unroll
                                for (int h = 0; h < 2; ++h)
#pragma unroll
                                    for (int e = 0; e < 2; ++e) {
                                        uint64_t& to = acc[h][e][ci * (CH / 8) + o];
                                        const uint32_t p0 = r[b][h][4 * o + 2 * e], p1 = r[b][h][4 * o + 2 * e + 1];
                                        if constexpr (C::kBiased) promote2(to, p0, p1, w2[h][e], b2[h][e], x2[b][o]);
                                        else promote2(to, p0, p1, w2[h][e], x2[b][o]);
                                    }
                            if constexpr (GM == 0) {
                                if (a.dump) {
#pragma unroll
                                    for (int o = 0; o < CH / 8; ++o)
#pragma unroll
                                        for (int i = 0; i < 8; ++i) {
                                            const int n = n0 + quad * 32 + 16 * (i >> 2) + 8 * ((i >> 1) & 1) + (lane >> 2);
                                            const int m = m0 + part * HC + ci * CH + 8 * o + 2 * (lane & 3) + (i & 1);
                                            if (m < a.M && n < a.N)
                                                a.dump[(static_cast<size_t>(m) * a.N + n) * G + j] = static_cast<int>(r[b][i >> 2][4 * o + (i & 3)]);
                                        }
                                }
                            }
                        }
                        if (q0 + BATCH < STEPS) load_sums(q0 + BATCH);
                    }
                    if (++as == C::kSlots) { as = 0; acc_parity ^= 1u; }
                    xs_addr += U * BT * 4;
                    ws_addr += U * BR * 4;
                }
                // the chunk's scales are used up
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sc_empty[slot]);
                if (++slot == C::kScRing) { slot = 0; sc_parity ^= 1u; }
            }
            int infinite = 0;
            if constexpr (C::kBiased) {
                const int ith = (tile - walker) / walkers;
                infinite = infinite_s[ith % kMarks] == ith + 1;
                const uint64_t up = pack2(0x1p38f, 0x1p38f);
#pragma unroll
                for (int i = 0; i < 4 * OCT; ++i) mul2(acc[i / (2 * OCT)][i / OCT % 2][i % OCT], up);
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
                    if constexpr (C::kBiased) {
                        int v;
                        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(map_to_rank(ptx::smem_u32(&infinite_s[0]), c)) : "memory");
                        infinite |= v;  // (a CTA's only tile: 0 or 1)
                    }
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
            if (et == 0) {
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the tile before has left it
                if constexpr (C::kBiased) infinite_tile_s = infinite;
            }
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
            if constexpr (C::kBiased) {
                if (infinite_tile_s) {
                    find_infinite_rows(a, infinite_rows_s, n0, et);
                    epi_barrier<kEpiThreads>();
                    infinite_rows<C>(a, infinite_rows_s, out_stage, m0, n0, min(BT, a.M - m0), swiglu, et);
                }
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
                        // Several rows at a time: their reads are memory latencies. (All of them at once with four parts, or four in the forms
                        // for any group size, spill registers in the loop above.)
                        constexpr int kRowStep = kEpiThreads / 16;
                        constexpr int kRows = GM == 0 ? 2 : C::kFewStore ? BT / kRowStep : BT % (4 * kRowStep) == 0 ? 4 : BT % (3 * kRowStep) == 0 ? 3 : 2;
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
                    auto staged = [&](int t) {
                        uint16_t b;
                        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(b)
                                     : "r"(out_stage + (col >> 6) * C::kPanelBytes + t * 128 + ((((col & 63) >> 3) ^ (t & 7)) << 4) + (col & 7) * 2));
                        return __ushort_as_half(b);
                    };
                    if constexpr (C::kFewStore) {
                        constexpr int kTok = BT / 16;  // (256 wide, 7071 x 7721 x 9984 592 us with eight, 562 with sixteen; 128 wide eight)
                        static_assert(BT % (kTok * C::kParts) == 0, "whole rounds");
                        if (col < width) {
#pragma unroll 1
                            for (int t0 = et >> 7; t0 < tokens; t0 += kTok * C::kParts) {
                                const size_t o0 = static_cast<size_t>(m0) * ycols + y0 + col;
                                __half y[kTok], r[kTok];
#pragma unroll
                                for (int i = 0; i < kTok; ++i) {
                                    const int t = t0 + i * C::kParts < tokens ? t0 + i * C::kParts : t0;
                                    y[i] = staged(t);
                                    r[i] = a.epilogue == W8A8_EPI_RESIDUAL ? a.residual[o0 + static_cast<size_t>(t) * ycols] : __float2half(0.0f);
                                }
#pragma unroll
                                for (int i = 0; i < kTok; ++i) {
                                    const int t = t0 + i * C::kParts;
                                    if (t >= tokens) break;
                                    if (a.epilogue == W8A8_EPI_RESIDUAL) y[i] = __float2half(__half2float(y[i]) + __half2float(r[i]));
                                    a.Y[o0 + static_cast<size_t>(t) * ycols] = y[i];
                                }
                            }
                        }
                    } else if (col < width) {
                        for (int t = et >> 7; t < tokens; t += C::kParts) {
                            const size_t o = static_cast<size_t>(m0 + t) * ycols + y0 + col;
                            __half y = staged(t);
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
// What a form's tiles take, ns: per 128 bytes of K, per K-group, per tile (conversion, TMA store), once per launch (the launch itself, the first
// operands, the end of a chain that nothing overlaps); and per tile on top, for rows that leave element by element, for a residual, for
// both. Least squares over 15,000 times of one of the forms under the model in choose(): the four projections and 9728 x 2560 at 30 token counts from
// 33 to 8192, 890 drawn shapes (33 to 8192 tokens, 128 to 24,000 rows, K from 128 to 12,800, every epilogue, odd rows) and 420 of up to 420
// tokens; the model's count three times. No cost is moved after the fit. Judged by its choice against the best form, groups of 64, 128 and 256, the
// rule loses on average 0.4, 0.6 and 1.0 % over 299 other drawn shapes, 0.6, 0.8 and 1.0 % over the drawn ones it was fitted to, 0.0, 0.2 and 0.2 %
// over the model's. (Costs per stage and tile alone, moved towards the choices that lose least over the model's shapes: 1.6, 2.1 and 2.3; 1.4, 2.2 and
// 2.7; 0.4 each.)
struct Cost {
    float stage, group, tile, start, odd, residual, odd_residual;
};
// A tile form: its kernel and what the launch needs to know about it.
struct Form {
    int bt;
    bool pair, split;
    Kernel kernel[2];  // tokens walked first, rows walked first (or none)
    int threads, smem;
    int launch_regs;  // per thread, if the form moves some between its warpgroups; else 0
    Cost cost;
    int unit_kb;  // Config::kUnitKb
    FormState* state;  // [2]
};
template <int BT, bool PAIR, int GM, bool SPLIT>
inline FormState form_state[2];
template <int BT, bool PAIR, int GM, bool SPLIT = false>
Form form(const Cost& cost) {
    using C = Config<BT, PAIR, GM, SPLIT>;
    Kernel rows_first = nullptr;
    if constexpr (BT >= 128 && !SPLIT && GM != 0) rows_first = gemm_i8_kernel<BT, PAIR, GM, SPLIT, true>;  // (a long prompt's forms)
    return Form{BT, PAIR, SPLIT, {gemm_i8_kernel<BT, PAIR, GM, SPLIT, false>, rows_first}, C::kThreads, C::kSmem, C::kMoveRegs ? C::kLaunchRegs : 0,
                cost, C::kUnitKb, form_state<BT, PAIR, GM, SPLIT>};
}
template <int GM>
const Form* all_forms(int* count) {
    // groups of 64, 128 and 256; token widths 32, 64, 96, 128, 192, 256
    static constexpr Cost kCost[3][6] = {
        {{188, 0, 489, 2990, 1330, 296, 1890}, {286, 0, 788, 3080, 2430, 611, 4200}, {363, 0, 1100, 2940, 2340, 770, 3830},
         {488, 0, 1190, 2970, 4210, 1200, 6100}, {729, 0, 1740, 4120, 3410, 1610, 8360}, {1080, 0, 1260, 4970, 7930, 4070, 14500}},
        {{136, 0, 298, 3050, 1260, 315, 2110}, {186, 0, 622, 3100, 2470, 519, 4350}, {260, 0, 861, 2730, 3120, 576, 6180},
         {303, 0, 1060, 2540, 3000, 702, 1470}, {466, 0, 1510, 3630, 3680, 1270, 5070}, {616, 0, 1610, 3760, 4740, 2060, 6100}},
        {{122, 0, 227, 2880, 1110, 221, 2150}, {142, 0, 573, 3020, 2280, 401, 4400}, {232, 0, 731, 2160, 2610, 448, 6620},
         {249, 0, 776, 2370, 2430, 518, 1960}, {297, 0, 1580, 3410, 3390, 1010, 6260}, {362, 0, 1950, 3010, 5940, 1660, 3410}}};
    const Cost* c = kCost[GM == 64 ? 0 : GM == 128 ? 1 : 2];
    static const Form table[] = {form<32, false, GM>(c[0]),       form<64, false, GM>(c[1]),       form<96, false, GM>(c[2]),
                                 form<128, false, GM>(c[3]),      form<192, true, GM>(c[4]),       form<256, true, GM>(c[5]),
                                 form<32, false, GM, true>(c[0]), form<64, false, GM, true>(c[1]), form<96, false, GM, true>(c[2]),
                                 form<128, false, GM, true>(c[3])};
    *count = static_cast<int>(sizeof(table) / sizeof(table[0]));
    return table;
}
const Form* forms_g64(int* count);
const Form* forms_g128(int* count);
const Form* forms_g256(int* count);
const Form* forms_any(int* count);

}  // namespace gemm
}  // namespace w8a8
