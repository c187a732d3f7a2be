// Host side of the packed decode linear (kernel and its reasons: w8a8_gemv_packed.cuh): the work split, the loader-side pack
// and the launches.
#include "w8a8_gemv_packed.cuh"

namespace w8a8 {
// How many CTAs share the row tiles of a linear. Up to two per SM (their shared memory fits twice when M <= 8),
// as many as make the tiles per CTA equal: 160 row tiles on 148 SMs are 160 CTAs of one tile, not 136 of one
// and 12 of two. An SM that hosts two CTAs has twice the copies in flight and pulls twice the bytes in the same
// time, so what matters is that no CTA is the last one left streaming. Measured over the decode step: 1.92 ->
// 1.72 ms. The one-launch decode step deals its tiles by the same rule.
int gemv_packed_ctas(int tiles, int sms, bool two_per_sm) {
    if (tiles <= sms) return tiles;
    if (!two_per_sm) return sms;
    const int per_cta = (tiles + 2 * sms - 1) / (2 * sms);
    return (tiles + per_cta - 1) / per_cta;
}

namespace {
using namespace gemv;

bool packable(int N, int K, int g) {
    return N > 0 && K > 0 && K % 256 == 0 && K % g == 0 && (g == 64 || g == 128 || g % 256 == 0);
}

size_t fused_smem_bytes(int K, int G) {  // norm weight + padded code rows + scales
    return static_cast<size_t>(K) * 2 + static_cast<size_t>(8) * (K + 64) + static_cast<size_t>(8) * G * 4;
}

}  // namespace

bool gemv::make_plan(const LinearArgs& a, Plan& pl, bool rows, int sms) {
    const bool fused = a.norm_weight != nullptr, quant = !fused && a.X && !a.Xq;
    if (a.M < 1 || a.M > 32) return false;
    if (rows) {  // TMA wants W 16-byte aligned; the scales of a unit are read as one word; whole-row prologues are the packed form's
        if (!a.W || (reinterpret_cast<uintptr_t>(a.W) & 15u) || fused) return false;
        if (reinterpret_cast<uintptr_t>(a.w_scale) & (a.g == 64 ? 7u : a.g == 128 ? 3u : 1u)) return false;
        if (a.tp.world > 0 || a.tail_kind != kTailNone) return false;
    } else if (!a.packed) {
        return false;
    }
    if (!packable(a.N, a.K, a.g)) return false;
    if (fused) {
        // one warp per row; the norm emulates the reference's 1024-thread block, which it launches for dim > 512
        if (a.M > 8 || !a.X || a.K <= 512 || a.K > 4096 || a.dump) return false;
        if (a.smooth_inv || a.act_scale) return false;
        if ((reinterpret_cast<uintptr_t>(a.X) | reinterpret_cast<uintptr_t>(a.norm_weight) |
             reinterpret_cast<uintptr_t>(a.norm_residual) | reinterpret_cast<uintptr_t>(a.norm_x_out) |
             reinterpret_cast<uintptr_t>(a.codes_out)) & 15u)
            return false;
        if (a.norm_residual && a.norm_x_out == a.X) return false;  // other CTAs still read X
    } else if (quant) {
        if (a.M > 8 || !(a.g == 64 || a.g == 128 || a.g == 256) || a.dump || a.smooth_inv || a.act_scale) return false;
        if (a.tail_kind != kTailNone || a.tp.world > 0 || (reinterpret_cast<uintptr_t>(a.X) & 15u)) return false;
        // CTAs that are done store rows of Y while others still quantise X: an output over the input (in place, N == K) needs
        // the two launches, where all of X is codes before the first store.
        const uintptr_t x0 = reinterpret_cast<uintptr_t>(a.X), y0 = reinterpret_cast<uintptr_t>(a.Y);
        const size_t x_bytes = static_cast<size_t>(a.M) * a.K * 2;
        const size_t y_bytes = static_cast<size_t>(a.M) * (a.epilogue == W8A8_EPI_SWIGLU ? a.N / 2 : a.N) * 2;
        if (x0 < y0 + y_bytes && y0 < x0 + x_bytes) return false;
    } else {
        if (!a.Xq || !a.Xs) return false;
        if (reinterpret_cast<uintptr_t>(a.Xq) & 15u) return false;
    }
    if (a.epilogue == W8A8_EPI_SWIGLU && a.N % 16 != 0) return false;
    if (a.tp.world > 0 && (a.epilogue != W8A8_EPI_NONE || a.M > a.tp.max_tokens || a.tail_kind != kTailNone)) return false;
    if (!a.Y && a.tp.world == 0) return false;
    if (a.tail_kind != kTailNone) {
        if (fused || a.M > 8 || !a.tail_counters) return false;
        const int tg = a.tail_g;
        if (a.tail_kind == kTailRowNorm) {
            // a CTA per row, two 16-byte pieces per thread; the norm emulates the reference's 1024-thread block
            if (a.epilogue != W8A8_EPI_NONE || a.N % 256 != 0 || a.N <= 512 || a.N > 4096) return false;
            if (!a.tail_x || !a.tail_norm_weight) return false;
            if (a.tail_Xq && (!a.tail_Xs || !(tg == 64 || tg == 128 || tg == 256))) return false;
            if ((reinterpret_cast<uintptr_t>(a.tail_x) | reinterpret_cast<uintptr_t>(a.tail_norm_weight) |
                 reinterpret_cast<uintptr_t>(a.Y) | reinterpret_cast<uintptr_t>(a.tail_normed_out) |
                 reinterpret_cast<uintptr_t>(a.tail_Xq)) & 15u)
                return false;
        } else {
            const int kout = a.epilogue == W8A8_EPI_SWIGLU ? a.N / 2 : a.N;
            const int cpt = a.epilogue == W8A8_EPI_SWIGLU ? 8 : 16;
            if (a.epilogue == W8A8_EPI_RESIDUAL || !a.tail_Xq || !a.tail_Xs) return false;
            if (tg <= 0 || tg % cpt != 0 || tg % 8 != 0 || kout % 8 != 0) return false;
            if ((kout + tg - 1) / tg > kTailCounterInts) return false;
            if ((reinterpret_cast<uintptr_t>(a.Y) | reinterpret_cast<uintptr_t>(a.tail_Xq)) & 15u) return false;
        }
    }
    pl.pro = fused ? kProNorm : quant ? kProQuant : kProCodes;
    pl.MT = a.M <= 8 ? 1 : (a.M <= 16 ? 2 : 4);
    pl.GM = a.g == 64 ? 64 : a.g == 128 ? 128 : 256;
    pl.bpu = a.g > 256 ? a.g / 256 : 1;
    pl.upt = a.K / (256 * pl.bpu);
    pl.block_bytes = kBlockW + 32 * (a.g >= 256 ? 1 : 256 / a.g);
    pl.tiles = (a.N + 15) / 16;
    pl.U = static_cast<long long>(pl.tiles) * pl.upt;
    // Up to two CTAs per SM where their registers and shared memory fit twice, never more CTAs than row tiles.
    // Two row tiles at once where the CTA that holds most has two at least and more than eight blocks per warp: half the reads of activations,
    // twice the code, which runs cold, and a longer first step. us, one tile and two: M = 16, g = 64 2560 x 9728 10.7 and 9.1, 19456 x 2560
    // 12.8 and 11.7, 155776 x 2560 77 and 64; g = 128 9728 x 11008 28.0 and 23.8; M = 32, g = 256 155776 x 2560 98 and 76 (with its quantiser); but
    // 6144 x 2560 at M = 32 11.1 and 12.3, at g >= 128 and M = 9, where the other form fits an SM twice, 2560 x 9728 9.4 and 9.7, and where no CTA
    // has two tiles, M = 32, g = 64 2048 x 16640, 13.0 and 17.4. Decode step, batch 16: g = 64 1790 and 1733, g = 128 1662 and 1610.
    // A lone last tile counts in the split over the warps as two do (its steps cost little less), so an odd number of tiles streams as long as
    // the next even one: M = 32, g = 64 6144 x 9728, three tiles, 21.5 and 23.6, row-major 21.9 and 26.2; M = 19, 19456 x 9728, nine, 50.1 and 54.2.
    // Dealing blocks out evenly instead is faster there but slower at M = 16 (19456 x 2560 11.5 and 12.2). So odd numbers only from where one
    // tile more is little against the gain, earlier while a run is short of what memory gives: M = 16, g = 64 9728 x 4096, five, 12.0 and 11.5, but
    // 9728 x 9728 21.1 and 21.3, row-major 22.6 and 23.3; M = 16, g = 256 9728 x 22784, five, 49.8 and 45.1.
    // (Packed and row-major weights take the same, so that they give the same bits; row-major alone, M > 16 at g = 128 would be better off with one tile:
    // 2560 x 9728 15.3 and 15.8, 8448 x 9728 24.9 and 27.0; packed 13.7 and 13.6, 22.1 and 22.4.)
    const int held = (pl.tiles + sms - 1) / sms, most = held * (a.K / 256);  // row tiles and blocks of the CTA that holds most, a CTA per SM
    const bool short_run = most <= 20 * kWarps;
    const int odd_from = pl.MT == 2 ? (pl.GM > 64 ? 3 : short_run ? 5 : 9) : pl.GM == 256 && short_run ? 9 : 15;
    // g >= 256 at 9..16 rows fits an SM twice and promotes little: only the longest runs (M = 16 155776 x 2560 65.3 and 62.2; 20000 x 2560 12.6 and 12.5; the
    // step at batch 16, context 200 1599 and 1613, at batch 14, context 900 1826 and 1842).
    const bool two = pl.MT == 4 || pl.GM == 64 || (pl.GM == 128 ? a.M > 12 : most > 32 * kWarps);
    pl.NR = pl.MT > 1 && most > 8 * kWarps && two && held >= 2 && (held % 2 == 0 || held >= odd_from) ? 2 : 1;
    pl.ctas = gemv_packed_ctas(pl.tiles, sms, two_per_sm(pl.MT, pl.GM, pl.NR));
    if ((pl.U + 1) * static_cast<long long>(pl.ctas) * kWarps >= (1ll << 32)) return false;  // 32-bit range math
    return true;
}

void gemv::fill_params(const LinearArgs& a, const Plan& pl, int* status, GemvPackedParams& p) {
    p.a = a;
    p.packed = static_cast<const unsigned char*>(a.packed);
    p.block_bytes = pl.block_bytes;
    p.upt = pl.upt;
    p.bpu = pl.bpu;
    p.U = static_cast<unsigned>(pl.U);
    p.status = status;
#ifdef W8A8_TRACE
    const char* v = std::getenv("W8A8_ABLATE");
    p.ablate = v ? std::atoi(v) : 0;
#endif
}

namespace {

template <int MT, int GM, int NR, int PRO, int ST, int KI, int EPI, bool EXTRA>
__global__ void __launch_bounds__(kThreads, two_per_sm(MT, GM, NR) ? 2 : 1)
gemv_packed_kernel(const __grid_constant__ GemvPackedParams p) {
    gemv_body<MT, GM, NR, PRO, ST, KI, EPI, EXTRA, false>(p, nullptr);
}

template <int MT, int GM, int NR, int PRO, int ST, int KI, int EPI, bool EXTRA>
int launch_variant(const LinearArgs& a, const Plan& pl, int* status, cudaStream_t stream) {
    GemvPackedParams p;
    fill_params(a, pl, status, p);
    auto kern = gemv_packed_kernel<MT, GM, NR, PRO, ST, KI, EPI, EXTRA>;
    const size_t ring = static_cast<size_t>(kWarps) * ST * kStagePitch + 128;
    const size_t smem = ring + (PRO == kProNorm ? fused_smem_bytes(a.K, a.G) : 0);
    const size_t most = ring + (PRO == kProNorm ? fused_smem_bytes(256 * KI, 4 * KI) : 0);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.ctas, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled(kPdlLinear) ? 1 : 0;
    static SmemAttribute attribute;
    cudaError_t e = launch_with_smem(attribute, static_cast<int>(most), cfg, kern, p);
    if (e != cudaSuccess) return fail(W8A8_ERR_CUDA, "gemv_packed launch: %s", cudaGetErrorString(e));
    return W8A8_OK;
}

template <int MT, int GM, int NR>
int launch_pro(const LinearArgs& a, const Plan& pl, int* status, cudaStream_t s) {
    if constexpr (MT == 1) {
        if (pl.pro == kProNorm) {
            if (a.K <= 2560) return launch_variant<1, GM, 1, kProNorm, 2, 10, -1, false>(a, pl, status, s);
            return launch_variant<1, GM, 1, kProNorm, 2, 16, -1, false>(a, pl, status, s);
        }
        if (pl.pro == kProQuant) return launch_variant<1, GM, 1, kProQuant, 3, 1, -1, false>(a, pl, status, s);
    }
    if (!plain_instance(a)) return launch_variant<MT, GM, NR, kProCodes, 3, 1, -1, true>(a, pl, status, s);
    switch (a.epilogue) {
        case W8A8_EPI_NONE: return launch_variant<MT, GM, NR, kProCodes, 3, 1, W8A8_EPI_NONE, false>(a, pl, status, s);
        case W8A8_EPI_SWIGLU: return launch_variant<MT, GM, NR, kProCodes, 3, 1, W8A8_EPI_SWIGLU, false>(a, pl, status, s);
        default: return launch_variant<MT, GM, NR, kProCodes, 3, 1, W8A8_EPI_RESIDUAL, false>(a, pl, status, s);
    }
}

template <int MT, int NR>
int launch_gm(const LinearArgs& a, const Plan& pl, int* status, cudaStream_t s) {
    switch (pl.GM) {
        case 64: return launch_pro<MT, 64, NR>(a, pl, status, s);
        case 128: return launch_pro<MT, 128, NR>(a, pl, status, s);
        default: return launch_pro<MT, 256, NR>(a, pl, status, s);
    }
}

// One thread per 16 bytes of the packed image.
__global__ void __launch_bounds__(256) pack_weight_kernel(const int8_t* __restrict__ W, const __half* __restrict__ S,
                                                          int N, int K, int g, int G, int block_bytes,
                                                          unsigned char* __restrict__ out, size_t total16) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= total16) return;
    const int per_block = block_bytes / 16;
    const size_t blk = i / per_block;
    const int r = static_cast<int>(i % per_block);
    const int kblocks = K / 256;
    const int rt = static_cast<int>(blk / kblocks), kb = static_cast<int>(blk % kblocks);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < kBlockW / 16) {
        // [chunk][half][lane]: 16 bytes of row (lane/4) + 8*half at K offset chunk*64 + (lane%4)*16
        const int lane = r & 31, half = (r >> 5) & 1, ch = r >> 6;
        const int row = rt * 16 + (lane >> 2) + 8 * half;
        const int k = kb * 256 + ch * 64 + (lane & 3) * 16;
        if (row < N) v = *reinterpret_cast<const uint4*>(W + static_cast<size_t>(row) * K + k);
    } else {
        // scales: [16 rows][gpb] fp16, 8 halves per 16-byte piece
        const int gpb = g >= 256 ? 1 : 256 / g;
        __align__(16) __half h[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int idx = (r - kBlockW / 16) * 8 + e;  // row * gpb + q
            const int row = rt * 16 + idx / gpb, q = idx % gpb;
            const int j = g >= 256 ? (kb * 256) / g : kb * gpb + q;
            h[e] = row < N ? S[static_cast<size_t>(row) * G + j] : __float2half(0.0f);
        }
        v = *reinterpret_cast<const uint4*>(h);
    }
    reinterpret_cast<uint4*>(out)[i] = v;
}

}  // namespace

size_t packed_weight_bytes(int N, int K, int g) {
    g = norm_group(K, g);
    if (!packable(N, K, g)) return 0;
    const size_t block_bytes = kBlockW + 32 * (g >= 256 ? 1 : 256 / g);
    return static_cast<size_t>((N + 15) / 16) * (K / 256) * block_bytes;
}

int launch_pack_weight(const int8_t* W, const __half* S, int N, int K, int g, void* out, cudaStream_t s) {
    g = norm_group(K, g);
    const size_t bytes = packed_weight_bytes(N, K, g);
    if (bytes == 0) return fail(W8A8_ERR_UNSUPPORTED, "N=%d K=%d group=%d cannot be packed (K %% 256, group 64/128/k*256)", N, K, g);
    if ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(out)) & 15u)
        return fail(W8A8_ERR_INVALID_ARG, "pack_weight needs 16-byte aligned W and output");
    const int block_bytes = kBlockW + 32 * (g >= 256 ? 1 : 256 / g);
    const size_t total16 = bytes / 16;
    pack_weight_kernel<<<static_cast<unsigned>((total16 + 255) / 256), 256, 0, s>>>(
        W, S, N, K, g, num_groups(K, g), block_bytes, static_cast<unsigned char*>(out), total16);
    return check_launch("pack_weight_kernel");
}

// At most three blocks per warp: there the fused quantiser costs what the launch it replaces costs in a replayed graph (packed,
// 4097 x 2560 at M = 8: 4.66 against 4.72 us; row-major, 6144 x 2560: 7.23 against 7.40) and saves that launch on the host
// (eager: 7.4 -> 5.2 and 7.4 -> 6.9 us a call). With longer runs every block is quantised by every row tile's warps again:
// packed 2560 x 9728 at M = 8 8.0 -> 9.5 us, row-major 19456 x 2560 12.4 -> 13.8.
bool quant_form_wins(const LinearArgs& a) {
    const int tiles = (a.N + 15) / 16, ctas = gemv_packed_ctas(tiles, device_sms(), true);
    return static_cast<long long>(tiles) * (a.K / 256) <= 3ll * kWarps * ctas;
}

bool gemv_packed_supports(const LinearArgs& a) {
    Plan pl;
    return make_plan(a, pl, false, device_sms());
}

int gemv_form(int M, int N, int K, int g, int sms, bool packed, int* out3) {
    alignas(16) static const unsigned char there[16] = {};  // (never read)
    LinearArgs a = {};
    a.M = M; a.N = N; a.K = K; a.g = g; a.G = num_groups(K, g);
    a.Xq = a.W = reinterpret_cast<const int8_t*>(there);
    a.Xs = reinterpret_cast<const float*>(there);
    a.w_scale = reinterpret_cast<const __half*>(there);
    a.packed = there;
    a.Y = reinterpret_cast<__half*>(const_cast<unsigned char*>(there));
    Plan pl;
    if (N < 1 || K < 1 || sms < 1 || !make_plan(a, pl, !packed, sms)) return W8A8_ERR_UNSUPPORTED;
    out3[0] = 8 * pl.MT;
    out3[1] = pl.NR;
    out3[2] = pl.ctas;
    return W8A8_OK;
}

int launch_linear_gemv_packed(const LinearArgs& a, int* device_status, cudaStream_t s) {
    Plan pl;
    if (!make_plan(a, pl, false, device_sms())) return fail(W8A8_ERR_UNSUPPORTED, "packed gemv kernel does not take this shape");
    if (pl.MT == 1) return launch_gm<1, 1>(a, pl, device_status, s);
    if (pl.NR == 1) return pl.MT == 2 ? launch_gm<2, 1>(a, pl, device_status, s) : launch_gm<4, 1>(a, pl, device_status, s);
    return pl.MT == 2 ? launch_gm<2, 2>(a, pl, device_status, s) : launch_gm<4, 2>(a, pl, device_status, s);
}

}  // namespace w8a8

W8A8_TRACE_READER(gemv_packed)
