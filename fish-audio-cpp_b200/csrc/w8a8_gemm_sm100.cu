// Chooses and launches the tcgen05 GEMM (kernel and its reasons: w8a8_gemm_sm100.cuh).
#include "w8a8_gemm_sm100.cuh"

#include <algorithm>

namespace w8a8 {
namespace gemm {

// Group sizes without a case of their own, and calls that want the group sums. (Costs fitted at groups of 32, 320, 512 and K, 40 to 4001
// tokens, within 15 %. Nowhere there was the pair the faster one: 5-15 % slower.)
const Form* forms_any(int* count) {
    static const Form table[] = {form<128, false, 0>({332, 332, 1250, 0, 1760, 0, 3500}), form<128, true, 0>({345, 355, 1840, 0, 1760, 0, 3500})};
    *count = static_cast<int>(sizeof(table) / sizeof(table[0]));
    return table;
}

namespace {

const Form* forms(int g, int* count) {
    return g == 64 ? forms_g64(count) : g == 128 ? forms_g128(count) : g == 256 ? forms_g256(count) : forms_any(count);
}

// Stages of 128 bytes that each CTA of a split takes: whole K-groups.
int split_kb(int K, int g, int splits) {
    const int unit = g > BK ? g / BK : 1;
    return (K / BK / unit + splits - 1) / splits * unit;
}

// The stages that a run of kb takes in the form: whole units.
int padded_kb(const Form& f, int kb) { return (kb + f.unit_kb - 1) / f.unit_kb * f.unit_kb; }

// setmaxnreg moves registers between the warpgroups of the widest form; the sums balance only for the register count the kernel
// was compiled to (Form::launch_regs per thread). An unbalanced sum blocks for ever in setmaxnreg.inc, a wait nothing bounds, so in a
// build that came out differently that form is not taken.
bool balanced(const Form& f) {
    if (f.launch_regs == 0) return true;
    for (int i = 0; i < 2 && f.kernel[i]; ++i) {
        int r = f.state[i].registers.load(std::memory_order_relaxed);
        if (r == 0) {
            cudaFuncAttributes fa;
            if (cudaFuncGetAttributes(&fa, f.kernel[i]) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
            f.state[i].registers.store(r = fa.numRegs, std::memory_order_relaxed);
        }
        if (r != f.launch_regs) return false;
    }
    return true;
}

// Which side of the tiles is walked first. Tokens, so that concurrent CTAs share weight tiles in L2 and each weight is read from memory once;
// but where the activation codes are the larger operand and do not stay in L2 beside the rest, every such sweep reads them from memory
// again. Then rows: the weights stay, and the codes are read once. us back to back, tokens and rows first: 8192 x 2560 x 9728 (80 MB of
// codes) g = 256 198 and 182, g = 128 294 and 256; 16384 x 2560 x 9728 407 and 337; 6500 (63 MB) 166 and 160; 5000 (49 MB) 129.6 and
// 129.9; 2048 59.8 and 62.2.
bool walk_rows_first(int M, int N, int K) { return M > N && static_cast<long long>(M) * K >= 60000000ll; }

struct Choice {
    const Form* form;
    int splits;
};

// The tile form that ends first: whole waves of tiles over the SMs (or pairs), each wave at its tiles' cost or at the time in which memory brings
// the weights that it is the first to read (6 TB/s), whichever is longer, and a quarter of the other: 19456 rows by 64 tokens are 152 tiles, a
// wave that memory bounds and four tiles more. A width that leaves the last wave nearly empty loses to one that fills it; narrow tiles win
// where there are few tokens.
// A tile's K is split over two or four CTAs where all of them fit the chip at once (a cluster of four leaves some SMs of a
// GPC over: 128 of 148 taken as usable); 1.9 and 3.4 us for meeting and adding up choose best, 1.4 and 2.9 at g = 64. A split adds the groups in
// another order than the other kernels do, so it has to save 6 % at least, and K = 2560 never splits.
// table_g: the group size whose forms are looked at (0: those of any group size). pair: -1 either, 0 one CTA per tile, 1 a pair.
// only_bt, only_splits: 0, or the token width and the split (1: none) to take; no form where they do not fit the shape.
template <class Usable>
Choice choose(int M, int N, int K, int table_g, int g, bool residual, int sms, int pair, int only_bt, int only_splits, Usable usable) {
    int count = 0;
    const Form* table = forms(table_g, &count);
    Choice best = {nullptr, 1};
    double best_ns = 0;
    for (int i = 0; i < count; ++i) {
        const Form& f = table[i];
        if (pair >= 0 && (f.pair != (pair != 0) || f.split)) continue;
        if (only_bt && f.bt != only_bt) continue;
        const int rows = f.pair ? 2 * BR : BR, walkers = f.pair ? sms / 2 : sms, kb_total = K / BK;
        const Cost& c = f.cost;
        const double tile_ns = c.tile + (N % 8 == 0 ? (residual ? c.residual : 0.0f) : residual ? c.odd_residual : c.odd);
        const long tiles_m = (M + f.bt - 1) / f.bt, tiles = tiles_m * ((N + rows - 1) / rows);
        for (int splits = f.split ? 2 : 1; splits <= (f.split ? 4 : 1); splits *= 2) {
            if (only_splits && splits != only_splits) continue;
            if (f.split && (tiles * splits > (splits == 2 ? sms / 2 * 2 : sms * 7 / 8 - 1) || (splits - 1) * split_kb(K, g, splits) >= kb_total))
                continue;
            const double kb = padded_kb(f, f.split ? split_kb(K, g, splits) : kb_total);
            const double wave_ns = kb * c.stage + kb * BK / g * c.group + tile_ns;
            const double memory_ns = static_cast<double>(rows) * K / tiles_m / splits / 6000;  // a tile's share of the weights it is the first to read
            const long waves = (tiles * splits + walkers - 1) / walkers, last = tiles * splits - (waves - 1) * walkers;
            auto both = [](double x, double y) { return std::max(x, y) + 0.25 * std::min(x, y); };
            double ns = c.start + (waves - 1) * both(wave_ns, walkers * memory_ns) + both(wave_ns, last * memory_ns);
            if (f.split) ns = (ns + (splits == 2 ? 1900 : 3400) - (g == 64 ? 500 : 0)) / 0.94;
            if ((!best.form || ns < best_ns) && usable(f)) { best = {&f, splits}; best_ns = ns; }
        }
    }
    return best;
}

}  // namespace
}  // namespace gemm

bool gemm_supports(const LinearArgs& a) {
    if (a.M < 1 || !a.Xq || !a.Xs) return false;
    if (a.K % gemm::BK != 0 || a.g % 32 != 0 || a.K % a.g != 0) return false;
    if ((reinterpret_cast<uintptr_t>(a.W) | reinterpret_cast<uintptr_t>(a.Xq)) & 15u) return false;
    if (a.epilogue == W8A8_EPI_SWIGLU && (a.N % 16 != 0 || (reinterpret_cast<uintptr_t>(a.Y) & 15u))) return false;
    if (a.epilogue != W8A8_EPI_SWIGLU && a.N % 8 == 0 && (reinterpret_cast<uintptr_t>(a.Y) & 15u)) return false;
    if (a.residual && a.N % 8 == 0 && (reinterpret_cast<uintptr_t>(a.residual) & 15u)) return false;
    return true;
}

int gemm_form(int M, int N, int K, int g, int sms, int form, int only_bt, int only_splits, bool moved_registers, int* out3) {
    using namespace gemm;
    if (M < 1 || N < 1 || K < 1 || sms < 2 || K % BK != 0 || g % 32 != 0 || K % g != 0) return W8A8_ERR_UNSUPPORTED;
    const Choice c = choose(M, N, K, g, g, false, sms, form, only_bt, only_splits, [&](const Form& f) { return moved_registers || f.launch_regs == 0; });
    if (!c.form) return W8A8_ERR_UNSUPPORTED;
    out3[0] = c.form->bt;
    out3[1] = c.form->pair ? 2 : 1;
    out3[2] = c.splits;
    return W8A8_OK;
}

int launch_linear_gemm(const LinearArgs& a, int* device_status, cudaStream_t stream, int form) {
    using namespace gemm;
    if (!gemm_supports(a)) return fail(W8A8_ERR_UNSUPPORTED, "tcgen05 GEMM does not take this shape");
    const int sms = device_sms();

    const Choice choice = choose(a.M, a.N, a.K, a.dump ? 0 : a.g, a.g, a.epilogue == W8A8_EPI_RESIDUAL, sms, form, a.gemm_bt, a.gemm_splits, balanced);
    const Form* best = choice.form;
    const int best_splits = choice.splits;
    if (!best) return fail(W8A8_ERR_UNSUPPORTED, "no tile form of the tcgen05 GEMM for this shape (token width %d, splits %d asked for)",
                           a.gemm_bt, a.gemm_splits);

    const int bt = best->bt, rows = best->pair ? 2 * BR : BR;
    CUtensorMap map_w, map_x, map_y;
    const uint64_t K = static_cast<uint64_t>(a.K);
    int rc = make_tensor_map_2d_u8(&map_w, a.W, K, static_cast<uint64_t>(a.N), K, BK, BR, 1);
    if (rc) return rc;
    rc = make_tensor_map_2d_u8(&map_x, a.Xq, K, static_cast<uint64_t>(a.M), K, BK, best->pair ? bt / 2 : bt, 1);
    if (rc) return rc;
    const int ycols = a.epilogue == W8A8_EPI_SWIGLU ? a.N / 2 : a.N;
    GemmParams p;
    p.a = a;
    p.status = device_status;
    const int tiles_m = (a.M + bt - 1) / bt, tiles_n = (a.N + rows - 1) / rows;
    const bool rows_first = best->kernel[1] && walk_rows_first(a.M, a.N, a.K);
    p.inner = rows_first ? tiles_n : tiles_m;
    p.tiles_total = tiles_m * tiles_n;
    p.splits = best_splits;
    p.split_kb = split_kb(a.K, a.g, best_splits);
    p.tma_store = ycols % 8 == 0 && (reinterpret_cast<uintptr_t>(a.Y) & 15u) == 0;
    map_y = map_x;  // (a valid map in either case; only the TMA store reads it)
    if (p.tma_store) {
        // Y as rows of bytes; a box is BT rows x 128 bytes (64 fp16 columns), 128-byte swizzle; stores clip at the
        // tensor's edges, so ragged last tiles need no care
        rc = make_tensor_map_2d_u8(&map_y, a.Y, static_cast<uint64_t>(ycols) * 2, static_cast<uint64_t>(a.M),
                                   static_cast<uint64_t>(ycols) * 2, 128, bt, 1);
        if (rc) return rc;
    }
    cudaLaunchConfig_t cfg = {};
    // persistent: one CTA (or CTA pair) per SM (pair of SMs) walks its tiles
    const int walkers_max = best->pair ? sms / 2 : sms;
    const int walkers = p.tiles_total < walkers_max ? p.tiles_total : walkers_max;
    cfg.gridDim = dim3(best->pair ? 2 * walkers : best->split ? best_splits * p.tiles_total : walkers, 1, 1);
    cfg.blockDim = dim3(best->threads, 1, 1);
    cfg.dynamicSmemBytes = best->smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (best->pair || best->split) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = best->pair ? 2 : best_splits;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (pdl_enabled(kPdlLinear)) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t e = launch_with_smem(best->state[rows_first].attribute, best->smem, cfg, best->kernel[rows_first], map_w, map_x, map_y, p);
    if (e != cudaSuccess) return fail(W8A8_ERR_CUDA, "gemm launch: %s", cudaGetErrorString(e));
    return W8A8_OK;
}

}  // namespace w8a8
