// The decode linear over the row-major matrix, for weights that were not packed: the kernel of w8a8_gemv_packed.cuh with TMA
// boxes of the matrix as its blocks. It replaces a stream-K form of one CTA per SM whose cut tiles met in global scratch through
// L2 atomics: at g = 64, M = 8, 6144 x 2560 10.4 -> 6.0 us, 2560 x 9728 14.4 -> 9.0, 19456 x 2560 22.4 -> 12.2 (4.1 TB/s); at
// M = 32 19456 x 2560 59 -> 22. Sixteen runs of 256 bytes per block reach a lower rate than the packed image's linear stream.
// The split, the sum of cut tiles and the arithmetic are the packed form's.
#include "w8a8_gemv_packed.cuh"

namespace w8a8 {
namespace {
using namespace gemv;

template <int MT, int GM, int NR, int PRO, bool EXTRA>
__global__ void __launch_bounds__(kThreads, two_per_sm(MT, GM, NR) ? 2 : 1)
gemv_rows_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ GemvPackedParams p) {
    gemv_body<MT, GM, NR, PRO, 3, 1, -1, EXTRA, true>(p, &map);
}

template <int MT, int GM, int NR, int PRO, bool EXTRA>
int launch_variant(const LinearArgs& a, const Plan& pl, int* status, cudaStream_t stream) {
    CUtensorMap map;
    // W seen as [N rows][K/128 blocks][128 bytes]; one box = 16 rows x 2 blocks, 128-byte swizzle
    int rc = make_tensor_map_3d_u8(&map, a.W, 128, static_cast<uint64_t>(a.K / 128), static_cast<uint64_t>(a.N), 128,
                                   static_cast<uint64_t>(a.K), 128, 2, 16, 1);
    if (rc) return rc;
    GemvPackedParams p;
    fill_params(a, pl, status, p);
    auto kern = gemv_rows_kernel<MT, GM, NR, PRO, EXTRA>;
    const size_t smem = static_cast<size_t>(kWarps) * 3 * kBlockW + 1024;
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
    cudaError_t e = launch_with_smem(attribute, static_cast<int>(smem), cfg, kern, map, p);
    if (e != cudaSuccess) return fail(W8A8_ERR_CUDA, "gemv_rows launch: %s", cudaGetErrorString(e));
    return W8A8_OK;
}

template <int GM, bool EXTRA>
int launch_codes(const LinearArgs& a, const Plan& pl, int* status, cudaStream_t s) {
    if (pl.MT == 1) return launch_variant<1, GM, 1, kProCodes, EXTRA>(a, pl, status, s);
    if (pl.NR == 1)
        return pl.MT == 2 ? launch_variant<2, GM, 1, kProCodes, EXTRA>(a, pl, status, s) : launch_variant<4, GM, 1, kProCodes, EXTRA>(a, pl, status, s);
    return pl.MT == 2 ? launch_variant<2, GM, 2, kProCodes, EXTRA>(a, pl, status, s) : launch_variant<4, GM, 2, kProCodes, EXTRA>(a, pl, status, s);
}

template <int GM>
int launch_gm(const LinearArgs& a, const Plan& pl, int* status, cudaStream_t s) {
    if (pl.pro == kProQuant) return launch_variant<1, GM, 1, kProQuant, false>(a, pl, status, s);
    return plain_instance(a) ? launch_codes<GM, false>(a, pl, status, s) : launch_codes<GM, true>(a, pl, status, s);
}

}  // namespace

bool gemv_rows_supports(const LinearArgs& a) {
    Plan pl;
    return make_plan(a, pl, true, device_sms());
}

int launch_linear_gemv_rows(const LinearArgs& a, int* device_status, cudaStream_t s) {
    Plan pl;
    if (!make_plan(a, pl, true, device_sms())) return fail(W8A8_ERR_UNSUPPORTED, "TMA gemv kernel does not take this shape");
    switch (pl.GM) {
        case 64: return launch_gm<64>(a, pl, device_status, s);
        case 128: return launch_gm<128>(a, pl, device_status, s);
        default: return launch_gm<256>(a, pl, device_status, s);
    }
}

}  // namespace w8a8

W8A8_TRACE_READER(gemv_rows)
