// The tcgen05 GEMM for groups of 64 (w8a8_gemm_sm100.cuh). A file of its own so that the instances compile side by side.
#include "w8a8_gemm_sm100.cuh"

namespace w8a8 {
namespace gemm {

const Form* forms_g64(int* count) { return all_forms<64>(count); }

}  // namespace gemm
}  // namespace w8a8
