// The decode-sized packed GEMM on 4-bit codes (one file per container: they compile side by side).
#include "linear_gv_launch.cuh"

namespace tsb {
namespace gv {
template cudaError_t launch<4>(const Params&, const Plan&, bool, bool, cudaStream_t);
}  // namespace gv
}  // namespace tsb
