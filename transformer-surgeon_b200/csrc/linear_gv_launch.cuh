// Launch of the decode-sized packed GEMM: the instantiations behind gv::launch.
#pragma once
#include "linear_gv.cuh"

namespace tsb {
namespace gv {

template <int BITS, int NT, int R, bool GATED>
cudaError_t launch_one(const Params& p, const Plan& plan, bool pdl, cudaStream_t s) {
  auto* kernel = linear_gv_kernel<BITS, NT, R, GATED>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)plan.grid);
  cfg.blockDim = dim3((unsigned)plan.warps * 32);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (plan.ranks > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = (unsigned)plan.ranks;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <int BITS, int NT>
cudaError_t launch_nt(const Params& p, const Plan& plan, bool gated, bool pdl, cudaStream_t s) {
  if (gated) return plan.R == 1 ? launch_one<BITS, NT, 1, true>(p, plan, pdl, s) : launch_one<BITS, NT, 2, true>(p, plan, pdl, s);
  return plan.R == 1 ? launch_one<BITS, NT, 1, false>(p, plan, pdl, s) : launch_one<BITS, NT, 2, false>(p, plan, pdl, s);
}

template <int BITS>
cudaError_t launch(const Params& p, const Plan& plan, bool gated, bool pdl, cudaStream_t s) {
  return token_tiles(p.M) == 1 ? launch_nt<BITS, 1>(p, plan, gated, pdl, s) : launch_nt<BITS, 2>(p, plan, gated, pdl, s);
}

}  // namespace gv
}  // namespace tsb
