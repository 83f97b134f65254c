// The team-cooperative block-sandwich kernel in FP64 (sandwich_warp.cuh).
#include "sandwich_warp.cuh"

namespace c2g {

cudaError_t launch_sandwich_warp_f64(const WarpLaunch& w, int ntiles, const SlotPtrs& sp, cudaStream_t stream) {
  if (ntiles <= 0) return cudaSuccess;
  sandwich_warp_kernel<double><<<ntiles, kWT, 0, stream>>>(w, sp);
  return cudaGetLastError();
}

}  // namespace c2g
