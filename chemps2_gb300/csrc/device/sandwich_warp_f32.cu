// The team-cooperative block-sandwich kernel in FP32 (sandwich_warp.cuh).
#include "sandwich_warp.cuh"

namespace c2g {

cudaError_t launch_sandwich_warp_f32(const WarpLaunch& w, int ntiles, const SlotPtrs& sp, cudaStream_t stream) {
  if (ntiles <= 0) return cudaSuccess;
  sandwich_warp_kernel<float><<<ntiles, kWT, 0, stream>>>(w, sp);
  return cudaGetLastError();
}

}  // namespace c2g
