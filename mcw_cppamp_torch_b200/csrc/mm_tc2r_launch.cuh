// Launches of the two-SM kernel, for the files that compile it (mm_tc2r_*.cu).
#ifndef THC_MM_TC2R_LAUNCH_CUH
#define THC_MM_TC2R_LAUNCH_CUH

#include "mm_tc2r.cuh"
#include "per_device.h"

namespace thc {
namespace mm {

template <class P, int BN2>
int tc2r_resident_clusters() {
  constexpr int SMEM = tc2r_smem_bytes<BN2, P::PREC>();
  static PerDevice resident;
  return resident.get(ctx().device, [] {
    THC_CUDA(cudaFuncSetAttribute(tc2r_kernel<P, BN2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * ctx().sm_count, 1, 1);
    cfg.blockDim = dim3(T2_THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM;
    int c = 0;
    if (cudaOccupancyMaxActiveClusters(&c, tc2r_kernel<P, BN2>, &cfg) != cudaSuccess || c < 1) {
      cudaGetLastError();
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
      cfg.attrs = &attr; cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&c, tc2r_kernel<P, BN2>, &cfg) != cudaSuccess || c < 1) {
        cudaGetLastError();
        c = ctx().sm_count / 2;
      }
    }
    return std::min(c, ctx().sm_count / 2);
  });
}
template <class P, int BN2>
void launch_tc2r_kernel(const P &p, long items, bool early) {
  const long clusters = std::min<long>(items, tc2r_resident_clusters<P, BN2>());
  launch_on_stream(early, tc2r_kernel<P, BN2>, dim3((unsigned)(2 * clusters), 1, 1), T2_THREADS, tc2r_smem_bytes<BN2, P::PREC>(), p, stall_ctl(),
                   sched_counter());
  check_launch("tc2r_kernel");
}

#define TC2R_WIDTH(BN2, ...) \
  template int tc2r_resident_clusters<__VA_ARGS__, BN2>(); \
  template void launch_tc2r_kernel<__VA_ARGS__, BN2>(const __VA_ARGS__ &, long, bool);
#define TC2R_NARROW(...) TC2R_WIDTH(64, __VA_ARGS__) TC2R_WIDTH(128, __VA_ARGS__)     // pixel pairs
#define TC2R_BLOCKS(...) TC2R_WIDTH(128, __VA_ARGS__) TC2R_WIDTH(256, __VA_ARGS__)    // MN-major 16-bit columns
#define TC2R_ALL(...) TC2R_NARROW(__VA_ARGS__) TC2R_WIDTH(192, __VA_ARGS__) TC2R_WIDTH(256, __VA_ARGS__)

}  // namespace mm
}  // namespace thc

#endif
