// Instances of the cluster-resident kernel (msx_resident.cuh) for lines of 64, 128 and 256.
#include "msx_resident.cuh"

namespace msx {

template <class LR, class LC>
struct ResidentImpl {
  using K = Resident<LR, LC>;
  static cudaLaunchConfig_t config(int w, int cl, int waves, cudaStream_t st, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(waves * cl));
    cfg.blockDim = dim3(kResidentThreads);
    cfg.dynamicSmemBytes = K::smem(w, cl);
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)cl;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
  }
  static cudaError_t configure() {
    cudaError_t e = cudaFuncSetAttribute(resident_kernel<LR, LC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(resident_kernel<LR, LC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
  }
  static int most(int w, int cl, int sms) {
    if (K::smem(w, cl) > 232448 || cl > K::NY) return 0;
    const size_t by_smem = 233472 / (K::smem(w, cl) + 1024), by_threads = 2048 / kResidentThreads;
    return (int)(by_smem < by_threads ? by_smem : by_threads) * sms / cl;
  }
  static cudaError_t clusters(int w, int cl, int* n) {
    *n = 0;
    if (K::smem(w, cl) > 232448 || cl > K::NY) return cudaSuccess;
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg = config(w, cl, 1, nullptr, &at);
    return cudaOccupancyMaxActiveClusters(n, resident_kernel<LR, LC>, &cfg);
  }
  static cudaError_t launch(ResidentArgs a, int waves, int cl, cudaStream_t st) {
    cudaLaunchAttribute at{};
    a.tbufs = K::tbufs(a.x_hi - a.x_lo, cl);
    const cudaLaunchConfig_t cfg = config(a.x_hi - a.x_lo, cl, waves, st, &at);
    return cudaLaunchKernelEx(&cfg, resident_kernel<LR, LC>, a);
  }
  static ResidentOps ops() {
    return ResidentOps{LR::FFT::tw_words(), LC::FFT::tw_words(), &LR::FFT::host_twiddles, &LC::FFT::host_twiddles,
                       &configure, &most, &clusters, &launch};
  }
};

namespace {
using Line64 = ResidentLine<64, 8, 8, 8>;
using Line128 = ResidentLine<128, 8, 16, 8>;
using Line256 = ResidentLine<256, 16, 16, 16>;

template <class LR>
const ResidentOps* of_rows(int ny) {
  static const ResidentOps table[] = {ResidentImpl<LR, Line64>::ops(), ResidentImpl<LR, Line128>::ops(),
                                      ResidentImpl<LR, Line256>::ops()};
  return ny == 64 ? &table[0] : ny == 128 ? &table[1] : ny == 256 ? &table[2] : nullptr;
}
}  // namespace

const ResidentOps* resident_ops(int ny, int nx) {
  return nx == 64 ? of_rows<Line64>(ny) : nx == 128 ? of_rows<Line128>(ny) : nx == 256 ? of_rows<Line256>(ny) : nullptr;
}

}  // namespace msx
