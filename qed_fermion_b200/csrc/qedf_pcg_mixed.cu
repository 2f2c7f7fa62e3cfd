// The persistent PCG kernels: mixed precision.
#include "qedf_pcg_kernel.cuh"

namespace qedf {

int launch_pcg_mixed(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st) {
  return launch_pcg_by<float, double, float, float>(p, taps, by, st);
}

}  // namespace qedf
