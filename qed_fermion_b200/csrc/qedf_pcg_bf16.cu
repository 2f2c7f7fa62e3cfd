// The persistent PCG kernels: mixed precision, p and z stored as bf16.
#include "qedf_pcg_kernel.cuh"

namespace qedf {

int launch_pcg_bf16(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st) {
  return launch_pcg_by<float, double, float, bf16>(p, taps, by, st);
}

}  // namespace qedf
