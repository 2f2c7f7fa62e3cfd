// The persistent PCG kernels: mixed precision, p and z stored as scaled fp16.
#include "qedf_pcg_kernel.cuh"

namespace qedf {

int launch_pcg_f16(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st) {
  return launch_pcg_by<float, double, float, __half>(p, taps, by, st);
}

}  // namespace qedf
