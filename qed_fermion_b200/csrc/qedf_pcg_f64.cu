// The persistent PCG kernels: double precision.
#include "qedf_pcg_kernel.cuh"

namespace qedf {

int launch_pcg_f64(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st) {
  return launch_pcg_by<double, double, double, double>(p, taps, by, st);
}

}  // namespace qedf
