// One-pass bond-bond correlators, complex64.
#include "qedf_corr.cuh"

extern "C" int qedf_bb_corr_c64(int kind, const float* eta, const float* g_eta, const float* ephase, const int* ps, const int* pt,
                                int npairs, int Nrv, int Lx, int Ltau, double* S, qedf_stream_t s) {
  if (kind == 0) return QEDF_ERR_ARG;
  return qedf::corr_entry<float>(kind, eta, g_eta, ephase, ps, pt, npairs, Nrv, Lx, Ltau, S,
                              reinterpret_cast<cudaStream_t>(s));
}

extern "C" int qedf_bb_corr_sum_c64(const float* eta, const float* g_eta, const float* ephase, const int* ps, const int* pt,
                                    int npairs, int Nrv, int Lx, int Ltau, double* S, qedf_stream_t s) {
  return qedf::corr_entry<float>(0, eta, g_eta, ephase, ps, pt, npairs, Nrv, Lx, Ltau, S,
                                reinterpret_cast<cudaStream_t>(s));
}
