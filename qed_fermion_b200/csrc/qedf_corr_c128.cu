// One-pass bond-bond correlators, complex128.
#include "qedf_corr.cuh"

extern "C" int qedf_bb_corr_c128(int kind, const double* eta, const double* g_eta, const double* ephase, const int* ps, const int* pt,
                                int npairs, int Nrv, int Lx, int Ltau, double* S, qedf_stream_t s) {
  if (kind == 0) return QEDF_ERR_ARG;
  return qedf::corr_entry<double>(kind, eta, g_eta, ephase, ps, pt, npairs, Nrv, Lx, Ltau, S,
                              reinterpret_cast<cudaStream_t>(s));
}

extern "C" int qedf_bb_corr_sum_c128(const double* eta, const double* g_eta, const double* ephase, const int* ps, const int* pt,
                                    int npairs, int Nrv, int Lx, int Ltau, double* S, qedf_stream_t s) {
  return qedf::corr_entry<double>(0, eta, g_eta, ephase, ps, pt, npairs, Nrv, Lx, Ltau, S,
                                reinterpret_cast<cudaStream_t>(s));
}
