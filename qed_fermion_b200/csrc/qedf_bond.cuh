// What the kernels of the bond-bond correlators share.
#pragma once
#include "qedf_common.cuh"
#include "qedf_internal.h"

namespace qedf {

struct BondArgs {
  int kind;  // 1: T1, 21: T21, 2: T2, 4: T4
  const void* eta;
  const void* g;
  const void* ep;  // e^{i phi_x} per site, [Ltau][Vs]
  const int* ps;
  const int* pt;
  int npairs, nrv, L, Nt;
  void* fa;
  void* fb;
};

template <typename R>
__device__ __forceinline__ Cx<R> ldcx(const R* base, int64_t i) {
  return *reinterpret_cast<const Cx<R>*>(base + 2 * i);
}
template <typename R>
__device__ __forceinline__ Cx<R> conjc(Cx<R> a) {
  return mk<R>(a.re, -a.im);
}

}  // namespace qedf
