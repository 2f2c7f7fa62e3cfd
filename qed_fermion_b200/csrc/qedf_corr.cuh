// One pass for a whole bond-bond correlator: per (pair, slice) the two fields,
// their 2-D transforms A(k) = sum_r a(r) e^{+2 pi i k.r / L} and B(k) = sum_r
// b(r) e^{-2 pi i k.r / L}, and A(k) B(k), none of which reaches memory.  A
// thread holds a whole line of L = P Q sites in registers: first a column (y),
// whose field values it forms from eta and G (neighbouring threads read
// neighbouring sites), then, after one exchange through shared memory, a row
// (x).  Lines are transformed by the prime-factor split where P and Q are
// coprime, else by Cooley-Tukey with twiddles.  A is the conjugate of the
// forward transform of conj(a).  A block takes a contiguous run of items, slice
// by slice and pairs within, so that its first vector and e^{i phi} stay in L1;
// its sum of products stays in shared memory.
//
// Eight warps per SM, which is what a line in registers leaves at L = 30 in
// double precision, bound it: the FP64 pipe is 37 % busy, shared memory 33 %.
// Measured against pair fields in memory, cuFFT and a k-space sum, 20 vectors
// and Ltau = 10 L, one correlator with 0.2 ms of host work: L = 30, complex128,
// 2.2 -> 1.1 ms, complex64 1.5 -> 0.6 ms; L = 20, 0.86 -> 0.39 and 0.58 -> 0.33;
// L = 48, complex64, 12 vectors, 2.0 -> 1.5 ms.  Lines of more than 32 sites in
// double precision leave one line per thread few registers (one correlator at
// L = 36: 1.33 against 1.31 ms), so a single correlator keeps the two passes
// there.  Blocks per SM: at L = 30, complex128, two with 255 registers a thread
// take 1.1 ms, three with 168 1.35 ms: the shared memory of the third is L1 that
// the vectors' slices need.  The sum of all four, in place of T1, T21 and T4 in
// turn: L = 30, 20 vectors, complex128 3.6 -> 1.57 ms, complex64 2.2 -> 0.94; L =
// 20, 1.5 -> 0.64 and 1.15 -> 0.51; L = 48, complex64, 12 vectors, 5.2 -> 1.5; L =
// 36, complex128, 12 vectors, 4.4 -> 1.4; L = 40, 6.8 -> 1.8.
#pragma once
#include <cooperative_groups.h>

#include <algorithm>

#include "qedf_bond.cuh"
#include "qedf_corr_any.cuh"

namespace qedf {

// X_k = sum_n x_n e^{-2 pi i n k / N}, in place
template <typename R, int N>
__device__ __forceinline__ void dft_odd(Cx<R> (&x)[N], const double (&c)[N], const double (&s)[N]) {
  constexpr int H = (N - 1) / 2;
  Cx<R> u[H], d[H];
  const Cx<R> x0 = x[0];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    u[j] = x[j + 1] + x[N - 1 - j];
    d[j] = x[j + 1] - x[N - 1 - j];
    x[0] = x[0] + u[j];
  }
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    Cx<R> a = x0, b = mk<R>(0, 0);
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      const R cj = (R)c[j * k % N], sj = (R)s[j * k % N];
      a = mk<R>(fma(cj, u[j - 1].re, a.re), fma(cj, u[j - 1].im, a.im));
      b = j == 1 ? mk<R>(sj * d[0].re, sj * d[0].im) : mk<R>(fma(sj, d[j - 1].re, b.re), fma(sj, d[j - 1].im, b.im));
    }
    x[k] = mk<R>(a.re + b.im, a.im - b.re);
    x[N - k] = mk<R>(a.re - b.im, a.im + b.re);
  }
}
template <typename R>
__device__ __forceinline__ void dft2(Cx<R>& a, Cx<R>& b) {
  const Cx<R> t = a - b;
  a = a + b;
  b = t;
}
template <typename R>
__device__ __forceinline__ void dft4(Cx<R>& a, Cx<R>& b, Cx<R>& c, Cx<R>& d) {
  dft2(a, c);
  dft2(b, d);
  d = mk<R>(d.im, -d.re);  // -i d
  dft2(a, b);
  dft2(c, d);
  const Cx<R> t = b;  // order 0, 2, 1, 3
  b = c;
  c = t;
}
template <typename R, int N>
__device__ __forceinline__ void dft(Cx<R> (&x)[N]) {
  static_assert(N <= 8 || N == 11 || N == 13, "no transform of this length");
  if constexpr (N == 3) {
    constexpr double c[] = {1.0, -0.5, -0.5};
    constexpr double s[] = {0.0, 0.8660254037844386, -0.8660254037844386};
    dft_odd<R, N>(x, c, s);
  } else if constexpr (N == 5) {
    constexpr double c[] = {1.0, 0.30901699437494745, -0.8090169943749475, -0.8090169943749475,
                              0.30901699437494745};
    constexpr double s[] = {0.0, 0.9510565162951535, 0.5877852522924731, -0.5877852522924731, -0.9510565162951535};
    dft_odd<R, N>(x, c, s);
  } else if constexpr (N == 7) {
    constexpr double c[] = {1.0, 0.6234898018587335, -0.2225209339563144, -0.9009688679024191, -0.9009688679024191,
                              -0.2225209339563144, 0.6234898018587335};
    constexpr double s[] = {0.0, 0.7818314824680298, 0.9749279121818236, 0.4338837391175581, -0.4338837391175581,
                              -0.9749279121818236, -0.7818314824680298};
    dft_odd<R, N>(x, c, s);
  } else if constexpr (N == 11) {
    constexpr double c[] = {1.0, 0.8412535328311812, 0.41541501300188644, -0.14231483827328514,
                              -0.6548607339452851, -0.9594929736144974, -0.9594929736144974, -0.6548607339452851,
                              -0.14231483827328514, 0.41541501300188644, 0.8412535328311812};
    constexpr double s[] = {0.0, 0.5406408174555976, 0.9096319953545183, 0.9898214418809327, 0.7557495743542583,
                              0.28173255684142967, -0.28173255684142967, -0.7557495743542583, -0.9898214418809327,
                              -0.9096319953545183, -0.5406408174555976};
    dft_odd<R, N>(x, c, s);
  } else if constexpr (N == 13) {
    constexpr double c[] = {1.0, 0.8854560256532099, 0.5680647467311558, 0.12053668025532305, -0.3546048870425356,
                              -0.7485107481711011, -0.970941817426052, -0.970941817426052, -0.7485107481711011,
                              -0.3546048870425356, 0.12053668025532305, 0.5680647467311558, 0.8854560256532099};
    constexpr double s[] = {0.0, 0.46472317204376856, 0.8229838658936564, 0.992708874098054, 0.9350162426854148,
                              0.6631226582407952, 0.23931566428755777, -0.23931566428755777, -0.6631226582407952,
                              -0.9350162426854148, -0.992708874098054, -0.8229838658936564, -0.46472317204376856};
    dft_odd<R, N>(x, c, s);
  } else if constexpr (N == 2) {
    dft2(x[0], x[1]);
  } else if constexpr (N == 4) {
    dft4(x[0], x[1], x[2], x[3]);
  } else if constexpr (N == 6) {  // 2 x 3, coprime: input 3 n1 + 2 n2, output 3 k1 + 4 k2
    Cx<R> e[3] = {x[0], x[2], x[4]}, o[3] = {x[3], x[5], x[1]};
    dft<R, 3>(e);
    dft<R, 3>(o);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dft2(e[k], o[k]);
      x[4 * k % 6] = e[k];
      x[(3 + 4 * k) % 6] = o[k];
    }
  } else if constexpr (N == 8) {
    dft4(x[0], x[2], x[4], x[6]);
    dft4(x[1], x[3], x[5], x[7]);
    const R q = (R)0.70710678118654752440;
    x[3] = mk<R>(q * (x[3].re + x[3].im), q * (x[3].im - x[3].re));
    x[5] = mk<R>(x[5].im, -x[5].re);
    x[7] = mk<R>(q * (x[7].im - x[7].re), -q * (x[7].re + x[7].im));
    // even outputs stand in x[0], x[2], x[4], x[6] in order, odd ones likewise
    Cx<R> y[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dft2(x[2 * k], x[2 * k + 1]);
      y[k] = x[2 * k];
      y[k + 4] = x[2 * k + 1];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = y[k];
  }
}

__host__ __device__ constexpr int gcd_of(int a, int b) { return b ? gcd_of(b, a % b) : a; }
// the inverse of a modulo m (1 if there is none)
__host__ __device__ constexpr int inverse_of(int a, int m) {
  for (int i = 1; i < m; ++i)
    if (a * i % m == 1) return i;
  return 1;
}

// the transform of a line of L = P Q in registers; element i of the result is
// the output out(i).  tw[m] = e^{-2 pi i m / L}, read where P and Q share a factor.
template <typename R, int P, int Q>
struct Line {
  static constexpr int L = P * Q;
  static constexpr bool coprime = gcd_of(P, Q) == 1;
  static constexpr int QI = Q * inverse_of(Q % P, P), PI = P * inverse_of(P % Q, Q);
  // input n1, n2 and output k1, k2 stand at
  __device__ static constexpr int in(int n1, int n2) { return coprime ? (Q * n1 + P * n2) % L : n1 + P * n2; }
  __device__ static constexpr int out(int k1, int k2) {
    return coprime ? (QI * k1 + PI * k2) % L : Q * k1 + k2;
  }
  // f(k, value) for every output
  template <typename F>
  __device__ static __forceinline__ void run(Cx<R> (&x)[L], const Cx<R>* tw, F f) {
#pragma unroll
    for (int n1 = 0; n1 < P; ++n1) {
      Cx<R> y[Q];
#pragma unroll
      for (int n2 = 0; n2 < Q; ++n2) y[n2] = x[in(n1, n2)];
      dft<R, Q>(y);
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) x[in(n1, k2)] = coprime || n1 == 0 || k2 == 0 ? y[k2] : cmul(tw[n1 * k2], y[k2]);
    }
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2) {
      Cx<R> y[P];
#pragma unroll
      for (int n1 = 0; n1 < P; ++n1) y[n1] = x[in(n1, k2)];
      dft<R, P>(y);
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) f(out(k1, k2), y[k1]);
    }
  }
};

// fields of a pair and slice: two of one correlator, or the four of all
constexpr int CORR_ONE = 2, CORR_ALL = 4;
constexpr int corr_threads(int L, int NF) { return NF * L <= 128 ? 128 : (NF * L + 31) / 32 * 32; }
// blocks that add up their sums; of eight, 33 clusters are resident at two blocks
// per SM, of four all but a few SMs are filled: L = 30, complex128, 1.68 -> 1.57 ms,
// L = 48, complex64, 1.54 -> 1.47, at the same error
constexpr int CORR_CLUSTER = 4;
// blocks per SM that leave a thread the registers of its line and fit in shared memory
constexpr int corr_blocks(int L, int words, int NF) {
  if (NF == CORR_ALL && words == 1) return L <= 32 ? 4 : L <= 36 ? 3 : 2;
  if (L * words > 72) return 1;
  return L * words <= 40 ? 4 : L * words <= 48 ? 3 : 2;
}

// NF = CORR_ALL: the sum of all four correlators, whose fields are sums of the
// same four: U_st(r) = conj(eta_s(r)) G_t(r + x) e^{i phi}, V_st(r) = conj(eta_s(r
// + x)) G_t(r) e^{-i phi}, and U_ts, V_ts.  T1 correlates U_st with U_ts, T4 V_st
// with V_ts, T21 (V_st + V_ts) / 2 with (U_st + U_ts) / 2, and T2 is T21 at -k.
// So four transforms do instead of six in three launches, one sum instead of
// three, and A(k), the transform of U_st at -k, needs no conjugation.
template <typename R, int P, int Q, int NF>
__global__ void __launch_bounds__(corr_threads(P* Q, NF), corr_blocks(P* Q, sizeof(R) / 4, NF))
    k_bb_corr(BondArgs a, int ni, double* S) {
  constexpr int L = P * Q, Vs = L * L, PITCH = L | 1;  // rows apart by an odd number of complex numbers
  using T = Line<R, P, Q>;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sum = reinterpret_cast<double2*>(smraw);   // [Vs]
  Cx<R>* F = reinterpret_cast<Cx<R>*>(sum + Vs);      // [ni][NF][L][PITCH]
  Cx<R>* tw = F + (size_t)ni * NF * L * PITCH;        // [L]
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < L; i += nt) {
    double sn, cs;
    sincospi(-2.0 * i / L, &sn, &cs);
    tw[i] = mk<R>((R)cs, (R)sn);
  }
  for (int i = tid; i < Vs; i += nt) sum[i] = make_double2(0, 0);
  __syncthreads();
  // this thread's item of the block's ni, its field (a or b, st or ts) and line
  const int it = tid / (NF * L), f = tid / L & 1, l = tid % L;
  const bool mine = it < ni;
  Cx<R>* Ff = F + (size_t)(tid / L) * L * PITCH;
  const bool two = NF == CORR_ONE && (a.kind == 21 || a.kind == 2);
  // conj(eta) at r, G at r + x, times e^{i phi}; else conj(eta) at r + x, G at r, times e^{-i phi}
  const bool up = NF == CORR_ALL ? (tid / L & 2) == 0 : a.kind == 1 || (a.kind == 21 && f) || (a.kind == 2 && !f);
  const int l1 = l + 1 == L ? 0 : l + 1;
  const R* eta = reinterpret_cast<const R*>(a.eta) + 2 * (up ? l : l1);
  const R* g = reinterpret_cast<const R*>(a.g) + 2 * (up ? l1 : l);
  const R* ep = reinterpret_cast<const R*>(a.ep) + 2 * l;
  const int64_t nsite = (int64_t)a.Nt * Vs;
  const int items = a.npairs * a.Nt;
  const int w0 = (int)((int64_t)items * blockIdx.x / gridDim.x), w1 = (int)((int64_t)items * (blockIdx.x + 1) / gridDim.x);
  for (int w = w0; w < w1; w += ni) {
    const int n = min(ni, w1 - w);
    if (mine && it < n) {
      const int tau = (w + it) / a.npairs, pr = (w + it) - tau * a.npairs;
      const int s = a.ps[pr], t = a.pt[pr];
      // a: conj(eta_s) G_t, b: conj(eta_t) G_s; T21 and T2 add the same with s and t exchanged
      const bool valid = (unsigned)s < (unsigned)a.nrv && (unsigned)t < (unsigned)a.nrv;  // not a noise vector: zero
      const int64_t sl = (int64_t)tau * Vs, ou = (f ? t : s) * nsite + sl, ov = (f ? s : t) * nsite + sl;
      Cx<R> x[L];
      if (!valid) {
#pragma unroll
        for (int y = 0; y < L; ++y) x[y] = mk<R>(0, 0);
      } else {
#pragma unroll
        for (int y = 0; y < L; ++y) {
          Cx<R> v = cmul(conjc(ldcx(eta, ou + y * L)), ldcx(g, ov + y * L));
          if (two) v = (R)0.5 * (v + cmul(conjc(ldcx(eta, ov + y * L)), ldcx(g, ou + y * L)));
          Cx<R> e = ldcx(ep, sl + y * L);
          if (!up) e = conjc(e);
          v = cmul(v, e);
          x[y] = f || NF == CORR_ALL ? v : conjc(v);
        }
      }
      T::run(x, tw, [&](int k, Cx<R> v) { Ff[k * PITCH + l] = v; });
    }
    __syncthreads();
    if (mine && it < n) {
      Cx<R> x[L];
      Cx<R>* row = Ff + l * PITCH;
#pragma unroll
      for (int i = 0; i < L; ++i) x[i] = row[i];
      T::run(x, tw, [&](int k, Cx<R> v) { row[k] = v; });
    }
    __syncthreads();
    if constexpr (NF == CORR_ALL) {
      // k and -k together: rows up to L / 2, of the first and the last row half
      for (int k = tid; k < (L / 2 + 1) * L; k += nt) {
        const int ky = k / L, kx = k % L;
        if (ky % (L / 2) == 0 && kx > L / 2) continue;
        const int my = ky ? L - ky : 0, mx = kx ? L - kx : 0, m = my * L + mx;
        const Cx<R>*q = F + ky * PITCH + kx, *r = F + my * PITCH + mx;
        double2 c = sum[k], d = sum[m];
        auto at = [](const Cx<R>* u, int j) {
          const Cx<R> v = u[j * L * PITCH];
          return make_double2(v.re, v.im);
        };
        auto add = [](double2& s, double2 u, double2 v) {
          s.x = fma(u.x, v.x, fma(-u.y, v.y, s.x));
          s.y = fma(u.x, v.y, fma(u.y, v.x, s.y));
        };
        for (int i = 0; i < n; ++i, q += NF * L * PITCH, r += NF * L * PITCH) {
          double2 u = at(q, 0), w = at(q, 1), um = at(r, 0), wm = at(r, 1);  // U_st, U_ts at k and -k
          add(c, um, w);
          add(d, u, wm);
          const double2 U = make_double2(u.x + w.x, u.y + w.y), Um = make_double2(um.x + wm.x, um.y + wm.y);
          u = at(q, 2), w = at(q, 3), um = at(r, 2), wm = at(r, 3);  // V_st, V_ts
          add(c, um, w);
          add(d, u, wm);
          double2 e = make_double2(0, 0);
          add(e, make_double2(um.x + wm.x, um.y + wm.y), U);
          add(e, make_double2(u.x + w.x, u.y + w.y), Um);
          c = make_double2(fma(0.25, e.x, c.x), fma(0.25, e.y, c.y));
          d = make_double2(fma(0.25, e.x, d.x), fma(0.25, e.y, d.y));
        }
        sum[k] = c;
        if (m != k) sum[m] = d;
      }
    } else {
      for (int k = tid; k < Vs; k += nt) {
        const Cx<R>* q = F + k / L * PITCH + k % L;
        double2 c = sum[k];
        for (int i = 0; i < n; ++i, q += 2 * L * PITCH) {
          const Cx<R> u = q[0], v = q[L * PITCH];
          const double ur = u.re, ui = -u.im, vr = v.re, vi = v.im;
          c.x = fma(ur, vr, fma(-ui, vi, c.x));
          c.y = fma(ur, vi, fma(ui, vr, c.y));
        }
        sum[k] = c;
      }
    }
    __syncthreads();
  }
  // the cluster's sums in a tree, then one addition to S per cluster: one per
  // block, a chain of hundreds of roundings, was half of the result's error
  auto cluster = cooperative_groups::this_cluster();
  cluster.sync();
  for (int k = tid + nt * (int)cluster.block_rank(); k < Vs; k += nt * CORR_CLUSTER) {
    double2 c[CORR_CLUSTER];
#pragma unroll
    for (int j = 0; j < CORR_CLUSTER; ++j) c[j] = cluster.map_shared_rank(sum, j)[k];
#pragma unroll
    for (int h = 1; h < CORR_CLUSTER; h *= 2)
#pragma unroll
      for (int j = 0; j < CORR_CLUSTER; j += 2 * h) c[j] = make_double2(c[j].x + c[j + h].x, c[j].y + c[j + h].y);
    atomicAdd(S + 2 * k, c[0].x);
    atomicAdd(S + 2 * k + 1, c[0].y);
  }
  cluster.sync();  // no block's shared memory goes while another reads it
}

template <typename R, int NF, int P, int Q>
static int launch_corr_pq(const BondArgs& a, double* S, cudaStream_t st) {
  constexpr int L = P * Q;
  if (a.npairs == 0) return QEDF_OK;
  const int ni = corr_threads(L, NF) / (NF * L), threads = (ni * NF * L + 31) / 32 * 32;
  const size_t smem = L * L * sizeof(double2) + ((size_t)ni * NF * L * (L | 1) + L) * sizeof(Cx<R>);
  if (cudaFuncSetAttribute(k_bb_corr<R, P, Q, NF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return QEDF_ERR_CUDA;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = CORR_CLUSTER;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = CORR_CLUSTER;
  cfg.blockDim = threads;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int clusters = 0;  // that are resident at a time
  if (cudaOccupancyMaxActiveClusters(&clusters, k_bb_corr<R, P, Q, NF>, &cfg) != cudaSuccess || clusters < 1)
    return QEDF_ERR_SIZE;
  const int64_t per = (int64_t)ni * CORR_CLUSTER, want = ((int64_t)a.npairs * a.Nt + per - 1) / per;
  cfg.gridDim = CORR_CLUSTER * (unsigned)std::min<int64_t>(want, clusters);
  if (cudaLaunchKernelEx(&cfg, k_bb_corr<R, P, Q, NF>, a, ni, S) != cudaSuccess) return QEDF_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}

// even sides (the sum of all takes k and -k together) whose factors have transforms and whose lines fit in registers
template <typename R, int NF>
static int launch_corr(const BondArgs& a, double* S, cudaStream_t st) {
  switch (a.L) {
    case 4: return launch_corr_pq<R, NF, 1, 4>(a, S, st);
    case 6: return launch_corr_pq<R, NF, 2, 3>(a, S, st);
    case 8: return launch_corr_pq<R, NF, 1, 8>(a, S, st);
    case 10: return launch_corr_pq<R, NF, 2, 5>(a, S, st);
    case 12: return launch_corr_pq<R, NF, 3, 4>(a, S, st);
    case 14: return launch_corr_pq<R, NF, 2, 7>(a, S, st);
    case 16: return launch_corr_pq<R, NF, 4, 4>(a, S, st);
    case 18: return launch_corr_pq<R, NF, 3, 6>(a, S, st);
    case 20: return launch_corr_pq<R, NF, 4, 5>(a, S, st);
    case 22: return launch_corr_pq<R, NF, 2, 11>(a, S, st);
    case 24: return launch_corr_pq<R, NF, 3, 8>(a, S, st);
    case 26: return launch_corr_pq<R, NF, 2, 13>(a, S, st);
    case 28: return launch_corr_pq<R, NF, 4, 7>(a, S, st);
    case 30: return launch_corr_pq<R, NF, 5, 6>(a, S, st);
    case 32: return launch_corr_pq<R, NF, 4, 8>(a, S, st);
  }
  if constexpr (NF == CORR_ALL && sizeof(R) == 8) {
    switch (a.L) {
      case 36: return launch_corr_pq<R, NF, 6, 6>(a, S, st);
      case 40: return launch_corr_pq<R, NF, 5, 8>(a, S, st);
    }
  }
  if constexpr (sizeof(R) == 4) {
    switch (a.L) {
      case 36: return launch_corr_pq<R, NF, 6, 6>(a, S, st);
      case 40: return launch_corr_pq<R, NF, 5, 8>(a, S, st);
      case 42: return launch_corr_pq<R, NF, 6, 7>(a, S, st);
      case 48: return launch_corr_pq<R, NF, 6, 8>(a, S, st);
    }
  }
  return QEDF_ERR_SIZE;
}

// kind 0: the sum of all four
template <typename R>
static int corr_entry(int kind, const R* eta, const R* g, const R* ep, const int* ps, const int* pt, int npairs,
                      int Nrv, int Lx, int Ltau, double* S, cudaStream_t st) {
  if (kind != 0 && kind != 1 && kind != 21 && kind != 2 && kind != 4) return QEDF_ERR_ARG;
  if (!eta || !g || !ep || !ps || !pt || !S) return QEDF_ERR_ARG;
  if (npairs < 0 || Lx < 2 || Ltau < 1 || Nrv < 2) return QEDF_ERR_ARG;
  BondArgs a;
  a.kind = kind;
  a.eta = eta;
  a.g = g;
  a.ep = ep;
  a.ps = ps;
  a.pt = pt;
  a.npairs = npairs;
  a.nrv = Nrv;
  a.L = Lx;
  a.Nt = Ltau;
  a.fa = nullptr;
  a.fb = nullptr;
  // (the line kernels count items in 32 bits)
  const bool lines = (int64_t)npairs * Ltau <= INT32_MAX - 256;
  if (kind == 0) return lines ? launch_corr<R, CORR_ALL>(a, S, st) : QEDF_ERR_SIZE;
  const int e = lines ? launch_corr<R, CORR_ONE>(a, S, st) : QEDF_ERR_SIZE;
  return e == QEDF_ERR_SIZE ? launch_corr_any<R>(a, S, st) : e;
}

}  // namespace qedf
