// Persistent batched preconditioned CG on M^dag M x = b: planning and launch
// (the kernel is qedf_pcg_kernel.cuh, instantiated by one unit per mode).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "qedf_internal.h"
#include "qedf_pcg_kernel.cuh"
#include "qedf_precon_table.h"

namespace qedf {

__constant__ PreTable c_pre = {QEDF_PRE_LAYOUT, QEDF_PRE_EDGE_VALUES, QEDF_PRE_TAIL_VALUES,
                               QEDF_PRE_MIDDLE_VALUES, QEDF_PRE_CORNER_VALUES};
static const PreTable h_pre = {QEDF_PRE_LAYOUT, QEDF_PRE_EDGE_VALUES, QEDF_PRE_TAIL_VALUES,
                               QEDF_PRE_MIDDLE_VALUES, QEDF_PRE_CORNER_VALUES};

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

int pcg_storage_bytes(int mode) { return mode == QEDF_PCG_PLAIN_F64 ? 8 : 4; }
static bool mode_mixed(int mode) {
  return mode == QEDF_PCG_MIXED || mode == QEDF_PCG_MIXED_BF16 || mode == QEDF_PCG_MIXED_F16;
}
static bool mode_narrow(int mode) { return mode == QEDF_PCG_MIXED_BF16 || mode == QEDF_PCG_MIXED_F16; }

// slices of side L that an SM holds, by the warps that the kernels' registers allow
static int resident_slices(int L, int by) {
  return std::min(PCG_MAX_PER_SM, (by == 2 ? 20 : 16) / std::max(4, slice_threads(L, by) / 32));
}

// Tau segments of the elementwise units: whole tau columns (one segment) where
// these fill the GPU, else as many segments as shorten the busiest block's
// work, counted in rows with twelve rows of the neighbours and about forty
// rows' worth of latency per unit.  At L = 10, Ltau = 100, 2 right-hand sides
// there are 14 columns for 148 SMs.  Split solves keep a second buffer of r,
// so only those whose vectors are small (9 MB) are split.
static int auto_segments(int64_t columns, int Nt, int blocks) {
  int best = 1;
  int64_t best_cost = -1;
  for (int n = 1; n <= Nt / 12; ++n) {
    const int len = (Nt + n - 1) / n;
    const int64_t cost = (columns * n + blocks - 1) / blocks * (len + (n > 1 ? 12 : 0) + 40);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = n;
    }
  }
  return best;
}

// The tile height where none is asked for; it must divide every system's L.
// 2 x 2 tiles unless they leave an SM a single one of the largest slices and 2
// x 4 ones more (by the warps that the kernels' 96 and 128 registers allow, up
// to PCG_MAX_PER_SM).  Then a block's run of n slices takes 2 n + 1 B's, half
// as many of them with two blocks per SM, each about 1.5 times as long: 2 x 2
// where runs are so short that rounding n up and the halo eat the difference.
// 2 x 6 tiles only where neither divides L.  us per iteration with 2 x 2 and 2 x
// 4 tiles, mixed: L = 36, 64 right-hand sides, 741 and 614; L = 44, 5 at Ltau =
// 308, 77 and 71; L = 44, 1 at Ltau = 440, 25.8 and 27.8 (double 63 and 86); L =
// 48, 2, 47 and 51.  With two 2 x 2 slices per SM: L = 28, 2, 17.0 and 21.3; L =
// 28, 6, 31.6 and 38.2 (double 85 and 108); L = 32, 4, 29.9 and 36.0; L = 28, 48,
// 194 and 191.
static int pcg_pick_by(const PcgParams& p) {
  int first = -1, Lmax = 0;
  bool ok[7] = {};
  int64_t slices = 0;
  for (int s = 0; s < p.nsys; ++s) {
    Lmax = std::max(Lmax, p.sys[s].L);
    slices += (int64_t)p.sys[s].nrhs * p.sys[s].Nt;
  }
  for (int by : {6, 4, 2}) {
    ok[by] = true;
    for (int s = 0; s < p.nsys; ++s) ok[by] = ok[by] && by_valid(p.sys[s].L, by);
    if (ok[by]) first = by;
  }
  if (first != 2 || !ok[4] || resident_slices(Lmax, 2) > 1 || resident_slices(Lmax, 4) < 2) return first;
  const int64_t sms = num_sms(), n2 = (slices + sms - 1) / sms, n4 = (slices + 2 * sms - 1) / (2 * sms);
  return 3 * (2 * n4 + 1) <= 2 * (2 * n2 + 1) ? 4 : 2;
}

// 32-site elementwise units instead of 16-site ones, where none are asked for:
// one block per SM (a wide unit's column is up to 169 KB of shared memory), two
// rounds of narrow units and one of wide ones, whose rows are then all in flight
// at once.  Single precision, us per iteration, 16 and 32 sites: L = 48, 2
// right-hand sides, 53.0 and 50.8; L = 60, 1: 42.0 and 39.7; L = 66, 1: 85.7 and 81.6.
// Three rounds against two lose (L = 52, 2: 57.6 and 59.4), and so does a wide
// column where it takes a second block's place or L1 (L = 40, 3: 52.4 and 56.9).
static bool wide_units(const PcgParams& p, int by, int64_t narrow, int64_t wide, int Ltau, int rhs) {
  int Lmax = 0;
  for (int s = 0; s < p.nsys; ++s) Lmax = std::max(Lmax, p.sys[s].L);
  if (by <= 0) by = pcg_pick_by(p);
  return by > 0 && resident_slices(Lmax, by) == 1 && narrow > num_sms() && wide <= num_sms() &&
         (size_t)Ltau * 2 * PCG_CHUNK * 8 + RhsState<true, true>::bytes(rhs) <= 200 * 1024;
}

int pcg_plan(PcgParams& p, const qedf_system* sys, int nsys, const qedf_pcg_opts* o) {
  std::memset(&p, 0, sizeof(p));
  if (!sys || !o || nsys <= 0 || nsys > PCG_MAX_SYS) return QEDF_ERR_ARG;
  if (o->mode != QEDF_PCG_PLAIN_F32 && o->mode != QEDF_PCG_PLAIN_F64 && !mode_mixed(o->mode)) return QEDF_ERR_ARG;
  p.mode = o->mode;
  p.nsys = nsys;
  p.x_init = o->x_init > 0 ? 1 : 0;
  p.l2 = o->l2_persist < 0 ? -1 : 0;
  if (o->chunk != 0 && o->chunk != 16 && o->chunk != 32) return QEDF_ERR_ARG;
  // 32-site elementwise units: twice the shared memory per unit
  int ntmax_all = 0;
  for (int s = 0; s < nsys; ++s) ntmax_all = std::max(ntmax_all, sys[s].Ltau);
  const bool wide_fits = o->mode != QEDF_PCG_PLAIN_F64 && ntmax_all <= 500;
  if (o->chunk == 32 && !wide_fits) return QEDF_ERR_SIZE;
  p.CH = o->chunk ? o->chunk : PCG_CHUNK;
  int Lmax = 0;
  int64_t columns = 0, wide = 0, elements = 0, slices = 0, all_rhs = 0;
  for (int s = 0; s < nsys; ++s) {
    const qedf_system& q = sys[s];
    if (q.Lx < 2 || q.Lx % 2 || q.Ltau < 2 || q.nrhs < 1) return QEDF_ERR_ARG;
    columns += (int64_t)q.nrhs * (((int64_t)q.Lx * q.Lx + p.CH - 1) / p.CH);
    wide += (int64_t)q.nrhs * (((int64_t)q.Lx * q.Lx + 2 * PCG_CHUNK - 1) / (2 * PCG_CHUNK));
    all_rhs += q.nrhs;
    p.sys[s].L = q.Lx;
    p.sys[s].Nt = q.Ltau;
    p.sys[s].nrhs = q.nrhs;
    elements += (int64_t)q.nrhs * q.Ltau * q.Lx * q.Lx;
    Lmax = std::max(Lmax, q.Lx);
    slices += (int64_t)q.nrhs * q.Ltau;
  }
  const bool may_split = elements * 2 * pcg_storage_bytes(o->mode) <= 9000000;
  if (!o->chunk && o->mode != QEDF_PCG_PLAIN_F64 && !may_split &&
      wide_units(p, o->by, columns, wide, ntmax_all, (int)all_rhs)) {
    p.CH = 2 * PCG_CHUNK;
    columns = wide;
  }
  // blocks that take them: two per SM, or as many as the operator's slices bring
  // and fit (double precision, whose units take twice as long: L = 20, 3
  // right-hand sides, 36.9 -> 33.2 us per iteration; L = 24, 2: 35.2 -> 33.2)
  const int64_t seg_most = (int64_t)num_sms() * std::max(2, resident_slices(Lmax, 2));
  const int seg_blocks = (int)std::min(std::max<int64_t>(slices, 2 * num_sms()), seg_most);
  int rhs = 0, pt = 0;
  int64_t vec = 0, phi = 0;
  for (int s = 0; s < nsys; ++s) {
    const qedf_system& q = sys[s];
    PcgSys& S = p.sys[s];
    S.L = q.Lx;
    S.Nt = q.Ltau;
    S.nrhs = q.nrhs;
    S.shared = q.shared_boson ? 1 : 0;
    S.precon = (o->use_precon && q.Ltau >= PRE_MIN_LTAU) ? 1 : 0;
    S.T = o->slab > 0 ? std::min(o->slab, q.Ltau) : 1;
    // the preconditioner rows that are the bulk band (middle values at every
    // distance, nothing else): one contiguous range away from both tau ends
    S.pmid_lo = S.pmid_hi = 0;
    if (S.precon) {
      int lo = -1, hi = -1;
      for (int t = 0; t < q.Ltau; ++t) {
        bool mid = t >= 6 && t + 6 < q.Ltau;
        int cnt = 0;
        pre_row(h_pre, q.Ltau, t, [&](int c, float val) {
          const int d = c > t ? c - t : t - c;
          mid = mid && d <= 6 && val == h_pre.middle[d];
          ++cnt;
        });
        mid = mid && cnt == 13;
        if (mid && lo < 0) lo = t;
        if (mid) hi = t + 1;
      }
      if (lo >= 0) {
        S.pmid_lo = lo;
        S.pmid_hi = hi;
      }
    }
    S.nslab = (q.Ltau + S.T - 1) / S.T;
    S.nchunk = (q.Lx * q.Lx + p.CH - 1) / p.CH;
    S.nseg = may_split ? auto_segments(columns, q.Ltau, seg_blocks) : 1;
    S.seg = (q.Ltau + S.nseg - 1) / S.nseg;
    S.nseg = (q.Ltau + S.seg - 1) / S.seg;
    if (S.nseg > 1) p.split = 1;
    S.rhs0 = rhs;
    S.vec0 = vec;
    S.phi0 = phi;
    S.ptab0 = pt;
    pt += 13 * q.Ltau;
    rhs += q.nrhs;
    vec += (int64_t)q.nrhs * q.Ltau * q.Lx * q.Lx;
    phi += (int64_t)(S.shared ? 1 : q.nrhs) * q.Ltau * q.Lx * q.Lx * 2;
    if (rhs > PCG_MAX_RHS) return QEDF_ERR_SIZE;
  }
  p.nrhs = rhs;
  p.nvec_total = vec;
  p.ptab_len = pt;
  p.max_iter = o->max_iter;
  p.rtol = o->rtol;
  // defaults measured on the benchmark solve: every 100 iterations or a
  // hundredfold residual drop take the iteration count of 50 / tenfold with
  // half the reliable-update time
  p.ru_interval = o->ru_interval > 0 ? o->ru_interval : 100;
  p.ru_delta = o->ru_delta > 0 ? o->ru_delta : 0.01;
  const FactorCoeffs f = factor_coeffs(o->dtau);
  p.c1 = f.c1;
  p.ch = f.ch;
  p.t1 = f.t1;
  p.th = f.th;
  p.Cb = f.Cb;
  // largest absolute row sum of the systems' preconditioners (a bound of its
  // 2-norm, P being symmetric); 1 for the identity
  p.pnorm = 1.0;
  for (int s = 0; s < nsys; ++s) {
    if (!p.sys[s].precon) continue;
    for (int t = 0; t < p.sys[s].Nt; ++t) {
      double row = 0;
      pre_row(h_pre, p.sys[s].Nt, t, [&](int, float val) { row += std::fabs((double)val); });
      p.pnorm = std::max(p.pnorm, row);
    }
  }
  return QEDF_OK;
}

// The workspace layout, in one place: r (twice where units are tau segments),
// p0, p1, z, Op and, in the mixed modes, x_lo, in the sloppy precision; p and z
// in half of it with narrow storage, which then has a buffer of its own for
// half of the reliable updates' M x (float storage uses z); the double
// accumulators, 256 bytes of grid-barrier words and the preconditioner
// tables, each 256-byte aligned.  Returns the bytes the layout needs; with a
// workspace it also points p's buffers into it, and *zero_bytes receives the
// length of the block that starts at zero every solve (accumulators and
// barrier words, contiguous from p.acc).
size_t pcg_carve(PcgParams& p, int sloppy_bytes, void* workspace, size_t* zero_bytes) {
  const size_t full = align_up((size_t)p.nvec_total * 2 * sloppy_bytes, 256);
  const size_t narrow = mode_narrow(p.mode) ? align_up((size_t)p.nvec_total * 4, 256) : full;
  const size_t accb = align_up(sizeof(double) * PCG_ACC_PER_RHS * p.nrhs, 256);
  const size_t barb = 256;
  const size_t tabb = align_up(sizeof(float) * (size_t)p.ptab_len, 256);
  if (zero_bytes) *zero_bytes = accb + barb;
  unsigned char* w = static_cast<unsigned char*>(workspace);
  size_t at = 0;
  auto take = [&](size_t n) -> void* {
    void* q = w ? w + at : nullptr;
    at += n;
    return q;
  };
  p.r = take(full);
  p.r2 = p.split ? take(full) : nullptr;
  p.p0 = take(narrow);
  p.p1 = take(narrow);
  p.z = take(narrow);
  p.Op = take(full);
  p.xlo = mode_mixed(p.mode) ? take(full) : nullptr;
  p.y0 = mode_narrow(p.mode) ? take(full) : mode_mixed(p.mode) ? p.z : nullptr;
  p.acc = static_cast<double*>(take(accb));
  p.bar = static_cast<unsigned long long*>(take(barb));
  p.ptab = static_cast<float*>(take(tabb));
  return at;
}

size_t pcg_workspace_bytes(const PcgParams& p, int sloppy_bytes) {
  PcgParams q = p;
  return pcg_carve(q, sloppy_bytes, nullptr, nullptr);
}

// Per solve: zero the accumulators and barrier words, and write each system's
// periodic 13-band preconditioner table (entry k of row t multiplies r at
// tau = t + k - 6 mod Nt).
__global__ void k_pcg_prep(const __grid_constant__ PcgParams p, int zero_words) {
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned int* z = reinterpret_cast<unsigned int*>(p.acc);
  for (int i = i0; i < zero_words; i += gridDim.x * blockDim.x) z[i] = 0u;
  for (int s = 0; s < p.nsys; ++s) {
    const int Nt = p.sys[s].Nt;
    float* tab = p.ptab + p.sys[s].ptab0;
    for (int e = i0; e < 13 * Nt; e += gridDim.x * blockDim.x) tab[e] = 0.f;
  }
  __syncthreads();
  // rows are independent; each thread fills whole rows (duplicate-free)
  for (int s = 0; s < p.nsys; ++s) {
    const int Nt = p.sys[s].Nt;
    if (!p.sys[s].precon) continue;
    float* tab = p.ptab + p.sys[s].ptab0;
    for (int t = i0; t < Nt; t += gridDim.x * blockDim.x)
      pre_row(c_pre, Nt, t, [&](int col, float val) {
        int k = col - t + 6;
        if (k < 0) k += Nt;
        if (k >= Nt) k -= Nt;
        tab[t * 13 + k] += val;
      });
  }
}

// L2 persistence for the iteration vectors.  p_old / p_new (p0, p1), z and
// M^dag M p (Op) are contiguous in the workspace; each is written in one phase
// and read in the next.  The launch carries an access-policy window over the
// four (z and Op alone when four exceed the largest window) whose hit ratio
// fits them to the context's persisting set-aside as it is: the limit is
// never changed, since a larger set-aside takes L2 from every other kernel of
// the process (measured: a solve without the window went from 30.8 to 41 ms
// after the limit was raised to 75 MB).  With the B200 default set-aside
// (about 25 MB) the bench solve takes about 4 % less time.  Errors of these
// queries only turn the window off.
// After the solve the window's lines would stay persisting and crowd every
// later kernel (another solver's workspace included) out of the set-aside.
// This kernel reads each 128-byte line of the window once under a window with
// the normal hit property, which returns the lines to normal status.
__global__ void k_l2_release(const uint4* base, size_t n16) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i * 8 < n16; i += (size_t)gridDim.x * blockDim.x) {
    unsigned int a, b, c, d;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
                 : "l"(base + i * 8));
  }
}

static bool pcg_l2_window(const PcgParams& p, cudaLaunchAttribute& at) {
  if (p.l2 < 0) return false;
  int dev = 0, maxw = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&maxw, cudaDevAttrMaxAccessPolicyWindowSize, dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const size_t maxwin = (size_t)std::max(maxw, 0);
  const char* end = static_cast<const char*>(p.Op) + align_up((size_t)p.nvec_total * 2 * pcg_storage_bytes(p.mode), 256);
  void* base = p.p0;
  size_t bytes = (size_t)(end - static_cast<const char*>(p.p0));  // p0, p1, z, Op
  if (bytes > maxwin) {
    base = p.z;
    bytes = (size_t)(end - static_cast<const char*>(p.z));  // z, Op
  }
  if (bytes == 0 || bytes > maxwin) return false;
  size_t cur = 0;  // the context's persisting set-aside, used as it is
  if (cudaDeviceGetLimit(&cur, cudaLimitPersistingL2CacheSize) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (cur == 0) return false;
  at.id = cudaLaunchAttributeAccessPolicyWindow;
  at.val.accessPolicyWindow.base_ptr = base;
  at.val.accessPolicyWindow.num_bytes = bytes;
  at.val.accessPolicyWindow.hitRatio = std::min(1.0f, (float)((double)cur / (double)bytes));
  at.val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
  at.val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
  return true;
}

int pcg_launch_kernel(const void* kern, const PcgParams& p, const BandTaps& taps, int threads, size_t smem, int nblk,
                      cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nblk);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const bool window = pcg_l2_window(p, attr[1]);
  if (window) cfg.numAttrs = 2;
  void* args[2] = {const_cast<PcgParams*>(&p), const_cast<BandTaps*>(&taps)};
  if (cudaLaunchKernelExC(&cfg, kern, args) != cudaSuccess) return QEDF_ERR_CUDA;
  if (p.l2 >= 0) {
    // one launch whenever the option is on (an empty one without a window)
    cudaLaunchConfig_t rc = {};
    rc.gridDim = dim3(window ? num_sms() * 4 : 1);
    rc.blockDim = dim3(256);
    rc.stream = st;
    cudaLaunchAttribute ra[1];
    size_t n16 = 0;
    const uint4* base = nullptr;
    if (window) {
      ra[0] = attr[1];
      ra[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyNormal;
      ra[0].val.accessPolicyWindow.missProp = cudaAccessPropertyNormal;
      rc.attrs = ra;
      rc.numAttrs = 1;
      base = static_cast<const uint4*>(attr[1].val.accessPolicyWindow.base_ptr);
      n16 = attr[1].val.accessPolicyWindow.num_bytes / 16;
    }
    if (cudaLaunchKernelEx(&rc, k_l2_release, base, n16) != cudaSuccess) return QEDF_ERR_CUDA;
  }
  return QEDF_OK;
}

int launch_pcg_prep(const PcgParams& p, int zero_words, cudaStream_t st) {
  k_pcg_prep<<<1, 256, 0, st>>>(p, zero_words);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}

int launch_pcg(PcgParams& p, int by, cudaStream_t st) {
  if (by <= 0) by = pcg_pick_by(p);
  if (by < 0) return QEDF_ERR_SIZE;
  BandTaps taps;
  for (int d = 0; d < 7; ++d) taps.c[d] = h_pre.middle[d];
  switch (p.mode) {
    case QEDF_PCG_PLAIN_F32: return launch_pcg_f32(p, taps, by, st);
    case QEDF_PCG_PLAIN_F64: return launch_pcg_f64(p, taps, by, st);
    case QEDF_PCG_MIXED: return launch_pcg_mixed(p, taps, by, st);
    case QEDF_PCG_MIXED_BF16: return launch_pcg_bf16(p, taps, by, st);
    case QEDF_PCG_MIXED_F16: return launch_pcg_f16(p, taps, by, st);
  }
  return QEDF_ERR_ARG;
}

}  // namespace qedf

extern "C" int qedf_precon_tau_csr(int Ltau, int* row_ptr, int* col, double* val, int* nnz) {
  using namespace qedf;
  if (Ltau < PRE_MIN_LTAU || !row_ptr || !nnz) return QEDF_ERR_ARG;
  int k = 0;
  for (int t = 0; t < Ltau; ++t) {
    row_ptr[t] = k;
    // collect and sort the row by column
    int cols[32];
    double vals[32];
    int n = 0;
    pre_row(h_pre, Ltau, t, [&](int c, float v) {
      cols[n] = c;
      vals[n] = (double)v;
      ++n;
    });
    for (int i = 1; i < n; ++i)
      for (int j = i; j > 0 && cols[j - 1] > cols[j]; --j) {
        std::swap(cols[j - 1], cols[j]);
        std::swap(vals[j - 1], vals[j]);
      }
    for (int i = 0; i < n; ++i, ++k)
      if (col && val) {
        col[k] = cols[i];
        val[k] = vals[i];
      }
  }
  row_ptr[Ltau] = k;
  *nnz = k;
  return QEDF_OK;
}
