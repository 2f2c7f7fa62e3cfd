// Persistent batched preconditioned CG on M^dag M x = b: the kernel.
//
// One cooperative launch runs the whole solve.  Each iteration is two
// grid-wide phases separated by grid barriers:
//
//   A  (runs of tau-slices of the active right-hand sides)
//        x    += alpha_old p_old          (the previous iteration's update,
//                                          on the run's own slices)
//        p_new = z + beta p_old          (halo slices recomputed, not exchanged)
//        Op    = M^dag M p_new            (slice engine, registers + smem)
//        pAp  += Re p_new^dag Op          (double)
//   BC (elementwise units: one right-hand side x a chunk of sites x a tau segment)
//        r -= alpha Op
//        z  = (P_tau (x) I) r             (the unit's r column stays in smem)
//        rr += |r|^2,  rz += Re r^dag z   (double)
//
// The last iteration's x update is applied by a reliable update's fold or at
// the end of the solve.
//
// This is the arithmetic of preconditioned_cg_fast_test
// (hmc_sampler_batch.py:751-846) with the reference's per-iteration torch
// kernels (einsum dots, axpys, _C.mhm_vec, _C.precon_vec) fused.  Every
// right-hand side has its own mask: once ||r||/||b|| <= rtol it stops
// updating (the reference's active_bs, :826).
//
// Mixed mode iterates in float and keeps x and b in double: x_lo (float)
// accumulates the update, and a reliable update folds it into x (double),
// recomputes the true residual r = b - A x with the double-precision engine
// and restarts r from it.  It runs every ru_interval iterations, when the
// iterated residual fell by ru_delta since the last one, and whenever the
// iterated residual claims convergence, so convergence is always decided on
// the true residual.
//
// Work.  The slices of the active right-hand sides form one line, cut into one
// contiguous run per block, and so do the elementwise units; the lines are laid
// anew whenever a right-hand side converges.  As many blocks share an SM as
// registers and shared memory allow, up to PCG_MAX_PER_SM: one block's barriers,
// loads and exchanges then overlap the others' arithmetic.
//
// Per-right-hand-side scalars (alpha, beta, masks) are recomputed by every
// thread block from the same double accumulators in the same order, so all
// blocks take identical decisions without another barrier.  Grid barriers
// spin with a clock budget; when it runs out the block raises an error flag
// that ends every block's loop, and the solve reports QEDF_ERR_TIMEOUT.
#pragma once

#include <algorithm>
#include <type_traits>

#include "qedf_barrier_word.h"
#include "qedf_internal.h"
#include "qedf_slice.cuh"

namespace qedf {

// ---------------------------------------------------------------------------
// bounded grid barrier
// ---------------------------------------------------------------------------
// *bar counts arrivals over the whole solve (zeroed per solve; qedf_barrier_word.h);
// barrier n of a block is passed once the count reaches n * nblocks.  Arrival is
// a release reduction without a reply, and waiting an acquire load of the
// count, so the last block's arrival ends the barrier directly (release and
// acquire at GPU scope, ordered after and before the block barriers, need no
// further fences).  The error code is in the same word: read apart, it doubled the
// time between two looks at the count and followed the last of them.  `target` is
// the calling block's count to wait for, kept by its thread 0 across calls.
__device__ __forceinline__ bool grid_barrier(unsigned long long* bar, unsigned int nblocks, long long budget,
                                             unsigned int& target) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    target += nblocks;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;\n" ::"l"(bar), "l"(1ull) : "memory");
    const long long t0 = clock64();
    while (true) {
      unsigned long long w;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(w) : "l"(bar) : "memory");
      ok = bar_error(w) == 0;
      if (!ok || bar_reached(w, target)) break;
      if (clock64() - t0 > budget) {
        atomicOr(bar, bar_error_bits(QEDF_ERR_TIMEOUT));
        ok = 0;
        break;
      }
    }
  }
  return __syncthreads_and(ok);
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sums over the block, results valid in thread 0 (sh: 32 doubles each)
__device__ __forceinline__ void block_sum_d(double& a, double* sh) {
  a = warp_sum_d(a);
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  __syncthreads();
  if (ln == 0) sh[w] = a;
  __syncthreads();
  if (threadIdx.x < 32) a = warp_sum_d(threadIdx.x < (blockDim.x + 31) / 32 ? sh[threadIdx.x] : 0.0);
}
__device__ __forceinline__ void block_sum2_d(double& a, double& b, double* sh) {
  a = warp_sum_d(a);
  b = warp_sum_d(b);
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  __syncthreads();
  if (ln == 0) {
    sh[w] = a;
    sh[32 + w] = b;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const bool in = threadIdx.x < (blockDim.x + 31) / 32;
    a = warp_sum_d(in ? sh[threadIdx.x] : 0.0);
    b = warp_sum_d(in ? sh[32 + threadIdx.x] : 0.0);
  }
}
// ---------------------------------------------------------------------------
// accumulator layout (doubles)
// ---------------------------------------------------------------------------
struct Acc {
  double* a;
  int NV;
  __device__ __forceinline__ double* bb() const { return a; }                         // [NV]
  __device__ __forceinline__ double* pAp(int k) const { return a + (1 + k) * NV; }    // [2][NV]
  __device__ __forceinline__ double* rr(int k) const { return a + (3 + k) * NV; }     // [2][NV]
  __device__ __forceinline__ double* rz(int k) const { return a + (5 + k) * NV; }     // [2][NV]
  __device__ __forceinline__ double* ru_rr() const { return a + 7 * NV; }             // [NV]
  __device__ __forceinline__ double* ru_rz() const { return a + 8 * NV; }             // [NV]
  // [2][NV] |p|^2 of the operator phase (scaled fp16 storage)
  __device__ __forceinline__ double* pp(int k) const { return a + (9 + k) * NV; }
};

// Per-block state of the right-hand sides (identical in all blocks), carved
// from the front of dynamic shared memory: its size follows their number, so
// that small solves keep room for more blocks per SM, and the mode, whose own
// arrays (resmax, lastru and ru: reliable updates; scz and scp: scaled fp16) come
// last: 71, 84 or 96 bytes each.  With all of them, 256 right-hand sides and
// the longest tau column of double precision would not fit together.
template <bool MIXED, bool H16>
struct RhsState {
  static constexpr int ND = 6 + MIXED, NI = 5 + MIXED + 3 * H16, NC = 3 + MIXED;  // doubles, ints, bytes each
  unsigned char* sm;
  int NV;
  __host__ __device__ static size_t bytes(int NV) {
    return ((size_t)NV * (8 * ND + 4 * NI + NC) + 2 * 4 + 127) / 128 * 128;
  }
  __device__ __forceinline__ double* d(int k) const { return reinterpret_cast<double*>(sm) + k * NV; }
  __device__ __forceinline__ int* i(int k) const { return reinterpret_cast<int*>(d(ND)) + k * NV; }
  __device__ __forceinline__ unsigned char* c(int k) const {
    return reinterpret_cast<unsigned char*>(i(NI) + 2) + k * NV;
  }
  __device__ __forceinline__ double* alpha() const { return d(0); }
  __device__ __forceinline__ double* beta() const { return d(1); }
  __device__ __forceinline__ double* rz() const { return d(2); }
  __device__ __forceinline__ double* rzold() const { return d(3); }
  __device__ __forceinline__ double* rr() const { return d(4); }
  __device__ __forceinline__ double* res() const { return d(5); }
  __device__ __forceinline__ double* resmax() const {
    static_assert(MIXED);
    return d(6);
  }
  __device__ __forceinline__ int* iters() const { return i(0); }
  __device__ __forceinline__ int* status() const { return i(1); }
  __device__ __forceinline__ int* list() const { return i(2); }  // a work line's right-hand sides,
  __device__ __forceinline__ int* pre_a() const { return i(3); }  // [NV + 1] prefix sums of their operator units
  __device__ __forceinline__ int* pre_e() const { return i(4) + 1; }  // [NV + 1] and of their elementwise units
  __device__ __forceinline__ int* lastru() const {
    static_assert(MIXED);
    return i(5) + 2;
  }
  // storage scales of z and the two p buffers (scaled fp16)
  __device__ __forceinline__ float* scz() const {
    static_assert(H16);
    return reinterpret_cast<float*>(i(5 + MIXED) + 2);
  }
  __device__ __forceinline__ float* scp(int par) const {
    static_assert(H16);
    return reinterpret_cast<float*>(i(6 + MIXED + par) + 2);
  }
  __device__ __forceinline__ unsigned char* active() const { return c(0); }
  __device__ __forceinline__ unsigned char* pending() const { return c(1); }
  __device__ __forceinline__ unsigned char* sys() const { return c(2); }
  __device__ __forceinline__ unsigned char* ru() const {
    static_assert(MIXED);
    return c(3);
  }
};

// What a block keeps about the solve, in shared memory: held in registers it
// would be live across the operator phase, whose slice loop needs them all.
struct PcgCtl {
  int any_active, any_ru, changed;
  int n;              // right-hand sides of the work line
  int u0a, u1a, ka;   // this block's operator units and their first line entry
  int u0e, u1e, ke;   // the same of the elementwise units
  int it;             // iterations done
  int slot;           // accumulator slot holding the current rr / rz
  int rcur;           // buffer that holds r
  int guess;          // plain modes with an initial guess: the pass that forms r = b - A x
  int relay;          // the line of active right-hand sides has to be laid
  unsigned int target;  // grid barrier count to wait for (thread 0)
  long long t0, t;    // clocks of the phase timing (thread 0)
};

// Optional phase timing (block 0, thread 0): prof[k] accumulates clock64 cycles of
//   0 init, 1 operator phase work, 2 wait after it, 3 elementwise phase work,
//   4 wait after it, 5 reliable updates (work + waits), 6 iterations, 7 total
__device__ __forceinline__ void lap(long long* prof, PcgCtl& c, int k) {
  if (prof && blockIdx.x == 0 && threadIdx.x == 0) {
    const long long n = clock64();
    prof[k] += n - c.t;
    c.t = n;
  }
}

// the coefficients of the preconditioner's bulk band by tau distance
struct BandTaps {
  float c[7];
};

// consecutive rows of z that a thread forms at a time; rows of r and Op that it has in flight
constexpr int PCG_ZROWS = 4;
constexpr int PCG_EW_ROWS = 6;

// Engine choices of the PCG for iteration precision RS and tile height BY.
// Double-precision tall tiles as the operator's CFG_TALL: phases in the
// records, one exchange buffer, y_t in Op's own slice.  The double-precision
// engine of the mixed modes' reliable updates always keeps its phases in the
// records and has one exchange buffer; it applies one B per pass, with y = M x
// in memory between the two.
template <typename RS, int BY>
struct PcgT {
  static constexpr bool TALL = sizeof(RS) == 8 && BY >= 4;
  static constexpr bool IN_OP = sizeof(RS) == 8;  // y_t waits in Op
  // x_lo or the angles of the next slice are on their way into shared memory
  // while B is applied (loaded when needed, their latency is exposed); z and
  // p_old go to registers (operator phase at L = 48, 2 right-hand sides: 62 K
  // cycles, 70 K through shared memory).
  static constexpr bool STAGE = !TALL;
  static constexpr bool PHS = IN_OP;
  static constexpr int threads = MaxT<RS, BY>::value;
};

// A thread's own slot for its tile of one slice, filled by cp.async with an L2
// evict-first policy (each thread waits for its own copies only).
template <typename SP, int BY>
struct TileSlot {
  static constexpr int ROW = 4 * sizeof(SP);  // bytes of two complex numbers or four angles: 16 or 32
  // odd multiples of the access width apart
  static constexpr int BYTES = 16 * ((ROW / 16 * BY) | 1);
  unsigned char* p;
  __device__ __forceinline__ void init(unsigned char* smem, int tid) { p = smem + (size_t)tid * BYTES; }
  __device__ __forceinline__ SP* row(int r) const { return reinterpret_cast<SP*>(p + r * ROW); }
  // src: the tile's first site, rs: reals per row of the slice
  __device__ __forceinline__ void fetch_first(const SP* src, int rs) const {
    const unsigned long long pol = evict_first_policy();
#pragma unroll
    for (int r = 0; r < BY; ++r)
#pragma unroll
      for (int k = 0; k < ROW / 16; ++k)
        cp_async16(row(r) + 16 / sizeof(SP) * k, src + r * rs + 16 / sizeof(SP) * k, pol);
  }
  __host__ __device__ static size_t smem(int threads) { return ((size_t)threads * BYTES + 15) / 16 * 16; }
};

// the engines of the operator phase and of the true residual
template <typename RS, int BY>
using OpSlice = Slice<RS, BY, PcgT<RS, BY>::PHS, PcgT<RS, BY>::TALL ? 1 : 2>;
template <typename RH, int BY>
using TrueSlice = Slice<RH, BY, true, 1>;

// shared memory of the phases behind the right-hand sides' state
template <typename RS, typename RH, typename SP, int BY>
inline size_t pcg_phase_smem(int eng_threads, int col_rows, int CH) {
  using T = PcgT<RS, BY>;
  size_t s = slice_smem<RS>(eng_threads, OpSlice<RS, BY>::REC) +
             (T::IN_OP ? 0 : 2 * stash_smem<RS, BY>(eng_threads)) + (T::STAGE ? TileSlot<RS, BY>::smem(eng_threads) : 0);
  if (!std::is_same<RS, RH>::value) s = std::max(s, slice_smem<RH>(eng_threads, TrueSlice<RH, BY>::REC));
  return std::max(s, sizeof(Cx<RS>) * (size_t)col_rows * CH);
}

// ---------------------------------------------------------------------------
// operator pass over one run of slices [a, b) of one right-hand side
// ---------------------------------------------------------------------------
// p_new = z + beta p_old on the run and its halo slices, Op = M^dag M p_new,
// pap += p_new^dag M^dag M p_new = sum_t |(M p_new)_t|^2 over the run, and the
// previous iteration's x += alpha p_old on the run's own slices while p_old is
// in registers anyway.  q lies in shared memory and is read where it is used:
// its pointers and scalars, kept in registers, make the slice loop spill.
template <typename RS, typename A, typename SP>
struct OpRun {
  int L, Nt, a, b, eng, x_too;
  int64_t sv;  // reals per slice
  const A* phi;
  const SP *zz, *pold;
  SP* pnew;
  RS *xl, *O;
  RS beta, al_old, s_z, s_po, s_pn, i_pn;  // storage scales: 1 unless scaled fp16
  RS t1, th, Cb;
};

template <typename RS, typename A, typename SP, int BY>
__device__ __forceinline__ void operator_run(const OpRun<RS, A, SP>& q, unsigned char* smem, double& pap_out, double& ppp_out) {
  using CT = PcgT<RS, BY>;
  constexpr bool H16 = std::is_same<SP, __half>::value, LOWP = !std::is_same<SP, RS>::value;
  using Eng = OpSlice<RS, BY>;
  // the first two slices' angles are asked for together: at BY = 2, where
  // registers hold them, 2 to 4 % of an iteration (L = 48, 2 right-hand sides,
  // 53.6 -> 52.3 us); with taller tiles or converted storage they spill
  constexpr bool AHEAD = sizeof(RS) == 4 && BY == 2 && !LOWP;
  const int tid = threadIdx.x;
  Eng E;
  E.init(q.L, smem, tid);
  size_t at = slice_smem<RS>(q.eng, Eng::REC);
  // y_t and y_{t+1} wait in two stashes in turn
  Stash<RS, BY> stash, other;
  if constexpr (!CT::IN_OP) {
    stash.init(smem + at, tid);
    at += stash_smem<RS, BY>(q.eng);
    other.init(smem + at, tid);
    at += stash_smem<RS, BY>(q.eng);
  }
  TileSlot<A, BY> slot;  // the angles and x in turn
  static_assert(sizeof(A) == sizeof(RS), "x and the angles share a slot");
  if constexpr (CT::STAGE) slot.init(smem + at, tid);
  const int a = q.a;
  double pap = 0, ppp = 0;
  Cx<RS> X0[BY][2], X1[BY][2], Y[BY][2];
  // z and p_old of slice t, and x of own slices with a pending update, on their way
  auto fetch = [&](Cx<RS> (&X)[BY][2], Cx<RS> (&T)[BY][2], int t, bool own) {
    if constexpr (CT::STAGE) {
      if (own && q.x_too) slot.fetch_first(q.xl + t * q.sv + E.off, E.rs);
      cp_async_commit();
    }
    E.load_st(X, q.zz + t * q.sv, q.s_z);
    E.load_st(T, q.pold + t * q.sv, q.s_po);
  };
  // the angles of slice t on their way, where x waited
  auto fetch_angles = [&](int t) {
    if constexpr (CT::STAGE) {
      slot.fetch_first(q.phi + t * q.sv + E.off, E.rs);
      cp_async_commit();
    }
  };
  auto phases = [&](int t) {
    A ang[BY][4];
    if constexpr (CT::STAGE) {
      cp_async_wait<0>();
#pragma unroll
      for (int r = 0; r < BY; ++r) {
        Cx<A> u, w;
        ld2c(slot.row(r), u, w);
        ang[r][0] = u.re;
        ang[r][1] = u.im;
        ang[r][2] = w.re;
        ang[r][3] = w.im;
      }
    } else {
      E.load_angles(ang, q.phi + t * q.sv);
    }
    E.phases(ang, q.t1, q.th);
  };
  // X <- p_new = z + q.beta p_old of slice t, rounded to the storage, row by row;
  // on own slices p_new is stored, with x += alpha_old p_old
  auto form = [&](Cx<RS> (&X)[BY][2], const Cx<RS> (&Z)[BY][2], const Cx<RS> (&T)[BY][2], int t, bool own) {
    if constexpr (CT::STAGE) cp_async_wait<0>();
#pragma unroll
    for (int r = 0; r < BY; ++r) {
      const int64_t i = t * q.sv + E.off + r * E.rs;
      const Cx<RS> Z0 = Z[r][0], Z1 = Z[r][1], T0 = T[r][0], T1 = T[r][1];
      X[r][0] = mk<RS>(fma(q.beta, T0.re, Z0.re), fma(q.beta, T0.im, Z0.im));
      X[r][1] = mk<RS>(fma(q.beta, T1.re, Z1.re), fma(q.beta, T1.im, Z1.im));
      if constexpr (LOWP) {
        X[r][0] = round_st<SP>(X[r][0], q.s_pn, q.i_pn);
        X[r][1] = round_st<SP>(X[r][1], q.s_pn, q.i_pn);
      }
      if (!own) continue;
      if (E.on) st2s(q.pnew + i, X[r][0], X[r][1], q.i_pn);
      if (q.x_too) {
        Cx<RS> l0, l1;
        if constexpr (CT::STAGE) ld2c(slot.row(r), l0, l1);
        else ld2c(q.xl + i, l0, l1);
        l0 = mk<RS>(fma(q.al_old, T0.re, l0.re), fma(q.al_old, T0.im, l0.im));
        l1 = mk<RS>(fma(q.al_old, T1.re, l1.re), fma(q.al_old, T1.im, l1.im));
        if (E.on) st2_first(q.xl + i, l0, l1);
      }
    }
    if constexpr (H16)
      if (own && E.on) ppp += sq_blk<RS, BY>(X);
  };
  const int tp = a == 0 ? q.Nt - 1 : a - 1;
  Cx<RS> Z[BY][2], T[BY][2];  // z and p_old of the slice after this one
  A first[BY][4];             // the angles of the first slice
  fetch_angles(tp);
  fetch(Z, T, tp, false);
  if constexpr (AHEAD) E.load_angles(first, q.phi + a * q.sv);
  phases(tp);
  form(X0, Z, T, tp, false);
  fetch(Z, T, a, true);
  E.template applyB<0>(X0);
  if constexpr (AHEAD) E.phases(first, q.t1, q.th);
  form(X1, Z, T, a, true);
  if constexpr (!AHEAD) fetch_angles(a);
  axpy_blk<RS, BY>(Y, X1, sigma_of<RS>(tp, q.Nt) * q.Cb, X0);  // y_a
  if constexpr (CT::IN_OP) E.store(q.O + a * q.sv, Y); else stash.park(Y);
  copy_blk<RS, BY>(X0, X1);
  for (int t = a; t < q.b; ++t) {
    const int tn = t + 1 == q.Nt ? 0 : t + 1;
    const bool own = t + 1 < q.b;
    if (!AHEAD || t > a) phases(t);
    const RS sg = sigma_of<RS>(t, q.Nt) * q.Cb;
    fetch(Z, T, tn, own);
    E.template applyB<1>(X0);            // B_t p_t
    form(X1, Z, T, tn, own);
    if (own) fetch_angles(t + 1);
    axpy_blk<RS, BY>(Y, X1, sg, X0);     // y_{t+1}
    // y_t and y_{t+1} are not in registers now
    if constexpr (CT::IN_OP) {
      if (own) E.store(q.O + (t + 1) * q.sv, Y);
    } else {
      other.park(Y);
    }
    E.template applyB<0>(Y);             // B_t y_{t+1}
    if constexpr (CT::IN_OP) {
      E.load_st(X0, q.O + t * q.sv);     // y_t
    } else {
      stash.unpark(X0);
      RS* w = stash.p;
      stash.p = other.p;
      other.p = w;
    }
    pap += E.on ? sq_blk<RS, BY>(X0) : 0.0;
    axpy_blk<RS, BY>(Y, X0, sg, Y);      // (M^dag M p)_t
    E.store(q.O + t * q.sv, Y);
    copy_blk<RS, BY>(X0, X1);
  }
  pap_out += pap;
  ppp_out += ppp;
}

// ---------------------------------------------------------------------------
// the true residual in the high precision (mixed modes): y = M x, then
// r = b - M^dag y, each one B per slice and slices independent; y, double,
// waits in two buffers of 16 bytes per site pair (first sites, second sites).
// Returns |r|^2 over the run.
// ---------------------------------------------------------------------------
template <typename RS, typename RH, typename A>
struct TrueRun {
  int L, Nt, a, b;
  const A* phi;
  const RH *x, *rhs;
  RS* r;
  double2 *ya, *yb;
  double t1, th, Cb;
};

template <typename RS, typename RH, typename A, int BY, bool SECOND>
__device__ __noinline__ double true_residual_run(const TrueRun<RS, RH, A>& q, int smem_at) {
  // (the address, formed here, is known to be a shared one)
  extern __shared__ __align__(128) unsigned char dsm_all[];
  unsigned char* smem = dsm_all + smem_at;
  TrueSlice<RH, BY> E;
  E.init(q.L, smem, threadIdx.x);
  const int Nt = q.Nt;
  const int64_t sv = 2 * (int64_t)q.L * q.L;
  const RH t1 = (RH)q.t1, th = (RH)q.th, Cb = (RH)q.Cb;
  double sum = 0;
  auto ypair = [&](int t, int r) { return (t * sv + E.off + r * E.rs) / 4; };
  for (int t = q.a; t < q.b; ++t) {
    Cx<RH> V[BY][2];
    if constexpr (!SECOND) {
      const int tp = t == 0 ? Nt - 1 : t - 1;
      E.load_st(V, q.x + tp * sv);
      E.phases_of(q.phi + tp * sv, t1, th);
      E.template applyB<0>(V);
      const RH sg = sigma_of<RH>(tp, Nt) * Cb;
#pragma unroll
      for (int r = 0; r < BY; ++r) {
        Cx<RH> x0, x1;
        ld2c(q.x + t * sv + E.off + r * E.rs, x0, x1);
        if (!E.on) continue;
        q.ya[ypair(t, r)] = make_double2(fma(-sg, V[r][0].re, x0.re), fma(-sg, V[r][0].im, x0.im));
        q.yb[ypair(t, r)] = make_double2(fma(-sg, V[r][1].re, x1.re), fma(-sg, V[r][1].im, x1.im));
      }
    } else {
      const int tn = t + 1 == Nt ? 0 : t + 1;
#pragma unroll
      for (int r = 0; r < BY; ++r) {
        const double2 u = q.ya[ypair(tn, r)], w = q.yb[ypair(tn, r)];
        V[r][0] = mk<RH>(u.x, u.y);
        V[r][1] = mk<RH>(w.x, w.y);
      }
      E.phases_of(q.phi + t * sv, t1, th);
      E.template applyB<0>(V);
      const RH sg = sigma_of<RH>(t, Nt) * Cb;
#pragma unroll
      for (int r = 0; r < BY; ++r) {
        const double2 u = q.ya[ypair(t, r)], w = q.yb[ypair(t, r)];
        const int64_t at = t * sv + E.off + r * E.rs;
        Cx<RH> b0, b1;
        ld2c(q.rhs + at, b0, b1);
        if (!E.on) continue;
        b0 = mk<RH>(b0.re - fma(-sg, V[r][0].re, u.x), b0.im - fma(-sg, V[r][0].im, u.y));
        b1 = mk<RH>(b1.re - fma(-sg, V[r][1].re, w.x), b1.im - fma(-sg, V[r][1].im, w.y));
        sum += b0.re * b0.re + b0.im * b0.im + b1.re * b1.re + b1.im * b1.im;
        st2(q.r + at, mk<RS>((RS)b0.re, (RS)b0.im), mk<RS>((RS)b1.re, (RS)b1.im));
      }
    }
  }
  return sum;
}

// ---------------------------------------------------------------------------
// the persistent kernel
// ---------------------------------------------------------------------------
// RS iteration precision, RH precision of b and x, A angles, SP storage of the
// search direction p and the preconditioned residual z: RS, bf16 pairs or
// scaled fp16 pairs (mixed-mode options).  r, M^dag M p and x_lo always keep
// the iteration precision, so that the residual recurrence r -= alpha M^dag M p
// stays that of x += alpha p.
template <typename RS, typename RH, typename A, typename SP, int BY>
__global__ void __launch_bounds__(PcgT<RS, BY>::threads, 1)
    k_pcg(const __grid_constant__ PcgParams p, const __grid_constant__ BandTaps taps) {
  constexpr bool MIXED = !std::is_same<RS, RH>::value;
  constexpr bool H16 = std::is_same<SP, __half>::value;
  constexpr bool LOWP = !std::is_same<SP, RS>::value;
  extern __shared__ __align__(128) unsigned char dsm_all[];
  __shared__ double red[64];
  __shared__ PcgCtl ctl;
  __shared__ OpRun<RS, A, SP> oprun;
#define NV p.nrhs
  using State = RhsState<MIXED, H16>;
  const State st{dsm_all, NV};
  const Acc acc{p.acc, NV};
#define dsm (dsm_all + State::bytes(NV))
  const int tid = threadIdx.x;
  // scales of z and of p buffer `par` (1 for every other storage type)
  auto sc_z = [&](int v) -> RS {
    if constexpr (H16) return (RS)st.scz()[v];
    else return (RS)1;
  };
  auto sc_p = [&](int par, int v) -> RS {
    if constexpr (H16) return (RS)st.scp(par)[v];
    else return (RS)1;
  };
  auto xs = [&]() { return MIXED ? reinterpret_cast<RS*>(p.xlo) : reinterpret_cast<RS*>(p.x); };
  auto xh = [&]() { return reinterpret_cast<RH*>(p.x); };
  auto bvec = [&]() { return reinterpret_cast<const RH*>(p.b); };
  auto phi_all = [&]() { return reinterpret_cast<const A*>(p.phi); };
  // r, double-buffered where units read their neighbours' rows (p.r2)
  auto rbuf = [&](int k) { return reinterpret_cast<RS*>(k && p.r2 ? p.r2 : p.r); };

  for (int s = 0; s < p.nsys; ++s)
    for (int v = p.sys[s].rhs0 + tid; v < p.sys[s].rhs0 + p.sys[s].nrhs; v += blockDim.x) st.sys()[v] = (unsigned char)s;
  for (int v = tid; v < NV; v += blockDim.x) {
    st.active()[v] = 1;
    st.iters()[v] = 0;
    st.status()[v] = QEDF_OK;
    st.res()[v] = 0.0;
    st.pending()[v] = 0;
    if constexpr (MIXED) {
      st.lastru()[v] = 0;
      st.resmax()[v] = 1.0;
      st.ru()[v] = 0;
    }
  }
  if (tid == 0) {
    ctl.it = ctl.slot = ctl.rcur = ctl.guess = 0;
    ctl.relay = 1;
    ctl.target = 0;
    ctl.t0 = ctl.t = p.prof ? clock64() : 0;
  }

  auto vec_base = [&](const PcgSys& S, int v) -> int64_t {
    return S.vec0 + (int64_t)(v - S.rhs0) * S.Nt * S.L * S.L;
  };

  // ---- work lines -------------------------------------------------------------
  // lay the line of the right-hand sides with pred(v) and find this block's run of it
  auto lay_line = [&](auto pred) {
    __syncthreads();
    if (tid == 0) {
      int n = 0, a = 0, e = 0;
      int *pa = st.pre_a(), *pe = st.pre_e();
      for (int v = 0; v < NV; ++v)
        if (pred(v)) {
          const PcgSys& S = p.sys[st.sys()[v]];
          st.list()[n] = v;
          pa[n] = a;
          pe[n] = e;
          a += S.nslab;
          e += S.nchunk * S.nseg;
          ++n;
        }
      pa[n] = a;
      pe[n] = e;
      ctl.n = n;
      ctl.u0a = (int)((int64_t)a * blockIdx.x / gridDim.x);
      ctl.u1a = (int)((int64_t)a * (blockIdx.x + 1) / gridDim.x);
      ctl.u0e = (int)((int64_t)e * blockIdx.x / gridDim.x);
      ctl.u1e = (int)((int64_t)e * (blockIdx.x + 1) / gridDim.x);
      // (a block without units starts at the line's end)
      int k = ctl.u0a < ctl.u1a ? 0 : n;
      while (k < n && pa[k + 1] <= ctl.u0a) ++k;
      ctl.ka = k;
      k = ctl.u0e < ctl.u1e ? 0 : n;
      while (k < n && pe[k + 1] <= ctl.u0e) ++k;
      ctl.ke = k;
    }
    __syncthreads();
  };
  // operator work of this block: f(v, S, a, b) for the tau-slices [a, b)
  auto for_slices = [&](auto f) {
    for (int k = ctl.ka; k < ctl.n && st.pre_a()[k] < ctl.u1a; ++k) {
      const int base = st.pre_a()[k];
      const int ua = max(ctl.u0a, base) - base, ub = min(ctl.u1a, st.pre_a()[k + 1]) - base;
      const int v = st.list()[k];
      const PcgSys& S = p.sys[st.sys()[v]];
      f(v, S, ua * S.T, min(ub * S.T, S.Nt));
    }
  };
  // elementwise work: f(v, S, unit), then done(v) after the last unit of a right-hand side
  auto for_units = [&](auto f, auto done) {
    for (int k = ctl.ke; k < ctl.n && st.pre_e()[k] < ctl.u1e; ++k) {
      const int base = st.pre_e()[k];
      const int ub = min(ctl.u1e, st.pre_e()[k + 1]) - base;
      const int v = st.list()[k];
      for (int u = max(ctl.u0e, base) - base; u < ub; ++u) f(v, p.sys[st.sys()[v]], u);
      done(v);
    }
  };
  auto barrier = [&]() { return grid_barrier(p.bar, gridDim.x, p.timeout_cycles, ctl.target); };

  // ---- BC-type elementwise pass over one unit ----------------------------------
  // kind 0: init (x = 0 unless it holds an initial guess, r = b, bb); 1:
  // iteration update; 2: preconditioner only (after a reliable update or the
  // initial guess's residual); 3: preconditioner only, r^dag z into the rz
  // slot (scaled fp16 init).  A unit is CH sites of one right-hand side over a
  // tau segment, the whole of tau unless that leaves SMs idle; a thread
  // handles two neighbouring sites (one 16-byte access per vector in single
  // precision) per row.  r of the unit stays in shared memory for the
  // tau-stencil of the preconditioner, with six rows of each neighbouring
  // segment, whose r this unit computes as well; r is double-buffered then.
  // The periodic 13-band table P_tab[t][k] (offset k - 6; the corners of the
  // reference's matrix are the band's wrap-around) was prepared per system.  A
  // thread forms PCG_ZROWS consecutive rows of z, reading PCG_ZROWS + 12 rows
  // of the column instead of 13 for each.
  auto elementwise = [&](auto kind_c, int v, const PcgSys& S, int u, double& acc_a, double& acc_b, double& acc_c) {
    constexpr int kind = decltype(kind_c)::value;
    const int Vs = S.L * S.L, Nt = S.Nt, CH = p.CH, PPR = CH / 2;
    const int c0 = (u % S.nchunk) * CH, w = min(CH, Vs - c0);
    const int t0 = (u / S.nchunk) * S.seg, len = min(S.seg, Nt - t0);
    const int h = S.nseg > 1 && S.precon ? 6 : 0;  // neighbours' rows on either side
    const int rows = len + 2 * h;
    RS* col = reinterpret_cast<RS*>(dsm);  // [rows][CH] complex
    const int j = tid % PPR, g0 = tid / PPR, gstep = blockDim.x / PPR;
    const bool jon = 2 * j < w && g0 < gstep;
    const int64_t base = 2 * (vec_base(S, v) + c0 + 2 * j);  // reals
    const int64_t sv = 2 * (int64_t)Vs;
    const RS* rin = rbuf(ctl.rcur);
    RS* rout = rbuf(kind == 1 ? ctl.rcur ^ 1 : ctl.rcur);
    const RS* Op = reinterpret_cast<const RS*>(p.Op);
    SP* z = reinterpret_cast<SP*>(p.z);
    // (alpha from its accumulator, whose latency is then the rows' own)
    const RS al = kind != 1 ? (RS)0 : ctl.guess ? (RS)1 : (RS)(st.rz()[v] / acc.pAp(ctl.it & 1)[v]);
    RS cpart = 0;
    // row i of the column is slice t0 - h + i (mod Nt); the unit's own rows are [h, h + len)
    auto slice_of = [&](int i) {
      int t = t0 - h + i;
      return t < 0 ? t + Nt : (t >= Nt ? t - Nt : t);
    };
    if constexpr (kind == 1) {
      // UN rows of both vectors in flight per thread (past the last row the
      // last one is loaded again and dropped)
      constexpr int UN = sizeof(RS) == 4 ? PCG_EW_ROWS : PCG_EW_ROWS / 2;
      const RS* o = reinterpret_cast<const RS*>(p.Op) + base;
      const RS* ri = rin + base;
      RS* ro = rout + base;
      const int svi = (int)sv;
      if (jon)
        for (int i0 = g0; i0 < rows; i0 += UN * gstep) {
          Cx<RS> o0[UN], o1[UN], r0[UN], r1[UN];
#pragma unroll
          for (int k = 0; k < UN; ++k) {
            const int at = slice_of(min(i0 + k * gstep, rows - 1)) * svi;
            ld2c(o + at, o0[k], o1[k]);
            ld2c(ri + at, r0[k], r1[k]);
          }
#pragma unroll
          for (int k = 0; k < UN; ++k) {
            const int i = i0 + k * gstep;
            if (i >= rows) break;
            r0[k] = mk<RS>(fma(-al, o0[k].re, r0[k].re), fma(-al, o0[k].im, r0[k].im));
            r1[k] = mk<RS>(fma(-al, o1[k].re, r1[k].re), fma(-al, o1[k].im, r1[k].im));
            st2(col + 2 * (i * CH + 2 * j), r0[k], r1[k]);
            if (i < h || i >= h + len) continue;
            st2(ro + slice_of(i) * svi, r0[k], r1[k]);
            cpart = fma(r0[k].re, r0[k].re, fma(r0[k].im, r0[k].im, fma(r1[k].re, r1[k].re, fma(r1[k].im, r1[k].im, cpart))));
          }
        }
      acc_c += (double)cpart;
    } else if (jon) {
#pragma unroll 2
      for (int i = g0; i < rows; i += gstep) {
        const int64_t q = base + slice_of(i) * sv;
        const bool own = i >= h && i < h + len;
        Cx<RS> r0, r1;
        if constexpr (kind == 0) {
          Cx<RH> b0, b1;
          ld2c(bvec() + q, b0, b1);
          r0 = mk<RS>((RS)b0.re, (RS)b0.im);
          r1 = mk<RS>((RS)b1.re, (RS)b1.im);
          if (own) {
            acc_a += (double)b0.re * b0.re + (double)b0.im * b0.im + (double)b1.re * b1.re + (double)b1.im * b1.im;
            // x_lo (mixed) always starts at 0; x itself unless it is the guess
            if (MIXED || !p.x_init) st2(xs() + q, mk<RS>(0, 0), mk<RS>(0, 0));
            if (MIXED && !p.x_init) st2(xh() + q, mk<RH>(0, 0), mk<RH>(0, 0));
            st2(rout + q, r0, r1);
          }
        } else {
          ld2c(rin + q, r0, r1);
        }
        if (own)
          acc_c += (double)r0.re * r0.re + (double)r0.im * r0.im + (double)r1.re * r1.re + (double)r1.im * r1.im;
        st2(col + 2 * (i * CH + 2 * j), r0, r1);
      }
    }
    __syncthreads();
    // scaled fp16: the scale of z follows from |r|, known only after the init
    // pass, so that pass leaves z to a kind-3 pass
    constexpr bool zpass = !(H16 && kind == 0);
    if (jon && zpass) {
      const RS szv = sc_z(v), izv = (RS)1 / szv;  // powers of two: exact
      RS bpart = 0;  // this thread's r^dag z in the iteration precision
      const RS* cj = col + 4 * j;
      const int rw = 2 * CH;  // reals per row of the column
      auto put = [&](int i, Cx<RS> z0, Cx<RS> z1) {  // row i of the segment
        Cx<RS> r0, r1;
        ld2c(cj + (h + i) * rw, r0, r1);
        z0 = round_st<SP>(z0, szv, izv);
        z1 = round_st<SP>(z1, szv, izv);
        st2s(z + base + (int64_t)(t0 + i) * sv, z0, z1, izv);
        bpart = fma(r0.re, z0.re, fma(r0.im, z0.im, fma(r1.re, z1.re, fma(r1.im, z1.im, bpart))));
      };
      if (S.precon) {
        // bulk rows [lo, lo + PCG_ZROWS nrun): constant coefficients, no wrap;
        // the others, a few at the ends of tau, one at a time from the table
        const int lo = max(S.pmid_lo - t0, 0), nrun = max(min(S.pmid_hi - t0, len) - lo, 0) / PCG_ZROWS;
        for (int m = g0; m < nrun; m += gstep) {
          const int i = lo + PCG_ZROWS * m;
          Cx<RS> a0[PCG_ZROWS], a1[PCG_ZROWS];
#pragma unroll
          for (int k = 0; k < PCG_ZROWS; ++k) a0[k] = a1[k] = mk<RS>(0, 0);
          const RS* q = cj + (h + i - 6) * rw;
#pragma unroll
          for (int n = 0; n < PCG_ZROWS + 12; ++n) {
            Cx<RS> q0, q1;
            ld2c(q + n * rw, q0, q1);
#pragma unroll
            for (int k = 0; k < PCG_ZROWS; ++k) {
              const int d = n - 6 - k;  // tau distance of row n from output row k
              if (d < -6 || d > 6) continue;
              const RS c = (RS)taps.c[d < 0 ? -d : d];
              a0[k] = mk<RS>(fma(c, q0.re, a0[k].re), fma(c, q0.im, a0[k].im));
              a1[k] = mk<RS>(fma(c, q1.re, a1[k].re), fma(c, q1.im, a1[k].im));
            }
          }
#pragma unroll
          for (int k = 0; k < PCG_ZROWS; ++k) put(i + k, a0[k], a1[k]);
        }
        const float* tab = p.ptab + S.ptab0;
        const int first = min(lo, len), rest = len - PCG_ZROWS * nrun;
        for (int e = gstep - 1 - g0; e < rest; e += gstep) {
          const int k = e < first ? e : e + PCG_ZROWS * nrun;
          Cx<RS> z0 = mk<RS>(0, 0), z1 = z0;
          int m = h + k - 6;  // without neighbours' rows the column wraps
          if (m < 0) m += Nt;
#pragma unroll
          for (int d = 0; d < 13; ++d) {
            const RS c = (RS)__ldg(tab + (t0 + k) * 13 + d);
            Cx<RS> q0, q1;
            ld2c(cj + m * rw, q0, q1);
            z0 = mk<RS>(fma(c, q0.re, z0.re), fma(c, q0.im, z0.im));
            z1 = mk<RS>(fma(c, q1.re, z1.re), fma(c, q1.im, z1.im));
            ++m;
            if (h == 0 && m == Nt) m = 0;
          }
          put(k, z0, z1);
        }
      } else {
        // z = r; the narrow-storage engines read z, rounded, the others r
        for (int i = g0; i < len; i += gstep) {
          Cx<RS> r0, r1;
          ld2c(cj + i * rw, r0, r1);
          if (LOWP) put(i, r0, r1);
          else bpart = fma(r0.re, r0.re, fma(r0.im, r0.im, fma(r1.re, r1.re, fma(r1.im, r1.im, bpart))));
        }
      }
      acc_b += (double)bpart;
    }
    __syncthreads();
  };
  // the pass over this block's units; sums go to the accumulators once per right-hand side
  auto elementwise_pass = [&](auto kind_c, int slot) {
    constexpr int kind = decltype(kind_c)::value;
    double a = 0, b = 0, c = 0;
    for_units([&](int v, const PcgSys& S, int u) { elementwise(kind_c, v, S, u, a, b, c); },
              [&](int v) {
                if (kind == 0) block_sum_d(a, red);
                block_sum2_d(b, c, red);
                if (tid == 0) {
                  if (kind == 0) atomicAdd(acc.bb() + v, a);
                  if (kind == 0 || kind == 1) atomicAdd(acc.rr(slot) + v, c);
                  if (kind == 2) atomicAdd(acc.ru_rz() + v, b);
                  else atomicAdd(acc.rz(slot) + v, b);
                }
                a = b = c = 0;
              });
  };

  // ---- operator pass over this block's runs of slices ------------------------------
  auto operator_pass = [&](int slot) {
    for_slices([&](int v, const PcgSys& S, int a, int b) {
      double pap = 0, ppp = 0;
      __syncthreads();
      if (tid == 0) {
        const int64_t vb = 2 * vec_base(S, v);  // reals
        const int64_t sv = 2 * (int64_t)S.L * S.L;
        const int it = st.iters()[v];
        OpRun<RS, A, SP>& q = oprun;
        q.L = S.L;
        q.sv = sv;
        q.Nt = S.Nt;
        q.a = a;
        q.b = b;
        q.eng = p.eng_threads;
        q.phi = phi_all() + S.phi0 + (S.shared ? 0 : (int64_t)(v - S.rhs0) * S.Nt * sv);
        q.zz = (ctl.guess ? reinterpret_cast<const SP*>(xs())
                           : (S.precon || LOWP) ? reinterpret_cast<const SP*>(p.z)
                                                     : reinterpret_cast<const SP*>(rbuf(ctl.rcur))) + vb;
        // the first iteration has no p_old: z stands in, with beta = 0
        q.pold = it > 0 ? reinterpret_cast<const SP*>((it & 1) ? p.p0 : p.p1) + vb : q.zz;
        q.pnew = reinterpret_cast<SP*>((it & 1) ? p.p1 : p.p0) + vb;
        q.xl = xs() + vb;
        q.O = reinterpret_cast<RS*>(p.Op) + vb;
        q.beta = it > 0 ? (RS)st.beta()[v] : (RS)0;
        // the previous iteration's x += alpha p (alpha = 0: none is pending)
        q.al_old = st.pending()[v] ? (RS)st.alpha()[v] : (RS)0;
        q.x_too = st.pending()[v];
        q.s_z = sc_z(v);
        q.s_po = it > 0 ? sc_p((it & 1) ^ 1, v) : q.s_z;
        q.s_pn = sc_p(it & 1, v);
        q.i_pn = (RS)1 / q.s_pn;
        q.t1 = (RS)p.t1;
        q.th = (RS)p.th;
        q.Cb = (RS)p.Cb;
      }
      __syncthreads();
      if (tid < p.eng_threads) operator_run<RS, A, SP, BY>(oprun, dsm, pap, ppp);
      else OpSlice<RS, BY>::idle_apply(1 + 2 * (b - a));
      if constexpr (H16) block_sum2_d(pap, ppp, red);
      else block_sum_d(pap, red);
      if (tid == 0) {
        atomicAdd(acc.pAp(slot) + v, pap);
        if constexpr (H16) atomicAdd(acc.pp(slot) + v, ppp);
      }
    });
  };

  // ---- the true residual's runs (mixed modes) ----------------------------------------
  auto true_run = [&](int v, const PcgSys& S, int a, int b) {
    const int64_t vb = 2 * vec_base(S, v);
    TrueRun<RS, RH, A> q;
    q.L = S.L;
    q.Nt = S.Nt;
    q.a = a;
    q.b = b;
    q.phi = phi_all() + S.phi0 + (S.shared ? 0 : (int64_t)(v - S.rhs0) * S.Nt * 2 * S.L * S.L);
    q.x = xh() + vb;
    q.rhs = bvec() + vb;
    q.r = rbuf(ctl.rcur) + vb;
    // a site pair is four reals
    q.ya = reinterpret_cast<double2*>(p.y0) + vb / 4;
    q.yb = reinterpret_cast<double2*>(p.Op) + vb / 4;
    q.t1 = p.t1;
    q.th = p.th;
    q.Cb = p.Cb;
    return q;
  };

  // the pending x += alpha p_last of right-hand side v at one site pair
  auto apply_pending = [&](int v, int64_t i2, Cx<RS>& l0, Cx<RS>& l1) {
    if (!st.pending()[v]) return;
    const SP* pl = reinterpret_cast<const SP*>((st.iters()[v] & 1) ? p.p0 : p.p1);  // p of the last iteration
    const RS al = (RS)st.alpha()[v];
    Cx<RS> p0v, p1v;
    ld2s(pl + i2, p0v, p1v, sc_p((st.iters()[v] & 1) ^ 1, v));
    l0 = mk<RS>(fma(al, p0v.re, l0.re), fma(al, p0v.im, l0.im));
    l1 = mk<RS>(fma(al, p1v.re, l1.re), fma(al, p1v.im, l1.im));
  };
  // f(i2) at every site pair of this block's units of the line (i2: reals)
  auto for_pairs = [&](auto f) {
    for_units(
        [&](int v, const PcgSys& S, int u) {
          const int CH = p.CH, PPR = CH / 2;
          const int Vs = S.L * S.L, c0 = (u % S.nchunk) * CH, t0 = (u / S.nchunk) * S.seg;
          const int j = tid % PPR, gstep = blockDim.x / PPR;
          if (2 * j >= min(CH, Vs - c0) || tid / PPR >= gstep) return;
          for (int t = t0 + tid / PPR; t < min(t0 + S.seg, S.Nt); t += gstep)
            f(v, 2 * (vec_base(S, v) + (int64_t)t * Vs + c0 + 2 * j));
        },
        [](int) {});
  };
  // mixed: x (double) += x_lo (+ the pending update), x_lo = 0; plain: the
  // pending update alone
  auto fold_pass = [&]() {
    for_pairs([&](int v, int64_t i2) {
      Cx<RS> l0, l1;
      if constexpr (MIXED) {
        Cx<RH> h0, h1;
        ld2c(xs() + i2, l0, l1);
        apply_pending(v, i2, l0, l1);
        ld2c(xh() + i2, h0, h1);
        st2(xh() + i2, mk<RH>(h0.re + (RH)l0.re, h0.im + (RH)l0.im), mk<RH>(h1.re + (RH)l1.re, h1.im + (RH)l1.im));
        st2(xs() + i2, mk<RS>(0, 0), mk<RS>(0, 0));
      } else {
        ld2c(xs() + i2, l0, l1);
        apply_pending(v, i2, l0, l1);
        st2(xs() + i2, l0, l1);
      }
    });
  };

  // ---------------------------------------------------------------------------
  // init: x = 0, r = b, z = P r
  lay_line([](int) { return true; });
  elementwise_pass(std::integral_constant<int, 0>(), 0);
  bool ok = barrier();
  if (ok) {
    for (int v = tid; v < NV; v += blockDim.x) {
      st.rz()[v] = acc.rz(0)[v];
      st.rzold()[v] = 1.0;
      st.rr()[v] = acc.rr(0)[v];
      if (acc.bb()[v] == 0.0) {  // b = 0: x = 0 is exact
        st.active()[v] = 0;
        st.res()[v] = 0.0;
      } else {
        st.res()[v] = sqrt(st.rr()[v] / acc.bb()[v]);
      }
    }
    __syncthreads();
  }
  if constexpr (H16) {
    // z = P r now that |r| = |b| fixes z's scale; r^dag z into the rz slot,
    // which the init pass left at zero
    if (ok) {
      for (int v = tid; v < NV; v += blockDim.x) st.scz()[v] = st_scale(st.rr()[v]);
      __syncthreads();
      elementwise_pass(std::integral_constant<int, 3>(), 0);
      ok = barrier();
    }
    if (ok) {
      for (int v = tid; v < NV; v += blockDim.x) st.rz()[v] = acc.rz(0)[v];
      __syncthreads();
    }
  }
  // initial guess: a right-hand side with b = 0 gets x = 0 (the exact
  // solution).  Mixed modes start the others with a reliable update (r = b -
  // A x in double, z = P r); plain modes with one pass of the iteration's own
  // two phases on p = x (guess pass: Op = A x, then r = b - 1 * Op and z = P
  // r), which counts no iteration and updates no x
  if (ok && p.x_init) {
    for_pairs([&](int v, int64_t i2) {
      if (acc.bb()[v] == 0.0) st2(xh() + i2, mk<RH>(0, 0), mk<RH>(0, 0));
    });
    if (tid == 0) ctl.guess = !MIXED;
    __syncthreads();
  }
  lap(p.prof, ctl, 0);

  while (ok) {
    // ---- convergence / reliable-update decisions (identical in every block)
    if (tid == 0) ctl.any_ru = ctl.any_active = ctl.changed = 0;
    __syncthreads();
    const int it = ctl.it;
    for (int v = tid; v < NV; v += blockDim.x) {
      if constexpr (MIXED) st.ru()[v] = 0;
      if (!st.active()[v]) continue;
      const double res = st.res()[v];
      if (!isfinite(res)) {
        st.active()[v] = 0;
        st.status()[v] = QEDF_ERR_NAN;
        ctl.changed = 1;
        continue;
      }
      if constexpr (MIXED) {
        // (the initial guess's residual is a reliable update's)
        if (res <= p.rtol || it - st.lastru()[v] >= p.ru_interval || res < p.ru_delta * st.resmax()[v] ||
            (it == 0 && p.x_init)) {
          st.ru()[v] = 1;
          ctl.any_ru = 1;
        }
      } else if (res <= p.rtol) {
        st.active()[v] = 0;
        ctl.changed = 1;
      }
      if (st.active()[v]) ctl.any_active = 1;
    }
    __syncthreads();
    if constexpr (MIXED) {
      if (ctl.any_ru) {
        lap(p.prof, ctl, 6);
        lay_line([&](int v) { return st.ru()[v] != 0; });
        if (blockIdx.x == 0)
          for (int v = tid; v < NV; v += blockDim.x) {
            acc.ru_rr()[v] = 0;
            acc.ru_rz()[v] = 0;
          }
        fold_pass();
        if (!(ok = barrier())) break;
        for_slices([&](int v, const PcgSys& S, int a, int b) {
          if (tid < p.eng_threads) {
            const TrueRun<RS, RH, A> q = true_run(v, S, a, b);
            true_residual_run<RS, RH, A, BY, false>(q, (int)State::bytes(NV));
          } else {
            TrueSlice<RH, BY>::idle_apply(b - a);
          }
        });
        if (!(ok = barrier())) break;
        for_slices([&](int v, const PcgSys& S, int a, int b) {
          double sum = 0;
          if (tid < p.eng_threads) {
            const TrueRun<RS, RH, A> q = true_run(v, S, a, b);
            sum = true_residual_run<RS, RH, A, BY, true>(q, (int)State::bytes(NV));
          } else {
            TrueSlice<RH, BY>::idle_apply(b - a);
          }
          block_sum_d(sum, red);
          if (tid == 0) atomicAdd(acc.ru_rr() + v, sum);
        });
        if (!(ok = barrier())) break;
        if constexpr (H16) {
          for (int v = tid; v < NV; v += blockDim.x)
            if (st.ru()[v]) st.scz()[v] = st_scale(acc.ru_rr()[v]);
          __syncthreads();
        }
        elementwise_pass(std::integral_constant<int, 2>(), 0);
        if (!(ok = barrier())) break;
        if (tid == 0) {
          ctl.any_active = 0;
          ctl.changed = 1;  // the line was laid for the reliable update
        }
        __syncthreads();
        for (int v = tid; v < NV; v += blockDim.x) {
          if (st.ru()[v]) {
            st.pending()[v] = 0;  // folded into x above
            st.rr()[v] = acc.ru_rr()[v];
            st.rz()[v] = acc.ru_rz()[v];
            const double res = sqrt(st.rr()[v] / acc.bb()[v]);
            st.res()[v] = res;
            st.resmax()[v] = res;
            st.lastru()[v] = it;
            if (!isfinite(res)) {
              st.active()[v] = 0;
              st.status()[v] = QEDF_ERR_NAN;
            } else if (res <= p.rtol) {
              st.active()[v] = 0;
            }
          }
          if (st.active()[v]) ctl.any_active = 1;
        }
        __syncthreads();
        lap(p.prof, ctl, 5);
      }
    }
    if (!ctl.any_active || it >= p.max_iter) break;
    if (ctl.changed || ctl.relay) {
      lay_line([&](int v) { return st.active()[v] != 0; });
      if (tid == 0) ctl.relay = 0;
    }

    // ---- phase A
    for (int v = tid; v < NV; v += blockDim.x) {
      st.beta()[v] = st.iters()[v] > 0 ? st.rz()[v] / st.rzold()[v] : 0.0;
      if constexpr (H16)
        if (st.active()[v]) {
          // the scale of the buffer p_new goes to, from a bound of its norm:
          // |z + beta p_old| <= |P| |r| + beta |p_old| (|p_old| measured in the
          // last operator phase); p grows far above r in ill-conditioned solves
          double est = p.pnorm * sqrt(st.rr()[v]);
          if (st.iters()[v] > 0) est += fabs(st.beta()[v]) * sqrt(acc.pp((it & 1) ^ 1)[v]);
          st.scp(st.iters()[v] & 1)[v] = st_scale(est * est);
        }
    }
    __syncthreads();
    // (the guess pass uses the pAp slot of odd iterations, so that its BC
    // phase clears the slot of iteration 0)
    operator_pass(ctl.guess ? 1 : ctl.it & 1);
    // the rr/rz slot that BC will fill was last read before the previous barrier
    if (blockIdx.x == 0)
      for (int v = tid; v < NV; v += blockDim.x) {
        acc.rr(ctl.slot ^ 1)[v] = 0;
        acc.rz(ctl.slot ^ 1)[v] = 0;
      }
    lap(p.prof, ctl, 1);
    if (!(ok = barrier())) break;
    lap(p.prof, ctl, 2);

    // ---- phase BC
    const int aslot = ctl.guess ? 1 : ctl.it & 1;
    // alpha of inactive systems stays that of their last iteration: a pending
    // x update still uses it
    for (int v = tid; v < NV; v += blockDim.x)
      if (st.active()[v]) {
        st.alpha()[v] = ctl.guess ? 1.0 : st.rz()[v] / acc.pAp(aslot)[v];
        if constexpr (H16) st.scz()[v] = st_scale(st.rr()[v]);  // |r| before this update
      }
    if constexpr (H16) __syncthreads();
    elementwise_pass(std::integral_constant<int, 1>(), ctl.slot ^ 1);
    if (blockIdx.x == 0)  // pAp (and |p|^2) slot of the next iteration
      for (int v = tid; v < NV; v += blockDim.x) {
        acc.pAp(aslot ^ 1)[v] = 0;
        if constexpr (H16) acc.pp(aslot ^ 1)[v] = 0;
      }
    lap(p.prof, ctl, 3);
    if (!(ok = barrier())) break;
    lap(p.prof, ctl, 4);
    const int slot = ctl.slot ^ 1;
    for (int v = tid; v < NV; v += blockDim.x) {
      if (!st.active()[v]) continue;
      st.rzold()[v] = st.rz()[v];
      st.rz()[v] = acc.rz(slot)[v];
      st.rr()[v] = acc.rr(slot)[v];
      st.res()[v] = sqrt(st.rr()[v] / acc.bb()[v]);
      if (ctl.guess) continue;
      st.iters()[v] += 1;
      st.pending()[v] = 1;
    }
    __syncthreads();
    if (tid == 0) {
      ctl.slot = slot;
      ctl.rcur ^= 1;
      if (!ctl.guess) ++ctl.it;
      ctl.guess = 0;
    }
    lap(p.prof, ctl, 6);
  }
  if (p.prof && blockIdx.x == 0 && tid == 0) p.prof[7] += clock64() - ctl.t0;

  // mixed: fold the remaining float updates of unconverged systems into x;
  // plain: apply the last iteration's x update
  if (ok) {
    lay_line([&](int v) { return st.pending()[v] != 0 || (MIXED && st.active()[v] != 0); });
    fold_pass();
  }
  if (blockIdx.x == 0) {
    const unsigned int err = bar_error(*((volatile unsigned long long*)p.bar));
    for (int v = tid; v < NV; v += blockDim.x) {
      int stt = st.status()[v];
      if (err) stt = (int)err;
      else if (stt == QEDF_OK && st.active()[v]) stt = QEDF_ERR_MAXITER;
      p.status[v] = stt;
      p.iters[v] = st.iters()[v];
      p.relres[v] = st.res()[v];
    }
  }
}
#undef NV
#undef dsm

// ---------------------------------------------------------------------------
// launch
// ---------------------------------------------------------------------------
int pcg_launch_kernel(const void* kern, const PcgParams& p, const BandTaps& taps, int threads, size_t smem, int nblk,
                      cudaStream_t st);

template <typename RS, typename RH, typename A, typename SP, int BY>
static int launch_pcg_t(PcgParams& p, const BandTaps& taps, cudaStream_t st) {
  int eng = 0, rows = 0, ntmax = 0;
  int64_t slices = 0, units = 0;
  for (int s = 0; s < p.nsys; ++s) {
    const PcgSys& S = p.sys[s];
    if (S.L % BY) return QEDF_ERR_ARG;
    eng = std::max(eng, slice_threads(S.L, BY));
    rows = std::max(rows, S.seg + (S.nseg > 1 ? 12 : 0));
    ntmax = std::max(ntmax, S.Nt);
    slices += (int64_t)S.nrhs * S.nslab;
    units += (int64_t)S.nrhs * S.nchunk * S.nseg;
  }
  if (eng > PcgT<RS, BY>::threads) return QEDF_ERR_SIZE;
  // whole tau columns of PCG_CHUNK sites are the documented limit, also where
  // they are split or wider
  if (sizeof(Cx<RS>) * (size_t)ntmax * PCG_CHUNK > pcg_column_limit(sizeof(RS), std::max(128, eng))) return QEDF_ERR_SIZE;
  // the elementwise phase wants four warps; the engine's records need `eng`
  const int threads = std::max(128, eng);
  p.eng_threads = eng;
  const size_t smem = RhsState<!std::is_same<RS, RH>::value, std::is_same<SP, __half>::value>::bytes(p.nrhs) +
                      pcg_phase_smem<RS, RH, SP, BY>(eng, rows, p.CH);
  // beside the kernel's static shared memory: red, ctl and oprun
  constexpr size_t fixed = (64 * sizeof(double) + sizeof(PcgCtl) + sizeof(OpRun<RS, A, SP>) + 127) / 128 * 128;
  if (smem + fixed > 227 * 1024) return QEDF_ERR_SIZE;
  auto kern = k_pcg<RS, RH, A, SP, BY>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return QEDF_ERR_CUDA;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess || per_sm < 1)
    return QEDF_ERR_SIZE;
  // one block per slice is the most that has work in the operator phase
  const int64_t most = (int64_t)num_sms() * std::min(per_sm, PCG_MAX_PER_SM);
  const int nblk = (int)std::max<int64_t>(1, std::min<int64_t>(most, std::max(slices, units)));
  return pcg_launch_kernel(reinterpret_cast<const void*>(kern), p, taps, threads, smem, nblk, st);
}

template <typename RS, typename RH, typename A, typename SP>
static int launch_pcg_by(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st) {
  switch (by) {
    case 2: return launch_pcg_t<RS, RH, A, SP, 2>(p, taps, st);
    case 4: return launch_pcg_t<RS, RH, A, SP, 4>(p, taps, st);
    case 6: return launch_pcg_t<RS, RH, A, SP, 6>(p, taps, st);
  }
  return QEDF_ERR_ARG;
}

// one translation unit per mode instantiates its kernels
int launch_pcg_f32(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st);
int launch_pcg_f64(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st);
int launch_pcg_mixed(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st);
int launch_pcg_bf16(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st);
int launch_pcg_f16(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st);

}  // namespace qedf
