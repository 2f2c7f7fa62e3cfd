// Operator, preconditioner, force, boson and reduction kernels of the
// qed_fermion B200 library, plus their host launchers.
//
// Layouts (all contiguous):
//   vectors  [nvec][Nt][L][L]    complex (re, im interleaved)
//   angles   [nphi][Nt][L][L][2] real, component 0 = x-bond, 1 = y-bond
//   forces   same as angles
#include <algorithm>
#include <cstdio>
#include <type_traits>

#include "qedf_internal.h"
#include "qedf_slice.cuh"

namespace qedf {

// ============================================================================
// M, M^dagger, M^dagger M
// ============================================================================
//
// With x_t the slices of the input and sigma_t = +1 (t < Nt-1) or -1
// (t = Nt-1):
//   (M x)_t      = x_t - sigma_{t-1} B_{t-1} x_{t-1}
//   (M^dag y)_t  = y_t - sigma_t B_t y_{t+1}
//   (M^dag M x)_t: y = M x is produced slice by slice in registers and M^dag
//                  applied to it, so x is read once and one extra slice of y
//                  (the run's lower halo) is recomputed.
// The slices of all right-hand sides form one line that is cut into one
// contiguous run per block (block_run), so every SM gets the same number of
// slices; with a slab length, a run is one slab instead.  Measured with the
// engine of qedf_slice.cuh at 8 right-hand sides, L = 48, Ltau = 480: 60 us
// complex64 (72 with fixed slabs and one block per SM) and 191 us complex128
// (328); the algorithmic bytes take 32 and 65 us at the copy bandwidth.  What
// is left is issue slots (52 % busy) and shared-memory wavefronts (44 %); in
// double precision the FP64 pipe, half of it for the phases' sincos.
//
// CFG_TALL (double precision, tall tiles with many threads): the phases live
// in the thread's record, there is one exchange buffer, and y_t waits in z's
// own slice instead of a stash, so that 384 or 512 threads fit in shared
// memory and registers.  2 x 2 double tiles also leave y_t in z, and fetch the
// next slice's angles by cp.async into the stash instead (185 against 189 us at
// L = 48, 95 against 107 at L = 36: no spills; in single precision the same
// costs 8 to 15 %, the shared-memory pipe being the busy one there).
enum { CFG_REG = 0, CFG_TALL = 1 };

// threads and resident blocks that an operator kernel is compiled for
template <typename R, int BY, int CFG>
struct OpT {
  // 2 x 4 double tiles keep 168 registers (384 threads) unless CFG_TALL
  static constexpr int threads = (sizeof(R) == 8 && BY == 4 && CFG == CFG_REG) ? 384 : MaxT<R, BY>::value;
  static constexpr int min_blocks = MaxT<R, BY>::min_blocks;
};

// first and one-past-last global slice (right-hand side * Nt + t) of a block
__device__ __forceinline__ void block_run(int bs, int Nt, int T, int64_t& w0, int64_t& w1) {
  if (T > 0) {
    const int per = (Nt + T - 1) / T, rb = blockIdx.x / per, k = blockIdx.x % per;
    w0 = (int64_t)rb * Nt + (int64_t)k * T;
    w1 = min(w0 + T, (int64_t)(rb + 1) * Nt);
  } else {
    const int64_t W = (int64_t)bs * Nt;
    w0 = W * blockIdx.x / gridDim.x;
    w1 = W * (blockIdx.x + 1) / gridDim.x;
  }
}

template <typename R, typename A, int BY, int OP, int CFG>
__global__ void __launch_bounds__(OpT<R, BY, CFG>::threads, OpT<R, BY, CFG>::min_blocks) k_operator(OpArgs p) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr bool TALL = CFG == CFG_TALL;
  // angles of the next slice wait in registers where these allow it
  constexpr bool PF = sizeof(R) == 4 && BY >= 4;
  using Eng = Slice<R, BY, TALL, TALL ? 1 : 2>;
  Eng S;
  S.init(p.L, smem, threadIdx.x);
  // where y_t and the next slice's angles wait (OP_MHM; see above)
  constexpr bool STAGE = OP == OP_MHM && sizeof(R) == 8 && BY == 2;
  constexpr bool IN_Z = TALL || STAGE;
  Stash<R, BY> st;
  if constexpr (OP == OP_MHM && !TALL) st.init(smem + slice_smem<R>(blockDim.x, Eng::REC), threadIdx.x);
  const size_t sv = 2 * (size_t)p.L * p.L;  // reals per slice (vector and angles)
  const R t1 = (R)p.t1, th = (R)p.th, Cb = (R)p.Cb;
  const int Nt = p.Nt;
  int64_t w, w1;
  block_run(p.bs, Nt, p.T, w, w1);
  while (w < w1) {
    const int rb = (int)(w / Nt), a = (int)(w - (int64_t)rb * Nt), b = (int)min((int64_t)Nt, a + (w1 - w));
    w += b - a;
    const A* phi = reinterpret_cast<const A*>(p.phi) + (size_t)(rb / p.rhs_per_phi) * Nt * sv;
    const R* x = reinterpret_cast<const R*>(p.x) + (size_t)rb * Nt * sv;
    R* z = reinterpret_cast<R*>(p.z) + (size_t)rb * Nt * sv;
    Cx<R> X0[BY][2], X1[BY][2];
    A ang[BY][4];
    if constexpr (OP == OP_M) {
      int tp = a == 0 ? Nt - 1 : a - 1;
      S.load(X0, x + tp * sv);
      if (PF) S.load_angles(ang, phi + tp * sv);
      for (int t = a; t < b; ++t) {
        if (!PF) S.load_angles(ang, phi + tp * sv);
        S.load(X1, x + t * sv);
        S.phases(ang, t1, th);
        if (PF && t + 1 < b) S.load_angles(ang, phi + t * sv);
        if ((t - a) & 1) S.template applyB<1>(X0);
        else S.template applyB<0>(X0);
        axpy_blk<R, BY>(X0, X1, sigma_of<R>(tp, Nt) * Cb, X0);
        S.store(z + t * sv, X0);
        copy_blk<R, BY>(X0, X1);
        tp = t;
      }
    } else if constexpr (OP == OP_MH) {
      if constexpr (sizeof(R) == 8) {
        // from the run's last slice down, so that one tile waits while B is applied, as
        // for M; upwards x_t and x_{t+1} both do (L = 28, 8 vectors: 39.3 -> 33.0 us)
        S.load(X0, x + (b == Nt ? 0 : b) * sv);
        for (int t = b - 1; t >= a; --t) {
          S.load_angles(ang, phi + t * sv);
          S.load(X1, x + t * sv);
          S.phases(ang, t1, th);
          if ((b - 1 - t) & 1) S.template applyB<1>(X0);
          else S.template applyB<0>(X0);
          axpy_blk<R, BY>(X0, X1, sigma_of<R>(t, Nt) * Cb, X0);
          S.store(z + t * sv, X0);
          copy_blk<R, BY>(X0, X1);
        }
      } else {
        S.load(X0, x + a * sv);
        if (PF) S.load_angles(ang, phi + a * sv);
        for (int t = a; t < b; ++t) {
          const int tn = t + 1 == Nt ? 0 : t + 1;
          if (!PF) S.load_angles(ang, phi + t * sv);
          S.load(X1, x + tn * sv);
          S.phases(ang, t1, th);
          if (PF && t + 1 < b) S.load_angles(ang, phi + (t + 1) * sv);
          Cx<R> Y[BY][2];
          copy_blk<R, BY>(Y, X1);
          if ((t - a) & 1) S.template applyB<1>(Y);
          else S.template applyB<0>(Y);
          axpy_blk<R, BY>(Y, X0, sigma_of<R>(t, Nt) * Cb, Y);
          S.store(z + t * sv, Y);
          copy_blk<R, BY>(X0, X1);
        }
      }
    } else {  // OP_MHM
      Cx<R> Y[BY][2];
      const int tp = a == 0 ? Nt - 1 : a - 1;
      S.load(X0, x + tp * sv);
      S.load_angles(ang, phi + tp * sv);
      S.load(X1, x + a * sv);
      S.phases(ang, t1, th);
      if (PF) S.load_angles(ang, phi + a * sv);
      if constexpr (STAGE) S.fetch_angles(st, phi + a * sv);
      S.template applyB<0>(X0);
      axpy_blk<R, BY>(Y, X1, sigma_of<R>(tp, Nt) * Cb, X0);  // y_a
      if constexpr (IN_Z) S.store(z + a * sv, Y); else st.park(Y);
      copy_blk<R, BY>(X0, X1);
      for (int t = a; t < b; ++t) {
        const int tn = t + 1 == Nt ? 0 : t + 1;
        if constexpr (STAGE) S.take_angles(ang, st);
        else if (!PF) S.load_angles(ang, phi + t * sv);
        S.load(X1, x + tn * sv);
        S.phases(ang, t1, th);
        if (t + 1 < b) {
          if constexpr (STAGE) S.fetch_angles(st, phi + (t + 1) * sv);
          else if (PF) S.load_angles(ang, phi + (t + 1) * sv);
        }
        const R sg = sigma_of<R>(t, Nt) * Cb;
        S.template applyB<1>(X0);             // B_t x_t
        axpy_blk<R, BY>(Y, X1, sg, X0);       // y_{t+1}
        if constexpr (IN_Z) {
          if (t + 1 < b) S.store(z + (t + 1) * sv, Y);
        } else {
          st.unpark(X0);                      // y_t
          st.park(Y);
        }
        S.template applyB<0>(Y);              // B_t y_{t+1}
        if constexpr (IN_Z) S.load_st(X0, z + t * sv);
        axpy_blk<R, BY>(Y, X0, sg, Y);        // z_t = y_t - sigma_t B_t y_{t+1}
        S.store(z + t * sv, Y);
        copy_blk<R, BY>(X0, X1);
      }
    }
    // the next run's first factor uses buffer 0, as may this run's last
    __syncthreads();
  }
}

// ============================================================================
// b_vec_per_tau: B_t v or its six partial products, one slice
// ============================================================================
template <typename R, typename A, int BY>
__global__ void __launch_bounds__(MaxT<R, BY>::value, 1) k_bvec(BvecArgs p) {
  extern __shared__ __align__(16) unsigned char smem[];
  Slice<R, BY> S;
  S.init(p.L, smem, threadIdx.x);
  const size_t sv = 2 * (size_t)p.L * p.L;
  const R* v = reinterpret_cast<const R*>(p.v) + blockIdx.x * sv;
  R* out = reinterpret_cast<R*>(p.out) + blockIdx.x * sv * (p.interm ? 6 : 1);
  Cx<R> W[BY][2];
  S.load(W, v);
  S.phases_of(reinterpret_cast<const A*>(p.phi), (R)p.t1, (R)p.th);
  R scale = 1;  // the product of the applied factors' cosh
  auto put = [&](R* to) {
    if (!S.on) return;
#pragma unroll
    for (int r = 0; r < BY; ++r) st2(to + S.off + r * S.rs, scale * W[r][0], scale * W[r][1]);
  };
  const R c1 = (R)p.c1, ch = (R)p.ch;
  S.template factor<3, 0>(W);
  scale *= ch;
  if (p.interm) put(out);
  S.template factor<2, 1>(W);
  scale *= ch;
  if (p.interm) put(out + 1 * sv);
  S.template factor<1, 0>(W);
  scale *= ch;
  if (p.interm) put(out + 2 * sv);
  S.template factor<0, 1>(W);
  scale *= c1;
  if (p.interm) put(out + 3 * sv);
  S.template factor<1, 0>(W);
  scale *= ch;
  if (p.interm) put(out + 4 * sv);
  S.template factor<2, 1>(W);
  scale *= ch;
  if (p.interm) {
    put(out + 5 * sv);
  } else {
    S.template factor<3, 0>(W);
    scale *= ch;
    put(out);
  }
}

// ============================================================================
// preconditioner z = (P_tau (x) I) r, P_tau given as a tau-space CSR matrix
// ============================================================================
//
// A warp forms C consecutive output rows of 32 sites; a block's warps take
// neighbouring segments of tau, whose common rows meet in L1.  The C + 2H rows
// of r that a banded P_tau needs are all loaded at once, into registers, while
// the warp finds out which of three forms each row of its segment has:
// * the middle CSR row (t = Ltau/2) shifted along tau - taps t-H .. t+H with the
//   same values, as in the bulk: registers only, with the taps as constants;
// * up to 2H+1 entries within t-H .. t+H in ascending order: registers too, with
//   the row's own taps from shared memory, absent ones left out;
// * any other: dealt to all warps of the block, which run over the CSR row 32
//   entries at a time, the next ones on their way; from shared memory an
//   entry is one broadcast where shuffles took two or three.
// All orders of summation are the CSR order, so the forms agree bit for bit.
// What is left is loads in flight against the 60 MB of the first size below.
// Device times, us, 8 vectors: with columns staged in shared memory, with the first
// and the last form alone and shuffled entries, and now.  The builtin matrix, L = 36,
// Ltau = 359: complex64 27.0, 17.6, 15.6, complex128 49.4, 34.5, 30.4; L = 48, Ltau =
// 480, complex64: 50.9, 41.9, 38.3; there a diagonal 56.8, 112, 41.1, three taps
// 67.0, 113, 42.0, 41 taps 256, 327, 235, a dense matrix 3211, 3085, 2421.  With the
// rows of r asked for before the entries, a quarter more: a load that depends on
// another one waits for both behind the queue.  Four warps to a block: with
// eight, a fifth more, the blocks' last wave being emptier.
template <typename R>
struct Tap;  // a real tap times a complex number
template <>
struct Tap<float> {
  static constexpr int ROWS = 16;
  using V = float2;
  struct __align__(8) Entry {
    float v;
    int c;
  };
  unsigned long long c;  // the tap twice: one instruction for both parts
  __device__ __forceinline__ explicit Tap(float t) { asm("mov.b64 %0, {%1, %1};" : "=l"(c) : "f"(t)); }
  __device__ __forceinline__ V fma(V q, V a) const {
    unsigned long long qa = *reinterpret_cast<unsigned long long*>(&q), aa = *reinterpret_cast<unsigned long long*>(&a);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(aa) : "l"(c), "l"(qa));
    return *reinterpret_cast<V*>(&aa);
  }
};
template <>
struct Tap<double> {
  static constexpr int ROWS = 8;
  using V = double2;
  struct __align__(16) Entry {
    double v;
    int c;
  };
  double c;
  __device__ __forceinline__ explicit Tap(double t) : c(t) {}
  __device__ __forceinline__ V fma(V q, V a) const { return make_double2(::fma(c, q.x, a.x), ::fma(c, q.y, a.y)); }
};

constexpr int PRE_H = 6;      // half-width of the banded form (13 taps, the builtin P_tau)
constexpr int PRE_WARPS = 4;  // segments of tau per block

template <typename R>
__global__ void __launch_bounds__(32 * PRE_WARPS, 4) k_precon(PreconArgs p) {
  using V = typename Tap<R>::V;
  constexpr int H = PRE_H, C = Tap<R>::ROWS, TAPS = 2 * H + 1;
  constexpr unsigned ALL = 0xffffffffu;
  using Entry = typename Tap<R>::Entry;
  __shared__ unsigned odd[PRE_WARPS];  // rows of the last form
  __shared__ R taps[PRE_WARPS][C][TAPS];  // of rows of the second form
  __shared__ __align__(16) Entry entries[PRE_WARPS][2][32];
  const int Vs = p.L * p.L, Nt = p.Nt, nchunk = (Vs + 31) / 32;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t rb = blockIdx.x / nchunk;
  const int s = (blockIdx.x % nchunk) * 32 + lane;
  const bool on = s < Vs;
  const V* r = reinterpret_cast<const V*>(p.r) + rb * Nt * Vs + (on ? s : Vs - 1);
  V* z = reinterpret_cast<V*>(p.z) + rb * Nt * Vs + s;
  // the ends of tau, which take longer, first
  const int b0 = (blockIdx.y == 0 ? gridDim.y - 1 : blockIdx.y - 1) * (PRE_WARPS * C), t0 = b0 + w * C;
  // the segment's entries, asked for before the rows of r, behind which they would queue:
  // if each of its rows has TAPS of them, entry lane + 32 n is tap i of row g
  constexpr int NE = (C * TAPS + 31) / 32;
  const int rows = min(max(Nt - t0, 0), C);
  const int km = p.row_ptr[Nt / 2], k0 = p.row_ptr[min(t0, Nt)], kl = p.row_ptr[min(t0 + min(lane, C), Nt)];
  const bool full = rows > 0 && p.row_ptr[Nt / 2 + 1] - km == TAPS && __all_sync(ALL, lane > rows || kl == k0 + TAPS * lane);
  double vm = 0, ve[NE];
  int cm = 0, ce[NE];
  if (full) {
    vm = p.val[km + min(lane, TAPS - 1)];
    cm = p.col[km + min(lane, TAPS - 1)];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int k = k0 + min(32 * e + lane, TAPS * rows - 1);
      ve[e] = p.val[k];
      ce[e] = p.col[k];
    }
  }
  V q[C + 2 * H];
  if (t0 >= H && t0 + C + H <= Nt) {
    const V* r0 = r + (int64_t)(t0 - H) * Vs;
#pragma unroll
    for (int k = 0; k < C + 2 * H; ++k) q[k] = r0[(int64_t)k * Vs];
  } else {  // (rows outside tau are not used: a row that is the middle row shifted has none)
#pragma unroll
    for (int k = 0; k < C + 2 * H; ++k) q[k] = r[(int64_t)min(max(t0 - H + k, 0), Nt - 1) * Vs];
  }
  unsigned mask = 0;
  if (full) {
    int i = lane % TAPS, g = lane / TAPS;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const double want = __shfl_sync(ALL, vm, i);  // (all lanes)
      if (ce[e] != t0 + g - H + i || ve[e] != want) mask |= 1u << g;
      i += 32 % TAPS;
      g += 32 / TAPS;
      if (i >= TAPS) i -= TAPS, ++g;
    }
    mask = __reduce_or_sync(ALL, mask);
    mask = __all_sync(ALL, lane >= TAPS || cm == Nt / 2 - H + lane) ? ~mask & ((1u << rows) - 1) : 0u;
    // (taps reach outside tau in the first and last H rows)
    if (t0 < H) mask &= ALL << (H - t0);
    if (t0 + C > Nt - H) mask &= t0 < Nt - H ? (1u << (Nt - H - t0)) - 1 : 0u;
  }
  // rows whose own taps lie within H slices
  const unsigned rest = ~mask & ((1u << rows) - 1);
  unsigned near = 0, have = 0;
  if (rest) {
    constexpr int PARTS = 32 / C, PER = (TAPS + PARTS - 1) / PARTS;  // lanes to a row, entries to a lane
    const int g = lane % C, part = lane / C;
    const int kg = __shfl_sync(ALL, kl, g), ng = __shfl_sync(ALL, kl, g + 1) - kg;
    bool ok = (rest >> g & 1) && ng <= TAPS;
    int off[PER];
    double v[PER];
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      const int i = part * PER + n;
      off[n] = -1;
      if (ok && i < ng) {
        off[n] = p.col[kg + i];
        v[n] = p.val[kg + i];
      }
    }
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      if (!ok || part * PER + n >= ng) continue;
      const bool in = (unsigned)off[n] < (unsigned)Nt;
      off[n] -= t0 + g - H;
      ok = in && (unsigned)off[n] < (unsigned)TAPS;
      if (!ok) continue;
      have |= 1u << off[n];
      taps[w][g][off[n]] = (R)v[n];
    }
#pragma unroll
    for (int o = C; o < 32; o *= 2) have |= __shfl_xor_sync(ALL, have, o);
    // ascending: as many of the row's entries lie below each as precede it
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      const int i = part * PER + n;
      if (ok && i < ng) ok = __popc(have & ((1u << off[n]) - 1)) == i;
    }
    ok = ok && __popc(have) == ng;
    near = __ballot_sync(ALL, ok);
#pragma unroll
    for (int o = C; o < 32; o *= 2) near &= near >> o;
    near &= rest;
    __syncwarp();
  }
  if (lane == 0) odd[w] = rest & ~near;
  if (mask) {
    const R vr = (R)vm;
    R c[TAPS];
#pragma unroll
    for (int k = 0; k < TAPS; ++k) c[k] = __shfl_sync(ALL, vr, k);
    V* z0 = z + (int64_t)t0 * Vs;
#pragma unroll
    for (int i = 0; i < C; ++i) {
      if (!(mask >> i & 1)) continue;
      V acc = {0, 0};
#pragma unroll
      for (int k = 0; k < TAPS; ++k) acc = Tap<R>(c[k]).fma(q[i + k], acc);
      if (on) __stcg(z0 + (int64_t)i * Vs, acc);
    }
  }
  if (near) {
    V* z0 = z + (int64_t)t0 * Vs;
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const unsigned h = __shfl_sync(ALL, have, i);
      if (!(near >> i & 1)) continue;
      V acc = {0, 0};
#pragma unroll
      for (int k = 0; k < TAPS; ++k)
        if (h >> k & 1) acc = Tap<R>(taps[w][i][k]).fma(q[i + k], acc);
      if (on) __stcg(z0 + (int64_t)i * Vs, acc);
    }
  }
  __syncthreads();
  // this warp's rows of the last form, one per lane: the block's w-th, (w + PRE_WARPS)-th ...
  int mine = -1, left = w + PRE_WARPS * lane;
#pragma unroll
  for (int g = 0; g < PRE_WARPS; ++g) {
    unsigned m = odd[g];
    const int n = __popc(m);
    if (mine < 0 && left < n) {
      for (int k = 0; k < left; ++k) m &= m - 1;
      mine = g * C + __ffs(m) - 1;
    }
    left -= n;
  }
  const int own = __popc(__ballot_sync(ALL, mine >= 0));  // (at most C)
  if (!own) return;
  int first = 0, end = 0;
  if (mine >= 0) {
    first = p.row_ptr[b0 + mine];
    end = p.row_ptr[b0 + mine + 1];
  }
  int cl = -1, buf = 0;
  R vl = 0;
  auto ask = [&](int k, int k1) {  // entries k .. k + 31 below k1
    cl = -1;
    if (k + lane < k1) {
      cl = p.col[k + lane];
      vl = (R)p.val[k + lane];
    }
  };
  ask(__shfl_sync(ALL, first, 0), __shfl_sync(ALL, end, 0));
  for (int j = 0; j < own; ++j) {
    int k = __shfl_sync(ALL, first, j);
    const int k1 = __shfl_sync(ALL, end, j), t = b0 + __shfl_sync(ALL, mine, j);
    const int kn = __shfl_sync(ALL, first, min(j + 1, own - 1)), kn1 = j + 1 < own ? __shfl_sync(ALL, end, j + 1) : 0;
    V acc = {0, 0};
    do {
      // (two buffers: the one before this is read by all once they meet here)
      entries[w][buf][lane] = {vl, cl};
      // (a lane without an entry has column -1)
      const bool inside = __all_sync(ALL, (unsigned)cl < (unsigned)Nt || k + lane >= k1);
      __syncwarp();
      constexpr int N = 16 / sizeof(Entry);  // entries to an access
      struct __align__(16) Entries {
        Entry e[N];
      };
      const Entries* en = reinterpret_cast<const Entries*>(entries[w][buf]);
      buf ^= 1;
      const int n = min(32, k1 - k);
      k += 32;
      if (k < k1) ask(k, k1);
      else ask(kn, kn1);
      auto add = [&](auto count, auto check, int e) {  // entries e .. e + count - 1
        constexpr int M = decltype(count)::value;
        constexpr bool CHECK = decltype(check)::value;
        V qe[M];
        Entries x[M / N];
#pragma unroll
        for (int i = 0; i < M; ++i) {
          if (i % N == 0) x[i / N] = en[(e + i) / N];
          const unsigned c = x[i / N].e[i % N].c;
          qe[i] = r[(int64_t)(CHECK ? min(c, (unsigned)Nt - 1) : c) * Vs];
        }
#pragma unroll
        for (int i = 0; i < M; ++i) {
          const Entry& q = x[i / N].e[i % N];
          const V next = Tap<R>(q.v).fma(qe[i], acc);
          if (!CHECK || (unsigned)q.c < (unsigned)Nt) acc = next;  // else: outside the matrix
        }
      };
      int e = 0;
      if (inside)
        for (; n - e >= 8; e += 8) add(std::integral_constant<int, 8>(), std::false_type(), e);
      for (; n - e > 4; e += 8) add(std::integral_constant<int, 8>(), std::true_type(), e);
      if (e < n) add(std::integral_constant<int, 4>(), std::true_type(), e);
    } while (k < k1);
    if (on) __stcg(z + (int64_t)t * Vs, acc);
  }
}

// ============================================================================
// fermion force  F = -dS_f/dphi,  S_f = psi^dag (M^dag M)^{-1} psi,  given xi
// ============================================================================
//
// Per slice t (right vector R = xi_t, left vector u = B_t xi_t - sigma_t
// xi_{t+1} = -sigma_t (M xi)_{t+1}):
//   F(bond of group g) = 2 Re sum_{k: F_g at position k of B}
//                          l_{k-1}^dag dF_g/dphi R_{7-k}
// where R_m is xi_t after the m rightmost factors and l_k is u after the k
// leftmost factors (F_g Hermitian).  R_7 = B xi_t is produced forward; the
// R_m needed afterwards are recovered backwards with F_g^{-1} = c (I - tK)
// while l is advanced forwards, so no partial product is stored.  This is the
// sum that the reference evaluates with explicit partial products
// (force_f_fast, hmc_sampler_batch.py:2150-2227; force_f_sparse :2230-2330).
//
// Unlike the operators, the force exchanges plain values and its bonds' phases
// (once per slice, in the record's last entries) and applies the factors with
// their scalars: every rounding is then that of the textbook update of each
// site, so that trajectories in single precision, whose energies show a change
// of the last bit of the force at 1e-9, do not depend on the tiling.  Every
// slice is independent of the others: the slices of all right-hand sides are
// dealt as block_run does.  Measured, 2 right-hand sides at L = 48, Ltau = 480,
// complex64: 35 us, against 39 with fixed slabs and one block per SM.
template <typename R, int BY>
struct ForceT {
  static constexpr int threads = MaxT<R, BY>::value;
};

template <typename R, int BY>
struct ForceSlice : Slice<R, BY, false, 2, 2, BY + 2> {
  using Base = Slice<R, BY, false, 2, 2, BY + 2>;
  static constexpr int PHX = Base::PH0, PHY = PHX + BY;  // x-bond phases of column x0+1, y-bond ones of the last row
  R c1, ch;

  // makes the phases that the neighbours need visible at the next barrier
  __device__ __forceinline__ void publish() {
#pragma unroll
    for (int r = 0; r < BY; ++r) this->me[PHX + r] = this->px(r, 1);
    this->me[PHY] = this->py(BY - 1, 0);
    this->me[PHY + 1] = this->py(BY - 1, 1);
  }
  // v_i + a v_j and v_j + conj(a) v_i, times c
  __device__ static __forceinline__ Cx<R> upd(R c, Cx<R> a, Cx<R> vj, Cx<R> vi) { return c * cfma(a, vj, vi); }
  __device__ static __forceinline__ Cx<R> updj(R c, Cx<R> a, Cx<R> vi, Cx<R> vj) { return c * cjfma(a, vi, vj); }

  // v <- F_g v, plain values exchanged
  template <int G, int BUF>
  __device__ __forceinline__ void factor_true(Cx<R> (&v)[BY][2]) {
    constexpr int B0 = BUF * 2 * BY;
    const R c = G == 0 ? c1 : ch;
    Cx<R>* me = this->me;
    auto local = [&](Cx<R>& vi, Cx<R>& vj, Cx<R> a) {
      const Cx<R> oi = vi, oj = vj;
      vi = upd(c, a, oj, oi);
      vj = updj(c, a, oi, oj);
    };
    if constexpr (G == 0 || G == 2) {
      constexpr int RC = G == 0 ? 1 : 0;
#pragma unroll
      for (int r = RC; r < BY; r += 2) {
        me[B0 + (r & ~1)] = v[r][0];
        me[B0 + (r & ~1) + 1] = v[r][1];
      }
#pragma unroll
      for (int r = 1 - RC; r < BY; r += 2) local(v[r][0], v[r][1], this->px(r, 0));
      __syncthreads();
#pragma unroll
      for (int r = RC; r < BY; r += 2) {
        v[r][1] = upd(c, this->px(r, 1), this->rt[B0 + (r & ~1)], v[r][1]);
        v[r][0] = updj(c, this->lf[PHX + r], this->lf[B0 + (r & ~1) + 1], v[r][0]);
      }
    } else {
      constexpr int CL = (G == 1) ? 0 : 1, CC = 1 - CL;
      me[B0] = v[0][CC];
      me[B0 + 1] = v[BY - 1][CC];
#pragma unroll
      for (int r = 0; r < BY; r += 2) local(v[r][CL], v[r + 1][CL], this->py(r, CL));
#pragma unroll
      for (int r = 1; r + 1 < BY; r += 2) local(v[r][CC], v[r + 1][CC], this->py(r, CC));
      __syncthreads();
      v[BY - 1][CC] = upd(c, this->py(BY - 1, CC), this->dn[B0], v[BY - 1][CC]);
      v[0][CC] = updj(c, this->up[PHY + CC], this->up[B0 + 1], v[0][CC]);
    }
  }

  // term for one bond: 2 c Re[conj(l_i) (i a) R_j + conj(l_j) conj(i a) R_i]
  __device__ static __forceinline__ R term(Cx<R> li, Cx<R> lj, Cx<R> Ri, Cx<R> Rj, Cx<R> a, R c) {
    const Cx<R> ia = mk<R>(-a.im, a.re);
    const Cx<R> u = cjmul(li, cmul(ia, Rj));
    const Cx<R> w = cjmul(lj, cjmul(ia, Ri));
    return (R)2 * c * (u.re + w.re);
  }
  // a bond inside the tile
  __device__ static __forceinline__ void local(Cx<R>& Ri, Cx<R>& Rj, Cx<R>& li, Cx<R>& lj, Cx<R> a, R c, R& F) {
    const Cx<R> nRi = upd(c, cneg(a), Rj, Ri), nRj = updj(c, cneg(a), Ri, Rj);
    F += term(li, lj, nRi, nRj, a, c);
    const Cx<R> oi = li, oj = lj;
    li = upd(c, a, oj, oi);
    lj = updj(c, a, oi, oj);
    Ri = nRi;
    Rj = nRj;
  }
  // the owner's side of a cross bond: i is its own site, j the neighbour's
  __device__ static __forceinline__ void edge(Cx<R>& Ri, Cx<R>& li, Cx<R> Rj, Cx<R> lj, Cx<R> a, R c, R& F) {
    const Cx<R> nRi = upd(c, cneg(a), Rj, Ri), nRj = updj(c, cneg(a), Ri, Rj);
    F += term(li, lj, nRi, nRj, a, c);
    li = upd(c, a, lj, li);
    Ri = nRi;
  }
  // the other side: j is its own site
  __device__ static __forceinline__ void far(Cx<R>& Rj, Cx<R>& lj, Cx<R> Ri, Cx<R> li, Cx<R> a, R c) {
    Rj = updj(c, cneg(a), Ri, Rj);
    lj = updj(c, a, li, lj);
  }

  // one factor position: R <- F_g^{-1} R, accumulate the force, l <- F_g l
  template <int G, int BUF>
  __device__ __forceinline__ void step(Cx<R> (&Rv)[BY][2], Cx<R> (&l)[BY][2], R (&Fx)[BY][2], R (&Fy)[BY][2]) {
    constexpr int B0 = BUF * 2 * BY, B1 = B0 + BY;  // exchange slots of R and l
    const R c = G == 0 ? c1 : ch;
    Cx<R>* me = this->me;
    if constexpr (G == 0 || G == 2) {
      constexpr int RC = G == 0 ? 1 : 0;
#pragma unroll
      for (int r = RC; r < BY; r += 2) {
        const int q = r & ~1;
        me[B0 + q] = Rv[r][0];
        me[B0 + q + 1] = Rv[r][1];
        me[B1 + q] = l[r][0];
        me[B1 + q + 1] = l[r][1];
      }
#pragma unroll
      for (int r = 1 - RC; r < BY; r += 2)
        local(Rv[r][0], Rv[r][1], l[r][0], l[r][1], this->px(r, 0), c, Fx[r][0]);
      __syncthreads();
#pragma unroll
      for (int r = RC; r < BY; r += 2) {
        const int q = r & ~1;
        edge(Rv[r][1], l[r][1], this->rt[B0 + q], this->rt[B1 + q], this->px(r, 1), c, Fx[r][1]);
        far(Rv[r][0], l[r][0], this->lf[B0 + q + 1], this->lf[B1 + q + 1], this->lf[PHX + r], c);
      }
    } else {
      constexpr int CL = (G == 1) ? 0 : 1, CC = 1 - CL;
      me[B0] = Rv[0][CC];
      me[B0 + 1] = Rv[BY - 1][CC];
      me[B1] = l[0][CC];
      me[B1 + 1] = l[BY - 1][CC];
#pragma unroll
      for (int r = 0; r < BY; r += 2)
        local(Rv[r][CL], Rv[r + 1][CL], l[r][CL], l[r + 1][CL], this->py(r, CL), c, Fy[r][CL]);
#pragma unroll
      for (int r = 1; r + 1 < BY; r += 2)
        local(Rv[r][CC], Rv[r + 1][CC], l[r][CC], l[r + 1][CC], this->py(r, CC), c, Fy[r][CC]);
      __syncthreads();
      edge(Rv[BY - 1][CC], l[BY - 1][CC], this->dn[B0], this->dn[B1], this->py(BY - 1, CC), c, Fy[BY - 1][CC]);
      far(Rv[0][CC], l[0][CC], this->up[B0 + 1], this->up[B1 + 1], this->up[PHY + CC], c);
    }
  }
};

template <typename R, typename A, int BY>
__global__ void __launch_bounds__(ForceT<R, BY>::threads, 1) k_force(ForceArgs p) {
  extern __shared__ __align__(16) unsigned char smem[];
  ForceSlice<R, BY> S;
  S.init(p.L, smem, threadIdx.x);
  const size_t sv = 2 * (size_t)p.L * p.L;
  const int Nt = p.Nt;
  const R t1 = (R)p.t1, th = (R)p.th;
  S.c1 = (R)p.c1;
  S.ch = (R)p.ch;
  int64_t w, w1;
  block_run(p.bs, Nt, p.T, w, w1);
  for (; w < w1; ++w) {
    const int rb = (int)(w / Nt), t = (int)(w - (int64_t)rb * Nt), tn = t + 1 == Nt ? 0 : t + 1;
    const A* phi = reinterpret_cast<const A*>(p.phi) + (size_t)(rb / p.rhs_per_phi) * Nt * sv;
    const R* xi = reinterpret_cast<const R*>(p.xi) + (size_t)rb * Nt * sv;
    A* F = reinterpret_cast<A*>(p.F) + ((size_t)rb * Nt + t) * sv;
    Cx<R> Rv[BY][2], l[BY][2];
    S.load(Rv, xi + t * sv);
    S.phases_of(phi + t * sv, t1, th);
    S.load(l, xi + tn * sv);
    S.publish();
    S.template factor_true<3, 0>(Rv);  // R_7 = B_t xi_t
    S.template factor_true<2, 1>(Rv);
    S.template factor_true<1, 0>(Rv);
    S.template factor_true<0, 1>(Rv);
    S.template factor_true<1, 0>(Rv);
    S.template factor_true<2, 1>(Rv);
    S.template factor_true<3, 0>(Rv);
    axpy_blk<R, BY>(l, Rv, sigma_of<R>(t, Nt), l);
    R Fx[BY][2], Fy[BY][2];
#pragma unroll
    for (int r = 0; r < BY; ++r) Fx[r][0] = Fx[r][1] = Fy[r][0] = Fy[r][1] = 0;
    // positions k = 1..7 of B = F4 F3 F2 F1 F2 F3 F4
    S.template step<3, 1>(Rv, l, Fx, Fy);
    S.template step<2, 0>(Rv, l, Fx, Fy);
    S.template step<1, 1>(Rv, l, Fx, Fy);
    S.template step<0, 0>(Rv, l, Fx, Fy);
    S.template step<1, 1>(Rv, l, Fx, Fy);
    S.template step<2, 0>(Rv, l, Fx, Fy);
    S.template step<3, 1>(Rv, l, Fx, Fy);
    if (S.on) {
#pragma unroll
      for (int r = 0; r < BY; ++r) {
        A o[4] = {(A)Fx[r][0], (A)Fy[r][0], (A)Fx[r][1], (A)Fy[r][1]};
        st4(F + S.off + r * S.rs, o);
      }
    }
    __syncthreads();  // the phases of this slice are read
  }
}

// ============================================================================
// boson action / force (layout [bs][Nt][L][L][2])
// ============================================================================
template <typename A>
__device__ __forceinline__ A curl_at(const A* ph, int L, int x, int y) {
  const int xp = (x + 1) % L, yp = (y + 1) % L;
  return ph[2 * (x + L * y)] + ph[2 * (xp + L * y) + 1] - ph[2 * (x + L * yp)] - ph[2 * (x + L * y) + 1];
}

// F_b = -d(S_plaq + S_tau)/dphi at every bond
template <typename A>
__device__ __forceinline__ void boson_force_site(const A* phi, int L, int Nt, int t, int x, int y, A K,
                                                 A ctau, int compact, A& fx, A& fy) {
  const size_t sv = 2 * (size_t)L * L;
  const A* ph = phi + t * sv;
  const A sc = sin(curl_at(ph, L, x, y));
  const A sdy = sin(curl_at(ph, L, x, (y + L - 1) % L));
  const A sdx = sin(curl_at(ph, L, (x + L - 1) % L, y));
  fx = K * (sc - sdy);
  fy = K * (-sc + sdx);
  const A* pn = phi + ((t + 1) % Nt) * sv;
  const A* pp = phi + ((t + Nt - 1) % Nt) * sv;
  const int s2 = 2 * (x + L * y);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const A v = ph[s2 + c], vn = pn[s2 + c], vp = pp[s2 + c];
    A f;
    if (compact)
      f = -(-sin(vn - v) + sin(v - vp));
    else
      f = -(-(vn - v) + (v - vp));
    if (c == 0)
      fx += ctau * f;
    else
      fy += ctau * f;
  }
}

template <typename A>
// grid (site blocks, slice, chain): one site per thread, both bond directions
__global__ void k_boson_force(BosonArgs p) {
  const int Vs = p.L * p.L;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= Vs) return;
  const int t = blockIdx.y, b = blockIdx.z;
  const A* phi = reinterpret_cast<const A*>(p.x) + (size_t)b * p.Nt * 2 * Vs;
  A fx, fy;
  boson_force_site<A>(phi, p.L, p.Nt, t, s % p.L, s / p.L, (A)p.K, (A)p.ctau, p.compact, fx, fy);
  A* F = reinterpret_cast<A*>(p.F) + 2 * (((size_t)b * p.Nt + t) * Vs + s);
  F[0] = fx;
  F[1] = fy;
}

// The same force with one block per (slice, chain): the slice's angles are
// staged in shared memory with 16-byte loads, sin(curl) is formed once per
// plaquette (instead of three times per site), and each bond's force is the
// difference of its two plaquettes' sines plus the tau term.  The arithmetic
// of every term is that of boson_force_site, so the results are identical.
// (x, y) of the sites s = threadIdx.x + k blockDim.x of an L x L slice,
// advanced without integer division
struct SiteWalk {
  int s, x, y, dx, dy;
  __device__ explicit SiteWalk(int L)
      : s(threadIdx.x), x(threadIdx.x % L), y(threadIdx.x / L), dx(blockDim.x % L), dy(blockDim.x / L) {}
  __device__ void next(int L) {
    s += blockDim.x;
    x += dx;
    y += dy;
    if (x >= L) {
      x -= L;
      ++y;
    }
  }
};

template <typename A>
inline size_t boson_slice_smem(int L, int curls) {
  return sizeof(A) * (size_t)L * L * (2 + curls);
}

template <typename A>
__global__ void __launch_bounds__(256) k_boson_force_slice(BosonArgs p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = p.L, Vs = L * L, Nt = p.Nt, t = blockIdx.x, b = blockIdx.y;
  A* ph = reinterpret_cast<A*>(smem_raw);  // [Vs][2] angles of slice t
  A* sc = ph + 2 * Vs;                     // [Vs] sin(curl)
  const size_t sv = 2 * (size_t)Vs;
  const A* phi = reinterpret_cast<const A*>(p.x) + (size_t)b * Nt * sv;
  const float4* src = reinterpret_cast<const float4*>(phi + t * sv);
  const int nvec = (int)(sv * sizeof(A) / 16);  // L even: whole 16-byte vectors
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) reinterpret_cast<float4*>(ph)[i] = __ldg(src + i);
  __syncthreads();
  for (SiteWalk w(L); w.s < Vs; w.next(L)) {
    const int s = w.s, x = w.x, y = w.y;
    const int xp = x + 1 == L ? 0 : x + 1, yp = y + 1 == L ? 0 : y + 1;
    sc[s] = sin(ph[2 * (x + L * y)] + ph[2 * (xp + L * y) + 1] - ph[2 * (x + L * yp)] - ph[2 * (x + L * y) + 1]);
  }
  __syncthreads();
  const Cx<A>* pn = reinterpret_cast<const Cx<A>*>(phi + ((t + 1) % Nt) * sv);
  const Cx<A>* pp = reinterpret_cast<const Cx<A>*>(phi + ((t + Nt - 1) % Nt) * sv);
  Cx<A>* F = reinterpret_cast<Cx<A>*>(p.F) + ((size_t)b * Nt + t) * Vs;
  const A K = (A)p.K, ctau = (A)p.ctau;
  for (SiteWalk w(L); w.s < Vs; w.next(L)) {
    const int s = w.s, x = w.x, y = w.y;
    const int xm = x == 0 ? L - 1 : x - 1, ym = y == 0 ? L - 1 : y - 1;
    const A c = sc[s];
    A fx = K * (c - sc[x + L * ym]);
    A fy = K * (-c + sc[xm + L * y]);
    const Cx<A> vn = pn[s], vp = pp[s];
    const A v0 = ph[2 * s], v1 = ph[2 * s + 1];
    if (p.compact) {
      fx += ctau * -(-sin(vn.re - v0) + sin(v0 - vp.re));
      fy += ctau * -(-sin(vn.im - v1) + sin(v1 - vp.im));
    } else {
      fx += ctau * -(-(vn.re - v0) + (v0 - vp.re));
      fy += ctau * -(-(vn.im - v1) + (v1 - vp.im));
    }
    F[s] = mk<A>(fx, fy);
  }
}

// p += ca[b] * F * mask[t];  then (if cb != 0) x += cb[b] * p * mask[t]
template <typename A>
__global__ void k_kick_drift(KickArgs p) {
  const int Vs = p.L * p.L;
  const size_t n = (size_t)p.bs * p.Nt * Vs * 2;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t site = i / 2;
    const int t = (site / Vs) % p.Nt;
    const int b = site / ((size_t)Vs * p.Nt);
    const A m = p.mask ? (A)p.mask[t] : (A)1;
    A* P = reinterpret_cast<A*>(p.p);
    const A* F = reinterpret_cast<const A*>(p.F);
    A pv = P[i];
    if (F) pv += (A)(p.kick_scale * p.dt[b]) * F[i] * m;
    P[i] = pv;
    if (p.drift_scale != 0.0) {
      A* X = reinterpret_cast<A*>(p.x);
      X[i] += (A)(p.drift_scale * p.dt[b]) * pv * m;
    }
  }
}

// ============================================================================
// reductions (double accumulation)
// ============================================================================
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-wide sum; every thread of the block must call it
__device__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  __syncthreads();
  if (ln == 0) sh[w] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x < (blockDim.x + 31) / 32) t = sh[threadIdx.x];
  if (w == 0) t = warp_sum(t);
  return t;
}

// out[b] (+)= Re sum conj(u) v over n complex entries per row (double accum)
template <typename R>
__global__ void k_cdot(const R* u, const R* v, int64_t n, double* out) {
  __shared__ double sh[32];
  const int b = blockIdx.y;
  const R* ub = u + (size_t)b * 2 * n;
  const R* vb = v + (size_t)b * 2 * n;
  double acc = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if ((n & 1) == 0 && ((reinterpret_cast<uintptr_t>(ub) | reinterpret_cast<uintptr_t>(vb)) & 15) == 0) {
    // two complex numbers per access
    for (int64_t k = i0; 2 * k < n; k += stride) {
      Cx<R> a0, a1, b0, b1;
      ld2(ub + 4 * k, a0, a1);
      ld2(vb + 4 * k, b0, b1);
      acc += (double)a0.re * (double)b0.re + (double)a0.im * (double)b0.im + (double)a1.re * (double)b1.re +
             (double)a1.im * (double)b1.im;
    }
  } else {
    for (int64_t i = i0; i < n; i += stride)
      acc += (double)ub[2 * i] * (double)vb[2 * i] + (double)ub[2 * i + 1] * (double)vb[2 * i + 1];
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) atomicAdd(out + b, acc);
}

// out[b] (+)= sum of the boson action per chain and (kin != 0) sum p^2 / (2m)
template <typename A>
__global__ void k_boson_action(BosonArgs p, double* out) {
  __shared__ double sh[32];
  const int Vs = p.L * p.L;
  const int b = blockIdx.y;
  const int n = p.Nt * Vs;  // sites of one chain (below 2^31)
  const A* phi = reinterpret_cast<const A*>(p.x) + (size_t)b * n * 2;
  const A* mom = p.F ? reinterpret_cast<const A*>(p.F) + (size_t)b * n * 2 : nullptr;
  double acc = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int s = i % Vs;
    const int t = i / Vs;
    const A* ph = phi + t * 2 * (size_t)Vs;
    acc += p.K * (double)cos(curl_at(ph, p.L, s % p.L, s / p.L));
    const A* pn = phi + ((t + 1) % p.Nt) * 2 * (size_t)Vs;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double d = (double)pn[2 * s + c] - (double)ph[2 * s + c];
      acc += p.compact ? p.ctau * (1.0 - cos(d)) : p.ctau * 0.5 * d * d;
      if (mom) {
        const double q = mom[2 * i + c];
        acc += q * q / (2.0 * p.mass);
      }
    }
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) atomicAdd(out + b, acc);
}

// The same sums with one block per (slice, chain), the slice staged in shared
// memory with 16-byte loads.
template <typename A>
__global__ void __launch_bounds__(256) k_boson_action_slice(BosonArgs p, double* out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[32];
  const int L = p.L, Vs = L * L, Nt = p.Nt, t = blockIdx.x, b = blockIdx.y;
  A* ph = reinterpret_cast<A*>(smem_raw);  // [Vs][2] angles of slice t
  const size_t sv = 2 * (size_t)Vs;
  const A* phi = reinterpret_cast<const A*>(p.x) + (size_t)b * Nt * sv;
  const float4* src = reinterpret_cast<const float4*>(phi + t * sv);
  const int nvec = (int)(sv * sizeof(A) / 16);
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) reinterpret_cast<float4*>(ph)[i] = __ldg(src + i);
  __syncthreads();
  const Cx<A>* pn = reinterpret_cast<const Cx<A>*>(phi + ((t + 1) % Nt) * sv);
  const Cx<A>* mom = p.F ? reinterpret_cast<const Cx<A>*>(p.F) + ((size_t)b * Nt + t) * Vs : nullptr;
  double acc = 0;
  for (SiteWalk w(L); w.s < Vs; w.next(L)) {
    const int s = w.s, x = w.x, y = w.y;
    const int xp = x + 1 == L ? 0 : x + 1, yp = y + 1 == L ? 0 : y + 1;
    acc += p.K * (double)cos(ph[2 * (x + L * y)] + ph[2 * (xp + L * y) + 1] - ph[2 * (x + L * yp)] -
                             ph[2 * (x + L * y) + 1]);
    const Cx<A> vn = pn[s];
    const double d0 = (double)vn.re - (double)ph[2 * s], d1 = (double)vn.im - (double)ph[2 * s + 1];
    acc += p.compact ? p.ctau * (1.0 - cos(d0)) : p.ctau * 0.5 * d0 * d0;
    acc += p.compact ? p.ctau * (1.0 - cos(d1)) : p.ctau * 0.5 * d1 * d1;
    if (mom) {
      const Cx<A> q = mom[s];
      acc += (double)q.re * (double)q.re / (2.0 * p.mass);
      acc += (double)q.im * (double)q.im / (2.0 * p.mass);
    }
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) atomicAdd(out + b, acc);
}

// ============================================================================
// host launchers
// ============================================================================
static int g_num_sms = 0;
int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

template <typename K>
static int prepare_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return QEDF_ERR_CUDA;
  }
  return QEDF_OK;
}

bool by_valid(int L, int by) {
  return (by == 2 || by == 4 || by == 6) && L % by == 0 && (L / 2) * (L / by) <= max_threads_by(by);
}

// slices of an operator kernel that one SM holds at a time, by the warps that
// its registers allow (the launch bounds above)
static int resident_slices(int L, int by, int real_bytes) {
  const int warps = slice_threads(L, by) / 32;
  const int room = real_bytes == 4 ? (by == 2 ? 36 : by == 4 ? 16 : 12) : (by == 2 ? 20 : warps > 12 ? 16 : 12);
  return room / warps;
}

// The tile height that keeps most slices resident per SM; at equal numbers the
// taller tile in single precision (less exchange per site: L = 36, 8 right-hand
// sides, M^dag M 31 us with 2 x 6, 35 with 2 x 2 tiles; L = 30, 22.8 and 24.9),
// the lower one in double, whose taller tiles spill (L = 48: 185 us with 2 x 2,
// 209 with 2 x 4; where 2 x 4 fits two slices and 2 x 2 one, L = 36, 86 against
// 95 us; 2 x 6 only where nothing else divides L: L = 30, 80 against 58 us,
// L = 60, 149 against 142 us with 2 x 4).
int pick_by(int L, int requested, int real_bytes) {
  if (requested > 0) return by_valid(L, requested) ? requested : -1;
  int best = -1, most = 0;
  for (int by : {2, 4, 6}) {
    if (!by_valid(L, by) || (real_bytes == 8 && by == 6 && best > 0)) continue;
    const int n = resident_slices(L, by, real_bytes);
    if (best < 0 || n > most || (n == most && real_bytes == 4)) {
      best = by;
      most = n;
    }
  }
  return best;
}

// slices that the busiest block place of the GPU gets, `resident` slices to an SM
static int64_t rounds_of(int64_t slices, int resident) {
  const int64_t places = (int64_t)num_sms() * resident;
  return (slices + places - 1) / places;
}

// The operators' tile height.  In single precision 2 x 2 tiles in place of 2 x 6 ones
// where the slices would fill half of the block places of 2 x 2 tiles at most: a slice's
// own time counts there (L = 18, M^dag M, us with 2 x 2 and 2 x 6 tiles: 1 vector 3.8
// and 5.5, 4: 4.7 and 5.7, 8: 7.0 and 6.8).  In double precision 2 x 4 tiles, where
// pick_by prefers them, have to shorten the busiest block's run: a run of n slices
// applies B n times and starts up once, M^dag M 2 n + 1 times, each the longer
// the more slices share the SM.  Measured with 2 x 2 and 2 x 4 tiles, us:
// M^dag M at L = 28, 2 vectors, 16.9 and 20.9, 8: 45.6 and 45.5; L = 32, 3: 30.7 and
// 29.1, 8: 55.9 and 51.6; L = 36, 1: 20.9 and 23.3, 8: 98.8 and 84.9; L = 20, 2: 10.8
// and 12.7, 8: 26.9 and 20.9; M at L = 36, 1: 14.7 and 16.6, 3: 31.1 and 27.1.
static int pick_operator_by(int op, const OpArgs& a, int requested, int real_bytes) {
  const int by = pick_by(a.L, requested, real_bytes);
  if (requested > 0 || !by_valid(a.L, 2)) return by;
  const int64_t W = (int64_t)a.bs * a.Nt;
  const int r2 = resident_slices(a.L, 2, real_bytes), r4 = resident_slices(a.L, 4, real_bytes);
  if (real_bytes == 4) return by == 6 && rounds_of(2 * W, r2) == 1 ? 2 : by;
  if (by != 4) return by;
  auto cost = [&](int r) { return op == OP_MHM ? 2 * rounds_of(W, r) + 1 : rounds_of(W, r) + 1; };
  return (r2 + r4) * cost(r4) < 2 * r2 * cost(r2) ? 4 : 2;
}

static size_t smem_limit() { return 227 * 1024; }

// blocks of a run-per-block kernel: as many as the GPU holds at once, but
// with a slab length one per slab.  Of runs of one and a few of two slices, chance gives
// some SM two of the longer ones; runs of two alone, where they fit with a block per SM
// less, are even (complex128, L = 26, 3 vectors of 188 slices: M^dag M 17.2 -> 13.9 us, the
// force 19.0 -> 14.3; complex64, L = 28, 3 of 280: 12.8 -> 9.2).
template <typename K>
static int run_grid(K kernel, int threads, size_t smem, int bs, int Nt, int T, int& grid) {
  if (prepare_smem(kernel, smem)) return QEDF_ERR_CUDA;
  const int64_t W = (int64_t)bs * Nt;
  int64_t g = (int64_t)bs * ((Nt + (T > 0 ? T : 1) - 1) / (T > 0 ? T : 1));
  if (T <= 0 && W > num_sms()) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
      return QEDF_ERR_SIZE;
    g = std::min<int64_t>(W, (int64_t)num_sms() * per_sm);
    const int64_t twos = (W + 1) / 2;
    if (W > g && 5 * W <= 8 * g && twos <= (int64_t)num_sms() * (per_sm - 1)) g = twos;
  }
  if (g > INT32_MAX) return QEDF_ERR_SIZE;
  grid = (int)g;
  return QEDF_OK;
}

template <typename R, typename A, int BY, int OP, int CFG>
static int launch_operator_t(const OpArgs& a, cudaStream_t st) {
  const int threads = slice_threads(a.L, BY);
  constexpr int rec = Slice<R, BY, CFG == CFG_TALL, CFG == CFG_TALL ? 1 : 2>::REC;
  const size_t smem =
      slice_smem<R>(threads, rec) + (OP == OP_MHM && CFG == CFG_REG ? stash_smem<R, BY>(threads) : 0);
  if (smem > smem_limit() || threads > OpT<R, BY, CFG>::threads) return QEDF_ERR_SIZE;
  auto kern = k_operator<R, A, BY, OP, CFG>;
  int grid = 0;
  if (int e = run_grid(kern, threads, smem, a.bs, a.Nt, a.T, grid)) return e;
  kern<<<grid, threads, smem, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}

template <typename R, typename A, int BY>
static int launch_operator_by(int op, const OpArgs& a, cudaStream_t st) {
  // double precision: 2 x 6 tiles and 2 x 4 tiles above 384 threads
  if constexpr (sizeof(R) == 8 && BY >= 4) {
    if (BY == 6 || slice_threads(a.L, BY) > OpT<R, BY, CFG_REG>::threads) {
      if (op == OP_M) return launch_operator_t<R, A, BY, OP_M, CFG_TALL>(a, st);
      if (op == OP_MH) return launch_operator_t<R, A, BY, OP_MH, CFG_TALL>(a, st);
      return launch_operator_t<R, A, BY, OP_MHM, CFG_TALL>(a, st);
    }
  }
  if constexpr (!(sizeof(R) == 8 && BY == 6)) {
    if (op == OP_M) return launch_operator_t<R, A, BY, OP_M, CFG_REG>(a, st);
    if (op == OP_MH) return launch_operator_t<R, A, BY, OP_MH, CFG_REG>(a, st);
    return launch_operator_t<R, A, BY, OP_MHM, CFG_REG>(a, st);
  }
  return QEDF_ERR_ARG;
}

template <typename R, typename A>
int launch_operator(int op, OpArgs a, int by, cudaStream_t st) {
  by = pick_operator_by(op, a, by, sizeof(R));
  switch (by) {
    case 2: return launch_operator_by<R, A, 2>(op, a, st);
    case 4: return launch_operator_by<R, A, 4>(op, a, st);
    case 6: return launch_operator_by<R, A, 6>(op, a, st);
  }
  return QEDF_ERR_ARG;
}
template int launch_operator<float, float>(int, OpArgs, int, cudaStream_t);
template int launch_operator<double, double>(int, OpArgs, int, cudaStream_t);

template <typename R, typename A, int BY>
static int launch_bvec_by(const BvecArgs& a, int nvec, cudaStream_t st) {
  const int threads = slice_threads(a.L, BY);
  const size_t smem = slice_smem<R>(threads, Slice<R, BY>::REC);
  if (smem > smem_limit()) return QEDF_ERR_SIZE;
  if (prepare_smem(k_bvec<R, A, BY>, smem)) return QEDF_ERR_CUDA;
  k_bvec<R, A, BY><<<nvec, threads, smem, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}

template <typename R, typename A>
int launch_bvec(BvecArgs a, int nvec, cudaStream_t st) {
  const int by = pick_by(a.L, 0, sizeof(R));
  switch (by) {
    case 2: return launch_bvec_by<R, A, 2>(a, nvec, st);
    case 4: return launch_bvec_by<R, A, 4>(a, nvec, st);
    case 6: return launch_bvec_by<R, A, 6>(a, nvec, st);
  }
  return QEDF_ERR_ARG;
}
template int launch_bvec<float, float>(BvecArgs, int, cudaStream_t);
template int launch_bvec<double, double>(BvecArgs, int, cudaStream_t);

template <typename R>
int launch_precon(const PreconArgs& a, cudaStream_t st) {
  const int64_t chunks = (int64_t)((a.L * a.L + 31) / 32) * a.bs;
  const int rows = PRE_WARPS * Tap<R>::ROWS;
  if (chunks > 0x7fffffff || (a.Nt + rows - 1) / rows > 65535) return QEDF_ERR_SIZE;
  k_precon<R><<<dim3((unsigned)chunks, (a.Nt + rows - 1) / rows), 32 * PRE_WARPS, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}
template int launch_precon<float>(const PreconArgs&, cudaStream_t);
template int launch_precon<double>(const PreconArgs&, cudaStream_t);

template <typename R, typename A, int BY>
static int launch_force_by(const ForceArgs& a, cudaStream_t st) {
  const int threads = slice_threads(a.L, BY);
  const size_t smem = slice_smem<R>(threads, ForceSlice<R, BY>::REC);
  if (smem > smem_limit() || threads > ForceT<R, BY>::threads) return QEDF_ERR_SIZE;
  auto kern = k_force<R, A, BY>;
  int grid = 0;
  if (int e = run_grid(kern, threads, smem, a.bs, a.Nt, a.T, grid)) return e;
  kern<<<grid, threads, smem, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}

// The force's tile height.  Its kernels keep 112, 128 and 168 registers (18, 16
// and 12 warps per SM), and where 2 x 2 tiles leave an SM two slices or more (in
// double precision one), the taller tile that pick_by prefers has to cut the rounds
// of slices by more than each one's longer time: 1.7 times with 2 x 4 and twice with 2 x
// 6 tiles in single, 1.95 times with 2 x 4 in double precision.  Measured with 2 x 2 and
// the taller tiles, us: complex64, L = 30, 2 vectors, 14.6 and 17.3 (2 x 6), 8: 33.4 and
// 39.0; L = 18, 8: 12.7 and 10.5; L = 32, 2: 13.4 and 15.0 (2 x 4), 8: 33.4 and 31.5;
// complex128, L = 32, 1: 19.0 and 17.0, 2: 27.3 and 33.5; L = 36, 1: 23.1 and 29.3, 8:
// 136 and 134.
static int pick_force_by(const ForceArgs& a, int requested, int real_bytes) {
  const int by = pick_by(a.L, requested, real_bytes);
  if (requested > 0 || by <= 2 || !by_valid(a.L, 2)) return by;
  auto slices = [&](int h) { return (h == 2 ? 18 : h == 4 ? 16 : 12) / (slice_threads(a.L, h) / 32); };
  auto rounds = [&](int h) { return rounds_of((int64_t)a.bs * a.Nt, slices(h)); };
  if (slices(by) < 1 || (real_bytes == 4 && slices(2) < 2)) return by;
  return (real_bytes == 8 ? 1.95 : by == 4 ? 1.7 : 2.0) * rounds(by) <= rounds(2) ? by : 2;
}

template <typename R, typename A>
int launch_force(ForceArgs a, int by, cudaStream_t st) {
  by = pick_force_by(a, by, sizeof(R));
  switch (by) {
    case 2: return launch_force_by<R, A, 2>(a, st);
    case 4: return launch_force_by<R, A, 4>(a, st);
    case 6: return launch_force_by<R, A, 6>(a, st);
  }
  return QEDF_ERR_ARG;
}
template int launch_force<float, float>(ForceArgs, int, cudaStream_t);
template int launch_force<double, double>(ForceArgs, int, cudaStream_t);

template <typename A>
int launch_boson_force(const BosonArgs& a, cudaStream_t st) {
  const int threads = 256;
  const size_t smem = boson_slice_smem<A>(a.L, 1);
  if (smem <= smem_limit()) {
    if (prepare_smem(k_boson_force_slice<A>, smem)) return QEDF_ERR_CUDA;
    k_boson_force_slice<A><<<dim3(a.Nt, a.bs), threads, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
  }
  dim3 grid((a.L * a.L + threads - 1) / threads, a.Nt, a.bs);
  k_boson_force<A><<<grid, threads, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}
template int launch_boson_force<float>(const BosonArgs&, cudaStream_t);
template int launch_boson_force<double>(const BosonArgs&, cudaStream_t);

template <typename A>
int launch_kick_drift(const KickArgs& a, cudaStream_t st) {
  const size_t n = (size_t)a.bs * a.Nt * a.L * a.L * 2;
  const int threads = 256;
  const int blocks = (int)std::min<size_t>((n + threads - 1) / threads, (size_t)num_sms() * 8);
  k_kick_drift<A><<<blocks, threads, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}
template int launch_kick_drift<float>(const KickArgs&, cudaStream_t);
template int launch_kick_drift<double>(const KickArgs&, cudaStream_t);

template <typename A>
int launch_boson_action(const BosonArgs& a, double* out, cudaStream_t st) {
  const size_t n = (size_t)a.Nt * a.L * a.L;
  const int threads = 256;
  const size_t smem = boson_slice_smem<A>(a.L, 0);
  if (smem + 32 * sizeof(double) <= smem_limit()) {
    if (prepare_smem(k_boson_action_slice<A>, smem)) return QEDF_ERR_CUDA;
    k_boson_action_slice<A><<<dim3(a.Nt, a.bs), threads, smem, st>>>(a, out);
    return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
  }
  const int bx = (int)std::max<size_t>(1, std::min<size_t>((n + threads - 1) / threads,
                                                           (size_t)num_sms() * 16 / std::max(1, a.bs) + 1));
  k_boson_action<A><<<dim3(bx, a.bs), threads, 0, st>>>(a, out);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}
template int launch_boson_action<float>(const BosonArgs&, double*, cudaStream_t);
template int launch_boson_action<double>(const BosonArgs&, double*, cudaStream_t);

template <typename R>
int launch_cdot(const R* u, const R* v, int64_t n, int rows, double* out, cudaStream_t st) {
  const int threads = 256;
  const int bx = (int)std::max<int64_t>(1, std::min<int64_t>((n / 2 + threads - 1) / threads,
                                                             (int64_t)num_sms() * 8 / std::max(1, rows) + 1));
  k_cdot<R><<<dim3(bx, rows), threads, 0, st>>>(u, v, n, out);
  return cudaGetLastError() == cudaSuccess ? QEDF_OK : QEDF_ERR_CUDA;
}
template int launch_cdot<float>(const float*, const float*, int64_t, int, double*, cudaStream_t);
template int launch_cdot<double>(const double*, const double*, int64_t, int, double*, cudaStream_t);

}  // namespace qedf
