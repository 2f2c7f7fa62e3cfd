// Slice engine: applies the checkerboard bond factors of one imaginary-time
// slice to a vector held in registers by one thread block.
//
// Thread mapping.  The L x L slice is tiled by 2 x BY site blocks ("tiles");
// tile (bx, by) owns x in {2bx, 2bx+1} and y in [BY*by, BY*by + BY) and has
// the id by * nbx + bx, its thread index.  Because x0 and y0 are even, every
// bond factor pairs sites either inside the tile ("local") or across its edge
// with the neighbouring tile ("cross"):
//
//   g1 (x-bond A -> A+x):  local in even rows, cross in odd rows
//   g3 (x-bond A-x -> A):  local in odd rows,  cross in even rows
//   g2 (y-bond A -> A+y):  local in column x0, cross at the ends of x0+1
//   g4 (y-bond A-y -> A):  local in column x0+1, cross at the ends of x0
//
// (A = sites with x = y mod 2, the ordering of the reference's
// initialize_geometry, hmc_sampler_batch.py:937-969).  The factors are applied
// without their scalar cosh: I + K with K_ij = a = t e^{i phi}, K_ji = conj(a).
//
// Exchange.  A cross pair (i in this tile's last column or row, j in the next
// tile's first) is updated from both sides: the owner of the bond, which alone
// holds its phase a, exports conj(a) v_i, and the other side exports v_j.  So
// no thread ever needs a neighbour's phase: a slice's phases are computed from
// the thread's own angles, without tables or a barrier.  Every factor costs
// one block barrier, with two exchange buffers in turn (BUF = 0, 1; the seven
// factors of B use P, 1-P, ..., P, so two applications in a row alternate P).
//
// Shared memory is one record per thread: the exchange slots of both buffers
// (and the phases, with PHS), an odd number of complex entries apart.  Every
// slot is then a compile-time offset from one of five thread pointers (own,
// left, right, up, down), whatever L is, and the lanes of a warp hit distinct
// banks.  A thread without a tile works on tile 0's data in its own record,
// whose slots nobody else reads: the factors hold no per-thread condition,
// which keeps the compiler from predicating (and spilling) whole tiles.
//
// What bounds it: with one block per SM its warps move in lockstep from
// barrier to barrier and the exchange, the FMA chains and the loads add up.
// Two and more blocks per SM overlap them, so the launch bounds (MaxT) trade
// registers for co-resident blocks.  Taller tiles exchange less per site: M^dag M
// of 8 complex64 vectors at L = 48, Ltau = 480 takes 63 us on the device with 2 x 2
// tiles (56 registers, two 576-thread blocks per SM), 76 us with 2 x 4 (one block of
// nine warps per SM) and 55 us with 2 x 6 (168 registers, two 192-thread blocks per
// SM; 1.15 warp instructions per site against 1.68 of an engine that also exchanged
// phases and was compiled per L, 70 us).
#pragma once

#include <type_traits>

#include "qedf_common.cuh"

namespace qedf {

// Largest thread block of each tile height; it fixes the register budget
// together with min_blocks.  Single precision: 2 x 2 tiles keep 56 registers
// for two 576-thread blocks per SM, 2 x 4 tiles 128 and 2 x 6 tiles 168 for as
// many smaller blocks as their threads allow.
template <typename R, int BY>
struct MaxT {
  static constexpr int value = BY == 2 ? 576 : (BY == 4 ? 512 : 384);
  static constexpr int min_blocks = (BY == 2 && sizeof(R) == 4) ? 2 : 1;
};

inline int max_threads_by(int by) { return by == 2 ? 576 : (by == 4 ? 512 : 384); }

// threads of one slice (a multiple of 32)
__host__ __device__ inline int slice_threads(int L, int BY) { return ((L / 2) * (L / BY) + 31) / 32 * 32; }

// complex entries of a thread's record: nbuf exchange buffers of `vecs`
// vectors, BY slots each, and with phs its 4 BY bond phases; odd
__host__ __device__ constexpr int slice_record(int BY, int nbuf, int vecs, bool phs, int extra) {
  return (nbuf * vecs * BY + (phs ? 4 * BY : 0) + extra) | 1;
}
// complex entries of a thread's stash of one tile (16-byte units an odd number apart)
template <typename R, int BY>
__host__ __device__ constexpr int stash_record() {
  return sizeof(R) == 4 ? 2 * (BY | 1) : ((2 * BY) | 1);
}

// A thread's own parking place of one tile in shared memory (no
// synchronisation), in 16-byte units an odd number apart.
template <typename R, int BY>
struct Stash {
  R* p;
  __device__ __forceinline__ void init(unsigned char* smem, int tid) {
    p = reinterpret_cast<R*>(smem) + 2 * (size_t)tid * stash_record<R, BY>();
  }
  __device__ __forceinline__ void park(const Cx<R> (&v)[BY][2]) const {
#pragma unroll
    for (int r = 0; r < BY; ++r) st2(p + 4 * r, v[r][0], v[r][1]);
  }
  __device__ __forceinline__ void unpark(Cx<R> (&v)[BY][2]) const {
#pragma unroll
    for (int r = 0; r < BY; ++r) ld2c(p + 4 * r, v[r][0], v[r][1]);
  }
};

// NBUF exchange buffers of VECS vectors per thread.  NBUF = 1 (a second
// barrier per factor instead of a second buffer) is for kernels short of
// shared memory.
// A block may have more warps than its engine: those call idle_apply instead, so
// that every barrier is the whole block's.  A barrier that counts the engine's
// threads alone takes their number from a register: 3 to 5 % of a solver's
// iteration (L = 48, 2 right-hand sides, 50.2 -> 48.1 us; L = 66, 1, 81.2 -> 77.1).
// EXTRA: further entries of the record, the kernel's own.
template <typename R, int BY, bool PHS = false, int NBUF = 2, int VECS = 1, int EXTRA = 0>
struct Slice {
  static_assert(BY % 2 == 0, "BY must be even");
  static constexpr int REC = slice_record(BY, NBUF, VECS, PHS, EXTRA);
  static constexpr int PH0 = NBUF * VECS * BY;  // first phase (or extra entry) of a record
  int off, rs;  // reals: this tile's first site in a slice, one row
  bool on;      // owns a tile
  Cx<R>*me, *lf, *rt, *up, *dn;  // records: own and the four neighbours'
  Cx<R> px_[PHS ? 1 : BY][2], py_[PHS ? 1 : BY][2];

  // smem: blockDim.x records of REC complex entries
  __device__ __forceinline__ void init(int L, unsigned char* smem, int tid) {
    const int nbx = L / 2, nby = L / BY;
    on = tid < nbx * nby;
    const int q = on ? tid : 0;
    const int bx = q % nbx, by = q / nbx;
    off = 2 * (BY * by * L + 2 * bx);
    rs = 2 * L;
    Cx<R>* base = reinterpret_cast<Cx<R>*>(smem);
    me = base + tid * REC;
    lf = base + (on ? by * nbx + (bx == 0 ? nbx - 1 : bx - 1) : tid) * REC;
    rt = base + (on ? by * nbx + (bx + 1 == nbx ? 0 : bx + 1) : tid) * REC;
    up = base + (on ? (by == 0 ? nby - 1 : by - 1) * nbx + bx : tid) * REC;
    dn = base + (on ? (by + 1 == nby ? 0 : by + 1) * nbx + bx : tid) * REC;
  }
  // phase of the x-bond / y-bond starting at own site (x0+c, y0+r)
  __device__ __forceinline__ Cx<R> px(int r, int c) const {
    return PHS ? me[PH0 + 4 * r + 2 * c] : px_[PHS ? 0 : r][c];
  }
  __device__ __forceinline__ Cx<R> py(int r, int c) const {
    return PHS ? me[PH0 + 4 * r + 2 * c + 1] : py_[PHS ? 0 : r][c];
  }

  // ---- global memory: the tile's rows of a slice --------------------------
  __device__ __forceinline__ void load(Cx<R> (&v)[BY][2], const R* slice) const {
#pragma unroll
    for (int r = 0; r < BY; ++r) ld2(slice + off + r * rs, v[r][0], v[r][1]);
  }
  // coherent, through a storage type S (float, double, bf16 or scaled fp16
  // pairs: stored value times sc; see ld2s)
  template <typename S>
  __device__ __forceinline__ void load_st(Cx<R> (&v)[BY][2], const S* slice, R sc) const {
#pragma unroll
    for (int r = 0; r < BY; ++r) ld2s(slice + off + r * rs, v[r][0], v[r][1], sc);
  }
  template <typename S>
  __device__ __forceinline__ void load_st(Cx<R> (&v)[BY][2], const S* slice) const {
#pragma unroll
    for (int r = 0; r < BY; ++r) ld2s(slice + off + r * rs, v[r][0], v[r][1]);
  }
  __device__ __forceinline__ void store(R* slice, const Cx<R> (&v)[BY][2]) const {
    if (!on) return;
#pragma unroll
    for (int r = 0; r < BY; ++r) st2(slice + off + r * rs, v[r][0], v[r][1]);
  }
  template <typename S>
  __device__ __forceinline__ void store_st(S* slice, const Cx<R> (&v)[BY][2], R inv) const {
    if (!on) return;
#pragma unroll
    for (int r = 0; r < BY; ++r) st2s(slice + off + r * rs, v[r][0], v[r][1], inv);
  }

  // ---- bond phases of one slice -------------------------------------------
  // t1 = tanh(dtau), th = tanh(dtau/2)
  template <typename A>
  __device__ __forceinline__ void load_angles(A (&a)[BY][4], const A* ang) const {
#pragma unroll
    for (int r = 0; r < BY; ++r) ld4(ang + off + r * rs, a[r]);
  }
  template <typename A>
  __device__ __forceinline__ void phases(const A (&a)[BY][4], R t1, R th) {
#pragma unroll
    for (int r = 0; r < BY; ++r) {
      // the x-bond of (x0+c, y0+r) is in g1 when the site is an A site, else g3
      const Cx<R> q[4] = {tphase((R)a[r][0], (r & 1) == 0 ? t1 : th), tphase((R)a[r][1], th),
                          tphase((R)a[r][2], (r & 1) == 1 ? t1 : th), tphase((R)a[r][3], th)};
      if constexpr (PHS) {
#pragma unroll
        for (int k = 0; k < 4; ++k) me[PH0 + 4 * r + k] = q[k];
      } else {
        px_[r][0] = q[0];
        py_[r][0] = q[1];
        px_[r][1] = q[2];
        py_[r][1] = q[3];
      }
    }
  }
  // the tile's angles by cp.async into a stash (each thread waits for its own)
  __device__ __forceinline__ void fetch_angles(const Stash<R, BY>& st, const R* ang) const {
#pragma unroll
    for (int r = 0; r < BY; ++r)
#pragma unroll
      for (int k = 0; k < (int)(4 * sizeof(R) / 16); ++k)
        cp_async16(st.p + 4 * r + 16 / sizeof(R) * k, ang + off + r * rs + 16 / sizeof(R) * k);
    cp_async_commit();
  }
  __device__ __forceinline__ void take_angles(R (&a)[BY][4], const Stash<R, BY>& st) const {
    cp_async_wait<0>();
#pragma unroll
    for (int r = 0; r < BY; ++r) {
      Cx<R> u, v;
      ld2c(st.p + 4 * r, u, v);
      a[r][0] = u.re;
      a[r][1] = u.im;
      a[r][2] = v.re;
      a[r][3] = v.im;
    }
  }
  // straight from memory, row by row
  template <typename A>
  __device__ __forceinline__ void phases_of(const A* ang, R t1, R th) {
    A a[BY][4];
    load_angles(a, ang);
    phases(a, t1, th);
  }

  // conj(a) b
  __device__ static __forceinline__ Cx<R> cjm(Cx<R> a, Cx<R> b) {
    return mk<R>(fma(a.re, b.re, a.im * b.im), fma(a.re, b.im, -(a.im * b.re)));
  }
  // (v_i, v_j) <- (v_i + a v_j, v_j + conj(a) v_i)
  __device__ static __forceinline__ void pair(Cx<R>& vi, Cx<R>& vj, Cx<R> a) {
    const Cx<R> oi = vi, oj = vj;
    vi = cfma(a, oj, oi);
    vj = cjfma(a, oi, oj);
  }

  // ---- one factor: v <- (I + K_g) v -----------------------------------------
  // G: 0..3 for g1..g4; BUF: exchange buffer
  template <int G, int BUF>
  __device__ __forceinline__ void factor(Cx<R> (&v)[BY][2]) {
    constexpr int B0 = (NBUF == 2 ? BUF : 0) * BY;
    if constexpr (NBUF == 1) __syncthreads();  // the last factor's values are read
    if constexpr (G == 0 || G == 2) {
      constexpr int RC = G == 0 ? 1 : 0;  // parity of the cross rows
#pragma unroll
      for (int r = RC; r < BY; r += 2) {
        me[B0 + (r & ~1)] = v[r][0];
        me[B0 + (r & ~1) + 1] = cjm(px(r, 1), v[r][1]);
      }
#pragma unroll
      for (int r = 1 - RC; r < BY; r += 2) pair(v[r][0], v[r][1], px(r, 0));
      __syncthreads();
#pragma unroll
      for (int r = RC; r < BY; r += 2) {
        v[r][1] = cfma(px(r, 1), rt[B0 + (r & ~1)], v[r][1]);
        v[r][0] = v[r][0] + lf[B0 + (r & ~1) + 1];
      }
    } else {
      constexpr int CL = (G == 1) ? 0 : 1;  // column with only local pairs
      constexpr int CC = 1 - CL;            // column with cross pairs at its ends
      me[B0] = v[0][CC];
      me[B0 + 1] = cjm(py(BY - 1, CC), v[BY - 1][CC]);
#pragma unroll
      for (int r = 0; r < BY; r += 2) pair(v[r][CL], v[r + 1][CL], py(r, CL));
#pragma unroll
      for (int r = 1; r + 1 < BY; r += 2) pair(v[r][CC], v[r + 1][CC], py(r, CC));
      __syncthreads();
      v[BY - 1][CC] = cfma(py(BY - 1, CC), dn[B0], v[BY - 1][CC]);
      v[0][CC] = v[0][CC] + up[B0 + 1];
    }
  }

  // B = F4 F3 F2 F1 F2 F3 F4 without the scalar Cb.  Two applications in a row
  // alternate P (or are separated by a barrier).
  template <int P = 0>
  __device__ __forceinline__ void applyB(Cx<R> (&v)[BY][2]) {
    factor<3, P>(v);
    factor<2, 1 - P>(v);
    factor<1, P>(v);
    factor<0, 1 - P>(v);
    factor<1, P>(v);
    factor<2, 1 - P>(v);
    factor<3, P>(v);
  }
  // n applications' barriers, for a warp outside the engine
  __device__ static __forceinline__ void idle_apply(int n) {
    for (int i = 0; i < n * 7 * (NBUF == 1 ? 2 : 1); ++i) asm volatile("bar.sync 0;\n" ::: "memory");
  }
};

// bytes of a block's records, rounded to 16, where a stash may follow
template <typename R>
__host__ __device__ constexpr size_t slice_smem(int threads, int rec) {
  return ((size_t)threads * rec * sizeof(Cx<R>) + 15) / 16 * 16;
}
template <typename R, int BY>
__host__ __device__ constexpr size_t stash_smem(int threads) {
  return (size_t)threads * stash_record<R, BY>() * sizeof(Cx<R>);
}

// y = a - s * b  (s real)
template <typename R, int BY>
__device__ __forceinline__ void axpy_blk(Cx<R> (&y)[BY][2], const Cx<R> (&a)[BY][2], R s,
                                         const Cx<R> (&b)[BY][2]) {
#pragma unroll
  for (int r = 0; r < BY; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      y[r][c].re = fma(-s, b[r][c].re, a[r][c].re);
      y[r][c].im = fma(-s, b[r][c].im, a[r][c].im);
    }
}

// sum of |a|^2 over a tile in the tile's precision, then double
template <typename R, int BY>
__device__ __forceinline__ double sq_blk(const Cx<R> (&a)[BY][2]) {
  R s = 0;
#pragma unroll
  for (int r = 0; r < BY; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) s = fma(a[r][c].re, a[r][c].re, fma(a[r][c].im, a[r][c].im, s));
  return (double)s;
}

template <typename R, int BY>
__device__ __forceinline__ void copy_blk(Cx<R> (&y)[BY][2], const Cx<R> (&a)[BY][2]) {
#pragma unroll
  for (int r = 0; r < BY; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) y[r][c] = a[r][c];
}

// sigma_t: +1 for t < Nt-1 and -1 for the antiperiodic wrap t = Nt-1
template <typename R>
__device__ __forceinline__ R sigma_of(int t, int Nt) { return t == Nt - 1 ? R(-1) : R(1); }

}  // namespace qedf
