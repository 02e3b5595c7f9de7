// The TCI2 sweep step kernel (sm_103a): batched evaluation of f over Pi,
// full-pivot rank-revealing LU, and the per-bond post-processing, fused so that
// a Pi matrix that fits in shared memory never leaves the SM.
//
// One CTA takes one task at a time from an atomic queue (tasks are ordered
// largest first on the host).  Task kinds (tci_tasks.h):
//   RRLU : Pi[i,j] = f(rows[i] ++ cols[j]) (filltensor, tensorci2.jl:290-312,
//          batcheval.jl:32-61) or a given matrix, then rrLU exactly as
//          _optimizerrlu!/addpivot! (matrixlu.jl:98-181), then optionally
//          left/right of MatrixLUCI (matrixluci.jl:40-84).
//   SITE : setsitetensor!(tci, f, b) (tensorci2.jl:367-394): the pivot matrix P
//          is factored with partial pivoting in LAPACK's order and
//          T = Pi1 * inv(P) is solved row by row.
//   CORE : core = Pi1 (tensorci2.jl:379-383, :449-459).
//   EVAL : f and the tensor train at points (globalpivotfinder.jl:167-177,
//          abstracttensortrain.jl:124-132).
//
// Bit-exactness of the pivots: the rank-1 update is a separate IEEE multiply and
// subtract (as the reference's loop at matrixlu.jl:128-134 is compiled without FMA),
// scaling is an IEEE division (matrixlu.jl:119-123); the products and quotients are
// formed on the integer pipes, correctly rounded (ieee_int.h), and by __dmul_rn and
// __ddiv_rn for operands outside its range.  The argmax compares abs2 = v*v with
// strict '>' and breaks ties towards the first element in column-major order of the
// physically permuted matrix
// (matrixlu.jl:16-31).  The comparison of v*v is skipped for elements whose |v|
// is more than 16 ulps below the running maximum, where v*v is provably smaller.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <limits.h>
#include <mutex>
#include <stddef.h>
#include <stdint.h>
#include <type_traits>
#include <string>

#include "ieee_int.h"
#include "kernels.h"
#include "tci_functions.h"
#include "tci_tasks.h"

// The variant this translation unit builds (kernels.h): the threads of one task
// CTA and the task CTAs per SM, and the namespace of its kernels and launchers.
#ifndef TCI_KNS
#define TCI_KNS tci_k256
#define TCI_STEP_THREADS 256
#define TCI_CTAS_PER_SM 2
#endif

// Optional per-phase timing hook (defined by an instrumented build; no-op here).
#ifndef TCI_PHASE
#define TCI_PHASE(id) ((void)0)
#endif

namespace TCI_KNS {
namespace {

constexpr int NT = TCI_STEP_THREADS;
constexpr int NW = NT / 32;
constexpr unsigned FULL = 0xffffffffu;
constexpr uint64_t NAN_FLOOR = 0x7ff0000000000000ULL;  // bits above this are NaN
constexpr uint64_t SQ_SMALL = (uint64_t)(1023 - 500) << 52;  // below: squares may be subnormal
constexpr uint64_t SQ_BIG = (uint64_t)(1023 + 500) << 52;    // above: squares may overflow

template <int W>
struct CtlT {
  int task;
  int r, c, K, stop, kmax, need_exact, bar_err;
  int status;
  double piv, maxerror, err;
  int factors[2];  // flags of the entries that joined L and U, by pivot parity (JoinFlags)
  double red_s[W + 1];
  int red_k[W + 1];
  unsigned long long red_u[W + 1];
  unsigned long long red_b[W + 1];
  unsigned red_p[W + 1];
  long long red4[4][W + 1];
};
using Ctl = CtlT<NW>;
// The multi-CTA rrLU runs one 512-thread CTA per SM whatever the task CTAs are.
constexpr int BIG_NT = 512;
constexpr int BIG_NW = BIG_NT / 32;
using BigCtl = CtlT<BIG_NW>;

__device__ __forceinline__ double jmax(double a, double b) {
  if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000LL);
  return a > b ? a : b;
}

// Bit pattern of |v| computed on the integer pipe.  Written as a register move
// plus integer AND so that it cannot be lowered to an FP64 absolute-value
// instruction: on this GPU the FP64 pipe is 1/64 of the FP32 rate and is the
// bottleneck of the rank-1 update.
__device__ __forceinline__ uint64_t abs_bits(double v) {
  unsigned lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
  return ((uint64_t)(hi & 0x7fffffffu) << 32) | (uint64_t)lo;
}
// v is NaN, tested on the integer pipe (an FP64 self-comparison would take the
// slow FP64 pipe).
__device__ __forceinline__ bool is_nan_bits(double v) { return abs_bits(v) > 0x7ff0000000000000ULL; }

// Argmax of abs2 with first-in-column-major tie breaking, without squaring on
// the FP64 pipe in the common case: while updating, each thread tracks the
// largest |v| bit pattern, its first key and the next smaller pattern (integer
// ops, NaN excluded); one block reduction gives the winner unless another
// element lies within 16 ulps of the largest |v| (where v*v can tie with the
// largest square) or the magnitude is below 2^-500 or above 2^500 (squares can
// underflow or overflow).  Then a read-only pass squares the elements near the
// maximum and picks the largest square, ties to the smallest key.
// Element keys are (column << 16) | row: ordered like the column-major position
// (matrices have at most 65535 rows and columns).
__device__ __forceinline__ uint32_t pack_key(int i, int j) { return ((uint32_t)j << 16) | (uint32_t)i; }

// One thread's running argmax of |v| (pushed in any key order), integer pipe
// only: A = the largest |v| bit pattern + 1, k = its smallest key, B = the
// largest bit pattern + 1 below A (0 = none).  NaN never wins (the reference's
// scan starts from typemin and compares with '>').
struct ArgTrack {
  uint64_t A, B;
  uint32_t k, sgn;  // sgn: the sign bit of the element at k
  __device__ __forceinline__ void init() {
    A = B = 0;
    k = 0xffffffffu;
    sgn = 0;
  }
  __device__ __forceinline__ void push(double v, uint32_t key) {
    uint64_t b = abs_bits(v);
    if (b > NAN_FLOOR) return;
    b += 1;
    const bool win = b > A || (b == A && key < k);
    B = b > A ? A : (b < A && b > B ? b : B);
    if (win) {
      A = b;
      k = key;
      sgn = (uint32_t)__double2hiint(v) & 0x80000000u;
    }
  }
  // the element at k
  __device__ __forceinline__ double value() const {
    return __longlong_as_double((long long)((A ? A - 1 : 0) | ((uint64_t)sgn << 32)));
  }
};
// Warp-wide versions with the hardware reductions (redux.sync) instead of a
// shuffle tree; every lane gets the result.  warp_track: the largest A, the smallest
// key among the lanes that hold it, and B = the largest value below A held
// anywhere (a lane below the maximum offers its A, a lane at it its B).
__device__ __forceinline__ uint64_t warp_max_u64(uint64_t x) {
  const unsigned hi = __reduce_max_sync(FULL, (unsigned)(x >> 32));
  const unsigned lo = __reduce_max_sync(FULL, (unsigned)(x >> 32) == hi ? (unsigned)x : 0u);
  return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ void warp_track(uint64_t& A, uint32_t& k, uint64_t& B) {
  const uint64_t Am = warp_max_u64(A);
  const uint32_t km = __reduce_min_sync(FULL, A == Am ? k : 0xffffffffu);
  B = warp_max_u64(A == Am ? B : A);
  A = Am;
  k = km;
}
// The largest s and the smallest key among the lanes that hold it.
__device__ __forceinline__ void warp_best(uint64_t& s, uint32_t& key) {
  const uint64_t sm = warp_max_u64(s);
  key = __reduce_min_sync(FULL, s == sm ? key : 0xffffffffu);
  s = sm;
}

// Exact candidate of the second pass: abs2 = v*v (never NaN here, >= +0), so
// its bit pattern orders like its value; ties go to the smaller key.
struct ArgBest {
  uint64_t s;  // abs2 bits + 1, 0 = none
  uint32_t key;
  double val;  // the element at key
  __device__ __forceinline__ void init() {
    s = 0;
    key = 0xffffffffu;
    val = 0.0;
  }
  __device__ __forceinline__ void consider(double v, uint32_t k) {
    const uint64_t q = (uint64_t)__double_as_longlong(__dmul_rn(v, v)) + 1;
    if (q > s || (q == s && k < key)) {
      s = q;
      key = k;
      val = v;
    }
  }
};
__device__ __forceinline__ bool near_max(uint64_t b, uint64_t Mstar) {
  return b <= NAN_FLOOR && (b + 16 >= Mstar || Mstar < SQ_SMALL || Mstar >= SQ_BIG);
}

// Block-wide exact argmax; every thread gets (abs2 bits + 1, key).  Ends with a barrier.
__device__ void block_argmax(const ArgBest& a, Ctl& ctl, uint64_t& out_s, uint32_t& out_key) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t s = a.s;
  uint32_t key = a.key;
  warp_best(s, key);
  __syncthreads();  // the slots may still be read
  if (lane == 0) {
    ctl.red_u[warp] = s;
    ctl.red_k[warp] = (int)key;
  }
  __syncthreads();
  if (warp == 0) {
    s = lane < NW ? ctl.red_u[lane] : 0ULL;
    key = lane < NW ? (uint32_t)ctl.red_k[lane] : 0xffffffffu;
    warp_best(s, key);
    if (lane == 0) {
      ctl.red_u[NW] = s;
      ctl.red_k[NW] = (int)key;
    }
  }
  __syncthreads();
  out_s = ctl.red_u[NW];
  out_key = (uint32_t)ctl.red_k[NW];
  __syncthreads();
}

// Block-wide max of unsigned 64-bit values (|v| bit patterns: NaN sorts above Inf).
__device__ unsigned long long block_max_u64(unsigned long long v, Ctl& ctl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    unsigned long long o = __shfl_down_sync(FULL, v, off);
    v = o > v ? o : v;
  }
  if (lane == 0) ctl.red_u[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < NW ? ctl.red_u[lane] : 0ULL;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      unsigned long long o = __shfl_down_sync(FULL, v, off);
      v = o > v ? o : v;
    }
    if (lane == 0) ctl.red_u[NW] = v;
  }
  __syncthreads();
  unsigned long long r = ctl.red_u[NW];
  __syncthreads();
  return r;
}


// Second argmax pass over the block A[r0:r0+rows, c0:c0+cols]: squares only
// the elements near the largest |v| (Mstar).  Every thread gets the result;
// s == 0 means no element qualified (all NaN).
__device__ void exact_argmax(const double* A, int lda, int r0, int rows, int c0, int cols, uint64_t Mstar,
                             Ctl& ctl, uint64_t& s, uint32_t& key) {
  ArgBest ab;
  ab.init();
  if (rows > 0 && cols > 0) {
    const long long total = (long long)rows * cols;
    const int sq = NT / rows, sr = NT % rows;
    int jj = threadIdx.x / rows, ii = threadIdx.x % rows;
    for (long long e = threadIdx.x; e < total; e += NT) {
      const int i = r0 + ii, j = c0 + jj;
      const double v = A[i + (size_t)j * lda];
      if (near_max(abs_bits(v), Mstar)) ab.consider(v, pack_key(i, j));
      ii += sr;
      jj += sq;
      if (ii >= rows) {
        ii -= rows;
        jj += 1;
      }
    }
  }
  block_argmax(ab, ctl, s, key);
}

// The pivot of the next step (submatrixargmax of abs2, matrixlu.jl:1-32): its
// place and value.
struct Pick {
  int r, c;
  double piv;
};
// Whether the largest |v| (A - 1, runner-up B - 1) decides the argmax of abs2:
// no element other than the largest |v| lies within 16 ulps of it (its square
// could tie), and the magnitude is not where squares underflow or overflow.
__device__ __forceinline__ bool track_decides(uint64_t A, uint64_t B) {
  const uint64_t M = A - 1;
  return A != 0 && M >= SQ_SMALL && M < SQ_BIG && (B == 0 || (B - 1) + 16 < M);
}

// From every thread's ArgTrack over the block A[r0:, c0:] to every thread: one
// barrier.  Each warp writes its winner, and every warp reduces the NW winners
// itself: the pivot step needs no second barrier to hand the result out.  The
// winner's value travels with it, so no thread reads A here (the next step's
// swaps may already be under way in other warps).  The exact pass and a block
// of NaNs only (the scan keeps its start) do read A, with barriers of their own.
__device__ Pick argmax_pick(const ArgTrack& t, const double* A, int lda, int r0, int rows, int c0, int cols,
                            Ctl& ctl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t a = t.A, b = t.B;
  uint32_t k = t.k;
  warp_track(a, k, b);
  if (t.A == a && t.k == k) {  // one lane (any, when nothing was tracked)
    ctl.red_u[warp] = a;
    ctl.red_b[warp] = b;
    ctl.red_k[warp] = (int)k;
    ctl.red_s[warp] = t.value();
  }
  __syncthreads();
  const uint64_t wa = lane < NW ? ctl.red_u[lane] : 0ULL;
  const uint32_t wk = lane < NW ? (uint32_t)ctl.red_k[lane] : 0xffffffffu;
  const double wv = lane < NW ? ctl.red_s[lane] : 0.0;
  a = wa;
  k = wk;
  b = lane < NW ? ctl.red_b[lane] : 0ULL;
  warp_track(a, k, b);
  Pick p;
  if (track_decides(a, b)) {
    p.r = (int)(k & 0xffffu);
    p.c = (int)(k >> 16);
    p.piv = __shfl_sync(FULL, wv, __ffs(__ballot_sync(FULL, wa == a && wk == k)) - 1);
    return p;
  }
  p.r = r0;
  p.c = c0;
  if (a != 0) {
    uint64_t s;
    uint32_t key;
    exact_argmax(A, lda, r0, rows, c0, cols, a - 1, ctl, s, key);
    if (s) {
      p.r = (int)(key & 0xffffu);
      p.c = (int)(key >> 16);
    }
  }
  p.piv = A[p.r + (size_t)p.c * lda];
  __syncthreads();
  return p;
}

__device__ int block_or(int v, Ctl& ctl) {
  int r = __syncthreads_or(v);
  return r;
}

__device__ __forceinline__ size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// base + offset as integer arithmetic: in resident mode the base is zero and
// the offsets are absolute addresses.
__device__ __forceinline__ const char* at(const char* base, int64_t off) {
  return (const char*)((uintptr_t)base + (uintptr_t)off);
}
__device__ __forceinline__ char* atw(char* base, int64_t off) { return (char*)((uintptr_t)base + (uintptr_t)off); }

// Row / column partial sums of the registered f (tci_functions.h).  For a
// task that may tabulate f (int_states), the sums are exact integers and are
// stored as long long in the same 8-byte slots; make_filler turns them back
// into doubles if it decides against tables.
__device__ __forceinline__ bool int_states(const tci_task& T) {
  return tci_f_tables(T.fid) > 0 && T.lut != nullptr && T.lutcap0 > 0;
}
// The registered f of its two sums, and the sums of `len` sites from site0 on with
// local values v (site `over` of them taken as `val`).  Out of line: a task's fills
// and states share one copy of the code, which a small task would otherwise wait for
// more than once.
__device__ __noinline__ double f_finish(int fid, const double* prm, int nparams, double a0, double a1) {
  return tci_f_finish(fid, prm, nparams, a0, a1);
}
struct FSums {
  double a0, a1;
};
__device__ __forceinline__ bool f_digits(int fid, int site0, int len) {
  return (fid == TCI_F_QTT1D || fid == TCI_F_QTT2D) && len <= 53 && site0 + len <= 1022;
}
__device__ __noinline__ FSums f_sums(int fid, const double* prm, int site0, int len, const uint8_t* v, int over,
                                     int val) {
  FSums a{0.0, 0.0};
  if (f_digits(fid, site0, len)) {
    // binary digits: every partial sum is exact, so they are collected as an
    // integer (an FP64 addition per site takes a warp 64 cycles of its SM quarter)
    unsigned long long q0 = 0, q1 = 0;
    for (int p = 0; p < len; ++p) {
      const int d = p == over ? val : v[p];
      q0 = 2 * q0 + (fid == TCI_F_QTT1D ? d != 0 : d & 1);
      q1 = 2 * q1 + (d >> 1 & 1);
    }
    const double ulp = tci_pow2i(-(site0 + len));
    a.a0 = (double)q0 * ulp;
    if (fid == TCI_F_QTT2D) a.a1 = (double)q1 * ulp;
  } else {
    for (int p = 0; p < len; ++p) tci_f_term(fid, prm, site0 + p, p == over ? val : v[p], &a.a0, &a.a1);
  }
  return a;
}

// f at one multi-index, inline: in a task of points there is nothing to share the code
// with, and the calls made the search of a product function 14 % slower.
__device__ __forceinline__ double f_point(const tci_task& T, const double* prm, const uint8_t* v, int over, int val) {
  FSums a{0.0, 0.0};
  if (tci_f_tables(T.fid) > 0 && T.lutcap0 > 0) {  // the same sums, exact integers, off the FP64 pipe
    long long i0 = 0, i1 = 0;
    for (int s = 0; s < T.L; ++s) tci_f_term_int(T.fid, prm, s, s == over ? val : v[s], &i0, &i1);
    a.a0 = (double)i0;
    a.a1 = (double)i1;
  } else if (f_digits(T.fid, 0, T.L)) {
    a = f_sums(T.fid, prm, 0, T.L, v, over, val);
  } else {
    for (int s = 0; s < T.L; ++s) tci_f_term(T.fid, prm, s, s == over ? val : v[s], &a.a0, &a.a1);
  }
  return tci_f_finish(T.fid, prm, T.nparams, a.a0, a.a1);
}

// A list of `count` multi-indices of `len` sites from site0 on, and where their
// two sums go.
struct StateList {
  const uint8_t* idx;
  int count, len, site0;
  double *s0, *s1;
};
// All lists in one pass over the CTA's threads: of a small task each list has a
// few entries, and one after the other would use a warp at a time.
template <int G>
__device__ void compute_states(const tci_task& T, const double* params, const StateList (&g)[G]) {
  int total = 0;
#pragma unroll
  for (int k = 0; k < G; ++k) total += g[k].count;
  const bool ints = int_states(T);
  for (int e = threadIdx.x; e < total; e += NT) {
    StateList l = g[0];
    int i = e;
#pragma unroll
    for (int k = 1; k < G; ++k)
      if (i >= l.count) {
        i -= l.count;
        l = g[k];
      }
    const uint8_t* v = l.idx + (size_t)i * l.len;
    if (ints) {
      long long a0 = 0, a1 = 0;
      for (int p = 0; p < l.len; ++p) tci_f_term_int(T.fid, params, l.site0 + p, v[p], &a0, &a1);
      ((long long*)l.s0)[i] = a0;
      ((long long*)l.s1)[i] = a1;
    } else {
      const FSums a = f_sums(T.fid, params, l.site0, l.len, v, -1, 0);
      l.s0[i] = a.a0;
      l.s1[i] = a.a1;
    }
  }
}

// Element generator of a registered f from row/column partial sums.  When f
// factors through exact integer sums (tci_f_tables), the distinct values of
// part0 and of scale1(part1) over the task's range are computed once into
// T.lut and each element is combine_scaled(table0[s0], table1[s1]) -- one FP64
// operation; the direct path computes the same functions, so the bits are
// identical.
using At1 = std::integral_constant<int, 1>;  // elements taken at once by a fill's loop
using At4 = std::integral_constant<int, 4>;
struct Filler {
  int fid, nparams;
  const double* prm;
  const double* lut0;
  const double* lut1;
  int lo0, lo1;
  // element (i, j) from row states r0/r1 and column states c0/c1: from the tables, or either way
  __device__ __forceinline__ double tab(const double* r0, const double* r1, int i, const double* c0,
                                        const double* c1, int j) const {
    const double p0 = lut0[(int)(((const long long*)r0)[i] + ((const long long*)c0)[j]) - lo0];
    if (!lut1) return p0;
    const double q1 = lut1[(int)(((const long long*)r1)[i] + ((const long long*)c1)[j]) - lo1];
    return tci_f_combine_scaled(fid, p0, q1);
  }
  __device__ __forceinline__ double val(const double* r0, const double* r1, int i, const double* c0,
                                        const double* c1, int j) const {
    if (lut0) return tab(r0, r1, i, c0, c1, j);
    return f_finish(fid, prm, nparams, r0[i] + c0[j], r1[i] + c1[j]);
  }
};

// Block-wide max of four signed 64-bit integers (pass -x for a minimum).
__device__ void block_max4_i64(long long v[4], Ctl& ctl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const long long o = __shfl_down_sync(FULL, v[q], off);
      v[q] = o > v[q] ? o : v[q];
    }
    if (lane == 0) ctl.red4[q][warp] = v[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      long long x = lane < NW ? ctl.red4[q][lane] : LLONG_MIN;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const long long o = __shfl_down_sync(FULL, x, off);
        x = o > x ? o : x;
      }
      if (lane == 0) ctl.red4[q][NW] = x;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = ctl.red4[q][NW];
  __syncthreads();
}

// Decide on tabulation for a task whose elements are sums rs[i] + cs[j] over
// the given row-state groups, and fill the tables.  Ends with a barrier.
__device__ Filler make_filler(const tci_task& T, const double* prm, double* const* rs0, double* const* rs1,
                              const int* rcount, int ngroups, double* cs0, double* cs1, int n, int64_t elems,
                              Ctl& ctl) {
  Filler F;
  F.fid = T.fid;
  F.nparams = T.nparams;
  F.prm = prm;
  F.lut0 = F.lut1 = nullptr;
  F.lo0 = F.lo1 = 0;
  if (!int_states(T)) return F;
  const int tables = tci_f_tables(T.fid);
  if (T.lut_full) {  // the solve's tables, built once by its TABLE task
    F.lut0 = T.lut;
    F.lut1 = tables > 1 ? T.lut + T.lutcap0 : nullptr;
    F.lo0 = T.lut_base0;
    F.lo1 = 0;
    return F;
  }
  // max / -min of the row and column sums
  long long v[4] = {LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN};  // max r0, max r1, -min r0, -min r1
  long long w[4] = {LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN};
  for (int g = 0; g < ngroups; ++g) {
    const long long* a0 = (const long long*)rs0[g];
    const long long* a1 = (const long long*)rs1[g];
    for (int i = threadIdx.x; i < rcount[g]; i += NT) {
      v[0] = max(v[0], a0[i]);
      v[1] = max(v[1], a1[i]);
      v[2] = max(v[2], -a0[i]);
      v[3] = max(v[3], -a1[i]);
    }
  }
  {
    const long long* b0 = (const long long*)cs0;
    const long long* b1 = (const long long*)cs1;
    for (int j = threadIdx.x; j < n; j += NT) {
      w[0] = max(w[0], b0[j]);
      w[1] = max(w[1], b1[j]);
      w[2] = max(w[2], -b0[j]);
      w[3] = max(w[3], -b1[j]);
    }
  }
  block_max4_i64(v, ctl);
  block_max4_i64(w, ctl);
  bool use = v[0] != LLONG_MIN && w[0] != LLONG_MIN;  // rows and columns exist
  long long lo0 = 0, lo1 = 0, n0 = 0, n1 = 0;
  if (use) {
    lo0 = -v[2] - w[2];
    lo1 = -v[3] - w[3];
    n0 = v[0] + w[0] - lo0 + 1;
    n1 = tables > 1 ? v[1] + w[1] - lo1 + 1 : 0;
    use = n0 <= T.lutcap0 && (tables == 1 || n1 <= T.lutcap1) &&
          n0 + n1 <= elems;  // tabulating must cost less than it saves
  }
  if (!use) {  // direct evaluation: the sums become doubles (exact)
    for (int g = 0; g < ngroups; ++g)
      for (int i = threadIdx.x; i < rcount[g]; i += NT) {
        rs0[g][i] = (double)((const long long*)rs0[g])[i];
        rs1[g][i] = (double)((const long long*)rs1[g])[i];
      }
    for (int j = threadIdx.x; j < n; j += NT) {
      cs0[j] = (double)((const long long*)cs0)[j];
      cs1[j] = (double)((const long long*)cs1)[j];
    }
    __syncthreads();
    return F;
  }
  double* t0 = T.lut;
  double* t1 = T.lut + T.lutcap0;
  for (int k = threadIdx.x; k < (int)n0; k += NT) t0[k] = tci_f_part0(T.fid, prm, T.nparams, (double)(lo0 + k));
  for (int k = threadIdx.x; k < (int)n1; k += NT)
    t1[k] = tci_f_scale1(T.fid, prm, tci_f_part1(T.fid, prm, (double)(lo1 + k)));
  __syncthreads();
  F.lut0 = t0;
  F.lut1 = tables > 1 ? t1 : nullptr;
  F.lo0 = (int)lo0;
  F.lo1 = (int)lo1;
  return F;
}

// Result record pointers.
struct ResPtrs {
  tci_result_head* head;
  int* rowp;
  int* colp;
  double* diag;
};
__device__ ResPtrs res_ptrs(char* resb, const tci_task& T) {
  ResPtrs p;
  char* base = atw(resb, T.res);
  p.head = (tci_result_head*)base;
  const int kcap = T.kcap;
  size_t off = sizeof(tci_result_head);
  p.rowp = (int*)(base + off);
  off += align_up((size_t)kcap * 4, 8);
  p.colp = (int*)(base + off);
  off += align_up((size_t)kcap * 4, 8);
  p.diag = (double*)(base + off);
  return p;
}

// Bit pattern of a stopping threshold for integer comparison with |pivot| (the
// patterns of non-negative doubles order like their values): NaN and negative
// thresholds, below which nothing lies, become zero.
__device__ __forceinline__ uint64_t threshold_bits(double t) {
  const uint64_t b = (uint64_t)__double_as_longlong(t);
  return b > 0x7ff0000000000000ULL ? 0ull : b;
}

// State of the pivot loop, the same in every thread that runs it.
struct PivotState {
  uint64_t err, maxerror, thr;  // bit patterns of lu.error, maxerror and max(reltol * maxerror, abstol)
  __device__ __forceinline__ void init(double reltol, double abstol) {
    err = 0x7ff8000000000000ULL;
    maxerror = 0;
    thr = max(threshold_bits(reltol * 0.0), threshold_bits(abstol));
  }
  // Decision of _optimizerrlu! (matrixlu.jl:150-158) for a pivot: lu.error and
  // the stopping rule, on the integer pipe; reltol * maxerror is formed only
  // when maxerror grows.  Returns whether to stop.
  __device__ __forceinline__ bool decide(double piv, int K, double reltol, double abstol) {
    const uint64_t e = abs_bits(piv);
    err = e;
    if (e < thr && K > 0) return true;
    if (e > maxerror) {  // also when the pivot is NaN; a NaN maxerror stays
      maxerror = (uint64_t)__double_as_longlong(
          jmax(__longlong_as_double((long long)maxerror), __longlong_as_double((long long)e)));
      thr = max(threshold_bits(reltol * __longlong_as_double((long long)maxerror)), threshold_bits(abstol));
    }
    return false;
  }
};
// The permutation bookkeeping of addpivot! and the pivot's entry of diag, by one thread.
__device__ __forceinline__ void record_pivot(const Pick& p, int K, double* diag_out, int* rowperm, int* colperm) {
  diag_out[K] = __longlong_as_double((long long)abs_bits(p.piv));
  const int a = rowperm[K], b = rowperm[p.r], c = colperm[K], d = colperm[p.c];
  rowperm[K] = b;
  rowperm[p.r] = a;
  colperm[K] = d;
  colperm[p.c] = c;
}

// swaprow!(K, R), swapcol!(K, C) and the scaling of addpivot! (matrixlu.jl:98-124)
// in one pass: new(i, j) = old(pr(i), pc(j)) with pr, pc the two transpositions,
// divided by the pivot in column K below the diagonal (leftorthogonal) or in row
// K right of it.  Written for the scaled direction: "line" K and line C are the
// columns for leftorthogonal, and the rows otherwise (strides si within a line
// and sj across).  Item i < mi swaps entry i of the two lines and scales the new
// one; item R also does the four corners, so that one division site serves all
// entries; items mi + j swap entries (K, j) and (R, j) of the other lines.
// The body for threads t = 0, stride, ... of a group (no barrier).
// The entries of the new row K (columns >= K) and of the new column K (rows >=
// K) join U and L at this pivot; every other entry of L and U joined at an
// earlier one (swaps only move them), so the flags of all pivots cover the NaN
// check of L and U (matrixlu.jl:162-169).
struct JoinFlags {
  bool nan;     // an entry that joined is NaN
  int factors;  // of this pivot: 2 an entry is not int_safe, 1 one is not int_dense
  __device__ __forceinline__ void join(double v) {
    if (!int_dense(v)) factors |= 1;
    if (!int_safe(v)) {
      factors |= 2;
      if (is_nan_bits(v)) nan = true;
    }
  }
};
// How the products of a rank-1 update are taken: all factors dense, some of
// them not (decided per tile), or on the FP64 pipe.
enum { PROD_DENSE = 0, PROD_MIXED = 1, PROD_FP64 = 2 };
// The scaling divides a whole row or column by one pivot: on the integer pipe
// (int_div) unless the pivot or the entry is outside its range.  An FP64
// division holds an SM quarter's FP64 pipe for 548 cycles.
struct PivotDivisor {
  double piv;
  bool safe;
  IntDivisor d;
  __device__ __forceinline__ explicit PivotDivisor(double p) : piv(p), safe(int_safe(p) && (abs_bits(p) != 0)) {
    d = int_divisor(p);
  }
  __device__ __forceinline__ double quo(double v) const {
    return safe && int_safe(v) ? int_div(v, d) : __ddiv_rn(v, piv);
  }
};
__device__ __forceinline__ void swap_scale_body(double* A, int lda, int m, int n, int K, const Pick& p,
                                                bool leftorth, int t, int stride, JoinFlags& fl) {
  const PivotDivisor D(p.piv);
  const int mi = leftorth ? m : n, nj = leftorth ? n : m;
  const int R = leftorth ? p.r : p.c, C = leftorth ? p.c : p.r;
  const int si = leftorth ? 1 : lda, sj = leftorth ? lda : 1;
  for (int w = t; w < mi + nj; w += stride) {
    if (w < mi) {
      const int i = w;
      if (i == K && R != K) continue;  // done by item R
      double* const pk = A + (size_t)i * si + (size_t)K * sj;
      double* const pc = A + (size_t)i * si + (size_t)C * sj;
      double a = *pk, v = *pc;
      if (i == R && R != K) {
        double* const qk = A + (size_t)K * si + (size_t)K * sj;
        double* const qc = A + (size_t)K * si + (size_t)C * sj;
        const double ork = a;
        a = *qk;
        v = *qc;
        *qk = p.piv;
        if (C != K) {
          *qc = ork;
          fl.join(ork);
        }
      }
      if (i > K) {
        v = D.quo(v);
        fl.join(v);
      }
      *pk = v;
      if (C != K) {
        *pc = a;
        if (i == K) fl.join(a);
      }
    } else {
      const int j = w - mi;
      if (j == K || j == C) continue;
      double* const pk = A + (size_t)K * si + (size_t)j * sj;
      if (R != K) {
        double* const pr = A + (size_t)R * si + (size_t)j * sj;
        const double a = *pk, v = *pr;
        *pr = a;
        *pk = v;
        if (j > K) fl.join(v);
      } else if (j > K) {
        fl.join(*pk);
      }
    }
  }
  if (is_nan_bits(p.piv)) fl.nan = true;
}
// swap_scale_body by one warp for at most 32 scaled lines: each lane takes an entry
// by the place it comes from (rows K and R exchanged), so that all lanes run the
// same few instructions; the lines are read before any is written.  A pivot of an
// 8 x 8 matrix by one warp, with rank1_low: 3.1k cycles -> 2.55k.
__device__ __forceinline__ void swap_scale_warp(double* A, int lda, int m, int n, int K, const Pick& p, bool leftorth,
                                                int lane, JoinFlags& fl) {
  const PivotDivisor D(p.piv);
  const int mi = leftorth ? m : n, nj = leftorth ? n : m;
  const int R = leftorth ? p.r : p.c, C = leftorth ? p.c : p.r;
  const int si = leftorth ? 1 : lda, sj = leftorth ? lda : 1;
  for (int w0 = 0; w0 < mi + nj; w0 += 32) {
    const int w = w0 + lane, j = w - mi;
    const bool line = w < mi;
    const int from = w == R ? K : (w == K ? R : w);
    const int ov = line ? from * si + C * sj : R * si + j * sj, oa = line ? from * si + K * sj : K * si + j * sj;
    const int tv = line ? w * si + K * sj : oa, ta = line ? w * si + C * sj : ov;
    const bool on = line || (j < nj && j != K && j != C), past = line ? w > K : j > K;
    double v = 0.0, a = 0.0;
    if (on) {
      v = A[ov];
      a = A[oa];
    }
    __syncwarp();
    if (line && past) v = D.quo(v);
    if (on) {
      A[tv] = v;
      if (line ? C != K : R != K) A[ta] = a;
    }
    if (on && (past || (line && w == K && C != K))) fl.join(past ? v : a);
  }
  if (is_nan_bits(p.piv)) fl.nan = true;
}
// Every thread gets how the update's products are taken.  The flags go through
// a shared word per pivot parity (a barrier with a reduction costs three plain
// ones); rrlu_loop clears it.
__device__ int swap_scale(double* A, int lda, int m, int n, int K, const Pick& p, bool leftorth, JoinFlags& fl,
                          Ctl& ctl) {
  fl.factors = 0;
  swap_scale_body(A, lda, m, n, K, p, leftorth, threadIdx.x, NT, fl);
  if (fl.factors) atomicOr(&ctl.factors[K & 1], fl.factors);
  __syncthreads();
  return min(ctl.factors[K & 1], (int)PROD_FP64);
}

// x_i * y_j of an R x C group per lane.  The subtraction that follows stays on
// the FP64 pipe; the bits are those of the FP64 multiplication in every mode.
template <int MODE, int R, int C>
__device__ __forceinline__ void tile_products(const double (&x)[R], const double (&y)[C], double (&q)[R][C]) {
  bool dense = MODE == PROD_DENSE;
  if (MODE == PROD_MIXED) {
    bool d = true;
#pragma unroll
    for (int a = 0; a < R; ++a) d = d && int_dense(x[a]);
#pragma unroll
    for (int b = 0; b < C; ++b) d = d && int_dense(y[b]);
    dense = __all_sync(FULL, d);
  }
  if (MODE == PROD_FP64) {
#pragma unroll
    for (int b = 0; b < C; ++b)
#pragma unroll
      for (int a = 0; a < R; ++a) q[a][b] = __dmul_rn(x[a], y[b]);
  } else if (dense) {
    DenseFactor xf[R], yf[C];
#pragma unroll
    for (int a = 0; a < R; ++a) xf[a] = dense_split(x[a]);
#pragma unroll
    for (int b = 0; b < C; ++b) yf[b] = dense_split(y[b]);
#pragma unroll
    for (int b = 0; b < C; ++b)
#pragma unroll
      for (int a = 0; a < R; ++a) q[a][b] = int_mul_dense(xf[a], yf[b]);
  } else {
    IntFactor xf[R], yf[C];
#pragma unroll
    for (int a = 0; a < R; ++a) xf[a] = int_split(x[a]);
#pragma unroll
    for (int b = 0; b < C; ++b) yf[b] = int_split(y[b]);
#pragma unroll
    for (int b = 0; b < C; ++b)
#pragma unroll
      for (int a = 0; a < R; ++a) q[a][b] = int_mul(xf[a], yf[b]);
  }
}

// A[K:, K:] -= x y^T by warp `warp` of `nw`, each element tracked for the next
// pivot: x[i] and y[j * ystride] for i, j >= K, A column-major.
//
// FP64-bound: the products are taken on the integer pipes (ieee_int.h), so the
// FP64 pipe is used once per element instead of twice.  A warp takes 16 x 8
// tiles, its lanes laid out 8 x 4 with 2 x 2 elements each: x and y are taken
// apart once per four products, the four chains of a thread overlap, and the
// ragged ends waste at most half a tile.  Indices past the end repeat the last
// row or column (not stored).  104 x 104, two 256-thread CTAs per SM: 0.68
// cycles per element and SM (1.20 with FP64 products walked element by
// element); 16 x 16 tiles 0.76, 16 x 4 tiles 0.72.
// Tracking: only elements whose |v| has a top word of at least the warp's
// largest so far less one can be the maximum or lie within 16 ulps of it, so
// a tile costs one vote and is pushed element by element only if it reaches that.
template <int MODE, int R = 2>
__device__ __forceinline__ void rank1_tiles(double* A, int lda, int K, int m, int n, const double* x, const double* y,
                                            int ystride, int warp, int nw, ArgTrack& at) {
  const int lane = threadIdx.x & 31, lr = lane & 7, lc = lane >> 3;
  const int nti = (m - K + 8 * R - 1) / (8 * R), ntj = (n - K + 7) >> 3;
  // warp and nw over nti by an approximate reciprocal: a half added, a quotient is at
  // least 0.5 / nti from an integer (an integer division is some 25 instructions)
  const float rn = __fdividef(1.0f, (float)nti);
  int tj = nw == 1 ? 0 : (int)(((float)warp + 0.5f) * rn), ti = warp - tj * nti;
  const int dj = nw == 1 ? (nti == 1 ? 1 : 0) : (int)(((float)nw + 0.5f) * rn), di = nw - dj * nti;
  uint32_t top = 0;  // top word of the largest |v| pushed by the warp
  while (tj < ntj) {
    const int i0 = K + 8 * R * ti + lr, j0 = K + 8 * tj + lc;
    const bool vj[2] = {j0 < n, j0 + 4 < n};
    const int jj[2] = {min(j0, n - 1), min(j0 + 4, n - 1)};
    bool vi[R];
    int ii[R];
#pragma unroll
    for (int a = 0; a < R; ++a) {
      vi[a] = i0 + 8 * a < m;
      ii[a] = min(i0 + 8 * a, m - 1);
    }
    double* const p[2] = {A + (size_t)jj[0] * lda, A + (size_t)jj[1] * lda};
    double v[R][2], xv[R], yv[2], q[R][2];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int a = 0; a < R; ++a) v[a][b] = p[b][ii[a]];
#pragma unroll
    for (int a = 0; a < R; ++a) xv[a] = x[ii[a]];
#pragma unroll
    for (int b = 0; b < 2; ++b) yv[b] = y[(size_t)jj[b] * ystride];
    tile_products<MODE>(xv, yv, q);
    uint32_t h = 0;
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int a = 0; a < R; ++a) {
        v[a][b] = __dsub_rn(v[a][b], q[a][b]);
        if (vi[a] && vj[b]) p[b][ii[a]] = v[a][b];
        h = max(h, (uint32_t)__double2hiint(v[a][b]) & 0x7fffffffu);
      }
    if (__any_sync(FULL, h + 1 >= top)) {
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int a = 0; a < R; ++a)
          if (vi[a] && vj[b]) at.push(v[a][b], pack_key(ii[a], jj[b]));
      top = __reduce_max_sync(FULL, at.A ? (uint32_t)((at.A - 1) >> 32) : 0u);
    }
    ti += di;
    tj += dj;
    if (ti >= nti) {
      ti -= nti;
      tj += 1;
    }
  }
}
// The two rarer modes are kept out of line: their code is shared by the CTA and
// the one-warp loop.
__device__ __noinline__ ArgTrack rank1_mixed(double* A, int lda, int K, int m, int n, const double* x,
                                             const double* y, int ystride, int warp, int nw) {
  ArgTrack at;
  at.init();
  rank1_tiles<PROD_MIXED>(A, lda, K, m, n, x, y, ystride, warp, nw, at);
  return at;
}
__device__ __noinline__ ArgTrack rank1_fp64(double* A, int lda, int K, int m, int n, const double* x, const double* y,
                                            int ystride, int warp, int nw) {
  ArgTrack at;
  at.init();
  rank1_tiles<PROD_FP64>(A, lda, K, m, n, x, y, ystride, warp, nw, at);
  return at;
}
__device__ __forceinline__ ArgTrack rank1_update(double* A, int lda, int K, int m, int n, const double* x,
                                                 const double* y, int ystride, int warp, int nw, int mode) {
  if (mode == PROD_MIXED) return rank1_mixed(A, lda, K, m, n, x, y, ystride, warp, nw);
  if (mode == PROD_FP64) return rank1_fp64(A, lda, K, m, n, x, y, ystride, warp, nw);
  ArgTrack at;
  at.init();
  rank1_tiles<PROD_DENSE>(A, lda, K, m, n, x, y, ystride, warp, nw, at);
  return at;
}

// Eight rows or fewer, one warp: 8 x 8 tiles (inline: a call costs as much as they
// save, 500 cycles).
__device__ __forceinline__ ArgTrack rank1_low(double* A, int lda, int K, int m, int n, const double* x,
                                              const double* y) {
  ArgTrack at;
  at.init();
  rank1_tiles<PROD_DENSE, 1>(A, lda, K, m, n, x, y, lda, 0, 1, at);
  return at;
}

// Trailing blocks of at most this many elements are finished by warp 0 alone:
// with one warp no CTA barrier is needed per pivot.  Measured: up to ~6 elements
// per lane one warp beats the barriers of the whole CTA.
constexpr int WARP_TAIL_RRLU = 192;

// rrlu_loop from pivot K on (pick `p` taken, not stopped), warp 0 only; same
// arithmetic and argmax as the CTA path.  Returns the final K on every lane.
__device__ int rrlu_warp_tail(double* A, int lda, int m, int n, int K, int kmax, double reltol, double abstol,
                              bool leftorth, int* rowperm, int* colperm, double* diag_out, Pick p, PivotState& S,
                              JoinFlags& fl) {
  const int lane = threadIdx.x & 31;
  while (true) {
    fl.factors = 0;
    if ((leftorth ? m : n) <= 32) swap_scale_warp(A, lda, m, n, K, p, leftorth, lane, fl);
    else swap_scale_body(A, lda, m, n, K, p, leftorth, lane, 32, fl);
    int mode = PROD_DENSE;
    if (__any_sync(FULL, fl.factors != 0)) mode = __any_sync(FULL, fl.factors >= 2) ? PROD_FP64 : PROD_MIXED;
    __syncwarp();
    ++K;
    if (K == kmax) break;
    const double *x = A + (size_t)(K - 1) * lda, *y = A + (K - 1);
    const ArgTrack at = mode == PROD_DENSE && m - K <= 8 ? rank1_low(A, lda, K, m, n, x, y)
                                                         : rank1_update(A, lda, K, m, n, x, y, lda, 0, 1, mode);
    uint64_t a = at.A, b = at.B;
    uint32_t k = at.k;
    warp_track(a, k, b);
    __syncwarp();  // every lane's update is in place before the exact pass and the next swaps
    if (track_decides(a, b)) {
      p.r = (int)(k & 0xffffu);
      p.c = (int)(k >> 16);
      p.piv = __shfl_sync(FULL, at.value(), __ffs(__ballot_sync(FULL, at.A == a && at.k == k)) - 1);
    } else {
      p.r = p.c = K;
      if (a != 0) {  // squares of the elements near the maximum
        ArgBest ab;
        ab.init();
        const int rows = m - K, total = rows * (n - K);
        for (int e = lane; e < total; e += 32) {
          const int i = K + e % rows, j = K + e / rows;
          const double v = A[i + (size_t)j * lda];
          if (near_max(abs_bits(v), a - 1)) ab.consider(v, pack_key(i, j));
        }
        uint64_t sv = ab.s;
        uint32_t key = ab.key;
        warp_best(sv, key);
        if (sv) {
          p.r = (int)(key & 0xffffu);
          p.c = (int)(key >> 16);
        }
      }
      p.piv = A[p.r + (size_t)p.c * lda];
      __syncwarp();
    }
    if (S.decide(p.piv, K, reltol, abstol)) break;
    if (lane == 0) record_pivot(p, K, diag_out, rowperm, colperm);
  }
  return K;
}

// The rrLU main loop (matrixlu.jl:141-181) on A (m x n, leading dim lda) from
// the first pick.  rowperm/colperm are full permutations.  Per pivot: one
// swap/scale pass and the rank-1 update fused with the next argmax, whose
// decision every thread takes itself -- two barriers.
// xy: optional shared-memory copy (m + n doubles) of the pivot column and row
// for a matrix in global memory, so that each element of the update costs one
// load and one store.  Returns this thread's part of the NaN check of L and U
// (an OR over the CTA gives it).
__device__ bool rrlu_loop(double* A, int lda, int m, int n, int maxrank, double reltol, double abstol,
                          bool leftorth, int* rowperm, int* colperm, double* diag_out, Pick p, Ctl& ctl,
                          double* xy = nullptr, int warp_tail = WARP_TAIL_RRLU) {
  const int tid = threadIdx.x;
  const int kmax = min(maxrank, min(m, n));
  JoinFlags fl{false, 0};
  PivotState S;
  S.init(reltol, abstol);
  int K = 0;
  bool go = kmax > 0 && !S.decide(p.piv, 0, reltol, abstol);
  bool tail = false;
  if (go && tid == 0) record_pivot(p, 0, diag_out, rowperm, colperm);
  if (tid < 2) ctl.factors[tid] = 0;
  __syncthreads();
  while (go) {
    TCI_PHASE(1);
    if ((m - K) * (n - K) <= warp_tail) {
      tail = true;
      break;
    }
    const int mode = swap_scale(A, lda, m, n, K, p, leftorth, fl, ctl);
    TCI_PHASE(3);
    ++K;
    if (K == kmax) break;  // the trailing update after the last pivot is not observable
    // A[K:, K:] -= x * y^T fused with the argmax of abs2 for the next pivot
    const double *x = A + (size_t)(K - 1) * lda, *y = A + (K - 1);
    int ystride = lda;
    if (xy) {  // x = A[K:, K-1] and y = A[K-1, K:] on chip, indexed from K
      double* xs = xy;
      double* ys = xy + m;
      for (int i = K + tid; i < m; i += NT) xs[i] = x[i];
      for (int j = K + tid; j < n; j += NT) ys[j] = y[(size_t)j * lda];
      __syncthreads();
      x = xs;
      y = ys;
      ystride = 1;
    }
    const ArgTrack at = rank1_update(A, lda, K, m, n, x, y, ystride, tid >> 5, NW, mode);
    TCI_PHASE(4);
    p = argmax_pick(at, A, lda, K, m - K, K, n - K, ctl);
    if (tid == 0) ctl.factors[(K - 1) & 1] = 0;  // read by all before the pick's barrier, set again two pivots on
    go = !S.decide(p.piv, K, reltol, abstol);
    if (go && tid == 0) record_pivot(p, K, diag_out, rowperm, colperm);
    TCI_PHASE(6);
  }
  if (tail && tid < 32) K = rrlu_warp_tail(A, lda, m, n, K, kmax, reltol, abstol, leftorth, rowperm, colperm,
                                           diag_out, p, S, fl);
  if (tid == 0) {
    ctl.K = K;
    ctl.err = K >= min(m, n) ? 0.0 : __longlong_as_double((long long)S.err);
  }
  __syncthreads();
  return fl.nan;
}

// left(MatrixLUCI) for leftorthogonal (colstimespivotinv, matrixluci.jl:48-57):
// rows K.. of L solved against the unit-lower L11, rows scattered by rowperm.
// For !leftorthogonal: colmatrix = left(lu) * U[:, 1:K] (matrixluci.jl:40-42).
__device__ void post_left(double* A, int lda, int m, int n, int K, bool leftorth, const int* rowperm,
                          double* out) {
  const int tid = threadIdx.x;
  if (leftorth) {
    // X * L11 = L21 with unit-lower L11, one thread per row of L21, in the
    // oracle's order: X[p, q] = L21[p, q] - sum over t = q+1 .. K-1 (ascending)
    // of X[p, t] * L11[t, q], for q from K-1 down to 0 (the division by the
    // unit diagonal is exact and omitted).
    for (int p = K + tid; p < m; p += NT) {
      for (int q = K - 1; q >= 0; --q) {
        double s = A[p + (size_t)q * lda];
        for (int t = q + 1; t < K; ++t) s = s - A[p + (size_t)t * lda] * A[t + (size_t)q * lda];
        A[p + (size_t)q * lda] = s;
      }
    }
    __syncthreads();
    for (int q = 0; q < K; ++q)
      for (int p = tid; p < m; p += NT) {
        double v = p < K ? (p == q ? 1.0 : 0.0) : A[p + (size_t)q * lda];
        out[rowperm[p] + (size_t)q * m] = v;
      }
  } else {
    // colmatrix: (L with rows scattered) * U11, U11 unit upper; L keeps its diagonal
    for (int p = tid; p < m; p += NT)
      for (int q = 0; q < K; ++q) {
        double s = 0.0;
        const int tmax = min(p, q);
        for (int t = 0; t <= tmax; ++t) {
          double l = A[p + (size_t)t * lda];
          double u = (t == q) ? 1.0 : A[t + (size_t)q * lda];
          s = s + l * u;
        }
        out[rowperm[p] + (size_t)q * m] = s;
      }
  }
  __syncthreads();
}

// right(MatrixLUCI): for leftorthogonal rowmatrix = L11 * right(lu)
// (matrixluci.jl:44-46); otherwise pivotinvtimesrows (matrixluci.jl:59-68).
__device__ void post_right(double* A, int lda, int m, int n, int K, bool leftorth, const int* colperm,
                           double* out) {
  const int tid = threadIdx.x;
  if (leftorth) {
    for (int j = tid; j < n; j += NT)
      for (int q = 0; q < K; ++q) {
        double s = 0.0;
        for (int t = 0; t <= q; ++t) {
          double l = (t == q) ? 1.0 : A[q + (size_t)t * lda];
          double u = (t <= j) ? A[t + (size_t)j * lda] : 0.0;
          s = s + l * u;
        }
        out[q + (size_t)colperm[j] * K] = s;
      }
  } else {
    // U11 X = U12 with unit-upper U11, one thread per column of U12, in the
    // oracle's order: X[q, j] = U12[q, j] - sum over p = q+1 .. K-1 (ascending)
    // of U11[q, p] * X[p, j], for q from K-1 down to 0.
    for (int j = K + tid; j < n; j += NT) {
      double* col = A + (size_t)j * lda;
      for (int q = K - 1; q >= 0; --q) {
        double s = col[q];
        for (int p = q + 1; p < K; ++p) s = s - A[q + (size_t)p * lda] * col[p];
        col[q] = s;
      }
    }
    __syncthreads();
    for (int j = tid; j < n; j += NT)
      for (int q = 0; q < K; ++q) {
        double v = j < K ? (q == j ? 1.0 : 0.0) : A[q + (size_t)j * lda];
        out[q + (size_t)colperm[j] * K] = v;
      }
  }
  __syncthreads();
}

struct SmemCursor {
  char* p;
  __device__ char* take(size_t bytes) {
    char* r = p;
    p += align_up(bytes, 16);
    return r;
  }
};

// ---------------------------------------------------------------- RRLU task
__device__ void task_rrlu(const tci_task& T, const char* blob, char* resb, char* smem, Ctl& ctl, size_t smem_bytes) {
  const int m = T.m, n = T.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  ResPtrs rp = res_ptrs(resb, T);
  SmemCursor cur{smem};
  double* A = T.smem_mode == 1 ? (double*)cur.take((size_t)m * n * 8) : T.work;
  const int lda = m;
  int* rowperm = (int*)cur.take((size_t)m * 4);
  int* colperm = (int*)cur.take((size_t)n * 4);
  for (int i = tid; i < m; i += NT) rowperm[i] = i;
  for (int j = tid; j < n; j += NT) colperm[j] = j;
  int lut_used = 0;
  ArgTrack am;
  am.init();
  unsigned long long mx = 0;
  if (T.ain) {
    // the input is read once: evict-first loads keep it from pushing the
    // working matrices (re-read every pivot) out of L2
    // the input is one contiguous run (lda = m); eight loads in flight per thread
    const size_t total = (size_t)m * n;
    const int sq = NT / m, sr = NT - sq * m;
    int j = tid / m, i = tid - j * m;
    for (size_t e0 = tid; e0 < total; e0 += 8 * NT) {
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = e0 + q * NT < total ? __ldcs(T.ain + e0 + q * NT) : 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (e0 + q * NT < total) {
          A[e0 + q * NT] = v[q];
          am.push(v[q], pack_key(i, j));
          const unsigned long long b = abs_bits(v[q]);
          mx = b > mx ? b : mx;
        }
        i += sr;
        j += sq;
        if (i >= m) {
          i -= m;
          j += 1;
        }
      }
    }
  } else {
    const double* prm = (const double*)at(blob, T.params);
    // the row / column f states: on chip, or after the matrix in global scratch
    double* const st = T.smem_mode == 2 ? T.work + (size_t)m * n : nullptr;
    double* rs0 = st ? st : (double*)cur.take((size_t)m * 8);
    double* rs1 = st ? st + m : (double*)cur.take((size_t)m * 8);
    double* cs0 = st ? st + 2 * (size_t)m : (double*)cur.take((size_t)n * 8);
    double* cs1 = st ? st + 2 * (size_t)m + n : (double*)cur.take((size_t)n * 8);
    compute_states(T, prm, {{(const uint8_t*)at(blob, T.rows), m, T.nl, 0, rs0, rs1},
                            {(const uint8_t*)at(blob, T.cols), n, T.nr, T.nl, cs0, cs1}});
    __syncthreads();
    double* const rg0[1] = {rs0};
    double* const rg1[1] = {rs1};
    const int rc[1] = {m};
    const Filler F = make_filler(T, prm, rg0, rg1, rc, 1, cs0, cs1, n, (int64_t)m * n, ctl);
    lut_used = F.lut0 != nullptr;
    // consecutive elements over the CTA: f's FP64 chains cost a warp the same with
    // one lane or 32 (7 x 7 of a 40-site quantics function: 16.6k cycles with a
    // column per warp, 9.8k so, 6.8k with tci_math.h's short forms)
    const auto loop = [&](const auto& element, auto together) {
      const int sq = NT / m, sr = NT - sq * m, total = m * n;
      int j = tid / m, i = tid - j * m;
#pragma unroll decltype(together)::value
      for (int e = tid; e < total; e += NT) {
        const double v = element(i, j);
        A[e] = v;
        am.push(v, pack_key(i, j));
        const unsigned long long b = abs_bits(v);
        mx = b > mx ? b : mx;
        i += sr;
        j += sq;
        if (i >= m) {
          i -= m;
          j += 1;
        }
      }
    };
    if (F.lut0)
      loop([&](int i, int j) { return F.tab(rs0, rs1, i, cs0, cs1, j); }, At4{});
    else
      loop([&](int i, int j) { return F.val(rs0, rs1, i, cs0, cs1, j); }, At1{});
  }
  __syncthreads();
  unsigned long long mxall = block_max_u64(mx, ctl);
  if (tid == 0) ctl.status = 0;
  const Pick first = argmax_pick(am, A, lda, 0, m, 0, n, ctl);
  const bool leftorth = T.leftorth != 0;
  double* xy = nullptr;
  if (T.smem_mode != 1 && (size_t)(cur.p - smem) + (size_t)(m + n) * 8 <= smem_bytes) xy = (double*)cur.take((size_t)(m + n) * 8);
  const bool nan_part = rrlu_loop(A, lda, m, n, T.maxrank, T.reltol, T.abstol, leftorth, rowperm, colperm, rp.diag,
                                  first, ctl, xy, T.tail_elems > 0 ? T.tail_elems : WARP_TAIL_RRLU);
  const int K = ctl.K;
  // NaN check of L = tril(A[:, 1:K]) and U = triu(A[1:K, :]) (matrixlu.jl:162-169),
  // gathered while the pivots were taken
  int nan = block_or(nan_part ? 1 : 0, ctl);
  if (T.post == TCI_POST_LEFT && !nan) post_left(A, lda, m, n, K, leftorth, rowperm, T.core_out);
  if (T.post == TCI_POST_RIGHT && !nan) post_right(A, lda, m, n, K, leftorth, colperm, T.core_out);
  if (T.post == TCI_POST_FACTORS)
    for (int j = warp; j < n; j += NW)
      for (int i = lane; i < m; i += 32) T.core_out[i + (size_t)j * m] = A[i + (size_t)j * lda];
  if (tid == 0) {
    rp.head->status = nan ? TCI_ST_NAN : 0;
    rp.head->npivot = K;
    rp.head->error = ctl.err;
    rp.head->maxabs = __longlong_as_double((long long)mxall);
    rp.head->maxabs_nan = mxall > NAN_FLOOR ? 1 : 0;
    rp.head->lut_used = lut_used;
  }
  if (T.post == TCI_POST_FACTORS) {
    // full permutations go after the factors: rowperm (m) then colperm (n)
    int* fr = (int*)(T.core_out + (size_t)m * n);
    for (int i = tid; i < m; i += NT) fr[i] = rowperm[i];
    for (int j = tid; j < n; j += NT) fr[m + j] = colperm[j];
  }
  for (int k = tid; k < K; k += NT) {
    rp.rowp[k] = rowperm[k];
    rp.colp[k] = colperm[k];
  }
  __syncthreads();
}

// ---------------------------------------------------------------- SITE task
// Warp-wide pivot search of column j of A (lda = r) over rows j .. r-1 with the
// rule of LAPACK's partial pivoting as the oracle states it: start from |A[j,j]|
// and take the first row whose |a| is strictly larger than the running best
// (NaN never wins; a NaN diagonal keeps row j).  Bit patterns of |a| order like
// the values, so the search runs on the integer pipe.  Every lane gets the row.
__device__ int site_col_pivot(const double* col, int j, int r) {
  const int lane = threadIdx.x & 31;
  uint64_t s = 0;  // |a| bits + 1 of this lane's first maximum, 0 = none
  int si = INT_MAX;
  for (int i = j + 1 + lane; i < r; i += 32) {
    const uint64_t b = abs_bits(col[i]);
    if (b <= NAN_FLOOR && b + 1 > s) {
      s = b + 1;
      si = i;
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const uint64_t os = __shfl_xor_sync(FULL, s, off);
    const int oi = __shfl_xor_sync(FULL, si, off);
    if (os > s || (os == s && oi < si)) {
      s = os;
      si = oi;
    }
  }
  const uint64_t d = abs_bits(col[j]);
  if (d > NAN_FLOOR) return j;
  return s > d + 1 ? si : j;
}

// What a value, or the largest of several, allows: PROD_DENSE, PROD_MIXED
// (int_safe) or PROD_FP64.
__device__ __forceinline__ int prod_class(double v) {
  return int_safe(v) ? (int_dense(v) ? PROD_DENSE : PROD_MIXED) : PROD_FP64;
}

// w[i * ws] -= a[i * as] * b for i0 <= i < i1 (separate multiply and subtract),
// the products as MODE says: four elements at a time with their loads first, so
// that their chains overlap.  One warp alone is faster with FP64 products (one
// instruction instead of two dozen), many warps with integer ones.
template <int MODE>
__device__ __forceinline__ void row_axpy(double* w, size_t ws, const double* a, size_t as, int i0, int i1, double b) {
  const DenseFactor bd = dense_split(b);
  const IntFactor bi = int_split(b);
  auto mul = [&](double y) {
    return MODE == PROD_DENSE ? int_mul_dense(dense_split(y), bd)
                              : (MODE == PROD_MIXED ? int_mul(int_split(y), bi) : __dmul_rn(y, b));
  };
  int i = i0;
  for (; i + 4 <= i1; i += 4) {
    double x[4], y[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[q] = w[(size_t)(i + q) * ws];
      y[q] = a[(size_t)(i + q) * as];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = mul(y[q]);
#pragma unroll
    for (int q = 0; q < 4; ++q) w[(size_t)(i + q) * ws] = __dsub_rn(x[q], y[q]);
  }
  if (i < i1) {  // up to three more, the last one repeated (not stored)
    double x[3], y[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int k = min(i + q, i1 - 1);
      x[q] = w[(size_t)k * ws];
      y[q] = a[(size_t)k * as];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) y[q] = mul(y[q]);
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (i + q < i1) w[(size_t)(i + q) * ws] = __dsub_rn(x[q], y[q]);
  }
}
__device__ __forceinline__ void row_axpy_by(int mode, double* w, size_t ws, const double* a, int i0, int i1, double b) {
  if (mode == PROD_DENSE) row_axpy<PROD_DENSE>(w, ws, a, 1, i0, i1, b);
  else if (mode == PROD_MIXED) row_axpy<PROD_MIXED>(w, ws, a, 1, i0, i1, b);
  else row_axpy<PROD_FP64>(w, ws, a, 1, i0, i1, b);
}

// getrf with partial pivoting of the r x r matrix A (lda = r), in the oracle's
// order: per column j, the pivot row p (site_col_pivot), a whole-row swap of
// rows j and p, the column below the diagonal times the IEEE reciprocal of the
// pivot, then the rank-1 update of the trailing block as a separate multiply
// and subtract.  ipiv[j] = p.  Returns (to every thread) 1 when a pivot is
// exactly zero -- the reference's SingularException -- else 0.
// Two block barriers per column: (swap + scale) and (update + next pivot
// search); warp 0 owns the column being scaled and the next column, whose
// update it fuses with the search.  Matrices of at most 32 rows run on warp 0
// alone with warp-level synchronisation.
__device__ int site_getrf(double* A, int r, int* ipiv, Ctl& ctl) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (r <= 32) {
    if (warp == 0) {
      int sing = 0;
      for (int j = 0; j < r; ++j) {
        // lane i holds A[i, j]; the pivot rule of site_col_pivot by warp reductions
        double* cj = A + (size_t)j * r;
        const double v = lane < r ? cj[lane] : 0.0;
        const uint64_t bits = abs_bits(v);
        const uint64_t s = lane > j && lane < r && bits <= NAN_FLOOR ? bits + 1 : 0;
        const uint64_t best = warp_max_u64(s);
        const uint64_t d = __shfl_sync(FULL, bits, j);
        const int first = __ffs(__ballot_sync(FULL, s == best && s != 0)) - 1;
        const int p = d <= NAN_FLOOR && best > d + 1 ? first : j;
        const double piv = __shfl_sync(FULL, v, p), vj = __shfl_sync(FULL, v, j);
        if (abs_bits(piv) == 0) {
          sing = 1;
          break;
        }
        if (lane == 0) ipiv[j] = p;
        double y = 0.0;  // lane c: the new A[j, c]
        if (lane < r) {
          y = A[p + (size_t)lane * r];
          if (p != j) {
            const double a = A[j + (size_t)lane * r];
            A[j + (size_t)lane * r] = y;
            A[p + (size_t)lane * r] = a;
          }
        }
        const double rcp = PivotDivisor(piv).quo(1.0);
        const double l = __dmul_rn(lane == p ? vj : v, rcp);
        __syncwarp();
        if (lane > j && lane < r) cj[lane] = l;
        if (lane > j && lane < r) row_axpy<PROD_FP64>(A + lane, (size_t)r, A + j, (size_t)r, j + 1, r, l);
        __syncwarp();
      }
      if (lane == 0) ctl.status = sing;
    }
    __syncthreads();
    const int s = ctl.status;
    __syncthreads();
    return s;
  }
  if (warp == 0) {
    const int p = site_col_pivot(A, 0, r);
    if (lane == 0) {
      ctl.r = p;
      ctl.piv = A[p];
    }
  }
  __syncthreads();
  for (int j = 0; j < r; ++j) {
    const int p = ctl.r;
    const double piv = ctl.piv;
    if (abs_bits(piv) == 0) {
      __syncthreads();
      return 1;
    }
    // swap rows j and p (warp 0 takes column j and scales it)
    if (warp == 0) {
      double* cj = A + (size_t)j * r;
      const double djj = cj[j];
      __syncwarp();
      const double rcp = PivotDivisor(piv).quo(1.0);
      for (int i = j + 1 + lane; i < r; i += 32) {
        const double v = i == p ? djj : cj[i];
        cj[i] = v * rcp;
      }
      if (lane == 0) {
        cj[j] = piv;
        ipiv[j] = p;
      }
    } else if (p != j) {
      for (int c = tid - 32; c < r; c += NT - 32) {
        if (c == j) continue;
        const double a = A[j + (size_t)c * r], b = A[p + (size_t)c * r];
        A[j + (size_t)c * r] = b;
        A[p + (size_t)c * r] = a;
      }
    }
    __syncthreads();
    // trailing update; warp 0 updates column j+1 and searches its pivot
    const double* lj = A + (size_t)j * r;
    if (warp == 0) {
      if (j + 1 < r) {
        double* c1 = A + (size_t)(j + 1) * r;
        const double y = c1[j];
        for (int i = j + 1 + lane; i < r; i += 32) c1[i] = __dsub_rn(c1[i], __dmul_rn(lj[i], y));
        __syncwarp();
        const int pn = site_col_pivot(c1, j + 1, r);
        if (lane == 0) {
          ctl.r = pn;
          ctl.piv = c1[pn];
        }
      }
    } else {
      // four columns of a warp at a time: lane rows, loads first
      for (int c = j + 2 + 4 * (warp - 1); c < r; c += 4 * (NW - 1))
        for (int i = j + 1 + lane; i < r; i += 32)
          row_axpy<PROD_FP64>(A + i, (size_t)r, A + j, (size_t)r, c, min(c + 4, r), lj[i]);
    }
    __syncthreads();
  }
  return 0;
}

// setsitetensor!(tci, f, b) (tensorci2.jl:367-394): P (r x r) = f(prows x cols),
// Pi1 (m x r) = f(rows x cols), T = Pi1 * inv(P) from transpose(P) \ transpose(Pi1)
// (:391), i.e. getrf of A = P^T with partial pivoting and, per row of Pi1, the
// row interchanges, the unit-lower forward substitution and the upper back
// substitution (division by the diagonal) -- the order of the oracle's LAPACK
// restatement, so the tensor equals the oracle's bit for bit.
__device__ void task_site(const tci_task& T, const char* blob, char* resb, char* smem, Ctl& ctl,
                          size_t smem_bytes) {
  const int r = T.r, m = T.m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  ResPtrs rp = res_ptrs(resb, T);
  const double* prm = (const double*)at(blob, T.params);
  SmemCursor cur{smem};
  double* A = T.smem_mode == 1 ? (double*)cur.take((size_t)r * r * 8) : T.work;
  int* ipiv = (int*)cur.take((size_t)r * 4);
  int* colcls = (int*)cur.take((size_t)r * 4);  // prod_class of each column of the factored P
  double* ps0 = (double*)cur.take((size_t)r * 8);
  double* ps1 = (double*)cur.take((size_t)r * 8);
  double* cs0 = (double*)cur.take((size_t)r * 8);
  double* cs1 = (double*)cur.take((size_t)r * 8);
  // the row f states: on chip, or after P in global scratch
  double* rs0 = T.smem_mode == 2 ? T.work + (size_t)r * r : (double*)cur.take((size_t)m * 8);
  double* rs1 = T.smem_mode == 2 ? T.work + (size_t)r * r + m : (double*)cur.take((size_t)m * 8);
  compute_states(T, prm, {{(const uint8_t*)at(blob, T.prows), r, T.nl, 0, ps0, ps1},
                          {(const uint8_t*)at(blob, T.cols), r, T.nr, T.nl, cs0, cs1},
                          {(const uint8_t*)at(blob, T.rows), m, T.nl, 0, rs0, rs1}});
  __syncthreads();
  double* const rg0[2] = {ps0, rs0};
  double* const rg1[2] = {ps1, rs1};
  const int rc[2] = {r, m};
  const Filler F = make_filler(T, prm, rg0, rg1, rc, 2, cs0, cs1, r, (int64_t)(r + m) * r, ctl);
  uint64_t* rec = (uint64_t*)cur.take((size_t)r * 8);
  size_t used = (size_t)(cur.p - smem);
  int RB = (int)((smem_bytes > used ? smem_bytes - used : 0) / ((size_t)r * 8 + 8));
  RB = RB > NT ? NT : RB;
  RB = RB < 1 ? 1 : RB;
  double* W = (double*)cur.take((size_t)RB * r * 8);
  unsigned long long mx = 0;
  int nanflag = 0;
  // A[i, j] = P[j, i] = f(prows[j] ++ cols[i]) and, in the same pass, the first
  // block of rows, W[rr, q] = f(rows[base + rr] ++ cols[q])
  auto fill = [&](int base, int rows_here, int na) {
    const int total = na + rows_here * r;
    for (int e = tid; e < total; e += NT) {
      const bool p = e < na;
      const int f = p ? e : e - na, h = p ? r : rows_here, hi = f / h, lo = f - hi * h;
      const double v = F.val(p ? ps0 : rs0, p ? ps1 : rs1, p ? hi : base + lo, cs0, cs1, p ? lo : hi);
      if (p) {
        A[f] = v;
      } else {
        W[lo + (size_t)hi * RB] = v;
        const unsigned long long b = abs_bits(v);
        mx = b > mx ? b : mx;
      }
    }
    __syncthreads();
  };
  fill(0, min(RB, m), r * r);
  const int singular = site_getrf(A, r, ipiv, ctl);
  // reciprocals of the diagonal (int_divisor), for the back substitution of every row
  for (int j = tid; j < r; j += NT) rec[j] = int_divisor(A[j + (size_t)j * r]).R;
  // (up to one warp of rows per SM quarter: FP64 products, see row_axpy)
  for (int j = warp; j < r; j += NW) {
    int c = m <= 128 ? PROD_FP64 : PROD_DENSE;
    for (int i = lane; i < r; i += 32)
      if (i != j) c = max(c, prod_class(A[i + (size_t)j * r]));
    c = __reduce_max_sync(FULL, c);
    if (lane == 0) colcls[j] = c;
  }
  __syncthreads();
  for (int base = 0; base < m; base += RB) {
    const int rows_here = min(RB, m - base);
    if (base > 0) fill(base, rows_here, 0);
    if (!singular) {
      for (int rr = tid; rr < rows_here; rr += NT) {
        double* w = W + rr;
        for (int j = 0; j < r; ++j) {
          const int p = ipiv[j];
          if (p != j) {
            const double a = w[(size_t)j * RB];
            w[(size_t)j * RB] = w[(size_t)p * RB];
            w[(size_t)p * RB] = a;
          }
        }
        for (int j = 0; j + 1 < r; ++j) {
          const double bj = w[(size_t)j * RB];
          const int cc = colcls[j];
          row_axpy_by(cc == PROD_FP64 ? cc : max(cc, prod_class(bj)), w, (size_t)RB, A + (size_t)j * r, j + 1, r, bj);
        }
        for (int j = r - 1; j >= 0; --j) {
          const double d = A[j + (size_t)j * r], x = w[(size_t)j * RB];
          double bj;
          if (int_safe(d) && int_safe(x) && abs_bits(d) != 0) {
            const uint32_t dh = ii_hi(d);
            bj = int_div(x, IntDivisor{((uint64_t)((dh & 0xfffffu) | 0x100000u) << 32) | ii_lo(d), rec[j],
                                       dh & 0xfff00000u});
          } else {
            bj = __ddiv_rn(x, d);
          }
          w[(size_t)j * RB] = bj;
          const int cc = colcls[j];
          row_axpy_by(cc == PROD_FP64 ? cc : max(cc, prod_class(bj)), w, (size_t)RB, A + (size_t)j * r, 0, j, bj);
        }
      }
    }
    __syncthreads();
    for (int q = warp; q < r; q += NW)
      for (int rr = lane; rr < rows_here; rr += 32) {
        const double v = W[rr + (size_t)q * RB];
        if (is_nan_bits(v)) nanflag = 1;
        T.core_out[(base + rr) + (size_t)q * m] = v;
      }
    __syncthreads();
  }
  unsigned long long mxall = block_max_u64(mx, ctl);
  int nan = block_or(nanflag, ctl);
  if (tid == 0) {
    rp.head->status = (singular ? TCI_ST_SINGULAR : 0) | (nan ? TCI_ST_NAN : 0);
    rp.head->npivot = singular ? 0 : r;
    rp.head->error = 0.0;
    rp.head->maxabs = __longlong_as_double((long long)mxall);
    rp.head->maxabs_nan = mxall > NAN_FLOOR ? 1 : 0;
    rp.head->lut_used = F.lut0 != nullptr;
  }
  __syncthreads();
}

// ---------------------------------------------------------------- CORE task
__device__ void task_core(const tci_task& T, const char* blob, char* resb, char* smem, Ctl& ctl) {
  const int m = T.m, n = T.n, tid = threadIdx.x;
  const double* prm = (const double*)at(blob, T.params);
  SmemCursor cur{smem};
  double* rs0 = (double*)cur.take((size_t)m * 8);
  double* rs1 = (double*)cur.take((size_t)m * 8);
  double* cs0 = (double*)cur.take((size_t)n * 8);
  double* cs1 = (double*)cur.take((size_t)n * 8);
  compute_states(T, prm, {{(const uint8_t*)at(blob, T.rows), m, T.nl, 0, rs0, rs1},
                          {(const uint8_t*)at(blob, T.cols), n, T.nr, T.nl, cs0, cs1}});
  __syncthreads();
  double* const rg0[1] = {rs0};
  double* const rg1[1] = {rs1};
  const int rc[1] = {m};
  const Filler F = make_filler(T, prm, rg0, rg1, rc, 1, cs0, cs1, n, (int64_t)m * n, ctl);
  unsigned long long mx = 0;
  for (int e = tid; e < m * n; e += NT) {
    const int j = e / m, i = e - j * m;
    const double v = F.val(rs0, rs1, i, cs0, cs1, j);
    T.core_out[e] = v;
    const unsigned long long b = abs_bits(v);
    mx = b > mx ? b : mx;
  }
  unsigned long long mxall = block_max_u64(mx, ctl);
  if (tid == 0) {
    tci_result_head* h = (tci_result_head*)(atw(resb, T.res));
    h->status = 0;
    h->npivot = 0;
    h->error = 0.0;
    h->maxabs = __longlong_as_double((long long)mxall);
    h->maxabs_nan = mxall > NAN_FLOOR ? 1 : 0;
    h->lut_used = F.lut0 != nullptr;
  }
  __syncthreads();
}

// ---------------------------------------------------------------- EVAL task
constexpr int EVAL_THREAD_RMAX = TCI_EVAL_THREAD_RMAX;  // largest bond of the thread-per-point path

// f and the tensor train at T.m points (rows, L sites each).  The train: one
// thread per point for bonds up to EVAL_THREAD_RMAX, else one warp per point;
// out[q] = sum_p v[p] * core[p, i, q], summed in order of p with separate
// multiply and add, as the oracle's loop.
__device__ void task_eval(const tci_task& T, const char* blob, char* resb, char* smem, Ctl& ctl) {
  const int np = T.m, L = T.L, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* prm = (const double*)at(blob, T.params);
  const uint8_t* pts = (const uint8_t*)at(blob, T.rows);
  char* base = atw(resb, T.res);
  double* fout = (double*)(base + sizeof(tci_result_head));
  double* tout = fout + np;
  for (int p = tid; p < np; p += NT) fout[p] = f_point(T, prm, pts + (size_t)p * L, -1, 0);
  if (T.cores && T.r <= EVAL_THREAD_RMAX) {
    // bonds up to EVAL_THREAD_RMAX: one thread per point (a warp per point would
    // leave most lanes idle), the running vector in the thread's own column of
    // shared memory (2 x EVAL_THREAD_RMAX x NT doubles, within the step's plan)
    const tci_core_ref* cr = (const tci_core_ref*)at(blob, T.cores);
    double* vs = (double*)smem;
    double* ws = vs + (size_t)EVAL_THREAD_RMAX * NT;
    for (int p = tid; p < np; p += NT) {
      double* v = vs;
      double* w = ws;
      v[tid] = 1.0;
      for (int s = 0; s < L; ++s) {
        const tci_core_ref c = cr[s];
        const int i = pts[(size_t)p * L + s];
        for (int q = 0; q < c.r1; ++q) {
          const double* col = c.p + (size_t)c.r0 * (i + (size_t)c.d * q);
          double acc = 0.0;
          for (int t = 0; t < c.r0; ++t) acc = __dadd_rn(acc, __dmul_rn(v[(size_t)t * NT + tid], col[t]));
          w[(size_t)q * NT + tid] = acc;
        }
        double* tmp = v;
        v = w;
        w = tmp;
      }
      tout[p] = v[tid];
    }
  } else if (T.cores) {
    const tci_core_ref* cr = (const tci_core_ref*)at(blob, T.cores);
    const int rmax = T.r;
    double* va = (double*)smem + (size_t)warp * 2 * rmax;
    double* vb = va + rmax;
    for (int p = warp; p < np; p += NW) {
      if (lane == 0) va[0] = 1.0;
      __syncwarp();
      double* v = va;
      double* w = vb;
      for (int s = 0; s < L; ++s) {
        const tci_core_ref c = cr[s];
        const int i = pts[(size_t)p * L + s];
        for (int q = lane; q < c.r1; q += 32) {
          double acc = 0.0;
          const double* col = c.p + (size_t)c.r0 * (i + (size_t)c.d * q);
          for (int t = 0; t < c.r0; ++t) acc = __dadd_rn(acc, __dmul_rn(v[t], col[t]));
          w[q] = acc;
        }
        __syncwarp();
        double* tmp = v;
        v = w;
        w = tmp;
      }
      if (lane == 0) tout[p] = v[0];
      __syncwarp();
    }
  } else {
    for (int p = tid; p < np; p += NT) tout[p] = 0.0;
  }
  if (tid == 0) {
    tci_result_head* h = (tci_result_head*)base;
    h->status = 0;
    h->npivot = 0;
  }
  __syncthreads();
}

// ---------------------------------------------------------------- SEARCH task
// One start point of DefaultGlobalPivotFinder (globalpivotfinder.jl:160-177):
// f and the train at every point that differs from the start in one site.  The
// train values use left environments Le_p = C_0[i_0] ... C_{p-1}[i_{p-1}] and
// right environments Re_p = C_{p+1}[i_{p+1}] ... C_{L-1}[i_{L-1}] of the start,
// value(p, v) = sum_b (sum_a Le_p[a] C_p[a, v, b]) Re_p[b], every sum in index
// order with separate multiply and add (the oracle uses the same order).
// The order of every sum is fixed, so its additions are a serial chain; the
// products before it are not (chain_dot loads and multiplies eight at a time, on
// the integer pipes where many warps share the FP64 pipe).
// The two environment chains run side by side on the two halves of the CTA, and
// the inner sums of all (p, v, b) are spread over the threads before the outer
// ones.
template <bool INT>
__device__ __forceinline__ double chain_dot(double acc, const double* __restrict__ x, const double* __restrict__ y,
                                            size_t ystride, int n) {
  int t = 0;
  for (; t + 8 <= n; t += 8) {
    double p[8], q[8];
    bool safe = INT, dense = INT;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      p[k] = x[t + k];
      q[k] = y[(size_t)(t + k) * ystride];
    }
    if (INT) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        safe = safe && int_safe(p[k]) && int_safe(q[k]);
        dense = dense && int_dense(p[k]) && int_dense(q[k]);
      }
    }
    if (safe && dense) {
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = int_mul_dense(dense_split(p[k]), dense_split(q[k]));
    } else if (safe) {
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = int_mul(int_split(p[k]), int_split(q[k]));
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = __dmul_rn(p[k], q[k]);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) acc = __dadd_rn(acc, q[k]);
  }
  if (t < n) {  // the rest, its loads first as well
    double q[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) q[k] = y[(size_t)min(t + k, n - 1) * ystride];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      if (t + k >= n) break;
      acc = __dadd_rn(acc, __dmul_rn(x[t + k], q[k]));
    }
  }
  return acc;
}

__device__ void task_search(const tci_task& T, const char* blob, char* resb, char* smem, size_t smem_bytes) {
  const int L = T.L, tid = threadIdx.x;
  const double* prm = (const double*)at(blob, T.params);
  const uint8_t* st = (const uint8_t*)at(blob, T.rows);
  char* base = atw(resb, T.res);
  double* fout = (double*)(base + sizeof(tci_result_head));
  double* tout = fout + T.m;
  // environment offsets: Le_p has r0(p) entries, Re_p has r1(p) entries
  int* loff = (int*)smem;
  int* roff = loff + (L + 1);
  int* ioff = roff + (L + 1);  // first item of site p
  double* env = (double*)(smem + align_up((size_t)(3 * (L + 1)) * 4, 16));
  // the core table on chip: every site step below reads it, and in resident
  // mode the task's copy is in host memory (one round trip here instead of one
  // per read)
  tci_core_ref* cr = (tci_core_ref*)(smem + align_up((size_t)(3 * (L + 1)) * 4, 16) +
                                     align_up((size_t)T.n * 8, 16));
  {
    const tci_core_ref* src = (const tci_core_ref*)at(blob, T.cores);
    for (int p = tid; p < L; p += NT) cr[p] = src[p];
  }
  __syncthreads();
  if (tid == 0) {
    int a = 0, b = 0, c = 0;
    for (int p = 0; p < L; ++p) {
      loff[p] = a;
      a += cr[p].r0;
      ioff[p] = c;
      c += cr[p].d;
    }
    for (int p = 0; p < L; ++p) {
      roff[p] = a + b;
      b += cr[p].r1;
    }
    ioff[L] = c;
  }
  __syncthreads();
  // left environments on the first half of the threads, right ones on the second
  if (tid == 0) {
    env[loff[0]] = 1.0;
    env[roff[L - 1]] = 1.0;
  }
  __syncthreads();
  for (int k = 0; k + 1 < L; ++k) {
    const bool left = tid < NT / 2;
    const int p = left ? k : L - 1 - k;
    const tci_core_ref c = cr[p];
    const double* col0 = c.p + (size_t)c.r0 * st[p];
    const size_t slice = (size_t)c.r0 * c.d;
    if (left) {
      for (int b = tid; b < c.r1; b += NT / 2)
        env[loff[p + 1] + b] = chain_dot<false>(0.0, env + loff[p], col0 + slice * b, 1, c.r0);
    } else {
      for (int a = tid - NT / 2; a < c.r0; a += NT / 2)
        env[roff[p - 1] + a] = chain_dot<false>(0.0, env + roff[p], col0 + a, slice, c.r1);
    }
    __syncthreads();
  }
  // every (p, v): the inner sums of a block of items, then their outer sums
  const int nitems = ioff[L];
  double* wbuf = (double*)((char*)cr + align_up((size_t)L * sizeof(tci_core_ref), 16));
  const size_t used = (size_t)((char*)wbuf - smem);
  const int rmax = max(T.r, 1), block = (int)((smem_bytes > used ? smem_bytes - used : 0) / ((size_t)rmax * 8));
  for (int j0 = 0; block > 0 && j0 < nitems; j0 += block) {
    const int j1 = min(nitems, j0 + block);
    for (int e = tid; e < (j1 - j0) * rmax; e += NT) {
      const int it = j0 + e / rmax, b = e % rmax;
      int p = 0;
      while (ioff[p + 1] <= it) ++p;
      const tci_core_ref c = cr[p];
      if (b >= c.r1) continue;
      wbuf[e] = chain_dot<true>(0.0, env + loff[p], c.p + (size_t)c.r0 * ((it - ioff[p]) + (size_t)c.d * b), 1, c.r0);
    }
    __syncthreads();
    for (int it = j0 + tid; it < j1; it += NT) {
      int p = 0;
      while (ioff[p + 1] <= it) ++p;
      tout[it] = chain_dot<false>(0.0, wbuf + (size_t)(it - j0) * rmax, env + roff[p], 1, cr[p].r1);
    }
    __syncthreads();
  }
  for (int it = tid; it < nitems; it += NT) {
    int p = 0;
    while (ioff[p + 1] <= it) ++p;
    const int v = it - ioff[p];
    if (block == 0) {  // no room for one item's inner sums: each thread takes a whole item
      const tci_core_ref c = cr[p];
      double val = 0.0;
      for (int b = 0; b < c.r1; ++b)
        val = __dadd_rn(val, __dmul_rn(chain_dot<true>(0.0, env + loff[p], c.p + (size_t)c.r0 * (v + (size_t)c.d * b),
                                                       1, c.r0), env[roff[p] + b]));
      tout[it] = val;
    }
    fout[it] = f_point(T, prm, st, p, v);
  }
  if (tid == 0) {
    tci_result_head* h = (tci_result_head*)base;
    h->status = 0;
    h->npivot = 0;
    h->lut_used = 0;
  }
  __syncthreads();
}

// ---------------------------------------------------------------- SUM task
// sum(tt) (abstracttensortrain.jl:164-199): v <- v * (sum over the local index
// of core b), left to right; one thread per output bond index.
__device__ void task_sum(const tci_task& T, const char* blob, char* resb, char* smem) {
  const int L = T.L, tid = threadIdx.x;
  const tci_core_ref* cr = (const tci_core_ref*)at(blob, T.cores);
  double* v = (double*)smem;
  double* w = v + T.r;
  if (tid == 0) v[0] = 1.0;
  __syncthreads();
  for (int s = 0; s < L; ++s) {
    const tci_core_ref c = cr[s];
    for (int q = tid; q < c.r1; q += NT) {
      double acc = 0.0;
      for (int p = 0; p < c.r0; ++p) {
        double sm = 0.0;
        for (int i = 0; i < c.d; ++i) sm = __dadd_rn(sm, c.p[p + (size_t)c.r0 * (i + (size_t)c.d * q)]);
        acc = __dadd_rn(acc, __dmul_rn(v[p], sm));
      }
      w[q] = acc;
    }
    __syncthreads();
    double* t = v;
    v = w;
    w = t;
  }
  if (tid == 0) {
    tci_result_head* h = (tci_result_head*)(atw(resb, T.res));
    h->status = 0;
    h->npivot = 0;
    h->error = v[0];
  }
  __syncthreads();
}

// TABLE task: part0 over [lut_base0, lut_base0 + lutcap0) and scale1(part1)
// over [0, lutcap1) of the solve's f into T.lut -- the same functions the
// per-element path calls, so table entries equal direct evaluation bit for bit.
__device__ void task_table(const tci_task& T, const char* blob, char* resb) {
  const double* prm = (const double*)at(blob, T.params);
  for (int k = threadIdx.x; k < T.lutcap0; k += NT)
    T.lut[k] = tci_f_part0(T.fid, prm, T.nparams, (double)(T.lut_base0 + k));
  if (tci_f_tables(T.fid) > 1)
    for (int k = threadIdx.x; k < T.lutcap1; k += NT)
      T.lut[T.lutcap0 + k] = tci_f_scale1(T.fid, prm, tci_f_part1(T.fid, prm, (double)k));
  if (threadIdx.x == 0) {
    tci_result_head* h = (tci_result_head*)(atw(resb, T.res));
    h->status = 0;
    h->npivot = 0;
    h->lut_used = 1;
  }
  __syncthreads();
}

__device__ void run_task(const tci_task& T, const char* blob, char* resb, char* smem, Ctl& ctl,
                         size_t smem_bytes) {
  switch (T.kind) {
    case TCI_TASK_RRLU: task_rrlu(T, blob, resb, smem, ctl, smem_bytes); break;
    case TCI_TASK_SITE: task_site(T, blob, resb, smem, ctl, smem_bytes); break;
    case TCI_TASK_CORE: task_core(T, blob, resb, smem, ctl); break;
    case TCI_TASK_EVAL: task_eval(T, blob, resb, smem, ctl); break;
    case TCI_TASK_SUM: task_sum(T, blob, resb, smem); break;
    case TCI_TASK_SEARCH: task_search(T, blob, resb, smem, smem_bytes); break;
    case TCI_TASK_TABLE: task_table(T, blob, resb); break;
    default: break;
  }
}

// cta_area: the global scratch of each CTA (cta_stride doubles apiece), reused
// by the CTA's successive tasks: the working matrix of a task too large for
// shared memory, then its per-task f tables (the host sized the stride for the
// largest task).
__global__ void __launch_bounds__(NT, TCI_CTAS_PER_SM)
    tci_step_kernel(const char* __restrict__ blob, char* __restrict__ resb, const int* __restrict__ order,
                    int ntasks, int* counter, size_t smem_bytes, double* cta_area, size_t cta_stride) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Ctl ctl;
  const tci_task* tasks = (const tci_task*)blob;
  double* const area = cta_area + (size_t)blockIdx.x * cta_stride;
  for (;;) {
    if (threadIdx.x == 0) ctl.task = atomicAdd(counter, 1);
    __syncthreads();
    const int ti = ctl.task;
    __syncthreads();
    if (ti >= ntasks) break;
    tci_task T = tasks[order[ti]];
    size_t we = 0;
    if (T.smem_mode != 1) {
      we = tci_work_elems(&T);
      T.work = area;
    }
    if (!T.lut_full) T.lut = T.lutcap0 > 0 ? area + we : nullptr;
    const long long t0 = clock64();
    run_task(T, blob, resb, smem, ctl, smem_bytes);
    if (threadIdx.x == 0) ((tci_result_head*)(atw(resb, T.res)))->cycles = clock64() - t0;
  }
}

// ------------------------------------------------------------ resident kernel
// System-scope acquire / release on mapped host memory.
__device__ __forceinline__ uint64_t ld_acquire_sys(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(uint64_t* p, uint64_t v) {
  asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint64_t ld_acquire_gpu(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_acquire_gpu_s32(const int32_t* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(uint64_t* p, uint64_t v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_release_gpu_s32(int32_t* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr int RES_MAX_PARAMS = 64;                          // params copied to shared memory
constexpr long long RES_MAX_POLLS = 1LL << 31;  // a worker's most polls of one ticket
constexpr int TASK_WORDS = (int)(sizeof(tci_task) / 8);
static_assert(sizeof(tci_task) % 8 == 0, "task record is a whole number of words");

// Warp 0 of CTA 0: move published host-ring descriptors, 32 at a time, into
// the device ring (in ticket order, while the device ring has room), mark the
// host slots free, publish the device tickets.  Leaves -- and tells the
// workers -- when the host asks to stop and nothing published is left, after
// qc->idle_us with nothing published, when a worker has reported a failed
// wait, or after wait_ns without room in the device ring.
__device__ void resident_dispatch(tci_queue_slot* __restrict__ hs, uint32_t hmask, tci_resident_state* st,
                                  tci_queue_ctl* qc, uint64_t wait_ns) {
  const int lane = threadIdx.x;
  unsigned long long pos = *(volatile unsigned long long*)&st->host_pos;
  unsigned long long k = 0;
  const uint64_t idle_ns = (uint64_t)(*(volatile int32_t*)&qc->idle_us) * 1000ull;
  uint64_t t_idle = global_ns();
  unsigned sleep_ns = 32;
  for (;;) {
    const unsigned long long hp = pos + lane, dk = k + lane;
    tci_queue_slot* h = &hs[hp & hmask];
    tci_queue_slot* d = &st->ring[dk & (TCI_DRING - 1)];
    const bool pub = ld_acquire_sys(&h->seq) == hp + 1;
    const bool room = dk < TCI_DRING || ld_acquire_gpu(&d->taken) == dk - TCI_DRING + 1;
    const unsigned okm = __ballot_sync(FULL, pub && room);
    const int p = okm == FULL ? 32 : __ffs(~okm) - 1;
    if (p > 0) {
      if (lane < p) {
        // all loads first (independent, uncached: one trip over the host link),
        // then the stores; ordered after this lane's acquire of `seq`
        const unsigned long long* src = (const unsigned long long*)&h->t;
        unsigned long long* dst = (unsigned long long*)&d->t;
        unsigned long long w[TASK_WORDS];
#pragma unroll
        for (int q = 0; q < TASK_WORDS; ++q) w[q] = __ldcv(src + q);
#pragma unroll
        for (int q = 0; q < TASK_WORDS; ++q) dst[q] = w[q];
        st_release_sys(&h->taken, hp + 1);
        st_release_gpu(&d->seq, dk + 1);
      }
      pos += p;
      k += p;
      if (lane == 0) *(volatile unsigned long long*)&st->host_pos = pos;
      t_idle = global_ns();
      sleep_ns = 32;
      continue;
    }
    int leave = 0;
    if (lane == 0) {
      const uint64_t waited = global_ns() - t_idle;
      if (!pub)  // nothing published: the host is done, quiet for too long, or a worker failed
        leave = (*(volatile int32_t*)&qc->stop != 0) || waited > idle_ns || (*(volatile int32_t*)&st->error != 0);
      else       // published but no room: the workers must free slots; they may have failed
        leave = (*(volatile int32_t*)&st->error != 0) || waited > wait_ns;
    }
    if (__shfl_sync(FULL, leave, 0)) break;
    __nanosleep(sleep_ns);
    sleep_ns = sleep_ns < 512 ? sleep_ns * 2 : 512;
  }
  __syncwarp();
  if (lane == 0) {
    *(volatile unsigned long long*)&st->count = k;
    st_release_gpu_s32(&st->stop, 1);
  }
}

// Persistent kernel of the resident mode (every CTA resident: tci_resident_launch).
// CTA 0 hosts the dispatcher; every other CTA claims the next device ticket
// with one atomic, waits until it is dispatched (or the dispatcher has left:
// tickets past the last dispatched one are never used), runs the task and
// publishes the result record to the host.  A worker waits at most wait_ns for
// its ticket; then it sets st->error and every CTA leaves.
__global__ void __launch_bounds__(NT, TCI_CTAS_PER_SM)
    tci_resident_kernel(tci_queue_slot* __restrict__ hslots, uint32_t hmask, tci_resident_state* st,
                        tci_queue_ctl* qc, size_t smem_bytes, unsigned long long wait_ns) {
  if (blockIdx.x == 0) {
    if (threadIdx.x < 32) resident_dispatch(hslots, hmask, st, qc, wait_ns);
    return;
  }
  extern __shared__ __align__(16) char smem[];
  __shared__ Ctl ctl;
  __shared__ __align__(16) tci_task Ts;
  __shared__ double s_params[RES_MAX_PARAMS];
  __shared__ long long s_ticket;
  const int tid = threadIdx.x;
  for (;;) {
    if (tid == 0) {
      long long got = -1;
      const unsigned long long t = atomicAdd(&st->head, 1ull);
      tci_queue_slot* d = &st->ring[t & (TCI_DRING - 1)];
      const uint64_t t_begin = global_ns();
      unsigned sleep_ns = 32;
      for (long long it = 0;; ++it) {
        if (ld_acquire_gpu(&d->seq) == t + 1) {
          got = (long long)t;
          break;
        }
        if (ld_acquire_gpu_s32(&st->stop)) {  // every dispatch happened before the stop flag
          if (ld_acquire_gpu(&d->seq) == t + 1) got = (long long)t;
          break;
        }
        if (it >= RES_MAX_POLLS || global_ns() - t_begin > wait_ns) {
          atomicExch(&st->error, 1);
          break;
        }
        if (*(volatile int32_t*)&st->error) break;  // another wait has failed: leave too
        __nanosleep(sleep_ns);
        sleep_ns = sleep_ns < 256 ? sleep_ns * 2 : 256;
      }
      s_ticket = got;
    }
    __syncthreads();
    const long long ticket = s_ticket;
    if (ticket < 0) break;
    tci_queue_slot* d = &st->ring[(unsigned long long)ticket & (TCI_DRING - 1)];
    if (tid < TASK_WORDS) ((uint64_t*)&Ts)[tid] = ((const volatile uint64_t*)&d->t)[tid];
    __syncthreads();
    if (tid == 0) st_release_gpu(&d->taken, (uint64_t)ticket + 1);
    const long long t0 = clock64();
    size_t task_smem = smem_bytes;
    if (Ts.stage_bytes > 0) {
      // The record's input part (params, index lists, core table; 16-byte
      // multiple, 256-byte aligned block) to the top of shared memory, with
      // every thread's loads issued before its stores; pointers into it are
      // moved to the copy.
      const size_t sb = (size_t)Ts.stage_bytes;
      const char* base = (const char*)(uintptr_t)Ts.params;
      char* dst = smem + (smem_bytes - sb);
      const uint4* s4 = (const uint4*)base;
      uint4* d4 = (uint4*)dst;
      const int n4 = (int)(sb / 16);
      for (int k0 = tid; k0 < n4; k0 += 4 * NT) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (k0 + q * NT < n4) v[q] = s4[k0 + q * NT];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (k0 + q * NT < n4) d4[k0 + q * NT] = v[q];
      }
      __syncthreads();
      if (tid == 0) {
        const uintptr_t lo = (uintptr_t)base, hi = lo + sb;
        auto move = [&](int64_t p) -> int64_t {
          const uintptr_t q = (uintptr_t)p;
          return (q >= lo && q < hi) ? (int64_t)(uintptr_t)(dst + (q - lo)) : p;
        };
        Ts.params = move(Ts.params);
        Ts.rows = move(Ts.rows);
        Ts.cols = move(Ts.cols);
        Ts.prows = move(Ts.prows);
        Ts.cores = move(Ts.cores);
        Ts.ain = (const double*)(uintptr_t)move((int64_t)(uintptr_t)Ts.ain);
      }
      task_smem = smem_bytes - sb;
      __syncthreads();
    }
    if (Ts.nparams <= RES_MAX_PARAMS) {  // f parameters are read per element: keep them on chip
      const double* src = (const double*)(uintptr_t)Ts.params;
      for (int k = tid; k < Ts.nparams; k += NT) s_params[k] = src[k];
    }
    __syncthreads();
    if (tid == 0 && Ts.nparams <= RES_MAX_PARAMS) Ts.params = (int64_t)(uintptr_t)s_params;
    __syncthreads();
    run_task(Ts, nullptr, nullptr, smem, ctl, task_smem);
    __syncthreads();
    if (tid == 0) {
      tci_result_head* h = (tci_result_head*)(uintptr_t)Ts.res;
      h->cycles = clock64() - t0;
      __threadfence_system();
      st_release_sys(&h->done, Ts.ticket + 1);
    }
  }
}

// ------------------------------------------------------------ multi-CTA rrLU
// One rank-revealing LU spread over every SM (cooperative launch) for matrices
// far larger than shared memory.  The CTAs form a Pr x Pc grid; CTA (p, q) owns
// the row block p x column block q of the working matrix.  Nothing moves: the
// row and column swaps of swaprow!/swapcol! (matrixlu.jl:98-112) are tracked as
// permutations (pos: physical -> logical position, stor: logical -> physical),
// and the argmax key of an element is (logical column << 16) | logical row, so
// ties break exactly as in the physically permuted matrix.  The scaling of
// addpivot! (matrixlu.jl:114-124) is applied where it is needed with the same
// operands: the update of step k uses x_i = A[i, C] / piv (leftorthogonal) or
// y_j = A[R, j] / piv, each CTA dividing the entries of its own rows / columns
// (the pivot row R and column C are stable after the barrier: they leave the
// trailing block), and the stored factors are divided the same way when they
// are written out.  Per pivot: every CTA reduces the G partial argmaxes (same
// result everywhere), takes the decision, forms its x and y slices, updates its
// block of the trailing matrix fused with its partial argmax, and publishes that; the
// next pivot's wait for the partials is the only one on the other CTAs.  Products,
// quotients and subtractions are those of rrlu_loop, so the factors are bit-identical.

struct BigBar {
  unsigned int count, gen;
  int error;
  unsigned int arrived;  // partials published so far (G per pivot step; never reset)
};
struct BigPartial {
  unsigned long long A, B;
  unsigned int k, ph;  // key and physical position (row | column << 16) of the maximum
  double v;            // the element at key k (the next pivot's value)
  unsigned int nan, pad;
};

// Running argmax of |v| with the value and physical position at its key (push
// in any key order).
struct BigTrack {
  uint64_t A, B;
  uint32_t k, ph;
  double v;
  __device__ __forceinline__ void init() {
    A = B = 0;
    k = 0xffffffffu;
    ph = 0;
    v = 0.0;
  }
  __device__ __forceinline__ void push(double x, uint32_t key, uint32_t phys) {
    uint64_t b = abs_bits(x);
    if (b > NAN_FLOOR) return;
    b += 1;
    if (b > A) {
      B = A;
      A = b;
      k = key;
      ph = phys;
      v = x;
    } else if (b == A) {
      if (key < k) {
        k = key;
        ph = phys;
        v = x;
      }
    } else if (b > B) {
      B = b;
    }
  }
};
__device__ __forceinline__ void big_combine(uint64_t& A, uint32_t& k, uint32_t& ph, uint64_t& B, double& v,
                                            uint64_t A2, uint32_t k2, uint32_t ph2, uint64_t B2, double v2) {
  if (A2 > A) {
    B = B2 > A ? B2 : A;
    A = A2;
    k = k2;
    ph = ph2;
    v = v2;
  } else if (A2 == A) {
    B = B2 > B ? B2 : B;
    if (k2 < k) {
      k = k2;
      ph = ph2;
      v = v2;
    }
  } else if (A2 > B) {
    B = A2;
  }
}

// warp_track with the winner's physical position and value (from the first lane
// that holds the winning key); every lane gets the result.  Same result as
// folding big_combine over the lanes.
__device__ __forceinline__ void warp_track5(uint64_t& A, uint32_t& k, uint32_t& ph, uint64_t& B, double& v) {
  const uint64_t Am = warp_max_u64(A);
  const uint32_t km = __reduce_min_sync(FULL, A == Am ? k : 0xffffffffu);
  const int src = __ffs(__ballot_sync(FULL, A == Am && k == km)) - 1;
  B = warp_max_u64(A == Am ? B : A);
  ph = __shfl_sync(FULL, ph, src);
  v = __shfl_sync(FULL, v, src);
  A = Am;
  k = km;
}

__device__ __forceinline__ unsigned ld_acquire_gpu_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add_u32(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr long long BIG_BAR_POLLS = 1LL << 24;  // bounded wait of one grid barrier (a few seconds)

// Grid-wide barrier (sense by generation).  Returns false once any CTA has hit
// the wait bound; every CTA then leaves the factorization.
__device__ bool big_barrier(BigBar* bar, unsigned nblocks, unsigned& gen, BigCtl& ctl) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned g = gen;
    if (atomicAdd(&bar->count, 1u) == nblocks - 1) {
      atomicExch(&bar->count, 0u);
      __threadfence();
      atomicExch(&bar->gen, g + 1);
    } else {
      unsigned sleep_ns = 32;
      for (long long it = 0; ld_acquire_gpu_u32(&bar->gen) == g; ++it) {
        if (it > BIG_BAR_POLLS || *(volatile int*)&bar->error) {
          atomicExch(&bar->error, 1);
          break;
        }
        __nanosleep(sleep_ns);
        sleep_ns = sleep_ns < 128 ? sleep_ns * 2 : 128;
      }
    }
    gen = g + 1;
    ctl.bar_err = *(volatile int*)&bar->error;
  }
  __syncthreads();
  return ctl.bar_err == 0;
}

// Block reduction of every thread's BigTrack; every thread gets the result.
// Ends with a barrier.
__device__ void block_track(BigTrack& t, BigCtl& ctl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t a = t.A, b = t.B;
  uint32_t kk = t.k, ph = t.ph;
  double v = t.v;
  warp_track5(a, kk, ph, b, v);
  if (lane == 0) {
    ctl.red_u[warp] = a;
    ctl.red_b[warp] = b;
    ctl.red_k[warp] = (int)kk;
    ctl.red_p[warp] = ph;
    ctl.red_s[warp] = v;
  }
  __syncthreads();
  if (warp == 0) {
    a = lane < BIG_NW ? ctl.red_u[lane] : 0ULL;
    b = lane < BIG_NW ? ctl.red_b[lane] : 0ULL;
    kk = lane < BIG_NW ? (uint32_t)ctl.red_k[lane] : 0xffffffffu;
    ph = lane < BIG_NW ? ctl.red_p[lane] : 0u;
    v = lane < BIG_NW ? ctl.red_s[lane] : 0.0;
    warp_track5(a, kk, ph, b, v);
    if (lane == 0) {
      ctl.red_u[BIG_NW] = a;
      ctl.red_b[BIG_NW] = b;
      ctl.red_k[BIG_NW] = (int)kk;
      ctl.red_p[BIG_NW] = ph;
      ctl.red_s[BIG_NW] = v;
    }
  }
  __syncthreads();
  t.A = ctl.red_u[BIG_NW];
  t.B = ctl.red_b[BIG_NW];
  t.k = (uint32_t)ctl.red_k[BIG_NW];
  t.ph = ctl.red_p[BIG_NW];
  t.v = ctl.red_s[BIG_NW];
  __syncthreads();
}

// Block reduction of every thread's BigTrack into thread 0's (the others keep
// partial values).  One CTA barrier; the caller's next barrier orders the reuse
// of the staging slots.
__device__ void block_track_to0(BigTrack& t, BigCtl& ctl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t a = t.A, b = t.B;
  uint32_t kk = t.k, ph = t.ph;
  double v = t.v;
  warp_track5(a, kk, ph, b, v);
  if (lane == 0) {
    ctl.red_u[warp] = a;
    ctl.red_b[warp] = b;
    ctl.red_k[warp] = (int)kk;
    ctl.red_p[warp] = ph;
    ctl.red_s[warp] = v;
  }
  __syncthreads();
  if (warp == 0) {
    a = lane < BIG_NW ? ctl.red_u[lane] : 0ULL;
    b = lane < BIG_NW ? ctl.red_b[lane] : 0ULL;
    kk = lane < BIG_NW ? (uint32_t)ctl.red_k[lane] : 0xffffffffu;
    ph = lane < BIG_NW ? ctl.red_p[lane] : 0u;
    v = lane < BIG_NW ? ctl.red_s[lane] : 0.0;
    warp_track5(a, kk, ph, b, v);
    t.A = a;
    t.B = b;
    t.k = kk;
    t.ph = ph;
    t.v = v;
  }
}

// Publish this CTA's partial (one thread, after a CTA barrier that follows the
// CTA's update): the fields, then one arrival on the grid's counter with release
// semantics (cumulative: it also covers the other threads' update writes, which
// the CTA barrier ordered before it), so that a CTA that sees the count with
// acquire also sees the partial and the update.  The arrival is a reduction (no
// round trip).
__device__ __forceinline__ void big_publish(BigPartial& o, const BigTrack& t, BigBar* bar) {
  o.A = t.A;
  o.B = t.B;
  o.k = t.k;
  o.ph = t.ph;
  o.v = t.v;
  red_release_gpu_add_u32(&bar->arrived, 1u);
}

// Partials one lane of the gathering warp loads at once, and the most it handles
// (grids of up to 320 CTAs).
constexpr int BIG_GATHER_Q = 5;
constexpr int BIG_GATHER_MAX = 2 * BIG_GATHER_Q;

// Warp 0: wait until `target` partials have arrived in all (lane 0 polls the
// counter, bounded), then combine the G partials of this step, every lane
// loading its share at once; every lane gets the result.  This wait is the pivot
// step's only grid-wide synchronisation: a CTA publishes after its update, so
// once all G are in, every update of the step is done and visible.  Returns
// false if the wait hit its bound or another CTA has flagged an error (the flag
// is then set).
// Partials that are their own flags, polled by every CTA, save the counter's trip
// and cost more: 174 x 1653 to rank 136 takes 0.94 ms so and 1.10 to 1.15 with them,
// 513 x 512 to full rank 3.05 and 3.9 to 4.1, 2048 x 2048 to rank 512 8.94 and 9.07.
__device__ bool big_gather(const BigPartial* cur, int G, unsigned target, BigBar* bar, BigTrack& g) {
  const int lane = threadIdx.x & 31;
  g.init();
  int ok = 1;
  if (lane == 0) {
    unsigned sleep_ns = 16;
    for (long long it = 0; ld_acquire_gpu_u32(&bar->arrived) < target; ++it) {
      if (it > BIG_BAR_POLLS || *(volatile int*)&bar->error) {
        atomicExch(&bar->error, 1);
        ok = 0;
        break;
      }
      __nanosleep(sleep_ns);
      sleep_ns = sleep_ns < 64 ? sleep_ns * 2 : 64;
    }
  }
  ok = __shfl_sync(FULL, ok, 0);
  __syncwarp();  // lane 0's acquire orders the warp's loads below
  for (int base = 0; ok && base < G; base += 32 * BIG_GATHER_Q) {
    uint64_t qa[BIG_GATHER_Q], qb[BIG_GATHER_Q];
    uint32_t qk[BIG_GATHER_Q], qp[BIG_GATHER_Q];
    double qv[BIG_GATHER_Q];
#pragma unroll
    for (int q = 0; q < BIG_GATHER_Q; ++q) {
      if (base + lane + 32 * q < G) {
        const BigPartial* p = cur + base + lane + 32 * q;
        qa[q] = __ldcg(&p->A);
        qb[q] = __ldcg(&p->B);
        qk[q] = __ldcg(&p->k);
        qp[q] = __ldcg(&p->ph);
        qv[q] = __ldcg(&p->v);
      }
    }
#pragma unroll
    for (int q = 0; q < BIG_GATHER_Q; ++q)
      if (base + lane + 32 * q < G) big_combine(g.A, g.k, g.ph, g.B, g.v, qa[q], qk[q], qp[q], qb[q], qv[q]);
  }
  uint64_t a = g.A, b = g.B;
  uint32_t kk = g.k, ph = g.ph;
  double v = g.v;
  warp_track5(a, kk, ph, b, v);
  g.A = __shfl_sync(FULL, a, 0);
  g.B = __shfl_sync(FULL, b, 0);
  g.k = __shfl_sync(FULL, kk, 0);
  g.ph = __shfl_sync(FULL, ph, 0);
  g.v = __shfl_sync(FULL, v, 0);
  return ok != 0;
}

struct BigArgs {
  const double* ain;      // m x n input (column-major)
  double* A;              // m x n working copy (physical positions never change)
  double* fact;           // m x n factors in logical order, then int32 rowperm[m], colperm[n]
  char* res;              // result record (tci_result_head, rowp[kcap], colp[kcap], diag[kcap])
  BigPartial* parts;      // 2 x gridDim.x partials (double-buffered by pivot parity)
  double* pivs;           // signed pivot of every step (kmax)
  BigBar* bar;
  int m, n, kmax, kcap, leftorth;
  int pr, pc, mb, nb;     // CTA grid and block sizes
  int nres;               // columns of a block held in shared memory as well
  double reltol, abstol;
};

// The rank-1 update of a CTA's block: the active rows and columns (lists of
// local indices) of A at (r0, c0), x and y by list position, the logical
// positions for the argmax keys.  As rank1_tiles, but a warp takes 32 x 4 tiles
// with one row and four columns per lane, whole lines of A.  The first nres
// columns are also kept in shared memory (blk, leading dimension mb) and read
// from there; every result is written to A too, where the other CTAs read the
// pivot row and column.  A 2048 x 2048 matrix to rank 512: 9.0 ms, 1.06 cycles
// per element and SM in here; 10.5 ms and 1.3 when the block was read from L2.
struct BigBlock {
  double *A, *blk;
  int m, mb, nres, r0, c0, nr, nc;
  const double *xs, *ys;
  const uint16_t *act_r, *act_c, *pos_r, *pos_c;
  bool rev;
};
template <int MODE>
__device__ __forceinline__ void big_update(const BigBlock B, BigTrack& bt) {
  const int lane = threadIdx.x & 31;
  const int nti = (B.nr + 31) >> 5, ntj = (B.nc + 3) >> 2;
  const int di = BIG_NW % nti, dj = BIG_NW / nti;
  int tj = (threadIdx.x >> 5) / nti, ti = (threadIdx.x >> 5) - tj * nti;
  uint32_t top = 0;
  while (tj < ntj) {
    const int t = 32 * ti + lane, u0 = 4 * (B.rev ? ntj - 1 - tj : tj);
    const bool vi = t < B.nr;
    const int tt = min(t, B.nr - 1);
    const int ri = B.act_r[tt];
    double v[4], xv[1], yv[4], q[1][4];
    int cj[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int uu = min(u0 + b, B.nc - 1);
      cj[b] = B.act_c[uu];
      yv[b] = B.ys[uu];
    }
    double* const g = B.A + B.r0 + ri + (size_t)B.c0 * B.m;
#pragma unroll
    for (int b = 0; b < 4; ++b) v[b] = cj[b] < B.nres ? B.blk[ri + cj[b] * B.mb] : g[(size_t)cj[b] * B.m];
    xv[0] = B.xs[tt];
    tile_products<MODE>(xv, yv, q);
    uint32_t h = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      v[b] = __dsub_rn(v[b], q[0][b]);
      if (vi && u0 + b < B.nc) {
        if (cj[b] < B.nres) B.blk[ri + cj[b] * B.mb] = v[b];
        g[(size_t)cj[b] * B.m] = v[b];
      }
      h = max(h, (uint32_t)__double2hiint(v[b]) & 0x7fffffffu);
    }
    if (__any_sync(FULL, h + 1 >= top)) {
      const int lr = B.pos_r[ri];
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (vi && u0 + b < B.nc) bt.push(v[b], pack_key(lr, B.pos_c[cj[b]]), pack_key(B.r0 + ri, B.c0 + cj[b]));
      top = __reduce_max_sync(FULL, bt.A ? (uint32_t)((bt.A - 1) >> 32) : 0u);
    }
    ti += di;
    tj += dj;
    if (ti >= nti) {
      ti -= nti;
      tj += 1;
    }
  }
}

__global__ void __launch_bounds__(BIG_NT, 1) rrlu_big_kernel(BigArgs P) {
  extern __shared__ __align__(16) char smem[];
  __shared__ BigCtl ctl;
  const int tid = threadIdx.x, G = gridDim.x, b = blockIdx.x, m = P.m, n = P.n;
  const bool leftorth = P.leftorth != 0;
  const int r0 = (b / P.pc) * P.mb, c0 = (b % P.pc) * P.nb;
  const int r1 = min(m, r0 + P.mb), c1 = min(n, c0 + P.nb);
  const int nrb = max(0, r1 - r0), ncb = max(0, c1 - c0);  // block extent
  double* blk = (double*)smem;         // the block's first nres columns (mb x nres)
  double* xs = blk + (size_t)P.mb * P.nres;  // x of the active rows (mb)
  double* ys = xs + P.mb;              // y of the active columns (nb)
  uint16_t* stor_r = (uint16_t*)(ys + P.nb);  // logical row -> physical (m)
  uint16_t* stor_c = stor_r + m;              // (n)
  uint16_t* pos_r = stor_c + n;        // logical position of each block row, active rows, slot of each (mb each)
  uint16_t* act_r = pos_r + P.mb;
  uint16_t* slot_r = act_r + P.mb;
  uint16_t* pos_c = slot_r + P.mb;     // (nb each)
  uint16_t* act_c = pos_c + P.nb;
  uint16_t* slot_c = act_c + P.nb;
  unsigned gen = 0;
  for (int i = tid; i < m; i += BIG_NT) stor_r[i] = (uint16_t)i;
  for (int j = tid; j < n; j += BIG_NT) stor_c[j] = (uint16_t)j;
  for (int t = tid; t < nrb; t += BIG_NT) {
    pos_r[t] = (uint16_t)(r0 + t);
    act_r[t] = slot_r[t] = (uint16_t)t;
  }
  for (int u = tid; u < ncb; u += BIG_NT) {
    pos_c[u] = (uint16_t)(c0 + u);
    act_c[u] = slot_c[u] = (uint16_t)u;
  }
  PivotState S;  // thread 0's
  S.init(P.reltol, P.abstol);
  if (tid == 0) {
    ctl.factors[0] = ctl.factors[1] = 0;
    ctl.stop = 0;
    ctl.r = nrb;  // active row / column counts
    ctl.c = ncb;
  }
  // copy own block, first argmax
  BigTrack bt;
  bt.init();
  {
    const long long tot = (long long)nrb * ncb;
    for (long long e = tid; e < tot; e += BIG_NT) {
      const int i = r0 + (int)(e % nrb), j = c0 + (int)(e / nrb);
      const double v = P.ain[i + (size_t)j * m];
      P.A[i + (size_t)j * m] = v;
      if (j - c0 < P.nres) blk[i - r0 + (j - c0) * P.mb] = v;
      bt.push(v, pack_key(i, j), pack_key(i, j));
    }
  }
  block_track(bt, ctl);
  if (tid == 0) big_publish(P.parts[b], bt, P.bar);  // buffer 0: read at pivot 0
  bool ok = true;
  int K = 0;
  tci_result_head* head = (tci_result_head*)P.res;
  const int kcap = P.kcap;
  int* rowp = (int*)(P.res + sizeof(tci_result_head));
  int* colp = (int*)(P.res + sizeof(tci_result_head) + align_up((size_t)kcap * 4, 8));
  double* diag = (double*)(P.res + sizeof(tci_result_head) + 2 * align_up((size_t)kcap * 4, 8));
  // Decision of pivot step K (every CTA takes the same one), by one thread: the
  // error, the stopping rule, swaprow!(K, rl) / swapcol!(K, cl) on the maps, and
  // the pivot row and column leaving this block's active sets.
  auto decide = [&]() {
    const unsigned key = (unsigned)ctl.K, ph = (unsigned)ctl.kmax;
    const int rl = (int)(key & 0xffffu), cl = (int)(key >> 16);
    const int R = (int)(ph & 0xffffu), Cc = (int)(ph >> 16);
    const double piv = ctl.piv;
    ctl.stop = S.decide(piv, K, P.reltol, P.abstol) ? 1 : 0;
    ctl.err = __longlong_as_double((long long)S.err);
    ctl.factors[(K + 1) & 1] = 0;  // the flags of pivot K - 1: every thread has passed them
    if (!ctl.stop) {
      if (b == 0) {
        diag[K] = fabs(piv);
        P.pivs[K] = piv;
      }
      // swaprow!(K, rl), swapcol!(K, cl) on the maps
      const int sr = stor_r[K];
      stor_r[K] = (uint16_t)R;
      stor_r[rl] = (uint16_t)sr;
      if (sr >= r0 && sr < r1) pos_r[sr - r0] = (uint16_t)rl;
      const int sc = stor_c[K];
      stor_c[K] = (uint16_t)Cc;
      stor_c[cl] = (uint16_t)sc;
      if (sc >= c0 && sc < c1) pos_c[sc - c0] = (uint16_t)cl;
      // the pivot row and column leave this block's active sets
      if (R >= r0 && R < r1) {
        pos_r[R - r0] = (uint16_t)K;
        const int s = slot_r[R - r0], last = act_r[ctl.r - 1];
        act_r[s] = (uint16_t)last;
        slot_r[last] = (uint16_t)s;
        ctl.r -= 1;
      }
      if (Cc >= c0 && Cc < c1) {
        pos_c[Cc - c0] = (uint16_t)K;
        const int s = slot_c[Cc - c0], last = act_c[ctl.c - 1];
        act_c[s] = (uint16_t)last;
        slot_c[last] = (uint16_t)s;
        ctl.c -= 1;
      }
    }
  };
  while (ok) {
    // the partials of pivot K are in buffer K & 1: a CTA writes the next set to
    // the other buffer, so a fast CTA never overwrites what a slow one reads
    BigPartial* const cur = P.parts + (size_t)(K & 1) * G;
    // ---- the pivot: argmax of abs2 over the trailing block, from the G partials
    // (warp 0 waits for them); unless the exact pass is needed, lane 0 also takes
    // the decision
    if (tid < 32) {
      BigTrack g;
      const bool got = big_gather(cur, G, (unsigned)(K + 1) * (unsigned)G, P.bar, g);
      if (tid == 0) {
        ctl.bar_err = got ? 0 : 1;
        if (got) {
          const uint64_t Mstar = g.A ? g.A - 1 : 0;
          const bool safe = Mstar >= SQ_SMALL && Mstar < SQ_BIG;
          const bool close = g.B != 0 && (g.B - 1) + 16 >= Mstar;
          ctl.red_u[BIG_NW] = Mstar;
          ctl.need_exact = (g.A != 0 && !(safe && !close)) ? 1 : 0;
          if (g.A == 0) {  // every element NaN: the scan keeps its start
            ctl.kmax = (int)(((unsigned)stor_c[K] << 16) | (unsigned)stor_r[K]);
            ctl.K = (K << 16) | K;
            ctl.piv = __ldcg(&P.A[stor_r[K] + (size_t)stor_c[K] * m]);
          } else {
            ctl.kmax = (int)g.ph;
            ctl.K = (int)g.k;
            ctl.piv = g.v;
          }
          if (!ctl.need_exact) decide();
        }
      }
    }
    __syncthreads();
    if (ctl.bar_err) {
      ok = false;
      break;
    }
    if (ctl.need_exact) {  // squares of the elements near the maximum (rare)
      const uint64_t Mstar = ctl.red_u[BIG_NW];
      const int nr = ctl.r, nc = ctl.c;
      ArgBest ab;
      ab.init();
      uint32_t abph = 0;
      for (long long e = tid; e < (long long)nr * nc; e += BIG_NT) {
        const int i = r0 + act_r[(int)(e % nr)], j = c0 + act_c[(int)(e / nr)];
        const double v = P.A[i + (size_t)j * m];
        if (near_max(abs_bits(v), Mstar)) {
          const uint32_t key = pack_key(pos_r[i - r0], pos_c[j - c0]);
          const uint64_t q = (uint64_t)__double_as_longlong(__dmul_rn(v, v)) + 1;
          if (q > ab.s || (q == ab.s && key < ab.key)) {
            ab.s = q;
            ab.key = key;
            ab.val = v;
            abph = pack_key(i, j);
          }
        }
      }
      BigTrack et;
      et.A = ab.s;
      et.B = 0;
      et.k = ab.key;
      et.ph = abph;
      et.v = ab.val;
      ok = big_barrier(P.bar, G, gen, ctl);  // everyone has read the partials
      if (!ok) break;
      block_track(et, ctl);
      if (tid == 0) {
        BigPartial& o = cur[b];
        o.A = et.A;
        o.B = 0;
        o.k = et.k;
        o.ph = et.ph;
        o.v = et.v;
      }
      ok = big_barrier(P.bar, G, gen, ctl);
      if (!ok) break;
      BigTrack g;
      g.init();
      for (int t = tid; t < G; t += BIG_NT) {
        const BigPartial* q = cur + t;
        big_combine(g.A, g.k, g.ph, g.B, g.v, __ldcg(&q->A), __ldcg(&q->k), __ldcg(&q->ph), __ldcg(&q->B),
                    __ldcg(&q->v));
      }
      block_track(g, ctl);
      if (tid == 0) {
        if (g.A) {
          ctl.kmax = (int)g.ph;
          ctl.K = (int)g.k;
          ctl.piv = g.v;
        }
        decide();
      }
      __syncthreads();
    }
    const int R = (int)((unsigned)ctl.kmax & 0xffffu), Cc = (int)((unsigned)ctl.kmax >> 16);
    const double piv = ctl.piv;
    if (ctl.stop) break;
    ++K;
    if (K == P.kmax) break;  // the trailing update after the last pivot is not observable
    // ---- x (pivot column) for the active rows, y (pivot row) for the active columns
    // (one element per thread: the x and y entries on different threads)
    const int nr = ctl.r, nc = ctl.c;
    const PivotDivisor D(piv);
    JoinFlags fl{false, 0};
    for (int t = tid; t < nr + nc; t += BIG_NT) {
      if (t < nr) {
        const double v = __ldcg(&P.A[r0 + act_r[t] + (size_t)Cc * m]);
        xs[t] = leftorth ? D.quo(v) : v;
        fl.join(xs[t]);
      } else {
        const int u = t - nr;
        const double v = __ldcg(&P.A[R + (size_t)(c0 + act_c[u]) * m]);
        ys[u] = leftorth ? v : D.quo(v);
        fl.join(ys[u]);
      }
    }
    if (fl.factors) atomicOr(&ctl.factors[(K - 1) & 1], fl.factors);
    __syncthreads();
    const int mode = min(ctl.factors[(K - 1) & 1], (int)PROD_FP64);
    // ---- rank-1 update of the block's active part, fused with its argmax.
    // The columns are walked in reverse on odd pivots, so the part of the block
    // the last pass touched last is still in L1.
    bt.init();
    if (nr > 0 && nc > 0) {
      const BigBlock B{P.A, blk, m, P.mb, P.nres, r0, c0, nr, nc, xs, ys, act_r, act_c, pos_r, pos_c, (K & 1) != 0};
      if (mode == PROD_DENSE) big_update<PROD_DENSE>(B, bt);
      else if (mode == PROD_MIXED) big_update<PROD_MIXED>(B, bt);
      else big_update<PROD_FP64>(B, bt);
    }
    block_track_to0(bt, ctl);
    // read at pivot K (already incremented); no grid barrier: the next gather
    // waits for every CTA's partial
    if (tid == 0) big_publish(P.parts[(size_t)(K & 1) * G + b], bt, P.bar);
  }
  if (ok) ok = big_barrier(P.bar, G, gen, ctl);  // every pivot value is recorded
  if (!ok) {
    if (b == 0 && tid == 0) head->status = TCI_ST_TOO_LARGE;
    return;
  }
  // ---- the factors in logical order, with the deferred scaling of addpivot!,
  // and the NaN scan of L and U (matrixlu.jl:162-169)
  int bad = 0;
  {
    const long long tot = (long long)nrb * ncb;
    for (long long e = tid; e < tot; e += BIG_NT) {
      const int i = r0 + (int)(e % nrb), j = c0 + (int)(e / nrb);
      const int lr = pos_r[i - r0], lc = pos_c[j - c0];
      double v = P.A[i + (size_t)j * m];
      if (leftorth && lc < K && lr > lc) v = PivotDivisor(__ldcg(&P.pivs[lc])).quo(v);
      if (!leftorth && lr < K && lc > lr) v = PivotDivisor(__ldcg(&P.pivs[lr])).quo(v);
      const bool inL = lc < K && lr >= lc;
      const bool inU = lr < K && lr <= lc;
      if ((inL || inU) && is_nan_bits(v)) bad = 1;
      P.fact[lr + (size_t)lc * m] = v;
    }
  }
  bad = __syncthreads_or(bad);
  if (tid == 0) P.parts[b].nan = bad;
  ok = big_barrier(P.bar, G, gen, ctl);
  if (!ok) {
    if (b == 0 && tid == 0) head->status = TCI_ST_TOO_LARGE;
    return;
  }
  if (b == 0) {
    int nan = 0;
    for (int t = tid; t < G; t += BIG_NT) nan |= (int)__ldcg(&P.parts[t].nan);
    nan = __syncthreads_or(nan);
    int* fr = (int*)(P.fact + (size_t)m * n);
    for (int i = tid; i < m; i += BIG_NT) fr[i] = stor_r[i];
    for (int j = tid; j < n; j += BIG_NT) fr[m + j] = stor_c[j];
    for (int q = tid; q < K; q += BIG_NT) {
      rowp[q] = stor_r[q];
      colp[q] = stor_c[q];
    }
    if (tid == 0) {
      head->status = nan ? TCI_ST_NAN : 0;
      head->npivot = K;
      head->error = K >= min(m, n) ? 0.0 : ctl.err;
      head->maxabs = 0.0;
      head->maxabs_nan = 0;
      head->lut_used = 0;
    }
  }
}

// ------------------------------------------------------------ cluster rrLU
// One rank-revealing LU on a thread-block cluster: the matrix lives in the
// shared memory of the cluster's CTAs (a pr x pc grid, CTA (p, q) owns row block
// p x column block q), and nothing of it goes through L2 between the fill and
// the factors.  As in the multi-CTA kernel above, rows and columns stay where
// they are: logical positions are tracked as permutations, the argmax keys are
// logical, and the stored factors are scaled when they are written out, so
// pivots and factors are bit-identical to rrlu_loop's.
// Per pivot: each CTA reduces its block's argmax and writes it into every CTA's
// shared memory; one cluster barrier; every warp reduces the CTAs' winners and
// takes the decision itself; x and y come from the owners' shared memory (the
// pivot row and column have left the trailing block there, so they are stable);
// one CTA barrier; the rank-1 update of the block's active part.
// Bound by that chain (about 5 thousand cycles a pivot: block argmax and
// exchange 1.7, decision 0.7, x and y 1.4, one tile 1.6 thousand) until the
// update outgrows it.  381 x 517 to rank 140 on 16 CTAs: 1.03 ms; on one CTA,
// from L2, 14.1 ms.
namespace cg = cooperative_groups;
constexpr int CL_NT = 512;
constexpr int CL_NW = CL_NT / 32;
constexpr int CL_MAX = 16;  // CTAs of a cluster at most

struct ClusterCtl {
  unsigned long long red_a[CL_NW], red_b[CL_NW];
  unsigned red_k[CL_NW], red_p[CL_NW];
  double red_v[CL_NW];
  BigPartial parts[2][CL_MAX];
  int factors[2];
  int nr, nc;  // active rows and columns of the block
  int bad[CL_MAX];
  unsigned long long mx[CL_MAX];
};

struct ClusterJob {
  int m, n, kmax, leftorth;
  int pr, pc, mb, nb;  // CTA grid and block sizes
  int nres;            // columns of a block held in shared memory; the rest, if any, in `spill`
  double* spill;       // ncta x mb x (nb - nres) doubles of device scratch
  double reltol, abstol;
  double* pivs;        // kmax signed pivots (device scratch)
  double* fact;        // the factored m x n matrix, or null
  int *rowperm, *colperm;  // full permutations (m, n), or null
  int *rowk, *colk;        // their first npivot entries, or null
  double* diag;        // |pivots| (kmax), or null
};
struct ClusterResult {
  int K, nan;  // nan and mx (largest |value| bit pattern): valid in CTA 0
  double err;
  unsigned long long mx;
};

// Column u of CTA `rank`'s block: in its shared memory (blk), or in the spill.
template <bool SPILL>
struct ClusterBlock {
  double* blk;
  double* spill;
  int mb, nb, nres;
  __device__ __forceinline__ double* col(int u, int rank) const {
    if (SPILL && u >= nres) return spill + ((size_t)rank * (nb - nres) + (u - nres)) * mb;
    return blk + u * mb;
  }
  // entry (t, u) of another CTA's block; its spilled columns come from L2
  __device__ __forceinline__ double remote(const cg::cluster_group& cl, int t, int u, int rank) const {
    if (SPILL && u >= nres) return __ldcg(col(u, rank) + t);
    return cl.map_shared_rank(blk, rank)[t + u * mb];
  }
};

// Shared memory of one CTA: the block, x and y, the maps (16-bit: logical ->
// physical for all rows and columns; per block row and column its logical
// position, the active list and the slot in it).
__host__ __device__ inline size_t cluster_smem(int m, int n, int mb, int nb, int nres) {
  return ((size_t)mb * nres + mb + nb) * 8 + ((size_t)m + n) * 2 + ((size_t)mb + nb) * 6 + 64;
}

// This CTA's partial to every CTA of the cluster, then the cluster barrier.
__device__ __forceinline__ void cluster_exchange(const BigTrack& t, ClusterCtl& ctl, int par, const cg::cluster_group& cl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t a = t.A, b = t.B;
  uint32_t k = t.k, ph = t.ph;
  double v = t.v;
  warp_track5(a, k, ph, b, v);
  if (lane == 0) {
    ctl.red_a[warp] = a;
    ctl.red_b[warp] = b;
    ctl.red_k[warp] = k;
    ctl.red_p[warp] = ph;
    ctl.red_v[warp] = v;
  }
  __syncthreads();
  // The CTA barrier orders the other warps' writes before warp 0's release, so
  // only warp 0 pays for one (790 cycles a pivot when every warp did).
  if (warp == 0) {
    a = lane < CL_NW ? ctl.red_a[lane] : 0ULL;
    b = lane < CL_NW ? ctl.red_b[lane] : 0ULL;
    k = lane < CL_NW ? ctl.red_k[lane] : 0xffffffffu;
    ph = lane < CL_NW ? ctl.red_p[lane] : 0u;
    v = lane < CL_NW ? ctl.red_v[lane] : 0.0;
    warp_track5(a, k, ph, b, v);
    if (lane < (int)cl.num_blocks()) {
      BigPartial* o = cl.map_shared_rank(&ctl.parts[par][cl.block_rank()], lane);
      o->A = a;
      o->B = b;
      o->k = k;
      o->ph = ph;
      o->v = v;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  } else {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The winner over the CTAs, to every lane of every warp.
__device__ __forceinline__ BigTrack cluster_winner(const ClusterCtl& ctl, int par, int ncta) {
  const int lane = threadIdx.x & 31;
  BigTrack g;
  g.init();
  if (lane < ncta) {
    const BigPartial& q = ctl.parts[par][lane];
    g.A = q.A;
    g.B = q.B;
    g.k = q.k;
    g.ph = q.ph;
    g.v = q.v;
  }
  warp_track5(g.A, g.k, g.ph, g.B, g.v);
  return g;
}

template <int MODE, bool SPILL>
__device__ __forceinline__ void cluster_update(const ClusterBlock<SPILL>& B, int rank, int r0, int c0, int nr, int nc, const double* xs,
                                               const double* ys, const uint16_t* act_r, const uint16_t* act_c,
                                               const uint16_t* pos_r, const uint16_t* pos_c, BigTrack& bt) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane & 7, lc = lane >> 3;
  const int nti = (nr + 15) >> 4, ntj = (nc + 7) >> 3;
  int tj = warp / nti, ti = warp - tj * nti;
  const int dj = CL_NW / nti, di = CL_NW - dj * nti;
  uint32_t top = 0;
  while (tj < ntj) {
    const int t0 = 16 * ti + lr, u0 = 8 * tj + lc;
    const bool vi[2] = {t0 < nr, t0 + 8 < nr}, vj[2] = {u0 < nc, u0 + 4 < nc};
    int ri[2], cj[2];
    double v[2][2], xv[2], yv[2], q[2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      ri[a] = act_r[min(t0 + 8 * a, nr - 1)];
      cj[a] = act_c[min(u0 + 4 * a, nc - 1)];
      xv[a] = xs[ri[a]];
      yv[a] = ys[cj[a]];
    }
    double* const p[2] = {B.col(cj[0], rank), B.col(cj[1], rank)};
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int a = 0; a < 2; ++a) v[a][b] = p[b][ri[a]];
    tile_products<MODE>(xv, yv, q);
    uint32_t h = 0;
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        v[a][b] = __dsub_rn(v[a][b], q[a][b]);
        if (vi[a] && vj[b]) p[b][ri[a]] = v[a][b];
        h = max(h, (uint32_t)__double2hiint(v[a][b]) & 0x7fffffffu);
      }
    if (__any_sync(FULL, h + 1 >= top)) {
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int a = 0; a < 2; ++a)
          if (vi[a] && vj[b]) bt.push(v[a][b], pack_key(pos_r[ri[a]], pos_c[cj[b]]), pack_key(r0 + ri[a], c0 + cj[b]));
      top = __reduce_max_sync(FULL, bt.A ? (uint32_t)((bt.A - 1) >> 32) : 0u);
    }
    ti += di;
    tj += dj;
    if (ti >= nti) {
      ti -= nti;
      tj += 1;
    }
  }
}

// The body, by every thread of every CTA of the cluster.  fill(i, j) gives the
// matrix.
template <bool SPILL, class Fill>
__device__ ClusterResult cluster_rrlu(const ClusterJob& P, char* smem, ClusterCtl& ctl, const Fill& fill) {
  const cg::cluster_group cl = cg::this_cluster();
  // The first exchange writes to every CTA's shared memory, which is there once that
  // CTA has started: all arrive here, and the fill covers the wait.
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const int tid = threadIdx.x, ncta = P.pr * P.pc, rank = (int)cl.block_rank(), m = P.m, n = P.n;
  const bool leftorth = P.leftorth != 0;
  const int bp = rank / P.pc, bq = rank % P.pc, mb = P.mb, nb = P.nb;
  const int r0 = bp * mb, c0 = bq * nb;
  const int nrb = max(0, min(m, r0 + mb) - r0), ncb = max(0, min(n, c0 + nb) - c0);
  double* blk = (double*)smem;  // column-major, leading dimension mb
  const ClusterBlock<SPILL> B{blk, P.spill, mb, nb, P.nres};
  double* xs = blk + (size_t)mb * P.nres;
  double* ys = xs + mb;
  uint16_t* stor_r = (uint16_t*)(ys + nb);
  uint16_t* stor_c = stor_r + m;
  uint16_t* pos_r = stor_c + n;
  uint16_t* act_r = pos_r + mb;
  uint16_t* slot_r = act_r + mb;
  uint16_t* pos_c = slot_r + mb;
  uint16_t* act_c = pos_c + nb;
  uint16_t* slot_c = act_c + nb;
  for (int i = tid; i < m; i += CL_NT) stor_r[i] = (uint16_t)i;
  for (int j = tid; j < n; j += CL_NT) stor_c[j] = (uint16_t)j;
  for (int t = tid; t < nrb; t += CL_NT) {
    pos_r[t] = (uint16_t)(r0 + t);
    act_r[t] = slot_r[t] = (uint16_t)t;
  }
  for (int u = tid; u < ncb; u += CL_NT) {
    pos_c[u] = (uint16_t)(c0 + u);
    act_c[u] = slot_c[u] = (uint16_t)u;
  }
  if (tid == 0) {
    ctl.nr = nrb;
    ctl.nc = ncb;
    ctl.factors[0] = ctl.factors[1] = 0;
  }
  BigTrack bt;
  bt.init();
  unsigned long long mx = 0;
  if (nrb > 0 && ncb > 0) {
    // fill picks what gives an element and how many are taken at once, so that each
    // kind has its own loop (loads overlap; f's call among them would part them)
    fill([&](const auto& element, auto together) {
      const int sq = CL_NT / nrb, sr = CL_NT - sq * nrb;
      int u = tid / nrb, t = tid - u * nrb;
#pragma unroll decltype(together)::value
      for (int e = tid; e < nrb * ncb; e += CL_NT) {
        const double v = element(r0 + t, c0 + u);
        B.col(u, rank)[t] = v;
        mx = max(mx, (unsigned long long)abs_bits(v));
        const uint32_t key = pack_key(r0 + t, c0 + u);
        bt.push(v, key, key);
        t += sr;
        u += sq;
        if (t >= nrb) {
          t -= nrb;
          u += 1;
        }
      }
    });
  }
  PivotState S;
  S.init(P.reltol, P.abstol);
  int K = 0;
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // every CTA has started
  while (P.kmax > 0) {
    // ---- the pivot: argmax of abs2 over the cluster's trailing blocks
    const int par = K & 1;
    cluster_exchange(bt, ctl, par, cl);
    if (tid == 0 && K > 0) ctl.factors[(K - 1) & 1] = 0;  // read by all before the barrier
    BigTrack g = cluster_winner(ctl, par, ncta);
    if (!track_decides(g.A, g.B)) {
      if (g.A == 0) {  // every element NaN: the scan keeps its start
        g.k = (uint32_t)((K << 16) | K);
        g.ph = pack_key(stor_r[K], stor_c[K]);
        const int pi = stor_r[K], pj = stor_c[K];
        g.v = B.remote(cl, pi % mb, pj % nb, (pi / mb) * P.pc + pj / nb);
      } else {  // squares of the elements near the maximum
        const int nr = ctl.nr, nc = ctl.nc;
        BigTrack et;
        et.init();
        for (int e = tid; e < nr * nc; e += CL_NT) {
          const int i = act_r[e % nr], j = act_c[e / nr];
          const double v = B.col(j, rank)[i];
          if (near_max(abs_bits(v), g.A - 1)) {
            const uint32_t key = pack_key(pos_r[i], pos_c[j]);
            const uint64_t q = (uint64_t)__double_as_longlong(__dmul_rn(v, v)) + 1;
            if (q > et.A || (q == et.A && key < et.k)) {
              et.A = q;
              et.k = key;
              et.ph = pack_key(r0 + i, c0 + j);
              et.v = v;
            }
          }
        }
        cl.sync();  // everyone has read the partials
        cluster_exchange(et, ctl, par, cl);
        g = cluster_winner(ctl, par, ncta);
      }
    }
    if (S.decide(g.v, K, P.reltol, P.abstol)) break;
    const int rl = (int)(g.k & 0xffffu), cc = (int)(g.k >> 16), R = (int)(g.ph & 0xffffu), C = (int)(g.ph >> 16);
    if (tid == CL_NT - 32) {  // swaprow!(K, rl) on the maps; the pivot row leaves its block's active set
      const int sr = stor_r[K];
      stor_r[K] = (uint16_t)R;
      stor_r[rl] = (uint16_t)sr;
      if (sr >= r0 && sr < r0 + nrb) pos_r[sr - r0] = (uint16_t)rl;
      if (R >= r0 && R < r0 + nrb) {
        pos_r[R - r0] = (uint16_t)K;
        const int s = slot_r[R - r0], last = act_r[ctl.nr - 1];
        act_r[s] = (uint16_t)last;
        slot_r[last] = (uint16_t)s;
        ctl.nr -= 1;
      }
    } else if (tid == CL_NT - 64) {  // swapcol!(K, cc)
      const int sc = stor_c[K];
      stor_c[K] = (uint16_t)C;
      stor_c[cc] = (uint16_t)sc;
      if (sc >= c0 && sc < c0 + ncb) pos_c[sc - c0] = (uint16_t)cc;
      if (C >= c0 && C < c0 + ncb) {
        pos_c[C - c0] = (uint16_t)K;
        const int s = slot_c[C - c0], last = act_c[ctl.nc - 1];
        act_c[s] = (uint16_t)last;
        slot_c[last] = (uint16_t)s;
        ctl.nc -= 1;
      }
    } else if (tid == CL_NT - 96 && rank == 0) {
      P.pivs[K] = g.v;
      if (P.diag) P.diag[K] = __longlong_as_double((long long)abs_bits(g.v));
    }
    ++K;
    if (K == P.kmax) break;  // the trailing update after the last pivot is not observable
    // ---- x (pivot column) and y (pivot row) for the block, by physical place
    JoinFlags fl{false, 0};
    {
      const int xo = bp * P.pc + C / nb, yo = (R / mb) * P.pc + bq;  // owners
      auto entry = [&](int t) {
        return t < nrb ? B.remote(cl, t, C % nb, xo) : B.remote(cl, R % mb, t - nrb, yo);
      };
      double v = tid < nrb + ncb ? entry(tid) : 0.0;  // under way during the division set-up
      const PivotDivisor D(g.v);
      for (int t = tid; t < nrb + ncb; t += CL_NT) {
        const bool isx = t < nrb;
        if (t != tid) v = entry(t);
        if (isx == leftorth) v = D.quo(v);
        fl.join(v);
        if (isx) xs[t] = v;
        else ys[t - nrb] = v;
      }
    }
    if (fl.factors) atomicOr(&ctl.factors[(K - 1) & 1], fl.factors);
    __syncthreads();
    const int mode = min(ctl.factors[(K - 1) & 1], (int)PROD_FP64);
    bt.init();
    const int nr = ctl.nr, nc = ctl.nc;
    if (nr > 0 && nc > 0) {
      if (mode == PROD_DENSE)
        cluster_update<PROD_DENSE>(B, rank, r0, c0, nr, nc, xs, ys, act_r, act_c, pos_r, pos_c, bt);
      else if (mode == PROD_MIXED)
        cluster_update<PROD_MIXED>(B, rank, r0, c0, nr, nc, xs, ys, act_r, act_c, pos_r, pos_c, bt);
      else
        cluster_update<PROD_FP64>(B, rank, r0, c0, nr, nc, xs, ys, act_r, act_c, pos_r, pos_c, bt);
    }
  }
  // ---- permutations, and the factors in logical order with the deferred
  // scaling of addpivot! and the NaN check of L and U (matrixlu.jl:162-169);
  // without factors to write only L and U are visited, and dividing by a finite
  // pivot neither makes nor loses a NaN
  cl.sync();  // the maps and every pivot value are in place; no CTA reads another's block any more
  int bad = 0;
  for (int u = tid >> 5; u < ncb; u += CL_NW) {
    const int lc = pos_c[u];
    const PivotDivisor D(leftorth && lc < K ? __ldcg(&P.pivs[lc]) : 1.0);
    for (int t = tid & 31; t < nrb; t += 32) {
      const int lr = pos_r[t];
      if (!P.fact && lr >= K && lc >= K) continue;
      double v = B.col(u, rank)[t];
      if (leftorth && lc < K && lr > lc && (P.fact || !D.safe)) v = D.quo(v);
      if (!leftorth && lr < K && lc > lr) {
        const double piv = __ldcg(&P.pivs[lr]);
        if (P.fact || !int_safe(piv) || abs_bits(piv) == 0) v = PivotDivisor(piv).quo(v);
      }
      if ((lc < K && lr >= lc) || (lr < K && lr <= lc)) bad |= is_nan_bits(v) ? 1 : 0;
      if (P.fact) P.fact[lr + (size_t)lc * m] = v;
    }
  }
  bad = __syncthreads_or(bad);
  mx = warp_max_u64(mx);
  if ((tid & 31) == 0) ctl.red_a[tid >> 5] = mx;
  __syncthreads();
  if (tid < 32) {
    mx = warp_max_u64(tid < CL_NW ? ctl.red_a[tid] : 0ULL);
    if (tid == 0) {
      *cl.map_shared_rank(&ctl.bad[rank], 0) = bad;
      *cl.map_shared_rank(&ctl.mx[rank], 0) = mx;
    }
  }
  if (rank == 0) {
    for (int i = tid; i < m; i += CL_NT) {
      if (P.rowperm) P.rowperm[i] = stor_r[i];
      if (P.rowk && i < K) P.rowk[i] = stor_r[i];
    }
    for (int j = tid; j < n; j += CL_NT) {
      if (P.colperm) P.colperm[j] = stor_c[j];
      if (P.colk && j < K) P.colk[j] = stor_c[j];
    }
  }
  cl.sync();
  ClusterResult r;
  r.K = K;
  r.nan = 0;
  r.mx = 0;
  if (rank == 0)
    for (int t = 0; t < ncta; ++t) {
      r.nan |= ctl.bad[t];
      r.mx = max(r.mx, ctl.mx[t]);
    }
  r.err = K >= min(m, n) ? 0.0 : __longlong_as_double((long long)S.err);
  return r;
}

// The smallest cluster to try for a matrix of `elems` elements, of at most `most` CTAs:
// up to 100 x 100 the update does not fill eight.
inline int cluster_first(int64_t elems, int most) { return most > 8 && elems >= 10000 ? 16 : 8; }

// CTA grid of a cluster of `ncta` (a power of two) for an m x n matrix: the
// smallest block perimeter (x and y exchanged per pivot).
struct ClusterGrid {
  int pr, pc, mb, nb;
};
inline ClusterGrid cluster_grid(int m, int n, int ncta) {
  ClusterGrid best{1, ncta, m, (n + ncta - 1) / ncta};
  for (int pr = 1; pr <= ncta; pr *= 2) {
    const int pc = ncta / pr, mb = (m + pr - 1) / pr, nb = (n + pc - 1) / pc;
    if (mb + nb < best.mb + best.nb) best = ClusterGrid{pr, pc, mb, nb};
  }
  return best;
}

}  // namespace

// Shared-memory budget of one CTA of the step kernel.
size_t tci_step_smem_bytes() {
  // 228 KB per SM, 1 KB reserved per CTA, ~2 KB of static shared memory per CTA
  return (size_t)(228 * 1024) / TCI_CTAS_PER_SM - 3 * 1024 - 1024 * (TCI_CTAS_PER_SM - 1);
}

// Dynamic shared memory of the resident kernel (its static shared memory holds
// the task record and the f parameters as well).
size_t tci_resident_smem_bytes() { return tci_step_smem_bytes(); }

// Dynamic shared memory of one multi-CTA rrLU CTA (one per SM).
size_t tci_big_smem_limit() { return (size_t)(228 * 1024) - 3 * 1024; }

cudaError_t tci_step_configure() {
  cudaError_t e = cudaFuncSetAttribute(tci_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)tci_step_smem_bytes());
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(tci_resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)tci_resident_smem_bytes());
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(rrlu_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)tci_big_smem_limit());
}

// Multi-CTA rrLU (rrlu_big_kernel).  The CTA grid: pr x pc <= G CTAs with the
// largest count, then the most square blocks.  Shared memory per CTA: the
// permutations and lists (16-bit), x and y, and as many columns of the block as
// the rest takes.
namespace {
struct BigGrid {
  int pr, pc, mb, nb;
};
// G: the task kernels' grid (TCI_CTAS_PER_SM per SM); the multi-CTA rrLU runs
// one CTA per SM.
BigGrid big_grid(int64_t m, int64_t n, int G) {
  G = std::max(1, G / TCI_CTAS_PER_SM);
  G = std::min(G, 32 * BIG_GATHER_MAX);  // one gathering warp reads every partial
  BigGrid best{1, 1, (int)m, (int)n};
  double best_score = -1.0;
  for (int pr = 1; pr <= G; ++pr) {
    const int pc = G / pr;
    if (pr > m || pc > n || pc < 1) continue;
    const int mb = (int)((m + pr - 1) / pr), nb = (int)((n + pc - 1) / pc);
    const double aspect = (double)mb / nb;
    const double score = (double)pr * pc - 1e-3 * std::fabs(std::log(aspect));
    if (score > best_score) {
      best_score = score;
      best = BigGrid{pr, pc, mb, nb};
    }
  }
  return best;
}
}  // namespace
size_t tci_rrlu_big_smem(int64_t m, int64_t n, int G) {
  const BigGrid g = big_grid(m, n, G);
  return (size_t)(2 * (m + n) + 14 * ((int64_t)g.mb + g.nb) + 64);
}
bool tci_rrlu_big_fits(int64_t m, int64_t n, int G) {
  return m >= 1 && n >= 1 && m <= 65535 && n <= 65535 && tci_rrlu_big_smem(m, n, G) <= tci_big_smem_limit();
}
size_t tci_rrlu_big_scratch_bytes(int grid, int kmax) {
  return 64 + 2 * (size_t)grid * sizeof(BigPartial) + (size_t)std::max(kmax, 1) * sizeof(double);
}

// Launch on up to `grid` CTAs (all co-resident: cooperative launch).  scratch
// holds the grid barrier, the partials and the pivot values
// (tci_rrlu_big_scratch_bytes); it is cleared here.  res is a device result
// record with room for kcap pivots.
cudaError_t tci_rrlu_big_launch(const double* ain, double* work, double* fact, char* res, void* scratch, int m,
                                int n, int kmax, int kcap, int leftorth, double reltol, double abstol, int grid,
                                cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(scratch, 0, tci_rrlu_big_scratch_bytes(grid, kmax), stream);
  if (e != cudaSuccess) return e;
  const BigGrid g = big_grid(m, n, grid);
  BigArgs a;
  a.ain = ain;
  a.A = work;
  a.fact = fact;
  a.res = res;
  a.bar = (BigBar*)scratch;
  a.parts = (BigPartial*)((char*)scratch + 64);
  a.pivs = (double*)((char*)scratch + 64 + 2 * (size_t)grid * sizeof(BigPartial));
  a.m = m;
  a.n = n;
  a.kmax = kmax;
  a.kcap = kcap;
  a.leftorth = leftorth;
  a.pr = g.pr;
  a.pc = g.pc;
  a.mb = g.mb;
  a.nb = g.nb;
  a.reltol = reltol;
  a.abstol = abstol;
  const size_t fixed = tci_rrlu_big_smem(m, n, grid);
  a.nres = (int)std::min<size_t>((size_t)g.nb, (tci_big_smem_limit() - fixed) / ((size_t)g.mb * 8));
  const size_t smem = fixed + (size_t)a.nres * g.mb * 8;
  void* args[] = {(void*)&a};
  return cudaLaunchCooperativeKernel((const void*)rrlu_big_kernel, dim3(g.pr * g.pc), dim3(BIG_NT), args, smem,
                                     stream);
}

// Launch the resident kernel on every SM, all CTAs resident at once
// (cooperative launch), after clearing the per-launch part of its state.
// slots/qc are mapped pinned host memory, st device memory.
// cluster > 1: in clusters of that many CTAs, which leaves the other GPCs whole
// for a cluster kernel beside it (the grid is then far below one CTA per SM, so
// all of it is resident without a cooperative launch).
cudaError_t tci_resident_launch(tci_queue_slot* slots, uint32_t mask, tci_resident_state* st, tci_queue_ctl* qc,
                                int grid, int cluster, unsigned long long wait_ns, cudaStream_t stream) {
  const size_t off = offsetof(tci_resident_state, count);
  cudaError_t e = cudaMemsetAsync((char*)st + off, 0, sizeof(tci_resident_state) - off, stream);
  if (e != cudaSuccess) return e;
  size_t smem = tci_resident_smem_bytes();
  if (cluster > 1) {
    e = cudaFuncSetAttribute(tci_resident_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, tci_resident_kernel, slots, mask, st, qc, smem, wait_ns);
  }
  void* args[] = {(void*)&slots, (void*)&mask, (void*)&st, (void*)&qc, (void*)&smem, (void*)&wait_ns};
  return cudaLaunchCooperativeKernel((const void*)tci_resident_kernel, dim3(grid), dim3(NT), args, smem, stream);
}

// Launch one step.  counter must be zero (the launcher clears it on the stream).
cudaError_t tci_step_launch(const char* blob_dev, char* res_dev, const int* order_dev, int ntasks,
                            int* counter_dev, int grid, double* cta_area, size_t cta_stride, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(counter_dev, 0, sizeof(int), stream);
  if (e != cudaSuccess) return e;
  tci_step_kernel<<<grid, NT, tci_step_smem_bytes(), stream>>>(blob_dev, res_dev, order_dev, ntasks,
                                                              counter_dev, tci_step_smem_bytes(), cta_area,
                                                              cta_stride);
  return cudaGetLastError();
}

extern const tci_kernel_set kernels = {TCI_STEP_THREADS, TCI_CTAS_PER_SM, tci_step_smem_bytes,
                                       tci_resident_smem_bytes, tci_step_configure, tci_step_launch,
                                       tci_resident_launch};

}  // namespace TCI_KNS

// What follows is built once (in the throughput variant).
#ifndef TCI_SECONDARY

// ------------------------------------------------- RRLU tasks on a cluster
namespace TCI_KNS {
namespace {

constexpr size_t CL_SMEM = 224 * 1024;  // dynamic shared memory of a cluster's CTA at most

void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int ncta, size_t smem, cudaStream_t stream) {
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)ncta;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)ncta);
  cfg.blockDim = dim3(CL_NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}

// Shared memory of a task's CTA after the factorization's own: f's row and
// column states, and the index lists they are formed from.
__host__ __device__ inline size_t cluster_state_smem(int mb, int nb, int nl, int nr) {
  const size_t b = ((size_t)mb + nb) * 16 + (size_t)mb * nl + (size_t)nb * nr;
  return (b + 15) / 16 * 16;
}
__host__ __device__ inline size_t cluster_smem16(int m, int n, int mb, int nb) {
  return (cluster_smem(m, n, mb, nb, nb) + 15) / 16 * 16;
}

// One RRLU task (a given matrix, or f over its index lists) on the launched
// cluster, with post-processing NONE or FACTORS; the record as task_rrlu writes
// it.  A task's inputs may be in host memory: each CTA copies the lists of its
// own rows and columns in one pass.
__global__ void __launch_bounds__(CL_NT, 1) rrlu_cluster_task_kernel(const tci_task T, ClusterJob P) {
  extern __shared__ __align__(16) char smem[];
  __shared__ ClusterCtl ctl;
  __shared__ double s_params[RES_MAX_PARAMS];
  const long long t0 = clock64();
  const int tid = threadIdx.x, rank = (int)cg::this_cluster().block_rank();
  const int m = P.m, n = P.n, mb = P.mb, nb = P.nb, r0 = rank / P.pc * mb, c0 = rank % P.pc * nb;
  tci_result_head* head = (tci_result_head*)(uintptr_t)T.res;
  ClusterResult r;
  if (T.ain) {
    r = cluster_rrlu<false>(P, smem, ctl, [&](const auto& loop) {
      loop([&](int i, int j) { return __ldcs(T.ain + i + (size_t)j * m); }, At4{});
    });
  } else {
    const int nrb = max(0, min(m, r0 + mb) - r0), ncb = max(0, min(n, c0 + nb) - c0), nl = T.nl, nr = T.nr;
    double* rs0 = (double*)(smem + cluster_smem16(m, n, mb, nb));
    double *rs1 = rs0 + mb, *cs0 = rs1 + mb, *cs1 = cs0 + nb;
    uint8_t* li = (uint8_t*)(cs1 + nb);
    uint8_t* lj = li + (size_t)mb * nl;
    const uint8_t* gi = (const uint8_t*)(uintptr_t)T.rows + (size_t)r0 * nl;
    const uint8_t* gj = (const uint8_t*)(uintptr_t)T.cols + (size_t)c0 * nr;
    const double* prm = (const double*)(uintptr_t)T.params;
    for (int e = tid; e < nrb * nl; e += CL_NT) li[e] = gi[e];
    for (int e = tid; e < ncb * nr; e += CL_NT) lj[e] = gj[e];
    if (T.nparams <= RES_MAX_PARAMS) {
      for (int k = tid; k < T.nparams; k += CL_NT) s_params[k] = prm[k];
      prm = s_params;
    }
    __syncthreads();
    const bool tables = T.lut_full != 0;  // exact integer sums, kept in the same slots
    for (int e = tid; e < nrb + ncb; e += CL_NT) {
      const bool row = e < nrb;
      const int q = row ? e : e - nrb, len = row ? nl : nr, site0 = row ? 0 : nl;
      const uint8_t* v = row ? li + (size_t)q * nl : lj + (size_t)q * nr;
      double* d0 = (row ? rs0 : cs0) + q;
      double* d1 = (row ? rs1 : cs1) + q;
      if (tables) {
        long long a0 = 0, a1 = 0;
        for (int p = 0; p < len; ++p) tci_f_term_int(T.fid, prm, site0 + p, v[p], &a0, &a1);
        *(long long*)d0 = a0;
        *(long long*)d1 = a1;
      } else {
        const FSums a = f_sums(T.fid, prm, site0, len, v, -1, 0);
        *d0 = a.a0;
        *d1 = a.a1;
      }
    }
    __syncthreads();
    Filler F;
    F.fid = T.fid;
    F.nparams = T.nparams;
    F.prm = prm;
    F.lut0 = tables ? T.lut : nullptr;
    F.lut1 = tables && tci_f_tables(T.fid) > 1 ? T.lut + T.lutcap0 : nullptr;
    F.lo0 = T.lut_base0;
    F.lo1 = 0;
    r = cluster_rrlu<false>(P, smem, ctl, [&](const auto& loop) {
      if (tables)
        loop([&](int i, int j) { return F.tab(rs0, rs1, i - r0, cs0, cs1, j - c0); }, At4{});
      else
        loop([&](int i, int j) { return F.val(rs0, rs1, i - r0, cs0, cs1, j - c0); }, At1{});
    });
  }
  if (rank != 0) return;
  __syncthreads();  // the record's arrays before its head
  if (tid == 0) {
    head->status = r.nan ? TCI_ST_NAN : 0;
    head->npivot = r.K;
    head->error = r.err;
    head->maxabs = __longlong_as_double((long long)r.mx);
    head->maxabs_nan = r.mx > NAN_FLOOR ? 1 : 0;
    head->lut_used = !T.ain && T.lut_full;
    head->cycles = clock64() - t0;
    __threadfence_system();
    st_release_sys(&head->done, T.ticket + 1);
  }
}

}  // namespace

// CTAs of the largest cluster the device runs with a full CTA per SM, and how
// many such clusters at once (0: none).
int tci_rrlu_cluster_most(int* clusters) {
  static std::mutex mu;
  static int most[64], count[64];
  static bool ready[64];
  int dev = 0;
  if (clusters) *clusters = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lk(mu);
  if (!ready[dev]) {
    cudaError_t ce = cudaFuncSetAttribute(rrlu_cluster_task_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)CL_SMEM);
    if (ce == cudaSuccess)
      ce = cudaFuncSetAttribute(rrlu_cluster_task_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int c = CL_MAX; ce == cudaSuccess && c >= 8 && most[dev] == 0; c /= 2) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      cluster_config(cfg, at, c, CL_SMEM, nullptr);
      int fit = 0;
      if (cudaOccupancyMaxActiveClusters(&fit, rrlu_cluster_task_kernel, &cfg) == cudaSuccess && fit > 0) {
        most[dev] = c;
        count[dev] = fit;
      } else {
        (void)cudaGetLastError();
      }
    }
    ready[dev] = true;
  }
  if (clusters) *clusters = count[dev];
  return most[dev];
}

// CTAs for an RRLU task on clusters of at most `most`; 0 if it does not fit.
int tci_rrlu_cluster_ctas(const tci_task& t, int most) {
  if (t.m > 65535 || t.n > 65535 || t.m < 1 || t.n < 1) return 0;
  for (int c = cluster_first((int64_t)t.m * t.n, most); c <= most; c *= 2) {
    const ClusterGrid g = cluster_grid(t.m, t.n, c);
    const size_t state = t.ain ? 0 : cluster_state_smem(g.mb, g.nb, t.nl, t.nr);
    if (cluster_smem16(t.m, t.n, g.mb, g.nb) + state <= CL_SMEM) return c;
  }
  return 0;
}

// The task (absolute addresses, as in resident mode) on `ncta` CTAs; pivs: room
// for its largest rank in device memory.
cudaError_t tci_rrlu_cluster_launch(const tci_task& t, int ncta, double* pivs, cudaStream_t stream) {
  const ClusterGrid g = cluster_grid(t.m, t.n, ncta);
  ClusterJob P;
  P.m = t.m;
  P.n = t.n;
  P.kmax = std::min(t.maxrank, std::min(t.m, t.n));
  P.leftorth = t.leftorth;
  P.pr = g.pr;
  P.pc = g.pc;
  P.mb = g.mb;
  P.nb = g.nb;
  P.nres = g.nb;
  P.spill = nullptr;
  P.reltol = t.reltol;
  P.abstol = t.abstol;
  P.pivs = pivs;
  P.fact = t.post == TCI_POST_FACTORS ? t.core_out : nullptr;
  P.rowperm = P.fact ? (int*)(t.core_out + (size_t)t.m * t.n) : nullptr;
  P.colperm = P.fact ? P.rowperm + t.m : nullptr;
  char* arrays = (char*)(uintptr_t)t.res + sizeof(tci_result_head);
  const size_t kbytes = ((size_t)t.kcap * 4 + 7) / 8 * 8;
  P.rowk = (int*)arrays;
  P.colk = (int*)(arrays + kbytes);
  P.diag = (double*)(arrays + 2 * kbytes);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  const size_t state = t.ain ? 0 : cluster_state_smem(g.mb, g.nb, t.nl, t.nr);
  cluster_config(cfg, at, ncta, cluster_smem16(t.m, t.n, g.mb, g.nb) + state, stream);
  return cudaLaunchKernelEx(&cfg, rrlu_cluster_task_kernel, t, P);
}

}  // namespace TCI_KNS

// ===================================================================== rrLU
// without allocation (tci_rrlu_noalloc; no counterpart in the reference).
//
// Some callers cannot let the library allocate device memory: latency-critical
// serving loops where a cudaMalloc/cudaFree would stall the device, and hosts
// that own every device buffer through their own allocator (a Julia GPU array
// pool, a framework arena).  This entry point runs the same rank-revealing LU as the
// step kernel's RRLU task on caller-owned device buffers and keeps its working
// copy of the matrix, the factors and the result record in the fixed array
// below.  The array lives in every GPU that loads the library until the
// process exits.  Calls share it, so two calls that overlap on the GPU (on
// different streams, or interleaved with no ordering) race on it; calls issued
// on one stream are ordered and safe.  Nothing in it needs clearing between
// calls: every element a call reads is written earlier in the same call.

// error codes of include/tci_gb300.h (that header's function ids clash with
// tci_functions.h, so it is not included here)
#define TCI_ERR_ARG 1
#define TCI_ERR_NAN 3
#define TCI_ERR_CUDA 6

namespace tci {
void set_error(int code, const std::string& msg);
}

namespace TCI_KNS {
namespace {

constexpr int64_t NOALLOC_MAX_ELEMS = (int64_t)1 << 19;  // m * n
constexpr int64_t NOALLOC_MAX_DIM = 16384;               // m and n
constexpr int64_t NOALLOC_CLUSTER_ELEMS = 2500;          // from this size on a cluster
// working matrix | factors + full permutations | result record
constexpr int64_t NOALLOC_FACT_DOUBLES = NOALLOC_MAX_ELEMS + NOALLOC_MAX_DIM;
constexpr int64_t NOALLOC_RES_DOUBLES = 16 + 2 * NOALLOC_MAX_DIM;
constexpr int64_t NOALLOC_SCRATCH_DOUBLES = NOALLOC_MAX_ELEMS + NOALLOC_FACT_DOUBLES + NOALLOC_RES_DOUBLES;

static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_SCRATCH_DOUBLES];

// The caller's output buffers.
struct NoallocOut {
  int32_t *rowperm, *colperm, *npivot;
  double* error;
  int32_t* status;
};
template <bool SPILL>
__global__ void __launch_bounds__(CL_NT, 1) rrlu_noalloc_cluster_kernel(const double* __restrict__ ain, ClusterJob P,
                                                                        NoallocOut O) {
  extern __shared__ __align__(16) char smem[];
  __shared__ ClusterCtl ctl;
  const int m = P.m;
  const ClusterResult r =
      cluster_rrlu<SPILL>(P, smem, ctl, [&](const auto& loop) {
        loop([&](int i, int j) { return __ldcs(ain + i + (size_t)j * m); }, At4{});
      });
  if (cg::this_cluster().block_rank() == 0 && threadIdx.x == 0) {
    *O.npivot = r.K;
    *O.error = r.err;
    *O.status = r.nan ? TCI_ERR_NAN : 0;
  }
}

__global__ void __launch_bounds__(NT, TCI_CTAS_PER_SM) rrlu_noalloc_kernel(const tci_task T, char* resb) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Ctl ctl;
  task_rrlu(T, nullptr, resb, smem, ctl, 0);
}

// Copies the result record and the factors from the scratch array to the
// caller's buffers; *status = TCI_ERR_NAN when L or U holds a NaN (the
// reference's ErrorException "lu.L contains NaNs", matrixlu.jl:164-169), else 0.
__global__ void rrlu_noalloc_epilogue(const double* fact, const char* resb, int m, int n, int32_t* rowperm,
                                      int32_t* colperm, int32_t* npivot, double* error, int32_t* status,
                                      double* factors_out) {
  const tci_result_head* h = (const tci_result_head*)resb;
  const int32_t* perms = (const int32_t*)(fact + (size_t)m * n);
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  for (int i = tid; i < m; i += nth) rowperm[i] = perms[i];
  for (int j = tid; j < n; j += nth) colperm[j] = perms[m + j];
  if (factors_out)
    for (int64_t e = tid; e < (int64_t)m * n; e += nth) factors_out[e] = fact[e];
  if (tid == 0) {
    *npivot = h->npivot;
    *error = h->error;
    *status = (h->status & TCI_ST_NAN) ? TCI_ERR_NAN : 0;
  }
}

// CTAs of the cluster for an m x n matrix on a device whose clusters hold at
// most `most`; 0: one CTA of the step kernel.  A pivot costs some 5 thousand
// cycles on a cluster beside a large update, some 3 thousand on one CTA (swaps
// and argmax); full-rank factorizations cross at about 50 x 50: 32 x 32 takes
// 97 us on 8 CTAs and about 75 on one, 64 x 64 to rank 32 101 and 115, 104 x 104
// to rank 52 164 and 275, 160 x 160 to rank 80 274 and 1126 (from L2), 381 x 517
// to rank 140 1030 and 14100.
// *nres: the columns of a block that shared memory takes; past the fixed
// array's size nothing remains to spill to.
int noalloc_cluster(int64_t m, int64_t n, int most, int* nres) {
  if (m * n < NOALLOC_CLUSTER_ELEMS) return 0;
  for (int c = cluster_first(m * n, most); c <= most; c *= 2) {
    const ClusterGrid g = cluster_grid((int)m, (int)n, c);
    const size_t fixed = cluster_smem((int)m, (int)n, g.mb, g.nb, 0);
    if (fixed >= CL_SMEM) continue;
    *nres = (int)std::min<size_t>((size_t)g.nb, (CL_SMEM - fixed) / ((size_t)g.mb * 8));
    if (*nres == g.nb || (c == most && (int64_t)c * g.mb * (g.nb - *nres) <= NOALLOC_MAX_ELEMS)) return c;
  }
  return 0;
}

struct NoallocDevice {
  bool ready = false;
  int most = 0;  // CTAs of the largest cluster the device runs (0: none)
  double* scratch = nullptr;  // device address of g_noalloc_scratch
};

}  // namespace
}  // namespace TCI_KNS

// See include/tci_gb300.h.  The first call on a device resolves the device
// address of the scratch array (cudaGetSymbolAddress) and raises the kernel's
// shared-memory limit, with that device current; make that first call before
// any stream capture.  Later calls only launch one or two kernels on `stream_u`.  The
// address is cached per device for the life of the process, so a device reset
// (cudaDeviceReset) after the first call is not supported.
extern "C" int tci_rrlu_noalloc(const double* A_dev, int64_t m, int64_t n, int64_t maxrank, double reltol,
                                double abstol, int32_t leftorthogonal, int32_t* rowperm_dev, int32_t* colperm_dev,
                                int32_t* npivot_dev, double* error_dev, int32_t* status_dev, double* factors_dev,
                                uintptr_t stream_u) {
  using namespace TCI_KNS;
  static std::mutex mu;
  static NoallocDevice devs[64];
  if (m < 1 || n < 1 || m > NOALLOC_MAX_DIM || n > NOALLOC_MAX_DIM || m * n > NOALLOC_MAX_ELEMS) {
    tci::set_error(TCI_ERR_ARG, "tci_rrlu_noalloc: matrix must satisfy 1 <= m, n <= " +
                                            std::to_string(NOALLOC_MAX_DIM) + " and m*n <= " +
                                            std::to_string(NOALLOC_MAX_ELEMS) + " (got " + std::to_string(m) +
                                            " x " + std::to_string(n) + ")");
    return TCI_ERR_ARG;
  }
  if (!A_dev || !rowperm_dev || !colperm_dev || !npivot_dev || !error_dev || !status_dev) {
    tci::set_error(TCI_ERR_ARG, "tci_rrlu_noalloc: null input or output pointer");
    return TCI_ERR_ARG;
  }
  // A launch error left pending by earlier work on this thread is reported,
  // not cleared: the caller's own error check still sees it.
  cudaError_t ce = cudaPeekAtLastError();
  if (ce != cudaSuccess) {
    tci::set_error(TCI_ERR_CUDA, std::string("tci_rrlu_noalloc: a CUDA error was pending before the call: ") +
                                     cudaGetErrorString(ce));
    return TCI_ERR_CUDA;
  }
  int dev = 0;
  ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess || dev < 0 || dev >= 64) {
    tci::set_error(TCI_ERR_CUDA,std::string("tci_rrlu_noalloc: ") + cudaGetErrorString(ce));
    return TCI_ERR_CUDA;
  }
  NoallocDevice& D = devs[dev];
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!D.ready) {
      void* p = nullptr;
      ce = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (ce == cudaSuccess)
        ce = cudaFuncSetAttribute(rrlu_noalloc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)tci_step_smem_bytes());
      for (auto k : {rrlu_noalloc_cluster_kernel<false>, rrlu_noalloc_cluster_kernel<true>}) {
        if (ce == cudaSuccess)
          ce = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM);
        if (ce == cudaSuccess) ce = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      }
      for (int c = CL_MAX; ce == cudaSuccess && c >= 8 && D.most == 0; c /= 2) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        cluster_config(cfg, at, c, CL_SMEM, nullptr);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, rrlu_noalloc_cluster_kernel<true>, &cfg) == cudaSuccess && fit > 0)
          D.most = c;
        else
          (void)cudaGetLastError();
      }
      if (ce != cudaSuccess) {
        tci::set_error(TCI_ERR_CUDA,std::string("tci_rrlu_noalloc set-up: ") + cudaGetErrorString(ce));
        return TCI_ERR_CUDA;
      }
      D.scratch = (double*)p;
      D.ready = true;
    }
  }
  double* work = D.scratch;
  double* fact = D.scratch + NOALLOC_MAX_ELEMS;
  char* resb = (char*)(D.scratch + NOALLOC_MAX_ELEMS + NOALLOC_FACT_DOUBLES);
  tci_task T;
  memset(&T, 0, sizeof(T));
  T.kind = TCI_TASK_RRLU;
  T.m = (int32_t)m;
  T.n = (int32_t)n;
  int64_t kmax = maxrank <= 0 ? (m < n ? m : n) : maxrank;
  if (kmax > m) kmax = m;
  if (kmax > n) kmax = n;
  T.maxrank = (int32_t)kmax;
  T.kcap = (int32_t)kmax;
  T.reltol = reltol;
  T.abstol = abstol;
  T.leftorth = leftorthogonal ? 1 : 0;
  T.post = TCI_POST_FACTORS;
  T.ain = A_dev;
  T.core_out = fact;
  T.res = 0;
  cudaStream_t stream = (cudaStream_t)stream_u;
  int nres = 0;
  if (const int c = noalloc_cluster(m, n, D.most, &nres)) {
    const ClusterGrid g = cluster_grid((int)m, (int)n, c);
    ClusterJob P;
    P.m = (int)m;
    P.n = (int)n;
    P.kmax = (int)kmax;
    P.leftorth = T.leftorth;
    P.pr = g.pr;
    P.pc = g.pc;
    P.mb = g.mb;
    P.nb = g.nb;
    P.reltol = reltol;
    P.abstol = abstol;
    P.nres = nres;
    P.spill = work;
    P.pivs = fact;
    P.fact = factors_dev;
    P.rowperm = rowperm_dev;
    P.colperm = colperm_dev;
    P.rowk = P.colk = nullptr;
    P.diag = nullptr;
    const NoallocOut O{rowperm_dev, colperm_dev, npivot_dev, error_dev, status_dev};
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, c, cluster_smem((int)m, (int)n, g.mb, g.nb, nres), stream);
    ce = cudaLaunchKernelEx(&cfg, nres < g.nb ? rrlu_noalloc_cluster_kernel<true> : rrlu_noalloc_cluster_kernel<false>,
                            A_dev, P, O);
    if (ce == cudaSuccess) ce = cudaGetLastError();
    if (ce != cudaSuccess) {
      tci::set_error(TCI_ERR_CUDA, std::string("tci_rrlu_noalloc: ") + cudaGetErrorString(ce));
      return TCI_ERR_CUDA;
    }
    return 0;
  }
  const size_t smem = tci_step_smem_bytes();
  auto a16 = [](size_t x) { return (x + 15) / 16 * 16; };
  const size_t perms = a16((size_t)m * 4) + a16((size_t)n * 4);
  T.smem_mode = a16((size_t)m * n * 8) + perms <= smem ? 1 : 0;
  T.work = T.smem_mode ? nullptr : work;
  rrlu_noalloc_kernel<<<1, NT, smem, stream>>>(T, resb);
  rrlu_noalloc_epilogue<<<64, 256, 0, stream>>>(fact, resb, (int)m, (int)n, rowperm_dev, colperm_dev, npivot_dev,
                                                error_dev, status_dev, factors_dev);
  ce = cudaGetLastError();
  if (ce != cudaSuccess) {
    tci::set_error(TCI_ERR_CUDA,std::string("tci_rrlu_noalloc: ") + cudaGetErrorString(ce));
    return TCI_ERR_CUDA;
  }
  return 0;
}
#endif  // TCI_SECONDARY
