// Tensor-train contraction kernels (contraction.jl): the site contractions of
// contract_naive (:333-349) and contract_zipup (:442-486), the left/right
// factors of an rrLU (matrixlu.jl:374-392) and the small matrix products of
// compress! (tensortrain.jl:149-183).
//
// Every output element is one sum over the contracted index in a fixed
// ascending order with separate IEEE multiply and add (the file is compiled
// without FMA contraction), so the results are reproducible and equal, bit for
// bit, to the CPU oracle's loops.  The reference contracts through BLAS, whose
// summation order is unspecified, so against the reference itself these are
// tolerance-level results (as its own tests compare them).
//
// Layouts are column-major.  A 4-leg core is (link, s_in, s_out, link').
#include <cuda_runtime.h>
#include <stdint.h>

#include "ieee_int.h"
#include "tc_gemm.h"

namespace {

constexpr int CT = 256;

__device__ __forceinline__ int64_t gtid() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int64_t gstride() { return (int64_t)gridDim.x * blockDim.x; }

// _contractsitetensors (contraction.jl:333-349):
// out[(ia, ib), s1, s3, (ja, jb)] = sum_k a[ia, s1, k, ja] * b[ib, k, s3, jb],
// (ia, ib) and (ja, jb) fused with the a index fastest.
__global__ void naive_site_kernel(const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out,
                                  int ra, int s1, int s2, int ra2, int rb, int s3, int rb2) {
  const int64_t total = (int64_t)ra * rb * s1 * s3 * ra2 * rb2;
  for (int64_t e = gtid(); e < total; e += gstride()) {
    int64_t t = e;
    const int ia = (int)(t % ra); t /= ra;
    const int ib = (int)(t % rb); t /= rb;
    const int i1 = (int)(t % s1); t /= s1;
    const int i3 = (int)(t % s3); t /= s3;
    const int ja = (int)(t % ra2); t /= ra2;
    const int jb = (int)t;
    double acc = 0.0;
    for (int k = 0; k < s2; ++k) {
      const double x = a[ia + (int64_t)ra * (i1 + (int64_t)s1 * (k + (int64_t)s2 * ja))];
      const double y = b[ib + (int64_t)rb * (k + (int64_t)s2 * (i3 + (int64_t)s3 * jb))];
      acc = __dadd_rn(acc, __dmul_rn(x, y));
    }
    out[e] = acc;
  }
}

// C[c_row(i) + c_col(j)] = sum_k A[a_row(i) + a_k(k)] * B[b_k(k) + b_col(j)],
// k ascending, the legs of a tensor addressed through index maps.
//
// FP64-bound: one addition per multiply-add on the FP64 pipe, the product on the
// integer pipes (ieee_int.h).  A CTA computes a BM x BN tile from 16-deep slices
// in shared memory, each thread 4 x 4 outputs (4 x 2 in the narrowest tile): a value is taken apart once per
// four products, sixteen independent sums hide the latency, and the next slice
// is loaded while one is used.  How the products are taken is decided per slice
// from the values loaded (rank-revealing factors hold exact zeros and ones).
// 19200 x 60 x 240 (the larger product of a zip-up at bonds 24, 60 and 200):
// 0.60 ms against 0.53 for its additions on the FP64 pipe; 1.06 ms with one
// thread per output and FP64 products.
constexpr int GK = 16;  // depth of a slice
enum { VAL_DENSE = 0, VAL_ZEROS = 1, VAL_UNSAFE = 2 };
__device__ __forceinline__ int val_class(double v) {
  return int_safe(v) ? (int_dense(v) ? VAL_DENSE : VAL_ZEROS) : VAL_UNSAFE;
}
__device__ __forceinline__ int64_t map_at(const tci_map3& m, int64_t i) {
  if (i < m.d0) return i * m.s0;
  const int64_t a = i % m.d0, q = i / m.d0;
  return a * m.s0 + (q % m.d1) * m.s1 + (q / m.d1) * m.s2;
}

template <int MODE, int BM, int BN, int CB>
__device__ __forceinline__ void gemm_slice(const double (*As)[BM], const double (*Bs)[BN + 2], int kc, int ty, int tx,
                                           double (&acc)[4][CB]) {
  constexpr int TX = BN / CB;
#pragma unroll 1
  for (int k = 0; k < kc; ++k) {
    double x[4], y[CB];
#pragma unroll
    for (int a = 0; a < 4; ++a) x[a] = As[k][4 * ty + a];
#pragma unroll
    for (int b = 0; b < CB; ++b) y[b] = Bs[k][tx + TX * b];
    double q[4][CB];
    if (MODE == VAL_DENSE) {
      DenseFactor xf[4], yf[CB];
#pragma unroll
      for (int a = 0; a < 4; ++a) xf[a] = dense_split(x[a]);
#pragma unroll
      for (int b = 0; b < CB; ++b) yf[b] = dense_split(y[b]);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < CB; ++b) q[a][b] = int_mul_dense(xf[a], yf[b]);
    } else if (MODE == VAL_ZEROS) {
      IntFactor xf[4], yf[CB];
#pragma unroll
      for (int a = 0; a < 4; ++a) xf[a] = int_split(x[a]);
#pragma unroll
      for (int b = 0; b < CB; ++b) yf[b] = int_split(y[b]);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < CB; ++b) q[a][b] = int_mul(xf[a], yf[b]);
    } else {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < CB; ++b) q[a][b] = __dmul_rn(x[a], y[b]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < CB; ++b) acc[a][b] = __dadd_rn(acc[a][b], q[a][b]);
  }
}

template <int BN, int CB>
__global__ void __launch_bounds__(CT, 2)
    gemm_map_kernel(int64_t M, int64_t N, int64_t K, const double* __restrict__ A, tci_map3 a_row, tci_map3 a_k,
                    const double* __restrict__ B, tci_map3 b_k, tci_map3 b_col, double* __restrict__ C, tci_map3 c_row,
                    tci_map3 c_col) {
  constexpr int TX = BN / CB, TY = CT / TX, BM = 4 * TY;
  constexpr int LA = BM * GK / CT, LB = BN * GK / CT;  // values each thread loads of a slice
  // Past the edge: a dense value, so that it does not change how products are taken.
  const double pad = __hiloint2double(0x3ff00000, 1);
  __shared__ double As[2][GK][BM];
  __shared__ double Bs[2][GK][BN + 2];
  __shared__ int cls[3];  // class of the slices, in rotation: one in use, one being stored, one cleared
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int64_t tiles_n = (N + BN - 1) / BN, tiles = (M + BM - 1) / BM * tiles_n;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t m0 = tile / tiles_n * BM, n0 = tile % tiles_n * BN;
    // loads: A along its rows, B along k
    const int ar = tid % BM, ak = tid / BM, bk = tid % GK, bc = tid / GK;
    const bool a_in = m0 + ar < M;
    const double* ap = A + (a_in ? map_at(a_row, m0 + ar) : 0);
    const double* bp[LB];
    bool b_in[LB];
#pragma unroll
    for (int q = 0; q < LB; ++q) {
      const int64_t j = n0 + bc + q * (CT / GK);
      b_in[q] = j < N;
      bp[q] = B + (b_in[q] ? map_at(b_col, j) : 0);
    }
    double av[LA], bv[LB];
    auto load = [&](int64_t k0) {
#pragma unroll
      for (int q = 0; q < LA; ++q) {
        const int64_t k = k0 + ak + q * (GK / LA);
        av[q] = a_in && k < K ? ap[map_at(a_k, k)] : pad;
      }
      const int64_t ob = k0 + bk < K ? map_at(b_k, k0 + bk) : 0;
#pragma unroll
      for (int q = 0; q < LB; ++q) bv[q] = b_in[q] && k0 + bk < K ? bp[q][ob] : pad;
    };
    auto store = [&](int p, int slot) {
      int c = VAL_DENSE;
#pragma unroll
      for (int q = 0; q < LA; ++q) {
        As[p][ak + q * (GK / LA)][ar] = av[q];
        c = max(c, val_class(av[q]));
      }
#pragma unroll
      for (int q = 0; q < LB; ++q) {
        Bs[p][bk][bc + q * (CT / GK)] = bv[q];
        c = max(c, val_class(bv[q]));
      }
      if (c) atomicMax(&cls[slot], c);
    };
    if (tid < 3) cls[tid] = VAL_DENSE;
    double acc[4][CB];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < CB; ++b) acc[a][b] = 0.0;
    load(0);
    __syncthreads();
    store(0, 0);
    __syncthreads();
    int p = 0, slot = 0;
    for (int64_t k0 = 0; k0 < K; k0 += GK) {
      const bool more = k0 + GK < K;
      if (more) load(k0 + GK);
      const int kc = (int)min((int64_t)GK, K - k0), mode = cls[slot], next = slot == 2 ? 0 : slot + 1;
      if (tid == 0) cls[3 - slot - next] = VAL_DENSE;
      if (mode == VAL_DENSE) gemm_slice<VAL_DENSE, BM, BN, CB>(As[p], Bs[p], kc, ty, tx, acc);
      else if (mode == VAL_ZEROS) gemm_slice<VAL_ZEROS, BM, BN, CB>(As[p], Bs[p], kc, ty, tx, acc);
      else gemm_slice<VAL_UNSAFE, BM, BN, CB>(As[p], Bs[p], kc, ty, tx, acc);
      p ^= 1;
      slot = next;
      if (more) store(p, slot);
      __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int64_t i = m0 + 4 * ty + a;
      if (i >= M) continue;
      const int64_t o = map_at(c_row, i);
#pragma unroll
      for (int b = 0; b < CB; ++b) {
        const int64_t j = n0 + tx + TX * b;
        if (j < N) C[o + map_at(c_col, j)] = acc[a][b];
      }
    }
    __syncthreads();
  }
}

// The same with one thread per output, FP64 products: it spreads evenly over the SMs
// where tiles do not.  The offsets along k are formed once per CTA; eight loads in
// flight.
constexpr int EACH_K = 256;
__global__ void __launch_bounds__(128)
    gemm_each_kernel(int64_t M, int64_t N, int64_t K, const double* __restrict__ A, tci_map3 a_row, tci_map3 a_k,
                     const double* __restrict__ B, tci_map3 b_k, tci_map3 b_col, double* __restrict__ C, tci_map3 c_row,
                     tci_map3 c_col) {
  __shared__ int64_t ka[EACH_K], kb[EACH_K];
  const int64_t e = gtid();
  const bool on = e < M * N;
  const int64_t j = on ? e / M : 0, i = on ? e - j * M : 0;
  const double* a = A + map_at(a_row, i);
  const double* b = B + map_at(b_col, j);
  double acc = 0.0;
  for (int64_t k0 = 0; k0 < K; k0 += EACH_K) {
    const int kc = (int)(K - k0 < EACH_K ? K - k0 : EACH_K);
    __syncthreads();
    for (int k = threadIdx.x; k < kc; k += 128) {
      ka[k] = map_at(a_k, k0 + k);
      kb[k] = map_at(b_k, k0 + k);
    }
    __syncthreads();
    int k = 0;
    for (; k + 4 <= kc; k += 4) {
      double x[4], y[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        x[q] = __ldg(a + ka[k + q]);
        y[q] = __ldg(b + kb[k + q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) acc = __dadd_rn(acc, __dmul_rn(x[q], y[q]));
    }
    for (; k < kc; ++k) acc = __dadd_rn(acc, __dmul_rn(__ldg(a + ka[k]), __ldg(b + kb[k])));
  }
  if (on) C[map_at(c_row, i) + map_at(c_col, j)] = acc;
}

// Tiles or one thread per output.  The tile's width goes by the number of columns: a
// wider one than needed computes columns past the edge.  Up to one tile per SM takes
// the time of one, from there on each pair per SM the time of two; against that, one
// thread per output costs 1.75 times as much an output (two FP64 instructions a term
// instead of one) and has no edges.  A product of host matrices, microseconds, one
// thread per output and tiles: 60 x 60 x 60 52 and 125, 512 x 513 x 2000 2277 and 2722,
// 20000 x 40 x 300 1406 and 1919, 4864 x 65 x 200 402 and 405, 16384 x 16 x 1024 1930
// and 1568, 4864 x 128 x 200 678 and 459, 900 x 900 x 900 3065 and 2453.
cudaError_t gemm_map(int64_t M, int64_t N, int64_t K, const double* A, tci_map3 a_row, tci_map3 a_k, const double* B,
                     tci_map3 b_k, tci_map3 b_col, double* C, tci_map3 c_row, tci_map3 c_col, cudaStream_t st) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int64_t bn = N <= 16 ? 16 : N <= 32 ? 32 : 64, bm = bn == 64 ? 64 : 128;
  const int64_t tiles = (M + bm - 1) / bm * ((N + bn - 1) / bn);
  const int64_t turns = tiles <= sms ? 1 : 2 * ((tiles + 2 * sms - 1) / (2 * sms));
  const unsigned grid = (unsigned)(tiles < 65535 * 16 ? tiles : 65535 * 16);
  if ((double)(turns * bm * bn) * sms > 1.75 * (double)M * (double)N)
    gemm_each_kernel<<<(unsigned)((M * N + 127) / 128), 128, 0, st>>>(M, N, K, A, a_row, a_k, B, b_k, b_col, C, c_row,
                                                                      c_col);
  else if (bn == 16)
    gemm_map_kernel<16, 2><<<grid, CT, 0, st>>>(M, N, K, A, a_row, a_k, B, b_k, b_col, C, c_row, c_col);
  else if (bn == 32)
    gemm_map_kernel<32, 4><<<grid, CT, 0, st>>>(M, N, K, A, a_row, a_k, B, b_k, b_col, C, c_row, c_col);
  else
    gemm_map_kernel<64, 4><<<grid, CT, 0, st>>>(M, N, K, A, a_row, a_k, B, b_k, b_col, C, c_row, c_col);
  return cudaGetLastError();
}

// left(lu) and right(lu) (matrixlu.jl:374-392) from the factored m x n matrix F
// (L below the diagonal, U on and above; unit diagonal on L when leftorth,
// else on U) and the full 0-based permutations:
// left[rowperm[i], k] = L[i, k] (m x K), right[k, colperm[j]] = U[k, j] (K x n).
__global__ void lu_left_right_kernel(const double* __restrict__ F, const int32_t* __restrict__ rowperm,
                                     const int32_t* __restrict__ colperm, int m, int n, int K, int leftorth,
                                     double* __restrict__ left, double* __restrict__ right) {
  const int64_t nl = left ? (int64_t)m * K : 0, nr = right ? (int64_t)K * n : 0;
  for (int64_t e = gtid(); e < nl + nr; e += gstride()) {
    if (e < nl) {
      const int i = (int)(e % m), k = (int)(e / m);
      const double v = i < k ? 0.0 : (i == k && leftorth ? 1.0 : F[i + (int64_t)m * k]);
      left[rowperm[i] + (int64_t)m * k] = v;
    } else {
      const int64_t f = e - nl;
      const int k = (int)(f % K), j = (int)(f / K);
      const double v = k > j ? 0.0 : (k == j && !leftorth ? 1.0 : F[k + (int64_t)m * j]);
      right[k + (int64_t)K * colperm[j]] = v;
    }
  }
}

// L = tril(A[:, 1:K]) (m x K) and U = triu(A[1:K, :]) (K x n) with the unit
// diagonal (matrixlu.jl:162-174) from the factored m x n matrix F.
__global__ void lu_factors_kernel(const double* __restrict__ F, int m, int n, int K, int leftorth,
                                  double* __restrict__ L, double* __restrict__ U) {
  const int64_t nl = (int64_t)m * K, nu = (int64_t)K * n;
  for (int64_t e = gtid(); e < nl + nu; e += gstride()) {
    if (e < nl) {
      const int i = (int)(e % m), j = (int)(e / m);
      L[e] = i < j ? 0.0 : (i == j && leftorth ? 1.0 : F[e]);
    } else {
      const int64_t f = e - nl;
      const int i = (int)(f % K), j = (int)(f / K);
      U[f] = i > j ? 0.0 : (i == j && !leftorth ? 1.0 : F[i + (int64_t)m * j]);
    }
  }
}

// MatrixLUCI left/right (matrixluci.jl:40-84) from the factored matrix F as
// above: one thread per row of left (m threads), then one per column of right
// (n threads), each in the order of the oracle's loops (separate multiply,
// add/subtract and divide).
//   leftorth:  left = colstimespivotinv (rows K.. of L against LowerTriangular(L11),
//              rows scattered by rowperm), right = rowmatrix = L[1:K, :] * right(lu)
//   !leftorth: left = colmatrix = left(lu) * U[:, 1:K], right = pivotinvtimesrows
//              (UpperTriangular(U11) \ U12, columns scattered by colperm)
__device__ __forceinline__ double f_L(const double* F, int m, int i, int p, int leftorth) {
  return i < p ? 0.0 : (i == p && leftorth ? 1.0 : F[i + (int64_t)m * p]);
}
__device__ __forceinline__ double f_U(const double* F, int m, int p, int j, int leftorth) {
  return p > j ? 0.0 : (p == j && !leftorth ? 1.0 : F[p + (int64_t)m * j]);
}

__global__ void luci_left_right_kernel(const double* __restrict__ F, const int32_t* __restrict__ rowperm,
                                       const int32_t* __restrict__ colperm, int m, int n, int K, int leftorth,
                                       double* __restrict__ left, double* __restrict__ right) {
  for (int64_t e = gtid(); e < (int64_t)m + n; e += gstride()) {
    if (e < m) {
      const int i = (int)e;
      double* out = left + rowperm[i];  // out[q * m] = entry (rowperm[i], q)
      if (leftorth) {
        if (i < K) {
          for (int q = 0; q < K; ++q) out[(int64_t)m * q] = i == q ? 1.0 : 0.0;
        } else {
          for (int q = K - 1; q >= 0; --q) {
            double s = f_L(F, m, i, q, 1);
            for (int p = q + 1; p < K; ++p) s = __dsub_rn(s, __dmul_rn(out[(int64_t)m * p], f_L(F, m, p, q, 1)));
            out[(int64_t)m * q] = __ddiv_rn(s, f_L(F, m, q, q, 1));
          }
        }
      } else {
        for (int q = 0; q < K; ++q) {
          double s = 0.0;
          for (int p = 0; p <= q; ++p) s = __dadd_rn(s, __dmul_rn(f_L(F, m, i, p, 0), f_U(F, m, p, q, 0)));
          out[(int64_t)m * q] = s;
        }
      }
    } else {
      const int j = (int)(e - m);
      double* out = right + (int64_t)K * colperm[j];  // out[q] = entry (q, colperm[j])
      if (leftorth) {
        for (int q = 0; q < K; ++q) {
          double s = 0.0;
          for (int p = 0; p <= q; ++p) s = __dadd_rn(s, __dmul_rn(f_L(F, m, q, p, 1), f_U(F, m, p, j, 1)));
          out[q] = s;
        }
      } else if (j < K) {
        for (int q = 0; q < K; ++q) out[q] = j == q ? 1.0 : 0.0;
      } else {
        for (int q = K - 1; q >= 0; --q) {
          double s = f_U(F, m, q, j, 0);
          for (int p = q + 1; p < K; ++p) s = __dsub_rn(s, __dmul_rn(f_U(F, m, q, p, 0), out[p]));
          out[q] = __ddiv_rn(s, f_U(F, m, q, q, 0));
        }
      }
    }
  }
}

// ---- environments of the Contraction evaluator (contraction.jl:103-176) ----
// One level of new environments: entry e extends parent[e] (ra x rb) by site
// value (ii[e], jj[e]) of A (ra x s x S x ra2) and B (rb x S x s2 x rb2).
//   left:  tmp[b, t, a'] = sum_a P[a, b] A[a, i, t, a']
//          E[a', b']     = sum_(b, t), b fastest, tmp[b, t, a'] B[b, t, j, b']
//   right: tmp[b2, t, a] = sum_a2 P[a2, b2] A[a, i, t, a2]     (P is ra2 x rb2)
//          E[a, b]       = sum_(b2, t), b2 fastest, tmp[b2, t, a] B[b, t, j, b2]
// (_extend_cache, contraction.jl:103-109, with the permuted cores of :165-169).
struct EnvLevel {
  const double* A;
  const double* B;
  int ra, s, S, ra2, rb, s2, rb2;
  int right;
  int n;  // entries
  const double* const* parent;
  double* const* out;
  double* const* tmp;
  const int32_t* ii;
  const int32_t* jj;
};

__global__ void env_tmp_kernel(EnvLevel v) {
  // left: per entry rb * S * ra2 values; right: rb2 * S * ra values
  const int64_t per = v.right ? (int64_t)v.rb2 * v.S * v.ra : (int64_t)v.rb * v.S * v.ra2;
  for (int64_t g = gtid(); g < per * v.n; g += gstride()) {
    const int e = (int)(g / per);
    const int64_t x = g % per;
    const double* P = v.parent[e];
    const int i = v.ii[e];
    double acc = 0.0;
    if (!v.right) {
      const int b = (int)(x % v.rb), t = (int)((x / v.rb) % v.S), a2 = (int)(x / ((int64_t)v.rb * v.S));
      const double* Ac = v.A + (int64_t)v.ra * (i + (int64_t)v.s * (t + (int64_t)v.S * a2));
      for (int a = 0; a < v.ra; ++a) acc = __dadd_rn(acc, __dmul_rn(P[a + (int64_t)v.ra * b], Ac[a]));
    } else {
      const int b2 = (int)(x % v.rb2), t = (int)((x / v.rb2) % v.S), a = (int)(x / ((int64_t)v.rb2 * v.S));
      for (int a2 = 0; a2 < v.ra2; ++a2)
        acc = __dadd_rn(acc, __dmul_rn(P[a2 + (int64_t)v.ra2 * b2],
                                       v.A[a + (int64_t)v.ra * (i + (int64_t)v.s * (t + (int64_t)v.S * a2))]));
    }
    v.tmp[e][x] = acc;
  }
}

__global__ void env_out_kernel(EnvLevel v) {
  const int64_t per = v.right ? (int64_t)v.ra * v.rb : (int64_t)v.ra2 * v.rb2;
  for (int64_t g = gtid(); g < per * v.n; g += gstride()) {
    const int e = (int)(g / per);
    const int64_t x = g % per;
    const double* T = v.tmp[e];
    const int j = v.jj[e];
    double acc = 0.0;
    if (!v.right) {
      const int a2 = (int)(x % v.ra2), b2 = (int)(x / v.ra2);
      for (int t = 0; t < v.S; ++t) {
        const double* Tc = T + (int64_t)v.rb * (t + (int64_t)v.S * a2);
        const double* Bc = v.B + (int64_t)v.rb * (t + (int64_t)v.S * (j + (int64_t)v.s2 * b2));
        for (int b = 0; b < v.rb; ++b) acc = __dadd_rn(acc, __dmul_rn(Tc[b], Bc[b]));
      }
    } else {
      const int a = (int)(x % v.ra), b = (int)(x / v.ra);
      for (int t = 0; t < v.S; ++t) {
        const double* Tc = T + (int64_t)v.rb2 * (t + (int64_t)v.S * a);
        for (int b2 = 0; b2 < v.rb2; ++b2)
          acc = __dadd_rn(acc, __dmul_rn(Tc[b2], v.B[b + (int64_t)v.rb * (t + (int64_t)v.S * (j + (int64_t)v.s2 * b2))]));
      }
    }
    v.out[e][x] = acc;
  }
}

// out[k] = sum_t L[k][t] R[k][t], t = 0 .. len[k]-1 in order (the (link_a,
// link_b) contraction of batchevaluate, contraction.jl:325-329, a fastest).
__global__ void env_dot_kernel(const double* const* L, const double* const* R, const int32_t* len, int n,
                               double* out) {
  for (int64_t k = gtid(); k < n; k += gstride()) {
    const double* l = L[k];
    const double* r = R[k];
    double acc = 0.0;
    for (int t = 0; t < len[k]; ++t) acc = __dadd_rn(acc, __dmul_rn(l[t], r[t]));
    out[k] = acc;
  }
}

int grid_for(int64_t total) {
  int64_t g = (total + CT - 1) / CT;
  if (g < 1) g = 1;
  if (g > 152 * 32) g = 152 * 32;
  return (int)g;
}

}  // namespace

cudaError_t tci_naive_site_launch(const double* a, const double* b, double* out, int ra, int s1, int s2, int ra2,
                                  int rb, int s3, int rb2, cudaStream_t st) {
  const int64_t total = (int64_t)ra * rb * s1 * s3 * ra2 * rb2;
  naive_site_kernel<<<grid_for(total), CT, 0, st>>>(a, b, out, ra, s1, s2, ra2, rb, s3, rb2);
  return cudaGetLastError();
}

// Zipup, first product (contraction.jl:461-463): RA[ab, bn, s, s', an'] =
// sum_an R[ab, an, bn] * A[an, s, s', an'].
cudaError_t tci_zip_ra_launch(const double* R, const double* A, double* RA, int nab, int nan_, int nbn, int s,
                              int sp, int nan2, cudaStream_t st) {
  const int64_t rows = (int64_t)nab * nbn;
  return gemm_map(rows, (int64_t)s * sp * nan2, nan_, R, tci_map_2(nab, 1, (int64_t)nab * nan_), tci_map_stride(nab), A,
                  tci_map_stride(1), tci_map_stride(nan_), RA, tci_map_stride(1), tci_map_stride(rows), st);
}

// Zipup, second product (contraction.jl:464-469): C[ab, s, s'', an', bn'] =
// sum_{s'} sum_{bn} RA[ab, bn, s, s', an'] * B[bn, s', s'', bn'], the fused
// contracted index (bn, s') ascending with bn fastest; rows (ab, s, an'),
// columns (s'', bn').
cudaError_t tci_zip_c_launch(const double* RA, const double* B, double* C, int nab, int nbn, int s, int sp, int nan2,
                             int spp, int nbn2, cudaStream_t st) {
  const int64_t ab = nab, abn = ab * nbn, abs_ = ab * s, k = (int64_t)nbn * sp;
  return gemm_map(abs_ * nan2, (int64_t)spp * nbn2, k, RA, tci_map_3(nab, s, 1, abn, abn * s * sp),
                  tci_map_2(nbn, nab, abn * s), B, tci_map_stride(1), tci_map_stride(k), C,
                  tci_map_3(nab, s, 1, ab, abs_ * spp), tci_map_2(spp, abs_, abs_ * spp * nan2), st);
}

cudaError_t tci_lu_left_right_launch(const double* F, const int32_t* rowperm, const int32_t* colperm, int m, int n,
                                     int K, int leftorth, double* left, double* right, cudaStream_t st) {
  const int64_t total = (left ? (int64_t)m * K : 0) + (right ? (int64_t)K * n : 0);
  if (total == 0) return cudaSuccess;
  lu_left_right_kernel<<<grid_for(total), CT, 0, st>>>(F, rowperm, colperm, m, n, K, leftorth, left, right);
  return cudaGetLastError();
}

cudaError_t tci_lu_factors_launch(const double* F, int m, int n, int K, int leftorth, double* L, double* U,
                                  cudaStream_t st) {
  const int64_t total = ((int64_t)m + n) * K;
  if (total == 0) return cudaSuccess;
  lu_factors_kernel<<<grid_for(total), CT, 0, st>>>(F, m, n, K, leftorth, L, U);
  return cudaGetLastError();
}

cudaError_t tci_luci_left_right_launch(const double* F, const int32_t* rowperm, const int32_t* colperm, int m,
                                       int n, int K, int leftorth, double* left, double* right, cudaStream_t st) {
  const int64_t total = (int64_t)m + n;
  if (K == 0 || total == 0) return cudaSuccess;
  luci_left_right_kernel<<<grid_for(total), CT, 0, st>>>(F, rowperm, colperm, m, n, K, leftorth, left, right);
  return cudaGetLastError();
}

// C (M x N) = A (M x K) * B (K x N), column-major with leading dimensions.
cudaError_t tci_gemm_launch(const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
                            int M, int N, int K, cudaStream_t st) {
  return gemm_map(M, N, K, A, tci_map_stride(1), tci_map_stride(lda), B, tci_map_stride(1), tci_map_stride(ldb), C,
                  tci_map_stride(1), tci_map_stride(ldc), st);
}

cudaError_t tci_env_level_launch(const double* A, const double* B, int ra, int s, int S, int ra2, int rb, int s2,
                                 int rb2, int right, int n, const double* const* parent, double* const* out,
                                 double* const* tmp, const int32_t* ii, const int32_t* jj, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  EnvLevel v{A, B, ra, s, S, ra2, rb, s2, rb2, right, n, parent, out, tmp, ii, jj};
  const int64_t t1 = (right ? (int64_t)rb2 * S * ra : (int64_t)rb * S * ra2) * n;
  const int64_t t2 = (right ? (int64_t)ra * rb : (int64_t)ra2 * rb2) * n;
  env_tmp_kernel<<<grid_for(t1), CT, 0, st>>>(v);
  env_out_kernel<<<grid_for(t2), CT, 0, st>>>(v);
  return cudaGetLastError();
}

cudaError_t tci_env_dot_launch(const double* const* L, const double* const* R, const int32_t* len, int n, double* out,
                               cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  env_dot_kernel<<<grid_for(n), CT, 0, st>>>(L, R, len, n, out);
  return cudaGetLastError();
}
