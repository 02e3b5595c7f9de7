// evaluate(tt, indexset) (abstracttensortrain.jl:124-132) at many points in FP64:
// v <- v * T_s[:, i_s, :] site by site, v[q] = sum_t v[t] T_s[t, i, q] summed in
// order of t with separate multiply and add, as the oracle's loop.
//
// FP64-bound once every SM has work: one addition per multiply-add on the FP64
// pipe, the product on the integer pipes (ieee_int.h).  A CTA carries a block of
// P points through the train, their vectors in shared memory as [bond][point];
// a thread takes one point and four outputs at a time, so each v[t] is loaded
// and taken apart once per four products, the points of a warp share the lines
// of the core (one per local value), and four independent sums hide the
// latency.  100 000 points of a 30-site train with bonds of 80: 447 ms with a
// warp per point in 25 tasks, 35 ms so (both with the copies).  Few points leave
// threads over: each then takes one output (a point of 16 sites with bonds of 30
// 0.21 ms, 0.32 with four outputs a thread, 0.22 with a warp per point).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "device_once.h"
#include "ieee_int.h"
#include "tci_tasks.h"

namespace {

constexpr int NT = 512;
// What the entries of a core, or of the vectors of a CTA's points, allow.
enum { VAL_DENSE = 0, VAL_ZEROS = 1, VAL_UNSAFE = 2 };

__device__ __forceinline__ int val_class(double v) {
  return int_safe(v) ? (int_dense(v) ? VAL_DENSE : VAL_ZEROS) : VAL_UNSAFE;
}

// Largest class of each core's entries into cls (cleared before).
__global__ void __launch_bounds__(256) core_class_kernel(const tci_core_ref* cores, int* cls) {
  const tci_core_ref c = cores[blockIdx.x];
  const int64_t n = (int64_t)c.r0 * c.d * c.r1;
  int k = VAL_DENSE;
  for (int64_t e = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.y * blockDim.x)
    k = max(k, val_class(c.p[e]));
  k = __reduce_max_sync(0xffffffffu, k);
  if ((threadIdx.x & 31) == 0 && k) atomicMax(&cls[blockIdx.x], k);
}

// acc[k] += v[t] * col[t + k * stride], t = 0 .. r0-1, k < Q; v has stride P.
template <int MODE, int Q>
__device__ __forceinline__ void row_times_cols(const double* __restrict__ v, int P, const double* __restrict__ col,
                                               size_t stride, int r0, double (&acc)[Q]) {
  double x = v[0], c[Q];
#pragma unroll
  for (int k = 0; k < Q; ++k) c[k] = __ldg(col + k * stride);
  for (int t = 0; t < r0; ++t) {
    // the next step's loads before this one's arithmetic
    const int tn = t + 1 < r0 ? t + 1 : t;
    const double xn = v[(size_t)tn * P];
    double cn[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) cn[k] = __ldg(col + tn + k * stride);
    double q[Q];
    if (MODE == VAL_DENSE) {
      const DenseFactor xf = dense_split(x);
#pragma unroll
      for (int k = 0; k < Q; ++k) q[k] = int_mul_dense(xf, dense_split(c[k]));
    } else if (MODE == VAL_ZEROS) {
      const IntFactor xf = int_split(x);
#pragma unroll
      for (int k = 0; k < Q; ++k) q[k] = int_mul(xf, int_split(c[k]));
    } else {
#pragma unroll
      for (int k = 0; k < Q; ++k) q[k] = __dmul_rn(x, c[k]);
    }
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      acc[k] = __dadd_rn(acc[k], q[k]);
      c[k] = cn[k];
    }
    x = xn;
  }
}

// The sum for one output, eight terms' loads and products before their additions.
template <int MODE>
__device__ __forceinline__ double row_times_col(const double* __restrict__ v, int P, const double* __restrict__ col,
                                                int r0) {
  double acc = 0.0;
  for (int t = 0; t < r0; t += 8) {
    double x[8], c[8], q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int tk = min(t + k, r0 - 1);
      x[k] = v[(size_t)tk * P];
      c[k] = __ldg(col + tk);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      q[k] = MODE == VAL_DENSE ? int_mul_dense(dense_split(x[k]), dense_split(c[k]))
                               : (MODE == VAL_ZEROS ? int_mul(int_split(x[k]), int_split(c[k])) : __dmul_rn(x[k], c[k]));
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (t + k < r0) acc = __dadd_rn(acc, q[k]);
  }
  return acc;
}

// One site for the CTA's points: w = v * T[:, i, :].  Returns the largest class
// of the values written by this thread.
template <int MODE>
__device__ __forceinline__ int site_step(const tci_core_ref& c, const uint8_t* __restrict__ pts, int L, int s, int np,
                                         int P, const double* v, double* w) {
  int cls = VAL_DENSE;
  if (P * c.r1 <= NT) {  // few points: a thread for each output
    const int p = threadIdx.x % P, q = threadIdx.x / P;
    if (q < c.r1 && p < np) {
      const double* col = c.p + (size_t)c.r0 * (pts[(size_t)p * L + s] + (size_t)c.d * q);
      const double a = P * c.r1 <= NT / 4 ? row_times_col<VAL_UNSAFE>(v + p, P, col, c.r0)
                                          : row_times_col<MODE>(v + p, P, col, c.r0);
      w[(size_t)q * P + p] = a;
      cls = val_class(a);
    }
    return cls;
  }
  const int nq = (c.r1 + 3) >> 2;
  for (int e = threadIdx.x; e < P * nq; e += NT) {
    const int p = e % P, q0 = (e / P) * 4;  // P is a power of two
    if (p >= np) continue;
    const int i = pts[(size_t)p * L + s];
    const size_t stride = (size_t)c.r0 * c.d;
    const double* col = c.p + (size_t)c.r0 * i + stride * q0;
    if (q0 + 4 <= c.r1) {
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      row_times_cols<MODE, 4>(v + p, P, col, stride, c.r0, acc);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w[(size_t)(q0 + k) * P + p] = acc[k];
        cls = max(cls, val_class(acc[k]));
      }
    } else {
      for (int q = q0; q < c.r1; ++q) {
        double acc[1] = {0.0};
        row_times_cols<MODE, 1>(v + p, P, col + stride * (q - q0), stride, c.r0, acc);
        w[(size_t)q * P + p] = acc[0];
        cls = max(cls, val_class(acc[0]));
      }
    }
  }
  return cls;
}

__global__ void __launch_bounds__(NT) tt_eval_kernel(const tci_core_ref* __restrict__ cores, const int* __restrict__ cls,
                                                     int L, int rmax, int P, const uint8_t* __restrict__ pts,
                                                     int64_t np, double* __restrict__ out) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int vcls[2];
  for (int64_t base = (int64_t)blockIdx.x * P; base < np; base += (int64_t)gridDim.x * P) {
    const int n = (int)min((int64_t)P, np - base);
    const uint8_t* my = pts + base * L;
    double* v = smem;
    double* w = smem + (size_t)rmax * P;
    for (int p = threadIdx.x; p < P; p += NT) v[p] = 1.0;
    if (threadIdx.x == 0) {
      vcls[0] = VAL_ZEROS;  // 1 is not dense
      vcls[1] = VAL_DENSE;
    }
    __syncthreads();
    for (int s = 0; s < L; ++s) {
      const tci_core_ref c = cores[s];
      const int mode = max(cls[s], vcls[s & 1]);
      int k;
      if (mode == VAL_DENSE) k = site_step<VAL_DENSE>(c, my, L, s, n, P, v, w);
      else if (mode == VAL_ZEROS) k = site_step<VAL_ZEROS>(c, my, L, s, n, P, v, w);
      else k = site_step<VAL_UNSAFE>(c, my, L, s, n, P, v, w);
      if (k) atomicMax(&vcls[(s + 1) & 1], k);
      __syncthreads();
      if (threadIdx.x == 0) vcls[s & 1] = VAL_DENSE;  // read by all; set again after the next barrier's step
      __syncthreads();
      double* t = v;
      v = w;
      w = t;
    }
    for (int p = threadIdx.x; p < n; p += NT) out[base + p] = v[p];
    __syncthreads();
  }
}

// Points (n values of np x L multi-indices, 1-based int64, in the caller's host
// memory read across the host link) to 0-based bytes; a value outside
// [1, dims[site]] raises *bad and becomes 0.  Bound by the link (190 GB/s), with
// eight values in flight per thread: split-precision evaluation at a million
// points of 40 sites takes 8.1 ms in all, 12.1 with the packing on eight host
// threads.
__global__ void __launch_bounds__(256) pack_points_kernel(const int64_t* __restrict__ pts, int64_t n, int L,
                                                          const int* __restrict__ dims, uint8_t* __restrict__ out,
                                                          int* bad) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int wrong = 0;
  for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e0 < n; e0 += 8 * stride) {
    int64_t v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = e0 + q * stride < n ? __ldcs(pts + e0 + q * stride) : 1;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int64_t e = e0 + q * stride;
      if (e >= n) continue;
      const bool ok = v[q] >= 1 && v[q] <= dims[e % L];
      wrong |= !ok;
      out[e] = ok ? (uint8_t)(v[q] - 1) : 0;
    }
  }
  if (__any_sync(0xffffffffu, wrong) && (threadIdx.x & 31) == 0) atomicExch(bad, 1);
}

}  // namespace

// *bad must be zero.
cudaError_t tci_pack_points_launch(const int64_t* pts, int64_t np, int L, const int* dims, uint8_t* out, int* bad,
                                   int num_sms, cudaStream_t st) {
  const int64_t n = np * L, blocks = (n + 2047) / 2048;
  if (n <= 0) return cudaSuccess;
  pack_points_kernel<<<(unsigned)std::min<int64_t>(blocks, 8 * (int64_t)num_sms), 256, 0, st>>>(pts, n, L, dims, out, bad);
  return cudaGetLastError();
}

// Largest bond the kernel's shared memory takes.
int tci_tt_eval_max_bond() { return 225 * 1024 / 16; }

// cores: L records on the device, cls: L words of scratch, pts: np x L local
// indices, rmax: the largest bond.
cudaError_t tci_tt_eval_launch(const tci_core_ref* cores, int* cls, int L, int rmax, const uint8_t* pts, int64_t np,
                               double* out, int num_sms, cudaStream_t st) {
  if (np <= 0) return cudaSuccess;
  static DeviceOnce limit;
  cudaError_t e = limit(
      [] { return cudaFuncSetAttribute(tt_eval_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024); });
  if (e == cudaSuccess) e = cudaMemsetAsync(cls, 0, (size_t)L * sizeof(int), st);
  if (e != cudaSuccess) return e;
  core_class_kernel<<<dim3(L, 4), 256, 0, st>>>(cores, cls);
  // Points per CTA: as many as shared memory takes, up to 256, but no more than
  // leaves every SM a block.
  const size_t per = (size_t)rmax * 2 * sizeof(double);
  int P = 256;
  while (P > 1 && (size_t)P * per > 225 * 1024) P >>= 1;
  while (P > 1 && (np + P - 1) / P < num_sms) P >>= 1;
  const int64_t blocks = (np + P - 1) / P;
  tt_eval_kernel<<<(unsigned)std::min<int64_t>(blocks, 8 * (int64_t)num_sms), NT, (size_t)P * per, st>>>(
      cores, cls, L, rmax, P, pts, np, out);
  return cudaGetLastError();
}
