// Kernels of the device value cache of a caller-supplied f (fcache.h): probe a
// product of row and column keys against the table and compact the misses,
// insert new values, and rehash into a larger table.  All HBM-bound integer
// work: one 32-byte slot per probe step, load factor at most 1/2.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fc_slot.h"
#include "fcache.h"

namespace tci {
namespace {

constexpr int FC_THREADS = 256;

int fc_grid(int64_t n) {
  int64_t g = (n + FC_THREADS - 1) / FC_THREADS;
  if (g > 152 * 16) g = 152 * 16;
  return (int)(g < 1 ? 1 : g);
}

__device__ __forceinline__ bool fc_find(const tci_fc_entry* tab, uint64_t mask, uint64_t k0, uint64_t k1) {
  uint64_t h = tci_fc_hash(k0, k1) & mask;
  for (uint64_t q = 0; q <= mask; ++q) {
    const uint64_t e0 = tab[h].k0;
    if (e0 == k0 && tab[h].k1 == k1) return true;
    if (e0 == TCI_FC_EMPTY) return false;
    h = (h + 1) & mask;
  }
  return false;
}

// Element e = i + nr * j of the product rows x columns: key = rk[i] + ck[j]
// (word by word; the halves of a row and a column cover disjoint sites).  A miss
// appends (j << 32 | i) to miss[].
__global__ void __launch_bounds__(FC_THREADS)
    fc_probe_kernel(const tci_fc_entry* __restrict__ tab, uint64_t mask, const int64_t* __restrict__ rk, int64_t nr,
                    const int64_t* __restrict__ ck, int64_t nc, unsigned long long* count,
                    uint64_t* __restrict__ miss) {
  const int64_t n = nr * nc;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % nr, j = e / nr;
    const uint64_t k0 = (uint64_t)(rk[2 * i] + ck[2 * j]);
    const uint64_t k1 = (uint64_t)(rk[2 * i + 1] + ck[2 * j + 1]);
    if (!fc_find(tab, mask, k0, k1)) {
      const unsigned long long at = atomicAdd(count, 1ull);
      miss[at] = ((uint64_t)j << 32) | (uint64_t)i;
    }
  }
}

// The misses of one product in order, as the points the caller gets: a flag per
// element, the blocks' offsets, then the points.  On the host the same (a sort of
// the misses, a set against repeats, multi-indices one by one) took some 90 ns a
// point: a solve with 100,000 evaluations 19.6 ms, 10.3 so.  A block takes FC_TILE
// elements, eight probes a thread; bound by the probes' latency and the host link.
constexpr int FC_TILE = 2048;

__global__ void __launch_bounds__(FC_THREADS)
    fc_flag_kernel(const tci_fc_entry* __restrict__ tab, uint64_t mask, const int64_t* __restrict__ rk, int64_t nr,
                   const int64_t* __restrict__ ck, int64_t nc, uint32_t* __restrict__ flags,
                   unsigned* __restrict__ counts) {
  const int64_t n = nr * nc, e0 = (int64_t)blockIdx.x * FC_TILE;
  __shared__ unsigned total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  unsigned mine = 0;
  for (int k = threadIdx.x; k < FC_TILE; k += FC_THREADS) {
    const int64_t e = e0 + k;
    bool miss = false;
    if (e < n) {
      const int64_t j = e / nr, i = e - j * nr;
      miss = !fc_find(tab, mask, (uint64_t)(rk[2 * i] + ck[2 * j]), (uint64_t)(rk[2 * i + 1] + ck[2 * j + 1]));
    }
    const unsigned word = __ballot_sync(0xffffffffu, miss);
    if ((threadIdx.x & 31) == 0) {
      flags[(e0 + k) / 32] = word;
      mine += __popc(word);
    }
  }
  if (mine) atomicAdd(&total, mine);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// Exclusive sums of the counts in place, by one warp; the total to *all (host memory).
__global__ void __launch_bounds__(32) fc_offsets_kernel(unsigned* counts, int nblocks, unsigned long long* all) {
  unsigned base = 0;
  for (int b0 = 0; b0 < nblocks; b0 += 32) {
    const int b = b0 + threadIdx.x;
    const unsigned c = b < nblocks ? counts[b] : 0u;
    unsigned s = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned o = __shfl_up_sync(0xffffffffu, s, off);
      if (threadIdx.x >= off) s += o;
    }
    if (b < nblocks) counts[b] = base + s - c;
    base += __shfl_sync(0xffffffffu, s, 31);
  }
  if (threadIdx.x == 0) *all = base;
}

// Miss x of the product: its element to where[x], its L values (1-based) to
// pts[x * L ..] (host memory, written in runs).
__global__ void __launch_bounds__(FC_THREADS)
    fc_points_kernel(const uint32_t* __restrict__ flags, const unsigned* __restrict__ offsets, int64_t nr, int64_t nc,
                     const uint8_t* __restrict__ rows, int rl, const uint8_t* __restrict__ cols, int cl,
                     uint64_t* __restrict__ where, int64_t* __restrict__ pts) {
  constexpr int WORDS = FC_TILE / 32;
  const int64_t n = nr * nc, e0 = (int64_t)blockIdx.x * FC_TILE;
  __shared__ uint32_t word[WORDS];
  __shared__ int before[WORDS + 1];
  __shared__ uint16_t list[FC_TILE];
  for (int q = threadIdx.x; q < WORDS; q += FC_THREADS) word[q] = e0 + 32 * q < n ? flags[e0 / 32 + q] : 0u;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int q = 0; q < WORDS; ++q) {
      before[q] = s;
      s += __popc(word[q]);
    }
    before[WORDS] = s;
  }
  __syncthreads();
  const int64_t x0 = offsets[blockIdx.x];
  for (int k = threadIdx.x; k < FC_TILE; k += FC_THREADS) {
    const uint32_t w = word[k / 32];
    if (w >> (k & 31) & 1u) {
      const int x = before[k / 32] + __popc(w & ((1u << (k & 31)) - 1u));
      list[x] = (uint16_t)k;
      where[x0 + x] = (uint64_t)(e0 + k);
    }
  }
  __syncthreads();
  const int L = rl + cl, total = before[WORDS] * L;
  for (int q = threadIdx.x; q < total; q += FC_THREADS) {
    const int x = q / L, c = q - x * L;
    const int64_t e = e0 + list[x], j = e / nr, i = e - j * nr;
    pts[x0 * L + q] = (int64_t)(c < rl ? rows[i * rl + c] : cols[j * cl + (c - rl)]) + 1;
  }
}

// Keys in `in` are distinct and absent from the table, so a slot whose word 0
// is taken (even by an equal word 0) belongs to another key: claim the first
// free slot on the probe path.
__device__ __forceinline__ void fc_put(tci_fc_entry* tab, uint64_t mask, const tci_fc_entry& x) {
  uint64_t h = tci_fc_hash(x.k0, x.k1) & mask;
  for (uint64_t q = 0; q <= mask; ++q) {
    const unsigned long long prev =
        atomicCAS((unsigned long long*)&tab[h].k0, (unsigned long long)TCI_FC_EMPTY, (unsigned long long)x.k0);
    if (prev == TCI_FC_EMPTY) {
      tab[h].k1 = x.k1;
      tab[h].v = x.v;
      return;
    }
    h = (h + 1) & mask;
  }
}

__global__ void __launch_bounds__(FC_THREADS)
    fc_insert_kernel(tci_fc_entry* tab, uint64_t mask, const tci_fc_entry* __restrict__ in, int64_t n) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    fc_put(tab, mask, in[e]);
}

// The values of a product's misses (distinct and absent as above; vals in host memory).
__global__ void __launch_bounds__(FC_THREADS)
    fc_store_kernel(tci_fc_entry* tab, uint64_t mask, const int64_t* __restrict__ rk, int64_t nr,
                    const int64_t* __restrict__ ck, const uint64_t* __restrict__ where,
                    const double* __restrict__ vals, int64_t n) {
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = (int64_t)where[x], j = e / nr, i = e - j * nr;
    tci_fc_entry y;
    y.k0 = (uint64_t)(rk[2 * i] + ck[2 * j]);
    y.k1 = (uint64_t)(rk[2 * i + 1] + ck[2 * j + 1]);
    y.v = vals[x];
    y.unused = 0;
    fc_put(tab, mask, y);
  }
}

__global__ void __launch_bounds__(FC_THREADS)
    fc_rehash_kernel(tci_fc_entry* dst, uint64_t dmask, const tci_fc_entry* __restrict__ src, uint64_t scap) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < scap; e += (uint64_t)gridDim.x * blockDim.x)
    if (src[e].k0 != TCI_FC_EMPTY) fc_put(dst, dmask, src[e]);
}

}  // namespace

void fc_probe_launch(const tci_fc_entry* tab, uint64_t mask, const int64_t* rk, int64_t nr, const int64_t* ck,
                     int64_t nc, unsigned long long* count, uint64_t* miss, cudaStream_t s) {
  if (nr <= 0 || nc <= 0) return;
  fc_probe_kernel<<<fc_grid(nr * nc), FC_THREADS, 0, s>>>(tab, mask, rk, nr, ck, nc, count, miss);
}

size_t fc_blocks(int64_t n) { return (size_t)((n + FC_TILE - 1) / FC_TILE); }

void fc_flag_launch(const tci_fc_entry* tab, uint64_t mask, const int64_t* rk, int64_t nr, const int64_t* ck,
                    int64_t nc, uint32_t* flags, unsigned* counts, unsigned long long* all, cudaStream_t s) {
  const int nb = (int)fc_blocks(nr * nc);
  fc_flag_kernel<<<nb, FC_THREADS, 0, s>>>(tab, mask, rk, nr, ck, nc, flags, counts);
  fc_offsets_kernel<<<1, 32, 0, s>>>(counts, nb, all);
}

void fc_points_launch(const uint32_t* flags, const unsigned* offsets, int64_t nr, int64_t nc, const uint8_t* rows,
                      int rl, const uint8_t* cols, int cl, uint64_t* where, int64_t* pts, cudaStream_t s) {
  fc_points_kernel<<<(int)fc_blocks(nr * nc), FC_THREADS, 0, s>>>(flags, offsets, nr, nc, rows, rl, cols, cl, where,
                                                                  pts);
}

void fc_store_launch(tci_fc_entry* tab, uint64_t mask, const int64_t* rk, int64_t nr, const int64_t* ck,
                     const uint64_t* where, const double* vals, int64_t n, cudaStream_t s) {
  if (n <= 0) return;
  fc_store_kernel<<<fc_grid(n), FC_THREADS, 0, s>>>(tab, mask, rk, nr, ck, where, vals, n);
}

void fc_insert_launch(tci_fc_entry* tab, uint64_t mask, const tci_fc_entry* in, int64_t n, cudaStream_t s) {
  if (n <= 0) return;
  fc_insert_kernel<<<fc_grid(n), FC_THREADS, 0, s>>>(tab, mask, in, n);
}

void fc_rehash_launch(tci_fc_entry* dst, uint64_t dmask, const tci_fc_entry* src, uint64_t scap, cudaStream_t s) {
  if (scap == 0) return;
  fc_rehash_kernel<<<fc_grid((int64_t)scap), FC_THREADS, 0, s>>>(dst, dmask, src, scap);
}

}  // namespace tci
