// HPL residual check (src/HPL_pdtest.cpp:307-438 with the norms of
// src/pauxil/HPL_pdlange_device.cpp:76-116), deterministic on the device.
//
// Two sources for [A|b]: a stored matrix (the reference regenerates A in
// place with HPL_pdrandmat before checking), or the LCG itself, regenerated
// inside the kernels with the same bit-exact value function, so the check
// needs no N x N buffer at all.
//
// Work split (all reductions in a fixed order, no floating-point atomics):
//   rows_partial, rows_cols_partial : grid (row blocks, column chunks); per row and
//                  chunk the partial sums of a_ij x_j and |a_ij|; the latter, for a
//                  stored matrix, also per row block and column that of |a_ij|.
//   rows_final   : per row r_i = b_i - sum, row sum of |a|; per block the
//                  maxima of |r|, row sums, |b|, |x| and the sum of |x|.
//   col_fold / col_sums : per column sum_i |a_ij| from those sums / regenerated, a
//                  warp per column; per block the max.
//   finish       : one block folds the per-block values into the 8 outputs.
#include <algorithm>

#include "common.cuh"
#include "internal.h"
#include "lcg.cuh"

namespace hplb {

namespace {

constexpr int kRowThreads = 256;
constexpr int kChunk      = 2048;  // columns per partial sum
// The stored-matrix pass (rows_cols_partial): columns whose sums wait in shared
// memory before they leave a CTA.
constexpr int kPassHalf = 512;

struct ResTabs {
  Jump pow2[64];
  Jump col;     // jump by n (next column, same row)
  Jump step32;  // jump by 32 (same column, 32 rows down)
  uint64_t x1;  // X(1)
};

HPLB_DEV uint64_t state_of(const ResTabs& T, uint64_t k) {
  Jump acc{1, 0};
  for(int b = 0; k; ++b, k >>= 1)
    if(k & 1) acc = compose(acc, T.pow2[b]);
  return apply(acc, T.x1);
}

template <bool LCG>
__global__ void __launch_bounds__(kRowThreads)
rows_partial(int n, const double* __restrict__ A, int64_t ld, const double* __restrict__ X,
             const __grid_constant__ ResTabs T, double* part_r, double* part_a) {
  const int i  = blockIdx.x * kRowThreads + threadIdx.x;
  const int j0 = blockIdx.y * kChunk;
  const int j1 = min(n, j0 + kChunk);
  if(i >= n) return;
  double acc = 0.0, asum = 0.0;
  if(LCG) {
    const Jump cj = T.col;
    uint64_t   s  = state_of(T, (uint64_t)i + (uint64_t)j0 * (uint64_t)n);
    for(int j = j0; j < j1; ++j) {
      const double a = lcg_value(s);
      acc += a * X[j];
      asum += fabs(a);
      s = apply(cj, s);
    }
  } else {
    const double* a = A + (size_t)i + (size_t)j0 * ld;
#pragma unroll 4
    for(int j = j0; j < j1; ++j, a += ld) {
      const double v = *a;
      acc += v * X[j];
      asum += fabs(v);
    }
  }
  part_r[(size_t)blockIdx.y * n + i] = acc;
  part_a[(size_t)blockIdx.y * n + i] = asum;
}

// Row sums of A x and |A| and column sums of |A| in one read of the stored A:
// HBM-bound, and a second read for the column sums would double it.  A column's
// sum over a warp's 32 rows is folded 16 columns at a time: in each of 4 steps a
// lane hands half of its columns to its partner, the last step adds neighbours
// (16 exchanges for 16 columns); the warps' sums meet in shared memory, the
// CTAs' in part_c (a row of n per 256 rows of A).  Four CTAs per SM, so that one's
// folding runs under the others' loads: the whole check at N = 16384 takes 480 us
// (858 with two passes, 725 with 32 columns at a time and two CTAs).  A has m rows
// from here on; the chunks' partial row sums are `rows` apart.  col_sums adds in the
// same order, so the stored and the regenerated check agree to the last bit.
__global__ void __launch_bounds__(kRowThreads, 4)
rows_cols_partial(int n, int m, int rows, const double* __restrict__ A, int64_t ld,
                  const double* __restrict__ X, double* part_r, double* part_a, double* part_c) {
  constexpr int     kW = kRowThreads / 32, kU = 16;
  __shared__ double sc[kW][kPassHalf];
  const int     lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int     i = blockIdx.x * kRowThreads + threadIdx.x;
  const bool    in = i < m;
  const int     jb = blockIdx.y * kChunk, je = min(n, jb + kChunk);
  const double* a = A + (in ? i : 0);
  double        acc = 0.0, asum = 0.0;
  for(int jh = jb; jh < je; jh += kPassHalf) {
    const int jhe = min(je, jh + kPassHalf);
    for(int j = jh; j < jhe; j += kU) {
      double c[kU];
#pragma unroll
      for(int u = 0; u < kU; ++u)
        c[u] = in && j + u < jhe ? __ldcs(a + (size_t)(j + u) * (size_t)ld) : 0.0;
#pragma unroll
      for(int u = 0; u < kU; ++u) {
        if(j + u < jhe) acc += c[u] * X[j + u];
        c[u] = fabs(c[u]);
        asum += c[u];
      }
#pragma unroll
      for(int s = kU / 2; s > 0; s >>= 1) {
        const bool up = (lane & (2 * s)) != 0;
#pragma unroll
        for(int u = 0; u < kU / 2; ++u)
          if(u < s) {
            const double give = up ? c[u] : c[u + s], keep = up ? c[u + s] : c[u];
            c[u]              = keep + __shfl_xor_sync(0xffffffffu, give, 2 * s);
          }
      }
      c[0] += __shfl_xor_sync(0xffffffffu, c[0], 1);
      if((lane & 1) == 0) sc[warp][j - jh + (lane >> 1)] = c[0];  // column j + lane / 2
    }
    __syncthreads();
    for(int j = threadIdx.x; j < jhe - jh; j += kRowThreads) {
      double t = 0.0;
#pragma unroll
      for(int w = 0; w < kW; ++w) t += sc[w][j];
      part_c[(size_t)blockIdx.x * n + jh + j] = t;
    }
    __syncthreads();
  }
  if(in) {
    part_r[(size_t)blockIdx.y * rows + i] = acc;
    part_a[(size_t)blockIdx.y * rows + i] = asum;
  }
}

HPLB_DEV double block_max(double v, double* sh) {
  for(int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, off));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if(lane == 0) sh[warp] = v;
  __syncthreads();
  v = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0;
  if(warp == 0)
    for(int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, off));
  return v;  // valid in thread 0
}

HPLB_DEV double block_sum(double v, double* sh) {
  for(int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if(lane == 0) sh[warp] = v;
  __syncthreads();
  v = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0;
  if(warp == 0)
    for(int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  return v;  // valid in thread 0
}

template <bool LCG>
__global__ void __launch_bounds__(kRowThreads)
rows_final(int n, int row0, int rows, int nch, const double* __restrict__ A, int64_t ld,
           const double* __restrict__ X, const __grid_constant__ ResTabs T, const double* part_r,
           const double* part_a, double* blk) {
  __shared__ double sh[32];
  const int il = blockIdx.x * kRowThreads + threadIdx.x, i = row0 + il;
  double rabs = 0.0, rsum = 0.0, babs = 0.0, xabs = 0.0, xs = 0.0;
  if(i < n) {
    double b;
    if(LCG)
      b = lcg_value(state_of(T, (uint64_t)i + (uint64_t)n * (uint64_t)n));
    else
      b = A[(size_t)i + (size_t)n * ld];
    double acc = 0.0;
    for(int c = 0; c < nch; ++c) {
      acc += part_r[(size_t)c * rows + il];
      rsum += part_a[(size_t)c * rows + il];
    }
    rabs = fabs(b - acc);
    babs = fabs(b);
    xabs = fabs(X[i]);
    xs   = xabs;
  }
  const double m0 = block_max(rabs, sh);
  const double m1 = block_max(rsum, sh);
  const double m2 = block_max(babs, sh);
  const double m3 = block_max(xabs, sh);
  const double s4 = block_sum(xs, sh);
  if(threadIdx.x == 0) {
    double* o = blk + (size_t)blockIdx.x * 5;
    o[0] = m0;
    o[1] = m1;
    o[2] = m2;
    o[3] = m3;
    o[4] = s4;
  }
}

// Column sums so far (sum; from zero if `first`) and nrg more row groups' of a CTA's
// 256 columns; the last time, their largest to blkc.
__global__ void __launch_bounds__(256)
col_fold(int n, int nrg, const double* __restrict__ part_c, bool first, bool last, double* sum,
         double* blkc) {
  __shared__ double sh[32];
  const int j = blockIdx.x * 256 + threadIdx.x;
  double    s = (first || j >= n) ? 0.0 : sum[j];
  if(j < n)
    for(int g = 0; g < nrg; ++g) s += part_c[(size_t)g * n + j];
  if(!last) {
    if(j < n) sum[j] = s;
    return;
  }
  const double m = block_max(s, sh);
  if(threadIdx.x == 0) blkc[blockIdx.x] = m;
}

// Column sums of the regenerated matrix, added in the order of rows_cols_partial's
// folds.  The regenerating check as a whole: N = 1000 0.11 ms, 16384 0.69, 131072 34.2
// (0.15, 0.73 and 35.3 with lanes that keep sums of their own to the end and four more
// FP64 steps per entry).
__global__ void __launch_bounds__(256)
col_sums(int n, const __grid_constant__ ResTabs T, double* blkc) {
  __shared__ double sh[32];
  const int lane = threadIdx.x & 31;
  const int j    = blockIdx.x * 8 + (threadIdx.x >> 5);
  double    s    = 0.0;
  if(j < n) {
    const Jump st = T.step32;
    uint64_t   x  = state_of(T, (uint64_t)lane + (uint64_t)j * (uint64_t)n);
    for(int i0 = 0; i0 < n; i0 += kRowThreads) {
      double t = 0.0;
      for(int i = i0 + lane; i - lane < min(n, i0 + kRowThreads); i += 32) {
        double v = i < n ? fabs(lcg_value(x)) : 0.0;
        x        = apply(st, x);
        for(int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        t += v;
      }
      s += t;
    }
  }
  // s valid in lane 0 of each warp; block max over the 8 columns.
  s = __shfl_sync(0xffffffffu, s, 0);
  const double m = block_max(lane == 0 ? s : 0.0, sh);
  if(threadIdx.x == 0) blkc[blockIdx.x] = m;
}

__global__ void __launch_bounds__(256) finish(int n, int nrb, int ncb, const double* blk,
                                              const double* blkc, double* out) {
  __shared__ double sh[32];
  double v[5] = {0, 0, 0, 0, 0};
  for(int b = threadIdx.x; b < nrb; b += blockDim.x) {
    const double* o = blk + (size_t)b * 5;
    v[0] = fmax(v[0], o[0]);
    v[1] = fmax(v[1], o[1]);
    v[2] = fmax(v[2], o[2]);
    v[3] = fmax(v[3], o[3]);
  }
  // The |x| sum in block order, one thread, for a fixed summation order.
  double cm = 0.0;
  for(int b = threadIdx.x; b < ncb; b += blockDim.x) cm = fmax(cm, blkc[b]);
  const double rn = block_max(v[0], sh);
  const double ai = block_max(v[1], sh);
  const double bn = block_max(v[2], sh);
  const double xi = block_max(v[3], sh);
  const double a1 = block_max(cm, sh);
  if(threadIdx.x == 0) {
    double x1 = 0.0;
    for(int b = 0; b < nrb; ++b) x1 += blk[(size_t)b * 5 + 4];
    const double eps = 0x1p-53;
    out[0] = n > 0 ? rn / (eps * (ai * xi + bn) * (double)n) : 0.0;
    out[1] = rn;
    out[2] = a1;
    out[3] = ai;
    out[4] = x1;
    out[5] = xi;
    out[6] = bn;
    out[7] = eps;
  }
}

// The LCG jumps of an n-row matrix, passed to the kernels by value.
ResTabs make_tabs(int n, uint64_t seed) {
  ResTabs T;
  Jump    p{kLcgMult, kLcgAdd};
  for(int b = 0; b < 64; ++b) {
    T.pow2[b] = p;
    p         = compose(p, p);
  }
  T.col    = jump_by((uint64_t)n);
  T.step32 = jump_by(32);
  T.x1     = kLcgMult * seed + kLcgAdd;
  return T;
}

}  // namespace

namespace {

// The stored check's partial column sums take n doubles per 256 rows (n^2 / 256 in
// all), its partial row sums 2 per row and 2048 columns (n^2 / 1024).  Matrices of
// more than kOneBand row groups (102400 rows, 84 GB) are read in kBands bands of rows
// that share the space of one, so that a matrix that fills the GPU needs no more
// than n^2 / 1024 (N = 131072: 128 MB, one band 671 MB).  Each band's last CTAs run
// alone for a moment: N = 131072 25.8 -> 26.5 ms, but N = 50000 3.4 -> 5.1, so smaller
// matrices stay in one.
constexpr int kOneBand = 400, kBands = 6;

struct Bands {
  int count, groups;  // bands, and 256-row groups of each but the last
};
Bands bands_of(int n) {
  const int nrb = (n + kRowThreads - 1) / kRowThreads;
  const int c   = nrb > kOneBand ? kBands : 1;
  const int g   = (nrb + c - 1) / c;
  return {(nrb + g - 1) / g, g};
}

}  // namespace

// Doubles of scratch of the check, and of launch_gemv_hpl, for a stored or a
// regenerated matrix.
size_t residual_ws_doubles(int n, bool lcg) {
  const size_t nch = (size_t)(n + kChunk - 1) / kChunk;
  const size_t nrb = (size_t)(n + kRowThreads - 1) / kRowThreads;
  const size_t ncb = (size_t)(n + 7) / 8;
  size_t       part = 2 * nch * (size_t)n;
  if(!lcg) {
    const Bands b = bands_of(n);
    part          = std::max(part, 2 * nch * (size_t)b.groups * kRowThreads +
                                       (size_t)(b.groups + 1) * (size_t)n);
  }
  return part + 5 * nrb + ncb + 16;
}

cudaError_t launch_residual(int n, const double* A, int64_t ld, bool lcg, uint64_t seed,
                            const double* X, double* ws, double* out8, cudaStream_t stream) {
  if(n <= 0) return cudaMemsetAsync(out8, 0, 8 * sizeof(double), stream);
  const int nrb = (n + kRowThreads - 1) / kRowThreads;
  const int nch = (n + kChunk - 1) / kChunk;
  if(!lcg) {
    const int    ncb    = (n + 255) / 256;
    const Bands  b      = bands_of(n);
    const int    rows   = b.groups * kRowThreads;
    double*      part_r = ws;
    double*      part_a = part_r + (size_t)nch * rows;
    double*      part_c = part_a + (size_t)nch * rows;
    double*      sum    = part_c + (size_t)b.groups * n;
    double*      blk    = sum + n;
    double*      blkc   = blk + (size_t)nrb * 5;
    for(int k = 0; k < b.count; ++k) {
      const int g0 = k * b.groups, ng = std::min(b.groups, nrb - g0), row0 = g0 * kRowThreads;
      rows_cols_partial<<<dim3(ng, nch), kRowThreads, 0, stream>>>(n, n - row0, rows, A + row0, ld, X,
                                                                   part_r, part_a, part_c);
      rows_final<false><<<ng, kRowThreads, 0, stream>>>(n, row0, rows, nch, A, ld, X, ResTabs{},
                                                        part_r, part_a, blk + (size_t)g0 * 5);
      col_fold<<<ncb, 256, 0, stream>>>(n, ng, part_c, k == 0, k + 1 == b.count, sum, blkc);
    }
    finish<<<1, 256, 0, stream>>>(n, nrb, ncb, blk, blkc, out8);
    return cudaGetLastError();
  }
  const int ncb = (n + 7) / 8;
  double* part_r = ws;
  double* part_a = part_r + (size_t)nch * n;
  double* blk    = part_a + (size_t)nch * n;
  double* blkc   = blk + (size_t)nrb * 5;
  const ResTabs T = make_tabs(n, seed);
  dim3 g1(nrb, nch);
  rows_partial<true><<<g1, kRowThreads, 0, stream>>>(n, A, ld, X, T, part_r, part_a);
  rows_final<true><<<nrb, kRowThreads, 0, stream>>>(n, 0, n, nch, A, ld, X, T, part_r, part_a, blk);
  col_sums<<<ncb, 256, 0, stream>>>(n, T, blkc);
  finish<<<1, 256, 0, stream>>>(n, nrb, ncb, blk, blkc, out8);
  return cudaGetLastError();
}

namespace {

// y[i] = sum of the per-chunk partials of row i (fixed order).
__global__ void rows_sum(int n, int nch, const double* __restrict__ part, double* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= n) return;
  double acc = 0.0;
  for(int c = 0; c < nch; ++c) acc += part[(size_t)c * n + i];
  y[i] = acc;
}

// out[i] = A(i, col), from the stored matrix or regenerated from the LCG.
template <bool LCG>
__global__ void column_of(int n, int col, const double* __restrict__ A, int64_t ld,
                          const __grid_constant__ ResTabs T, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= n) return;
  if(LCG)
    out[i] = lcg_value(state_of(T, (uint64_t)i + (uint64_t)col * (uint64_t)n));
  else
    out[i] = A[(size_t)i + (size_t)col * ld];
}

}  // namespace

// y = A x for the n x n part of [A|b], FP64, from the stored matrix or the LCG.
// ws: residual_ws_doubles(n, lcg) doubles.
cudaError_t launch_gemv_hpl(int n, const double* A, int64_t ld, bool lcg, uint64_t seed,
                            const double* x, double* y, double* ws, cudaStream_t stream) {
  if(n <= 0) return cudaSuccess;
  const int nch = (n + kChunk - 1) / kChunk;
  const int nrb = (n + kRowThreads - 1) / kRowThreads;
  double*   part_r = ws;
  double*   part_a = part_r + (size_t)nch * n;
  const ResTabs T = make_tabs(n, seed);
  dim3 g1(nrb, nch);
  if(lcg)
    rows_partial<true><<<g1, kRowThreads, 0, stream>>>(n, A, ld, x, T, part_r, part_a);
  else
    rows_partial<false><<<g1, kRowThreads, 0, stream>>>(n, A, ld, x, T, part_r, part_a);
  rows_sum<<<nrb, kRowThreads, 0, stream>>>(n, nch, part_r, y);
  return cudaGetLastError();
}

// out = column col of [A|b] (col = n gives b).
cudaError_t launch_column_hpl(int n, int col, const double* A, int64_t ld, bool lcg,
                              uint64_t seed, double* out, cudaStream_t stream) {
  if(n <= 0) return cudaSuccess;
  const ResTabs T = make_tabs(n, seed);
  const int nrb = (n + kRowThreads - 1) / kRowThreads;
  if(lcg)
    column_of<true><<<nrb, kRowThreads, 0, stream>>>(n, col, A, ld, T, out);
  else
    column_of<false><<<nrb, kRowThreads, 0, stream>>>(n, col, A, ld, T, out);
  return cudaGetLastError();
}

}  // namespace hplb

// ---------------------------------------------------------------------------
// Allocation-free residual check.
//
// For callers that must not allocate device memory at all: a host program that
// has handed every byte of device memory to its own pool, or a check that runs
// between solves in a loop where cudaMalloc's implicit device synchronisation is
// not allowed.  The scratch of the kernels above lives in the file-scope array
// below instead of a context workspace, so this entry point needs neither a
// context nor an allocation.  The array is fixed in size (it serves
// n <= HPLB_NOALLOC_MAX_N) and every GPU that loads the library holds it until
// the process exits.
// ---------------------------------------------------------------------------

#include <cstdio>
#include <mutex>

namespace hplb {
namespace {

constexpr int    kNoAllocMaxN = HPLB_NOALLOC_MAX_N;
constexpr size_t kNoAllocWs   = 2 * ((size_t)(kNoAllocMaxN + kChunk - 1) / kChunk) * kNoAllocMaxN +
                                5 * ((size_t)(kNoAllocMaxN + kRowThreads - 1) / kRowThreads) +
                                (size_t)(kNoAllocMaxN + 7) / 8 + 16 + 8;

// Shared by every call on a device; it keeps the last call's contents.  No
// kernel of the check accumulates into it (every partial sum, per-block value
// and output is overwritten before it is read), so nothing has to be cleared.
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocWs];

constexpr int kMaxDevices = 64;
std::mutex    g_noalloc_mu;
double*       g_noalloc_ptr[kMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device.  In host code the
// array's name is only a host-side stand-in, so the address is looked up once
// per device (with that device current) and cached.
cudaError_t noalloc_scratch(int dev, double** out) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if(!g_noalloc_ptr[dev]) {
    void*       p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if(e != cudaSuccess) return e;
    g_noalloc_ptr[dev] = (double*)p;
  }
  *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

}  // namespace
}  // namespace hplb

extern "C" hplb_status hplb_residual_lcg_noalloc(int n, uint64_t seed, const double* dX,
                                                 void* stream, hplb_resid* out) {
  using namespace hplb;
  if(!out || n < 0 || (n > 0 && !dX)) return HPLB_ERR_ARG;
  if(n > kNoAllocMaxN) {
    fprintf(stderr,
            "hplb_residual_lcg_noalloc: n = %d exceeds the static scratch limit "
            "HPLB_NOALLOC_MAX_N = %d; use hplb_residual_lcg\n",
            n, kNoAllocMaxN);
    return HPLB_ERR_ARG;
  }
  int dev = 0;
  if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return HPLB_ERR_CUDA;
  }
  double* ws = nullptr;
  if(noalloc_scratch(dev, &ws) != cudaSuccess) {
    cudaGetLastError();
    return HPLB_ERR_CUDA;
  }
  cudaStream_t st   = (cudaStream_t)stream;
  double*      out8 = ws + (kNoAllocWs - 8);
  if(launch_residual(n, nullptr, 0, true, seed, dX, ws, out8, st) != cudaSuccess) {
    cudaGetLastError();
    return HPLB_ERR_CUDA;
  }
  double o[8];
  if(cudaMemcpyAsync(o, out8, sizeof o, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
     cudaStreamSynchronize(st) != cudaSuccess) {
    cudaGetLastError();
    return HPLB_ERR_CUDA;
  }
  out->resid     = o[0];
  out->rnorm_inf = o[1];
  out->anorm_1   = o[2];
  out->anorm_inf = o[3];
  out->xnorm_1   = o[4];
  out->xnorm_inf = o[5];
  out->bnorm_inf = o[6];
  out->eps       = o[7];
  return HPLB_OK;
}
