// Back-solve U x = y at P = Q = 1 (src/pgesv/HPL_pdtrsv_device.cpp:29-346).
//
// y is column n of the factored [A|b] (or a vector of its own); x is written
// to X; A and y are not modified.
// The reference solves bottom-up in NB blocks: rocblas_dtrsv on the diagonal
// block, then rocblas_dgemv to remove that block's contribution from every row
// above, two serial library calls per block.  Here the whole solve is ONE
// persistent kernel, HBM-bound on the single pass over the upper triangle
// (n^2/2 * 8 bytes):
//
//  * CTA k (in the order CTAs start, from an atomic ticket) owns row block
//    bi = nblk - 1 - k of kTb rows, so row blocks are taken bottom first.
//  * It streams its row panel U[bi, j] for j = nblk-1 down to bi+1, 16-byte
//    column segments, the next tile loaded while it waits for the current one's
//    x block, and accumulates U[bi, j] x_j in registers (each warp owns 8 of
//    the 64 columns of every tile, each lane 2 rows).
//  * x_j is published by the CTA that owns row block j: a release store of
//    flag j after x_j is written; readers acquire it.  A CTA only waits for
//    row blocks below its own, whose tickets were taken by CTAs that started
//    before it, so every wait ends; each is also bounded (status site 41).
//  * While the first flag is awaited the CTA inverts its own diagonal block
//    U_ii in shared memory (off the critical path), so the serial chain
//    through the blocks costs one 64 x 64 product per block instead of a
//    64-step substitution: x_i = U_ii^-1 (y_i - sum_j U_ij x_j).
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace hplb {

namespace {

constexpr int kTb          = 64;   // rows (and columns) per block
constexpr int kTrsvThreads = 256;  // 8 warps
constexpr int kTrsvWarps   = kTrsvThreads / 32;
constexpr int kColsPerWarp = kTb / kTrsvWarps;  // columns of a tile per warp
constexpr int kTrsvSite    = 41;

struct TrsvSmem {
  double T[kTb][kTb + 1];          // U_ii, then U_ii^-1 (upper triangular)
  double red[kTrsvWarps][kTb];     // per-warp partial row sums
  double r[kTb];                   // right-hand side of the diagonal block
  double tmp[kTb];
  int    ticket;
};

// Spin (bounded) until flag == 1; false once this or any block timed out.
HPLB_DEV bool wait_flag(const int* flag, int* status, int site = kTrsvSite) {
  if(ld_acquire_gpu(flag) != 0) return true;
  const unsigned long long t0 = globaltimer();
  for(unsigned polls = 1;; ++polls) {
    if(ld_acquire_gpu(flag) != 0) return true;
    if((polls & 31u) == 0) {
      if(ld_acquire_gpu(status + ST_TIMEOUT) != 0) return false;
      if(globaltimer() - t0 > kWaitBudgetNs) {
        atomicCAS(status + ST_TIMEOUT, 0, site);
        return false;
      }
    }
    __nanosleep(32);
  }
}

template <bool VEC>
HPLB_DEV void load_tile(const double* __restrict__ A, int64_t ld, int r0, int c0, int kc,
                        int lane, int warp, double2 (&v)[kColsPerWarp]) {
#pragma unroll
  for(int q = 0; q < kColsPerWarp; ++q) {
    const int c = warp + kTrsvWarps * q;
    if(c < kc) {
      const double* p = A + (size_t)(r0 + 2 * lane) + (size_t)(c0 + c) * (size_t)ld;
      if(VEC) {
        v[q] = __ldcs(reinterpret_cast<const double2*>(p));
      } else {
        v[q].x = __ldcs(p);
        v[q].y = __ldcs(p + 1);
      }
    } else {
      v[q] = make_double2(0.0, 0.0);
    }
  }
}

// In-place inverse of the upper triangular kTb x kTb block T (column by
// column, left to right: column j of the inverse is -T_jj^-1 times the
// already-inverted leading block applied to column j of U).  256 threads; T is
// the identity from row and column kb on, which takes no step.
HPLB_DEV void invert_upper(double (*T)[kTb + 1], int kb) {
  const int t = threadIdx.x, row = t >> 2, part = t & 3;
  for(int j = 0; j < kb; ++j) {
    double s = 0.0;
    if(row < j)
      for(int k = row + part; k < j; k += 4) s = fma(T[row][k], T[k][j], s);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    const double d = 1.0 / T[j][j];
    __syncthreads();
    if(part == 0 && row < j) T[row][j] = -d * s;
    if(t == 0) T[j][j] = d;
    __syncthreads();
  }
}

template <bool VEC>
__global__ void __launch_bounds__(kTrsvThreads)
trsv_kernel(const double* __restrict__ A, int64_t ld, int n, const double* __restrict__ Y,
            double* __restrict__ X, int* flags, int* status) {
  __shared__ TrsvSmem S;
  const int nblk = (n + kTb - 1) / kTb;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if(t == 0) S.ticket = atomicAdd(flags + nblk, 1);
  __syncthreads();
  const int bi = nblk - 1 - S.ticket;
  const int r0 = bi * kTb;
  const int kb = min(kTb, n - r0);

  // First tile of the row panel in flight before anything else.
  double2 cur[kColsPerWarp], nxt[kColsPerWarp];
#pragma unroll
  for(int q = 0; q < kColsPerWarp; ++q) cur[q] = nxt[q] = make_double2(0.0, 0.0);
  int     j = nblk - 1;
  if(j > bi) load_tile<VEC>(A, ld, r0, j * kTb, min(kTb, n - j * kTb), lane, warp, cur);

  // Diagonal block (identity beyond kb), inverted while the loads fly.
  for(int idx = t; idx < kTb * kTb; idx += kTrsvThreads) {
    const int c = idx / kTb, r = idx % kTb;
    double    v = (r == c) ? 1.0 : 0.0;
    if(r < kb && c < kb) v = r <= c ? A[(size_t)(r0 + r) + (size_t)(r0 + c) * (size_t)ld] : 0.0;
    S.T[r][c] = v;
  }
  if(t < kTb) S.r[t] = t < kb ? Y[r0 + t] : 0.0;
  __syncthreads();
  invert_upper(S.T, kb);

  // Row panel: acc = sum_j U[bi, j] x_j over the rows 2 lane, 2 lane + 1.
  double acc0 = 0.0, acc1 = 0.0;
  bool   alive = true;
  for(; j > bi; --j) {
    if(j - 1 > bi) load_tile<VEC>(A, ld, r0, (j - 1) * kTb, kTb, lane, warp, nxt);
    if(alive) alive = wait_flag(flags + j, status);
    const double* xj = X + (size_t)j * kTb;
    const int     kc = min(kTb, n - j * kTb);
#pragma unroll
    for(int q = 0; q < kColsPerWarp; ++q) {
      const int    c  = warp + kTrsvWarps * q;
      const double xc = c < kc ? __ldcg(xj + c) : 0.0;
      acc0            = fma(cur[q].x, xc, acc0);
      acc1            = fma(cur[q].y, xc, acc1);
    }
#pragma unroll
    for(int q = 0; q < kColsPerWarp; ++q) cur[q] = nxt[q];
  }

  // r = y_i - sum_j U_ij x_j, then x_i = U_ii^-1 r.
  S.red[warp][2 * lane]     = acc0;
  S.red[warp][2 * lane + 1] = acc1;
  __syncthreads();
  if(t < kTb) {
    double s = 0.0;
#pragma unroll
    for(int w = 0; w < kTrsvWarps; ++w) s += S.red[w][t];
    S.tmp[t] = S.r[t] - s;
  }
  __syncthreads();
  {
    const int m = t & (kTb - 1), q = t / kTb;  // 4 quarters of the 64 columns
    double    s = 0.0;
#pragma unroll
    for(int k = 0; k < kTb / 4; ++k) s = fma(S.T[m][q * (kTb / 4) + k], S.tmp[q * (kTb / 4) + k], s);
    S.red[q][m] = s;
  }
  __syncthreads();
  if(t < kb) {
    X[r0 + t] = (S.red[0][t] + S.red[1][t]) + (S.red[2][t] + S.red[3][t]);
    __threadfence();
  }
  __syncthreads();
  if(t == 0) st_release_gpu(flags + bi, 1);
}

// ---- triangular solves with up to kNr right-hand sides per launch ----
//
// trsv_kernel's structure for blocks of kTb rows x kNg right-hand sides.  Upper:
// U X = Y from the last row block up.  Lower: X <- L^-1 X for the unit-lower
// ns x ns L from the first row block down, and for the rows below it (up to
// rows) X -= L21 X_top, their tiles consumed as the blocks of X_top appear.  A
// CTA (ticket order: it waits only for CTAs that started before it) owns one row
// block of one group of right-hand sides and walks its row panel; each 64 x 64
// tile is staged by asynchronous copies (two buffers) beside the published block
// x_j, and the CTA's product is a DMMA m16n8k8 per warp and 8 columns (4 row
// tiles, the 64 columns in two halves).  Then x = D^-1 (y - sum) with the
// diagonal block (of a lower one its halves of 32) inverted while the first tile
// lands.
//
// Bound by the chain of row blocks: flag, x_j, one tile product, D^-1 product,
// store, flag.  Eight right-hand sides per CTA (four CTAs share a tile through
// L2) and the tensor-core products keep that chain short: the earlier form, 32
// right-hand sides per CTA with FMA loops bound by shared-memory loads, took
// 12.3 us per row block (N = 8192: 1576 us, now 424 us).  Up to 128 right-hand sides
// run in one launch, their groups' chains beside each other; a launch per 32 was as
// many chains in turn (hplb_getrs, 64 right-hand sides, N = 1000, NB = 64: plain 1.30,
// transposed 3.20 ms; one launch 0.73 and 2.16).  Waits are bounded (status site 42).  X may
// alias Y: a block of Y is read only by its own CTA, before that CTA writes X there.
constexpr int kNr       = 128;      // right-hand sides per launch
constexpr int kNg       = 8;        // right-hand sides per CTA
constexpr int kTp       = kTb + 4;  // pitch = 4 mod 16: fragment loads free of conflicts
constexpr int kTrsmSite = 42;

struct TrsmSmem {
  double U[2][kTb][kTp];  // staged tiles, [column][row]
  double X[2][kNg][kTp];  // the staged tile's x_j, [rhs][row]; then y - sum
  double T[kTb][kTp];     // the diagonal block (lower: transposed), then its inverse
  int    ticket;
};

HPLB_DEV void cp_async16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
HPLB_DEV void cp_async8(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
HPLB_DEV void dmma(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// In-place inverse X by a warp of the upper triangular w x w block at (o, o) of T (the
// identity from w on), a row of X per lane, column by column: a step's column is final
// in s[0]; the columns after it move one register down.  So X T = I is solved for: with
// T X = I, a column per lane, U x - y is smaller but the solution of A x = b is worse
// (|A x - b| 1.3 times as large at n = 64); of L, whose transpose T is, it solves for
// the columns of L^-1.
template <bool UNIT>
HPLB_DEV void invert_upper32(double (*T)[kTp], int o, int w) {
  constexpr int kW = 32;
  const int     lane = threadIdx.x & 31;
  const double  d = UNIT ? 1.0 : 1.0 / T[o + lane][o + lane];
  double        s[kW];
#pragma unroll
  for(int i = 0; i < kW; ++i) s[i] = i == lane ? 1.0 : 0.0;
  int k = 0;
#pragma unroll
  for(int half = 0; half < 2; ++half) {  // the second with half of the columns left
#pragma unroll 1
    for(; k < w && (half == 1 || k < kW / 2); ++k) {
      const double dk = UNIT ? 1.0 : __shfl_sync(0xffffffffu, d, k);
      const double x  = lane <= k ? s[0] * dk : 0.0;
#pragma unroll
      for(int h = 0; h < (half == 0 ? kW : kW / 2); h += kW / 4) {
        double u[kW / 4];
#pragma unroll
        for(int t = 0; t < kW / 4; ++t)
          u[t] = k + 1 + h + t < w ? T[o + k][o + k + 1 + h + t] : 0.0;
#pragma unroll
        for(int t = 0; t < kW / 4; ++t)
          if(h + t < kW - 1) s[h + t] = fma(-u[t], x, s[h + t + 1]);
      }
      T[o + lane][o + k] = x;
    }
  }
}

// A 16 x 8 tile per warp of the 32 x 32 product A B.
HPLB_DEV void product32(double (&acc)[4], const double* A, const double* B) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  const double* a = A + ((warp & 1) * 16 + g) * kTp + t4;
  const double* b = B + t4 * kTp + (warp >> 1) * 8 + g;
#pragma unroll
  for(int e = 0; e < 4; ++e) acc[e] = 0.0;
#pragma unroll
  for(int k = 0; k < 32; k += 8) {
    const double af[4] = {a[k], a[8 * kTp + k], a[k + 4], a[8 * kTp + k + 4]};
    const double bf[2] = {b[k * kTp], b[(k + 4) * kTp]};
    dmma(acc, af, bf);
  }
}

// In-place inverse of the upper triangular kTb x kTb block T (the identity from row and
// column kb on): both 32 x 32 halves by a warp each, joined (of a unit-lower L's
// transpose left as they are) by X12 = -(X11 U12) X22, W (32 rows) between.  Every panel of hplb_getrs waits for one of these, the transposed
// solve for two: kTb steps with two block barriers and a division each (invert_upper)
// take about 17 us longer (N = 1000, NB = 64, 32 right-hand sides, plain 721 us, now
// 419; transposed 2.16 ms, now 1.59).
template <bool UNIT>
HPLB_DEV void invert_upper_halves(double (*T)[kTp], double (*W)[kTp], int kb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(warp == 0) invert_upper32<UNIT>(T, 0, min(32, kb));
  if(warp == 1 && kb > 32) invert_upper32<UNIT>(T, 32, kb - 32);
  if(UNIT || kb <= 32) return;  // (U12 is 0)
  const int r = (warp & 1) * 16 + (lane >> 2), c = (warp >> 1) * 8 + 2 * (lane & 3);
  double    acc[4];
  __syncthreads();
  product32(acc, &T[0][0], &T[0][32]);
#pragma unroll
  for(int e = 0; e < 4; ++e) W[r + (e >> 1) * 8][c + (e & 1)] = acc[e];
  __syncthreads();
  product32(acc, &W[0][0], &T[32][32]);
#pragma unroll
  for(int e = 0; e < 4; ++e) T[r + (e >> 1) * 8][32 + c + (e & 1)] = -acc[e];
}

// Copies of the tile rows r0 .. r0 + kb, columns c0 .. c0 + kc of A into U
// (zeros outside), as one commit group.  VEC: 16-byte copies of row pairs (A
// 16-byte aligned, ld and r0 even); else 8-byte copies.
template <bool VEC>
HPLB_DEV void stage_tile(double (*U)[kTp], const double* A, int64_t ld, int r0, int kb, int c0,
                         int kc) {
  if(VEC) {
    for(int id = threadIdx.x; id < kTb * kTb / 2; id += kTrsvThreads) {
      const int     c = id / (kTb / 2), p = id % (kTb / 2);
      const int     rows = c < kc ? min(2, max(0, kb - 2 * p)) : 0;
      const double* src  = rows ? A + (size_t)(r0 + 2 * p) + (size_t)(c0 + c) * (size_t)ld : A;
      cp_async16(&U[c][2 * p], src, 8 * rows);
    }
  } else {
    for(int id = threadIdx.x; id < kTb * kTb; id += kTrsvThreads) {
      const int  c = id / kTb, r = id % kTb;
      const bool in = c < kc && r < kb;
      cp_async8(&U[c][r], in ? A + (size_t)(r0 + r) + (size_t)(c0 + c) * (size_t)ld : A,
                in ? 8 : 0);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <bool LOWER, bool VEC>
__global__ void __launch_bounds__(kTrsvThreads, 2)
trsm_kernel(const double* __restrict__ A, int64_t ld, int ns, int rows, int nrhs, const double* Y,
            int64_t ldy, double* X, int64_t ldx, int* flags, int* status) {
  extern __shared__ __align__(16) unsigned char trsm_smem_raw[];
  TrsmSmem& S    = *reinterpret_cast<TrsmSmem*>(trsm_smem_raw);
  const int nblk = (ns + kTb - 1) / kTb, ng = (nrhs + kNg - 1) / kNg;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = lane >> 2, t4 = lane & 3;
  if(t == 0) S.ticket = atomicAdd(flags + nblk * ng, 1);
  __syncthreads();
  const int  grp = S.ticket % ng, blk = S.ticket / ng;
  const bool solve = blk < nblk;  // false: rows below the lower triangle
  const int  bi = LOWER ? blk : nblk - 1 - blk;
  const int  r0 = solve ? bi * kTb : ns + (blk - nblk) * kTb;
  const int  kb = min(kTb, (solve ? ns : rows) - r0);
  const int  nt = min(blk, nblk);  // tiles of the row panel
  const int  q0 = grp * kNg, nq = min(kNg, nrhs - q0);
  const int  rt = (warp & 3) * 16, kh = (warp >> 2) * (kTb / 2);
  auto       tile = [&](int i) { return LOWER ? i : nblk - 1 - i; };
  if(nt > 0) stage_tile<VEC>(S.U[0], A, ld, r0, kb, tile(0) * kTb, min(kTb, ns - tile(0) * kTb));

  if(solve) {  // the diagonal block (identity beyond kb), inverted
    for(int idx = t; idx < kTb * kTb; idx += kTrsvThreads) {
      const int c = idx / kTb, r = idx % kTb;
      double    v = (r == c) ? 1.0 : 0.0;
      if(r < kb && c < kb) {
        if(LOWER)
          v = r > c ? A[(size_t)(r0 + r) + (size_t)(r0 + c) * (size_t)ld] : v;
        else
          v = r <= c ? A[(size_t)(r0 + r) + (size_t)(r0 + c) * (size_t)ld] : 0.0;
      }
      if(LOWER)
        S.T[c][r] = v;
      else
        S.T[r][c] = v;
    }
    __syncthreads();
    invert_upper_halves<LOWER>(S.T, S.U[1], kb);  // U[1]: no tile is on its way to it yet
  }
  double y[4];  // this warp's entries of y (the warps of the first half)
#pragma unroll
  for(int e = 0; e < 4; ++e) {
    const int r = rt + g + (e >> 1) * 8, q = 2 * t4 + (e & 1);
    y[e] = (kh == 0 && r < kb && q < nq) ? Y[(size_t)(r0 + r) + (size_t)(q0 + q) * (size_t)ldy]
                                         : 0.0;
  }

  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  bool   alive  = true;
  for(int i = 0; i < nt; ++i) {
    const int b = i & 1, j = tile(i), kc = min(kTb, ns - j * kTb);
    if(alive) alive = wait_flag(flags + j * ng + grp, status, kTrsmSite);
#pragma unroll
    for(int h = 0; h < kTb * kNg / kTrsvThreads; ++h) {
      const int r = t % kTb, q = t / kTb + h * (kTrsvThreads / kTb);
      S.X[b][q][r] = (r < kc && q < nq)
                         ? __ldcg(X + (size_t)(j * kTb + r) + (size_t)(q0 + q) * (size_t)ldx)
                         : 0.0;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");  // this thread's copies of the tile
    __syncthreads();  // everyone's, and the other buffers are no longer read
    if(i + 1 < nt)
      stage_tile<VEC>(S.U[b ^ 1], A, ld, r0, kb, tile(i + 1) * kTb,
                      min(kTb, ns - tile(i + 1) * kTb));
#pragma unroll
    for(int s = 0; s < kTb / 2; s += 8) {
      const int    k    = kh + s + t4;
      const double a[4] = {S.U[b][k][rt + g], S.U[b][k][rt + g + 8], S.U[b][k + 4][rt + g],
                           S.U[b][k + 4][rt + g + 8]};
      const double x[2] = {S.X[b][g][k], S.X[b][g][k + 4]};
      dmma(acc, a, x);
    }
  }

  // y - sum: the second half's part through shared memory.
  bool bad = false;  // a value that 0 does not take out of a product
  __syncthreads();
  if(kh != 0)
#pragma unroll
    for(int e = 0; e < 4; ++e) S.X[1][2 * t4 + (e & 1)][rt + g + (e >> 1) * 8] = acc[e];
  __syncthreads();
  if(kh == 0) {
#pragma unroll
    for(int e = 0; e < 4; ++e) {
      const int r = rt + g + (e >> 1) * 8, q = 2 * t4 + (e & 1);
      y[e] -= acc[e] + S.X[1][q][r];
      S.X[0][q][r] = r < kb ? y[e] : 0.0;
      bad |= r < kb && !isfinite(y[e]);
    }
  }
  if(!solve) {
    if(kh == 0)
#pragma unroll
      for(int e = 0; e < 4; ++e) {
        const int r = rt + g + (e >> 1) * 8, q = 2 * t4 + (e & 1);
        if(r < kb && q < nq) X[(size_t)(r0 + r) + (size_t)(q0 + q) * (size_t)ldx] = y[e];
      }
    return;
  }
  if(LOWER) {
    // x = L^-1 (y - sum) by the halves of 32 rows, each with its own inverse: the
    // inverse of all 64 would multiply the first half's rounding by the second's
    // (|A^T x - b| 1.15 to 1.23 times as large, N = 128 to 700, NB = 64 to 256).
    auto times = [&](double (&x)[4], const double (*v)[kTp], int k0) {
#pragma unroll
      for(int s = 0; s < 32; s += 8) {
        const int    k = k0 + s + t4, r = rt + g;
        const double a[4] = {S.T[k][r], S.T[k][r + 8], S.T[k + 4][r], S.T[k + 4][r + 8]};
        const double w[2] = {v[g][k], v[g][k + 4]};
        dmma(x, a, w);
      }
    };
    const bool top = kh == 0 && rt < 32, bottom = kh == 0 && rt >= 32;
    double     x[4] = {0.0, 0.0, 0.0, 0.0}, z[4] = {0.0, 0.0, 0.0, 0.0};
    __syncthreads();
    if(top) {
      times(x, S.X[0], 0);
#pragma unroll
      for(int e = 0; e < 4; ++e) S.X[1][2 * t4 + (e & 1)][rt + g + (e >> 1) * 8] = x[e];
    }
    if(kb > 32) {
      __syncthreads();
      if(bottom) {
        times(z, S.X[1], 0);
#pragma unroll
        for(int e = 0; e < 4; ++e) {
          const int r = rt + g + (e >> 1) * 8;
          S.X[0][2 * t4 + (e & 1)][r] = r < kb ? y[e] - z[e] : 0.0;
        }
      }
      __syncthreads();
      if(bottom) times(x, S.X[0], 32);
    }
    if(kh == 0) {
#pragma unroll
      for(int e = 0; e < 4; ++e) {
        const int r = rt + g + (e >> 1) * 8, q = 2 * t4 + (e & 1);
        if(r < kb && q < nq) X[(size_t)(r0 + r) + (size_t)(q0 + q) * (size_t)ldx] = x[e];
      }
      __threadfence();
    }
  } else if(__syncthreads_or(bad)) {
    // x = U^-1 (y - sum) over the triangle alone: an infinity or NaN in y reaches only
    // the rows that depend on it, which the full products below would not keep.
    if(kh == 0) {
      for(int e = 0; e < 4; ++e) {
        const int r = rt + g + (e >> 1) * 8, q = 2 * t4 + (e & 1);
        if(r >= kb || q >= nq) continue;
        double x = 0.0;
        for(int k = r; k < kb; ++k) x = fma(S.T[r][k], S.X[0][q][k], x);
        X[(size_t)(r0 + r) + (size_t)(q0 + q) * (size_t)ldx] = x;
      }
      __threadfence();
    }
  } else if(kh == 0) {  // x = U^-1 (y - sum), two chains
    double x0[4] = {0.0, 0.0, 0.0, 0.0}, x1[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for(int s = 0; s < kTb; s += 8) {
      const int    k = s + t4, r = rt + g;
      const double a[4] = {S.T[r][k], S.T[r + 8][k], S.T[r][k + 4], S.T[r + 8][k + 4]};
      const double v[2] = {S.X[0][g][k], S.X[0][g][k + 4]};
      if(s & 8)
        dmma(x1, a, v);
      else
        dmma(x0, a, v);
    }
#pragma unroll
    for(int e = 0; e < 4; ++e) {
      const int r = rt + g + (e >> 1) * 8, q = 2 * t4 + (e & 1);
      if(r < kb && q < nq) X[(size_t)(r0 + r) + (size_t)(q0 + q) * (size_t)ldx] = x0[e] + x1[e];
    }
    __threadfence();
  }
  __syncthreads();
  if(t == 0) st_release_gpu(flags + bi * ng + grp, 1);
}

// z[r] += sum_c U[r, c] x[c] for r < m, c < k: a thread per row (coalesced
// down each column), x staged in shared memory in chunks of 1024.
__global__ void __launch_bounds__(256)
gemv_acc_kernel(int m, int k, const double* __restrict__ U, int64_t ld,
                const double* __restrict__ x, double* __restrict__ z) {
  __shared__ double xs[1024];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  double    acc = 0.0;
  for(int c0 = 0; c0 < k; c0 += 1024) {
    const int kc = min(1024, k - c0);
    __syncthreads();
    for(int i = threadIdx.x; i < kc; i += blockDim.x) xs[i] = x[c0 + i];
    __syncthreads();
    if(r < m) {
      const double* u = U + (size_t)r + (size_t)c0 * (size_t)ld;
#pragma unroll 8
      for(int c = 0; c < kc; ++c) acc = fma(u[(size_t)c * (size_t)ld], xs[c], acc);
    }
  }
  if(r < m) z[r] += acc;
}

__global__ void vsub_kernel(int n, const double* __restrict__ y, const double* __restrict__ s,
                            double* __restrict__ r) {
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    r[i] = y[i] - s[i];
}

}  // namespace

size_t trsv_flag_ints(int n) { return (size_t)(n + kTb - 1) / kTb * (kNr / kNg) + 1; }

cudaError_t launch_gemv_acc(int m, int k, const double* U, int64_t ld, const double* x,
                            double* z, cudaStream_t stream) {
  if(m <= 0 || k <= 0) return cudaSuccess;
  gemv_acc_kernel<<<(m + 255) / 256, 256, 0, stream>>>(m, k, U, ld, x, z);
  return cudaGetLastError();
}

cudaError_t launch_vsub(int n, const double* y, const double* s, double* r, cudaStream_t stream) {
  if(n <= 0) return cudaSuccess;
  vsub_kernel<<<(n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024, 256, 0, stream>>>(n, y, s, r);
  return cudaGetLastError();
}

cudaError_t launch_trsv(const double* A, int64_t ld, int n, double* X, int* flags, int* status,
                        cudaStream_t stream, int* launches) {
  return launch_trsv_y(A, ld, n, A + (size_t)n * (size_t)ld, X, flags, status, stream, launches);
}

cudaError_t launch_trsv_y(const double* A, int64_t ld, int n, const double* Y, double* X,
                          int* flags, int* status, cudaStream_t stream, int* launches) {
  if(n <= 0) return cudaSuccess;
  const int   nblk = (n + kTb - 1) / kTb;
  cudaError_t e    = cudaMemsetAsync(flags, 0, trsv_flag_ints(n) * sizeof(int), stream);
  if(e != cudaSuccess) return e;
  const bool vec = (reinterpret_cast<uintptr_t>(A) % 16 == 0) && (ld % 2 == 0);
  if(vec)
    trsv_kernel<true><<<nblk, kTrsvThreads, 0, stream>>>(A, ld, n, Y, X, flags, status);
  else
    trsv_kernel<false><<<nblk, kTrsvThreads, 0, stream>>>(A, ld, n, Y, X, flags, status);
  ++*launches;
  return cudaGetLastError();
}

namespace {

template <bool LOWER, bool VEC>
cudaError_t launch_trsm_form(const double* A, int64_t ld, int ns, int rows, int nrhs,
                             const double* Y, int64_t ldy, double* X, int64_t ldx, int* flags,
                             int* status, cudaStream_t stream) {
  static bool attr = false;
  if(!attr) {
    const cudaError_t e = cudaFuncSetAttribute(
        trsm_kernel<LOWER, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrsmSmem));
    if(e != cudaSuccess) return e;
    attr = true;
  }
  const int blocks = (ns + kTb - 1) / kTb + (rows - ns + kTb - 1) / kTb;
  trsm_kernel<LOWER, VEC><<<blocks * ((nrhs + kNg - 1) / kNg), kTrsvThreads, sizeof(TrsmSmem),
                            stream>>>(A, ld, ns, rows, nrhs, Y, ldy, X, ldx, flags, status);
  return cudaGetLastError();
}

// One launch per kNr right-hand sides.  Upper: their flags zeroed here; lower: flags of
// their own (trsv_flag_ints(ns) each), zeroed by the caller for many solves at once.
template <bool LOWER>
cudaError_t launch_trsm_blocks(const double* A, int64_t ld, int ns, int rows, int nrhs,
                               const double* Y, int64_t ldy, double* X, int64_t ldx, int* flags,
                               int* status, cudaStream_t stream, int* launches) {
  if(ns <= 0 || nrhs <= 0) return cudaSuccess;
  const bool vec = reinterpret_cast<uintptr_t>(A) % 16 == 0 && ld % 2 == 0 &&
                   (rows == ns || ns % 2 == 0);
  for(int q = 0; q < nrhs; q += kNr) {
    const int   nr = std::min(kNr, nrhs - q);
    cudaError_t e  = cudaSuccess;
    if(!LOWER) e = cudaMemsetAsync(flags, 0, trsv_flag_ints(ns) * sizeof(int), stream);
    if(e != cudaSuccess) return e;
    const double* Yq = Y + (size_t)q * (size_t)ldy;
    double*       Xq = X + (size_t)q * (size_t)ldx;
    e = vec ? launch_trsm_form<LOWER, true>(A, ld, ns, rows, nr, Yq, ldy, Xq, ldx, flags, status,
                                            stream)
            : launch_trsm_form<LOWER, false>(A, ld, ns, rows, nr, Yq, ldy, Xq, ldx, flags, status,
                                             stream);
    if(e != cudaSuccess) return e;
    ++*launches;
    if(LOWER) flags += trsv_flag_ints(ns);
  }
  return cudaSuccess;
}

}  // namespace

cudaError_t launch_trsm_upper(const double* A, int64_t ld, int n, int nrhs, const double* Y,
                              int64_t ldy, double* X, int64_t ldx, int* flags, int* status,
                              cudaStream_t stream, int* launches) {
  return launch_trsm_blocks<false>(A, ld, n, n, nrhs, Y, ldy, X, ldx, flags, status, stream,
                                   launches);
}

cudaError_t launch_trsm_lower(const double* L, int64_t ldl, int ns, int rows, int nrhs, double* X,
                              int64_t ldx, int* flags, int* status, cudaStream_t stream,
                              int* launches) {
  return launch_trsm_blocks<true>(L, ldl, ns, rows, nrhs, X, ldx, X, ldx, flags, status, stream,
                                  launches);
}

}  // namespace hplb
