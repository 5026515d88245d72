// A whole panel in a few launches: the recursive factorisation of an M x NB panel
// (HPL_pdrpanrlT / HPL_pdrpanllT / HPL_pdrpancrT, src/pfact/HPL_pdrpanrlT.cpp:74-160),
// its interchanges, the row map and L11^-1, on ONE thread-block cluster of up
// to 16 CTAs that walks a list of operations made by the host's recursion.
//
// What bounds it: a panel is a chain of NB pivot searches over all its rows,
// so it is latency-bound, and beside the trailing update it also waits for SMs
// at every launch.  Hence one launch for a whole run of the recursion's
// operations (N = 16384, NB = 512: 5 to 8 launches per panel instead of 46), the
// cluster's SMs held from start to end, and a column step built around one
// one-way message:
//   * the leaf's rows live in registers (RPT rows of W columns per thread), the
//     current column always in register 0: the update writes each column one
//     register down, so one short loop body serves every column (eight unrolled
//     bodies spent a third of their time fetching instructions); finished
//     columns wait in shared memory;
//   * rows never move while the leaf is factored: each thread tracks the
//     position its row has under the interchanges and writes it there at the
//     end, so no diagonal row is exchanged;
//   * every CTA pushes its candidate row (the columns from the current one on,
//     and its position) into every CTA's shared memory with st.async, whose
//     arrival completes the receiver's mbarrier: no cluster barrier and no
//     remote read per column, the search for the winner is local;
//   * only column k + 1 is updated before the next candidate is published; the
//     remaining columns are updated while the messages travel (the published
//     row's share is done by the publishing warp, two columns per lane).
// Between the leaves, the recursion's U12 = L11^-1 A12 (a warp per column,
// blocked substitution with inverted 32 x 32 diagonal blocks) and
// A22 -= L21 U12 (DMMA m16n8k8 in FP64, FFMA in FP32, a share of the rows per
// CTA, cp.async-staged), separated by cluster barriers.
//
// Measured on one B200: a column step 2.7 us (one launch per leaf, 4096 rows)
// -> 1.2 us, of which about 0.45 us is staging and sending the candidate, 0.3 us
// its way to the other CTAs and the rest the search and the updates' latency; a
// panel of 4096 x 256 about 1.1 ms -> 0.55 ms, of 8192 x 512 in FP32 3.7 -> 1.3 ms.
//
// Every operation is the one of the launch-per-step path (panel.cu, dgemm_tma.cu,
// sgemm.cu) in the same order per element, so both give identical bits; leaves
// too tall for W = 32 are split into narrower ones.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "panel_msgs.h"

namespace hplb {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps   = kThreads / 32;
constexpr int kMaxG    = 16;  // CTAs per cluster at most (non-portable above 8)
constexpr int kTri     = 32;  // diagonal block size of the blocked substitution
constexpr int kMaxOps  = 400;
constexpr int kMaxNb   = 1024;

// off, jb, c2, n2 relative to the panel's first row / column:
//   n2 > 0           U12 and A22 of a node: L11 at (off, off), jb wide, applied
//                    to columns [c2, c2 + n2) (rows below off + jb included)
//   n2 = 0, c2 = 0   leaf of jb columns at (off, off)
//   n2 = 0, c2 = 1   inverses of the 32 x 32 diagonal blocks of [off, off + jb)
// The inverses of a node at off are kept from block off / 32 on.
// kSplit in n2: U12 only; the product is a launch of its own over all SMs after
// this launch.
constexpr int kSplit = 0x8000;
struct Op {
  unsigned short off, jb, c2, n2;
};

template <typename T>
struct FusedParams {
  T*      A;
  int64_t ld;
  int     r0, c0, n, jb;  // panel rows [r0, n), columns [c0, c0 + jb)
  int*    ipiv;           // ipiv[c] = global pivot row of column c
  int*    status;
  T*      dinv;           // ((jb + 31) / 32 + 1) blocks of 32 x 32
  T*      linv;           // jb x jb, or null: no row map and L11^-1
  int*    permU;          // 2 jb
  int     nops;
  Op      ops[kMaxOps];
};

HPLB_DEV uint32_t s_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
HPLB_DEV uint32_t peer_addr(uint32_t a, unsigned rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
HPLB_DEV unsigned cta_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
HPLB_DEV unsigned cta_count() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Orders every CTA's global and shared memory accesses before and after it.
HPLB_DEV void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
HPLB_DEV void mbar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_addr(b)),
               "r"(bytes)
               : "memory");
}
HPLB_DEV bool mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(s_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: on expiry the site goes to the status word and every later
// wait of the CTA returns at once; the kernel then runs to its end on what it
// has (all positions are range-checked), so no peer is left alone, and arms and
// sends nothing more (panel_msgs.h).  True once the phase has completed.
HPLB_DEV bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort, int* status) {
  if(mbar_try(b, parity)) return true;
  const unsigned long long t0 = globaltimer();
  while(!mbar_try(b, parity)) {
    if(*abort) return false;
    if(globaltimer() - t0 > kWaitBudgetNs) {
      atomicCAS(status + ST_TIMEOUT, 0, 51);
      *abort = 1;
      return false;
    }
  }
  return true;
}
// 16 bytes into a peer's shared memory, counted by its barrier on arrival.
HPLB_DEV void push16(uint32_t dst, const double (&v)[2], uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::
          "r"(dst), "l"(__double_as_longlong(v[0])), "l"(__double_as_longlong(v[1])), "r"(bar)
      : "memory");
}
HPLB_DEV void push16(uint32_t dst, const float (&v)[4], uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4},"
      " [%5];" ::"r"(dst),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
      "r"(__float_as_uint(v[3])), "r"(bar)
      : "memory");
}

// Pivot order as an integer: 2 |v| + 1 of a candidate's bits, 0 for none (a NaN
// ranks above every number, as in warp_argmax).
HPLB_DEV unsigned long long key_of(double v) {
  return ((unsigned long long)__double_as_longlong(v) << 1) | 1ull;
}
HPLB_DEV unsigned key_of(float v) { return (__float_as_uint(v) << 1) | 1u; }

// The lane holding the largest key, the lowest pos among equal keys; -1 if
// every key is 0.  One reduction and one vote unless high words tie.
HPLB_DEV int warp_best(unsigned long long key, int pos) {
  const unsigned hi = (unsigned)(key >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  unsigned       b  = __ballot_sync(0xffffffffu, hi == mh);
  if((b & (b - 1)) != 0 || mh == 0) {
    bool           c  = hi == mh && key != 0;
    const unsigned ml = __reduce_max_sync(0xffffffffu, c ? (unsigned)key : 0u);
    c                 = c && (unsigned)key == ml;
    const unsigned mp = __reduce_min_sync(0xffffffffu, c ? (unsigned)pos : 0xffffffffu);
    b                 = __ballot_sync(0xffffffffu, c && (unsigned)pos == mp);
  }
  return __ffs(b) - 1;
}
HPLB_DEV int warp_best(unsigned key, int pos) {
  const unsigned m = __reduce_max_sync(0xffffffffu, key);
  if(m == 0) return -1;
  bool     c = key == m;
  unsigned b = __ballot_sync(0xffffffffu, c);
  if(b & (b - 1)) {
    const unsigned p  = c ? (unsigned)pos : 0xffffffffu;
    const unsigned mp = __reduce_min_sync(0xffffffffu, p);
    b                 = __ballot_sync(0xffffffffu, c && p == mp);
  }
  return __ffs(b) - 1;
}

HPLB_DEV double recip(double v) { return __drcp_rn(v); }
HPLB_DEV float  recip(float v) { return __frcp_rn(v); }
HPLB_DEV double fma_(double a, double b, double c) { return fma(a, b, c); }
HPLB_DEV float  fma_(float a, float b, float c) { return fmaf(a, b, c); }

// x / piv, correctly rounded: from r = RN(1 / piv), q = x r is within two ulps;
// one residual correction makes it faithful and, by Markstein's theorem (IBM
// J. Res. Dev. 34, 1990: a faithful quotient corrected with the correctly
// rounded reciprocal is correctly rounded), a second one exact to the last
// bit.  Five dependent operations with the reciprocal shared by the column
// instead of a division per row.  Only for operands whose exponents keep every
// intermediate exact (exponent_safe); the rest divide.
template <typename T>
HPLB_DEV T quotient(T x, T piv, T r) {
  T q = x * r;
  T e = fma_(-q, piv, x);
  q   = fma_(e, r, q);
  e   = fma_(-q, piv, x);
  return fma_(e, r, q);
}
// Out of line: its code stays out of the column loop, which lives off the
// instruction cache.
template <typename T>
__device__ __noinline__ T divide(T x, T piv) {
  return x / piv;
}
// |v| in [2^-400, 2^500) (FP64), [2^-60, 2^60) (FP32).
HPLB_DEV bool exponent_safe(double v) {
  const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
  return h - ((1023u - 400u) << 20) < (900u << 20);
}
HPLB_DEV bool exponent_safe(float v) {
  const unsigned h = __float_as_uint(v) & 0x7fffffffu;
  return h - ((127u - 60u) << 23) < (120u << 23);
}

// A row's registers from FROM on to shared memory, 16 bytes at a time (the last
// value repeats).
template <int FROM, int N>
HPLB_DEV void store_row(double* s, const double (&v)[N]) {
#pragma unroll
  for(int i = 0; i < N; i += 2)
    *reinterpret_cast<double2*>(s + i) = make_double2(v[i + FROM], v[i + 1 + FROM < N ? i + 1 + FROM : N - 1]);
}
template <int FROM, int N>
HPLB_DEV void store_row(float* s, const float (&v)[N]) {
#pragma unroll
  for(int i = 0; i < N; i += 4)
    *reinterpret_cast<float4*>(s + i) =
        make_float4(v[i + FROM], v[i + 1 + FROM], v[i + 2 + FROM],
                    v[i + 3 + FROM < N ? i + 3 + FROM : N - 1]);
}
HPLB_DEV void load8(double (&v)[8], const double* s) {
#pragma unroll
  for(int i = 0; i < 8; i += 2) {
    const double2 t = *reinterpret_cast<const double2*>(s + i);
    v[i]            = t.x;
    v[i + 1]        = t.y;
  }
}
HPLB_DEV void load8(float (&v)[8], const float* s) {
#pragma unroll
  for(int i = 0; i < 8; i += 4) {
    const float4 t = *reinterpret_cast<const float4*>(s + i);
    v[i]           = t.x;
    v[i + 1]       = t.y;
    v[i + 2]       = t.z;
    v[i + 3]       = t.w;
  }
}

constexpr int kTopPitch = kTri + 1;

// Static shared memory of the panel kernel.
template <typename T, int W>
struct Shared {
  uint64_t           full[kBufs];
  unsigned long long key[2][kWarps];
  int                pos[2][kWarps];
  __align__(16) T    stage[W];  // the published row as its owner holds it, from its column on
  T                  lstage;    // and its multiplier of the last column
  int                pv[W];     // the leaf's pivots, relative to its first row
  int                src[kTri], dst[kTri];
  volatile int       abort;
  uint32_t           peer[kMaxG];            // offset of a CTA's shared memory in the cluster's window
  T                  top[kTri * kTopPitch];  // the leaf's pivot rows: U11 (L11 too in the last CTA)
};

// Dynamic shared memory while a leaf is factored: the messages, by buffer and
// sender, and the finished columns of this CTA's rows.
struct alignas(16) Cand {
  double    val;  // a candidate's entry of its column
  long long pos;  // and its position, -1: no candidate
};
template <typename T, int W, int RPT>
struct LeafMem {
  static constexpr int pitch = RPT * kThreads + 1;  // odd: a column of a row set, or a row, is free of conflicts
  T         row[kBufs][kMaxG][W];  // entry i < w - k: column k + i of the candidate row for column k
  Cand      cand[kBufs][kMaxG];
  T         done[W * pitch];
};

template <typename T, int W, int RPT>
struct Leaf {
  using Mem = LeafMem<T, W, RPT>;
  using Key = decltype(key_of(T(0)));
  const FusedParams<T>& P;
  Shared<T, W>&         S;
  Mem&                  M;
  unsigned              G, me;
  int                   warp, lane;
  int                   r0, w;
  unsigned              kc;  // columns done since the kernel started

  T   x[RPT][W];  // register i: column k + i of the thread's rows
  int pos[RPT];   // the rows' positions under the interchanges so far, -1: no row
  T   l[RPT];

  HPLB_DEV bool wait(int buf, uint32_t parity) {
    return mbar_wait(&S.full[buf], parity, &S.abort, P.status);
  }
  HPLB_DEV bool expired() const { return S.abort != 0; }
  HPLB_DEV void arm(int buf) { mbar_expect(&S.full[buf], G * (uint32_t)(W * sizeof(T) + 16)); }

  // The block's best candidate of column k1 (register FIRST ? 0 : 1) and its
  // publication by the warp that holds it.  Unless FIRST, the row's columns
  // beyond k1 still lack column k1 - 1's update (pivot row u) and get it here,
  // a lane per column; the columns before k1 come from their store.
  template <bool FIRST>
  HPLB_DEV void publish(int k1, const T* u) {
    constexpr int I  = FIRST ? 0 : 1;
    const int     d1 = r0 + k1;
    const bool    sends = may_send(*this);
    Key           key = 0;
    int           bp = -1, bq = 0;
#pragma unroll
    for(int q = 0; q < RPT; ++q) {
      const Key  kq = pos[q] >= d1 ? key_of(x[q][I]) : (Key)0;
      const bool up = kq > key || (kq == key && pos[q] < bp);
      key           = up ? kq : key;
      bp            = up ? pos[q] : bp;
      bq            = up ? q : bq;
    }
    const int wl  = max(warp_best(key, bp), 0);
    const int par = kc & 1;
    if(lane == wl) {
      S.key[par][warp] = key;
      S.pos[par][warp] = bp;
    }
    __syncthreads();
    Key ck = 0;
    int cp = -1;
    if(lane < kWarps) {
      ck = (Key)S.key[par][lane];
      cp = S.pos[par][lane];
    }
    const int ww = warp_best(ck, cp);
    if(warp != max(ww, 0) || !sends) return;
    if(lane == wl) {
#pragma unroll
      for(int q = 0; q < RPT; ++q)
        if(q == bq) {
          store_row<I>(S.stage, x[q]);
          S.lstage = l[q];
        }
    }
    const int p1  = ww < 0 ? -1 : __shfl_sync(0xffffffffu, bp, wl);
    const int buf = kc & (kBufs - 1);
    // A lane's 16 bytes of the row: entries i0 .., columns k1 + i0 ...
    constexpr int V = 16 / (int)sizeof(T), per_row = W / V, at_once = 32 / per_row;
    const int     i0 = lane % per_row * V, sub = lane / per_row;
    uint32_t      to[kMaxG / at_once];
#pragma unroll
    for(int t = 0; t < kMaxG / at_once; ++t) to[t] = S.peer[t * at_once + sub];
    __syncwarp();
    T v[V];
#pragma unroll
    for(int j = 0; j < V; ++j) {
      v[j] = S.stage[i0 + j];
      if(!FIRST) {
        const T f = fma_(-S.lstage, u[(i0 + j + 1) & (W - 1)], v[j]);
        v[j]      = i0 + j > 0 ? f : v[j];
      }
    }
    const uint32_t at = s_addr(&M.row[buf][me][i0]), bar = s_addr(&S.full[buf]);
#pragma unroll
    for(int t = 0; t < kMaxG / at_once; ++t)
      if(t * at_once + sub < (int)G) push16(at + to[t], v, bar + to[t]);
    if(lane < (int)G) {
      const uint32_t pl    = S.peer[lane];
      const double   cv[2] = {(double)S.stage[0], __longlong_as_double((long long)p1)};
      push16(s_addr(&M.cand[buf][me]) + pl, cv, bar + pl);
    }
    __syncwarp();
  }

  // Factor rows [r0, n) of columns [ca, ca + w) in place.
  HPLB_DEV void factor(int ca) {
    const int    rowsn = P.n - r0;
    const int    rpb   = ((rowsn + (int)G - 1) / (int)G + 31) / 32 * 32;
    const int    lo    = r0 + (int)me * rpb;
    const size_t ld    = (size_t)P.ld;
    T*           A     = P.A + (size_t)ca * ld;
#pragma unroll
    for(int q = 0; q < RPT; ++q) {
      const int  t  = (int)threadIdx.x + q * kThreads;
      const bool in = t < rpb && lo + t < P.n;
      pos[q]        = in ? lo + t : -1;
      l[q]          = (T)0;
#pragma unroll
      for(int c = 0; c < W; ++c)
        x[q][c] = (in && c < w) ? __ldcg(A + (size_t)pos[q] + (size_t)c * ld) : (T)0;
    }
    publish<true>(0, nullptr);
#pragma unroll 1
    for(int k = 0; k < w; ++k) {
      const int d   = r0 + k;
      const int buf = kc & (kBufs - 1);
      bool      odd = false;  // a quotient that needs the division
#pragma unroll
      for(int q = 0; q < RPT; ++q) odd |= pos[q] >= d && !exponent_safe(x[q][0]);
      odd = __any_sync(0xffffffffu, odd);
      const bool arrived = await_column(*this, kc);
      // The winner among the CTAs' candidates; each lane has the reciprocal of
      // its candidate under way while the search runs.
      Key  ck = 0;
      int  cp = -1;
      T    cv = (T)1;
      if(lane < (int)G) {
        const Cand c = M.cand[buf][lane];
        cv = (T)c.val;
        cp = (int)c.pos;
        ck = cp >= d ? key_of(cv) : (Key)0;
      }
      const T    cr  = recip(cv);
      const bool div = __any_sync(0xffffffffu, ck != 0 && !exponent_safe(cv)) || odd;
      const int  win = max(warp_best(ck, cp), 0);
      const T*   u   = M.row[buf][win];
      const T    piv = u[0], u1 = u[1];
      const T    r   = __shfl_sync(0xffffffffu, cr, win);
      int        p   = __shfl_sync(0xffffffffu, cp, win);
      if(p < d || p >= P.n) p = d;  // only after an expired wait
#pragma unroll
      for(int q = 0; q < RPT; ++q) {
        l[q]   = quotient(x[q][0], piv, r);
        pos[q] = pos[q] == p ? d : (pos[q] == d ? p : pos[q]);
      }
      if(div) {
#pragma unroll
        for(int q = 0; q < RPT; ++q) l[q] = divide(x[q][0], piv);
      }
#pragma unroll
      for(int q = 0; q < RPT; ++q) {
        if(pos[q] > d) M.done[k * Mem::pitch + threadIdx.x + q * kThreads] = l[q];
        x[q][1] = fma_(-l[q], u1, x[q][1]);
      }
      const unsigned kd = kc++;
      if(k + 1 < w) publish<false>(k + 1, u);
      // The other columns, while the candidates travel; the update also moves
      // every column one register down.  Rows that are pivot rows by now, and
      // registers past the leaf's last column, take values nobody reads.
#pragma unroll
      for(int q = 0; q < RPT; ++q) x[q][0] = x[q][1];
#pragma unroll
      for(int h = 0; h < (W + 15) / 16; ++h)
        if(16 * h + k < w) {
#pragma unroll
          for(int i0 = 16 * h; i0 < 16 * h + 16 && i0 < W; i0 += 8) {
            T uc[8];
            load8(uc, u + i0);
#pragma unroll
            for(int i = 0; i < 8; ++i)
              if(i0 + i >= 2)
#pragma unroll
                for(int q = 0; q < RPT; ++q)
                  x[q][i0 + i - 1] = fma_(-l[q], uc[i], x[q][i0 + i]);
          }
        }
      if(warp == kWarps - 1) {
        if(lane >= k && lane < W) S.top[k * kTopPitch + lane] = u[lane - k];
        if(lane == 0) {
          rearm(*this, kd, arrived);
          S.pv[k] = p - r0;
          if(me == 0) {
            P.ipiv[ca + k] = p;
            if(piv == (T)0) record_info(P.status, ca + k + 1);
          }
        }
      }
    }
    __syncthreads();
    // Rows to their positions: columns before a row's pivot column (all w of a
    // row that is no pivot row) from its owner's store; the rest of the pivot
    // rows, known to every CTA, by the first one.
#pragma unroll
    for(int q = 0; q < RPT; ++q)
      if(pos[q] >= r0) {
        const T*  f  = M.done + threadIdx.x + q * kThreads;
        const int nc = min(w, pos[q] - r0);
        for(int c = 0; c < nc; ++c) A[(size_t)pos[q] + (size_t)c * ld] = f[c * Mem::pitch];
      }
    if(me == 0)
      for(int c = warp; c < w; c += kWarps)
        if(lane <= c) A[(size_t)(r0 + lane) + (size_t)c * ld] = S.top[lane * kTopPitch + c];
  }
};

// Column `lane` of the inverse of the unit-lower w x w block whose rows are at
// L (row stride kTopPitch), padded with the identity to 32 x 32, into out: per
// step the next row's value is final and the rows below move one register down.
template <typename T>
HPLB_DEV void invert_block(const T* L, int w, T* out) {
  const int lane = threadIdx.x & 31;
  T         s[kTri];
#pragma unroll
  for(int i = 0; i < kTri; ++i) s[i] = i == lane ? (T)1 : (T)0;
  // Two halves, the second with half of the rows left; the loads of a step all
  // issue before its updates.  Rows beyond w (and 32) update nothing.
#pragma unroll
  for(int half = 0; half < 2; ++half) {
    constexpr int kHalf = kTri / 2;
#pragma unroll 1
    for(int k = half * kHalf; k < (half + 1) * kHalf; ++k) {
      const T* col = L + (size_t)k * kTopPitch + k;
      T        lv[kTri];
#pragma unroll
      for(int i = 1; i < kTri; ++i)
        if(half == 0 || i < kHalf) lv[i] = k + i < w ? col[i * kTopPitch] : (T)0;
      out[lane * kTri + k] = s[0];
      const T xk = s[0];
#pragma unroll
      for(int i = 1; i < kTri; ++i)
        if(half == 0 || i < kHalf) s[i - 1] = fma_(-lv[i], xk, s[i]);
    }
  }
}

// The leaf's w interchanges (S.pv) on the panel's columns outside the leaf, a
// warp per column, lane = row of the leaf's top block; the last warp of the
// cluster inverts the leaf's diagonal block meanwhile.
template <typename T, int W>
HPLB_DEV void leaf_finish(const FusedParams<T>& P, Shared<T, W>& S, unsigned G, unsigned me,
                          int off, int w, T* dinv) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int id = (int)me * kWarps + warp, last = (int)G * kWarps - 1;
  if((int)threadIdx.x < 2 * w) {
    // Half of the threads trace where a top row's value comes from, half where
    // the old row goes.
    const bool fwd = (int)threadIdx.x >= w;
    const int  x   = fwd ? (int)threadIdx.x - w : (int)threadIdx.x;
    int        at  = x;
    for(int t = 0; t < w; ++t) {
      const int i  = fwd ? t : w - 1 - t;
      const int pp = S.pv[i];
      at           = (at == i) ? pp : (at == pp ? i : at);
    }
    if(fwd)
      S.dst[x] = at >= w ? at : -1;
    else
      S.src[x] = at;
  }
  __syncthreads();
  if(id == last) {
    const T* a = P.A + (size_t)(P.r0 + off) + (size_t)(P.c0 + off) * (size_t)P.ld;
#pragma unroll 8
    for(int c = 0; c < w; ++c)
      if(lane < w) S.top[lane * kTopPitch + c] = __ldcg(a + lane + (size_t)c * (size_t)P.ld);
    __syncwarp();
    invert_block(S.top, w, dinv);
    return;
  }
  const int ncols = P.jb - w;
  const int src = lane < w ? S.src[lane] : 0, dst = lane < w ? S.dst[lane] : -1;
  constexpr int kAtOnce = 4;
  for(int j0 = id; j0 < ncols; j0 += kAtOnce * last) {
    T  v[kAtOnce], o[kAtOnce];
    T* a[kAtOnce];
#pragma unroll
    for(int t = 0; t < kAtOnce; ++t) {
      const int j   = j0 + t * last;
      const int col = P.c0 + (j < off ? j : j + w);
      a[t]          = P.A + (size_t)(P.r0 + off) + (size_t)col * (size_t)P.ld;
      v[t] = o[t] = (T)0;
      if(j < ncols && lane < w) {
        v[t] = __ldcg(a[t] + src);
        if(dst >= 0) o[t] = __ldcg(a[t] + lane);
      }
    }
    __syncwarp();  // every read of a column before any write to it
#pragma unroll
    for(int t = 0; t < kAtOnce; ++t)
      if(j0 + t * last < ncols) {
        if(dst >= 0) a[t][dst] = o[t];
        if(lane < w) a[t][lane] = v[t];
      }
    __syncwarp();
  }
}

// Inverses of the diagonal blocks of [off, off + jb), a warp per block.
template <typename T>
HPLB_DEV void invert_blocks(const FusedParams<T>& P, unsigned G, unsigned me, int off, int jb,
                            T* sm) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T*        L = sm + (size_t)warp * kTri * kTopPitch;
  for(int b = (int)me + (int)G * warp; b * kTri < jb; b += (int)G * kWarps) {
    const int w = min(kTri, jb - b * kTri);
    const T*  a = P.A + (size_t)(P.r0 + off + b * kTri) +
                 (size_t)(P.c0 + off + b * kTri) * (size_t)P.ld;
    T v[kTri];
#pragma unroll
    for(int c = 0; c < kTri; ++c)
      v[c] = (lane < w && c < w) ? __ldcg(a + lane + (size_t)c * (size_t)P.ld) : (T)0;
#pragma unroll
    for(int c = 0; c < kTri; ++c) L[lane * kTopPitch + c] = v[c];
    __syncwarp();
    invert_block(L, w, P.dinv + (size_t)(off / kTri + b) * kTri * kTri);
    __syncwarp();
  }
}

// X (jb x ncols at X, leading dimension ldx) <- L^-1 X, CP columns of a warp at
// a time.
template <typename T, int CP>
HPLB_DEV void trsm_cols(T* X, int64_t ldx, int jb, const T* L, int64_t ldl, const T* dinv,
                        int ncols, int first, int nw, T* sx) {
  const int    lane = threadIdx.x & 31;
  const int    lds  = jb + 1;
  const size_t ll   = (size_t)ldl;
  for(int c0 = first; c0 < ncols; c0 += CP * nw) {
#pragma unroll
    for(int q = 0; q < CP; ++q) {
      const int c = c0 + q * nw;
      for(int i = lane; i < jb; i += 32)
        sx[q * lds + i] = c < ncols ? __ldcg(X + (size_t)i + (size_t)c * (size_t)ldx) : (T)0;
    }
    __syncwarp();
    for(int b = 0; b * kTri < jb; ++b) {
      const int row0 = b * kTri, gr = row0 + lane;
      T         dv[kTri];
#pragma unroll
      for(int kk = 0; kk < kTri; ++kk)
        dv[kk] = __ldcg(dinv + (size_t)b * kTri * kTri + kk * kTri + lane);
      T acc[CP];
#pragma unroll
      for(int q = 0; q < CP; ++q) acc[q] = (T)0;
      if(gr < jb)
        for(int kk = 0; kk < row0; kk += 16) {
          T lv[16];
#pragma unroll
          for(int t = 0; t < 16; ++t) lv[t] = L[(size_t)gr + (size_t)(kk + t) * ll];
#pragma unroll
          for(int t = 0; t < 16; ++t)
#pragma unroll
            for(int q = 0; q < CP; ++q) acc[q] = fma_(lv[t], sx[q * lds + kk + t], acc[q]);
        }
#pragma unroll
      for(int q = 0; q < CP; ++q)
        if(gr < jb) sx[q * lds + gr] -= acc[q];
      __syncwarp();
#pragma unroll
      for(int q = 0; q < CP; ++q) acc[q] = (T)0;
#pragma unroll
      for(int kk = 0; kk < kTri; ++kk)
        if(row0 + kk < jb)
#pragma unroll
          for(int q = 0; q < CP; ++q) acc[q] = fma_(dv[kk], sx[q * lds + row0 + kk], acc[q]);
      __syncwarp();
#pragma unroll
      for(int q = 0; q < CP; ++q)
        if(gr < jb) sx[q * lds + gr] = acc[q];
      __syncwarp();
    }
#pragma unroll
    for(int q = 0; q < CP; ++q) {
      const int c = c0 + q * nw;
      if(c < ncols)
        for(int i = lane; i < jb; i += 32) X[(size_t)i + (size_t)c * (size_t)ldx] = sx[q * lds + i];
    }
    __syncwarp();
  }
}

template <typename T>
HPLB_DEV void trsm(T* X, int64_t ldx, int jb, const T* L, int64_t ldl, const T* dinv, int ncols,
                   unsigned G, unsigned me, T* sm) {
  const int warp = threadIdx.x >> 5;
  const int first = (int)me + (int)G * warp, nw = (int)G * kWarps;
  if(ncols > nw)
    trsm_cols<T, 2>(X, ldx, jb, L, ldl, dinv, ncols, first, nw, sm + (size_t)warp * 2 * (jb + 1));
  else
    trsm_cols<T, 1>(X, ldx, jb, L, ldl, dinv, ncols, first, nw, sm + (size_t)warp * (jb + 1));
}

HPLB_DEV void cp_async4(uint32_t s, const void* g, bool p) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(g), "r"(p ? 4 : 0)
               : "memory");
}
HPLB_DEV void cp_async8(uint32_t s, const void* g, bool p) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(g), "r"(p ? 8 : 0)
               : "memory");
}
HPLB_DEV void cp_async16(uint32_t s, const void* g, bool p) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(p ? 16 : 0)
               : "memory");
}
HPLB_DEV void cp_async1(uint32_t s, const double* g, bool p) { cp_async8(s, g, p); }
HPLB_DEV void cp_async1(uint32_t s, const float* g, bool p) { cp_async4(s, g, p); }
HPLB_DEV void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
HPLB_DEV void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

HPLB_DEV void dmma(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// C (m x n) -= A (m x k) B (k x n) by the cluster, each CTA a contiguous share
// of the rows.  The CTA's tile is (8 / WN) x 64 rows by 32 WN columns: the
// narrow updates of a panel's lower recursion levels (32 or 64 columns) keep
// all warps busy on rows.  k-slices of 16 through a cp.async ring; A in
// k-rows of pitch = 4 mod 16 doubles and B in columns of pitch 20, so every
// fragment load is free of bank conflicts.
constexpr int kBK = 16;
template <typename T>
struct GemmCfg {  // stage geometry in elements
  static constexpr int  apitch(int wn) { return 512 / wn + 4; }
  static constexpr int  bpitch(int wn) { return sizeof(T) == 8 ? kBK + 4 : 32 * wn + 4; }
  static constexpr int  bsize(int wn) { return sizeof(T) == 8 ? 32 * wn * bpitch(wn) : kBK * bpitch(wn); }
  static constexpr int  stage(int wn) { return kBK * apitch(wn) + bsize(wn); }
  static constexpr int  stages(int wn) { return wn == 1 ? 3 : 4; }
};

// Order of the reduction index inside a 16-deep slice: that of the
// trailing-update kernel's fragments (dgemm_tma.cu), so that both sum alike.
__constant__ const signed char kSliceOrder[16] = {0, 3, 12, 15, 2, 1, 14, 13,
                                                  4, 7, 8,  11, 6, 5, 10, 9};

// Stage slice kt: rows [row, row + nr) of A, columns [col, col + nc) of B.
template <typename T, int WN>
HPLB_DEV void load_slice(T* st, const T* A, int64_t lda, const T* B, int64_t ldb, int k, int kt,
                         int row, int nr, int col, int nc, bool vec) {
  constexpr int V = 16 / sizeof(T);
  const int     warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for(int h = 0; h < kBK / kWarps; ++h) {
    const int      kp = warp + h * kWarps;
    const int      kk = kt * kBK + (sizeof(T) == 8 ? (int)kSliceOrder[kp] : kp);
    const bool     in = kk < k;
    const T*       g  = A + (size_t)row + (size_t)(in ? kk : 0) * (size_t)lda;
    const uint32_t s  = s_addr(st + kp * GemmCfg<T>::apitch(WN));
    if(vec) {
      for(int r = V * lane; r < nr; r += 32 * V) cp_async16(s + r * sizeof(T), g + r, in);
    } else {
      for(int r = lane; r < nr; r += 32) cp_async1(s + r * sizeof(T), g + r, in);
    }
  }
  T* sb = st + kBK * GemmCfg<T>::apitch(WN);
#pragma unroll
  for(int h = 0; h < kBK * 32 * WN / kThreads; ++h) {
    const int idx = threadIdx.x + h * kThreads;
    const int kp = idx % kBK, nn = idx / kBK;
    const int kk = kt * kBK + (sizeof(T) == 8 ? (int)kSliceOrder[kp] : kp);
    const bool in = kk < k && nn < nc;
    const T*   g  = B + (size_t)(in ? kk : 0) + (size_t)(col + (in ? nn : 0)) * (size_t)ldb;
    T*         d  = sizeof(T) == 8 ? sb + nn * GemmCfg<T>::bpitch(WN) + kp
                                   : sb + kp * GemmCfg<T>::bpitch(WN) + nn;
    cp_async1(s_addr(d), g, in);
  }
}

template <int WN>
HPLB_DEV void gemm_tiles(int m, int n, int k, const double* A, int64_t lda, const double* B,
                         int64_t ldb, double* C, int64_t ldc, unsigned G, unsigned me,
                         double* sm) {
  using Cfg           = GemmCfg<double>;
  constexpr int WM    = kWarps / WN;
  constexpr int NST   = Cfg::stages(WN);
  const int     warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int     g = lane >> 2, t4 = lane & 3;
  const int     wm = warp % WM, wn = warp / WM;
  const int     KT    = (k + kBK - 1) / kBK;
  const int     slabs = (m + 15) / 16, share = (slabs + (int)G - 1) / (int)G;
  const int     sb = (int)me * share, se = min(slabs, sb + share);
  const bool    vec = (uintptr_t)A % 16 == 0 && lda % 2 == 0;
  for(int col = 0; col < n; col += 32 * WN)
    for(int s0 = sb; s0 < se;) {
      const int ns   = min(4, (se - s0 + WM - 1) / WM);  // 16-row slabs per warp
      const int row  = s0 * 16;
      // Rows staged: the pass's, to an even count (a 16-byte copy's pair never
      // leaves the column: lda is even and above the row).
      const int nr   = min(WM * ns * 16, m - row);
      const int nc   = min(32 * WN, n - col);
      double    acc[4][4][4];
#pragma unroll
      for(int i = 0; i < 4; ++i)
#pragma unroll
        for(int j = 0; j < 4; ++j)
#pragma unroll
          for(int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;
#pragma unroll
      for(int s = 0; s < NST - 1; ++s) {
        if(s < KT)
          load_slice<double, WN>(sm + s * Cfg::stage(WN), A, lda, B, ldb, k, s, row, nr, col, nc,
                                 vec);
        cp_commit();
      }
      for(int kt = 0; kt < KT; ++kt) {
        cp_wait<NST - 2>();
        __syncthreads();
        {
          const int nk = kt + NST - 1;
          if(nk < KT)
            load_slice<double, WN>(sm + (nk % NST) * Cfg::stage(WN), A, lda, B, ldb, k, nk, row,
                                   nr, col, nc, vec);
          cp_commit();
        }
        const double* as = sm + (kt % NST) * Cfg::stage(WN);
        const double* bs = as + kBK * Cfg::apitch(WN);
#pragma unroll
        for(int st = 0; st < 2; ++st) {
          double bf[4][2];
#pragma unroll
          for(int j = 0; j < 4; ++j) {
            const double* p = bs + (wn * 32 + j * 8 + g) * Cfg::bpitch(WN) + st * 8 + t4;
            bf[j][0]        = p[0];
            bf[j][1]        = p[4];
          }
#pragma unroll
          for(int i = 0; i < 4; ++i)
            if(i < ns) {
              const double* p =
                  as + (st * 8 + t4) * Cfg::apitch(WN) + (wm * ns + i) * 16 + g;
              double af[4];
              af[0] = p[0];
              af[1] = p[8];
              af[2] = p[4 * Cfg::apitch(WN)];
              af[3] = p[4 * Cfg::apitch(WN) + 8];
#pragma unroll
              for(int j = 0; j < 4; ++j) dmma(acc[i][j], af, bf[j]);
            }
        }
      }
      cp_wait<0>();
      __syncthreads();
#pragma unroll
      for(int h = 0; h < 2; ++h) {  // two slabs' loads in flight at once
        double    cv[2][4][4];
        const int c0 = col + wn * 32 + 2 * t4;
#pragma unroll
        for(int i = 0; i < 2; ++i) {
          const int  sl = wm * ns + 2 * h + i, r0 = row + sl * 16 + g;
          const bool in = 2 * h + i < ns && s0 + sl < se;
#pragma unroll
          for(int j = 0; j < 4; ++j)
#pragma unroll
            for(int r = 0; r < 4; ++r) {
              const int rr = r0 + (r >> 1) * 8, cc = c0 + j * 8 + (r & 1);
              cv[i][j][r] =
                  (in && rr < m && cc < n) ? __ldcg(C + (size_t)rr + (size_t)cc * ldc) : 0.0;
            }
        }
#pragma unroll
        for(int i = 0; i < 2; ++i) {
          const int  sl = wm * ns + 2 * h + i, r0 = row + sl * 16 + g;
          const bool in = 2 * h + i < ns && s0 + sl < se;
#pragma unroll
          for(int j = 0; j < 4; ++j)
#pragma unroll
            for(int r = 0; r < 4; ++r) {
              const int rr = r0 + (r >> 1) * 8, cc = c0 + j * 8 + (r & 1);
              if(in && rr < m && cc < n)
                C[(size_t)rr + (size_t)cc * ldc] = cv[i][j][r] - acc[2 * h + i][j][r];
            }
        }
      }
      s0 += WM * ns;
    }
}

// FP32: 8 x 8 values per thread (rows ty*4 + {0..3} of both halves of the tile,
// columns likewise), the sum over k in order.
template <int WN>
HPLB_DEV void gemm_tiles(int m, int n, int k, const float* A, int64_t lda, const float* B,
                         int64_t ldb, float* C, int64_t ldc, unsigned G, unsigned me, float* sm) {
  using Cfg         = GemmCfg<float>;
  constexpr int RT  = 512 / WN, NT = 32 * WN;
  constexpr int NST = Cfg::stages(WN);
  constexpr int TY  = RT / 8;  // lanes along rows: C in whole segments
  const int     ty = threadIdx.x % TY, tx = threadIdx.x / TY;
  const int     KT    = (k + kBK - 1) / kBK;
  const int     share = ((m + (int)G - 1) / (int)G + 7) / 8 * 8;
  const int     rb = (int)me * share, re = min(m, rb + share);
  const bool    vec = (uintptr_t)A % 16 == 0 && lda % 4 == 0;
  const bool    vec_c = (uintptr_t)C % 16 == 0 && ldc % 4 == 0;
  for(int col = 0; col < n; col += NT)
    for(int row = rb; row < re; row += RT) {
      const int nr = min(RT, re - row), nc = min(NT, n - col);
      float     acc[8][8];
#pragma unroll
      for(int i = 0; i < 8; ++i)
#pragma unroll
        for(int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll
      for(int s = 0; s < NST - 1; ++s) {
        if(s < KT)
          load_slice<float, WN>(sm + s * Cfg::stage(WN), A, lda, B, ldb, k, s, row, nr, col, nc,
                                vec);
        cp_commit();
      }
      for(int kt = 0; kt < KT; ++kt) {
        cp_wait<NST - 2>();
        __syncthreads();
        {
          const int nk = kt + NST - 1;
          if(nk < KT)
            load_slice<float, WN>(sm + (nk % NST) * Cfg::stage(WN), A, lda, B, ldb, k, nk, row,
                                  nr, col, nc, vec);
          cp_commit();
        }
        const float* as = sm + (kt % NST) * Cfg::stage(WN);
        const float* bs = as + kBK * Cfg::apitch(WN);
#pragma unroll 2
        for(int kk = 0; kk < kBK; ++kk) {
          const float*  pa = as + kk * Cfg::apitch(WN) + ty * 4;
          const float*  pb = bs + kk * Cfg::bpitch(WN) + tx * 4;
          const float4  a0 = *(const float4*)pa, a1 = *(const float4*)(pa + RT / 2);
          const float4  b0 = *(const float4*)pb, b1 = *(const float4*)(pb + NT / 2);
          const float   a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          const float   b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
          for(int i = 0; i < 8; ++i)
#pragma unroll
            for(int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
      }
      cp_wait<0>();
      __syncthreads();
      // Four columns' loads at once; four rows in one access where C allows it.
#pragma unroll
      for(int j0 = 0; j0 < 8; j0 += 4) {
        float cv[4][8];
#pragma unroll
        for(int j = 0; j < 4; ++j)
#pragma unroll
          for(int h = 0; h < 2; ++h) {
            const int    c = col + (j0 ? NT / 2 : 0) + tx * 4 + j, r = row + h * (RT / 2) + ty * 4;
            const float* q = C + (size_t)r + (size_t)c * ldc;
            if(vec_c && c < n && r + 3 < re) {
              const float4 t   = __ldcg(reinterpret_cast<const float4*>(q));
              cv[j][4 * h]     = t.x;
              cv[j][4 * h + 1] = t.y;
              cv[j][4 * h + 2] = t.z;
              cv[j][4 * h + 3] = t.w;
            } else {
#pragma unroll
              for(int i = 0; i < 4; ++i) cv[j][4 * h + i] = c < n && r + i < re ? __ldcg(q + i) : 0.f;
            }
          }
#pragma unroll
        for(int j = 0; j < 4; ++j)
#pragma unroll
          for(int h = 0; h < 2; ++h) {
            const int c = col + (j0 ? NT / 2 : 0) + tx * 4 + j, r = row + h * (RT / 2) + ty * 4;
            float*    q = C + (size_t)r + (size_t)c * ldc;
            if(vec_c && c < n && r + 3 < re) {
              *reinterpret_cast<float4*>(q) = make_float4(
                  cv[j][4 * h] - acc[4 * h][j0 + j], cv[j][4 * h + 1] - acc[4 * h + 1][j0 + j],
                  cv[j][4 * h + 2] - acc[4 * h + 2][j0 + j], cv[j][4 * h + 3] - acc[4 * h + 3][j0 + j]);
            } else {
#pragma unroll
              for(int i = 0; i < 4; ++i)
                if(c < n && r + i < re) q[i] = cv[j][4 * h + i] - acc[4 * h + i][j0 + j];
            }
          }
      }
    }
}

// X (jb x jb, leading dimension ldx) = L^-1 for the unit-lower L at L, from its
// inverted 32 x 32 diagonal blocks (dinv): substitution on the identity, CP
// neighbouring columns a warp, x in shared memory, one 32-row block after the other.
// Bound by the loads of L from L2, a batch of 16 columns on its way while the one
// before is used (FP64 / FP32 at jb = 256 37 / 34 us, 512 132 / 124; 171 / 188 without).
// Doubling ([A 0; B C]^-1 = [A^-1 0; -C^-1 (B A^-1) C^-1]) has a shorter chain and
// takes 77 us at 512, but multiplies the rounding of its products by C once more:
// |L X - I| is then 1.5 times substitution's at jb = 128, 2.7 at 256, 5.4 at 512.
constexpr int kClusterInverse = 512;  // the widest made here (see launch_unit_lower_inverse)
constexpr size_t kInverseBytes = (size_t)kWarps * 4 * kClusterInverse * sizeof(double);
template <typename T, int CP>
HPLB_DEV void lower_inverse_cols(const T* L, int64_t ldl, int jb, const T* dinv, T* X, int64_t ldx,
                                 int gw, int nw, T* sm) {
  const int lane = threadIdx.x & 31;
  T*        x    = sm + (size_t)(threadIdx.x >> 5) * CP * kClusterInverse;  // by column
  for(int c = gw * CP; c < jb; c += nw * CP) {
    const int first = c / kTri * kTri;  // the columns' own 32 rows; zeros above
#pragma unroll
    for(int q = 0; q < CP; ++q)
      if(c + q < jb)
        for(int r = lane; r < first; r += 32) X[(size_t)r + (size_t)(c + q) * (size_t)ldx] = (T)0;
    for(int row0 = first; row0 < jb; row0 += kTri) {
      const int r = row0 + lane;
      const T*  d = dinv + (size_t)row0 * kTri;
      T         v[CP];
      if(row0 == first) {
#pragma unroll
        for(int q = 0; q < CP; ++q) v[q] = __ldcg(d + (c % kTri + q) * kTri + lane);
      } else {
        T dv[kTri];
#pragma unroll
        for(int k = 0; k < kTri; ++k) dv[k] = row0 + k < jb ? __ldcg(d + k * kTri + lane) : (T)0;
#pragma unroll
        for(int q = 0; q < CP; ++q) v[q] = (T)0;
        const T* l = L + min(r, jb - 1);
        T        lv[2][16];
#pragma unroll
        for(int t = 0; t < 16; ++t) lv[0][t] = __ldcg(l + (size_t)(first + t) * (size_t)ldl);
        for(int k = first; k < row0; k += 32) {
#pragma unroll
          for(int h = 0; h < 2; ++h) {
            const int kn = min(k + 16 * (h + 1), row0 - 16);
#pragma unroll
            for(int t = 0; t < 16; ++t) lv[h ^ 1][t] = __ldcg(l + (size_t)(kn + t) * (size_t)ldl);
#pragma unroll
            for(int t = 0; t < 16; ++t)
#pragma unroll
              for(int q = 0; q < CP; ++q)
                v[q] = fma_(-lv[h][t], x[q * kClusterInverse + k + 16 * h + t], v[q]);
          }
        }
#pragma unroll
        for(int q = 0; q < CP; ++q) x[q * kClusterInverse + r] = r < jb ? v[q] : (T)0;
        __syncwarp();
#pragma unroll
        for(int q = 0; q < CP; ++q) v[q] = (T)0;
#pragma unroll
        for(int k = 0; k < kTri; ++k)
#pragma unroll
          for(int q = 0; q < CP; ++q) v[q] = fma_(dv[k], x[q * kClusterInverse + row0 + k], v[q]);
        __syncwarp();
      }
#pragma unroll
      for(int q = 0; q < CP; ++q) {
        x[q * kClusterInverse + r] = v[q];
        if(r < jb && c + q < jb) X[(size_t)r + (size_t)(c + q) * (size_t)ldx] = v[q];
      }
      __syncwarp();
    }
  }
}

template <typename T>
HPLB_DEV void lower_inverse(const T* L, int64_t ldl, int jb, const T* dinv, T* X, int64_t ldx,
                            unsigned G, unsigned me, T* sm) {
  const int gw = (int)me + (int)G * (int)(threadIdx.x >> 5), nw = (int)G * kWarps;
  // Columns per warp: as few passes as four at once allow.
  if(jb <= nw)
    lower_inverse_cols<T, 1>(L, ldl, jb, dinv, X, ldx, gw, nw, sm);
  else if(jb <= 2 * nw)
    lower_inverse_cols<T, 2>(L, ldl, jb, dinv, X, ldx, gw, nw, sm);
  else
    lower_inverse_cols<T, 4>(L, ldl, jb, dinv, X, ldx, gw, nw, sm);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
lower_inverse_kernel(const T* L, int64_t ldl, int jb, const T* dinv, T* X, int64_t ldx) {
  extern __shared__ __align__(128) unsigned char dyn[];
  lower_inverse<T>(L, ldl, jb, dinv, X, ldx, gridDim.x, blockIdx.x, reinterpret_cast<T*>(dyn));
}

constexpr size_t at_least(size_t a, size_t b) { return a > b ? a : b; }
template <typename T, int W, int RPT>
constexpr size_t dyn_bytes() {
  size_t b = sizeof(LeafMem<T, W, RPT>);
  b = at_least(b, (size_t)GemmCfg<T>::stages(1) * GemmCfg<T>::stage(1) * sizeof(T));
  b = at_least(b, (size_t)GemmCfg<T>::stages(2) * GemmCfg<T>::stage(2) * sizeof(T));
  b = at_least(b, (size_t)GemmCfg<T>::stages(4) * GemmCfg<T>::stage(4) * sizeof(T));
  b = at_least(b, kInverseBytes);
  b = at_least(b, (size_t)kWarps * 2 * (kMaxNb + 1) * sizeof(T));           // trsm_cols<T, 2>
  return at_least(b, (size_t)kWarps * kTri * kTopPitch * sizeof(T));        // invert_blocks
}

template <typename T, int W, int RPT>
__global__ void __launch_bounds__(kThreads, 1)
panel_fused_kernel(const __grid_constant__ FusedParams<T> P) {
  extern __shared__ __align__(128) unsigned char dyn[];
  __shared__ Shared<T, W>                        S;
  const unsigned G = cta_count(), me = cta_rank();
  T*             sm  = reinterpret_cast<T*>(dyn);
  auto&          mem = *reinterpret_cast<LeafMem<T, W, RPT>*>(dyn);
  if(threadIdx.x < kMaxG) {
    const uint32_t at = s_addr(&S.full[0]);
    S.peer[threadIdx.x] = threadIdx.x < G ? peer_addr(at, threadIdx.x) - at : 0;
  }
  if(threadIdx.x == 0) {
    S.abort = 0;
    for(int b = 0; b < kBufs; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s_addr(&S.full[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for(int b = 0; b < kBufs; ++b) mbar_expect(&S.full[b], G * (uint32_t)(W * sizeof(T) + 16));
  }
  cluster_sync();
  unsigned kc = 0;
  for(int o = 0; o < P.nops; ++o) {
    const int off = P.ops[o].off, jb = P.ops[o].jb, c2 = P.ops[o].c2, n2 = P.ops[o].n2 & ~kSplit;
    T*        a   = P.A + (size_t)(P.r0 + off) + (size_t)(P.c0 + off) * (size_t)P.ld;
    T*        inv = P.dinv + (size_t)(off / kTri) * kTri * kTri;
    if(n2 == 0 && c2 == 0) {
      {
        Leaf<T, W, RPT> F{P, S, mem, G, me, (int)(threadIdx.x >> 5), (int)(threadIdx.x & 31),
                          P.r0 + off, jb, kc};
        F.factor(P.c0 + off);
        kc = F.kc;
      }
      cluster_sync();  // L11 is in place
      leaf_finish<T, W>(P, S, G, me, off, jb, inv);
    } else if(n2 == 0) {
      invert_blocks(P, G, me, off, jb, sm);
    } else {
      T* x = P.A + (size_t)(P.r0 + off) + (size_t)(P.c0 + c2) * (size_t)P.ld;
      trsm<T>(x, P.ld, jb, a, P.ld, inv, n2, G, me, sm);
      const int m = P.n - (P.r0 + off + jb);
      if(m > 0 && !(P.ops[o].n2 & kSplit)) {
        cluster_sync();
        if(n2 <= 32)
          gemm_tiles<1>(m, n2, jb, a + jb, P.ld, x, P.ld, x + jb, P.ld, G, me, sm);
        else if(n2 <= 64)
          gemm_tiles<2>(m, n2, jb, a + jb, P.ld, x, P.ld, x + jb, P.ld, G, me, sm);
        else
          gemm_tiles<4>(m, n2, jb, a + jb, P.ld, x, P.ld, x + jb, P.ld, G, me, sm);
      }
    }
    cluster_sync();
  }
  if(P.linv == nullptr) return;
  // The row map of the panel's interchanges (the maps of perm_kernel), a thread
  // per entry, and L11^-1.
  int* s_piv = reinterpret_cast<int*>(dyn);
  if((int)me * kThreads < 2 * P.jb) {
    for(int i = threadIdx.x; i < P.jb; i += kThreads) s_piv[i] = __ldcg(P.ipiv + P.c0 + i) - P.r0;
    __syncthreads();
    for(int e = (int)me * kThreads + threadIdx.x; e < 2 * P.jb; e += (int)G * kThreads) {
      const bool fwd = e >= P.jb;
      int        at  = fwd ? e - P.jb : e;
      for(int t = 0; t < P.jb; ++t) {
        const int i  = fwd ? t : P.jb - 1 - t;
        const int pp = s_piv[i];
        at           = (at == i) ? pp : (at == pp ? i : at);
      }
      P.permU[e] = fwd ? (at >= P.jb ? at : -1) : at;
    }
    __syncthreads();  // s_piv is read: its memory is the inverse's now
  }
  lower_inverse<T>(P.A + (size_t)P.r0 + (size_t)P.c0 * (size_t)P.ld, P.ld, P.jb, P.dinv, P.linv,
                   P.jb, G, me, sm);
}

// The operations of a panel, in the order of the recursion (rfact 2: right-
// looking; else each piece is first brought up to date from the pieces before
// it, as HPL_pdrpanllT / HPL_pdrpancrT).
struct Builder {
  std::vector<Op> ops;
  int             nbmin, ndiv, rfact, W, rows;
  double          split;                     // products above this go to the whole GPU
  int             inv_off = -1, inv_jb = 0;  // the inverses written last

  void add(int off, int jb, int c2, int n2) {
    ops.push_back(Op{(unsigned short)off, (unsigned short)jb, (unsigned short)c2,
                     (unsigned short)n2});
  }
  // With NBMIN = 32 every leaf is one diagonal block of every node it is in, so
  // its inverse is kept; otherwise a node's blocks are inverted before its use.
  bool aligned() const { return nbmin == kTri; }
  void inverses(int off, int jb) {
    if(inv_off == off && inv_jb == jb) return;
    add(off, jb, 1, 0);
    inv_off = off;
    inv_jb  = jb;
  }
  void leaf(int off, int w) {
    for(int s = 0; s < w; s += W) {
      const int wl = std::min(W, w - s), rem = w - s - wl;
      add(off + s, wl, 0, 0);
      inv_off = off + s;
      inv_jb  = wl;
      if(rem > 0) add(off + s, wl, off + s + wl, rem);
    }
    if(w > W) inverses(off, w);
  }
  void update(int off, int jb, int c2, int n2) {
    if(!aligned()) inverses(off, jb);
    const double work = (double)(rows - off - jb) * jb * n2;
    add(off, jb, c2, work > split ? n2 | kSplit : n2);
  }
  void panel(int off, int N) {
    if(N <= nbmin) return leaf(off, N);
    const int nbs = (((N + nbmin - 1) / nbmin + ndiv - 1) / ndiv) * nbmin;
    int       jj = 0, rem = N, jb = nbs;
    do {
      rem -= jb;
      if(rfact != 2 && jj > 0) update(off, jj, off + jj, jb);
      panel(off + jj, jb);
      if(rfact == 2 && rem > 0) update(off + jj, jb, off + jj + jb, rem);
      jj += jb;
      jb = std::min(rem, nbs);
    } while(rem > 0);
  }
};

// Launches a cluster of g CTAs; *done stays false where the GPU has no place for one,
// which is what placeable[g] keeps.  An error is returned and not kept: it may be
// over by the next call (no memory to load the kernel, say).
template <typename Kern, typename... Args>
cudaError_t launch_cluster(Kern kern, int g, size_t smem, signed char* placeable,
                           cudaStream_t stream, bool* done, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim            = dim3((unsigned)g);
  cfg.blockDim           = dim3(kThreads);
  cfg.dynamicSmemBytes   = smem;
  cfg.stream             = stream;
  cudaLaunchAttribute at[1];
  at[0].id               = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)g;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs              = at;
  cfg.numAttrs           = 1;
  cudaError_t e          = cudaSuccess;
  if(placeable[g] == 0) {  // 0 unknown, 1 yes, -1 no
    int n = 0;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if(e == cudaSuccess && g > 8)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if(e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
    if(e == cudaSuccess || e == cudaErrorInvalidClusterSize) {
      placeable[g] = e == cudaSuccess && n >= 1 ? 1 : -1;
      if(e != cudaSuccess) cudaGetLastError();
      e = cudaSuccess;
    }
  }
  if(e == cudaSuccess && placeable[g] < 0) return cudaSuccess;
  if(e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kern, args...);
  *done = e == cudaSuccess;
  if(!*done) cudaGetLastError();
  return e;
}

template <typename T, int W, int RPT>
cudaError_t launch_form(FusedParams<T>& P, int g, cudaStream_t stream, bool* done) {
  static signed char placeable[kMaxG + 1] = {};
  return launch_cluster(panel_fused_kernel<T, W, RPT>, g, dyn_bytes<T, W, RPT>(), placeable,
                        stream, done, P);
}

// Rows per thread and leaf width by the rows a cluster of 16 must hold: the
// widest leaf whose RPT x W values stay within 192 of a thread's registers.  A
// narrower leaf costs an update and its barriers more per 32 columns (12288 rows
// as one leaf of 32: 76 us, 16384 rows as two of 16: 111 us).
template <typename T>
int form_width(int rows) {
  if(sizeof(T) == 8) return rows <= 12288 ? 32 : (rows <= 24576 ? 16 : (rows <= 32768 ? 8 : 0));
  return rows <= 24576 ? 32 : (rows <= 32768 ? 16 : 0);
}

cudaError_t launch_rows(FusedParams<double>& P, int rows, int g, cudaStream_t st, bool* done) {
  if(rows <= 4096) return launch_form<double, 32, 1>(P, g, st, done);
  if(rows <= 8192) return launch_form<double, 32, 2>(P, g, st, done);
  if(rows <= 12288) return launch_form<double, 32, 3>(P, g, st, done);
  if(rows <= 16384) return launch_form<double, 16, 4>(P, g, st, done);
  if(rows <= 24576) return launch_form<double, 16, 6>(P, g, st, done);
  return launch_form<double, 8, 8>(P, g, st, done);
}
cudaError_t launch_rows(FusedParams<float>& P, int rows, int g, cudaStream_t st, bool* done) {
  if(rows <= 4096) return launch_form<float, 32, 1>(P, g, st, done);
  if(rows <= 8192) return launch_form<float, 32, 2>(P, g, st, done);
  if(rows <= 16384) return launch_form<float, 32, 4>(P, g, st, done);
  if(rows <= 24576) return launch_form<float, 32, 6>(P, g, st, done);
  return launch_form<float, 16, 8>(P, g, st, done);
}

cudaError_t launch_product(int m, int n, int k, const double* A, int64_t lda, const double* B,
                           int64_t ldb, double* C, int64_t ldc, int* status, cudaStream_t st) {
  return launch_dgemm_sub(m, n, k, A, lda, B, ldb, C, ldc, status, st);
}
cudaError_t launch_product(int m, int n, int k, const float* A, int64_t lda, const float* B,
                           int64_t ldb, float* C, int64_t ldc, int*, cudaStream_t st) {
  return launch_sgemm(m, n, k, A, lda, B, ldb, C, ldc, true, st);
}

// CTAs of a cluster for `units` pieces of work that a CTA should have at least
// one of.
int cluster_for(int units) {
  int g = 1;
  while(g < kMaxG && units > g) g *= 2;
  return g;
}

}  // namespace

template <typename T>
cudaError_t launch_panel_fused(T* A, int64_t ld, int r0, int c0, int n, int jb, int nbmin,
                               int ndiv, int rfact, int* ipiv, int* status, T* dinv, T* linv,
                               int* permU, cudaStream_t stream, int* launches, bool* done) {
  *done          = false;
  const int rows = n - r0, W = form_width<T>(rows);
  if(W == 0 || jb < 1 || jb > kMaxNb || nbmin > kTri) return cudaSuccess;
  Builder B;
  B.nbmin = nbmin;
  B.ndiv  = ndiv;
  B.rfact = rfact;
  B.W     = W;
  B.rows  = rows;
  // Products of more work than this take longer on 16 SMs than a launch over all of
  // them with the cluster's own relaunch (8192 x 512 panel: everything in the
  // cluster 2.43 ms FP64 and 3.54 ms FP32, with this line 1.53 and 1.76 ms).
  B.split = sizeof(T) == 8 ? 5e7 : 2.5e7;
  B.panel(0, jb);
  if(linv && !B.aligned()) B.inverses(0, jb);
  if(B.ops.size() > (size_t)kMaxOps) return cudaSuccess;
  FusedParams<T> P;
  P.A      = A;
  P.ld     = ld;
  P.r0     = r0;
  P.c0     = c0;
  P.n      = n;
  P.jb     = jb;
  P.ipiv   = ipiv;
  P.status = status;
  P.dinv   = dinv;
  P.linv   = nullptr;
  P.permU  = permU;
  // At least 64 rows per CTA (64, 128 and 256 are within 2% of each other from 100
  // to 4096 rows, 256 is 5% slower at 500).
  const int g = cluster_for((rows + 63) / 64);
  for(size_t at = 0; at < B.ops.size();) {
    size_t end = at;
    while(end < B.ops.size() && !(B.ops[end].n2 & kSplit)) ++end;
    const bool last = end == B.ops.size();
    if(!last) ++end;
    P.nops = (int)(end - at);
    std::memcpy(P.ops, B.ops.data() + at, (end - at) * sizeof(Op));
    if(last && jb <= kClusterInverse) P.linv = linv;
    bool        did = false;
    cudaError_t e   = launch_rows(P, rows - B.ops[at].off, g, stream, &did);
    if(!did && at == 0) return cudaSuccess;  // (the other path meets a lasting error itself)
    if(!did) return e != cudaSuccess ? e : cudaErrorLaunchFailure;
    *launches += 1;
    if(!last) {
      const Op& o = B.ops[end - 1];
      const int m = rows - o.off - o.jb;
      T*        a = A + (size_t)(r0 + o.off) + (size_t)(c0 + o.off) * (size_t)ld;
      T*        x = A + (size_t)(r0 + o.off) + (size_t)(c0 + o.c2) * (size_t)ld;
      e = launch_product(m, o.n2 & ~kSplit, o.jb, a + o.jb, ld, x, ld, x + o.jb, ld, status, stream);
      if(e != cudaSuccess) return e;
      *launches += 1;
    }
    at = end;
  }
  if(linv && jb > kClusterInverse) {
    cudaError_t e = launch_perm(ipiv + c0, r0, jb, permU, stream);
    if(e != cudaSuccess) return e;
    *launches += 1;
    e = launch_unit_lower_inverse_wide(A + (size_t)r0 + (size_t)c0 * (size_t)ld, ld, jb, dinv, linv,
                                       jb, stream, launches);
    if(e != cudaSuccess) return e;
  } else if(linv && P.linv == nullptr) {
    return cudaErrorLaunchFailure;  // (a panel ends with a leaf)
  }
  *done = true;
  return cudaSuccess;
}

// As in the panel up to kClusterInverse columns, with a CTA per 8 columns over the GPU
// beyond, where 16 SMs are too few (us at 512 columns, 16 CTAs / the GPU: FP64 132 /
// 175, FP32 124 / 143; the GPU at 640 181 and 151).
template <typename T>
cudaError_t launch_unit_lower_inverse(const T* L, int64_t ldl, int jb, const T* dinv, T* Linv,
                                      int64_t ldinv, cudaStream_t stream, int* launches) {
  if(jb <= 0) return cudaSuccess;
  if(jb > kClusterInverse)
    return launch_unit_lower_inverse_wide(L, ldl, jb, dinv, Linv, ldinv, stream, launches);
  static bool attr = false;
  cudaError_t e    = cudaSuccess;
  if(!attr)
    e = cudaFuncSetAttribute(lower_inverse_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kInverseBytes);
  if(e != cudaSuccess) return e;
  attr = true;
  // As many warps as a panel's cluster has; they do not wait for each other.
  lower_inverse_kernel<T><<<cluster_for((jb + 31) / 32), kThreads, kInverseBytes, stream>>>(
      L, ldl, jb, dinv, Linv, ldinv);
  *launches += 1;
  return cudaGetLastError();
}

#define HPLB_FUSED_INSTANTIATE(T)                                                               \
  template cudaError_t launch_panel_fused<T>(T*, int64_t, int, int, int, int, int, int, int,    \
                                             int*, int*, T*, T*, int*, cudaStream_t, int*,      \
                                             bool*);                                            \
  template cudaError_t launch_unit_lower_inverse<T>(const T*, int64_t, int, const T*, T*,       \
                                                    int64_t, cudaStream_t, int*);
HPLB_FUSED_INSTANTIATE(double)
HPLB_FUSED_INSTANTIATE(float)

}  // namespace hplb
