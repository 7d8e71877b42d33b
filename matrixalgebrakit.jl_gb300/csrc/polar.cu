// Left polar decomposition by the scaled Newton iteration, GB300 native.
//
// Replaces the reference's left_polar!(A, (W, P), ::PolarNewton)
// (src/implementations/polar.jl:99-111) and left_polar_newton!
// (polar.jl:128-166) with _avgdiff! (polar.jl:209-220; GPU kernel
// ext/MatrixAlgebraKitCUDAExt/MatrixAlgebraKitCUDAExt.jl:154-173) and
// project_hermitian! (src/implementations/projections.jl:61-108).
//
//   m > n : A = Q R (qr_run), iterate on X0 = R;   m == n : iterate on X0 = A
//   X <- (g X + X^{-H}/g)/2,   g = sqrt(||X^{-H}||_F / ||X||_F)
//   stop when max|X^{-H}/g - g X| <= tol  or after maxiter iterations
//   W = Q X  (m > n)  or  W = X,     P = herm(W^H A)
//
// The inverse is an in-place blocked Gauss-Jordan elimination with partial
// pivoting (gje_inverse): per block column of 32 a panel kernel (pivot
// search + row exchange + elimination, one barrier per column, panel rows
// resident in shared memory; a thread-block cluster of up to 16 CTAs for n up
// to 4096 in Float64, 2048 in ComplexF64 and 8192 in the FP32 types as far as
// its rows fit, a cooperative grid with a bounded global barrier beyond), a
// row-exchange/save kernel for the other columns and one rank-32 GEMM update
// -- 2n^3 flops in total, the same count as the reference's LU + inverse.  The
// triangular first iterate of a tall A is inverted by substitution.  The Newton update reads
// X^{-H} straight out of the eliminated matrix through the inverse column
// permutation (no separate transpose or permutation pass) and fuses the
// avgdiff step, the scaling and the max-abs convergence measure.  For
// m > n, P is formed as herm(X^H R) (= herm(W^H A) since A = QR, W = QX),
// an n^3 instead of an m n^2 product.
#include "gemm.cuh"
#include "internal.h"
#include "util.cuh"

#include <climits>
#include <mutex>

namespace mak {

constexpr int GJ_NB = 32;
constexpr int GJ_OUTER_NB = 128;  // block column of the mixed-precision path
constexpr int GJ_THREADS = 256;

template <class T>
struct GjArgs {
  T* X;
  int64_t ldx;
  int n, k0, b, rpc;
  int* piv;
  real_t<T>* part_val;
  unsigned long long* part_key;  // [2][gstride] the same by key (register panel)
  int* part_idx;
  T* swapbuf;  // [2][GJ_NB]: row jj by column parity
  T* cand;     // [2][gstride][GJ_NB]: each CTA's pivot candidate row, by column parity
  T* low;       // [GJ_NB][GJ_NB]: the pivot rows' multipliers, for gje_laswp_save_kernel
  int gstride;  // allocation stride of the per-CTA partials
  unsigned* bar;
  int* status;
  int* singular;
  const int* skip;  // device stop flag of a fixed-iteration loop (or nullptr)
};

__device__ __forceinline__ double cabs1_(double x) { return fabs(x); }
__device__ __forceinline__ float cabs1_(float x) { return fabsf(x); }
template <class R> __device__ __forceinline__ R cabs1_(cplx<R> x) { return fabs(x.re) + fabs(x.im); }

// (value desc, index asc) arg-max merge
template <class R>
__device__ __forceinline__ void amax_merge(R& v, int& i, R v2, int i2) {
  if (v2 > v || (v2 == v && i2 < i)) { v = v2; i = i2; }
}

// The panel of an inverse whose rows do not fit shared memory twice (from
// about 200 rows per CTA, n beyond 10^4): one grid round per column, the slab
// once in shared memory.  All smaller ones take gje_panel_ahead_kernel.
template <class T>
__global__ void __launch_bounds__(GJ_THREADS) gje_panel_kernel(GjArgs<T> a) {
  using R = real_t<T>;
  if (skipped(a.skip)) return;  // the same in every CTA: no barrier is reached
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Ps = reinterpret_cast<T*>(smem_raw);  // rpc x b, ld = rpc
  T* fsh = Ps + (size_t)a.rpc * a.b;        // rpc multipliers of the current column
  __shared__ R sv[32];
  __shared__ int si[32];
  __shared__ T prow[GJ_NB];
  __shared__ T srow[GJ_NB];
  __shared__ T dinv_s;
  __shared__ int pivs, pivq;
  const int G = gridDim.x, cb = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int rpc = a.rpc, b = a.b, k0 = a.k0;
  const int r0 = cb * rpc;
  const int nr = max(0, min(a.n, r0 + rpc) - r0);
  T* Xp = a.X + (int64_t)k0 * a.ldx;
  for (int c = 0; c < b; c++)
    for (int r = tid; r < nr; r += blockDim.x) Ps[r + c * rpc] = Xp[(r0 + r) + (int64_t)c * a.ldx];
  __syncthreads();

  // Per column one grid-wide round: every CTA publishes its local arg-max
  // (value desc, index asc) together with that candidate row, and the CTA
  // holding row jj publishes row jj.  After the barrier every CTA merges the
  // partials in the same fixed order, reads the winning candidate as the
  // pivot row, and the CTA holding the pivot's old row receives row jj: no
  // second round for the exchange.  The published values are
  // double-buffered by column parity (a CTA writes column j+1's slot only
  // after every CTA passed barrier j, i.e. finished reading column j-1's).
  for (int j = 0; j < b; j++) {
    const int jj = k0 + j;
    const int par = j & 1;
    R* pval = a.part_val + par * a.gstride;
    int* pidx = a.part_idx + par * a.gstride;
    T* rowjj = a.swapbuf + par * GJ_NB;
    T* cand = a.cand + (int64_t)par * a.gstride * GJ_NB;
    // ---- local pivot candidate over global rows >= jj
    R best = R(-1);
    int bidx = INT_MAX;
    for (int r = tid; r < nr; r += blockDim.x) {
      const int gr = r0 + r;
      if (gr >= jj) amax_merge(best, bidx, cabs1_(Ps[r + j * rpc]), gr);
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
      R v2 = __shfl_xor_sync(0xffffffffu, best, m);
      int i2 = __shfl_xor_sync(0xffffffffu, bidx, m);
      amax_merge(best, bidx, v2, i2);
    }
    if (lane == 0) { sv[wid] = best; si[wid] = bidx; }
    if (jj >= r0 && jj < r0 + nr)
      for (int c = tid; c < b; c += blockDim.x) {
        rowjj[c] = Ps[(jj - r0) + c * rpc];
      }
    __syncthreads();
    if (wid == 0) {
      R v = lane < nw ? sv[lane] : R(-1);
      int ix = lane < nw ? si[lane] : INT_MAX;
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) {
        R v2 = __shfl_xor_sync(0xffffffffu, v, m);
        int i2 = __shfl_xor_sync(0xffffffffu, ix, m);
        amax_merge(v, ix, v2, i2);
      }
      if (lane == 0) {
        pval[cb] = v;
        pidx[cb] = ix;
        pivs = ix;
      }
    }
    __syncthreads();
    {
      const int li = pivs;  // this CTA's candidate row (global index)
      if (li != INT_MAX)
        for (int c = tid; c < b; c += blockDim.x) {
          cand[(int64_t)cb * GJ_NB + c] = Ps[(li - r0) + c * rpc];
        }
    }
    if (!panel_sync<SYNC_GRID>(a.bar, G, a.status)) return;

    // ---- global pivot (identical in every CTA), then the exchange
    if (wid == 0) {
      R v = R(-1);
      int ix = INT_MAX, iq = -1;
      for (int q = lane; q < G; q += 32) {
        const R v2 = ld_cg(&pval[q]);
        const int i2 = ld_cg(&pidx[q]);
        if (v2 > v || (v2 == v && i2 < ix)) { v = v2; ix = i2; iq = q; }
      }
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) {
        R v2 = __shfl_xor_sync(0xffffffffu, v, m);
        int i2 = __shfl_xor_sync(0xffffffffu, ix, m);
        int q2 = __shfl_xor_sync(0xffffffffu, iq, m);
        if (v2 > v || (v2 == v && i2 < ix)) { v = v2; ix = i2; iq = q2; }
      }
      if (lane == 0) {
        pivs = (ix == INT_MAX) ? jj : ix;
        pivq = (ix == INT_MAX || ix == jj) ? -1 : iq;
      }
    }
    __syncthreads();
    const int p = pivs, q = pivq;
    // pivot row: the winning CTA's candidate (row jj itself when p == jj)
    for (int c = tid; c < b; c += blockDim.x)
      prow[c] = q < 0 ? ld_cg(&rowjj[c]) : ld_cg(&cand[(int64_t)q * GJ_NB + c]);
    if (p != jj && p >= r0 && p < r0 + nr)
      for (int c = tid; c < b; c += blockDim.x) Ps[(p - r0) + c * rpc] = ld_cg(&rowjj[c]);
    if (cb == 0 && tid == 0) a.piv[jj] = p;
    __syncthreads();
    if (tid == 0) {
      const T d = prow[j];
      if (d == zero_<T>()) atomicExch(a.singular, 1);
      dinv_s = inv_fast(d);  // once per column: a dependent FP64 chain
    }
    __syncthreads();
    const T dinv = dinv_s;
    // the scaled pivot row, formed once (GB300 issues about 1.6 FP64
    // operations per clock per SM, so the elimination keeps one FMA per
    // element); its own column holds the new pivot-column entry 1/d
    for (int c = tid; c < b; c += blockDim.x) srow[c] = (c == j) ? dinv : prow[c] * dinv;
    __syncthreads();
    // the rows' multipliers f_r = X[r, jj] first, then the elimination with
    // each warp on its own columns (lanes over rows), so that all eight
    // warps share the FP64 work even when a CTA owns only a few dozen rows
    for (int r = tid; r < nr; r += blockDim.x) fsh[r] = Ps[r + j * rpc];
    __syncthreads();
    for (int c = wid; c < b; c += nw) {
      const T sc = srow[c];
      T* pc = Ps + c * rpc;
      for (int r = lane; r < nr; r += 32) {
        if (r0 + r == jj) pc[r] = sc;
        else if (c == j) pc[r] = -(fsh[r] * dinv);
        else pc[r] = fma_(-fsh[r], sc, pc[r]);
      }
    }
    __syncthreads();
  }
  for (int c = 0; c < b; c++)
    for (int r = tid; r < nr; r += blockDim.x) Xp[(r0 + r) + (int64_t)c * a.ldx] = Ps[r + c * rpc];
}

// ---- the panel one column ahead ------------------------------------------------
// The panel's rows sit row-major in shared memory, in two buffers by column
// parity.  Warp 0 of a CTA runs one column ahead of the others: after the
// pivot of column j is known it updates column j + 1 alone (lane = row),
// picks the CTA's next candidate (the largest magnitude at or below row
// jj + 1, the first row on ties; complex: the larger component), forms that
// row, scales it by its pivot's reciprocal and publishes it, while the other
// warps eliminate column j from all rows.  So a column's chain is one search,
// one reciprocal and one round between the CTAs, and the elimination's FP64
// work (rows x 32 per column at 1.66 per clock per SM; kDefer: the half of it to
// the column's right) runs beside it.  In a
// cluster (SYNC_CLUSTER) the candidates are pushed into every CTA's shared
// memory before the cluster barrier, so that nothing is fetched after it; the
// 16-byte type pushes keys only and one warp pulls the winner's row (remote
// stores run at about 5 bytes per clock: pushing all rows to 16 CTAs took 1650
// of a ComplexF64 column's 7100 cycles, 5540 with the pull; a Float64 column
// takes 3220 with the push, 3650 with the pull); in a grid they go through L2.  Elementwise arithmetic only: the result does
// not depend on the number of CTAs.
__device__ __forceinline__ unsigned long long pivot_key(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
  return b > 0x7FF0000000000000ull ? 0ull : b;  // NaN is never preferred
}
__device__ __forceinline__ unsigned long long pivot_key(float x) {
  const unsigned b = __float_as_uint(x) & 0x7FFFFFFFu;
  return b > 0x7F800000u ? 0ull : (unsigned long long)b << 32;
}
template <class R> __device__ __forceinline__ unsigned long long pivot_key(cplx<R> x) {
  const unsigned long long a = pivot_key(x.re), b = pivot_key(x.im);
  return a > b ? a : b;
}
// by integer comparison (a comparison of doubles would take the FP64 pipe)
__device__ __forceinline__ bool is_nan_(double x) {
  return ((unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull) >
         0x7FF0000000000000ull;
}
__device__ __forceinline__ bool is_nan_(float x) {
  return (__float_as_uint(x) & 0x7FFFFFFFu) > 0x7F800000u;
}
template <class R> __device__ __forceinline__ bool is_nan_(cplx<R> x) {
  return is_nan_(x.re) || is_nan_(x.im);
}
// the lanes' largest key, the smallest index among equals; the lane it is in
__device__ __forceinline__ int warp_pivot(unsigned long long& key, int& idx) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
  bool in = (unsigned)(key >> 32) == hi;
  const unsigned lo = __reduce_max_sync(0xffffffffu, in ? (unsigned)key : 0u);
  in = in && (unsigned)key == lo;
  const int i = __reduce_min_sync(0xffffffffu, in ? idx : INT_MAX);
  const unsigned at = __ballot_sync(0xffffffffu, in && idx == i);
  key = (unsigned long long)hi << 32 | lo;
  idx = i;
  return __ffs((int)at) - 1;
}
// 1 / d into y (1 + p): y close to 1/d with r = 1 - d y, p = r + r^2; beyond
// the normal range y is the IEEE quotient and p = 0
__device__ __forceinline__ void inv_split(double d, double& y, double& p) {
  const int e = exp2_of(d);
  if (e > -1000 && e < 1000) {
    y = rcp_seed(d);
    const double r = fma(-d, y, 1.0);
    p = fma(r, r, r);
  } else {
    y = 1.0 / d;
    p = 0.0;
  }
}
__device__ __forceinline__ void inv_split(float d, float& y, float& p) {
  y = 1.0f / d;
  p = 0.0f;
}
template <class R> __device__ __forceinline__ void inv_split(cplx<R> d, cplx<R>& y, R& p) {
  const R w = fmax(fabs(d.re), fabs(d.im));
  const int e = exp2_of(w);
  const int lim = sizeof(R) == 8 ? 480 : 50;
  if (w > R(0) && e > -lim && e < lim) {
    R q;
    inv_split(fma_(d.re, d.re, d.im * d.im), q, p);
    y = conj_(d) * q;
  } else {
    y = inv_fast(d);
    p = R(0);
  }
}

constexpr int kGjClusterWide = 16;
constexpr int GJA_LD = GJ_NB + 1;
// Warps 1-3 and 5-7 eliminate; warp 4 shares warp 0's SM sub-partition, whose
// FP64 pipe is left to it, and only passes row jj + 1 on.
constexpr int GJA_MAIN = 6;
// kDefer: a column is eliminated from the columns to its right only (lane =
// row), the columns to its left keep their multipliers, and the row exchange's
// kernel, which follows every panel, multiplies them by the inverse of the
// pivot rows' unit triangle (gje_finish_rows) on all SMs that are free.  That
// halves the FP64 work of the panel's 16 SMs.  Column c of the multipliers
// stays in buffer c & 1, whose columns up to j nothing else uses any more.
// From GJA_DEFER_ROWS rows per CTA on: there the halved elimination (per
// panel, 256 rows of Float64: 137 -> 90 us) is worth more than what the
// finishing rows add to the row exchange (6 -> 12 us).  left_polar, all in the
// panel / deferred: Float64 n = 1600 43.8 / 44.7 ms, 1800 59.7 / 59.6, 2040
// 65.8 / 62.0, 4096 187 / 163; ComplexF64 1100 51.7 / 54.7, 1280 76.4 / 76.0,
// 1440 83.4 / 80.6; Float32 2100 48.1 / 48.8, 3000 96.2 / 88.5; ComplexF32
// 1400 35.8 / 36.1, 2100 74.2 / 72.1.
template <class T>
constexpr int GJA_DEFER_ROWS = sizeof(real_t<T>) == 8 ? (traits<T>::cpx ? 80 : 112)
                                                      : (traits<T>::cpx ? 104 : 128);
// NL: rows per lane of warp 0 (32 NL rows per CTA at most)
template <class T, int SYNC, int NL, bool kDefer>
__global__ void __launch_bounds__(GJ_THREADS, 1) gje_panel_ahead_kernel(GjArgs<T> a) {
  using R = real_t<T>;
  if (skipped(a.skip)) return;  // the same in every CTA: no barrier is reached
  constexpr bool kCl = SYNC == SYNC_CLUSTER;
  constexpr int GC = kCl ? kGjClusterWide : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const Xs = reinterpret_cast<T*>(smem_raw);  // [2][rpc][GJA_LD]
  // by column parity: the CTAs' candidates, the scaled candidate rows and row
  // jj (written by the other CTAs; kPull: this CTA's own, read by the others)
  constexpr bool kPull = kCl && sizeof(T) == 16;
  __shared__ ulonglong2 x_key[2][GC];  // key, row index
  __shared__ T x_row[2][kPull ? 1 : GC][GJ_NB];
  __shared__ T x_rowjj[2][GJ_NB];
  __shared__ T s_row[GJ_NB], s_rjj[GJ_NB];  // what warp 0 pulled, for the others
  const int G = gridDim.x, cb = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, wid = tid >> 5, nw = GJ_THREADS / 32;
  const int b = a.b, k0 = a.k0, rpc = a.rpc;
  const int r0 = cb * rpc;
  const int nr = max(0, min(a.n, r0 + rpc) - r0);
  const size_t slab = (size_t)rpc * GJA_LD;
  T* Xp = a.X + (int64_t)k0 * a.ldx + r0;
  {
    T* const X0 = Xs + slab;  // "column -1"
    for (int r = lane; r < nr; r += 32) {
      T v[GJ_NB / 8];
#pragma unroll
      for (int q = 0; q < GJ_NB / 8; q++) {
        const int c = wid + q * nw;
        v[q] = c < b ? Xp[r + (int64_t)c * a.ldx] : zero_<T>();
      }
#pragma unroll
      for (int q = 0; q < GJ_NB / 8; q++) X0[r * GJA_LD + wid + q * nw] = v[q];
    }
  }
  __syncthreads();
  // a CTA may be written to only once it runs
  if constexpr (kCl) cluster_sync_all();

  // publish row v (lane = column) of column j's round as this CTA's candidate
  auto put_cand = [&](int par, unsigned long long key, int idx, T v) {
    if constexpr (kCl) {
      if constexpr (kPull)
        x_row[par][0][lane] = v;
      else
        for (int q = 0; q < G; q++) dsmem_st(&x_row[par][cb][lane], (unsigned)q, v);
      if (lane < G)
        dsmem_st(&x_key[par][cb], (unsigned)lane,
                 make_ulonglong2(key, (unsigned long long)(unsigned)idx));
    } else {
      if (lane < b) a.cand[((int64_t)par * a.gstride + cb) * GJ_NB + lane] = v;
      if (lane == 0) {
        a.part_key[par * a.gstride + cb] = key;
        a.part_idx[par * a.gstride + cb] = idx;
      }
    }
  };
  auto put_rowjj = [&](int par, T v) {
    if constexpr (kCl) {
      if constexpr (kPull)
        x_rowjj[par][lane] = v;
      else
        for (int q = 0; q < G; q++) dsmem_st(&x_rowjj[par][lane], (unsigned)q, v);
    } else {
      if (lane < b) a.swapbuf[par * GJ_NB + lane] = v;
    }
  };
  // the candidate among warp 0's column values cv (rows r0 + lane + 32 l, at
  // or below row jj): key, row index (INT_MAX: none) and value
  T cv[NL];
  auto pick = [&](int jj, unsigned long long& key, int& idx, T& d) {
    key = 0;
    idx = INT_MAX;
    d = zero_<T>();
#pragma unroll
    for (int l = 0; l < NL; l++) {
      const int r = lane + 32 * l;
      const unsigned long long k2 = pivot_key(cv[l]);
      // a NaN is no candidate, as in a comparison by magnitude
      if (r < nr && r0 + r >= jj && !is_nan_(cv[l]) && (idx == INT_MAX || k2 > key)) {
        key = k2;
        idx = r0 + r;
        d = cv[l];
      }
    }
    const int at = warp_pivot(key, idx);
    d = shfl_idx_(d, at);
  };

  if (wid == 0) {
    const T* X0 = Xs + slab;
#pragma unroll
    for (int l = 0; l < NL; l++)
      cv[l] = lane + 32 * l < nr ? X0[(lane + 32 * l) * GJA_LD] : zero_<T>();
    unsigned long long key;
    int idx;
    T d, y;
    R pr;
    pick(k0, key, idx, d);
    inv_split(d, y, pr);
    const T v = idx == INT_MAX ? zero_<T>() : X0[(idx - r0) * GJA_LD + lane];
    put_cand(0, key, idx, fma_real_(lane == 0 ? y : v * y, pr));
  } else if (wid == 4 && k0 >= r0 && k0 < r0 + nr) {
    put_rowjj(0, Xs[slab + (k0 - r0) * GJA_LD + lane]);
  }

  for (int j = 0; j < b; j++) {
    const int jj = k0 + j, par = j & 1;
    const T* const Xo = Xs + (par ^ 1) * slab;  // through column j - 1
    T* const Xn = Xs + par * slab;
    if (!panel_sync<SYNC>(a.bar, G, a.status)) return;

    // ---- the pivot, the same in every warp of every CTA
    int p, q = 0;
    unsigned long long key = 0;
    {
      int idx = INT_MAX;
      if constexpr (kCl) {
        if (lane < G) {
          const ulonglong2 c = x_key[par][lane];
          key = c.x;
          idx = (int)(unsigned)c.y;
          q = lane;
        }
      } else {
        for (int g = lane; g < G; g += 32) {
          const unsigned long long k2 = __ldcg(&a.part_key[par * a.gstride + g]);
          const int i2 = ld_cg(&a.part_idx[par * a.gstride + g]);
          if (k2 > key || (k2 == key && i2 < idx)) {
            key = k2;
            idx = i2;
            q = g;
          }
        }
      }
      q = __shfl_sync(0xffffffffu, q, warp_pivot(key, idx));
      p = idx == INT_MAX ? jj : idx;
      if (idx == INT_MAX) q = -1;
    }
    T srow, rjj = zero_<T>();
    if (kPull && wid != 0) {
      asm volatile("bar.sync 1, %0;" ::"n"(GJ_THREADS) : "memory");
      srow = s_row[lane];
      rjj = s_rjj[lane];
    } else {
      // row jj is wanted where the pivot's old row is (and by all without a
      // candidate)
      if constexpr (kPull) {
        if (q < 0 || (p != jj && p >= r0 && p < r0 + nr))
          rjj = dsmem_ld(&x_rowjj[par][lane], (unsigned)(jj / rpc));
        if (q >= 0) srow = dsmem_ld(&x_row[par][0][lane], (unsigned)q);
      } else if constexpr (kCl) {
        if (q < 0 || p != jj) rjj = x_rowjj[par][lane];
        if (q >= 0) srow = x_row[par][q][lane];
      } else {
        if (q < 0 || p != jj)
          rjj = lane < b ? ld_cg(&a.swapbuf[par * GJ_NB + lane]) : zero_<T>();
        if (q >= 0)
          srow = lane < b ? ld_cg(&a.cand[((int64_t)par * a.gstride + q) * GJ_NB + lane])
                          : zero_<T>();
      }
      if (q < 0) {  // no candidate (NaN only): row jj itself
        T y;
        R pr;
        inv_split(shfl_idx_(rjj, j), y, pr);
        srow = kDefer && lane < j ? rjj : fma_real_(lane == j ? y : rjj * y, pr);
      }
      if constexpr (kPull) {
        s_row[lane] = srow;
        s_rjj[lane] = rjj;
        asm volatile("bar.arrive 1, %0;" ::"n"(GJ_THREADS) : "memory");
      }
    }
    if (cb == 0 && tid == 0) {
      a.piv[jj] = p;
      if (q >= 0 && key == 0) atomicExch(a.singular, 1);
    }
    if (kDefer && cb == 0 && wid == 4) a.low[j * GJ_NB + lane] = lane < j ? srow : zero_<T>();
    const int lp = p != jj ? p - r0 : -1;  // the pivot's old row here: row jj moves into it
    const T rjj_j = shfl_idx_(rjj, j);
    // row r (not row jj) through column j - 1 and through column j (lane = column)
    auto before = [&](int r) -> T {
      return r == lp ? rjj
                     : Xs[(kDefer && lane < j ? lane & 1 : par ^ 1) * slab + r * GJA_LD + lane];
    };
    auto through = [&](T x, T f) -> T {
      return kDefer && lane < j ? x : fma_(-f, srow, lane == j ? zero_<T>() : x);
    };

    if (wid == 0) {
      if (j + 1 < b) {
        const T sj1 = shfl_idx_(srow, j + 1), rj1 = shfl_idx_(rjj, j + 1);
        T fv[NL];
#pragma unroll
        for (int l = 0; l < NL; l++) {
          const int r = lane + 32 * l;
          const bool at = r == lp;
          fv[l] = at ? rjj_j : cv[l];
          const T x = at ? rj1 : (r < nr ? Xo[r * GJA_LD + j + 1] : zero_<T>());
          cv[l] = fma_(-fv[l], sj1, x);
        }
        unsigned long long k2;
        int idx;
        T d, y;
        R pr;
        pick(jj + 1, k2, idx, d);
        inv_split(d, y, pr);
        T v = zero_<T>();
        if (idx != INT_MAX) {
          const int r = idx - r0;
          T f = fv[0];
#pragma unroll
          for (int l = 1; l < NL; l++)
            if (r >> 5 == l) f = fv[l];
          f = shfl_idx_(f, r & 31);
          v = through(before(r), f);
        }
        put_cand(par ^ 1, k2, idx,
                 kDefer && lane <= j ? v : fma_real_(lane == j + 1 ? y : v * y, pr));
      }
    } else if (wid == 4) {
      const int r = jj + 1 - r0;
      if (j + 1 < b && r >= 0 && r < nr)
        put_rowjj(par ^ 1, through(before(r), r == lp ? rjj_j : Xo[r * GJA_LD + j]));
      // the multipliers of the exchanged rows: the pivot row keeps none
      if (kDefer && lane < j) {
        T* const M = Xs + (lane & 1) * slab + lane;
        if (lp >= 0 && lp < nr) M[lp * GJA_LD] = rjj;
        if (jj >= r0 && jj < r0 + nr) M[(jj - r0) * GJA_LD] = zero_<T>();
      }
    } else if constexpr (!kDefer) {
      // lane = column
      const int mi = wid < 4 ? wid - 1 : wid - 2;
      for (int rb = mi; rb < nr; rb += 4 * GJA_MAIN) {
        T x[4], f[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int r = rb + k * GJA_MAIN;
          if (r < nr) {
            x[k] = before(r);
            f[k] = r == lp ? rjj_j : Xo[r * GJA_LD + j];
          }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int r = rb + k * GJA_MAIN;
          if (r < nr) Xn[r * GJA_LD + lane] = r0 + r == jj ? srow : through(x[k], f[k]);
        }
      }
    } else {
      // lane = row: a third of the columns and half of the rows per warp
      constexpr int H = 2, NH = NL / H;
      const int mi = wid < 4 ? wid - 1 : wid - 2;
      const int rb = lane + (mi & 1) * 32 * NH;
      T f[NH];
#pragma unroll
      for (int l = 0; l < NH; l++) {
        const int r = rb + 32 * l;
        f[l] = r < nr ? (r == lp ? rjj_j : Xo[r * GJA_LD + j]) : zero_<T>();
      }
      for (int c = j + mi / H; c < b; c += GJA_MAIN / H) {
        const T sc = shfl_idx_(srow, c), rc = shfl_idx_(rjj, c);
        T x[NH];
#pragma unroll
        for (int l = 0; l < NH; l++) {
          const int r = rb + 32 * l;
          x[l] = (c == j || r >= nr) ? zero_<T>() : r == lp ? rc : Xo[r * GJA_LD + c];
        }
#pragma unroll
        for (int l = 0; l < NH; l++) {
          const int r = rb + 32 * l;
          if (r < nr) Xn[r * GJA_LD + c] = r0 + r == jj ? sc : fma_(-f[l], sc, x[l]);
        }
      }
    }
  }
  // kPull: no CTA leaves while another may still read its rows; pushes into a
  // CTA came before the last column's barrier
  if constexpr (kPull) cluster_sync_all();
  else __syncthreads();
  for (int c = wid; c < b; c += nw)
    for (int r = lane; r < nr; r += 32)
      Xp[r + (int64_t)c * a.ldx] = Xs[((kDefer ? c : b - 1) & 1) * slab + r * GJA_LD + c];
}

// For every column outside the panel [k0, k0 + b): apply the panel's row
// exchanges, save rows k0 .. k0+b-1 into buf (b x n) and zero them in X.
// Only columns c in [c_lo, c_hi) are touched.
//
// The exchanges are composed first: only rows k0 .. k0+b-1 and the pivots
// take part, and the source of each is found by walking the exchanges
// backwards (every CTA repeats this small integer work).  Then a column is
// one batch of independent loads and one of stores, instead of b dependent
// exchanges through memory (4096 rows: 140 us per call before).
// perm, when given, is the composed row permutation of the whole
// elimination so far, exchanged along by one extra CTA.
//
// low, when given: the panel holds multipliers, and the CTAs from fin0 on
// finish its rows: row w becomes the x with x_q = w_q + sum_{k > q} x_k low[k][q].
// A row is spread over FIN_LPR lanes (four columns each; two of the 16-byte
// type): with 32 rows per CTA the work reaches 128 CTAs at 4096 rows.
constexpr int LASWP_MAX_B = 128;
template <class T> constexpr int FIN_LPR = sizeof(T) == 16 ? 16 : 8;
template <class T> constexpr int FIN_ROWS = 256 / FIN_LPR<T>;
template <class T>
__device__ __forceinline__ void gje_finish_rows(int n, T* Xp, int64_t ldx, int b, const T* low,
                                                int blk) {
  constexpr int LPR = FIN_LPR<T>, NC = GJ_NB / LPR;
  __shared__ T Ls[GJ_NB * GJ_NB];
  const int tid = threadIdx.x, q = tid % LPR;
  const int r = blk * FIN_ROWS<T> + tid / LPR;
  T x[NC];
#pragma unroll
  for (int i = 0; i < NC; i++) {
    const int c = q + LPR * i;
    x[i] = r < n && c < b ? Xp[r + (int64_t)c * ldx] : zero_<T>();
  }
  for (int e = tid; e < GJ_NB * GJ_NB; e += 256) Ls[e] = e < b * GJ_NB ? low[e] : zero_<T>();
  __syncthreads();
#pragma unroll
  for (int k = GJ_NB - 1; k > 0; k--) {
    if (k < b) {
      T u = x[k / LPR];
      if constexpr (traits<T>::cpx) {
        u.re = __shfl_sync(0xffffffffu, u.re, k % LPR, LPR);
        u.im = __shfl_sync(0xffffffffu, u.im, k % LPR, LPR);
      } else {
        u = __shfl_sync(0xffffffffu, u, k % LPR, LPR);
      }
#pragma unroll
      for (int i = 0; i < NC; i++)
        if (LPR * i < k && q + LPR * i < k) x[i] = fma_(u, Ls[k * GJ_NB + q + LPR * i], x[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < NC; i++) {
    const int c = q + LPR * i;
    if (r < n && c < b) Xp[r + (int64_t)c * ldx] = x[i];
  }
}
template <class T>
__global__ void __launch_bounds__(256) gje_laswp_save_kernel(int n, T* X, int64_t ldx, int k0,
                                                             int b, const int* piv, T* buf,
                                                             int c_lo, int c_hi, int* perm,
                                                             const T* low, int fin0,
                                                             const int* skip) {
  if (skipped(skip)) return;
  if (low != nullptr && (int)blockIdx.x >= fin0) {
    gje_finish_rows<T>(n, X + (int64_t)k0 * ldx, ldx, b, low, (int)blockIdx.x - fin0);
    return;
  }
  __shared__ int pv[LASWP_MAX_B];
  __shared__ int pos[2 * LASWP_MAX_B], src[2 * LASWP_MAX_B];
  const int tid = threadIdx.x;
  for (int t = tid; t < b; t += blockDim.x) {
    const int p = piv[k0 + t];
    pv[t] = (p >= k0 + t && p < n) ? p : k0 + t;
  }
  __syncthreads();
  // entry t < b: row k0 + t; entry b + t: row pv[t] if it lies below the
  // panel's rows (a row that is the pivot twice is listed twice with the same
  // source, so both entries store the same value)
  for (int e = tid; e < 2 * b; e += blockDim.x) {
    const int x = e < b ? k0 + e : pv[e - b];
    int s = -1;
    if (e < b || x >= k0 + b) {
      s = x;
      for (int t = b - 1; t >= 0; t--) {
        if (s == k0 + t) s = pv[t];
        else if (s == pv[t]) s = k0 + t;
      }
    }
    pos[e] = x;
    src[e] = s;
  }
  __syncthreads();
  if (perm != nullptr && (int)blockIdx.x == fin0 - 1) {
    // at most 2 x 128 entries: one per thread
    const int s = tid < 2 * b ? src[tid] : -1;
    const int v = s >= 0 ? perm[s] : 0;
    __syncthreads();
    if (s >= 0) perm[pos[tid]] = v;
    return;
  }
  // a warp per column
  const int lane = tid & 31;
  const int c = c_lo + blockIdx.x * (int)(blockDim.x >> 5) + (tid >> 5);
  if (c >= c_hi || (c >= k0 && c < k0 + b)) return;
  T* col = X + (int64_t)c * ldx;
  constexpr int U = 2 * LASWP_MAX_B / 32;
  T v[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const int e = lane + 32 * u;
    if (32 * u < 2 * b && e < 2 * b && src[e] >= 0) v[u] = col[src[e]];
  }
  __syncwarp();  // every load of the column before any store to it
#pragma unroll
  for (int u = 0; u < U; u++) {
    const int e = lane + 32 * u;
    if (32 * u < 2 * b && e < 2 * b && src[e] >= 0) {
      if (e < b) {
        buf[e + (int64_t)c * b] = v[u];
        col[pos[e]] = zero_<T>();
      } else {
        col[pos[e]] = v[u];
      }
    }
  }
}

__global__ void iota_kernel(int n, int* v, int* w) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    v[i] = i;
    w[i] = i;
  }
}

// iperm = inverse of the composed row permutation
__global__ void gje_perm_kernel(int n, const int* perm, int* iperm, const int* skip) {
  if (skipped(skip)) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const int p = perm[i];
    if (p >= 0 && p < n) iperm[p] = i;
  }
}

// slab capacity of the panel kernel, whose dynamic shared-memory limit is
// raised once per type and device
template <class T>
static size_t gj_slab_cap() {
  static PerDevice<size_t> pd;
  return pd.get([] {
    cudaFuncAttributes fa;
    size_t stat = 16 * 1024;
    if (cudaFuncGetAttributes(&fa, gje_panel_kernel<T>) == cudaSuccess) stat = fa.sharedSizeBytes;
    const size_t cap = (size_t)max_smem_optin() - stat - 1024;
    cudaFuncSetAttribute(gje_panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cap);
    return cap;
  });
}

// Launches the panel that runs one column ahead on G CTAs of ga.rpc rows; 1 if
// it does not fit (shared memory, or the cluster or grid cannot be resident).
template <class T, int SYNC, int NL, bool kDefer>
static int gje_ahead_launch_nl(cudaStream_t s, GjArgs<T>& ga, int G) {
  auto kern = gje_panel_ahead_kernel<T, SYNC, NL, kDefer>;
  const size_t smem = 2 * (size_t)ga.rpc * GJA_LD * sizeof(T);
  static PerDevice<int> pd;  // the dynamic shared memory the kernel may take (0: cannot run)
  const int cap = pd.get([&] {
    cudaFuncAttributes fa;
    int v = 0;
    if (cudaFuncGetAttributes(&fa, kern) == cudaSuccess) v = max_smem_optin() - (int)fa.sharedSizeBytes;
    if (v <= 0 || cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, v) !=
                      cudaSuccess)
      v = 0;
    if (SYNC == SYNC_CLUSTER && v > 0) {
      // 16 CTAs at the largest slab this instance takes
      cudaLaunchConfig_t c16 = {};
      cudaLaunchAttribute at[1];
      c16.gridDim = dim3(kGjClusterWide);
      c16.blockDim = dim3(GJ_THREADS);
      const size_t most = 2 * (size_t)32 * NL * GJA_LD * sizeof(T);
      c16.dynamicSmemBytes = most < (size_t)v ? most : (size_t)v;
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = kGjClusterWide;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      c16.attrs = at;
      c16.numAttrs = 1;
      int nc = 0;
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
              cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&nc, kern, &c16) != cudaSuccess || nc < 1)
        v = 0;
    }
    (void)cudaGetLastError();
    return v;
  });
  if (smem > (size_t)cap) return 1;
  if (SYNC == SYNC_GRID) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, GJ_THREADS, smem) !=
            cudaSuccess ||
        (int64_t)per_sm * num_sms() < G) {
      (void)cudaGetLastError();
      return 1;
    }
    ProfScope prof(s, PROF_GJ_PANEL, 2.0 * (double)ga.n * ga.b * sizeof(T));
    note_launch();
    void* args[] = {&ga};
    MAK_CUDA_TRY(cudaLaunchCooperativeKernel((void*)kern, dim3((unsigned)G), dim3(GJ_THREADS),
                                             args, smem, s));
    return 0;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)G);
  cfg.blockDim = dim3(GJ_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)G;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ProfScope prof(s, PROF_GJ_PANEL, 2.0 * (double)ga.n * ga.b * sizeof(T));
  note_launch();
  MAK_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, ga));
  return 0;
}
// deferred: the panel holds multipliers, whose rows gje_laswp_save_kernel finishes
template <class T, int SYNC>
static int gje_ahead_launch(cudaStream_t s, GjArgs<T>& ga, int G, bool& deferred) {
  const int nl = (int)ceil_div(ga.rpc, 32);
  deferred = ga.rpc > GJA_DEFER_ROWS<T>;
  if (deferred) {
    if (nl <= 4) return gje_ahead_launch_nl<T, SYNC, 4, true>(s, ga, G);
    if (nl <= 8) return gje_ahead_launch_nl<T, SYNC, 8, true>(s, ga, G);
    if constexpr (SYNC == SYNC_CLUSTER && sizeof(real_t<T>) == 4)
      if (nl <= 16) return gje_ahead_launch_nl<T, SYNC, 16, true>(s, ga, G);
    return 1;
  }
  if (nl <= 1) return gje_ahead_launch_nl<T, SYNC, 1, false>(s, ga, G);
  if (nl <= 2) return gje_ahead_launch_nl<T, SYNC, 2, false>(s, ga, G);
  static_assert(GJA_DEFER_ROWS<T> <= 128, "the largest instance below has 4 x 32 rows");
  return gje_ahead_launch_nl<T, SYNC, 4, false>(s, ga, G);
}

template <class T>
int gje_inverse(cudaStream_t st, int64_t n, T* X, int64_t ldx, int* iperm, int precision,
                Arena& ar, mak_info* info) {
  const int sms = num_sms();
  // mixed precision: 128-wide block columns, eliminated with 32-wide panels
  // whose updates stay inside the block; the other columns then receive one
  // rank-128 update through the split-precision tensor-core GEMM
  // the 128-wide blocking from n^2 128 >= 2^25 multiply-adds (complex
  // counted 4x: n >= 512 real, n >= 256 complex; MAK_GJ_SPLIT_MIN overrides
  // it).  Below that the native elimination runs even when mixed precision
  // is asked for (a gate of its own: the general split-product gate does not
  // move it).  Measured on the 300 uneven blocks (mixed polar, CUDA-graph
  // replay, 16 streams): gate 2^29 / 2^25 / 2^23 gave 2.23 / 1.80 / 1.75 s;
  // the launches the lower gates add only cost when they are not replayed
  // from a graph (the same batch issued eagerly: 2.68 / 5.47 / 5.64 s).
  const double gate = tuning(TUNE_GJ_SPLIT_MIN);
  const bool mixed = precision == MAK_PREC_MIXED && sizeof(real_t<T>) == 8 &&
                     (traits<T>::cpx ? 4.0 : 1.0) * (double)n * (double)n * GJ_OUTER_NB >= gate;
  const int NBO = mixed ? GJ_OUTER_NB : GJ_NB;
  int* piv = ar.take<int>(n > 0 ? n : 1);
  int* perm = ar.take<int>(n > 0 ? n : 1);
  // per-CTA pivot partials and candidate rows, double-buffered by column parity
  real_t<T>* part_val = ar.take<real_t<T>>(2 * sms);
  unsigned long long* part_key = ar.take<unsigned long long>(2 * sms);
  int* part_idx = ar.take<int>(2 * sms);
  T* swapbuf = ar.take<T>(2 * GJ_NB);
  T* cand = ar.take<T>((size_t)2 * sms * GJ_NB);
  T* low = ar.take<T>((size_t)GJ_NB * GJ_NB);
  T* buf = ar.take<T>((size_t)NBO * (n > 0 ? n : 1));
  T* bufo = mixed ? ar.take<T>((size_t)NBO * (n > 0 ? n : 1)) : nullptr;
  unsigned* bar = ar.take<unsigned>(2);
  char* ozs = nullptr;
  size_t oz_bytes = 0;
  if (mixed) {
    Arena meas(nullptr, 0);
    gemm_prec<T>(st, precision, n, n, NBO, one_<T>(), opnd<T>(nullptr, 1), opnd<T>(nullptr, 1),
                 one_<T>(), nullptr, 1, meas, nullptr);
    oz_bytes = meas.off + 1024;
    ozs = ar.take<char>(oz_bytes);
  }
  if (ar.base == nullptr) return 0;
  if (!ar.ok()) return MAK_ERR_WORKSPACE;
  if (n <= 0) return 0;
  // (the largest n whose inverse is provided)
  if ((size_t)n * sizeof(int) > (size_t)max_smem_optin() - 1024) return MAK_ERR_UNSUPPORTED;
  MAK_CUDA_TRY(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), st));
  // pivots start as the identity so that an aborted panel (bounded barrier
  // timeout) still leaves every index in range; so does the permutation
  note_launch();
  iota_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>((int)n, piv, perm);
  const size_t cap = gj_slab_cap<T>();
  // one 32-wide panel (cooperative launch, at most max_ctas CTAs: on the
  // look-ahead side stream it leaves the other SMs to the main stream)
  auto panel = [&](int64_t k0, int b, cudaStream_t s, int max_ctas, bool& unfinished) -> int {
    GjArgs<T> ga{X, ldx, (int)n, (int)k0, b, 0, piv, part_val, part_key, part_idx, swapbuf,
                 cand, low, sms, bar, &info->status, &info->singular, skip_flag()};
    // The panel that runs one column ahead: one cluster of up to 16 CTAs (at
    // least 32 rows each) up to the size where a column's elimination on 16 SMs
    // (half of rows per CTA x 32, complex four times that) takes longer than a
    // grid's round between its CTAs, about 4.5 us per column; beyond, a
    // cooperative grid while a CTA's rows fit shared memory twice.  left_polar
    // (mixed), cluster / grid: Float64 n = 4200 116.8 / 115.4 ms, 6000 229.0 /
    // 227.7; ComplexF64 2048 60.4 / 64.3, 2500 104.7 / 93.5; Float32 4200 73.9 /
    // 110.8, 8000 298 / 372; ComplexF32 4200 148 / 177, 6000 333 / 379.
    const int64_t cluster_max =
        sizeof(real_t<T>) == 4 ? 8192 : traits<T>::cpx ? 2048 : 4096;
    if (n <= cluster_max) {
      int64_t G = ceil_div(n, 32);
      if (G > kGjClusterWide) G = kGjClusterWide;
      const int64_t rpc = ceil_div(n, G);
      G = ceil_div(n, rpc);
      ga.rpc = (int)rpc;
      const int rc = gje_ahead_launch<T, SYNC_CLUSTER>(s, ga, (int)G, unfinished);
      if (rc != 1) return rc;
    }
    {
      int64_t G = ceil_div(n, 32);
      if (G > max_ctas) G = max_ctas;
      const int64_t rpc = ceil_div(n, G);
      G = ceil_div(n, rpc);
      ga.rpc = (int)rpc;
      const int rc = gje_ahead_launch<T, SYNC_GRID>(s, ga, (int)G, unfinished);
      if (rc != 1) return rc;
    }
    unfinished = false;
    // grid: rows per CTA >= 64, at most one CTA per SM, slab within shared memory
    int64_t G = ceil_div(n, 64);
    if (G > max_ctas) G = max_ctas;
    // the slab holds rpc x (b + 1) values: the panel rows and their multipliers
    int64_t rpc = ceil_div(n, G);
    if ((size_t)rpc * (b + 1) * sizeof(T) > cap) {
      G = ceil_div(n, (int64_t)(cap / ((size_t)(b + 1) * sizeof(T))));
      if (G > sms) return MAK_ERR_UNSUPPORTED;
      rpc = ceil_div(n, G);
    }
    G = ceil_div(n, rpc);
    size_t smem = (size_t)rpc * (b + 1) * sizeof(T);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gje_panel_kernel<T>,
                                                      GJ_THREADS, smem) != cudaSuccess ||
        (int64_t)per_sm * sms < G)
      return MAK_ERR_UNSUPPORTED;
    ga.rpc = (int)rpc;
    void* args[] = {&ga};
    ProfScope prof(s, PROF_GJ_PANEL, 2.0 * (double)n * b * sizeof(T));
    note_launch();
    MAK_CUDA_TRY(cudaLaunchCooperativeKernel((void*)gje_panel_kernel<T>,
                                             dim3((unsigned)G), dim3(GJ_THREADS), args, smem, s));
    return 0;
  };
  // the panels of block column [K0, K0 + KB) with their updates confined to
  // the block's columns (the whole elimination when not mixed: KB = n)
  auto factor_block = [&](int64_t K0, int64_t KB, cudaStream_t s, int max_ctas) -> int {
    const int64_t c_lo = K0, c_hi = K0 + KB;
    for (int64_t k0 = K0; k0 < K0 + KB; k0 += GJ_NB) {
      const int b = (int)((K0 + KB - k0) < GJ_NB ? (K0 + KB - k0) : GJ_NB);
      bool unfinished = false;  // the panel holds multipliers
      MAK_TRY(panel(k0, b, s, max_ctas, unfinished));
      note_launch();
      const int fin0 = (int)ceil_div(c_hi - c_lo, 8) + 1;
      const unsigned fin = unfinished ? (unsigned)ceil_div(n, FIN_ROWS<T>) : 0u;
      gje_laswp_save_kernel<T><<<(unsigned)fin0 + fin, 256, 0, s>>>(
          (int)n, X, ldx, (int)k0, b, piv, buf, (int)c_lo, (int)c_hi, perm,
          unfinished ? low : nullptr, fin0, skip_flag());
      MAK_CUDA_TRY(cudaGetLastError());
      const T* F = X + k0 * ldx;
      if (k0 > c_lo)
        MAK_TRY(gemm<T>(s, n, k0 - c_lo, b, one_<T>(), opnd<T>(F, ldx),
                        opnd<T>(buf + c_lo * b, b), one_<T>(), X + c_lo * ldx, ldx));
      if (k0 + b < c_hi)
        MAK_TRY(gemm<T>(s, n, c_hi - k0 - b, b, one_<T>(), opnd<T>(F, ldx),
                        opnd<T>(buf + (k0 + b) * b, b), one_<T>(), X + (k0 + b) * ldx, ldx));
    }
    return 0;
  };
  // block column [K0, K0 + KB) applied to the columns [c_lo, c_hi) outside
  // it: its row exchanges, then one rank-KB update (split-precision product)
  auto apply_block = [&](int64_t K0, int64_t KB, int64_t c_lo, int64_t c_hi, cudaStream_t s,
                         int max_ctas) -> int {
    if (c_hi <= c_lo) return 0;
    note_launch();
    gje_laswp_save_kernel<T><<<(unsigned)ceil_div(c_hi - c_lo, 8), 256, 0, s>>>(
        (int)n, X, ldx, (int)K0, (int)KB, piv, bufo, (int)c_lo, (int)c_hi, nullptr, nullptr,
        0, skip_flag());
    MAK_CUDA_TRY(cudaGetLastError());
    const T* Fb = X + K0 * ldx;
    const int64_t l1 = c_hi < K0 ? c_hi : K0;  // left part [c_lo, l1)
    if (l1 > c_lo) {
      Arena oz(ozs, oz_bytes);
      MAK_TRY(gemm_prec<T>(s, precision, n, l1 - c_lo, KB, one_<T>(), opnd<T>(Fb, ldx),
                           opnd<T>(bufo + c_lo * KB, KB), one_<T>(), X + c_lo * ldx, ldx, oz,
                           &info->status, max_ctas));
    }
    const int64_t r0 = c_lo > K0 + KB ? c_lo : K0 + KB;  // right part [r0, c_hi)
    if (c_hi > r0) {
      Arena oz(ozs, oz_bytes);
      MAK_TRY(gemm_prec<T>(s, precision, n, c_hi - r0, KB, one_<T>(), opnd<T>(Fb, ldx),
                           opnd<T>(bufo + r0 * KB, KB), one_<T>(), X + r0 * ldx, ldx, oz,
                           &info->status, max_ctas));
    }
    return 0;
  };

  if (!mixed) {
    MAK_TRY(factor_block(0, n, st, sms));
  } else {
    // Look-ahead: block K is applied first to block K+1's columns; the side
    // stream then factors block K+1 (its panels touch only its own columns,
    // and its row exchanges reach the other columns when block K+1 is
    // applied) while the main stream applies block K to the remaining
    // columns.
    const int64_t nblk = ceil_div(n, (int64_t)NBO);
    LookAhead* la = (nblk > 1 && lookahead_enabled() && n >= 2048) ? lookahead() : nullptr;
    const int la_ctas = lookahead_ctas();
    MAK_TRY(factor_block(0, n < NBO ? n : NBO, st, sms));
    for (int64_t K = 0; K < nblk; K++) {
      const int64_t K0 = K * NBO, KB = (n - K0) < NBO ? (n - K0) : NBO;
      const int64_t nx = K0 + KB;
      const bool has_next = nx < n;
      const int64_t nKB = has_next ? ((n - nx) < NBO ? (n - nx) : NBO) : 0;
      if (has_next && la) {
        MAK_TRY(apply_block(K0, KB, nx, nx + nKB, st, 0));
        MAK_CUDA_TRY(cudaEventRecord(la->ev_ready, st));
        MAK_CUDA_TRY(cudaStreamWaitEvent(la->side, la->ev_ready, 0));
        MAK_TRY(factor_block(nx, nKB, la->side, la_ctas));
        MAK_CUDA_TRY(cudaEventRecord(la->ev_done, la->side));
        MAK_TRY(apply_block(K0, KB, 0, K0, st, sms - la_ctas));
        MAK_TRY(apply_block(K0, KB, nx + nKB, n, st, sms - la_ctas));
        MAK_CUDA_TRY(cudaStreamWaitEvent(st, la->ev_done, 0));
      } else {
        MAK_TRY(apply_block(K0, KB, 0, n, st, 0));
        if (has_next) MAK_TRY(factor_block(nx, nKB, st, sms));
      }
    }
  }
  note_launch();
  gje_perm_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>((int)n, perm, iperm, skip_flag());
  MAK_CUDA_TRY(cudaGetLastError());
  return 0;
}

// ---- inverse of a triangular matrix --------------------------------------------
// Back substitution on R X = I by row blocks of 32 from the last one up: the
// block's rows are solved for (tri_solve_kernel) and their product with the
// columns of R above them subtracted from the rows above, two launches per
// block and n^3 / 3 multiply-adds, against a pivoted panel, an exchange and
// updates of all n columns per block in gje_inverse.
//
// Substitution because its residual R X - I is bounded by n eps |R| |X| entry
// by entry whatever R's condition.  Doubling (X_ab = -X_aa R_ab X_bb on ever
// larger blocks, log2(n / 32) levels) multiplies by the inverses of whole
// blocks, whose size R X no longer shows: on the factor of 100 smooth columns
// of condition 3e6 it is wrong by 1e-7 where this is by 5e-12, on 260 of them
// in every digit.  FP64 products in either precision: rows and columns that
// meet are graded against each other when R is, and a split product is
// accurate to the product of their maxima only.
constexpr int TRI_NB = 32;
constexpr int TRI_WARPS = 4;
// FP64 work grows with n^3 and the elimination's split products hardly, so in
// mixed precision the elimination takes over where it is the faster.  QR
// pullback by substitution / by elimination: Float64 n = 520 0.69 / 1.83 ms,
// 2000 6.6 / 10.7, 2800 15.0 / 19.5, 4000 38.3 / 37.7; ComplexF64 520 1.38 /
// 3.06, 2000 21.9 / 26.4, 2800 53.2 / 51.3.
template <class T>
constexpr int64_t TRI_SOLVE_MAX_N = traits<T>::cpx ? 2432 : 3584;

// X <- I
template <class T>
__global__ void __launch_bounds__(256) tri_eye_kernel(int n, T* X, const int* skip) {
  if (skipped(skip)) return;
  const int i = blockIdx.x * 256 + threadIdx.x;
  for (int j = blockIdx.y; j < n; j += gridDim.y)
    if (i < n) X[i + (int64_t)j * n] = i == j ? one_<T>() : zero_<T>();
}
// Rows i0 .. i0 + 31 of X from their right-hand sides in place, the columns
// from i0 on: a warp per column, lane = row, x_l = b_l / R_ll and b_i -= R_il
// x_l from the last row up.  A chain of 32 steps of about 150 cycles.
template <class T>
__global__ void __launch_bounds__(32 * TRI_WARPS) tri_solve_kernel(int n, int i0, const T* R,
                                                                   int64_t ldr, T* X,
                                                                   int* singular,
                                                                   const int* skip) {
  if (skipped(skip)) return;
  __shared__ T U[TRI_NB][TRI_NB + 1];  // U[l][i] = R[i, l]
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nb = min(TRI_NB, n - i0);
  for (int l = wid; l < nb; l += TRI_WARPS)
    U[l][lane] = lane <= l ? R[i0 + lane + (int64_t)(i0 + l) * ldr] : zero_<T>();
  __syncthreads();
  const T d = lane < nb ? U[lane][lane] : one_<T>();
  if (blockIdx.x == 0 && d == zero_<T>()) atomicExch(singular, 1);
  const T dinv = inv_fast(d);
  const int c = i0 + (int)blockIdx.x * TRI_WARPS + wid;
  if (c >= n) return;
  T* const x = X + i0 + lane + (int64_t)c * n;
  T b = lane < nb ? *x : zero_<T>();
  for (int l = nb - 1; l >= 0; l--) {
    if (lane == l) b = b * dinv;
    const T u = lane < l ? U[l][lane] : zero_<T>();
    b = fma_(-u, shfl_idx_(b, l), b);
  }
  if (lane < nb) *x = b;
}

// Y <- the upper triangle of R, zero below
template <class T>
__global__ void __launch_bounds__(256) tri_copy_kernel(int n, const T* R, int64_t ldr, T* Y,
                                                       const int* skip) {
  if (skipped(skip)) return;
  const int i = blockIdx.x * 256 + threadIdx.x;
  for (int j = blockIdx.y; j < n; j += gridDim.y)
    if (i < n) Y[i + (int64_t)j * n] = i <= j ? R[i + (int64_t)j * ldr] : zero_<T>();
}
// X[:, j] = Y[:, iperm[j]] above the diagonal, zero below
template <class T>
__global__ void __launch_bounds__(256) tri_gather_kernel(int n, const T* Y, const int* iperm,
                                                         T* X, const int* skip) {
  if (skipped(skip)) return;
  const int i = blockIdx.x * 256 + threadIdx.x;
  for (int j = blockIdx.y; j < n; j += gridDim.y)
    if (i < n) X[i + (int64_t)j * n] = i <= j ? Y[i + (int64_t)iperm[j] * n] : zero_<T>();
}

template <class T>
bool tri_substitution(int64_t n, int precision) {
  constexpr int64_t most = TRI_SOLVE_MAX_N<T>;
  return precision != MAK_PREC_MIXED || sizeof(real_t<T>) != 8 || n <= most;
}

template <class T>
int tri_inverse(cudaStream_t st, int64_t n, const T* R, int64_t ldr, T* X, int precision,
                Arena& ar, mak_info* info) {
  const bool direct = tri_substitution<T>(n, precision);
  T* Y = nullptr;
  int* iperm = nullptr;
  char* gjs = nullptr;
  size_t gj_bytes = 0;
  if (!direct) {
    Arena meas(nullptr, 0);
    gje_inverse<T>(st, n, nullptr, n, nullptr, precision, meas, nullptr);
    gj_bytes = meas.off + 256;
    Y = ar.take<T>((size_t)n * n + 1);
    iperm = ar.take<int>(n + 1);
    gjs = ar.take<char>(gj_bytes);
  }
  if (ar.base == nullptr) return 0;
  if (!ar.ok()) return MAK_ERR_WORKSPACE;
  if (n <= 0) return 0;
  if (!direct) {
    const dim3 g((unsigned)ceil_div(n, 256), (unsigned)(n < 16384 ? n : 16384));
    note_launch();
    tri_copy_kernel<T><<<g, 256, 0, st>>>((int)n, R, ldr, Y, skip_flag());
    MAK_CUDA_TRY(cudaGetLastError());
    Arena gj(gjs, gj_bytes);
    MAK_TRY(gje_inverse<T>(st, n, Y, n, iperm, precision, gj, info));
    note_launch();
    tri_gather_kernel<T><<<g, 256, 0, st>>>((int)n, Y, iperm, X, skip_flag());
    MAK_CUDA_TRY(cudaGetLastError());
    return 0;
  }
  const dim3 g((unsigned)ceil_div(n, 256), (unsigned)(n < 16384 ? n : 16384));
  note_launch();
  tri_eye_kernel<T><<<g, 256, 0, st>>>((int)n, X, skip_flag());
  MAK_CUDA_TRY(cudaGetLastError());
  for (int64_t i0 = (n - 1) / TRI_NB * TRI_NB; i0 >= 0; i0 -= TRI_NB) {
    const int64_t nb = (n - i0) < TRI_NB ? (n - i0) : TRI_NB;
    note_launch();
    tri_solve_kernel<T><<<(unsigned)ceil_div(n - i0, TRI_WARPS), 32 * TRI_WARPS, 0, st>>>(
        (int)n, (int)i0, R, ldr, X, &info->singular, skip_flag());
    MAK_CUDA_TRY(cudaGetLastError());
    if (i0 > 0)
      MAK_TRY(gemm<T>(st, i0, n - i0, nb, -one_<T>(), opnd<T>(R + i0 * ldr, ldr),
                      opnd<T>(X + i0 + i0 * n, n), one_<T>(), X + i0 * n, n));
  }
  return 0;
}
#define MAK_INST_TRI(T)                               \
  template bool tri_substitution<T>(int64_t, int);        \
  template int tri_inverse<T>(cudaStream_t, int64_t, const T*, int64_t, T*, int, Arena&, mak_info*);
MAK_INST_TRI(double)
MAK_INST_TRI(float)
MAK_INST_TRI(zcomplex)
MAK_INST_TRI(ccomplex)

// ---- Newton step -----------------------------------------------------------
__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
  atomicMax((unsigned long long*)addr, (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ void atomic_max_nonneg(float* addr, float v) {
  atomicMax((unsigned int*)addr, __float_as_uint(v));
}

// X <- (g X + Y^H/g)/2 with Y^H[i,j] = conj(Xi[j, iperm[i]]) (Xi = eliminated
// inverse), g = (||Xi||_F^2 / ||X||_F^2)^(1/4); *conv = max |Y^H/g - g X|.
template <class T>
__global__ void __launch_bounds__(256) newton_update_kernel(int n, T* X, int64_t ldx,
                                                            const T* Xi, int64_t ldi,
                                                            const int* iperm,
                                                            const real_t<T>* nrm2,
                                                            real_t<T>* conv,
                                                            const int* skip) {
  if (skipped(skip)) return;
  using R = real_t<T>;
  __shared__ T t[32][33];
  __shared__ R sh[32];
  __shared__ R gs[2];
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (threadIdx.x == 0) {  // two roots and two divisions, once per CTA
    gs[0] = sqrt(sqrt(nrm2[1] / nrm2[0]));
    gs[1] = R(1) / gs[0];
  }
  for (int r = ty; r < 32; r += 8) {
    const int i = i0 + r, j = j0 + tx;
    t[r][tx] = (i < n && j < n) ? Xi[j + (int64_t)iperm[i] * ldi] : zero_<T>();  // t[i'][j'] = Xi[j, iperm[i]]
  }
  __syncthreads();
  const R g = gs[0], ginv = gs[1];
  R dmax = R(0);  // complex: of |D|^2, so that no square root is taken per element
  for (int r = ty; r < 32; r += 8) {
    const int i = i0 + tx, j = j0 + r;
    if (i < n && j < n) {
      const T y = conj_(t[tx][r]) * ginv;
      const T x = g * X[i + (int64_t)j * ldx];
      X[i + (int64_t)j * ldx] = R(0.5) * (x + y);
      dmax = fmax(dmax, traits<T>::cpx ? abs2_(y - x) : abs_(y - x));
    }
  }
  dmax = block_max(dmax, sh);
  if (traits<T>::cpx) dmax = sqrt(dmax);
  if (threadIdx.x == 0) atomic_max_nonneg(conv, dmax);
}

// Newton-Schulz finish (mixed precision, Float64 types): once a Newton step
// had ||D||_F <= 1/2 (so ||D||_2 <= 1/2 and the new iterate's singular values
// lie in [1, 1.05]), the iteration continues with
// X <- X (3 I - X^H X) / 2, two products on the split tensor-core path
// instead of a latency-bound Gauss-Jordan inverse; it converges
// quadratically there (error e -> 1.5 e^2).  Its measure 2 max|dX| is on the
// Newton step's scale (max|D| = 2 max|dX|) and meets the same tolerance.
constexpr double NS_SWITCH = 0.5;  // ||D||_F at which Newton-Schulz takes over
// ||D||_F from the two norms: D = Y/g - g X with Y = X^-H and g^2 = ||Y||/||X||,
// and <Y, X> = tr(X^-1 X) = n, so ||D||_F^2 = 2 (||X|| ||Y|| - n); n max|D|
// bounds it from above and decides where rounding hides the difference.
template <class R>
__host__ __device__ inline bool ns_takes_over(R conv, R nx2, R ny2, int64_t n) {
  return (R)n * conv <= (R)NS_SWITCH ||
         R(2) * (sqrt(nx2) * sqrt(ny2) - (R)n) <= (R)(NS_SWITCH * NS_SWITCH);
}

// Z <- 1.5 I - 0.5 Z  (n x n, ld n)
template <class T>
__global__ void ns_prepare_kernel(int n, T* Z, const int* skip) {
  if (skipped(skip)) return;
  using R = real_t<T>;
  const int64_t nn = (int64_t)n * n;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nn;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % n, j = e / n;
    const T d = (i == j) ? make_scalar<T>(R(1.5), R(0)) : zero_<T>();
    Z[e] = d - R(0.5) * Z[e];
  }
}

// X <- Xn and *conv = max(*conv, 2 max|Xn - X|)
template <class T>
__global__ void __launch_bounds__(256) ns_update_kernel(int64_t nn, T* X, const T* Xn,
                                                        real_t<T>* conv, const int* skip) {
  if (skipped(skip)) return;
  using R = real_t<T>;
  __shared__ R sh[32];
  R dmax = R(0);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nn;
       e += (int64_t)gridDim.x * blockDim.x) {
    const T xn = Xn[e];
    dmax = fmax(dmax, abs_(xn - X[e]));
    X[e] = xn;
  }
  dmax = block_max(dmax, sh);
  if (threadIdx.x == 0) atomic_max_nonneg(conv, R(2) * dmax);
}

// Fixed-iteration mode: after each step, count it and stop the loop on the
// device once its measure is within tol (or is not a number), as the
// reference's host loop does; the Newton-Schulz switch is decided here too.
// w: [0] stopped, [1] steps taken, [2] Newton-Schulz phase, [3] skip flag of
// the Newton step's kernels, [4] skip flag of the Newton-Schulz step's.
template <class R>
__global__ void newton_stop_kernel(const R* conv, const R* nrm2, R tol, int* w, R* conv_last,
                                   int n, int ns_ok) {
  if (w[0]) return;
  w[1] += 1;
  *conv_last = *conv;
  if (!(*conv > tol)) w[0] = 1;
  else if (ns_ok && !w[2] && ns_takes_over(*conv, nrm2[0], nrm2[1], (int64_t)n)) w[2] = 1;
  w[3] = w[0] | w[2];
  w[4] = w[0] | !w[2];
}

template <class T>
__global__ void info_polar_fixed_kernel(mak_info* info, const int* stopw,
                                        const real_t<T>* conv_last, real_t<T> tol) {
  info->iterations = stopw[1];
  info->residual = (double)*conv_last;
  info->converged = (*conv_last <= tol) ? 1 : 0;
}

template <class T>
__global__ void info_polar_kernel(mak_info* info, int it, double conv, int converged) {
  info->iterations = it;
  info->residual = conv;
  info->converged = converged;
}

template <class T>
int polar_newton_run(cudaStream_t st, int64_t m, int64_t n, T* A, int64_t lda, T* W, int64_t ldw,
                     T* P, int64_t ldp, int maxiter, double tol, int precision, Arena& ar,
                     mak_info* info) {
  using R = real_t<T>;
  const bool want_p = P != nullptr;
  T* X = ar.take<T>((size_t)n * n + 1);
  T* Y = ar.take<T>((size_t)n * n + 1);
  int* iperm = ar.take<int>(n + 1);
  R* red = ar.take<R>(RED_CTAS + 8);
  int* stopw = ar.take<int>(5);  // fixed-iteration mode: see newton_stop_kernel
  const bool ns_ok = precision == MAK_PREC_MIXED && sizeof(real_t<T>) == 8;
  T* Yn = ns_ok ? ar.take<T>((size_t)n * n + 1) : nullptr;  // Newton-Schulz product
  // Without host synchronization (the batched driver) both step kinds are
  // launched every iteration and flags let one run.  There the finish is
  // used from n >= 256 (MAK_NS_FIXED_MIN_N / _MAX_N override the range):
  // below, the extra launches cost more than the Gauss-Jordan inverses
  // saved.  Measured on the 300 uneven blocks (mixed, CUDA-graph replay, 16
  // streams, tensor-core Gauss-Jordan updates from 2^25): finish for
  // 256 <= n <= 384 only 1.80 s, for every n >= 256 1.54 s.  The
  // host-checked loop launches just the step it takes and uses the finish
  // at every n.
  const double ns_lo = tuning(TUNE_NS_FIXED_MIN_N), ns_hi = tuning(TUNE_NS_FIXED_MAX_N);
  const bool ns_fixed_ok = ns_ok && n >= ns_lo && n <= ns_hi;
  T* Qw = (m > n) ? ar.take<T>((size_t)m * n) : nullptr;
  T* Rw = (m > n) ? ar.take<T>((size_t)n * n) : nullptr;
  T* A0 = (m == n && want_p) ? ar.take<T>((size_t)n * n) : nullptr;
  // the QR (m > n, once) and Gauss-Jordan (every iteration) workspaces are
  // used one after the other, so they share one tail region
  size_t qr_ws = 0, gj_ws = 0;
  if (m > n) {
    Arena meas(nullptr, 0);
    qr_run<T>(st, m, n, nullptr, lda, nullptr, m, n, nullptr, n, n, 1, 0, precision, meas,
              nullptr);
    qr_ws = meas.off + 256;
  }
  {
    Arena meas(nullptr, 0);
    gje_inverse<T>(st, n, nullptr, n, nullptr, precision, meas, nullptr);
    gj_ws = meas.off + 256;
    if (m > n && tri_substitution<T>(n, precision)) {  // the first iterate is triangular
      Arena mt(nullptr, 0);
      tri_inverse<T>(st, n, nullptr, n, nullptr, precision, mt, nullptr);
      if (mt.off + 256 > gj_ws) gj_ws = mt.off + 256;
    }
    for (int64_t mm : {m, n}) {  // W = Q X and P = X^H R products
      Arena m2(nullptr, 0);
      gemm_prec<T>(st, precision, mm, n, n, one_<T>(), opnd<T>(nullptr, 1), opnd<T>(nullptr, 1),
                   zero_<T>(), nullptr, 1, m2, nullptr);
      if (m2.off + 256 > gj_ws) gj_ws = m2.off + 256;
    }
  }
  const size_t tail_bytes = qr_ws > gj_ws ? qr_ws : gj_ws;
  // tol < 0: no host synchronization (graph-capturable); the loop launches
  // maxiter iterations and stops on the device once |tol| is reached
  const bool fixed_iters = tol < 0;
  if (fixed_iters) tol = -tol;
  char* tail = ar.take<char>(tail_bytes);
  if (ar.base == nullptr) return 0;
  if (!ar.ok()) return MAK_ERR_WORKSPACE;
  R* nrm2 = red + RED_CTAS;      // [0] ||X||^2, [1] ||Xi||^2
  R* conv = red + RED_CTAS + 2;  // max |D|
  R* conv_last = red + RED_CTAS + 3;

  if (m > n) {
    Arena sub(tail, tail_bytes);
    MAK_TRY(qr_run<T>(st, m, n, A, lda, Qw, m, n, Rw, n, n, 1, 0, precision, sub, info));
    MAK_TRY(copy_mat<T>(st, n, n, Rw, n, X, n));
  } else {
    if (want_p) MAK_TRY(copy_mat<T>(st, n, n, A, lda, A0, n));
    MAK_TRY(copy_mat<T>(st, n, n, A, lda, X, n));
  }
  int it = 0;
  R hconv = R(0);
  bool converged = (n == 0);
  if (fixed_iters) {
    MAK_CUDA_TRY(cudaMemsetAsync(stopw, 0, 4 * sizeof(int), st));
    MAK_CUDA_TRY(cudaMemsetAsync(stopw + 4, 1, sizeof(int), st));  // non-zero: Newton first
    MAK_CUDA_TRY(cudaMemsetAsync(conv_last, 0, sizeof(R), st));
  }
  const int64_t nn = n * n;
  const unsigned gnn = (unsigned)(ceil_div(nn > 0 ? nn : 1, (int64_t)256) < RED_CTAS
                                      ? ceil_div(nn > 0 ? nn : 1, (int64_t)256)
                                      : RED_CTAS);
  // one Newton step: X <- (g X + X^{-H}/g) / 2, measure max|D| into conv.  The
  // first iterate of a tall A is the triangular R.
  const bool tri_first = m > n && tri_substitution<T>(n, precision);
  auto newton_step = [&](bool triangular) -> int {
    if (triangular) {
      Arena sub(tail, tail_bytes);
      MAK_TRY(tri_inverse<T>(st, n, X, n, Y, precision, sub, info));
      note_launch();
      iota_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>((int)n, iperm, iperm);
      MAK_CUDA_TRY(cudaGetLastError());
    } else {
      MAK_TRY(copy_mat<T>(st, n, n, X, n, Y, n));
      Arena sub(tail, tail_bytes);
      MAK_TRY(gje_inverse<T>(st, n, Y, n, iperm, precision, sub, info));
    }
    MAK_TRY(reduce_mat<T>(st, n, n, X, n, 0, red, nrm2));
    MAK_TRY(reduce_mat<T>(st, n, n, Y, n, 0, red, nrm2 + 1));
    dim3 g((unsigned)ceil_div(n, 32), (unsigned)ceil_div(n, 32));
    note_launch();
    newton_update_kernel<T><<<g, 256, 0, st>>>((int)n, X, n, Y, n, iperm, nrm2, conv,
                                               skip_flag());
    return cudaGetLastError() == cudaSuccess ? 0 : MAK_ERR_CUDA;
  };
  // one Newton-Schulz step: X <- X (3 I - X^H X) / 2 (Y holds X^H X, then
  // 1.5 I - 0.5 X^H X), measure 2 max|dX| into conv
  auto ns_step = [&]() -> int {
    {
      Arena oz(tail, tail_bytes);
      MAK_TRY(gemm_prec<T>(st, precision, n, n, n, one_<T>(), opnd<T>(X, n, OP_C), opnd<T>(X, n),
                           zero_<T>(), Y, n, oz, &info->status));
    }
    note_launch();
    ns_prepare_kernel<T><<<gnn, 256, 0, st>>>((int)n, Y, skip_flag());
    MAK_CUDA_TRY(cudaGetLastError());
    {
      Arena oz(tail, tail_bytes);
      MAK_TRY(gemm_prec<T>(st, precision, n, n, n, one_<T>(), opnd<T>(X, n), opnd<T>(Y, n),
                           zero_<T>(), Yn, n, oz, &info->status));
    }
    note_launch();
    ns_update_kernel<T><<<gnn, 256, 0, st>>>(nn, X, Yn, conv, skip_flag());
    return cudaGetLastError() == cudaSuccess ? 0 : MAK_ERR_CUDA;
  };
  bool in_ns = false;  // tolerance mode: the host decides the phase
  for (it = 1; it <= maxiter && n > 0; it++) {
    MAK_CUDA_TRY(cudaMemsetAsync(conv, 0, sizeof(R), st));
    if (fixed_iters) {
      // both step kinds are launched; device flags let exactly one run (and
      // neither once the loop has stopped)
      {
        SkipScope skip_newton(stopw + 3);
        MAK_TRY(newton_step(it == 1 && tri_first));
      }
      if (ns_fixed_ok) {
        SkipScope skip_ns(stopw + 4);
        MAK_TRY(ns_step());
      }
      note_launch();
      newton_stop_kernel<R><<<1, 1, 0, st>>>(conv, nrm2, (R)tol, stopw, conv_last, (int)n,
                                             ns_fixed_ok ? 1 : 0);
      MAK_CUDA_TRY(cudaGetLastError());
    } else {
      MAK_TRY(in_ns ? ns_step() : newton_step(it == 1 && tri_first));
      R h[3];  // the two squared norms and max|D|
      MAK_CUDA_TRY(cudaMemcpyAsync(h, nrm2, sizeof(h), cudaMemcpyDeviceToHost, st));
      MAK_CUDA_TRY(cudaStreamSynchronize(st));
      hconv = h[2];
      if (!(hconv > (R)tol)) {  // also stops on NaN
        converged = hconv <= (R)tol;
        break;
      }
      if (ns_ok && !in_ns && ns_takes_over(hconv, h[0], h[1], n)) in_ns = true;
    }
  }
  if (it > maxiter) it = maxiter;
  note_launch();
  if (fixed_iters)
    info_polar_fixed_kernel<T><<<1, 1, 0, st>>>(info, stopw, conv_last, (R)tol);
  else
    info_polar_kernel<T><<<1, 1, 0, st>>>(info, n > 0 ? it : 0, (double)hconv, converged ? 1 : 0);
  MAK_CUDA_TRY(cudaGetLastError());

  auto G = [&](int64_t M_, int64_t N_, int64_t K_, Operand<T> a, Operand<T> b, T* C_,
               int64_t ldc) -> int {
    Arena oz(tail, tail_bytes);
    return gemm_prec<T>(st, precision, M_, N_, K_, one_<T>(), a, b, zero_<T>(), C_, ldc, oz,
                        &info->status);
  };
  if (m > n) {
    MAK_TRY(G(m, n, n, opnd<T>(Qw, m), opnd<T>(X, n), W, ldw));
    if (want_p) {
      MAK_TRY(G(n, n, n, opnd<T>(X, n, OP_C), opnd<T>(Rw, n, OP_N, MASK_UPPER), P, ldp));
      MAK_TRY(herm_project<T>(st, n, P, ldp));
    }
  } else {
    MAK_TRY(copy_mat<T>(st, n, n, X, n, W, ldw));
    if (want_p) {
      MAK_TRY(G(n, n, n, opnd<T>(X, n, OP_C), opnd<T>(A0, n), P, ldp));
      MAK_TRY(herm_project<T>(st, n, P, ldp));
    }
  }
  return 0;
}

#define MAK_INST_POLAR(T)                                                                     \
  template int gje_inverse<T>(cudaStream_t, int64_t, T*, int64_t, int*, int, Arena&,          \
                              mak_info*);                                                     \
  template int polar_newton_run<T>(cudaStream_t, int64_t, int64_t, T*, int64_t, T*, int64_t, \
                                   T*, int64_t, int, double, int, Arena&, mak_info*);
MAK_INST_POLAR(double)
MAK_INST_POLAR(float)
MAK_INST_POLAR(zcomplex)
MAK_INST_POLAR(ccomplex)

template <class T>
static double default_tol() {
  // defaulttol = eps(real T)^(2/3)  (src/common/defaults.jl:10)
  return pow(sizeof(real_t<T>) == 8 ? 2.220446049250313e-16 : 1.1920928955078125e-7, 2.0 / 3.0);
}

template <class T>
static int polar_entry(int64_t m, int64_t n, void* Av, int64_t lda, void* Wv, int64_t ldw,
                       void* Pv, int64_t ldp, const mak_polar_opts* opts, void* work,
                       size_t work_bytes, mak_info* info, mak_stream_t stream) {
  T* A = (T*)Av;
  T* W = (T*)Wv;
  T* P = (T*)Pv;
  if (m < 0) return -1;
  if (n < 0 || n > m) return -2;  // m >= n required (polar.jl:9-10)
  if (A == nullptr && m * n > 0) return -3;
  if (lda < (m > 1 ? m : 1)) return -4;
  if (W == nullptr && m * n > 0) return -5;
  if ((void*)W == (void*)A && m * n > 0) return -5;
  if (ldw < (m > 1 ? m : 1)) return -6;
  if (P != nullptr && ldp < (n > 1 ? n : 1)) return -8;
  mak_polar_opts o{10, MAK_PREC_NATIVE, 0.0};
  if (opts) o = *opts;
  if (o.maxiter < 1) return -9;
  if (o.precision != MAK_PREC_NATIVE && o.precision != MAK_PREC_MIXED) return -9;
  // tol < 0 selects the fixed-iteration (no host sync) mode, reported
  // against the default tolerance
  const double tol = o.tol > 0 ? o.tol : (o.tol < 0 ? -default_tol<T>() : default_tol<T>());
  if (info == nullptr) return -12;
  cudaStream_t st = (cudaStream_t)stream;
  {
    Arena meas(nullptr, 0);
    polar_newton_run<T>(st, m, n, nullptr, lda, nullptr, ldw, P, ldp, o.maxiter, tol, o.precision,
                        meas, nullptr);
    if (meas.off > work_bytes) return -11;
  }
  Arena ar(work, work_bytes);
  MAK_TRY(info_reset(st, info));
  return polar_newton_run<T>(st, m, n, A, lda, W, ldw, P, ldp, o.maxiter, tol, o.precision, ar,
                             info);
}

}  // namespace mak

using namespace mak;

extern "C" {

int mak_left_polar_workspace(int dtype, int64_t m, int64_t n, int want_p,
                             const mak_polar_opts* opts, size_t* bytes) {
  if (bytes == nullptr) return -6;
  if (m < 0) return -2;
  if (n < 0 || n > m) return -3;
  mak_polar_opts o{10, MAK_PREC_NATIVE, 0.0};
  if (opts) o = *opts;
  Arena meas(nullptr, 0);
  void* P = want_p ? (void*)16 : nullptr;  // only nullness matters when measuring
  switch (dtype) {
    case MAK_F64: polar_newton_run<double>(0, m, n, nullptr, m, nullptr, m, (double*)P, n, o.maxiter, 1.0, o.precision, meas, nullptr); break;
    case MAK_C64: polar_newton_run<zcomplex>(0, m, n, nullptr, m, nullptr, m, (zcomplex*)P, n, o.maxiter, 1.0, o.precision, meas, nullptr); break;
    case MAK_F32: polar_newton_run<float>(0, m, n, nullptr, m, nullptr, m, (float*)P, n, o.maxiter, 1.0, o.precision, meas, nullptr); break;
    case MAK_C32: polar_newton_run<ccomplex>(0, m, n, nullptr, m, nullptr, m, (ccomplex*)P, n, o.maxiter, 1.0, o.precision, meas, nullptr); break;
    default: return -1;
  }
  *bytes = meas.off + 256;
  return 0;
}

#define MAK_POLAR_ENTRY(NAME, T, PT)                                                            \
  int NAME(int64_t m, int64_t n, PT* A, int64_t lda, PT* W, int64_t ldw, PT* P, int64_t ldp,    \
           const mak_polar_opts* opts, void* work, size_t work_bytes, mak_info* info,           \
           mak_stream_t stream) {                                                               \
    return polar_entry<T>(m, n, A, lda, W, ldw, P, ldp, opts, work, work_bytes, info, stream); \
  }
MAK_POLAR_ENTRY(mak_left_polar_newton_d, double, double)
MAK_POLAR_ENTRY(mak_left_polar_newton_z, zcomplex, void)
MAK_POLAR_ENTRY(mak_left_polar_newton_s, float, float)
MAK_POLAR_ENTRY(mak_left_polar_newton_c, ccomplex, void)

}  // extern "C"
