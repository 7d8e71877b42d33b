// Blocked Householder QR with positive-diagonal gauge, GB300 native.
//
// Replaces the reference's LAPACK/cuSOLVER path
//   qr_householder!  (src/implementations/qr.jl:132-188)
//   = geqrt!/geqrf!  (panel + T factor, src/yalapack.jl:303-333 / 168-199)
//   + gemqrt!/unmqr! on one!(Q)  (Q formation, src/yalapack.jl:882-927)
//   + uppertriangular! R copy   (src/common/initialization.jl:18-26)
//   + gaugefix!(qr_householder!) (src/common/gauge.jl:16-25, sign_safe
//     src/common/safemethods.jl:10-11)
//
// Structure on the device, per panel of jb <= 32 columns starting at j0:
//  1. qr_panel_kernel: ONE launch factors the (m-j0) x jb panel: a
//     thread-block cluster of up to 16 CTAs for panels of up to 8 x 256 rows
//     (hardware cluster barrier; clusters of different streams run side by
//     side, which the batched driver relies on), a cooperative grid of up to
//     one CTA per SM beyond that (bounded global barrier).
//     Each CTA keeps a contiguous slab of panel rows resident in shared
//     memory for the whole panel; a column costs one barrier:
//     the reflector norm and the dot products of the still unscaled column
//     with the columns to its right are published together, and w = v^H A
//     follows from them once beta/tau are known.  Norms are plain sums of
//     squares with a rescaled two-round path when the largest magnitude is
//     outside a safe range, and every cross-CTA reduction is done in a fixed
//     order, so all CTAs derive bit-identical beta/tau/w.  The panel's Gram
//     matrix V^H V is reduced at the end and the CTAs form the T factor's
//     columns (forward, column-wise larft recurrence).  Panels whose columns
//     are far from dependent take ONE round for all columns instead
//     (panel_block_round).
//  2. larfb on the trailing columns:  W = V^H C (split-K GEMM, V read in
//     place through a unit-lower mask), W2 = T^H W (reduce_trmm_kernel),
//     C -= V W2 (GEMM).
// Q is then accumulated backwards (orgqr order, exploiting the identity
// structure: block b only touches Q[j0:, j0:]) starting from [diag(s); 0]
// where s = sign_safe(diag R): the gauge fix Q <- Q diag(s) is folded into the
// starting matrix because Q diag(s) = H_1...H_k [diag(s); 0].  R is written
// once, already multiplied by conj(s) row-wise.
#include "gemm.cuh"
#include "householder.cuh"
#include "internal.h"
#include "util.cuh"

#include <cstdlib>
#include <mutex>

namespace mak {

constexpr int NBMAX = 32;      // widest panel handled by one cooperative launch
constexpr int PANEL_THREADS = 256;

template <class T>
struct PanelArgs {
  T* A;                 // panel (row j0, col j0) of the packed matrix
  int64_t lda;
  int mp;               // panel rows
  int jb;               // panel columns
  int rpc;              // panel rows owned by one CTA
  T* tau;               // [jb]
  T* Tm;                // [NBMAX x NBMAX], ld NBMAX
  real_t<T>* part_nrm;  // [2][3][gstride] by round parity (sums of squares, largest
                        // magnitudes of columns j and j+1), then [gstride] rescaled sums
  T* part_w;            // [2][gstride][NBMAX] dot partials by round parity, then
                        // [gstride][NBMAX] for the rescaled path, then
                        // [2][gstride][NBMAX] column j+1's dot partials (pair rounds)
  T* part_g;            // [G][NBMAX*NBMAX]
  T* alpha_buf;         // [2][NBMAX]: row j of the panel by round parity, then
                        // [2][NBMAX] row j+1 (pair rounds)
  T* gram;              // [NBMAX*NBMAX]: the panel's reduced Gram matrix V^H V
  unsigned* bar;        // grid barrier words
  int* cflag;           // [gstride] outcome of the last global round, per cluster (SYNC_HIER)
  int* status;
  int gstride;          // allocation stride of the per-CTA partial rows
  int pair;             // two columns per barrier round where the norms allow
  int block;            // the whole panel in one round where its conditioning allows (the
                        // launch's shared memory then has block_extra_bytes after the slab)
};

// ---- block round: the whole panel from one Gram matrix -----------------------
// The pair rounds below form two reflectors per barrier from the Gram entries
// of two columns.  When the panel's columns are far from dependent, all of
// them follow from ONE round: with G = A^H A of the panel (rows >= j0),
// column j's |beta_j| and the row R_jc = G_jc / beta_j are one step of the
// Cholesky factorization of G, and the reflectors follow from the panel's top
// jb x jb block alone (Householder reconstruction, G. Ballard et al.,
// "Reconstructing Householder vectors from TSQR", 2014): with s_j =
// -sign(Re alpha_j), beta_j = s_j |beta_j|,
//   F_jc = T0_jc - R_jc (c > j),  F_jj = alpha_j - beta_j,
//   v_ij = T0_ij / F_jj,  T0_ic -= v_ij F_jc   (i > j),
// an LU elimination of the top block whose rows are shifted by R, since
// A = V F + [R; 0].  The rows below the top block follow by substitution,
// V_bot = A_bot F^-1, and the T factor from A = (I - V T V^H) [R; 0]:
// T = -F R^-1 V_top^-H.
//
// The Gram entries carry an error of eps |a_j| |a_c|, which R's inverse
// amplifies: with R' the factor of the panel with columns of norm one, Q^H Q
// - I is of the order of eps ||R'^-1||^2.  Every pivot well above zero does
// not bound that (32 columns that each keep half their squared norm can reach
// cond(R') = 10^4), so the round is taken only if every column keeps at least
// half its squared norm after the columns before it are projected out (the
// factorization of G is then safe to finish) and ||R'^-1||_F^2, formed from
// the finished factor, is at most BLK_INV_LIMIT per column; and if every
// squared norm is finite and far from overflow and underflow.  Every CTA
// repeats the jb x jb work on identical numbers, so all of them take the same
// branch; nothing has been written when a test fails, and the panel is
// factored column by column as before.
//
// Bound: FP64 throughput (about 1.6 DFMA per clock per SM): rows x jb^2 / 2
// multiply-adds for G and as many for V_bot, spread over the CTAs, plus the
// jb x jb work, a chain of dependent FP64 operations of about 0.8 us per
// column.  1000 x 501 Float64 QR 7.40 -> 4.52 ms, 2049 x 1000 full mixed QR
// 19.0 -> 11.0 ms, 300 uneven blocks 257 -> 188 ms against the pair rounds
// (a 1000-row panel: 236 us before, 80 us on 8 CTAs and 60 us on 16 now).
constexpr int BLK_TILES = 36;   // 4 x 4 tiles of the upper triangle of a 32 x 32 Gram matrix
constexpr int BLK_ROWGRP = 7;   // row groups: 36 x 7 = 252 of the 256 threads
constexpr int BLK_LD = NBMAX + 1;
constexpr int BLK_MIN_COLS = 8;
constexpr int BLK_MIN_MP_PER_COL = 3;  // fewer rows per column rarely pass the test
// ||R'^-1||_F^2 per column: the mean over the columns of their squared norm
// over their squared distance from the span of the others; about mp / (mp -
// jb) for Gaussian columns, 1.5 for three rows per column (96 x 32: 1.4 - 1.6).
// ||Q^H Q - I||_2 of accepted 32-column panels over that of the column rounds,
// 96 to 9000 rows, Float64 (Float32): 1.0 - 1.1 0.7 - 1.5 (1.7), 1.3 1.2 - 1.8
// (3.9), 1.6 0.7 - 2.5 (4.1), 2.0 1.0 - 1.5 (2.1), 2.7 2 - 6.5 (8), 4.4 4 - 8
// (6), 28 30 - 180 (70).  Columns correlated by 0.6 with the next one (2.1 -
// 2.4) are refused: 1000 x 501 Float64 2.63 ms accepted, 5.55 refused, 7.4 by
// column rounds on 8 CTAs without the round.
constexpr float BLK_INV_LIMIT = 2.0f;
template <class T>
constexpr size_t block_extra_bytes() {
  // partial Gram tiles, G / L / scaled F (one square), top block, a pair's raw
  // rows by step, 1 / F_jj; four vectors of reals; the steps' failures and the
  // four warps' parts of ||R'^-1||_F^2.  All
  // behind the slab, not static: static shared memory would take rows from the
  // slab of every panel, and with them from the tallest matrix there is.
  return sizeof(T) * (size_t)(BLK_TILES * 16 + 2 * NBMAX * BLK_LD + 9 * NBMAX) +
         sizeof(real_t<T>) * 4 * NBMAX + sizeof(int) * (NBMAX + 8);
}
__device__ __forceinline__ void blk_tile(int t, int& bi, int& bj) {
  bj = 0;
  while ((bj + 1) * (bj + 2) / 2 <= t) bj++;
  bi = t - bj * (bj + 1) / 2;
}

// x 2^e as a float, for results below 2^127 (e.g. ratios of the panel's column
// norms taken out of an entry of its factor); integer operations only, so that
// the FP64 pipe is left to the recurrence that runs beside it
__device__ __forceinline__ float narrow_exp(double x, int e) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int ex = (int)((hi >> 20) & 0x7FFu) - 1023 + 127 + e;
  if (ex <= 0) return 0.0f;
  return __uint_as_float((hi & 0x80000000u) | (unsigned)(ex < 254 ? ex : 254) << 23 |
                         (hi & 0xFFFFFu) << 3 | lo >> 29);
}
__device__ __forceinline__ float narrow_exp(float x, int e) { return x * pow2_(0.0f, e); }
template <class R> __device__ __forceinline__ cplx<float> narrow_exp(cplx<R> x, int e) {
  return {narrow_exp(x.re, e), narrow_exp(x.im, e)};
}
__device__ __forceinline__ float sq_(float x) { return x * x; }
__device__ __forceinline__ float sq_(cplx<float> x) { return fmaf(x.re, x.re, x.im * x.im); }

// Warp w4's part of ||R'^-1||_F^2 (lane = row): R' = D'^1/2 U with U_ik = L_ik
// |a_i| / |a_k| unit upper triangular and D'_c = D_c / |a_c|^2, so the columns
// c = w4, w4 + 4, ... of U^-1 by substitution, each divided by D'_c.  In FP32,
// which is enough: a norm below the limit is that of a matrix within 32
// 2^-23 |U| of U, and those of the panels refused need no digits.  Beside the
// elimination's last steps it costs 0.5 us per panel (Float32 1.3); after them
// 4 us (Float32 2).
template <class T>
__device__ __forceinline__ float panel_inverse_norm2(const T* Gs, const real_t<T>* dg, int jb,
                                                     int w4) {
  using F = typename std::conditional<traits<T>::cpx, cplx<float>, float>::type;
  const int lane = threadIdx.x & 31;
  const int ic = min(lane, jb - 1);
  const int E = exp2_of(dg[ic]) >> 1;               // |a_i| = 2^E times [1, 2)
  const float m = narrow_exp(dg[ic], -2 * E);
  const float rs = rsqrtf(m), s = m * rs;
  const float w = __fdividef(m, narrow_exp(re_(Gs[ic * BLK_LD + ic]), -2 * E));  // 1 / D'
  F x[NBMAX / 4];
#pragma unroll
  for (int q = 0; q < NBMAX / 4; q++) x[q] = lane == w4 + 4 * q ? one_<F>() : zero_<F>();
  // a small body, not unrolled: the code runs once per panel, and fetching it
  // costs more than its arithmetic; the next row is read ahead of the chain
  T g = lane < jb - 1 ? Gs[lane * BLK_LD + jb - 1] : zero_<T>();
#pragma unroll 1
  for (int k = jb - 1; k > 0; k--) {
    const int Ek = __shfl_sync(0xffffffffu, E, k);
    const float sk = s * __shfl_sync(0xffffffffu, rs, k);
    const F u = lane < k ? narrow_exp(g, E - Ek) * sk : zero_<F>();
    g = lane < k - 1 ? Gs[lane * BLK_LD + k - 1] : zero_<T>();
#pragma unroll
    for (int q = 0; q < NBMAX / 4; q++) x[q] = fma_(-u, shfl_idx_(x[q], k), x[q]);
  }
  float sum = 0.0f;
#pragma unroll
  for (int q = 0; q < NBMAX / 4; q++) {
    const int c = w4 + 4 * q;
    const float wc = __shfl_sync(0xffffffffu, w, c);
    if (c < jb) sum = fmaf(sq_(x[q]), wc, sum);
  }
  return warp_sum(sum);
}

// 1: the panel is factored and stored; 0: not taken (nothing written);
// -1: a bounded barrier gave up
template <class T, int SYNC>
__device__ __forceinline__ int panel_block_round(const PanelArgs<T>& a, T* Ps, int ldp, int r0, int nr,
                                 unsigned char* extra) {
  using R = real_t<T>;
  constexpr bool kCl = SYNC == SYNC_CLUSTER;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int b = blockIdx.x, G = gridDim.x, jb = a.jb;
  T* Gp = reinterpret_cast<T*>(extra);       // [36][4][4] this CTA's partial Gram
  T* Gs = Gp + BLK_TILES * 16;               // upper: G, then D and L; lower: F_jc / F_jj, transposed
  T* T0 = Gs + NBMAX * BLK_LD;               // lower: V_top; upper: F
  T(*raw)[2][NBMAX] = reinterpret_cast<T(*)[2][NBMAX]>(T0 + NBMAX * BLK_LD);  // [4]: a pair's rows of
                                                                 // G before they are scaled, by step
  T* scl = &raw[4][0][0];                    // 1 / F_jj
  R* dg = reinterpret_cast<R*>(scl + NBMAX); // squared norms of the panel's columns
  R* rsv = dg + NBMAX;                       // 1 / |beta_j|
  R* nrm_s = rsv + NBMAX;                    // |beta_j|
  R* sgn_s = nrm_s + NBMAX;                  // sign of beta_j
  int* fail_s = reinterpret_cast<int*>(sgn_s + NBMAX);  // per step, and [NBMAX]: the norms' range
  float* inv2_s = reinterpret_cast<float*>(fail_s + NBMAX + 1);  // [4] parts of ||R'^-1||_F^2
  // the top block, straight from the (still unmodified) panel
  T top[NBMAX / 8];
#pragma unroll
  for (int q = 0; q < NBMAX / 8; q++) {
    const int c = wid + q * nw;
    top[q] = (lane < jb && c < jb) ? ld_cg(&a.A[lane + (int64_t)c * a.lda]) : zero_<T>();
  }
  if (tid <= NBMAX) fail_s[tid] = 0;

  // ---- partial Gram over this CTA's rows: one 4 x 4 tile per thread and row
  // group, the groups folded in order
  {
    const int t = tid % BLK_TILES, grp = tid / BLK_TILES;
    int bi, bj;
    blk_tile(t, bi, bj);
    T acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[p][q] = zero_<T>();
    if (grp < BLK_ROWGRP) {
      const T *pi[4], *pj[4];
#pragma unroll
      for (int p = 0; p < 4; p++) {
        pi[p] = Ps + min(4 * bi + p, jb - 1) * ldp;
        pj[p] = Ps + min(4 * bj + p, jb - 1) * ldp;
      }
      for (int r = grp; r < nr; r += BLK_ROWGRP) {
        T x[4], y[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
          x[p] = conj_(pi[p][r]);
          y[p] = pj[p][r];
        }
#pragma unroll
        for (int p = 0; p < 4; p++)
#pragma unroll
          for (int q = 0; q < 4; q++) acc[p][q] = fma_(x[p], y[q], acc[p][q]);
      }
    }
    // fold the row groups: 0-3 into four buffers (the later three over the
    // squares, which are filled afterwards), 4-6 added to the first three
    T* const buf[4] = {Gp, Gs, Gs + BLK_TILES * 16, Gs + 2 * BLK_TILES * 16};
    T* dst = grp < 4 ? buf[grp] : buf[(grp - 4) & 3];
    if (grp < 4) {
#pragma unroll
      for (int p = 0; p < 16; p++) dst[t * 16 + p] = acc[p >> 2][p & 3];
    }
    __syncthreads();
    if (grp >= 4 && grp < BLK_ROWGRP) {
#pragma unroll
      for (int p = 0; p < 16; p++) dst[t * 16 + p] += acc[p >> 2][p & 3];
    }
    __syncthreads();
    for (int e = tid; e < BLK_TILES * 16; e += blockDim.x)
      Gp[e] = (Gp[e] + buf[1][e]) + (buf[2][e] + buf[3][e]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NBMAX / 8; q++) T0[lane * BLK_LD + wid + q * nw] = top[q];
  }
  // ---- sum over the CTAs in a fixed order, the same bits in every CTA
  if constexpr (kCl) {
    cluster_sync_all();
    for (int e = tid; e < BLK_TILES * 16; e += blockDim.x) {
      T s = zero_<T>();
      for (int q0 = 0; q0 < G; q0 += 8) {
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; q++)
          v[q] = q0 + q < G ? dsmem_ld(&Gp[e], (unsigned)(q0 + q)) : zero_<T>();
#pragma unroll
        for (int q = 0; q < 8; q++) s += v[q];
      }
      int bi, bj;
      blk_tile(e >> 4, bi, bj);
      const int d = 4 * bi + ((e >> 2) & 3), c = 4 * bj + (e & 3);
      if (d <= c) Gs[d * BLK_LD + c] = s;
    }
    // from here on no CTA reads another's shared memory; the barrier's second
    // half comes before anything the other CTAs may still read is rewritten
    cluster_arrive();
  } else {
    for (int e = tid; e < BLK_TILES * 16; e += blockDim.x)
      a.part_g[(int64_t)b * NBMAX * NBMAX + e] = Gp[e];
    if (!panel_sync<SYNC>(a.bar, G, a.status)) return -1;
    // one warp per entry
    for (int e = b * nw + wid; e < BLK_TILES * 16; e += G * nw) {
      T s = zero_<T>();
      for (int q = lane; q < G; q += 32) s += ld_cg(&a.part_g[(int64_t)q * NBMAX * NBMAX + e]);
      s = warp_sum(s);
      if (lane == 0) a.gram[e] = s;
    }
    if (!panel_sync<SYNC>(a.bar, G, a.status)) return -1;
    for (int e = tid; e < BLK_TILES * 16; e += blockDim.x) {
      int bi, bj;
      blk_tile(e >> 4, bi, bj);
      const int d = 4 * bi + ((e >> 2) & 3), c = 4 * bj + (e & 3);
      if (d <= c) Gs[d * BLK_LD + c] = ld_cg(&a.gram[e]);
    }
  }
  __syncthreads();
  if (wid == 0) {
    const R g = lane < jb ? re_(Gs[lane * BLK_LD + lane]) : R(1);
    const int lim = sizeof(R) == 8 ? 900 : 90;
    const int e = exp2_of(g);
    if (!(g > R(0) && finite_(g) && e > -lim && e < lim)) fail_s[NBMAX] = 1;
    dg[lane] = g;
  }
  __syncthreads();
  int failed = fail_s[NBMAX];

  // ---- warps 0-3: G = L^H D L (L unit upper), then |beta_j| = sqrt(D_j), one
  // step behind; warps 4-7: the elimination of the top block, two steps
  // behind.  A step takes the column pair 2P, 2P + 1, whose two rows one warp
  // owns (pair P: warp P mod 4 of each group; lane = column): the owner forms
  // both in registers and publishes them, a barrier follows, then the other
  // rows.  On GB300 a dependent FP64 operation takes 61 cycles (measured) and a
  // warp-wide one holds its sub-partition's FP64 pipe for 64, so the chains
  // are kept short (four operations from D_j to D_{j+1} with no square root
  // between them, five from alpha_j to alpha_{j+1}), and the next owner
  // updates only the pair it needs before it goes on, the rest of its rows a
  // step later.
  if (!failed) {
    const int w4 = wid & 3;
    const bool chol = wid < 4;
    const int np = (jb + 1) >> 1;
    // one step of G = L^H D L on row g (lanes >= j): D_j returned, L_j in l
    auto chol_row = [&](T g, int j, T& l) -> bool {
      const R d = shfl_idx_(re_(g), j);
      if (!(d >= R(0.5) * dg[j])) return false;
      const R y = rcp_seed(d);
      const R r = fma_(-d, y, R(1));
      l = fma_real_(g * y, fma_(r, r, r));
      return true;
    };
    // one step of the elimination on the top block's row t (current, lanes =
    // columns): F_j (lanes >= j) over t, F_jc / F_jj in fn (lanes > j).  The
    // sign of beta_j is opposite to alpha_j's real part.
    auto lu_row = [&](T& t, int j, T& fn) {
      const T alpha = shfl_idx_(t, j);
      const R nrm = nrm_s[j];
      const R sg = re_(alpha) >= R(0) ? R(-1) : R(1);
      const R bj = sg * nrm;
      const T fjj = alpha - make_scalar<T>(bj, R(0));
      const T f = lane > j ? t - Gs[j * BLK_LD + lane] * bj : zero_<T>();
      T y;
      R p;
      if constexpr (traits<T>::cpx) {
        const R z2 = fma_(fjj.re, fjj.re, fjj.im * fjj.im);
        const R y0 = rcp_seed(z2);
        const R r = fma_(-z2, y0, R(1));
        p = fma_(r, r, r);
        y = conj_(fjj) * y0;
      } else {
        y = rcp_seed(fjj);
        const R r = fma_(-fjj, y, R(1));
        p = fma_(r, r, r);
      }
      fn = fma_real_(f * y, p);
      if (lane > j) t = f;
      if (lane == j) {
        t = fjj;
        sgn_s[j] = sg;
        scl[j] = fma_real_(y, p);
      }
    };
#pragma unroll 1
    for (int it = 0; it < np + 2; it++) {
      const int P = chol ? it : it - 2;
      const bool live = P >= 0 && P < np;
      const int j0 = 2 * P, j1 = j0 + 1;
      const bool two = j1 < jb;
      if (live && w4 == (P & 3)) {
        if (chol) {
          T* const G0 = Gs + j0 * BLK_LD;
          T* const G1 = G0 + BLK_LD;
          const T g0 = lane >= j0 ? G0[lane] : zero_<T>();
          T l0 = zero_<T>(), l1 = zero_<T>(), g1 = zero_<T>();
          bool ok = chol_row(g0, j0, l0);
          if (two && ok) {
            const T f = conj_(shfl_idx_(g0, j1));
            g1 = lane >= j1 ? fma_(-f, l0, G1[lane]) : zero_<T>();
            ok = chol_row(g1, j1, l1);
          }
          if (!ok) {
            if (lane == 0) fail_s[P] = 1;
          } else {
            raw[P & 3][0][lane] = g0;
            raw[P & 3][1][lane] = g1;
            if (lane > j0) G0[lane] = l0;
            if (two && lane >= j1) G1[lane] = lane == j1 ? g1 : l1;
          }
        } else {
          T* const t0p = T0 + j0 * BLK_LD;
          T t0 = t0p[lane], t1 = two ? t0p[BLK_LD + lane] : zero_<T>(), fn;
          lu_row(t0, j0, fn);
          t0p[lane] = t0;
          if (lane > j0) Gs[lane * BLK_LD + j0] = fn;
          if (two) {
            const T e = shfl_idx_(t1, j0);
            if (lane > j0) t1 = fma_(-e, fn, t1);
            lu_row(t1, j1, fn);
            t0p[BLK_LD + lane] = t1;
            if (lane > j1) Gs[lane * BLK_LD + j1] = fn;
          }
        }
      }
      if (chol && it >= 1 && it <= np && w4 == ((it + 2) & 3)) {
        const int j = 2 * (it - 1) + (lane & 1);
        if (j < jb) {
          const R d = re_(Gs[j * BLK_LD + j]);
          const R rs = rsqrt_b3(d), s = d * rs;
          if (lane < 2) {
            nrm_s[j] = fma_(fma_(-s, s, d), R(0.5) * rs, s);  // sqrt(d), corrected
            rsv[j] = rs;
          }
        }
      }
      // L and D are complete: while the elimination takes its last two steps,
      // warps 0-3 look at the whole factor
      if (it >= np) {
        if (chol) {
          asm volatile("bar.arrive 2, %0;" ::"n"(PANEL_THREADS) : "memory");  // the last |beta_j|
          const float v = panel_inverse_norm2<T>(Gs, dg, jb, w4);
          if (lane == 0) inv2_s[w4] = v;
          break;
        }
        if (it == np) asm volatile("bar.sync 2, %0;" ::"n"(PANEL_THREADS) : "memory");
      } else {
        __syncthreads();
      }
      // this step's flag (written by its owner before the barrier; one word
      // per step, so that a later step's owner cannot race a slow reader)
      if (it < np && fail_s[it]) {
        failed = 1;
        break;
      }
      if (!live) continue;
      // the rows below: the next owner its next pair only; this step's owner
      // its remaining pairs with the previous step's columns and this step's
      const bool next = w4 == ((P + 1) & 3), prev = w4 == (P & 3) && P > 0;
      const int pend = next ? min(P + 2, np) : np;
      for (int p = P + 1 + ((w4 - P - 1) & 3); p < pend; p += 4) {
        const int d0 = 2 * p, d1 = d0 + 1;
        if (chol) {
          T* const X = Gs + d0 * BLK_LD;
          T a0 = X[lane], a1 = d1 < jb ? X[BLK_LD + lane] : zero_<T>();
          for (int q = prev ? P - 1 : P; q <= P; q++) {
            const T l0 = Gs[2 * q * BLK_LD + lane], l1 = Gs[(2 * q + 1) * BLK_LD + lane];
            const T* r0p = raw[q & 3][0];
            const T* r1p = raw[q & 3][1];
            a0 = fma_(-conj_(r0p[d0]), l0, a0);
            a1 = fma_(-conj_(r0p[d1]), l0, a1);
            a0 = fma_(-conj_(r1p[d0]), l1, a0);
            a1 = fma_(-conj_(r1p[d1]), l1, a1);
          }
          if (lane >= d0) X[lane] = a0;
          if (lane >= d1 && d1 < jb) X[BLK_LD + lane] = a1;
        } else {
          T* const X = T0 + d0 * BLK_LD;
          T a0 = X[lane], a1 = d1 < jb ? X[BLK_LD + lane] : zero_<T>();
          for (int q = prev ? 2 * (P - 1) : 2 * P; q <= 2 * P + 1; q++) {
            const T fn = lane > q ? Gs[lane * BLK_LD + q] : zero_<T>();
            const T e0 = shfl_idx_(a0, q), e1 = shfl_idx_(a1, q);
            a0 = fma_(-e0, fn, a0);
            a1 = fma_(-e1, fn, a1);
          }
          X[lane] = a0;
          if (d1 < jb) X[BLK_LD + lane] = a1;
        }
      }
    }
  }
  if constexpr (kCl) cluster_wait();
  if (failed) return 0;
  __syncthreads();
  if (!((inv2_s[0] + inv2_s[1]) + (inv2_s[2] + inv2_s[3]) <= BLK_INV_LIMIT * jb)) return 0;
  // V_top's entries, scaled
  for (int c = wid; c < jb; c += nw)
    if (lane > c && lane < jb) T0[lane * BLK_LD + c] = T0[lane * BLK_LD + c] * scl[c];
  __syncthreads();

  // ---- T = -F R^-1 V_top^-H, a warp per row, spread over the CTAs
  for (int i = b * nw + wid; i < NBMAX; i += G * nw) {
    T t = zero_<T>();
    if (i < jb) {
      const bool in = lane >= i && lane < jb;
      if (in) t = -T0[i * BLK_LD + lane];
      for (int k = i; k < jb; k++) {
        const T u = shfl_idx_(t, k);
        if (lane > k && lane < jb) t = fma_(-u, Gs[k * BLK_LD + lane], t);
      }
      if (in) t = t * (sgn_s[lane] * rsv[lane]);
      for (int k = i; k < jb; k++) {
        const T u = shfl_idx_(t, k);
        if (lane > k && lane < jb) t = fma_(-u, conj_(T0[lane * BLK_LD + k]), t);
      }
      if (!in) t = zero_<T>();
    }
    a.Tm[i + lane * NBMAX] = t;
  }
  // ---- rows below the top block: V_bot F = A_bot by substitution.  Eight
  // threads per row hold four columns each (cyclic); u_j = x_j unscaled is
  // passed on by a shuffle and F is read scaled by 1 / F_jj, so a step is one
  // multiply-add per column.
  {
    const int q = lane & 7, rl = lane >> 3;
    for (int rb = wid * 4; rb < nr; rb += nw * 4) {
      const int r = rb + rl;
      const bool in = r < nr && r0 + r >= jb;
      T x[4];
#pragma unroll
      for (int k = 0; k < 4; k++)
        x[k] = (in && q + 8 * k < jb) ? Ps[r + (q + 8 * k) * ldp] : zero_<T>();
#pragma unroll
      for (int j = 0; j < NBMAX; j++) {
        if (j < jb) {
          T u = x[j >> 3];
          if constexpr (traits<T>::cpx) {
            u.re = __shfl_sync(0xffffffffu, u.re, j & 7, 8);
            u.im = __shfl_sync(0xffffffffu, u.im, j & 7, 8);
          } else {
            u = __shfl_sync(0xffffffffu, u, j & 7, 8);
          }
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (8 * k + 7 > j) {
              const int c = q + 8 * k;
              if (c > j && c < jb) x[k] = fma_(-u, Gs[c * BLK_LD + j], x[k]);
            }
        }
      }
      if (in) {
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (q + 8 * k < jb) Ps[r + (q + 8 * k) * ldp] = x[k] * scl[q + 8 * k];
      }
    }
  }
  __syncthreads();
  for (int c = wid; c < jb; c += nw)
    for (int r = max(0, jb - r0) + lane; r < nr; r += 32)
      a.A[(r0 + r) + (int64_t)c * a.lda] = Ps[r + c * ldp];
  if (b == 0) {
    // R above V_top, and tau_j = (beta_j - alpha_j) / beta_j
    for (int c = wid; c < jb; c += nw)
      if (lane < jb)
        a.A[lane + (int64_t)c * a.lda] =
            lane < c ? Gs[lane * BLK_LD + c] * (sgn_s[lane] * nrm_s[lane])
                     : (lane == c ? make_scalar<T>(sgn_s[c] * nrm_s[c], R(0))
                                  : T0[lane * BLK_LD + c]);
    if (wid == 0 && lane < jb)
      a.tau[lane] = -(T0[lane * BLK_LD + lane] * (sgn_s[lane] * rsv[lane]));
  }
  return 1;
}

template <class T, int SYNC>
__global__ void __launch_bounds__(PANEL_THREADS, SYNC == SYNC_CLUSTER ? 2 : 1)
qr_panel_kernel(PanelArgs<T> a) {
  using R = real_t<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Ps = reinterpret_cast<T*>(smem_raw);  // rpc x jb, column-major, ld = ldp
  __shared__ R red_r[32];
  __shared__ typename NormKey<R>::K red_k[32];
  __shared__ typename NormKey<R>::K red_k2[32];
  __shared__ R sc_r[3];
  __shared__ int sc_flag, sc_flag2, sc_pair;
  __shared__ T wsh[NBMAX], wsh1[NBMAX];
  __shared__ T red_w[PANEL_THREADS / 32][NBMAX];
  __shared__ T red_g[PANEL_THREADS / 32][NBMAX];  // pair rounds: column j+1's dots
  __shared__ T sc[3], sc1[3];
  __shared__ T rowj[NBMAX], rowj1[NBMAX];
  // cluster variant: this CTA's published partials of the current column
  // (by column parity), read by the other CTAs through distributed shared
  // memory after the cluster barrier
  __shared__ R x_nrm[2][3];       // sum of squares, largest magnitude (of column j+1 too)
  __shared__ T x_w[2][NBMAX];     // dot partials
  __shared__ T x_g[2][NBMAX];     // pair rounds: column j+1's dot partials
  __shared__ T x_row[2][NBMAX];   // row j (the CTA that holds it)
  __shared__ T x_row1[2][NBMAX];  // pair rounds: row j+1
  constexpr bool kCl = SYNC == SYNC_CLUSTER;
  constexpr bool kH = SYNC == SYNC_HIER;
  constexpr bool kSm = kCl || kH;  // partials published in shared memory first
  const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  // hierarchical grid: C CTAs per cluster, H clusters; the global round
  // then carries one partial row per cluster
  const int C = kH ? (int)cluster_nctarank() : 1;
  const int H = G / C;
  const unsigned nsync = kH ? (unsigned)H : (unsigned)G;
  int* const cflag = kH ? a.cflag + b / C : nullptr;
  const int lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int rpc = a.rpc, jb = a.jb;
  const int ldp = rpc | 1;  // slab leading dimension (odd: conflict-free column strides)
  const int r0 = b * rpc;
  const int nr = max(0, min(a.mp, r0 + rpc) - r0);

  // a warp takes four columns at a time: four independent loads per thread
  for (int r = lane; r < nr; r += 32) {
    T v[NBMAX / 8];
#pragma unroll
    for (int q = 0; q < NBMAX / 8; q++) {
      const int c = wid + q * nw;
      v[q] = c < jb ? a.A[(r0 + r) + (int64_t)c * a.lda] : zero_<T>();
    }
#pragma unroll
    for (int q = 0; q < NBMAX / 8; q++)
      if (wid + q * nw < jb) Ps[r + (wid + q * nw) * ldp] = v[q];
  }
  __syncthreads();
  if constexpr (!kH) {
    if (a.block) {
      const size_t slab = ((size_t)ldp * jb * sizeof(T) + 15) / 16 * 16;
      const int done = panel_block_round<T, SYNC>(a, Ps, ldp, r0, nr, smem_raw + slab);
      if (done != 0) return;
    }
  }

  // Per column one grid-wide reduction: the partial sums of squares of x =
  // column j below the diagonal, its largest magnitude, the partial dot
  // products d_c = sum_{r>j} conj(x_r) A[r, c] of the still unscaled x with
  // the columns c > j, and row j, all published in one round.  Since
  // v = [1; scal x], w_c = v^H A[:, c] = A[j, c] + conj(scal) d_c follows
  // once larfg has fixed scal, without a second round.  The partials are
  // double-buffered by column parity: a CTA writes column j+1's slot only
  // after every CTA passed barrier j, i.e. finished reading column j-1's.
  // A column whose largest magnitude lies outside [2^lo, 2^hi] takes the
  // rescaled two-round path instead (the same decision in every CTA).
  // Pair rounds (pair_mode): one round publishes, next to column j's
  // partials, the dot products of column j+1 below row j+1 with the columns
  // c > j and row j+1.  Since H_j is unitary, column j+1's sum of squares
  // and dot products after the reflection follow from those Gram entries,
  // H_j's scalars and rows j, j+1, so column j+1's reflector is formed in
  // the same round (a rank-2 update follows).  When that derivation would
  // cancel (column j+1 keeps less than half of its norm below row j+1) or
  // a magnitude is outside the safe range, column j+1 takes its own round
  // instead; the test sees the same numbers in every CTA.
  const bool pair_mode = !kH && a.pair != 0;
  for (int j = 0, rnd = 0; j < jb; rnd++) {
    T* col = Ps + j * ldp;
    T* col1 = col + ldp;  // column j+1 (pair rounds)
    const int par = rnd & 1;
    const bool two = pair_mode && j + 1 < jb;
    R* pn = a.part_nrm + (int64_t)par * 3 * a.gstride;
    T* pw = a.part_w + (int64_t)par * a.gstride * NBMAX;
    T* pwg = a.part_w + (int64_t)(3 + par) * a.gstride * NBMAX;
    T* prow = a.alpha_buf + par * NBMAX;
    T* prow1 = a.alpha_buf + (2 + par) * NBMAX;
    using NK = NormKey<R>;
    using Key = typename NK::K;
    const int rs = max(0, j + 1 - r0);  // first local row below the diagonal
    const int jy = j + 1 - r0;          // local index of row j+1
    // ---- phase A: warp w takes a slice of this CTA's rows below the
    // diagonal; lane c >= j accumulates conj(x_r) A[r, c] over the slice
    // (lane j: conj(x_r) x_r, the sum of squares) and the largest magnitude
    // of x (pair rounds: also conj(y_r) A[r, c] for y = column j+1 below row
    // j+1, and y's largest magnitude).  No cross-lane reductions (GB300
    // issues about two FP64 operations per clock per SM, so butterflies over
    // 32 lanes would cost more than the products); warp 0 adds the eight
    // slices.  The slab's odd leading dimension keeps the column-strided
    // reads conflict-free.
    {
      const int nx = nr - rs;
      const int per = nx > 0 ? (nx + nw - 1) / nw : 0;
      const int ra = rs + wid * per, rb = min(nr, ra + per);
      T s0 = zero_<T>(), s1 = zero_<T>(), g0 = zero_<T>(), g1 = zero_<T>();
      Key mk = 0, mk2 = 0;
      if (lane >= j && lane < jb) {
        const T* pc = Ps + lane * ldp;
        int r = ra;
        if (two) {
          for (; r + 1 < rb; r += 2) {
            const T x0 = col[r], x1 = col[r + 1];
            const T y0 = r == jy ? zero_<T>() : col1[r];
            const T y1 = r + 1 == jy ? zero_<T>() : col1[r + 1];
            const T c0 = pc[r], c1 = pc[r + 1];
            s0 = fma_(conj_(x0), c0, s0);
            s1 = fma_(conj_(x1), c1, s1);
            g0 = fma_(conj_(y0), c0, g0);
            g1 = fma_(conj_(y1), c1, g1);
            const Key k0 = mag_key(x0), k1 = mag_key(x1);
            const Key k = k0 > k1 ? k0 : k1;
            mk = k > mk ? k : mk;
            const Key q0 = mag_key(y0), q1 = mag_key(y1);
            const Key q = q0 > q1 ? q0 : q1;
            mk2 = q > mk2 ? q : mk2;
          }
          if (r < rb) {
            const T x0 = col[r];
            const T y0 = r == jy ? zero_<T>() : col1[r];
            const T c0 = pc[r];
            s0 = fma_(conj_(x0), c0, s0);
            g0 = fma_(conj_(y0), c0, g0);
            const Key k = mag_key(x0);
            mk = k > mk ? k : mk;
            const Key q = mag_key(y0);
            mk2 = q > mk2 ? q : mk2;
          }
        } else {
          for (; r + 1 < rb; r += 2) {
            const T x0 = col[r], x1 = col[r + 1];
            s0 = fma_(conj_(x0), pc[r], s0);
            s1 = fma_(conj_(x1), pc[r + 1], s1);
            const Key k0 = mag_key(x0), k1 = mag_key(x1);
            const Key k = k0 > k1 ? k0 : k1;
            mk = k > mk ? k : mk;
          }
          if (r < rb) {
            const T x0 = col[r];
            s0 = fma_(conj_(x0), pc[r], s0);
            const Key k = mag_key(x0);
            mk = k > mk ? k : mk;
          }
        }
      }
      red_w[wid][lane] = s0 + s1;
      if (two) red_g[wid][lane] = g0 + g1;
      if (lane == j) {
        red_k[wid] = mk;
        red_k2[wid] = mk2;
      }
    }
    if (j >= r0 && j < r0 + nr)
      for (int c = j + tid; c < jb; c += blockDim.x) {
        if constexpr (kSm) x_row[par][c] = Ps[(j - r0) + c * ldp];
        else prow[c] = Ps[(j - r0) + c * ldp];
      }
    if (two && jy >= 0 && jy < nr)
      for (int c = j + tid; c < jb; c += blockDim.x) {
        if constexpr (kSm) x_row1[par][c] = Ps[jy + c * ldp];
        else prow1[c] = Ps[jy + c * ldp];
      }
    __syncthreads();
    if (wid == 0) {
      T s = zero_<T>();
      for (int w = 0; w < nw; w++) s += red_w[w][lane];
      if (lane > j && lane < jb) {
        if constexpr (kSm) x_w[par][lane] = s;
        else pw[(int64_t)b * NBMAX + lane] = s;
      }
      if (two) {
        T sg = zero_<T>();
        for (int w = 0; w < nw; w++) sg += red_g[w][lane];
        if (lane > j && lane < jb) {
          if constexpr (kSm) x_g[par][lane] = sg;
          else pwg[(int64_t)b * NBMAX + lane] = sg;
        }
      }
      if (lane == j) {
        Key m = 0, m2 = 0;
        for (int w = 0; w < nw; w++) {
          m = red_k[w] > m ? red_k[w] : m;
          m2 = red_k2[w] > m2 ? red_k2[w] : m2;
        }
        if constexpr (kSm) {
          x_nrm[par][0] = re_(s);
          x_nrm[par][1] = NK::val(m);
          x_nrm[par][2] = NK::val(m2);
        } else {
          pn[b] = re_(s);
          pn[a.gstride + b] = NK::val(m);
          pn[2 * a.gstride + b] = NK::val(m2);
        }
      }
    }
    if constexpr (kH) {
      // the cluster's first CTA combines its C CTAs' partials (rank order)
      // and publishes one row per cluster for the global round
      cluster_sync_all();
      if (cluster_ctarank() == 0) {
        const int h = b / C;
        if (wid == 0) {
          if (lane == j) {
            R s2 = R(0);
            Key m2 = 0;
            for (int r = 0; r < C; r++) {
              s2 += dsmem_ld(&x_nrm[par][0], (unsigned)r);
              const Key k = NK::key(dsmem_ld(&x_nrm[par][1], (unsigned)r));
              m2 = k > m2 ? k : m2;
            }
            pn[h] = s2;
            pn[a.gstride + h] = NK::val(m2);
          }
          if (lane > j && lane < jb) {
            T s2 = zero_<T>();
            for (int r = 0; r < C; r++) s2 += dsmem_ld(&x_w[par][lane], (unsigned)r);
            pw[(int64_t)h * NBMAX + lane] = s2;
          }
        }
        const int own = j / rpc;  // the CTA holding row j
        if (own / C == h && wid == 1 && lane >= j && lane < jb)
          prow[lane] = dsmem_ld(&x_row[par][lane], (unsigned)(own % C));
      }
      if (!hier_leader_barrier(a.bar, nsync, a.status, cflag)) return;
    } else {
      if (!panel_sync<SYNC>(a.bar, G, a.status)) return;
    }

    // ---- phase B: every CTA combines the partials in the same fixed order
    // and so derives bit-identical beta / tau / w.  Warp 0: the norm; every
    // warp: a slice of the CTAs' dot partials (lane = column); lane j of
    // warp 1 (or of warp 0 with one warp): row j; warp 2: row j+1.
    const int NP = kH ? H : G;  // partial rows to combine
    if (wid == 0) {
      R s = R(0);
      Key m = 0, m2 = 0;
      for (int q = lane; q < NP; q += 32) {
        if constexpr (kCl) {
          s += dsmem_ld(&x_nrm[par][0], (unsigned)q);
          const Key k = NK::key(dsmem_ld(&x_nrm[par][1], (unsigned)q));
          m = k > m ? k : m;
          if (two) {
            const Key k2 = NK::key(dsmem_ld(&x_nrm[par][2], (unsigned)q));
            m2 = k2 > m2 ? k2 : m2;
          }
        } else {
          s += ld_cg(&pn[q]);
          const Key k = NK::key(ld_cg(&pn[a.gstride + q]));
          m = k > m ? k : m;
          if (two) {
            const Key k2 = NK::key(ld_cg(&pn[2 * a.gstride + q]));
            m2 = k2 > m2 ? k2 : m2;
          }
        }
      }
      s = warp_sum(s);
      m = warp_max_key(m);
      if (two) m2 = warp_max_key(m2);
      if (lane == 0) {
        sc_r[0] = s;
        sc_r[1] = NK::val(m);
        sc_flag = norm_needs_rescale<R>(m);
        sc_flag2 = norm_needs_rescale<R>(m2);
      }
    }
    {
      const int per = (NP + nw - 1) / nw;
      const int q0 = wid * per, q1 = min(NP, q0 + per);
      T a0 = zero_<T>(), a1 = zero_<T>(), a2 = zero_<T>(), a3 = zero_<T>();
      T b0 = zero_<T>(), b1 = zero_<T>(), b2 = zero_<T>(), b3 = zero_<T>();
      if (lane > j && lane < jb) {
        int q = q0;
        if constexpr (kCl) {
          for (; q < q1; q++) {
            a0 += dsmem_ld(&x_w[par][lane], (unsigned)q);
            if (two) b0 += dsmem_ld(&x_g[par][lane], (unsigned)q);
          }
        } else {
          for (; q + 3 < q1; q += 4) {
            a0 += ld_cg(&pw[(int64_t)q * NBMAX + lane]);
            a1 += ld_cg(&pw[(int64_t)(q + 1) * NBMAX + lane]);
            a2 += ld_cg(&pw[(int64_t)(q + 2) * NBMAX + lane]);
            a3 += ld_cg(&pw[(int64_t)(q + 3) * NBMAX + lane]);
            if (two) {
              b0 += ld_cg(&pwg[(int64_t)q * NBMAX + lane]);
              b1 += ld_cg(&pwg[(int64_t)(q + 1) * NBMAX + lane]);
              b2 += ld_cg(&pwg[(int64_t)(q + 2) * NBMAX + lane]);
              b3 += ld_cg(&pwg[(int64_t)(q + 3) * NBMAX + lane]);
            }
          }
          for (; q < q1; q++) {
            a0 += ld_cg(&pw[(int64_t)q * NBMAX + lane]);
            if (two) b0 += ld_cg(&pwg[(int64_t)q * NBMAX + lane]);
          }
        }
      }
      red_w[wid][lane] = (a0 + a1) + (a2 + a3);
      if (two) red_g[wid][lane] = (b0 + b1) + (b2 + b3);
    }
    if (wid == (nw > 1 ? 1 : 0) && lane >= j && lane < jb) {
      // row j is held by the CTA whose rows contain j
      if constexpr (kCl) rowj[lane] = dsmem_ld(&x_row[par][lane], (unsigned)(j / rpc));
      else rowj[lane] = ld_cg(&prow[lane]);
    }
    if (two && wid == (nw > 2 ? 2 : 0) && lane >= j && lane < jb) {
      if constexpr (kCl) rowj1[lane] = dsmem_ld(&x_row1[par][lane], (unsigned)((j + 1) / rpc));
      else rowj1[lane] = ld_cg(&prow1[lane]);
    }
    __syncthreads();
    const bool rescale = sc_flag != 0;
    if (two && !rescale) {
      // ---- both reflectors on warp 0 (every lane derives the scalars, lane
      // c the column-c quantities).  H_j: f_c = conj(tau) w_c as below.
      // Column j+1 after H_j^H: with v = [1; scal x] and x_1 = A[j+1, j],
      //   p_c = sum_{r>j+1} conj(v_r) A[r, c] = conj(scal) (d_c - conj(x_1) A[j+1, c])
      //   q   = sum_{r>j+1} |v_r|^2 = |scal|^2 (|x|^2 - |x_1|^2)
      //   G_c = sum_{r>j+1} conj(A'[r, j+1]) A'[r, c]
      //       = g_c - conj(p_{j+1}) f_c - conj(f_{j+1}) p_c + conj(f_{j+1}) f_c q
      //   A'[j+1, c] = A[j+1, c] - scal x_1 f_c,
      // and column j+1's reflector follows from alpha = A'[j+1, j+1] and the
      // sum of squares G_{j+1}, with d'_c = G_c (c > j+1).
      if (wid == 0) {
        T d = zero_<T>(), g = zero_<T>();
        for (int w = 0; w < nw; w++) {
          d += red_w[w][lane];
          g += red_g[w][lane];
        }
        T beta, tau, scal;
        larfg_scalars_ssq(rowj[j], sc_r[0], sc_r[1], beta, tau, scal);
        const bool act = lane > j && lane < jb;
        const T f = act ? conj_(tau) * fma_(conj_(scal), d, rowj[lane]) : zero_<T>();
        const T x1 = rowj1[j];
        const T v1 = x1 * scal;
        const T p = act ? conj_(scal) * fma_(-conj_(x1), rowj1[lane], d) : zero_<T>();
        const R q = abs2_(scal) * (sc_r[0] - abs2_(x1));
        const T f1 = shfl_idx_(f, j + 1), p1 = shfl_idx_(p, j + 1);
        const T gp = act ? (g - conj_(p1) * f - conj_(f1) * p) + (conj_(f1) * f) * q : zero_<T>();
        const T r1 = act ? fma_(-v1, f, rowj1[lane]) : zero_<T>();
        const R ssq1 = re_(shfl_idx_(gp, j + 1));
        const T alpha1 = shfl_idx_(r1, j + 1);
        const R nrm1 = re_(shfl_idx_(g, j + 1)) + abs2_(rowj1[j + 1]) + abs2_(rowj[j + 1]);
        const bool fin = __all_sync(0xffffffffu, !act || (finite_(gp) && finite_(r1)));
        const int en = exp2_of(nrm1);
        const int lim = sizeof(R) == 8 ? 1000 : 100;
        const bool ok = fin && sc_flag2 == 0 && en > -lim && en < lim && ssq1 >= R(0.5) * nrm1;
        T beta1 = zero_<T>(), tau1 = zero_<T>(), scal1 = one_<T>(), f2 = zero_<T>();
        if (ok) {
          // a power of two within a factor 2 sqrt(2) of sqrt(ssq1) scales the
          // square root in place of column j+1's largest magnitude
          const R prox = ssq1 > R(0) ? pow2_(R(0), exp2_of(ssq1) >> 1) : R(0);
          larfg_scalars_ssq(alpha1, ssq1, prox, beta1, tau1, scal1);
          if (lane > j + 1 && lane < jb) f2 = conj_(tau1) * fma_(conj_(scal1), gp, r1);
        }
        wsh[lane] = f;
        wsh1[lane] = f2;
        if (lane == 0) {
          sc[0] = beta;
          sc[1] = tau;
          sc[2] = scal;
          sc1[0] = beta1;
          sc1[1] = tau1;
          sc1[2] = scal1;
          sc_pair = ok ? 1 : 0;
        }
      }
      __syncthreads();
      const T beta = sc[0], tau = sc[1], scal = sc[2];
      const bool ok = sc_pair != 0;
      if (b == 0 && tid == 0) {
        a.tau[j] = tau;
        if (ok) a.tau[j + 1] = sc1[1];
      }
      const int rj = max(0, j - r0);
      if (ok) {
        // column j: scale to v; column j+1: apply H_j^H, then scale below
        // row j+1 to v' (row j+1 becomes beta')
        const T f1 = wsh[j + 1], scal1 = sc1[2];
        for (int r = rj + tid; r < nr; r += blockDim.x) {
          const int gr = r0 + r;
          T v = one_<T>();
          if (gr > j) {
            v = col[r] * scal;
            col[r] = v;
          }
          const T y = fma_(-v, f1, col1[r]);
          col1[r] = gr > j + 1 ? y * scal1 : y;
        }
        __syncthreads();
        // rank-2 update of the columns c > j+1: rows >= j take v f_c, rows
        // >= j+1 also v' f'_c (v_j = 1, v'_{j+1} = 1)
        for (int c = j + 2 + wid; c < jb; c += nw) {
          const T fa = wsh[c], fb = wsh1[c];
          T* pc = Ps + c * ldp;
          for (int r = rj + lane; r < nr; r += 32) {
            const int gr = r0 + r;
            const T v = gr == j ? one_<T>() : col[r];
            T y = fma_(-v, fa, pc[r]);
            if (gr > j) y = fma_(gr == j + 1 ? -one_<T>() : -col1[r], fb, y);
            pc[r] = y;
          }
        }
        if (tid == 0 && j >= r0 && j < r0 + nr) col[j - r0] = beta;
        if (tid == 0 && jy >= 0 && jy < nr) col1[jy] = sc1[0];
        __syncthreads();
        j += 2;
      } else {
        for (int r = rs + tid; r < nr; r += blockDim.x) col[r] = col[r] * scal;
        __syncthreads();
        for (int c = j + 1 + wid; c < jb; c += nw) {
          const T f = wsh[c];
          T* pc = Ps + c * ldp;
          for (int r = rj + lane; r < nr; r += 32) {
            const T v = (r0 + r == j) ? one_<T>() : col[r];
            pc[r] = fma_(-v, f, pc[r]);
          }
        }
        if (tid == 0 && j >= r0 && j < r0 + nr) col[j - r0] = beta;
        __syncthreads();
        j += 1;
      }
      continue;
    }
    R xnorm = R(0);  // meaningful in thread 0 only (the scalars below)
    if (rescale) {
      // rare: rescale by 2^-e, e the exponent of the largest magnitude
      // (clamped so the scale itself stays finite), then sum again
      int e = 0;
      frexp(sc_r[1], &e);
      e = e > 1000 ? 1000 : (e < -1000 ? -1000 : e);
      const R scale = ldexp(R(1), -e);
      R ss2 = R(0);
      for (int r = rs + tid; r < nr; r += blockDim.x) ssq_scaled_add(ss2, col[r], scale);
      ss2 = block_sum(ss2, red_r);
      if (tid == 0) a.part_nrm[6 * a.gstride + b] = ss2;
      if (!panel_sync<SYNC>(a.bar, nsync, a.status, cflag)) return;
      if (wid == 0) {
        R s2 = R(0);
        for (int q = lane; q < G; q += 32) s2 += ld_cg(&a.part_nrm[6 * a.gstride + q]);
        s2 = warp_sum(s2);
        if (lane == 0) sc_r[2] = sqrt(s2) * ldexp(R(1), e);
      }
      __syncthreads();
      xnorm = sc_r[2];
    }
    if (tid == 0) {
      T beta, tau, scal;
      if (rescale) larfg_scalars(rowj[j], xnorm, beta, tau, scal);
      else larfg_scalars_ssq(rowj[j], sc_r[0], sc_r[1], beta, tau, scal);
      sc[0] = beta;
      sc[1] = tau;
      sc[2] = scal;
    }
    __syncthreads();
    const T beta = sc[0], tau = sc[1], scal = sc[2];
    if (b == 0 && tid == 0) a.tau[j] = tau;
    if (j + 1 >= jb) {
      for (int r = rs + tid; r < nr; r += blockDim.x) col[r] = col[r] * scal;
      if (tid == 0 && j >= r0 && j < r0 + nr) col[j - r0] = beta;
      __syncthreads();
      break;
    }
    if (!rescale) {
      // f_c = conj(tau) w_c, w_c = A[j, c] + conj(scal) d_c, formed once
      if (wid == 0) {
        T sum = zero_<T>();
        for (int w = 0; w < nw; w++) sum += red_w[w][lane];
        if (lane > j && lane < jb) wsh[lane] = conj_(tau) * fma_(conj_(scal), sum, rowj[lane]);
      }
    } else {
      // the two-round form on the scaled column: w = v^H A from v itself
      for (int r = rs + tid; r < nr; r += blockDim.x) col[r] = col[r] * scal;
      __syncthreads();
      const int rj = max(0, j - r0);
      T* pw2 = a.part_w + (int64_t)2 * a.gstride * NBMAX;
      for (int c = j + 1 + wid; c < jb; c += nw) {
        T s = zero_<T>();
        for (int r = rj + lane; r < nr; r += 32) {
          const T v = (r0 + r == j) ? one_<T>() : col[r];
          s = fma_(conj_(v), Ps[r + c * ldp], s);
        }
        s = warp_sum(s);
        if (lane == 0) pw2[(int64_t)b * NBMAX + c] = s;
      }
      if (!panel_sync<SYNC>(a.bar, nsync, a.status, cflag)) return;
      {
        const int per = (G + nw - 1) / nw;
        const int q0 = wid * per, q1 = min(G, q0 + per);
        T acc = zero_<T>();
        if (lane > j && lane < jb)
          for (int q = q0; q < q1; q++) acc += ld_cg(&pw2[(int64_t)q * NBMAX + lane]);
        red_w[wid][lane] = acc;
      }
      __syncthreads();
      if (wid == 0) {
        T sum = zero_<T>();
        for (int w = 0; w < nw; w++) sum += red_w[w][lane];
        if (lane > j && lane < jb) wsh[lane] = conj_(tau) * sum;
      }
    }
    __syncthreads();
    // ---- update rows >= j of the columns c > j: A[r, c] -= v_r f_c, with
    // v_j = 1 and v_r = scal x_r below (stored back as the reflector)
    // The reflector is scaled in place first; the update then gives each
    // warp its own columns (lanes over rows), so that all eight warps share
    // the FP64 work even when a CTA owns only a few dozen rows.
    const int rj = max(0, j - r0);
    if (!rescale)
      for (int r = rs + tid; r < nr; r += blockDim.x) col[r] = col[r] * scal;
    __syncthreads();
    for (int c = j + 1 + wid; c < jb; c += nw) {
      const T f = wsh[c];
      T* pc = Ps + c * ldp;
      for (int r = rj + lane; r < nr; r += 32) {
        const T v = (r0 + r == j) ? one_<T>() : col[r];
        pc[r] = fma_(-v, f, pc[r]);
      }
    }
    if (tid == 0 && j >= r0 && j < r0 + nr) col[j - r0] = beta;
    __syncthreads();
    j += 1;
  }

  // ---- Gram partials of V (unit lower trapezoidal) for the T factor: one
  // thread per pair (i, jj), i < jj, over this CTA's rows (no reductions)
  const int npairs = jb * (jb - 1) / 2;
  for (int pq = tid; pq < npairs; pq += blockDim.x) {
    int jj = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)pq)) * 0.5f);
    while (jj * (jj - 1) / 2 > pq) jj--;
    while (jj * (jj + 1) / 2 <= pq) jj++;
    const int i = pq - jj * (jj - 1) / 2;
    T s0 = zero_<T>(), s1 = zero_<T>();
    const int rb = max(0, jj - r0);
    int r = rb;
    if (r < nr && r0 + r == jj) {  // v_jj = 1 on its diagonal row
      s0 = conj_(Ps[r + i * ldp]);
      r++;
    }
    for (; r + 1 < nr; r += 2) {
      s0 = fma_(conj_(Ps[r + i * ldp]), Ps[r + jj * ldp], s0);
      s1 = fma_(conj_(Ps[r + 1 + i * ldp]), Ps[r + 1 + jj * ldp], s1);
    }
    if (r < nr) s0 = fma_(conj_(Ps[r + i * ldp]), Ps[r + jj * ldp], s0);
    a.part_g[(int64_t)b * NBMAX * NBMAX + i + jj * NBMAX] = s0 + s1;
  }
  for (int c = 0; c < jb; c++)
    for (int r = tid; r < nr; r += blockDim.x) a.A[(r0 + r) + (int64_t)c * a.lda] = Ps[r + c * ldp];
  if (!panel_sync<SYNC>(a.bar, nsync, a.status, cflag)) return;

  // ---- reduce the Gram over the CTAs: one thread per pair, the CTAs'
  // partials in a fixed order (four interleaved accumulators)
  for (int pq = b * (int)blockDim.x + tid; pq < npairs; pq += G * (int)blockDim.x) {
    int jj = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)pq)) * 0.5f);
    while (jj * (jj - 1) / 2 > pq) jj--;
    while (jj * (jj + 1) / 2 <= pq) jj++;
    const int i = pq - jj * (jj - 1) / 2;
    const T* src = a.part_g + i + jj * NBMAX;
    constexpr int64_t NN = NBMAX * NBMAX;
    T s0 = zero_<T>(), s1 = zero_<T>(), s2 = zero_<T>(), s3 = zero_<T>();
    int q = 0;
    for (; q + 3 < G; q += 4) {
      s0 += ld_cg(src + q * NN);
      s1 += ld_cg(src + (q + 1) * NN);
      s2 += ld_cg(src + (q + 2) * NN);
      s3 += ld_cg(src + (q + 3) * NN);
    }
    for (; q < G; q++) s0 += ld_cg(src + q * NN);
    a.gram[i + jj * NBMAX] = (s0 + s1) + (s2 + s3);
  }
  if (!panel_sync<SYNC>(a.bar, nsync, a.status, cflag)) return;

  // ---- T factor (larft, forward, column-wise): T = U^{-1} with U_ii =
  // 1/tau_i and U_il = G_il (i < l), each column an independent back
  // substitution x_k = tau_k, x_i = -tau_i sum_{l=i+1..k} G_il x_l (tau_i as
  // a factor: tau_i = 0 needs no division).  Column k goes to warp k mod 8
  // of CTA k / 8 (then every G * 8 columns); lane i owns row i.  tau and the
  // strict upper triangle of the Gram matrix are staged in shared memory
  // first (one batch of independent loads), so the substitution chain
  // itself waits on no L2 round trip.
  const int kfirst = b * nw;
  if (kfirst >= NBMAX) return;  // the same for every thread of the CTA
  __shared__ T gs[NBMAX * NBMAX];
  __shared__ T ts[NBMAX];
  if (kfirst < jb) {
    for (int e = tid; e < NBMAX * NBMAX; e += blockDim.x) {
      const int i = e % NBMAX, l = e / NBMAX;
      if (i < l && l < jb) gs[e] = ld_cg(&a.gram[e]);
    }
    if (tid < NBMAX) ts[tid] = tid < jb ? ld_cg(&a.tau[tid]) : zero_<T>();
  }
  __syncthreads();
  for (int k = kfirst + wid; k < NBMAX; k += G * nw) {
    T x = zero_<T>();
    if (k < jb) {
      T acc = zero_<T>();
      for (int l = k; l >= 0; l--) {
        const T mine = (l == k) ? ts[k] : -(ts[l] * acc);
        const T xl = shfl_idx_(mine, l);
        if (lane == l) x = xl;
        if (lane < l) acc = fma_(gs[lane + l * NBMAX], xl, acc);
      }
    }
    a.Tm[lane + k * NBMAX] = (k < jb && lane <= k) ? x : zero_<T>();
  }
}

// W2[:, c] = op(Tm) * sum_s Wpart[s][:, c]   (op = ^H for the factorization,
// identity for Q formation).  Fixed summation order -> deterministic.  One
// output per thread, eight columns per CTA of 32 rows: the FP64 work of the
// product is spread over as many SMs as there are column groups (32 columns per
// CTA left most of them idle: 500 columns 17.5 us).  16 or 32 columns where 16
// or 8 rows are all there are (8 x 100000: 68 us with 32 rows of threads).
constexpr int TRMM_THREADS = 256;
__host__ __device__ constexpr int trmm_rows(int jb) { return jb <= 8 ? 8 : (jb <= 16 ? 16 : 32); }
__host__ __device__ constexpr int trmm_cols(int jb) { return TRMM_THREADS / trmm_rows(jb); }
template <class T>
__global__ void __launch_bounds__(TRMM_THREADS) reduce_trmm_kernel(int jb, int nt, int splits,
                                                          const T* __restrict__ Wpart,
                                                          int64_t sstride,
                                                          const T* __restrict__ Tm, int conjtrans,
                                                          T* __restrict__ W2) {
  __shared__ T Ts[NBMAX][NBMAX + 1];
  __shared__ T Ws[TRMM_THREADS];
  const int rows = trmm_rows(jb);
  const int i = threadIdx.x & (rows - 1);
  const int c = blockIdx.x * trmm_cols(jb) + threadIdx.x / rows;
  for (int e = threadIdx.x; e < jb * jb; e += blockDim.x) {
    const int r = e % jb, l = e / jb;
    if (conjtrans) Ts[l][r] = conj_(Tm[r + l * NBMAX]);
    else Ts[r][l] = Tm[r + l * NBMAX];
  }
  T w = zero_<T>();
  if (i < jb && c < nt) {
    const T* src = Wpart + i + (int64_t)c * jb;
    int q = 0;
    for (; q + 3 < splits; q += 4) {
      const T a = src[q * sstride], b = src[(q + 1) * sstride];
      const T d = src[(q + 2) * sstride], f = src[(q + 3) * sstride];
      w += (a + b) + (d + f);
    }
    for (; q < splits; q++) w += src[q * sstride];
  }
  Ws[threadIdx.x] = w;
  __syncthreads();
  if (i >= jb || c >= nt) return;
  const T* const wc = Ws + threadIdx.x - i;  // the column's entries
  T s[4] = {zero_<T>(), zero_<T>(), zero_<T>(), zero_<T>()};
  int l = 0;
  for (; l + 3 < jb; l += 4)
#pragma unroll
    for (int q = 0; q < 4; q++) s[q] = fma_(Ts[i][l + q], wc[l + q], s[q]);
  for (; l < jb; l++) s[0] = fma_(Ts[i][l], wc[l], s[0]);
  W2[i + (int64_t)c * jb] = (s[0] + s[1]) + (s[2] + s[3]);
}

constexpr int QR_OUTER_NB = 128;  // block of the mixed-precision path
constexpr double QR_WIDE_MIN_MN = 4.0e6;  // m n from which its block reflectors are merged
// SMs given to the look-ahead side stream (panels and the block Gram) while
// the main stream's persistent tensor-core grid takes the rest; 48 by
// default, MAK_LOOKAHEAD_CTAS overrides it (read once, clamped to 8..120).
int lookahead_ctas() { return (int)tuning(TUNE_LOOKAHEAD_CTAS); }
// In the tail of the factorization the far update shrinks below the time
// of the next block's panels; from MAK_LOOKAHEAD_TAIL_COLS far columns
// down, the side stream takes MAK_LOOKAHEAD_TAIL_CTAS SMs instead.
static int side_ctas(int64_t far_cols) {
  const double tail = tuning(TUNE_LOOKAHEAD_TAIL_COLS);
  return (double)far_cols <= tail ? (int)tuning(TUNE_LOOKAHEAD_TAIL_CTAS) : lookahead_ctas();
}
static thread_local int tl_side_ctas = 0;  // the side stream's SMs for the block being factored

static thread_local bool tl_no_lookahead = false;
bool lookahead_enabled() { return !tl_no_lookahead; }
void set_lookahead(bool on) { tl_no_lookahead = !on; }
static thread_local int tl_gemm_budget = 0;
int split_gemm_cta_budget() { return tl_gemm_budget; }
void set_split_gemm_cta_budget(int ctas) { tl_gemm_budget = ctas > 0 ? ctas : 0; }

// Side stream (highest priority, so its panel CTAs are scheduled ahead of
// the trailing GEMM's) and events of the look-ahead, one set per (host
// thread, device) so that calls from several threads never share an event
// and a call on another device never queues work on this device's stream;
// created by the first large call of that thread on that device (which must
// precede any graph capture there).
LookAhead* lookahead() {
  static thread_local LookAhead la[kMaxDevices];
  static thread_local int state[kMaxDevices] = {};  // 0 not created, 1 ready, -1 failed
  const int d = current_device();
  if (state[d] == 0) {
    int lo = 0, hi = 0;
    cudaDeviceGetStreamPriorityRange(&lo, &hi);
    state[d] =
        (cudaStreamCreateWithPriority(&la[d].side, cudaStreamNonBlocking, hi) == cudaSuccess &&
         cudaEventCreateWithFlags(&la[d].ev_ready, cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&la[d].ev_done, cudaEventDisableTiming) == cudaSuccess)
            ? 1
            : -1;
  }
  return state[d] == 1 ? &la[d] : nullptr;
}

// T factor of a JB-wide block reflector H_1 ... H_JB = I - V T V^H (forward,
// column-wise storage) from the Gram matrix G = V^H V and the T factors of its
// nb-wide panels.  With the panels' columns V_0, V_1, ... and Ta the T factor
// of panel a, T is block upper triangular with the Ta on its diagonal and
// satisfies T_ab = -Ta sum_{a < c <= b} G_ac T_cb, so every column is an
// independent block back substitution.  One warp per column, lane = row of a
// block; eight columns of G in flight.  A warp-wide FP64 operation holds its
// sub-partition's pipe for 64 cycles: four warps per CTA, and 288 operations
// for the last column of 128 against 640 by single rows (Float64 70 us,
// ComplexF64 197 us per 128 columns before).
constexpr int LARFT_WARPS = 4;
template <class T>
__global__ void __launch_bounds__(32 * LARFT_WARPS)
larft_blocks_kernel(int jb, int nb, const T* __restrict__ G, int ldg, const T* __restrict__ Ts,
                    T* Tout, int ldt) {
  __shared__ T xs[LARFT_WARPS][QR_OUTER_NB];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int k = blockIdx.x * LARFT_WARPS + wid;
  if (k >= jb) return;
  T* const x = xs[wid];
  const int b = k / nb, kc = k - b * nb;
  for (int i = lane; i < QR_OUTER_NB; i += 32) x[i] = zero_<T>();
  __syncwarp();
  if (lane <= kc) x[b * nb + lane] = Ts[(int64_t)b * NBMAX * NBMAX + lane + kc * NBMAX];
  __syncwarp();
  for (int a = b - 1; a >= 0; a--) {
    const bool in = lane < nb;
    const T* g = G + a * nb + (in ? lane : 0);
    T y0 = zero_<T>(), y1 = zero_<T>();
    int l = (a + 1) * nb;
    for (; l + 7 <= k; l += 8) {
      T v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = g[(int64_t)(l + q) * ldg];
#pragma unroll
      for (int q = 0; q < 8; q += 2) {
        y0 = fma_(v[q], x[l + q], y0);
        y1 = fma_(v[q + 1], x[l + q + 1], y1);
      }
    }
    for (; l <= k; l++) y0 = fma_(g[(int64_t)l * ldg], x[l], y0);
    const T y = in ? -(y0 + y1) : zero_<T>();
    const T* t = Ts + (int64_t)a * NBMAX * NBMAX + lane;
    T s = zero_<T>();
#pragma unroll 8
    for (int c = 0; c < nb; c++) {
      const T yc = shfl_idx_(y, c);
      s = fma_(t[c * NBMAX], yc, s);  // Ta is stored with its lower zeros
    }
    if (in) x[a * nb + lane] = s;
    __syncwarp();
  }
  for (int i = lane; i < jb; i += 32) Tout[i + (int64_t)k * ldt] = i <= k ? x[i] : zero_<T>();
}

template <class T>
__global__ void signs_kernel(int k, const T* A, int64_t lda, int positive, T* s) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < k) s[j] = positive ? sign_safe_(A[j + j * lda]) : one_<T>();
}

// R[i, j] = (i <= j && i < k) ? conj(s_i) A[i, j] : 0   for i < rrows, j < n
template <class T>
__global__ void extract_r_kernel(int64_t rrows, int64_t n, int64_t k, const T* A, int64_t lda,
                                 const T* s, T* R, int64_t ldr) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t j = blockIdx.y;
  for (; j < n; j += gridDim.y) {
    if (i >= rrows) return;
    T v = zero_<T>();
    if (i <= j && i < k) v = conj_(s[i]) * A[i + j * lda];
    R[i + j * ldr] = v;
  }
}

// Q = [diag(s); 0] on the first k columns, identity beyond (qr_full)
template <class T>
__global__ void init_q_kernel(int64_t m, int64_t qcols, int64_t k, const T* s, T* Q, int64_t ldq) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t j = blockIdx.y; j < qcols; j += gridDim.y) {
    if (i >= m) return;
    T v = zero_<T>();
    if (i == j) v = (j < k) ? s[j] : one_<T>();
    Q[i + j * ldq] = v;
  }
}

__global__ void info_reset_kernel(mak_info* info) {
  info->status = 0;
  info->iterations = 0;
  info->rank = 0;
  info->converged = 0;
  info->residual = 0.0;
  info->gauge = 0.0;
  info->gauge_atol = 0.0;
  info->singular = 0;
  info->pad = 0;
}

int info_reset(cudaStream_t st, mak_info* info) {
  note_launch();
  info_reset_kernel<<<1, 1, 0, st>>>(info);
  return cudaGetLastError() == cudaSuccess ? 0 : MAK_ERR_CUDA;
}

std::atomic<unsigned long long>& launch_counter() {
  static std::atomic<unsigned long long> c{0};
  return c;
}

int num_sms() {
  static PerDevice<int> pd;
  return pd.get([] {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, current_device());
    return v > 0 ? v : 152;
  });
}
int max_smem_optin() {
  static PerDevice<int> pd;
  return pd.get([] {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, current_device());
    return v > 0 ? v : 227 * 1024;
  });
}

// Shared memory available to the panel slab: the opt-in maximum minus the
// kernel's static shared memory (T-factor scratch); queried, and the
// kernel's dynamic shared-memory limit raised, once per type and device.
template <class T>
static size_t panel_slab_cap() {
  static PerDevice<size_t> pd;
  return pd.get([] {
    cudaFuncAttributes fa;
    size_t stat = 48 * 1024;
    if (cudaFuncGetAttributes(&fa, qr_panel_kernel<T, SYNC_GRID>) == cudaSuccess)
      stat = fa.sharedSizeBytes;
    if (cudaFuncGetAttributes(&fa, qr_panel_kernel<T, SYNC_CLUSTER>) == cudaSuccess &&
        fa.sharedSizeBytes > stat)
      stat = fa.sharedSizeBytes;
    const size_t cap = (size_t)max_smem_optin() - stat - 1024;
    cudaFuncSetAttribute(qr_panel_kernel<T, SYNC_GRID>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
    cudaFuncSetAttribute(qr_panel_kernel<T, SYNC_CLUSTER>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
    cudaFuncSetAttribute(qr_panel_kernel<T, SYNC_HIER>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
    cudaFuncSetAttribute(qr_panel_kernel<T, SYNC_CLUSTER>,
                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return cap;
  });
}

constexpr int kPanelClusterWide = 16;
// Panels of at most this many rows per CTA (times the cluster limit) run as
// one thread-block cluster: below it a column's FP64 work per CTA stays
// smaller than what a global barrier costs.
constexpr int PANEL_CLUSTER_ROWS = 256;

// Launch shape of the panel kernel.  Cluster (sync = SYNC_CLUSTER): panels
// of up to kPanelClusterMax x PANEL_CLUSTER_ROWS rows, at least 32 rows per
// CTA.  Cooperative grid (SYNC_GRID) beyond that: rows per CTA bounded below
// by 64 (a grid barrier is only paid when there is real parallel work) and
// above by the shared-memory slab size; at most one CTA per SM.
struct PanelShape {
  int G, rpc, sync;
  int block = 0;  // the block round may be tried (its shared memory follows the slab)
  int cl = 1;  // CTAs per cluster (SYNC_CLUSTER: G; SYNC_HIER: the cluster size)
  size_t smem;
};
// shared memory of a launch: the slab, and the block round's scratch where
// the panel is tall enough to take it and the scratch fits beside the slab
template <class T>
static void panel_smem(PanelShape& ps, int64_t mp, int jb, size_t cap) {
  const size_t slab = (size_t)(ps.rpc | 1) * jb * sizeof(T);
  const size_t both = align_up(slab, 16) + block_extra_bytes<T>();
  ps.block = tuning(TUNE_PANEL_PAIR) != 0 && jb >= BLK_MIN_COLS &&
             mp >= (int64_t)BLK_MIN_MP_PER_COL * jb && both <= cap;
  ps.smem = ps.block ? both : slab;
}
template <class T>
static int panel_shape(int64_t mp, int jb, PanelShape& ps, int want_ctas, bool main_stream) {
  const int max_ctas = num_sms();
  const size_t cap = panel_slab_cap<T>();
  int64_t rpc_max = (int64_t)(cap / ((size_t)jb * sizeof(T))) - 1;  // ld = rpc | 1
  const int64_t cl_rows = rpc_max < PANEL_CLUSTER_ROWS ? rpc_max : PANEL_CLUSTER_ROWS;
  // Clusters of up to 16 CTAs (a non-portable size) of at least 32 rows: the
  // block round's FP64 work is shared by the CTAs (1000 x 501 Float64 QR 4.72
  // -> 4.50 ms against 8 CTAs of at least 64 rows, 2049 x 1000 mixed 11.65 ->
  // 10.76 ms, the 300 uneven blocks 189.7 -> 186.6 ms).  8 CTAs on the
  // look-ahead side stream, where the main stream's grid leaves 16 free SMs of
  // one cluster group only by chance, and where 16 do not fit.
  for (int cmax = main_stream ? kPanelClusterWide : kPanelClusterMax;
       mp <= (int64_t)kPanelClusterMax * cl_rows; cmax = kPanelClusterMax) {
    int64_t G = ceil_div(mp, 32);
    if (G > cmax) G = cmax;
    int64_t rpc = ceil_div(mp, G);
    if (rpc < 1) rpc = 1;
    G = ceil_div(mp, rpc);
    if (G < 1) G = 1;
    ps.G = (int)G;
    ps.rpc = (int)rpc;
    ps.sync = SYNC_CLUSTER;
    ps.cl = (int)G;
    panel_smem<T>(ps, mp, jb, cap);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3((unsigned)G);
    cfg.blockDim = dim3(PANEL_THREADS);
    cfg.dynamicSmemBytes = ps.smem;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, qr_panel_kernel<T, SYNC_CLUSTER>, &cfg) ==
            cudaSuccess &&
        nclusters >= 1)
      return 0;
    (void)cudaGetLastError();  // the smaller cluster, then the cooperative grid
    if (cmax == kPanelClusterMax) break;
  }
  // taller panels: a cooperative grid of clusters of C CTAs when the tuning
  // table asks for it (MAK_PANEL_HIER_C), else a plain cooperative grid
  const int hc = (int)tuning(TUNE_PANEL_HIER_C);
  if (hc == 2 || hc == 4 || hc == 8) {
    int64_t H = ceil_div(ceil_div(mp, 64), hc);
    if (H * hc > want_ctas) H = want_ctas / hc;
    if (H * hc > max_ctas) H = max_ctas / hc;
    if (H >= 1) {
      int64_t rpc = ceil_div(mp, H * hc);
      if (rpc <= rpc_max) {
        ps.G = (int)(H * hc);
        ps.rpc = (int)rpc;
        ps.sync = SYNC_HIER;
        ps.cl = hc;
        ps.smem = (size_t)(ps.rpc | 1) * jb * sizeof(T);
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        cfg.gridDim = dim3((unsigned)ps.G);
        cfg.blockDim = dim3(PANEL_THREADS);
        cfg.dynamicSmemBytes = ps.smem;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)hc;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int nclusters = 0;
        if (cudaOccupancyMaxActiveClusters(&nclusters, qr_panel_kernel<T, SYNC_HIER>, &cfg) ==
                cudaSuccess &&
            nclusters >= H)
          return 0;
        (void)cudaGetLastError();
      }
    }
  }
  int64_t G = ceil_div(mp, 64);
  if (G > want_ctas) G = want_ctas;
  if (G > max_ctas) G = max_ctas;
  if (G < 1) G = 1;
  int64_t rpc = ceil_div(mp, G);
  if (rpc > rpc_max) {
    G = ceil_div(mp, rpc_max);
    if (G > max_ctas) return MAK_ERR_UNSUPPORTED;
    rpc = ceil_div(mp, G);
  }
  if (rpc < 1) rpc = 1;
  G = ceil_div(mp, rpc);
  if (G < 1) G = 1;
  ps.G = (int)G;
  ps.rpc = (int)rpc;
  ps.sync = SYNC_GRID;
  ps.cl = 1;
  panel_smem<T>(ps, mp, jb, cap);
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, qr_panel_kernel<T, SYNC_GRID>,
                                                    PANEL_THREADS, ps.smem) != cudaSuccess)
    return MAK_ERR_CUDA;
  if ((int64_t)per_sm * max_ctas < G) return MAK_ERR_UNSUPPORTED;
  return 0;
}

template <class T>
int qr_run(cudaStream_t st, int64_t m, int64_t n, T* A, int64_t lda, T* Q, int64_t ldq,
           int64_t qcols, T* R, int64_t ldr, int64_t rrows, int positive, int blocksize,
           int precision, Arena& ar, mak_info* info) {
  const int64_t k = m < n ? m : n;
  const int nb = (blocksize > 0 && blocksize < NBMAX) ? blocksize : NBMAX;
  const int64_t nblk = ceil_div(k, nb);
  const int64_t wmax = (n > qcols ? n : qcols);
  const int sms = num_sms();
  const int gmax = sms;  // upper bound on panel CTAs (for workspace sizing)
  const int max_splits = 64;
  // mixed precision: 128-wide outer blocks whose block reflector is applied
  // with split-precision tensor-core GEMMs (K = 128 or K = m)
  // the 128-wide blocking pays only when its products are large enough to
  // take the split tensor-core path (gemm_prec's threshold); smaller
  // problems run the native blocking even when mixed precision is asked for
  const bool mixed = precision == MAK_PREC_MIXED && sizeof(real_t<T>) == 8 &&
                     (traits<T>::cpx ? 4.0 : 1.0) * (double)m * (double)n * QR_OUTER_NB >=
                         split_min_mnk();
  // outer block of the mixed path: 128 columns, or 64 for blocks whose
  // columns number at most MAK_QR_OUTER64_MAX_N (default 0: never), where
  // fewer 32-wide panels per block leave fewer within-block native updates
  const int NBM = mixed ? ((double)n <= tuning(TUNE_QR_OUTER64_MAX_N) ? 64 : QR_OUTER_NB) : nb;
  // Large problems apply wider block reflectors: two 128-wide blocks merged
  // for the trailing updates (the second is updated with the first on its
  // own), four for Q, whose T factors all exist by then.  A product with K =
  // 256 or 512 reads and writes C, cuts C's digit planes and finds C's maxima
  // half or a quarter as often, and amortises its epilogue over more of K
  // (16384 x 8192: K = 128 643, 256 955, 512 1005 bf16 TFLOP/s).  From the
  // size that takes the look-ahead: below it a block's panels are longer than
  // the update they would merge.
  const bool wide = mixed && NBM == QR_OUTER_NB && (double)m * n >= QR_WIDE_MIN_MN;
  const int NBO = wide ? 2 * NBM : NBM;
  const int NBQ = wide ? 4 * NBM : NBM;
  const int64_t nblk_o = ceil_div(k, NBO);

  T* tau = ar.take<T>(k > 0 ? k : 1);
  T* Ts = ar.take<T>((size_t)(nblk > 0 ? nblk : 1) * NBMAX * NBMAX);
  T* sgn = ar.take<T>(k > 0 ? k : 1);
  T* Wpart = ar.take<T>((size_t)max_splits * nb * (wmax > 0 ? wmax : 1));
  T* W2 = ar.take<T>((size_t)nb * (wmax > 0 ? wmax : 1));
  // norm partials [2 round parities][3][gmax] + the rescaled sums [gmax];
  // dot partials [2 parities][gmax][NBMAX] + the rescaled path's [gmax][NBMAX]
  // + column j+1's [2 parities][gmax][NBMAX]
  real_t<T>* part_nrm = ar.take<real_t<T>>((size_t)7 * gmax);
  T* part_w = ar.take<T>((size_t)5 * gmax * NBMAX);
  T* part_g = ar.take<T>((size_t)gmax * NBMAX * NBMAX);
  T* alpha_buf = ar.take<T>(4 * NBMAX);  // rows j and j+1 of the panel, by round parity
  T* gram_buf = ar.take<T>((size_t)NBMAX * NBMAX);
  unsigned* bar = ar.take<unsigned>(2);
  int* cflag = ar.take<int>(gmax);
  T *To = nullptr, *Gm = nullptr, *Xm = nullptr, *Tq = nullptr, *Wm = nullptr, *W2m = nullptr;
  char* ozs = nullptr;
  size_t oz_bytes = 0;
  auto scratch_for = [&](const int64_t (*shapes)[3], int count) -> size_t {
    size_t bytes = 0;
    for (int q = 0; q < count; q++) {
      Arena meas(nullptr, 0);
      gemm_prec<T>(st, precision, shapes[q][0], shapes[q][1], shapes[q][2], one_<T>(),
                   opnd<T>(nullptr, 1), opnd<T>(nullptr, 1), zero_<T>(), nullptr, 1, meas,
                   nullptr);
      if (meas.off + 1024 > bytes) bytes = meas.off + 1024;
    }
    return bytes;
  };
  if (mixed) {
    To = ar.take<T>((size_t)(nblk_o > 0 ? nblk_o : 1) * NBO * NBO);
    Gm = ar.take<T>((size_t)NBO * NBO);
    Wm = ar.take<T>((size_t)NBQ * (wmax > 0 ? wmax : 1));
    W2m = ar.take<T>((size_t)NBQ * (wmax > 0 ? wmax : 1));
    if (wide) {
      Xm = ar.take<T>((size_t)NBO * NBO);
      Tq = ar.take<T>((size_t)NBQ * NBQ);
    }
    // the tensor-core GEMMs run one after another and share one scratch region
    const int64_t shapes[4][3] = {{NBQ, wmax, m}, {m, wmax, NBQ}, {NBQ, wmax, NBQ}, {NBO, NBO, m}};
    oz_bytes = scratch_for(shapes, 4);
    ozs = ar.take<char>(oz_bytes);
  }
  // the block Gram matrix and the within-block updates of the panels run on
  // the look-ahead stream: their own scratch, and (mixed) W / T^H W of a
  // panel's update or of a 128-wide block's update inside its pair
  size_t gram_bytes = 0;
  char* grams = nullptr;
  T *Wp = nullptr, *W2p = nullptr;
  const bool panel_split = mixed && tuning(TUNE_QR_PANEL_SPLIT) != 0;
  if (mixed) {
    const int64_t shapes[5][3] = {{NBM, NBM, m}, {NBMAX, NBM, m}, {m, NBM, NBMAX},
                                  {m, NBM, NBM}, {NBM, NBM, NBM}};
    gram_bytes = scratch_for(shapes, wide ? 5 : (panel_split ? 3 : 1));
    grams = ar.take<char>(gram_bytes);
    if (panel_split || wide) {
      Wp = ar.take<T>((size_t)(wide ? NBM : NBMAX) * NBM);
      W2p = ar.take<T>((size_t)(wide ? NBM : NBMAX) * NBM);
    }
  }
  if (ar.base == nullptr) return 0;
  if (!ar.ok()) return MAK_ERR_WORKSPACE;
  int* status = &info->status;

  MAK_CUDA_TRY(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), st));

  // C <- (I - V op(T) V^H) C with the tensor-core GEMMs; op(T) = T^H for the
  // factorization, T for Q formation (T is JB x JB upper, leading dimension
  // ldt), on the scratch W / W2 / sb[0, sbytes) of the stream it runs on
  // max_ctas > 0 leaves the other SMs to the look-ahead side stream
  auto larfb_on = [&](const T* V, int64_t mp, int JB, const T* Tm, int ldt, int conjtrans, T* Cm,
                      int64_t ldc, int64_t nc, cudaStream_t s, int max_ctas, T* W, T* W2,
                      char* sb, size_t sbytes) -> int {
    if (nc <= 0) return 0;
    {
      Arena oz(sb, sbytes);
      MAK_TRY(gemm_prec<T>(s, precision, JB, nc, mp, one_<T>(),
                           opnd<T>(V, lda, OP_C, MASK_UNIT_LOWER), opnd<T>(Cm, ldc), zero_<T>(),
                           W, JB, oz, status, max_ctas));
    }
    {
      Arena oz(sb, sbytes);
      MAK_TRY(gemm_prec<T>(s, precision, JB, nc, JB, one_<T>(),
                           opnd<T>(Tm, ldt, conjtrans ? OP_C : OP_N, MASK_UPPER), opnd<T>(W, JB),
                           zero_<T>(), W2, JB, oz, status, max_ctas));
    }
    Arena oz(sb, sbytes);
    return gemm_prec<T>(s, precision, mp, nc, JB, -one_<T>(),
                        opnd<T>(V, lda, OP_N, MASK_UNIT_LOWER), opnd<T>(W2, JB), one_<T>(), Cm,
                        ldc, oz, status, max_ctas);
  };
  auto larfb_mixed = [&](const T* V, int64_t mp, int JB, const T* Tm, int ldt, int conjtrans,
                         T* Cm, int64_t ldc, int64_t nc, cudaStream_t s, int max_ctas) -> int {
    return larfb_on(V, mp, JB, Tm, ldt, conjtrans, Cm, ldc, nc, s, max_ctas, Wm, W2m, ozs,
                    oz_bytes);
  };
  // T of two block reflectors side by side (ja columns from j0, then jb): its
  // diagonal blocks Ta, Tb are in place in Tm, its corner is -Ta (Va^H Vb) Tb
  // (V = [Va Vb], Vb zero above row j0 + ja).  G and X: scratch of ja x jb.
  auto merge_t = [&](int64_t j0, int ja, int jb, T* Tm, int ldt, T* G, T* X, cudaStream_t s,
                     char* sb, size_t sbytes, int max_ctas) -> int {
    const int64_t j1 = j0 + ja;
    {
      Arena oz(sb, sbytes);
      MAK_TRY(gemm_prec<T>(s, precision, ja, jb, m - j1, one_<T>(),
                           opnd<T>(A + j1 + j0 * lda, lda, OP_C),
                           opnd<T>(A + j1 + j1 * lda, lda, OP_N, MASK_UNIT_LOWER), zero_<T>(), G,
                           ja, oz, status, max_ctas));
    }
    MAK_TRY(gemm<T>(s, ja, jb, jb, one_<T>(), opnd<T>(G, ja),
                    opnd<T>(Tm + ja + (int64_t)ja * ldt, ldt, OP_N, MASK_UPPER), zero_<T>(), X, ja));
    return gemm<T>(s, ja, jb, ja, -one_<T>(), opnd<T>(Tm, ldt, OP_N, MASK_UPPER), opnd<T>(X, ja),
                   zero_<T>(), Tm + (int64_t)ja * ldt, ldt);
  };
  // C = A[j0:, c0:c1] <- (I - V T^H V^H)... with the native SIMT kernels
  auto larfb_native = [&](int64_t j0, int jb, const T* Tb, int64_t c0, int64_t c1,
                          cudaStream_t s) -> int {
    const int64_t nt = c1 - c0;
    if (nt <= 0) return 0;
    const int64_t mp = m - j0;
    const T* Ap = A + j0 + j0 * lda;
    T* C = A + j0 + c0 * lda;
    int splits = pick_splits<T>(jb, nt, mp, sms);
    if (splits > max_splits) splits = max_splits;
    int used = 1;
    MAK_TRY(gemm<T>(s, jb, nt, mp, one_<T>(), opnd<T>(Ap, lda, OP_C, MASK_UNIT_LOWER),
                    opnd<T>(C, lda), zero_<T>(), Wpart, jb, splits, (int64_t)jb * nt, &used));
    note_launch();
    reduce_trmm_kernel<T><<<(unsigned)ceil_div(nt, trmm_cols(jb)), 256, 0, s>>>(jb, (int)nt, used, Wpart,
                                                                      (int64_t)jb * nt, Tb, 1, W2);
    MAK_CUDA_TRY(cudaGetLastError());
    return gemm<T>(s, mp, nt, jb, -one_<T>(), opnd<T>(Ap, lda, OP_N, MASK_UNIT_LOWER),
                   opnd<T>(W2, jb), one_<T>(), C, lda);
  };
  // mixed: a 32-wide panel's reflector applied to the rest of its 128-wide
  // block with split products (W = V^H C, W2 = T^H W, C -= V W2) on the
  // side stream's scratch; gemm_prec keeps products below the split gate
  // native
  auto larfb_panel_split = [&](int64_t j0, int jb, const T* Tb, int64_t c0, int64_t c1,
                               cudaStream_t s) -> int {
    const int64_t nt = c1 - c0;
    if (nt <= 0) return 0;
    const int64_t mp = m - j0;
    const T* Ap = A + j0 + j0 * lda;
    T* C = A + j0 + c0 * lda;
    const int mc = s == st ? 0 : tl_side_ctas;
    {
      Arena ga(grams, gram_bytes);
      MAK_TRY(gemm_prec<T>(s, precision, jb, nt, mp, one_<T>(),
                           opnd<T>(Ap, lda, OP_C, MASK_UNIT_LOWER), opnd<T>(C, lda), zero_<T>(),
                           Wp, jb, ga, status, mc));
    }
    note_launch();
    reduce_trmm_kernel<T><<<(unsigned)ceil_div(nt, trmm_cols(jb)), 256, 0, s>>>(jb, (int)nt, 1, Wp,
                                                                      (int64_t)jb * nt, Tb, 1, W2p);
    MAK_CUDA_TRY(cudaGetLastError());
    Arena ga(grams, gram_bytes);
    return gemm_prec<T>(s, precision, mp, nt, jb, -one_<T>(),
                        opnd<T>(Ap, lda, OP_N, MASK_UNIT_LOWER), opnd<T>(W2p, jb), one_<T>(), C,
                        lda, ga, status, mc);
  };
  // one 32-wide panel (cooperative launch)
  // on the look-ahead stream the panel takes a few SMs only, leaving the
  // rest to the trailing GEMM it overlaps with
  auto panel = [&](int64_t j0, int jb, cudaStream_t s) -> int {
    const int64_t mp = m - j0;
    PanelShape ps;
    MAK_TRY(panel_shape<T>(mp, jb, ps, s == st ? sms : tl_side_ctas, s == st));
    PanelArgs<T> pa{A + j0 + j0 * lda, lda, (int)mp, jb, ps.rpc, tau + j0,
                    Ts + (j0 / nb) * NBMAX * NBMAX, part_nrm, part_w, part_g, alpha_buf,
                    gram_buf, bar, cflag, status, gmax, ps.sync != SYNC_HIER && tuning(TUNE_PANEL_PAIR) != 0,
                    ps.block};
    ProfScope prof(s, PROF_QR_PANEL, 2.0 * (double)mp * jb * sizeof(T));
    note_launch();
    if (ps.sync == SYNC_CLUSTER || ps.sync == SYNC_HIER) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[2];
      cfg.gridDim = dim3((unsigned)ps.G);
      cfg.blockDim = dim3(PANEL_THREADS);
      cfg.dynamicSmemBytes = ps.smem;
      cfg.stream = s;
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)ps.cl;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeCooperative;
      attr[1].val.cooperative = 1;
      cfg.attrs = attr;
      cfg.numAttrs = ps.sync == SYNC_HIER ? 2 : 1;
      if (ps.sync == SYNC_HIER)
        MAK_CUDA_TRY(cudaLaunchKernelEx(&cfg, qr_panel_kernel<T, SYNC_HIER>, pa));
      else
        MAK_CUDA_TRY(cudaLaunchKernelEx(&cfg, qr_panel_kernel<T, SYNC_CLUSTER>, pa));
      return 0;
    }
    void* args[] = {&pa};
    MAK_CUDA_TRY(cudaLaunchCooperativeKernel((void*)qr_panel_kernel<T, SYNC_GRID>, dim3(ps.G),
                                             dim3(PANEL_THREADS), args, ps.smem, s));
    return 0;
  };
  // factor outer block b: its panels with updates confined to their 128-wide
  // block, (mixed) the block's T factor from its Gram matrix, and (wide) the
  // first block's reflector applied to the second, then their T merged
  auto factor_block = [&](int64_t b, cudaStream_t s) -> int {
    const int64_t J0 = b * NBO;
    const int JB = (int)((k - J0) < NBO ? (k - J0) : NBO);
    const int mc = s == st ? 0 : tl_side_ctas;
    T* const Tb = mixed ? To + b * NBO * NBO : nullptr;
    for (int64_t M0 = J0; M0 < J0 + JB; M0 += NBM) {
      const int MB = (int)((J0 + JB - M0) < NBM ? (J0 + JB - M0) : NBM);
      for (int64_t j0 = M0; j0 < M0 + MB; j0 += nb) {
        const int jb = (int)((M0 + MB - j0) < nb ? (M0 + MB - j0) : nb);
        MAK_TRY(panel(j0, jb, s));
        if (panel_split)
          MAK_TRY(larfb_panel_split(j0, jb, Ts + (j0 / nb) * NBMAX * NBMAX, j0 + jb, M0 + MB, s));
        else
          MAK_TRY(larfb_native(j0, jb, Ts + (j0 / nb) * NBMAX * NBMAX, j0 + jb, M0 + MB, s));
      }
      if (!mixed) return 0;
      const T* V = A + M0 + M0 * lda;
      {
        // the Gram matrix fixes the orthogonality of the block reflector; the
        // split-precision product is FP64-accurate, and 2 m 128^2 flops per
        // block on the FP64 pipe would sit on the look-ahead's critical path
        Arena ga(grams, gram_bytes);
        MAK_TRY(gemm_prec<T>(s, precision, MB, MB, m - M0, one_<T>(),
                             opnd<T>(V, lda, OP_C, MASK_UNIT_LOWER),
                             opnd<T>(V, lda, OP_N, MASK_UNIT_LOWER), zero_<T>(), Gm, MB, ga,
                             status, mc));
      }
      T* const Tmid = Tb + (M0 - J0) * (NBO + 1);
      note_launch();
      larft_blocks_kernel<T><<<(unsigned)ceil_div(MB, LARFT_WARPS), 32 * LARFT_WARPS, 0, s>>>(
          MB, nb, Gm, MB, Ts + (M0 / nb) * NBMAX * NBMAX, Tmid, NBO);
      MAK_CUDA_TRY(cudaGetLastError());
      const int rest = (int)(J0 + JB - M0 - MB);
      if (rest > 0)
        MAK_TRY(larfb_on(V, m - M0, MB, Tmid, NBO, 1, A + M0 + (M0 + MB) * lda, lda, rest, s, mc,
                         Wp, W2p, grams, gram_bytes));
    }
    if (JB > NBM)
      MAK_TRY(merge_t(J0, NBM, JB - NBM, Tb, NBO, Gm, Xm, s, grams, gram_bytes, mc));
    return 0;
  };
  // block b's reflector applied to the columns [c0, c1)
  auto apply_block = [&](int64_t b, int64_t c0, int64_t c1, cudaStream_t s,
                         int max_ctas) -> int {
    const int64_t J0 = b * NBO;
    const int JB = (int)((k - J0) < NBO ? (k - J0) : NBO);
    if (mixed)
      return larfb_mixed(A + J0 + J0 * lda, m - J0, JB, To + b * NBO * NBO, NBO, 1,
                         A + J0 + c0 * lda, lda, c1 - c0, s, max_ctas);
    return larfb_native(J0, JB, Ts + (J0 / nb) * NBMAX * NBMAX, c0, c1, s);
  };

  // ------------------------------------------------------------ factor
  // Look-ahead: block b's reflector is applied first to block b+1's columns;
  // a high-priority side stream then factors block b+1 while the main stream
  // applies block b to the remaining columns, so the latency-bound panels
  // hide behind the large trailing GEMMs.
  LookAhead* la = (nblk_o > 1 && lookahead_enabled() && (double)m * n >= 4.0e6) ? lookahead()
                                                                                  : nullptr;
  if (nblk_o > 0) MAK_TRY(factor_block(0, st));
  for (int64_t b = 0; b < nblk_o; b++) {
    const int64_t J0 = b * NBO;
    const int64_t nx = J0 + ((k - J0) < NBO ? (k - J0) : NBO);          // first column of b+1
    const bool has_next = b + 1 < nblk_o;
    const int64_t nx_end = has_next ? nx + ((k - nx) < NBO ? (k - nx) : NBO) : nx;
    if (has_next && la) {
      MAK_TRY(apply_block(b, nx, nx_end, st, 0));
      MAK_CUDA_TRY(cudaEventRecord(la->ev_ready, st));
      MAK_CUDA_TRY(cudaStreamWaitEvent(la->side, la->ev_ready, 0));
      tl_side_ctas = side_ctas(n - nx_end);
      if (tl_side_ctas > sms - 8) tl_side_ctas = sms - 8;
      MAK_TRY(factor_block(b + 1, la->side));
      MAK_CUDA_TRY(cudaEventRecord(la->ev_done, la->side));
      // the persistent tensor-core grid leaves the side stream its SMs
      MAK_TRY(apply_block(b, nx_end, n, st, sms - tl_side_ctas));
      MAK_CUDA_TRY(cudaStreamWaitEvent(st, la->ev_done, 0));
    } else {
      MAK_TRY(apply_block(b, nx, n, st, 0));
      if (has_next) MAK_TRY(factor_block(b + 1, st));
    }
  }

  // ------------------------------------------------------ R and the gauge
  if (k > 0) {
    note_launch();
    signs_kernel<T><<<(unsigned)ceil_div(k, 256), 256, 0, st>>>((int)k, A, lda, positive, sgn);
    MAK_CUDA_TRY(cudaGetLastError());
  }
  if (R != nullptr && rrows > 0 && n > 0) {
    dim3 g((unsigned)ceil_div(rrows, 256), (unsigned)(n < 65535 ? n : 65535));
    note_launch();
    extract_r_kernel<T><<<g, 256, 0, st>>>(rrows, n, k, A, lda, sgn, R, ldr);
    MAK_CUDA_TRY(cudaGetLastError());
  }
  if (m > 0 && qcols > 0) {
    dim3 g((unsigned)ceil_div(m, 256), (unsigned)(qcols < 65535 ? qcols : 65535));
    note_launch();
    init_q_kernel<T><<<g, 256, 0, st>>>(m, qcols, k, sgn, Q, ldq);
    MAK_CUDA_TRY(cudaGetLastError());
  }

  // ------------------------------------------- Q = H_1 ... H_k [diag(s); 0]
  if (mixed) {
    for (int64_t bq = ceil_div(k, NBQ) - 1; bq >= 0; bq--) {
      const int64_t J0 = bq * NBQ;
      const int JB = (int)((k - J0) < NBQ ? (k - J0) : NBQ);
      const int64_t qt = qcols - J0;
      if (qt <= 0) continue;
      const T* Tm = To + (J0 / NBO) * NBO * NBO;
      int ldt = NBO;
      if (JB > NBO) {  // two outer blocks' T factors merged
        const int jb = JB - NBO;
        MAK_TRY(copy_mat<T>(st, NBO, NBO, Tm, NBO, Tq, NBQ));
        MAK_TRY(copy_mat<T>(st, jb, jb, Tm + NBO * NBO, NBO, Tq + NBO * (NBQ + 1), NBQ));
        MAK_TRY(merge_t(J0, NBO, jb, Tq, NBQ, Gm, Xm, st, ozs, oz_bytes, 0));
        Tm = Tq;
        ldt = NBQ;
      }
      MAK_TRY(larfb_mixed(A + J0 + J0 * lda, m - J0, JB, Tm, ldt, 0, Q + J0 + J0 * ldq, ldq, qt,
                          st, 0));
    }
    return 0;
  }
  for (int64_t bi = nblk - 1; bi >= 0; bi--) {
    const int64_t j0 = bi * nb;
    const int jb = (int)((k - j0) < nb ? (k - j0) : nb);
    const int64_t mp = m - j0;
    const int64_t qt = qcols - j0;
    if (qt <= 0) continue;
    const T* Ap = A + j0 + j0 * lda;
    const T* Tb = Ts + bi * NBMAX * NBMAX;
    T* Qs = Q + j0 + j0 * ldq;
    int splits = pick_splits<T>(jb, qt, mp, sms);
    if (splits > max_splits) splits = max_splits;
    int used = 1;
    MAK_TRY(gemm<T>(st, jb, qt, mp, one_<T>(), opnd<T>(Ap, lda, OP_C, MASK_UNIT_LOWER),
                    opnd<T>(Qs, ldq), zero_<T>(), Wpart, jb, splits, (int64_t)jb * qt, &used));
    note_launch();
    reduce_trmm_kernel<T><<<(unsigned)ceil_div(qt, trmm_cols(jb)), 256, 0, st>>>(
        jb, (int)qt, used, Wpart, (int64_t)jb * qt, Tb, 0, W2);
    MAK_CUDA_TRY(cudaGetLastError());
    MAK_TRY(gemm<T>(st, mp, qt, jb, -one_<T>(), opnd<T>(Ap, lda, OP_N, MASK_UNIT_LOWER),
                    opnd<T>(W2, jb), one_<T>(), Qs, ldq));
  }
  return 0;
}

#define MAK_INST_QR(T)                                                                        \
  template int qr_run<T>(cudaStream_t, int64_t, int64_t, T*, int64_t, T*, int64_t, int64_t, \
                         T*, int64_t, int64_t, int, int, int, Arena&, mak_info*);
MAK_INST_QR(double)
MAK_INST_QR(float)
MAK_INST_QR(zcomplex)
MAK_INST_QR(ccomplex)

// ------------------------------------------------------------ C entry ---

template <class T>
static int qr_entry(int full, int64_t m, int64_t n, void* Av, int64_t lda, void* Qv, int64_t ldq,
                    void* Rv, int64_t ldr, const mak_qr_opts* opts, void* work, size_t work_bytes,
                    mak_info* info, mak_stream_t stream) {
  T* A = (T*)Av;
  T* Q = (T*)Qv;
  T* R = (T*)Rv;
  if (m < 0) return -1;
  if (n < 0) return -2;
  const int64_t k = m < n ? m : n;
  const int64_t qcols = full ? m : k;
  const int64_t rrows = full ? m : k;
  if (A == nullptr && m * n > 0) return -3;
  if (lda < (m > 1 ? m : 1)) return -4;
  if (Q == nullptr && m * qcols > 0) return -5;
  if (Q != nullptr && (void*)Q == (void*)A) return -5;  // in-place Q is not provided
  if (ldq < (m > 1 ? m : 1)) return -6;
  if (R != nullptr && ldr < (rrows > 1 ? rrows : 1)) return -8;
  mak_qr_opts o{1, 0, MAK_PREC_NATIVE, 0};
  if (opts) o = *opts;
  if (o.blocksize < 0 || o.blocksize > NBMAX) return -9;
  if (o.precision != MAK_PREC_NATIVE && o.precision != MAK_PREC_MIXED) return -9;
  cudaStream_t st = (cudaStream_t)stream;
  Arena ar(work, work_bytes);
  mak_info* inf = info ? info : ar.take<mak_info>(1);
  if (work == nullptr && info == nullptr) return -11;
  // size check first (a measuring pass)
  {
    Arena meas(nullptr, 0);
    if (!info) meas.take<mak_info>(1);
    qr_run<T>(st, m, n, nullptr, lda, nullptr, ldq, qcols, nullptr, ldr, rrows, o.positive,
              o.blocksize, o.precision, meas, nullptr);
    if (meas.off > work_bytes) return -12;
  }
  MAK_TRY(info_reset(st, inf));
  return qr_run<T>(st, m, n, A, lda, Q, ldq, qcols, R, ldr, rrows, o.positive, o.blocksize,
                   o.precision, ar, inf);
}

}  // namespace mak

using namespace mak;

extern "C" {

int mak_qr_workspace(int dtype, int64_t m, int64_t n, int full, const mak_qr_opts* opts,
                     size_t* bytes) {
  if (bytes == nullptr) return -6;
  if (m < 0) return -2;
  if (n < 0) return -3;
  mak_qr_opts o{1, 0, MAK_PREC_NATIVE, 0};
  if (opts) o = *opts;
  const int64_t k = m < n ? m : n;
  const int64_t qcols = full ? m : k;
  const int64_t rrows = full ? m : k;
  Arena meas(nullptr, 0);
  meas.take<mak_info>(1);
  switch (dtype) {
    case MAK_F64: qr_run<double>(0, m, n, nullptr, m, nullptr, m, qcols, nullptr, rrows, rrows, o.positive, o.blocksize, o.precision, meas, nullptr); break;
    case MAK_C64: qr_run<zcomplex>(0, m, n, nullptr, m, nullptr, m, qcols, nullptr, rrows, rrows, o.positive, o.blocksize, o.precision, meas, nullptr); break;
    case MAK_F32: qr_run<float>(0, m, n, nullptr, m, nullptr, m, qcols, nullptr, rrows, rrows, o.positive, o.blocksize, o.precision, meas, nullptr); break;
    case MAK_C32: qr_run<ccomplex>(0, m, n, nullptr, m, nullptr, m, qcols, nullptr, rrows, rrows, o.positive, o.blocksize, o.precision, meas, nullptr); break;
    default: return -1;
  }
  *bytes = meas.off + 256;
  return 0;
}

#define MAK_QR_ENTRY(NAME, FULL, T, PT)                                                        \
  int NAME(int64_t m, int64_t n, PT* A, int64_t lda, PT* Q, int64_t ldq, PT* R, int64_t ldr,   \
           const mak_qr_opts* opts, void* work, size_t work_bytes, mak_info* info,             \
           mak_stream_t stream) {                                                              \
    return qr_entry<T>(FULL, m, n, A, lda, Q, ldq, R, ldr, opts, work, work_bytes, info,       \
                       stream);                                                                \
  }
MAK_QR_ENTRY(mak_qr_compact_d, 0, double, double)
MAK_QR_ENTRY(mak_qr_compact_z, 0, zcomplex, void)
MAK_QR_ENTRY(mak_qr_compact_s, 0, float, float)
MAK_QR_ENTRY(mak_qr_compact_c, 0, ccomplex, void)
MAK_QR_ENTRY(mak_qr_full_d, 1, double, double)
MAK_QR_ENTRY(mak_qr_full_z, 1, zcomplex, void)
MAK_QR_ENTRY(mak_qr_full_s, 1, float, float)
MAK_QR_ENTRY(mak_qr_full_c, 1, ccomplex, void)

uint64_t mak_kernel_launches(void) { return (uint64_t)launch_counter().load(); }

const char* mak_version(void) { return "mak_gb300 0.1.0 (sm_103a)"; }

const char* mak_status_string(int code) {
  if (code == MAK_OK) return "ok";
  if (code < 0) return "invalid argument (-index of the offending argument)";
  switch (code) {
    case MAK_ERR_CUDA: return "CUDA launch or runtime error";
    case MAK_ERR_TIMEOUT: return "bounded device-side wait gave up";
    case MAK_ERR_UNSUPPORTED: return "shape outside the supported envelope";
    case MAK_ERR_WORKSPACE: return "workspace too small";
    default: return "unknown status";
  }
}

}  // extern "C"
