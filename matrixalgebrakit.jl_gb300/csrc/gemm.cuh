// Native-precision tiled GEMM on the SIMT pipes (FP64 DFMA, FP32 FFMA,
// complex as 4 real FMAs), with structured operands.
//
//   C = alpha * op(A) * op(B) + beta * C
//
// op(X) in {N, T, C}; each operand may additionally be read through a
// structure mask of its *stored* matrix: unit-lower-trapezoidal (Householder
// V: implicit 1 on the diagonal, 0 above), upper or lower triangular.  This
// lets the larfb / orgqr / pullback products read V and R straight out of the
// packed QR storage without materialising copies.
//
// On GB300 FP64 runs at ~1 TFLOP/s for the whole chip (measured: DFMA and
// DMMA alike), i.e. ~2 multiply-adds per clock per SM, so even a 16 x 16 tile
// is bound by the FP64 pipe and the only question is whether every SM has
// work; the tensor-core path is the split-precision GEMM in ozaki.cu.
#pragma once
#include "mak_common.cuh"

namespace mak {

enum Op { OP_N = 0, OP_T = 1, OP_C = 2 };
enum Mask { MASK_FULL = 0, MASK_UNIT_LOWER = 1, MASK_UPPER = 2, MASK_LOWER = 3 };

template <class T>
struct Operand {
  const T* p;
  int64_t ld;
  int op;
  int mask;
};
template <class T>
inline Operand<T> opnd(const T* p, int64_t ld, int op = OP_N, int mask = MASK_FULL) {
  return Operand<T>{p, ld, op, mask};
}

// element (i, k) of op(X); (r, c) is the position in the stored matrix
template <class T>
__device__ __forceinline__ T load_op(const Operand<T>& X, int64_t i, int64_t k) {
  int64_t r = (X.op == OP_N) ? i : k;
  int64_t c = (X.op == OP_N) ? k : i;
  switch (X.mask) {
    case MASK_UNIT_LOWER:
      if (r < c) return zero_<T>();
      if (r == c) return one_<T>();
      break;
    case MASK_UPPER:
      if (r > c) return zero_<T>();
      break;
    case MASK_LOWER:
      if (r < c) return zero_<T>();
      break;
    default:
      break;
  }
  T v = X.p[r + c * X.ld];
  return X.op == OP_C ? conj_(v) : v;
}

int num_sms();
constexpr int GEMM_BK = 32;  // K per step (and the granule of a K split)
constexpr int GEMM_GRID_Y = 65535;  // column tiles per launch

template <class T>
__device__ __forceinline__ bool is_zero_(T v) { return v == zero_<T>(); }

// A thread's share (L elements) of the B x BK tile of an operand at (i0, k0),
// i along the tile's B side (rows of op(A), columns of op(B)).  `ci`: the
// stored matrix is contiguous along i, so that i runs fastest over the
// threads; else k does.  A tile inside the operand that no structure mask
// touches (decided once, for the whole CTA) is read with one address step per
// element; the general form costs tens of instructions per element, three
// quarters of all issued in an FP32 update of K = 32.
template <class T, int B, int BK, int NT, int L>
__device__ __forceinline__ void fetch_tile(const Operand<T>& X, bool ci, int64_t i0, int64_t ilim,
                                           int k0, int kend, T (&v)[L]) {
  const int tid = threadIdx.x;
  bool plain = i0 + B <= ilim && k0 + BK <= kend;
  if (X.mask != MASK_FULL) {
    const int64_t rlo = ci ? i0 : k0, rhi = rlo + (ci ? B : BK) - 1;
    const int64_t clo = ci ? k0 : i0, chi = clo + (ci ? BK : B) - 1;
    plain = plain && (X.mask == MASK_UPPER ? rhi <= clo
                                           : (X.mask == MASK_LOWER ? rlo >= chi : rlo > chi));
  }
  if (plain) {
    const T* p = X.p + (ci ? (i0 + tid % B) + (int64_t)(k0 + tid / B) * X.ld
                           : (int64_t)(k0 + tid % BK) + (i0 + tid / BK) * X.ld);
    const int64_t step = (ci ? NT / B : NT / BK) * X.ld;
#pragma unroll
    for (int q = 0; q < L; q++) v[q] = p[q * step];
    if (traits<T>::cpx && X.op == OP_C) {
#pragma unroll
      for (int q = 0; q < L; q++) v[q] = conj_(v[q]);
    }
    return;
  }
#pragma unroll
  for (int q = 0; q < L; q++) {
    const int e = tid + q * NT;
    const int64_t gi = i0 + (ci ? e % B : e / BK);
    const int gk = k0 + (ci ? e / B : e % BK);
    T x = zero_<T>();
    if (gi < ilim && gk < kend) {
      const int64_t r = ci ? gi : gk, c = ci ? gk : gi;
      if (X.mask == MASK_UNIT_LOWER && r <= c) x = r == c ? one_<T>() : zero_<T>();
      else if ((X.mask == MASK_UPPER && r > c) || (X.mask == MASK_LOWER && r < c)) x = zero_<T>();
      else x = X.p[r + c * X.ld];
      if (X.op == OP_C) x = conj_(x);
    }
    v[q] = x;
  }
}

// One BM x BN tile of C per CTA of 256 threads (TM x TN outputs each).  The
// next K step's elements are fetched into registers while the current one is
// multiplied.
template <class T, int BM, int BN, int BK, int TM, int TN, bool kCut>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_kernel(int M, int N, int K, T alpha, Operand<T> A, Operand<T> B, T beta, T* C,
            int64_t ldc, int kchunk, int64_t split_stride, int64_t col0, const int* skip) {
  if (skipped(skip)) return;
  constexpr int RX = BM / TM;  // threads along rows
  constexpr int RY = BN / TN;  // threads along columns
  constexpr int NT = RX * RY;
  constexpr int LA = BM * BK / NT, LB = BN * BK / NT;  // elements fetched per thread
  static_assert(LA * NT == BM * BK && LB * NT == BN * BK, "whole tiles");
  __shared__ T As[BK][BM + 1];
  __shared__ T Bs[BK][BN + 1];
  const int64_t m0 = (int64_t)blockIdx.x * BM;
  const int64_t n0 = col0 + (int64_t)blockIdx.y * BN;
  const int kbeg = blockIdx.z * kchunk;
  const int kend = min(K, kbeg + kchunk);
  C += blockIdx.z * split_stride;
  const int tid = threadIdx.x;
  const int tx = tid % RX, ty = tid / RX;
  T acc[TM][TN];
#pragma unroll
  for (int r = 0; r < TM; r++)
#pragma unroll
    for (int c = 0; c < TN; c++) acc[r][c] = zero_<T>();

  T ra[LA], rb[LB];
  static_assert(NT % BM == 0 && NT % BN == 0 && NT % BK == 0, "whole address steps");
  auto fetch = [&](int k0) {
    fetch_tile<T, BM, BK, NT, LA>(A, A.op == OP_N, m0, M, k0, kend, ra);
    fetch_tile<T, BN, BK, NT, LB>(B, B.op != OP_N, n0, N, k0, kend, rb);
  };
  if (kbeg < kend) fetch(kbeg);
  // C before the products: its loads are then in flight together (after them,
  // each would wait for the store before it, which may alias)
  const bool use_beta = !is_zero_(beta);
  T cv[TM][TN];
  if (use_beta) {
#pragma unroll
    for (int c = 0; c < TN; c++)
#pragma unroll
      for (int r = 0; r < TM; r++) {
        const int64_t i = m0 + tx + r * RX, j = n0 + ty + c * RY;
        cv[r][c] = (i < M && j < N) ? C[i + j * ldc] : zero_<T>();
      }
  }
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
    for (int q = 0; q < LA; q++) {
      const int e = tid + q * NT;
      if (A.op == OP_N) As[e / BM][e % BM] = ra[q];
      else As[e % BK][e / BK] = ra[q];
    }
#pragma unroll
    for (int q = 0; q < LB; q++) {
      const int e = tid + q * NT;
      if (B.op == OP_N) Bs[e % BK][e / BK] = rb[q];
      else Bs[e / BN][e % BN] = rb[q];
    }
    __syncthreads();
    if (k0 + BK < kend) fetch(k0 + BK);
    const auto mul = [&](int kk) {
      T a[TM], b[TN];
#pragma unroll
      for (int r = 0; r < TM; r++) a[r] = As[kk][tx + r * RX];
#pragma unroll
      for (int c = 0; c < TN; c++) b[c] = Bs[kk][ty + c * RY];
#pragma unroll
      for (int r = 0; r < TM; r++)
#pragma unroll
        for (int c = 0; c < TN; c++) acc[r][c] = fma_(a[r], b[c], acc[r][c]);
    };
    if (!kCut || k0 + BK <= kend) {
#pragma unroll 4
      for (int kk = 0; kk < BK; kk++) mul(kk);
    } else {
      for (int kk = 0; kk < kend - k0; kk++) mul(kk);
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < TN; c++) {
    int64_t j = n0 + ty + c * RY;
    if (j >= N) continue;
#pragma unroll
    for (int r = 0; r < TM; r++) {
      int64_t i = m0 + tx + r * RX;
      if (i >= M) continue;
      T v = alpha * acc[r][c];
      if (use_beta) v = fma_(beta, cv[r][c], v);
      C[i + j * ldc] = v;
    }
  }
}

// The FP32 types' tile: 128 multiply-adds per clock per SM, so the operands'
// shared-memory reads decide.  A thread's TN columns are adjacent and read as
// 16-byte vectors; its TM rows are RX apart (lanes along the rows, C accessed
// in whole lines) or, with ROWC, adjacent and read as vectors too.  Reads per
// warp and k (in 128-byte wavefronts) against FMA cycles: 128 x 64 (TM 4, TN
// 8, RX 32) 6 : 8, 64 x 64 (TM 2) 4 : 4, 32 x 128 (TM 4, TN 4, RX 8, ROWC)
// 2 : 4; the scalar reads of a 4 x 4 tile were 8 : 4.
template <class T, int BM, int BN, int BK, int TM, int TN, int RX, bool ROWC, bool kCut>
__global__ void __launch_bounds__(256)
gemm_f32_kernel(int M, int N, int K, T alpha, Operand<T> A, Operand<T> B, T beta, T* C,
                int64_t ldc, int kchunk, int64_t split_stride, int64_t col0, const int* skip) {
  if (skipped(skip)) return;
  constexpr int NT = 256, RY = NT / RX;
  static_assert(RX * TM == BM && RY * TN == BN, "256 threads cover the tile");
  constexpr int LA = BM * BK / NT, LB = BN * BK / NT;
  constexpr int V = 16 / sizeof(T);  // elements per vector read
  static_assert(TN % V == 0 && (!ROWC || TM % V == 0), "whole vectors");
  struct alignas(16) Vec { T v[V]; };
  __shared__ alignas(16) T As[BK][BM + V];
  __shared__ alignas(16) T Bs[BK][BN + V];
  const int64_t m0 = (int64_t)blockIdx.x * BM;
  const int64_t n0 = col0 + (int64_t)blockIdx.y * BN;
  const int kbeg = blockIdx.z * kchunk;
  const int kend = min(K, kbeg + kchunk);
  C += blockIdx.z * split_stride;
  const int tid = threadIdx.x, tx = tid % RX, ty = tid / RX;
  T acc[TM][TN];
#pragma unroll
  for (int r = 0; r < TM; r++)
#pragma unroll
    for (int c = 0; c < TN; c++) acc[r][c] = zero_<T>();
  T ra[LA], rb[LB];
  static_assert(NT % BM == 0 && NT % BN == 0 && NT % BK == 0, "whole address steps");
  auto fetch = [&](int k0) {
    fetch_tile<T, BM, BK, NT, LA>(A, A.op == OP_N, m0, M, k0, kend, ra);
    fetch_tile<T, BN, BK, NT, LB>(B, B.op != OP_N, n0, N, k0, kend, rb);
  };
  if (kbeg < kend) fetch(kbeg);
  // C before the products: its loads are then in flight together (after them,
  // each would wait for the store before it, which may alias)
  const bool use_beta = !is_zero_(beta);
  T cv[TM][TN];
  // (a tile inside C takes one address step per element)
  constexpr int RS = ROWC ? 1 : RX;
  const bool inner = m0 + BM <= M && n0 + BN <= N;
  const int64_t i0 = m0 + (ROWC ? tx * TM : tx), j0 = n0 + ty * TN;
  T* const C0 = C + i0 + j0 * ldc;
  if (use_beta) {
#pragma unroll
    for (int c = 0; c < TN; c++)
#pragma unroll
      for (int r = 0; r < TM; r++)
        cv[r][c] = inner || (i0 + r * RS < M && j0 + c < N) ? C0[r * RS + c * ldc] : zero_<T>();
  }
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
    for (int q = 0; q < LA; q++) {
      const int e = tid + q * NT;
      if (A.op == OP_N) As[e / BM][e % BM] = ra[q];
      else As[e % BK][e / BK] = ra[q];
    }
#pragma unroll
    for (int q = 0; q < LB; q++) {
      const int e = tid + q * NT;
      if (B.op == OP_N) Bs[e % BK][e / BK] = rb[q];
      else Bs[e / BN][e % BN] = rb[q];
    }
    __syncthreads();
    if (k0 + BK < kend) fetch(k0 + BK);
    const auto mul = [&](int kk) {
      T a[TM], b[TN];
      if constexpr (ROWC) {
#pragma unroll
        for (int r = 0; r < TM; r += V) {
          const Vec v = *reinterpret_cast<const Vec*>(&As[kk][tx * TM + r]);
#pragma unroll
          for (int q = 0; q < V; q++) a[r + q] = v.v[q];
        }
      } else {
#pragma unroll
        for (int r = 0; r < TM; r++) a[r] = As[kk][tx + r * RX];
      }
#pragma unroll
      for (int c = 0; c < TN; c += V) {
        const Vec v = *reinterpret_cast<const Vec*>(&Bs[kk][ty * TN + c]);
#pragma unroll
        for (int q = 0; q < V; q++) b[c + q] = v.v[q];
      }
#pragma unroll
      for (int r = 0; r < TM; r++)
#pragma unroll
        for (int c = 0; c < TN; c++) acc[r][c] = fma_(a[r], b[c], acc[r][c]);
    };
    if (!kCut || k0 + BK <= kend) {
#pragma unroll 4
      for (int kk = 0; kk < BK; kk++) mul(kk);
    } else {
      for (int kk = 0; kk < kend - k0; kk++) mul(kk);
    }
    __syncthreads();
  }
  if (use_beta) {
#pragma unroll
    for (int c = 0; c < TN; c++)
#pragma unroll
      for (int r = 0; r < TM; r++) acc[r][c] = fma_(beta, cv[r][c], alpha * acc[r][c]);
  } else {
#pragma unroll
    for (int c = 0; c < TN; c++)
#pragma unroll
      for (int r = 0; r < TM; r++) acc[r][c] = alpha * acc[r][c];
  }
  if (inner) {
#pragma unroll
    for (int c = 0; c < TN; c++)
#pragma unroll
      for (int r = 0; r < TM; r++) C0[r * RS + c * ldc] = acc[r][c];
  } else {
#pragma unroll
    for (int c = 0; c < TN; c++)
#pragma unroll
      for (int r = 0; r < TM; r++)
        if (i0 + r * RS < M && j0 + c < N) C0[r * RS + c * ldc] = acc[r][c];
  }
}

template <class T>
__global__ void scale_kernel(int M, int N, T beta, T* C, int64_t ldc) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t j = blockIdx.y;
  if (i < M && j < N) C[i + j * ldc] = is_zero_(beta) ? zero_<T>() : beta * C[i + j * ldc];
}

// Host launcher.  `splits` > 1 partitions K; split s writes its partial
// product (beta ignored, treated as 0) to C + s * split_stride.
template <class T>
int gemm(cudaStream_t st, int64_t M, int64_t N, int64_t K, T alpha, Operand<T> A,
         Operand<T> B, T beta, T* C, int64_t ldc, int splits = 1, int64_t split_stride = 0,
         int* used_splits = nullptr) {
  if (used_splits) *used_splits = 1;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) {
    dim3 g((unsigned)ceil_div(M, 256), (unsigned)N);
    note_launch();
    scale_kernel<T><<<g, 256, 0, st>>>((int)M, (int)N, beta, C, ldc);
    return cudaGetLastError() == cudaSuccess ? 0 : MAK_ERR_CUDA;
  }
  if (splits < 1) splits = 1;
  int kchunk = (int)ceil_div(ceil_div(K, splits), GEMM_BK) * GEMM_BK;
  splits = (int)ceil_div(K, kchunk);
  if (used_splits) *used_splits = splits;
  if (splits > 1) beta = zero_<T>();
  ProfScope prof(st, PROF_GEMM_NATIVE, (traits<T>::cpx ? 8.0 : 2.0) * M * N * K);
  // Column tiles are blockIdx.y, of which a grid has 65535: wider outputs (more
  // than 2,097,120 columns of 32) take one launch per that many tiles.
#define MAK_GEMM_COLS(BM, BN, ...)                                                               \
  for (int64_t col0 = 0; col0 < N; col0 += (int64_t)GEMM_GRID_Y * BN) {                          \
    const int64_t cols = N - col0 < (int64_t)GEMM_GRID_Y * BN ? N - col0                         \
                                                              : (int64_t)GEMM_GRID_Y * BN;       \
    note_launch();                                                                               \
    __VA_ARGS__                                                                                  \
        <<<dim3((unsigned)ceil_div(M, BM), (unsigned)ceil_div(cols, BN), (unsigned)splits), 256, \
           0, st>>>((int)M, (int)N, (int)K, alpha, A, B, beta, C, ldc, kchunk, split_stride,     \
                    col0, skip_flag());                                                          \
  }
  // Short products with a ragged K: the last step multiplies no padding (kCut).
  // Elsewhere the padding is less than a quarter, and the second loop would cost
  // more: 8192 x 4096 Float64 QR 419 -> 433 ms.
  const bool cut = K % GEMM_BK != 0 && K <= 4 * GEMM_BK;
#define MAK_GEMM_TILE(BM, BN, BK, TM, TN)                                                        \
  if (cut) {                                                                                     \
    MAK_GEMM_COLS(BM, BN, gemm_kernel<T, BM, BN, BK, TM, TN, true>)                              \
  } else {                                                                                       \
    MAK_GEMM_COLS(BM, BN, gemm_kernel<T, BM, BN, BK, TM, TN, false>)                             \
  }
  const int64_t t32 = ceil_div(M, 32) * ceil_div(N, 32) * splits;
  if constexpr (sizeof(real_t<T>) == 8) {
    // The FP64 pipe is so slow that the operand traffic of a small tile costs
    // nothing, while every SM left without a tile costs its share of the
    // chip's FP64 rate: 32 x 32 tiles from three per SM, else 16 x 16.
    // Against 64 x 64 (and 32 x 64) tiles: a 512 x 64 x 32 complex update 140
    // -> 14.5 us, 1000 x 501 Float64 QR 4.5 -> 2.6 ms, 300 uneven blocks 188
    // -> 139 ms; 3000^3 45.3 -> 44.4 ms (1.22 TFLOP/s), 700^3 0.85 -> 0.83 ms.
    // Outputs of at most 16 rows take 16 x 16 tiles at any width: half of a 32-row
    // tile would be padding (gemm call of 8 x 100000 x 8: 286 us with 32-row tiles
    // and K padded to 32, 139 now; ComplexF64 814 and 239).
    if (t32 >= 3 * (int64_t)num_sms() && M > 16) {
      MAK_GEMM_TILE(32, 32, GEMM_BK, 2, 2)
    } else {
      MAK_GEMM_TILE(16, 16, GEMM_BK, 1, 1)
    }
  } else {
    // wide tiles where they fill the GPU (their operand reads are the
    // cheapest), smaller ones before SMs idle.  The 4093 x 1537 Float32 QR:
    // W = V^H C 33 -> 20 us, C -= V W2 29 -> 19 us per panel, the LQ 6.0 ->
    // 5.0 ms (issue slots, 63 % busy; the tiles' sizes hardly matter)
#define MAK_GEMM32_TILE(BM, BN, BK, TM, TN, RX, ROWC)                                            \
  if (cut) {                                                                                     \
    MAK_GEMM_COLS(BM, BN, gemm_f32_kernel<T, BM, BN, BK, TM, TN, RX, ROWC, true>)                \
  } else {                                                                                       \
    MAK_GEMM_COLS(BM, BN, gemm_f32_kernel<T, BM, BN, BK, TM, TN, RX, ROWC, false>)               \
  }
    const int64_t sms = num_sms();
    constexpr int BK32 = 32 / (sizeof(T) / 4);
    if (M <= 32 && ceil_div(N, 128) * splits >= sms) {
      // (a short K: half the step, whose padding costs fetches; QR of 8 x
      // 1000000 Float32 579 -> 505 us, 8 x 1000000 ComplexF32 780 -> 555)
      if (2 * K <= BK32) {
        MAK_GEMM32_TILE(32, 128, BK32 / 2, 4, 4, 8, true)
      } else {
        MAK_GEMM32_TILE(32, 128, BK32, 4, 4, 8, true)
      }
    } else if (ceil_div(M, 128) * ceil_div(N, 64) * splits >= 2 * sms) {
      MAK_GEMM32_TILE(128, 64, 16, 4, 8, 32, false)
    } else if (t32 >= 4 * sms) {
      MAK_GEMM32_TILE(64, 64, 16, 2, 8, 32, false)
    } else {
      MAK_GEMM_TILE(32, 32, GEMM_BK, 2, 2)
    }
#undef MAK_GEMM32_TILE
  }
#undef MAK_GEMM_TILE
#undef MAK_GEMM_COLS
  return cudaGetLastError() == cudaSuccess ? 0 : MAK_ERR_CUDA;
}

// number of K-splits that fills the GPU for an output of M x N: two 32 x 32
// tiles per SM for the FP64 types (at least 32 of K per split), two 32 x 128
// or 64 x 64 tiles for the FP32 types (at least 64)
template <class T>
inline int pick_splits(int64_t M, int64_t N, int64_t K, int sms) {
  constexpr bool f64 = sizeof(real_t<T>) == 8;
  const int64_t tiles = f64 ? ceil_div(M, 32) * ceil_div(N, 32)
                            : ceil_div(M, M <= 32 ? 32 : 64) * ceil_div(N, M <= 32 ? 128 : 64);
  int64_t want = 2LL * sms;
  if (tiles >= want) return 1;
  int64_t s = ceil_div(want, tiles);
  int64_t maxs = ceil_div(K, f64 ? 32 : 64);
  if (s > maxs) s = maxs;
  if (s < 1) s = 1;
  if (s > 64) s = 64;
  return (int)s;
}

}  // namespace mak
