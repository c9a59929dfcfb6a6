// FP64 dense linear algebra of the sparse-GP solve (SparseGP::
// update_matrices_QR, sparse_gp.cpp:607-641): the Cholesky factor of
// Kuu + jitter, lower-triangular inverses (L_inv, and R_inv through R^T),
// and the symmetric products Kuu^-1 = L_inv^T L_inv and Sigma = R_inv
// R_inv^T.
//
// Matrices are row-major.  The O(M^3) work runs as FP64-level products on
// the tensor cores (ozaki.cu: 9 exact BF16 slices, exact integer sums, one
// rounding; about 35x this GPU's FP64 DGEMM rate); the O(M nb^2) work on
// diagonal blocks of nb = 128 in shared memory:
//   Cholesky, right-looking by block columns: factor the diagonal block
//     and invert it (k_potrf_cluster, k_potrf_inverse), L21 = A21 L11^-T as a product with
//     that inverse, then the trailing update A22 -= L21 L21^T;
//   lower-triangular inverse, recursive: X = [X11 0; X21 X22] with X11,
//     X22 the inverses of the diagonal halves (leaves of nb from the
//     factorisation, or all at once by k_trtri_block for a given L) and X21 = -X22 (L21 X11).
// Operation orders differ from Eigen's (the reference's LLT and triangular
// solves), so results agree with it to FP64 rounding, not bit for bit.
#include <cmath>
#include <cstdint>
#include <utility>
#include <vector>

#include "fgb_dense.h"
#include "fgb_internal.h"
#include "fgb_ozaki.h"

namespace fgb {
namespace dense {
namespace {

constexpr int kNB = 128;          // diagonal block
constexpr int kBlockThreads = 512;

// ------------------------------------------------- diagonal block, cluster
// Cholesky factor of a kb x kb diagonal block (kb <= kNB) and the factor's
// inverse, by a cluster of kCl = 16 CTAs.  An SM finishes an FP64 warp
// instruction every 16 cycles and a warp one of its own every 64, dependent
// or not, so one CTA needs at least 180 us for the 700,000 multiply-adds of a
// 128-block (and took 820 us, with three barriers a column and the inverse
// by one thread a column).  Sixteen CTAs, blocked by kIB = 32 columns:
//   every CTA factors the 32 x 32 diagonal block for itself (the chain of 32
//     pivots; identical results, so no exchange);
//   the rows below and the 32 rows of the identity, which become the block's
//     inverse, are dealt out cyclically, a warp solving for a row;
//   their trailing updates need all of L21: through global memory (L2 loads)
//     between cluster barriers.
// The rest of the inverse follows in k_potrf_inverse.
// 72 us a 128-block and 8 for k_potrf_inverse; of the 72, 45 are the four
// chains of 32 pivots (720 cycles each: five dependent FP64 instructions of
// 66, the exchange between warps 140, the division's estimate and the stores)
// and 9 the cluster's barriers.  With the 32 x 32 inverses beside the pivots in
// every CTA, square roots on the chain and the rest of the inverse in the
// cluster it took 118 us (1,190 cycles a pivot).
constexpr int kIB = 32, kCl = 16, kClT = 256, kClW = kClT / 32;
// warps that factor a block: as many as the FP64 unit serves in the 64 cycles
// of one instruction, so that the pivot's never wait behind the updates
constexpr int kFW = 4, kFT = 32 * kFW;
constexpr int kLd = kIB + 1;
// shared doubles: the panel, the block's columns V and U, 1/sqrt(pivot)
constexpr int kClSmem = (kNB - kIB) * kLd + 2 * kIB * kIB + kIB;

__device__ __forceinline__ void cluster_barrier() {
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release;\n"
               "barrier.cluster.wait.acquire;" ::: "memory");
}
template <int ID, int N>
__device__ __forceinline__ void bar_sync() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void bar_arrive() {
  __threadfence_block();
  asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
  __syncwarp();
}
// d positive and far from the ends of the exponent range, by its upper word
// (an FP64 comparison takes an FP64 instruction's time).
__device__ __forceinline__ bool ordinary(double d) {
  return (unsigned)(__double2hiint(d) >> 20) - 60u < 1920u;
}
// 1/d of an ordinary d from the hardware's estimate y (20 bits of mantissa)
// by one third-order step of Householder's iteration, y (1 + e + e^2) with e =
// 1 - d y: e^3 leaves 2^-60, so within one ulp of the rounded quotient.
__device__ __forceinline__ double rcp64(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// v / d where the estimate does not serve; a pivot that is not positive
// counts as 1 and is reported.  Out of line: nothing of it on the pivots'
// chain.
static __device__ __noinline__ double div_rare(double v, double d, int k,
                                               int *flag) {
  if (d > 0.0) return v / d;
  if ((threadIdx.x & 31) == 0 && *flag == 0) *flag = k + 1;
  return v;
}

// Column k from its updated values v (a lane per row): V and U = v / d for
// the updates v_ij -= V_i U_j that need no square root.
__device__ __forceinline__ void pivot_column(int k, double v, double *V,
                                             double *U, int *flag) {
  const int lane = threadIdx.x & 31;
  const double d = __shfl_sync(0xffffffffu, v, k);
  V[k * kIB + lane] = lane >= k ? v : 0.0;
  double u = v * rcp64(d);
  if (!ordinary(d)) u = div_rare(v, d, k, flag);
  U[k * kIB + lane] = lane > k ? u : 0.0;
}

// The step of column K in factor_block32 (a template, so that the barrier
// ids are constants).  Column K + 1's warp brings that column up to date
// first, writes it and only arrives at the barrier that its readers wait at:
// its other updates follow while they go on.  Chain of a step: one update,
// the pivot (4 dependent FP64 instructions), the exchange.
template <int K>
__device__ __forceinline__ void factor_step(double (&v)[kIB / kFW], double *V,
                                            double *U, int *flag) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w != K % kFW) bar_sync<1 + (K & 3), kFT>();
  const double li = V[K * kIB + lane];
  constexpr int n1 = K + 1, o1 = n1 % kFW, q1 = n1 / kFW;
  if (n1 < kIB && w == o1) {
    constexpr int q = q1 % (kIB / kFW);
    v[q] = fma(-li, U[K * kIB + n1 % kIB], v[q]);
    pivot_column(n1, v[q], V, U, flag);
    bar_arrive<1 + (n1 & 3), kFT>();
  }
#pragma unroll
  for (int q = 0; q < kIB / kFW; q++)
    if (kFW * q + w > K && !(w == o1 && q == q1))
      v[q] = fma(-li, U[K * kIB + kFW * q + w], v[q]);
  if constexpr (K + 1 < kIB) factor_step<K + 1>(v, V, U, flag);
}

// Factors the block whose lower part is in v (v[q]: row lane, column
// kFW q + w; rows and columns past jb the identity's) into its columns V and
// U and y = 1/sqrt(pivot): L_ik = V_ik y_k.  Returns 0 or 1 + the first bad
// pivot.
__device__ int factor_block32(int jb, double (&v)[kIB / kFW], double *V,
                              double *U, double *y, int *flag) {
  const int t = threadIdx.x, w = t >> 5;
  if (t == 0) *flag = 0;
  __syncthreads();
  if (w == 0) {
    pivot_column(0, v[0], V, U, flag);
    bar_arrive<1, kFT>();
  }
  if (w < kFW) factor_step<0>(v, V, U, flag);
  __syncthreads();
  if (*flag && *flag <= jb) return *flag;
  if (w == 0) {
    const double d = V[t * kIB + t];
    y[t] = d > 0.0 ? rsqrt(d) : 1.0;
  }
  __syncthreads();
  return 0;
}

__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kClT)
k_potrf_cluster(int kb, double *__restrict__ A, long long lda,
                double *__restrict__ X, long long ldx, int base,
                int *__restrict__ info) {
  extern __shared__ double sh[];
  double *P = sh;                                    // panel rows
  double *V = P + (kNB - kIB) * kLd;
  double *U = V + kIB * kIB;
  double *y = U + kIB * kIB;
  __shared__ int flag;
  const int t = threadIdx.x, rank = blockIdx.x % kCl, w = t >> 5, lane = t & 31;
  for (int j0 = 0; j0 < kb; j0 += kIB) {
    const int jb = min(kIB, kb - j0);
    double v[kIB / kFW];
#pragma unroll
    for (int q = 0; q < kIB / kFW; q++) {
      const int c = kFW * q + w;
      v[q] = lane == c ? 1.0 : 0.0;
      if (w < kFW && lane < jb && c <= lane)
        v[q] = __ldcg(A + (long long)(j0 + lane) * lda + j0 + c);
    }
    // a warp's row: every kCl-th row below the block, then of the identity
    const int r0 = j0 + kIB, m = kb - r0;
    const int nown = m > rank ? (m - rank + kCl - 1) / kCl : 0;
    static_assert((kNB - kIB) / kCl + kIB / kCl <= kClW, "a row for each warp");
    const int e = rank + kCl * (w - nown);   // row of the identity, w >= nown
    double r = 0.0;
    if (w >= nown)
      r = lane == e ? 1.0 : 0.0;
    else if (lane < jb)
      r = __ldcg(A + (long long)(r0 + rank + kCl * w) * lda + j0 + lane);
    const int bad = factor_block32(jb, v, V, U, y, &flag);
    if (bad) {   // the same in every CTA: all leave here
      if (rank == 0 && t == 0) atomicCAS(info, 0, base + j0 + bad);
      return;
    }
    if (w < nown + kIB / kCl) {   // a warp with a row
#pragma unroll 8
      for (int k = 0; k < kIB; k++)
        r = fma(-__shfl_sync(0xffffffffu, r, k), U[k * kIB + lane], r);
    }
    r *= y[lane];
    if (lane < jb) {
      if (w < nown)
        A[(long long)(r0 + rank + kCl * w) * lda + j0 + lane] = r;
      else if (e < jb)
        X[(long long)(j0 + lane) * ldx + j0 + e] = r;
    }
    // every CTA has read the diagonal block before this barrier: the factor
    // may replace it
    cluster_barrier();
    if (rank == 0 && lane < jb)
#pragma unroll
      for (int q = 0; q < kIB / kClW; q++) {
        const int c = kClW * q + w;
        if (c < jb)
          A[(long long)(j0 + lane) * lda + j0 + c] =
              lane >= c ? V[c * kIB + lane] * y[c] : 0.0;
      }
    if (m <= 0) break;
    for (int e = t; e < m * kIB; e += kClT)
      P[(e / kIB) * kLd + e % kIB] =
          __ldcg(A + (long long)(r0 + e / kIB) * lda + j0 + e % kIB);
    __syncthreads();
    // own rows' updates, a warp for 32 columns of a row
    int item = 0;
    for (int q = 0; q < nown; q++) {
      const int i = rank + kCl * q;
      for (int c0 = 0; c0 <= i; c0 += 32) {
        if (item++ % kClW != w) continue;
        const int c = c0 + lane;
        if (c > i) continue;
        double s = 0.0;
#pragma unroll 8
        for (int k = 0; k < kIB; k++) s = fma(P[i * kLd + k], P[c * kLd + k], s);
        double *a = A + (long long)(r0 + i) * lda + r0 + c;
        *a = __ldcg(a) - s;
      }
    }
    cluster_barrier();
  }
}

// fgb_fp64_check: 1/x as a pivot's column is scaled (k = 0), or x / k.
__global__ void k_fp64_check(int k, long long n, const double *__restrict__ x,
                             double *__restrict__ y) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double d = x[i];
  int flag = 0;
  if (k > 0) y[i] = div_int(d, k);
  else y[i] = ordinary(d) ? rcp64(d) : div_rare(1.0, d, 0, &flag);
}

// The rest of the inverse X of a diagonal block's factor, a CTA for each
// column c: by 32-row blocks i below the column's own, X_i = -Xd_i (sum over
// k L_ik X_k) with the inverses Xd of the 32 x 32 diagonal blocks that
// k_potrf_cluster has left in X; zeros above.  A warp has one FP64 instruction
// in flight, so four warps take every fourth term of each sum.  By the
// sixteen CTAs of the cluster, eight columns each, this was 41,000 of its
// cycles.
constexpr int kInvT = 128, kInvB = kNB / kIB;
constexpr int kInvSmem =
    (kInvB * (kInvB - 1) / 2 + kInvB - 1) * kIB * kLd;   // doubles
__global__ void __launch_bounds__(kInvT)
k_potrf_inverse(int kb, const double *__restrict__ A, long long lda,
                double *X, long long ldx) {
  extern __shared__ double sh[];
  constexpr int kBlk = kIB * kLd;
  double *L = sh;                                  // blocks (i, k), k < i
  double *D = L + kInvB * (kInvB - 1) / 2 * kBlk;  // Xd_i, i > 0
  __shared__ double x[kNB], part[4][kIB], sum[kIB];
  const int c = blockIdx.x, t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int cb = c / kIB, nb = (kb + kIB - 1) / kIB;
  for (int i = cb + 1; i < nb; i++)
    for (int k = cb; k <= i; k++) {
      double *dst = k < i ? L + (i * (i - 1) / 2 + k) * kBlk : D + (i - 1) * kBlk;
#pragma unroll
      for (int e = t; e < kIB * kIB; e += kInvT) {
        const int r = e / kIB, q = e % kIB, row = i * kIB + r;
        const bool in = row < kb && (k < i || q <= r);
        const double *src = k < i ? A + (long long)row * lda + k * kIB + q
                                  : X + (long long)row * ldx + k * kIB + q;
        // all in flight at once; nothing read (zeros) outside the factor
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;"
                     ::"r"((unsigned)__cvta_generic_to_shared(dst + r * kLd + q)),
                       "l"(in ? src : A), "r"(in ? 8 : 0) : "memory");
      }
    }
  if (t < kIB) {
    const int row = cb * kIB + t;
    x[row] = row < kb ? X[(long long)row * ldx + c] : 0.0;
  }
  for (int row = t; row < cb * kIB; row += kInvT) X[(long long)row * ldx + c] = 0.0;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int i = cb + 1; i < nb; i++) {
    double s = 0.0;
    for (int k = cb; k < i; k++) {
      const double *l = L + (i * (i - 1) / 2 + k) * kBlk + lane * kLd;
#pragma unroll
      for (int q = 0; q < kIB; q += 4) s = fma(l[q + w], x[k * kIB + q + w], s);
    }
    part[w][lane] = s;
    __syncthreads();
    if (w == 0)
      sum[lane] = (part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane]);
    __syncthreads();
    const double *d = D + (i - 1) * kBlk + lane * kLd;
    s = 0.0;
#pragma unroll
    for (int q = 0; q < kIB; q += 4) s = fma(-d[q + w], sum[q + w], s);
    part[w][lane] = s;
    __syncthreads();
    if (w == 0) {
      const double v =
          (part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane]);
      const int row = i * kIB + lane;
      x[row] = v;
      if (row < kb) X[(long long)row * ldx + c] = v;
    }
    __syncthreads();
  }
}

// Inverses of the diagonal blocks of a lower-triangular M x M matrix L,
// one CTA per block of kNB (the last may be smaller), written into the same
// positions of X (the rest of X is left alone).
__global__ void __launch_bounds__(kBlockThreads)
k_trtri_block(int M, const double *__restrict__ L, long long ldl,
              double *__restrict__ X, long long ldx) {
  extern __shared__ double sh[];
  const int b0 = blockIdx.x * kNB;
  const int kb = min(kNB, M - b0);
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int idx = tid; idx < kb * kb; idx += nt) {
    const int i = idx / kb, j = idx - i * kb;
    sh[idx] = j <= i ? L[(long long)(b0 + i) * ldl + b0 + j] : 0.0;
  }
  __syncthreads();
  double *Xb = X + (long long)b0 * ldx + b0;
  for (int j = tid; j < kb; j += nt) {
    for (int i = 0; i < j; i++) Xb[(long long)i * ldx + j] = 0.0;
    Xb[(long long)j * ldx + j] = 1.0 / sh[j * kb + j];
    for (int i = j + 1; i < kb; i++) {
      double s = 0.0;
      for (int k = j; k < i; k++) s += sh[i * kb + k] * Xb[(long long)k * ldx + j];
      Xb[(long long)i * ldx + j] = -s / sh[i * kb + i];
    }
  }
}

// The diagonal blocks of the M x M matrix X from D (nblk x kNB x kNB).
__global__ void k_put_blocks(int M, const double *__restrict__ D,
                             double *__restrict__ X, long long ldx) {
  const int b0 = blockIdx.x * kNB, kb = min(kNB, M - b0);
  const double *d = D + (size_t)blockIdx.x * kNB * kNB;
  for (int i = threadIdx.x / kNB; i < kb; i += blockDim.x / kNB) {
    const int j = threadIdx.x % kNB;
    if (j < kb) X[(long long)(b0 + i) * ldx + b0 + j] = d[i * kNB + j];
  }
}

// out (cols x rows, ld ldo) = in^T (in: rows x cols, ld ldi), 32 x 32 tiles.
__global__ void k_transpose_tile(int rows, int cols, const double *__restrict__ in,
                                 long long ldi, double *__restrict__ out,
                                 long long ldo) {
  __shared__ double t[32][33];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = r0 + k, c = c0 + threadIdx.x;
    if (r < rows && c < cols) t[k][threadIdx.x] = in[(long long)r * ldi + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int c = c0 + k, r = r0 + threadIdx.x;
    if (r < rows && c < cols) out[(long long)c * ldo + r] = t[threadIdx.x][k];
  }
}

__global__ void k_zero_strict_upper(int M, double *__restrict__ A, long long lda) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)M * M) return;
  const int i = (int)(idx / M), j = (int)(idx - (long long)i * M);
  if (j > i) A[(long long)i * lda + j] = 0.0;
}

// At (M x (nl + M), row-major) = [Kuf diag(sqrt(noise)) | L]: the
// transpose of the reference's A = [sqrt(noise) Kuf^T ; L^T]
// (sparse_gp.cpp:621-630), built without a transpose (Kuf is M x nl
// row-major, L lower row-major); b = [sqrt(noise) y ; 0].
__global__ void k_build_At(int M, int nl, const double *__restrict__ Kuf,
                           const double *__restrict__ noise,
                           const double *__restrict__ y,
                           const double *__restrict__ L, double *__restrict__ At,
                           double *__restrict__ b) {
  const long long n = (long long)nl + M;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)M * n) return;
  const int c = (int)(idx / n);
  const long long r = idx - (long long)c * n;
  At[idx] = r < nl ? sqrt(noise[r]) * Kuf[(long long)c * nl + r]
                   : L[(long long)c * M + (r - nl)];
  if (c == 0) b[r] = r < nl ? sqrt(noise[r]) * y[r] : 0.0;
}

// Per-block partial sums of squares (fixed order), then each block adds them.
__global__ void k_sumsq_part(long long n, const double *__restrict__ x,
                             double *__restrict__ part) {
  __shared__ double red[256];
  double s = 0.0;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n;
       i += (long long)gridDim.x * 256)
    s += x[i] * x[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// A += s I (M x M, row-major) with s = kShift * part sum (the shifted
// Cholesky QR's shift from the squared Frobenius norm).
__global__ void k_add_shift(int M, double *__restrict__ A, long long lda,
                            const double *__restrict__ part, int nparts,
                            double factor) {
  __shared__ double red[256];
  double v = 0.0;
  for (int k = threadIdx.x; k < nparts; k += 256) v += part[k];
  red[threadIdx.x] = v;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  const double tot = red[0] * factor;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += gridDim.x * blockDim.x)
    A[(long long)i * lda + i] += tot;
}

// part[ch][j] = sum of Q[r][j] b[r] over the chunk's rows (Q n x M,
// row-major): 32 columns per block (lane = column), 8 row groups, fixed-order
// sums; k_gemv_t_final adds the chunks.
constexpr int kGemvChunks = 32;
__global__ void k_gemv_t(long long n, int M, const double *__restrict__ Q,
                         const double *__restrict__ b,
                         double *__restrict__ part) {
  __shared__ double red[8][33];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  const long long per = (n + kGemvChunks - 1) / kGemvChunks;
  const long long r1 = min(n, (blockIdx.y + 1) * per);
  double s = 0.0;
  if (j < M)
    for (long long r = blockIdx.y * per + g; r < r1; r += 8)
      s += Q[r * M + j] * b[r];
  red[g][lane] = s;
  __syncthreads();
  if (g == 0 && j < M) {
    double t = 0.0;
    for (int k = 0; k < 8; k++) t += red[k][lane];
    part[(long long)blockIdx.y * M + j] = t;
  }
}
__global__ void k_gemv_t_final(int M, const double *__restrict__ part,
                               double *__restrict__ y) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  double t = 0.0;
  for (int k = 0; k < kGemvChunks; k++) t += part[(long long)k * M + j];
  y[j] = t;
}

int transpose(int rows, int cols, const double *in, long long ldi, double *out,
              long long ldo, cudaStream_t st) {
  if (rows == 0 || cols == 0) return FGB_OK;
  dim3 g(ceil_div(cols, 32), ceil_div(rows, 32)), b(32, 8);
  k_transpose_tile<<<g, b, 0, st>>>(rows, cols, in, ldi, out, ldo);
  FGB_LAUNCH_CHECK("k_transpose_tile");
  return FGB_OK;
}

// Scratch of one factorisation: slices of the two operands and the
// tensor-core GEMM's time-out flag.
// A factorisation's diagonal-block inverses (nblk x kNB x kNB) are kept
// for the triangular inverse that follows; info[f] is factorisation f's
// first bad pivot (1-based; 0: none).
constexpr int kMaxFactors = 4;
struct Work {
  oz::Sliced A, B;
  DevBuf flags, t1, t2, dinv;   // flags: time-out, then info[kMaxFactors]
  explicit Work(cudaStream_t st)
      : A(st), B(st), flags(st), t1(st), t2(st), dinv(st) {}
  int *err() const { return flags.as<int>(); }
  int *info(int f) const { return flags.as<int>() + 1 + f; }
  int start(cudaStream_t st) {
    const int rc = flags.ensure(sizeof(int) * (1 + kMaxFactors));
    if (rc) return rc;
    FGB_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(int) * (1 + kMaxFactors), st));
    return FGB_OK;
  }
};

// C (m x n, ldc) = a A B^T + b C with A (m x k, lda) and B (n x k, ldb) at
// FP64 level on the tensor cores.
int gemm_nt(int m, int n, int k, const double *A, long long lda,
            const double *B, long long ldb, double *C, long long ldc,
            double a, double b, Work &w, cudaStream_t st, bool lower = false) {
  if (m == 0 || n == 0) return FGB_OK;
  int rc;
  if ((rc = oz::slice_pair(
           {m, k, oz::kTM, A, lda, nullptr, nullptr}, w.A,
           {n, k, oz::kTN64v[oz::tile64(m, n)], B, ldb, nullptr, nullptr}, w.B,
           st)))
    return rc;
  return oz::gemm_axpby(w.A, w.B, C, ldc, a, b, w.err(), st, lower);
}

// Waits for the stream and reports a product whose bounded wait ran out, then
// the first factorisation that met a bad pivot (one copy of all flags).
int finish(Work &w, cudaStream_t st, const char *what) {
  int h[1 + kMaxFactors] = {};
  FGB_CUDA(cudaMemcpyAsync(h, w.flags.p, sizeof(h), cudaMemcpyDeviceToHost, st));
  FGB_CUDA(cudaStreamSynchronize(st));
  if (h[0]) {
    set_error("%s: a bounded device wait ran out", what);
    return FGB_ETIMEOUT;
  }
  for (int f = 1; f <= kMaxFactors; f++)
    if (h[f]) {
      set_error("Cholesky of Kuu + jitter failed (leading minor %d not "
                "positive definite)", h[f]);
      return FGB_EINVAL;
    }
  return FGB_OK;
}

int smem_for(int kb) {
  return (int)(sizeof(double) * (size_t)kb * kb);
}

// X (lower part, row-major, ld ldx) = L^-1 for rows/cols [lo, lo + n),
// given the diagonal blocks already inverted in place.
int trtri_rec(int lo, int n, const double *L, long long ldl, double *X,
              long long ldx, Work &w, cudaStream_t st) {
  if (n <= kNB) return FGB_OK;
  const int nblk = ceil_div(n, kNB);
  const int h = kNB * ((nblk + 1) / 2);
  const int n2 = n - h;
  int rc;
  if ((rc = trtri_rec(lo, h, L, ldl, X, ldx, w, st)) ||
      (rc = trtri_rec(lo + h, n2, L, ldl, X, ldx, w, st)))
    return rc;
  // T = L21 X11 (n2 x h): B operand X11^T
  if ((rc = w.t1.ensure(sizeof(double) * (size_t)h * h)) ||
      (rc = w.t2.ensure(sizeof(double) * (size_t)n2 * h)))
    return rc;
  const double *L21 = L + (long long)(lo + h) * ldl + lo;
  const double *X11 = X + (long long)lo * ldx + lo;
  const double *X22 = X + (long long)(lo + h) * ldx + lo + h;
  double *X21 = X + (long long)(lo + h) * ldx + lo;
  if ((rc = transpose(h, h, X11, ldx, w.t1.as<double>(), h, st))) return rc;
  // T into X21's place (n2 x h), then its transpose into t2 (h x n2)
  if ((rc = gemm_nt(n2, h, h, L21, ldl, w.t1.as<double>(), h, X21, ldx, 1.0,
                    0.0, w, st)))
    return rc;
  if ((rc = transpose(n2, h, X21, ldx, w.t2.as<double>(), n2, st))) return rc;
  // X21 = -X22 T
  return gemm_nt(n2, h, n2, X22, ldx, w.t2.as<double>(), n2, X21, ldx, -1.0,
                 0.0, w, st);
}

// Lower Cholesky factor of the symmetric M x M matrix A (row-major; the
// lower triangle is read), in place (strict upper part zeroed); the diagonal
// blocks' inverses into w.dinv, a bad pivot into info[f].
int factor(int M, double *A, long long lda, int f, Work &w, cudaStream_t st) {
  int rc;
  const int nblk = ceil_div(M, kNB);
  if ((rc = w.dinv.ensure(sizeof(double) * (size_t)nblk * kNB * kNB)))
    return rc;
  constexpr int kSmem = (int)sizeof(double) * kClSmem;
  FGB_CUDA(cudaFuncSetAttribute(k_potrf_cluster,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSmem));
  FGB_CUDA(cudaFuncSetAttribute(k_potrf_cluster,
                                cudaFuncAttributeNonPortableClusterSizeAllowed,
                                1));
  constexpr int kInvBytes = (int)sizeof(double) * kInvSmem;
  FGB_CUDA(cudaFuncSetAttribute(k_potrf_inverse,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kInvBytes));
  for (int k0 = 0; k0 < M; k0 += kNB) {
    const int kb = std::min(kNB, M - k0);
    double *A11 = A + (long long)k0 * lda + k0;
    double *X = w.dinv.as<double>() + (size_t)(k0 / kNB) * kNB * kNB;
    k_potrf_cluster<<<kCl, kClT, kSmem, st>>>(kb, A11, lda, X, kNB, k0,
                                              w.info(f));
    FGB_LAUNCH_CHECK("k_potrf_cluster");
    k_potrf_inverse<<<kb, kInvT, kInvBytes, st>>>(kb, A11, lda, X, kNB);
    FGB_LAUNCH_CHECK("k_potrf_inverse");
    const int r = M - k0 - kb;
    if (r == 0) break;
    double *A21 = A + (long long)(k0 + kb) * lda + k0;
    double *A22 = A + (long long)(k0 + kb) * lda + k0 + kb;
    // L21 = A21 L11^-T, in place (the product reads slices of A21), then
    // A22 -= L21 L21^T (lower tiles)
    if ((rc = gemm_nt(r, kb, kb, A21, lda, X, kNB, A21, lda, 1.0, 0.0, w,
                      st)) ||
        (rc = gemm_nt(r, r, kb, A21, lda, A21, lda, A22, lda, -1.0, 1.0, w,
                      st, true)))
      return rc;
  }
  k_zero_strict_upper<<<ceil_div((long long)M * M, 256), 256, 0, st>>>(M, A,
                                                                       lda);
  FGB_LAUNCH_CHECK("k_zero_strict_upper");
  return FGB_OK;
}

// X = L^-1 of the factor just made (diagonal inverses from w.dinv) or, with
// `own`, of any lower-triangular L; X's strict upper part zeroed.
int invert(int M, const double *L, long long ldl, double *X, long long ldx,
           bool own, Work &w, cudaStream_t st) {
  k_zero_strict_upper<<<ceil_div((long long)M * M, 256), 256, 0, st>>>(M, X,
                                                                       ldx);
  FGB_LAUNCH_CHECK("k_zero_strict_upper");
  if (own) {
    FGB_CUDA(cudaFuncSetAttribute(k_trtri_block,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  smem_for(kNB)));
    k_trtri_block<<<ceil_div(M, kNB), kBlockThreads,
                    smem_for(std::min(M, kNB)), st>>>(M, L, ldl, X, ldx);
    FGB_LAUNCH_CHECK("k_trtri_block");
  } else {
    k_put_blocks<<<ceil_div(M, kNB), 256, 0, st>>>(M, w.dinv.as<double>(), X,
                                                   ldx);
    FGB_LAUNCH_CHECK("k_put_blocks");
  }
  return trtri_rec(0, M, L, ldl, X, ldx, w, st);
}

}  // namespace

// L = chol(A) in place and X = L^-1 (SparseGP's Kuu + jitter).
int cholesky_inverse(int M, double *A, double *X, cudaStream_t st) {
  if (M == 0) return FGB_OK;
  Work w(st);
  int rc;
  if ((rc = w.start(st)) || (rc = factor(M, A, M, 0, w, st)) ||
      (rc = invert(M, A, M, X, M, false, w, st)))
    return rc;
  return finish(w, st, "Cholesky");
}

int cholesky(int M, double *A, long long lda, cudaStream_t st) {
  if (M == 0) return FGB_OK;
  Work w(st);
  int rc;
  if ((rc = w.start(st)) || (rc = factor(M, A, lda, 0, w, st))) return rc;
  return finish(w, st, "Cholesky");
}

// X = L^-1 for a lower-triangular M x M matrix L (row-major; X's strict
// upper part zeroed).
int trtri_lower(int M, const double *L, long long ldl, double *X,
                long long ldx, cudaStream_t st) {
  if (M == 0) return FGB_OK;
  Work w(st);
  int rc;
  if ((rc = w.start(st)) || (rc = invert(M, L, ldl, X, ldx, true, w, st)))
    return rc;
  return finish(w, st, "triangular inverse");
}

// C = A^T A (transpose_first) or A A^T for a square M x M matrix A, FP64
// level on the tensor cores; C is symmetric (both triangles written).
int sym_product(int M, const double *A, bool transpose_first, double *C,
                cudaStream_t st) {
  if (M == 0) return FGB_OK;
  Work w(st);
  DevBuf At(st);
  int rc;
  if ((rc = w.start(st))) return rc;
  const double *op = A;
  if (transpose_first) {
    if ((rc = At.ensure(sizeof(double) * (size_t)M * M))) return rc;
    if ((rc = transpose(M, M, A, M, At.as<double>(), M, st))) return rc;
    op = At.as<double>();
  }
  if ((rc = gemm_nt(M, M, M, op, M, op, M, C, M, 1.0, 0.0, w, st))) return rc;
  return finish(w, st, "symmetric product");
}

// The factor R (returned as R_inv = R^-1, row-major upper) and Q^T b of the
// Householder QR in update_matrices_QR (sparse_gp.cpp:621-640), by shifted
// Cholesky QR with two refinement passes: pass 0 factors A^T A + s I (s =
// 11 (n M + M (M + 1)) u |A|_F^2), Q0 = A R0^-1; passes 1 and 2 factor
// Q^T Q without shift, Q <- Q R_k^-1; R = R2 R1 R0 and Q^T b = Q2^T b.
// That is backward stable like Householder QR for condition numbers below
// 1/u; A here = [sqrt(noise) Kuf^T; L^T] has sigma_min >= sqrt(jitter).
// Every O(n M^2) product is an FP64-level tensor-core product.  R agrees
// with a Householder R up to the signs of its rows, so alpha = R^-1 Q^T b
// and Sigma = R^-1 R^-T are the same quantities.  At (M x n, row-major) is
// read; b has n entries.
int cholqr_solve(int M, long long n, double *At, const double *b,
                 double *R_inv, double *Qtb, cudaStream_t st) {
  Work w(st);
  DevBuf G(st), X[3] = {DevBuf(st), DevBuf(st), DevBuf(st)}, A0(st), Q(st),
         Qt(st), part(st), P(st);
  int rc;
  const size_t MM = (size_t)M * M, nM = (size_t)n * M;
  if ((rc = w.start(st)) || (rc = G.ensure(sizeof(double) * MM)) ||
      (rc = X[0].ensure(sizeof(double) * MM)) ||
      (rc = X[1].ensure(sizeof(double) * MM)) ||
      (rc = X[2].ensure(sizeof(double) * MM)) ||
      (rc = P.ensure(sizeof(double) * MM)) ||
      (rc = A0.ensure(sizeof(double) * nM)) ||
      (rc = Q.ensure(sizeof(double) * nM)) ||
      (rc = part.ensure(sizeof(double) * std::max(1024, kGemvChunks * M))))
    return rc;
  if (n > (long long)INT32_MAX) {
    set_error("update_matrices_QR: %lld rows exceed the product kernels' "
              "limit", n);
    return FGB_EINVAL;
  }
  const int ni = (int)n;
  const double u = std::ldexp(1.0, -53);
  const double shift = 11.0 * ((double)n * M + (double)M * (M + 1)) * u;
  // the rows of A (n x M) for the products Q = A R^-1
  if ((rc = transpose(M, ni, At, n, A0.as<double>(), M, st))) return rc;
  const double *Qprev = A0.as<double>();
  const double *Tprev = At;   // Q_prev^T (M x n)
  for (int pass = 0; pass < 3; pass++) {
    if ((rc = gemm_nt(M, M, ni, Tprev, n, Tprev, n, G.as<double>(), M, 1.0,
                      0.0, w, st, true)))
      return rc;
    if (pass == 0) {
      const int nparts = 1024;
      k_sumsq_part<<<nparts, 256, 0, st>>>((long long)M * n, At,
                                          part.as<double>());
      FGB_LAUNCH_CHECK("k_sumsq_part");
      k_add_shift<<<ceil_div(M, 256), 256, 0, st>>>(
          M, G.as<double>(), M, part.as<double>(), nparts, shift);
      FGB_LAUNCH_CHECK("k_add_shift");
    }
    if ((rc = factor(M, G.as<double>(), M, pass, w, st)) ||
        (rc = invert(M, G.as<double>(), M, X[pass].as<double>(), M, false, w,
                     st)))
      return rc;
    // Q_pass = Q_prev R_pass^-1 = Q_prev X_pass^T (X = L^-1, R = L^T)
    if ((rc = gemm_nt(ni, M, M, Qprev, M, X[pass].as<double>(), M,
                      Q.as<double>(), M, 1.0, 0.0, w, st)))
      return rc;
    if (pass < 2) {
      // Q becomes the next pass's input (A0's storage is free after pass 0)
      Q.swap(A0);
      Qprev = A0.as<double>();
      if ((rc = Qt.ensure(sizeof(double) * nM))) return rc;
      if ((rc = transpose(ni, M, Qprev, M, Qt.as<double>(), n, st))) return rc;
      Tprev = Qt.as<double>();
    }
  }
  // Q^T b with the final Q
  k_gemv_t<<<dim3(ceil_div(M, 32), kGemvChunks), 256, 0, st>>>(
      n, M, Q.as<double>(), b, part.as<double>());
  FGB_LAUNCH_CHECK("k_gemv_t");
  k_gemv_t_final<<<ceil_div(M, 256), 256, 0, st>>>(M, part.as<double>(), Qtb);
  FGB_LAUNCH_CHECK("k_gemv_t_final");
  // R^-1 = R0^-1 R1^-1 R2^-1 = (X2 X1 X0)^T
  double *T1 = G.as<double>();
  if ((rc = transpose(M, M, X[1].as<double>(), M, T1, M, st)) ||
      (rc = gemm_nt(M, M, M, X[2].as<double>(), M, T1, M, P.as<double>(), M,
                    1.0, 0.0, w, st)) ||
      (rc = transpose(M, M, X[0].as<double>(), M, T1, M, st)) ||
      (rc = gemm_nt(M, M, M, P.as<double>(), M, T1, M, X[1].as<double>(), M,
                    1.0, 0.0, w, st)) ||
      (rc = transpose(M, M, X[1].as<double>(), M, R_inv, M, st)))
    return rc;
  return finish(w, st, "Cholesky QR");
}

int build_At(int M, int nl, const double *Kuf, const double *noise,
             const double *y, const double *L, double *At, double *b,
             cudaStream_t st) {
  const long long n = (long long)nl + M;
  k_build_At<<<ceil_div((long long)M * n, 256), 256, 0, st>>>(M, nl, Kuf, noise,
                                                             y, L, At, b);
  FGB_LAUNCH_CHECK("k_build_At");
  return FGB_OK;
}

}  // namespace dense
}  // namespace fgb

using namespace fgb;

extern "C" int fgb_fp64_check(int k, long long n, const double *d_x,
                              double *d_y, void *stream) {
  if (k < 0 || k >= kNumInv || n < 0 || n > (1LL << 30) ||
      (n > 0 && (!d_x || !d_y))) {
    set_error("fgb_fp64_check: invalid arguments (k in [0, %d])", kNumInv - 1);
    return FGB_EINVAL;
  }
  if (n == 0) return FGB_OK;
  dense::k_fp64_check<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(
      k, n, d_x, d_y);
  FGB_LAUNCH_CHECK("k_fp64_check");
  return FGB_OK;
}

extern "C" int fgb_cholesky(int M, double *d_A, void *stream) {
  if (M < 0 || (M > 0 && !d_A)) {
    set_error("fgb_cholesky: invalid arguments");
    return FGB_EINVAL;
  }
  return dense::cholesky(M, d_A, M, (cudaStream_t)stream);
}

extern "C" int fgb_trtri_lower(int M, const double *d_L, double *d_X,
                               void *stream) {
  if (M < 0 || (M > 0 && (!d_L || !d_X)) || d_L == d_X) {
    set_error("fgb_trtri_lower: invalid arguments (distinct L and X)");
    return FGB_EINVAL;
  }
  return dense::trtri_lower(M, d_L, M, d_X, M, (cudaStream_t)stream);
}

extern "C" int fgb_solve_products(int M, const double *d_L_inv,
                                  const double *d_R_inv, double *d_Kuu_inverse,
                                  double *d_Sigma, void *stream) {
  if (M < 0 || (d_Kuu_inverse && !d_L_inv) || (d_Sigma && !d_R_inv)) {
    set_error("fgb_solve_products: invalid arguments");
    return FGB_EINVAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if (d_Kuu_inverse &&
      (rc = dense::sym_product(M, d_L_inv, true, d_Kuu_inverse, st)))
    return rc;
  if (d_Sigma && (rc = dense::sym_product(M, d_R_inv, false, d_Sigma, st)))
    return rc;
  return FGB_OK;
}
