// Plain FP64 form: the reference's algorithm on the GPU (stored
// forward-mode descriptor gradients, envs_struc GEMM + scatter), envs_envs,
// and the FP64 QR solve.
#include <cusolverDn.h>

#include <type_traits>

#include "fgb_dense.h"
#include "fgb_internal.h"
#include "fgb_kernels.h"
#include "fgb_model.h"
#include "fgb_gemm64.cuh"

namespace fgb {
namespace {
using namespace gemm64;

// envs_envs block: K = sig2 (D1 D2^T / (n1 n2))^power
__global__ void __launch_bounds__(GT)
k_envs_envs(int M, int N, int K, const double *__restrict__ D1,
            const double *__restrict__ n1, const double *__restrict__ D2,
            const double *__restrict__ n2, double sig2, double power,
            double *__restrict__ out) {
  const int m0 = blockIdx.y * BM, nn0 = blockIdx.x * BN;
  double acc[4][4];
  gemm_mainloop<true>(acc, m0, nn0, M, N, K, D1, K, nullptr, D2, K);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    int m = m0 + ty + 16 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int n = nn0 + tx + 16 * j;
      if (n >= N) continue;
      double a = n1[m], b = n2[n];
      double v = 0.0;
      if (a >= kEmptyThresh && b >= kEmptyThresh)
        v = sig2 * powx(acc[i][j] / (a * b), power);
      out[(long long)m * N + n] = v;
    }
  }
}


// Stored forward-mode gradients (b2.cpp:181-242 with single-bond gradients
// from :367-395).  For pair p (i -> j, species s_j) the single-bond gradient
// is nonzero only in block s_j:
// dA_p[c][n][lm] = dg_n (x_c/r) Y_lm + g_n dY_lm/dx_c, and
// dB2_p[c][(n1,n2,l)] = sum_m A[n1][lm] dA_p[c][n2][lm] + dA_p[c][n1][lm] A[n2][lm].
// Two kernels over the flat pair list, both bound by FP64 instructions (64
// cycles each per warp on an SM quarter), so the pairs are spread over all
// SMs.  One block per atom that walked its pairs in series, one thread
// evaluating each pair's basis, took 913 us for 108 FCC atoms (3,456 pairs,
// n_d 144) where these take 84 us (k_pair_basis 14, k_b2_dervs 70).
constexpr int kBT = 32;   // pairs (threads) per block of k_pair_basis

// Basis values of every pair, value-major so that neighbouring pairs are
// neighbouring addresses: rows g[nm] | dg[nm] | Y[nh] | dY/dx[nh] | dY/dy[nh]
// | dY/dz[nh], each P long; zero for pairs beyond the species pair's cutoff.
// LC > 0 fixes l_max (the recurrence stays in registers).
template <int LC>
__global__ void __launch_bounds__(kBT)
k_pair_basis(B2Params p, long long P, const int *__restrict__ center,
             const int *__restrict__ nbr_j, const double4_16a *__restrict__ rel,
             const int *__restrict__ species, double *__restrict__ basis) {
  const long long pp = (long long)blockIdx.x * kBT + threadIdx.x;
  if (pp >= P) return;
  const double4_16a r = rel[pp];
  const double rc =
      p.cutoffs[species[center[pp]] * kMaxSpecies + species[nbr_j[pp]]];
  const int nm = p.n_max, nh = p.n_harm;
  double *o = basis + pp;
  if (!(r.x <= rc)) {
    for (int v = 0; v < 2 * nm + 4 * nh; v++) o[v * P] = 0.0;
    return;
  }
  double g[kMaxNmax], dg[kMaxNmax];
  radial_eval<double>(p, r.x, rc, g, dg);
  for (int n = 0; n < nm; n++) {
    o[n * P] = g[n];
    o[(nm + n) * P] = dg[n];
  }
  double *y = o + 2 * nm * P;
  ylm_visit<double, LC, true>(
      p.l_max, r.y, r.z, r.w,
      [&](int idx, double v, double gx, double gy, double gz) {
        y[idx * P] = v;
        y[(nh + idx) * P] = gx;
        y[(2 * nh + idx) * P] = gy;
        y[(3 * nh + idx) * P] = gz;
      });
}

// dB2 rows of PP consecutive pairs: dA in shared memory, then a thread per
// descriptor q for all PP x 3 rows, and the rows' dots with B2 by a
// fixed-order block sum.
constexpr int kDT = 128;
template <int PP>
__global__ void __launch_bounds__(kDT)
k_b2_dervs(B2Params p, long long P, const int *__restrict__ center,
           const int *__restrict__ nbr_j, const double4_16a *__restrict__ rel,
           const int *__restrict__ species, const double *__restrict__ basis,
           const double *__restrict__ A_in, const double *__restrict__ B2_in,
           double *__restrict__ dB2, double *__restrict__ fdots) {
  extern __shared__ double dA[];            // PP x 3 x nm x nh
  __shared__ double red[3 * PP][kDT + 1];
  const int nA = p.n_A, nh = p.n_harm, nm = p.n_max, nr = p.n_rad,
            L1 = p.l_max + 1, nd = p.n_d, nmh = nm * nh;
  const long long p0 = (long long)blockIdx.x * PP;
  const int t = threadIdx.x;
  int cen[PP], sj[PP];
#pragma unroll
  for (int k = 0; k < PP; k++) {
    cen[k] = p0 + k < P ? center[p0 + k] : center[p0];
    sj[k] = p0 + k < P ? species[nbr_j[p0 + k]] : -1;
  }
  for (int e = t; e < nmh; e += kDT) {
    const int n = e / nh, lm = e - n * nh;
    const double *bn = basis + n * P + p0;
    const double *by = basis + (2 * nm + lm) * P + p0;
#pragma unroll
    for (int k = 0; k < PP; k++) {
      if (p0 + k >= P) break;
      const double4_16a r = rel[p0 + k];
      const double ir = 1.0 / r.x;
      const double g = bn[k], dgy = bn[nm * P + k] * ir * by[k];
      double *d = dA + k * 3 * nmh + e;
      d[0] = fma(dgy, r.y, g * by[nh * P + k]);
      d[nmh] = fma(dgy, r.z, g * by[2 * nh * P + k]);
      d[2 * nmh] = fma(dgy, r.w, g * by[3 * nh * P + k]);
    }
  }
  __syncthreads();
  double fd[3 * PP];
#pragma unroll
  for (int k = 0; k < 3 * PP; k++) fd[k] = 0.0;
  for (int q = t; q < nd; q += kDT) {
    const int l = q % L1;
    int pidx = q / L1, n1 = 0;
    while (pidx >= nr - n1) { pidx -= nr - n1; n1++; }
    const int n2 = n1 + pidx, b1 = n1 / nm, b2 = n2 / nm;
    const int o1 = n1 * nh + l * l, o2 = n2 * nh + l * l;
    const int e1 = o1 - b1 * nmh, e2 = o2 - b2 * nmh;
#pragma unroll
    for (int k = 0; k < PP; k++) {
      if (p0 + k >= P) break;
      double v0 = 0.0, v1 = 0.0, v2 = 0.0;
      const double *A = A_in + (long long)cen[k] * nA;
      const double *d = dA + k * 3 * nmh;
      if (b2 == sj[k])
        for (int m = 0; m < 2 * l + 1; m++) {
          const double a = A[o1 + m];
          v0 = fma(a, d[e2 + m], v0);
          v1 = fma(a, d[nmh + e2 + m], v1);
          v2 = fma(a, d[2 * nmh + e2 + m], v2);
        }
      if (b1 == sj[k])
        for (int m = 0; m < 2 * l + 1; m++) {
          const double a = A[o2 + m];
          v0 = fma(a, d[e1 + m], v0);
          v1 = fma(a, d[nmh + e1 + m], v1);
          v2 = fma(a, d[2 * nmh + e1 + m], v2);
        }
      const double b = B2_in[(long long)cen[k] * nd + q];
      double *out = dB2 + 3 * (p0 + k) * nd + q;
      out[0] = v0;
      out[nd] = v1;
      out[2 * (long long)nd] = v2;
      fd[3 * k] = fma(v0, b, fd[3 * k]);
      fd[3 * k + 1] = fma(v1, b, fd[3 * k + 1]);
      fd[3 * k + 2] = fma(v2, b, fd[3 * k + 2]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3 * PP; k++) red[k][t] = fd[k];
  __syncthreads();
  for (int k = t >> 5; k < 3 * PP; k += kDT / 32) {
    double x = 0.0;
    for (int q = t & 31; q < kDT; q += 32) x += red[k][q];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      x += __shfl_down_sync(0xffffffffu, x, off);
    if ((t & 31) == 0 && p0 + k / 3 < P) fdots[3 * p0 + k] = x;
  }
}

// center[q] = a for the pairs q of atom a: a warp per atom.
__global__ void k_pair_center(int N, const long long *__restrict__ off,
                              int *__restrict__ center) {
  const int a = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (a >= N) return;
  for (long long q = off[a] + (threadIdx.x & 31); q < off[a + 1]; q += 32)
    center[q] = a;
}

// Dots_s = B2[perm] S_s^T (raw descriptors), Ns x Ms.
__global__ void __launch_bounds__(GT)
k_dots(int M, int N, int K, const double *__restrict__ B2,
       const int *__restrict__ perm, const double *__restrict__ S,
       double *__restrict__ out) {
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  double acc[4][4];
  gemm_mainloop<true>(acc, m0, n0, M, N, K, B2, K, perm, S, K);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    int m = m0 + ty + 16 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int n = n0 + tx + 16 * j;
      if (n < N) out[(long long)m * N + n] = acc[i][j];
    }
  }
}

// Force-kernel values for the pairs of species-s centres
// (normalized_dot_product.cpp:185-198): rows are dB2 rows 3p+c (gathered),
// columns the species' sparse environments.  Written into FK[3P x M].
__global__ void __launch_bounds__(GT)
k_force_kernel(int R, int Ms, int K, const double *__restrict__ dB2,
               const int *__restrict__ rows, const double *__restrict__ S,
               const int *__restrict__ pair_center,
               const int *__restrict__ inv_perm,
               const double *__restrict__ dots, const double *__restrict__ dnorm,
               const double *__restrict__ snorm,
               const double *__restrict__ fdots, double sig2, double power,
               int c_s, int M, double *__restrict__ FK) {
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  double acc[4][4];
  gemm_mainloop<true>(acc, m0, n0, R, Ms, K, dB2, K, rows, S, K);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    int m = m0 + ty + 16 * i;
    if (m >= R) continue;
    long long gr = rows[m];
    int pair = (int)(gr / 3);
    int atom = pair_center[pair];
    int jl = inv_perm[atom];
    double nj = dnorm[atom];
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      int n = n0 + tx + 16 * jj;
      if (n >= Ms) continue;
      double ni = snorm[n];
      double v = 0.0;
      if (ni >= kEmptyThresh && nj >= kEmptyThresh) {
        double nij = ni * nj, nij3 = nij * nj * nj;
        double dv = dots[(long long)jl * Ms + n];
        double nd_ = dv / nij;
        double dval = power * (power == 2.0 ? nd_
                                            : power == 1.0 ? 1.0
                                                           : pow(nd_, power - 1.0));
        double f1 = acc[i][jj] / nij;
        double f2 = dv * fdots[gr] / nij3;
        v = sig2 * dval * (f1 - f2);
      }
      FK[gr * M + c_s + n] = v;
    }
  }
}

// The energy and stress columns are sums over all atoms or pairs for every
// sparse row: block (32 sparse rows x 8 groups) x chunk of atoms or pairs,
// then k_col_final adds the chunks in order.  A thread per sparse row that
// walked every pair alone took 1,751 us (108 FCC atoms, 3,456 pairs, 200
// sparse rows) and every atom 406 us; the three kernels here take 12, 7 and
// 9 us, the stress part at 1.4 TB/s of FK (16.6 MB, partly in L2).
constexpr int kColRows = 32, kColGroups = 8;

// part[ch][i] = sum over the chunk's atoms j of sig2 (dot_ij / |s_i||d_j|)^power
__global__ void __launch_bounds__(kColRows * kColGroups)
k_energy_part(int Ns, int Ms, int per, const double *__restrict__ dots,
              const int *__restrict__ perm, const double *__restrict__ dnorm,
              const double *__restrict__ snorm, double sig2, double power,
              double *__restrict__ part, int ldp) {
  __shared__ double red[kColGroups][kColRows + 1];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int i = blockIdx.x * kColRows + x, ch = blockIdx.y;
  double acc = 0.0;
  if (i < Ms) {
    const double ni = snorm[i];
    const int j1 = min(Ns, (ch + 1) * per);
    if (ni >= kEmptyThresh)
      for (int j = ch * per + g; j < j1; j += kColGroups) {
        const double nj = dnorm[perm[j]];
        if (nj < kEmptyThresh) continue;
        acc += sig2 * powx(dots[(long long)j * Ms + i] / (ni * nj), power);
      }
  }
  red[g][x] = acc;
  __syncthreads();
  if (g == 0 && i < Ms) {
    for (int q = 1; q < kColGroups; q++) acc += red[q][x];
    part[(long long)ch * ldp + i] = acc;
  }
}

// part[ch][k][i] = sum over the chunk's pairs of fk_a r_b (b >= a, flare order)
__global__ void __launch_bounds__(kColRows * kColGroups)
k_stress_part(int M, long long P, long long per,
              const double4_16a *__restrict__ rel,
              const double *__restrict__ FK, double *__restrict__ part) {
  __shared__ double red[6][kColGroups][kColRows + 1];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int i = blockIdx.x * kColRows + x;
  const long long ch = blockIdx.y;
  double s[6] = {0, 0, 0, 0, 0, 0};
  if (i < M) {
    const long long p1 = min(P, (ch + 1) * per);
    for (long long p = ch * per + g; p < p1; p += kColGroups) {
      const double4_16a r = rel[p];
      const double *f = FK + 3 * p * M + i;
      const double f0 = f[0], f1 = f[M], f2 = f[2LL * M];
      s[0] = fma(f0, r.y, s[0]);
      s[1] = fma(f0, r.z, s[1]);
      s[2] = fma(f0, r.w, s[2]);
      s[3] = fma(f1, r.z, s[3]);
      s[4] = fma(f1, r.w, s[4]);
      s[5] = fma(f2, r.w, s[5]);
    }
  }
#pragma unroll
  for (int k = 0; k < 6; k++) red[k][g][x] = s[k];
  __syncthreads();
  if (g < 6 && i < M) {
    double t = 0.0;
    for (int q = 0; q < kColGroups; q++) t += red[g][q][x];
    part[(ch * 6 + g) * M + i] = t;
  }
}

// Energy column (k = 0) and stress columns (k = 1..6, times -1/V) from the
// chunks' partial sums: kern[i][col].
__global__ void k_col_final(int M, int nce, int ncs,
                            const double *__restrict__ epart,
                            const double *__restrict__ spart, double vol_inv,
                            int n_atoms, long long ncol,
                            double *__restrict__ kern) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (i >= M) return;
  double s = 0.0;
  if (k == 0) {
    for (int c = 0; c < nce; c++) s += epart[(long long)c * M + i];
    kern[(long long)i * ncol] = s;
  } else {
    for (int c = 0; c < ncs; c++) s += spart[((long long)c * 6 + k - 1) * M + i];
    kern[(long long)i * ncol + 1 + 3LL * n_atoms + k - 1] = -s * vol_inv;
  }
}

// Force columns by owner-computes: K[i][1+3a+c] = sum_{p in out(a)}
// FK[3p+c][i] - FK[3 twin(p)+c][i].  Thread per (sparse i, atom a).
__global__ void k_force_cols(int M, int N, const long long *__restrict__ off,
                             const long long *__restrict__ twin,
                             const double *__restrict__ FK, long long ncol,
                             double *__restrict__ kern) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)M * N) return;
  int i = (int)(idx % M), a = (int)(idx / M);
  double f[3] = {0.0, 0.0, 0.0};
  for (long long q = off[a]; q < off[a + 1]; q++) {
    long long tw = twin[q];
    for (int c = 0; c < 3; c++) {
      double v = FK[(3 * q + c) * M + i];
      if (tw >= 0) v -= FK[(3 * tw + c) * M + i];
      f[c] += v;
    }
  }
  for (int c = 0; c < 3; c++) kern[(long long)i * ncol + 1 + 3 * a + c] = f[c];
}

// mean_efs[o] = sum_i kern[i][o] alpha[i]
__global__ void k_kern_t_alpha(int M, long long ncol, const double *__restrict__ kern,
                               const double *__restrict__ alpha,
                               double *__restrict__ out) {
  long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= ncol) return;
  double acc = 0.0;
  for (int i = 0; i < M; i++) acc += kern[(long long)i * ncol + o] * alpha[i];
  out[o] = acc;
}

__global__ void k_rownorms(int M, int nd, const double *__restrict__ S,
                           double *__restrict__ out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M) return;
  double acc = 0.0;
  for (int q = 0; q < nd; q++) acc += S[(long long)i * nd + q] * S[(long long)i * nd + q];
  out[i] = sqrt(acc);
}

}  // namespace

int launch_b2_dervs(const B2Params &p, const fgb_nlist_s *nl,
                    const int *d_species, const double *d_A, const double *d_B2,
                    double *d_dB2, double *d_force_dots, DevBuf &center,
                    DevBuf &basis, cudaStream_t st) {
  const int N = nl->n_atoms;
  const long long P = nl->n_pairs;
  if (N == 0 || P == 0) return FGB_OK;
  // dA of a pair: PP = 8 pairs a block while they leave room for two blocks
  // on an SM, else 2
  const size_t per = sizeof(double) * 3 * (size_t)p.n_max * p.n_harm;
  const int PP = 8 * per <= 96 * 1024 ? 8 : 2;
  // descriptors whose A, B2 row and pair basis together exceed 200 KB are
  // refused by every stored-gradient entry point
  const size_t sm = sizeof(double) * ((size_t)p.n_A + p.n_d + 2 * p.n_max +
                                      4 * p.n_harm + 192) + per;
  if (sm > 200 * 1024) {
    set_error("stored-gradient form needs %zu bytes of shared memory", sm);
    return FGB_EINVAL;
  }
  int rc;
  if ((rc = center.ensure(sizeof(int) * P)) ||
      (rc = basis.ensure(sizeof(double) * (2 * p.n_max + 4 * p.n_harm) *
                         (size_t)P)))
    return rc;
  k_pair_center<<<ceil_div((long long)N * 32, 128), 128, 0, st>>>(
      N, nl->offsets.as<long long>(), center.as<int>());
  FGB_LAUNCH_CHECK("k_pair_center");
  const auto eval = [&](auto lc) {
    k_pair_basis<decltype(lc)::value><<<ceil_div(P, kBT), kBT, 0, st>>>(
        p, P, center.as<int>(), nl->nbr_j.as<int>(),
        nl->nbr_rel.as<double4_16a>(), d_species, basis.as<double>());
  };
  switch (p.l_max) {
    case 1: eval(std::integral_constant<int, 1>()); break;
    case 2: eval(std::integral_constant<int, 2>()); break;
    case 3: eval(std::integral_constant<int, 3>()); break;
    case 4: eval(std::integral_constant<int, 4>()); break;
    case 5: eval(std::integral_constant<int, 5>()); break;
    case 6: eval(std::integral_constant<int, 6>()); break;
    default: eval(std::integral_constant<int, 0>()); break;
  }
  FGB_LAUNCH_CHECK("k_pair_basis");
  const auto dervs = [&](auto pp) -> int {
    constexpr int K = decltype(pp)::value;
    FGB_CUDA(cudaFuncSetAttribute(k_b2_dervs<K>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(K * per)));
    k_b2_dervs<K><<<ceil_div(P, K), kDT, K * per, st>>>(
        p, P, center.as<int>(), nl->nbr_j.as<int>(),
        nl->nbr_rel.as<double4_16a>(), d_species, basis.as<double>(), d_A,
        d_B2, d_dB2, d_force_dots);
    return FGB_OK;
  };
  if ((rc = PP == 8 ? dervs(std::integral_constant<int, 8>())
                    : dervs(std::integral_constant<int, 2>())))
    return rc;
  FGB_LAUNCH_CHECK("k_b2_dervs");
  return FGB_OK;
}

}  // namespace fgb

using namespace fgb;

extern "C" int fgb_envs_envs(const double *d_desc1, const double *d_norm1,
                             int n1, const double *d_desc2,
                             const double *d_norm2, int n2, int n_desc,
                             double sig2, double power, double *d_kern,
                             void *stream) {
  if (n1 < 0 || n2 < 0 || n_desc <= 0 || (n1 && n2 && !d_kern)) {
    set_error("fgb_envs_envs: invalid arguments");
    return FGB_EINVAL;
  }
  if (n1 == 0 || n2 == 0) return FGB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  dim3 g(ceil_div(n2, BN), ceil_div(n1, BM));
  k_envs_envs<<<g, GT, 0, st>>>(n1, n2, n_desc, d_desc1, d_norm1, d_desc2,
                                d_norm2, sig2, power, d_kern);
  FGB_LAUNCH_CHECK("k_envs_envs");
  return FGB_OK;
}


extern "C" int fgb_b2_forward_dervs(fgb_b2_t b2, fgb_nlist_t nl,
                                    const int *d_species, double *d_B2,
                                    double *d_norms, double *d_dB2,
                                    double *d_force_dots, void *stream) {
  if (!b2 || !nl || !d_B2 || !d_norms || !d_dB2 || !d_force_dots) {
    set_error("fgb_b2_forward_dervs: invalid arguments");
    return FGB_EINVAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  DevBuf A, flag, center, basis;
  int rc;
  if ((rc = check_species(d_species, nl->n_atoms, b2->p.n_species, flag, st)))
    return rc;
  if ((rc = A.ensure(sizeof(double) * ((size_t)nl->n_atoms * b2->p.n_A + 1))))
    return rc;
  if ((rc = launch_b2_forward(b2->p, nl, d_species, A.as<double>(), d_B2,
                              d_norms, st)))
    return rc;
  rc = launch_b2_dervs(b2->p, nl, d_species, A.as<double>(), d_B2, d_dB2,
                       d_force_dots, center, basis, st);
  if (!rc) FGB_CUDA(cudaStreamSynchronize(st));
  return rc;
}

namespace fgb {
// envs_struc for one structure into d_kern; B2/norms of the structure are
// left in ws (for the plain prediction's variance stage).
int envs_struc_impl(const B2Params &p, double sigma, double power,
                           const int *h_counts, const double *d_sparse,
                           fgb_nlist_s *nl, const int *d_species,
                           double *d_kern, fgb_workspace &ws,
                           cudaStream_t st) {
  if (nl->n_struc != 1) {
    set_error("envs_struc needs a single-structure neighbour list");
    return FGB_EINVAL;
  }
  const int N = nl->n_atoms, S = p.n_species, nd = p.n_d;
  const long long P = nl->n_pairs;
  int rc;
  if ((rc = check_species(d_species, N, S, ws.flag, st))) return rc;
  std::vector<int> off(S + 1, 0);
  for (int s = 0; s < S; s++) off[s + 1] = off[s] + h_counts[s];
  const int M = off[S];
  const long long ncol = 1 + 3LL * N + 6;
  if (M == 0) return FGB_OK;
  FGB_CUDA(cudaMemsetAsync(d_kern, 0, sizeof(double) * M * ncol, st));
  if (N == 0) return FGB_OK;
  if ((rc = ws.A.ensure(sizeof(double) * ((size_t)N * p.n_A + 1))) ||
      (rc = ws.B2.ensure(sizeof(double) * ((size_t)N * nd + 1))) ||
      (rc = ws.norms.ensure(sizeof(double) * (N + 1))) ||
      (rc = ws.dB2.ensure(sizeof(double) * ((size_t)3 * P * nd + 1))) ||
      (rc = ws.fdots.ensure(sizeof(double) * (3 * P + 1))) ||
      (rc = ws.kern.ensure(sizeof(double) * ((size_t)3 * P * M + 1))) ||
      (rc = ws.var.ensure(sizeof(double) * (M + 1))) ||
      (rc = ws.pos.ensure(sizeof(int) * (P + 1))) ||
      (rc = ws.perm.ensure(sizeof(int) * (N + 1))) ||
      (rc = ws.flags.ensure(sizeof(int) * (N + 1))) ||
      (rc = ws.scal.ensure(sizeof(int) * (3 * P + 1))))
    return rc;
  if ((rc = launch_b2_forward(p, nl, d_species, ws.A.as<double>(),
                              ws.B2.as<double>(), ws.norms.as<double>(), st)))
    return rc;
  if ((rc = launch_b2_dervs(p, nl, d_species, ws.A.as<double>(),
                            ws.B2.as<double>(), ws.dB2.as<double>(),
                            ws.fdots.as<double>(), ws.pos, ws.basis, st)))
    return rc;
  // host-side species permutation and pair rows (plain path: sync is fine)
  std::vector<int> hs(N);
  std::vector<long long> hoff(N + 1);
  FGB_CUDA(cudaMemcpyAsync(hs.data(), d_species, sizeof(int) * N,
                           cudaMemcpyDeviceToHost, st));
  FGB_CUDA(cudaMemcpyAsync(hoff.data(), nl->offsets.p,
                           sizeof(long long) * (N + 1), cudaMemcpyDeviceToHost,
                           st));
  FGB_CUDA(cudaStreamSynchronize(st));
  std::vector<int> perm, inv(N), rows;
  std::vector<int> sbase(S + 1, 0);
  for (int s = 0; s < S; s++) {
    sbase[s] = (int)perm.size();
    for (int a = 0; a < N; a++)
      if (hs[a] == s) { inv[a] = (int)perm.size() - sbase[s]; perm.push_back(a); }
  }
  sbase[S] = N;
  FGB_CUDA(cudaMemcpyAsync(ws.perm.p, perm.data(), sizeof(int) * N,
                           cudaMemcpyHostToDevice, st));
  FGB_CUDA(cudaMemcpyAsync(ws.flags.p, inv.data(), sizeof(int) * N,
                           cudaMemcpyHostToDevice, st));
  DevBuf snorm, dots, rowsd;
  if ((rc = snorm.ensure(sizeof(double) * (M + 1)))) return rc;
  k_rownorms<<<ceil_div(M, 128), 128, 0, st>>>(M, nd, d_sparse,
                                               snorm.as<double>());
  FGB_LAUNCH_CHECK("k_rownorms");
  FGB_CUDA(cudaMemsetAsync(ws.kern.p, 0, sizeof(double) * 3 * P * M, st));
  const double sig2 = sigma * sigma;
  // chunks of the energy (atoms) and stress (pairs) sums: at least 32 atoms
  // or pairs each and at most 128 chunks
  const int eper = std::max(32, ceil_div(N, 128)), nce = ceil_div(N, eper);
  const long long sper = std::max(32LL, (P + 127) / 128);
  const int ncs = ceil_div(P, sper);
  if ((rc = ws.part.ensure(sizeof(double) * (size_t)M * (nce + 6 * ncs))))
    return rc;
  double *spart = ws.part.as<double>() + (size_t)M * nce;
  FGB_CUDA(cudaMemsetAsync(ws.part.p, 0, sizeof(double) * (size_t)M * nce, st));
  for (int s = 0; s < S; s++) {
    const int Ns = sbase[s + 1] - sbase[s], Ms = h_counts[s];
    if (Ns == 0 || Ms == 0) continue;
    const double *Ss = d_sparse + (size_t)off[s] * nd;
    const int *perm_s = ws.perm.as<int>() + sbase[s];
    if ((rc = dots.ensure(sizeof(double) * (size_t)Ns * Ms))) return rc;
    dim3 g1(ceil_div(Ms, BN), ceil_div(Ns, BM));
    k_dots<<<g1, GT, 0, st>>>(Ns, Ms, nd, ws.B2.as<double>(), perm_s, Ss,
                              dots.as<double>());
    FGB_LAUNCH_CHECK("k_dots");
    k_energy_part<<<dim3(ceil_div(Ms, kColRows), ceil_div(Ns, eper)),
                    kColRows * kColGroups, 0, st>>>(
        Ns, Ms, eper, dots.as<double>(), perm_s, ws.norms.as<double>(),
        snorm.as<double>() + off[s], sig2, power,
        ws.part.as<double>() + off[s], M);
    FGB_LAUNCH_CHECK("k_energy_part");
    rows.clear();
    for (int k = sbase[s]; k < sbase[s + 1]; k++) {
      int a = perm[k];
      for (long long q = hoff[a]; q < hoff[a + 1]; q++)
        for (int c = 0; c < 3; c++) rows.push_back((int)(3 * q + c));
    }
    const int R = (int)rows.size();
    if (R == 0) continue;
    if ((rc = rowsd.ensure(sizeof(int) * R))) return rc;
    FGB_CUDA(cudaMemcpyAsync(rowsd.p, rows.data(), sizeof(int) * R,
                             cudaMemcpyHostToDevice, st));
    dim3 g2(ceil_div(Ms, BN), ceil_div(R, BM));
    k_force_kernel<<<g2, GT, 0, st>>>(
        R, Ms, nd, ws.dB2.as<double>(), rowsd.as<int>(), Ss, ws.pos.as<int>(),
        ws.flags.as<int>(), dots.as<double>(), ws.norms.as<double>(),
        snorm.as<double>() + off[s], ws.fdots.as<double>(), sig2, power,
        off[s], M, ws.kern.as<double>());
    FGB_LAUNCH_CHECK("k_force_kernel");
    FGB_CUDA(cudaStreamSynchronize(st));   // rows buffer reused next species
  }
  k_force_cols<<<ceil_div((long long)M * N, 128), 128, 0, st>>>(
      M, N, nl->offsets.as<long long>(), nl->nbr_twin.as<long long>(),
      ws.kern.as<double>(), ncol, d_kern);
  FGB_LAUNCH_CHECK("k_force_cols");
  if (P > 0) {
    k_stress_part<<<dim3(ceil_div(M, kColRows), ncs), kColRows * kColGroups, 0,
                    st>>>(M, P, sper, nl->nbr_rel.as<double4_16a>(),
                          ws.kern.as<double>(), spart);
    FGB_LAUNCH_CHECK("k_stress_part");
  }
  k_col_final<<<dim3(ceil_div(M, 128), 7), 128, 0, st>>>(
      M, nce, ncs, ws.part.as<double>(), spart, 1.0 / nl->h_volume[0], N, ncol,
      d_kern);
  FGB_LAUNCH_CHECK("k_col_final");
  return FGB_OK;
}
}  // namespace fgb

extern "C" int fgb_envs_struc(fgb_b2_t b2, double sigma, double power,
                              const int *h_counts, const double *d_sparse,
                              fgb_nlist_t nl, const int *d_species,
                              double *d_kern, void *stream) {
  if (!b2 || !nl || !h_counts || !d_kern) {
    set_error("fgb_envs_struc: invalid arguments");
    return FGB_EINVAL;
  }
  fgb_workspace ws;
  cudaStream_t st = (cudaStream_t)stream;
  int rc = envs_struc_impl(b2->p, sigma, power, h_counts, d_sparse, nl,
                           d_species, d_kern, ws, st);
  if (!rc) FGB_CUDA(cudaStreamSynchronize(st));
  return rc;
}

extern "C" int fgb_predict_plain(fgb_model_t m, fgb_nlist_t nl,
                                 const int *d_species, double *d_mean_efs,
                                 double *d_local_var, void *stream) {
  if (!m || !nl || !d_mean_efs) {
    set_error("fgb_predict_plain: invalid arguments");
    return FGB_EINVAL;
  }
  if (!m->solved) {
    set_error("L_inv must be up to date to make predictions. Please call "
              "update_matrices_QR and try again.");
    return FGB_ESTALE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int N = nl->n_atoms, M = m->M;
  const long long ncol = 1 + 3LL * N + 6;
  int rc;
  DevBuf kern;
  if ((rc = kern.ensure(sizeof(double) * ((size_t)M * ncol + 1)))) return rc;
  if ((rc = envs_struc_impl(m->b2, m->sigma, m->power, m->h_counts.data(),
                            m->Sraw.as<double>(), nl, d_species,
                            kern.as<double>(), m->ws, st)))
    return rc;
  k_kern_t_alpha<<<ceil_div(ncol, 128), 128, 0, st>>>(
      M, ncol, kern.as<double>(), m->alpha.as<double>(), d_mean_efs);
  FGB_LAUNCH_CHECK("k_kern_t_alpha");
  if (d_local_var && N > 0) {
    // local variances: envs_envs(structure, sparse) then |L_inv k|^2
    // (sparse_gp.cpp:116-133), on the B2 values left in the workspace.
    std::vector<int> counts;
    if ((rc = species_permutation(m, d_species, N, counts, st))) return rc;
    if ((rc = m->ws.var.ensure(sizeof(double) * (N + 1)))) return rc;
    if ((rc = kernel_stage_fp64(m, N, counts, false, true, nullptr, nullptr,
                                m->ws.var.as<double>(), st)))
      return rc;
    FGB_CUDA(cudaMemcpyAsync(d_local_var, m->ws.var.p, sizeof(double) * N,
                             cudaMemcpyDeviceToDevice, st));
  }
  FGB_CUDA(cudaStreamSynchronize(st));
  return FGB_OK;
}

// ------------------------------------------------------------ QR solve
// SparseGP::update_matrices_QR (sparse_gp.cpp:607-641) in FP64:
//   L = chol(Kuu + jitter I);  L_inv = L^-1
//   A = [diag(sqrt(noise)) Kuf^T ; L^T],  b = [sqrt(noise) y ; 0]
//   A = QR;  alpha = R^-1 (Q^T b)[:M];  R_inv = R^-1
// (dense.cu holds the factorisations)
namespace fgb {
namespace {
__global__ void k_add_diag(int M, double *A, double v) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < M) A[(long long)i * M + i] += v;
}
// alpha = R_inv Qb (R_inv row-major upper): a warp per row, lanes over
// columns, fixed-order shuffle tree.
__global__ void k_upper_gemv(int M, const double *R, const double *x,
                             double *y) {
  const int row = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= M) return;
  double s = 0.0;
  for (int j = row + lane; j < M; j += 32) s += R[(long long)row * M + j] * x[j];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) y[row] = s;
}
}  // namespace
}  // namespace fgb

#define FGB_SOLVER(call, what)                                          \
  do {                                                                  \
    int s_ = (int)(call);                                               \
    if (s_ != 0) {                                                      \
      set_error("%s failed with status %d", what, s_);                  \
      rc = FGB_ECUDA;                                                   \
      goto done;                                                        \
    }                                                                   \
  } while (0)

// SparseGP::update_matrices_QR (sparse_gp.cpp:607-641) on the GPU in FP64,
// by the kernels of dense.cu: L = chol(Kuu + jitter I), L_inv = L^-1, the
// QR of A = [sqrt(noise) Kuf^T; L^T] by shifted Cholesky QR (R_inv and
// Q^T b; every O(n M^2) and O(M^3) product an FP64-level tensor-core
// product), alpha = R_inv (Q^T b)[:M] (the reference's R_inv * Q_b).
extern "C" int fgb_solve_qr(int M, int n_labels, const double *d_Kuu,
                            const double *d_Kuf, const double *d_y,
                            const double *d_noise, double jitter,
                            double *d_alpha, double *d_L_inv, double *d_R_inv,
                            void *stream) {
  if (M <= 0 || n_labels < 0 || !d_Kuu || !d_alpha || !d_L_inv ||
      (n_labels > 0 && (!d_Kuf || !d_y || !d_noise))) {
    set_error("fgb_solve_qr: invalid arguments");
    return FGB_EINVAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const long long rows = (long long)n_labels + M;
  int rc = FGB_OK;
  DevBuf L, At, b, Qtb, Rinv;
  double *R_inv = d_R_inv;
  if ((rc = L.ensure(sizeof(double) * (size_t)M * M)) ||
      (rc = At.ensure(sizeof(double) * (size_t)rows * M)) ||
      (rc = b.ensure(sizeof(double) * (size_t)rows)) ||
      (rc = Qtb.ensure(sizeof(double) * (size_t)M)))
    return rc;
  if (!R_inv) {
    if ((rc = Rinv.ensure(sizeof(double) * (size_t)M * M))) return rc;
    R_inv = Rinv.as<double>();
  }
  FGB_CUDA(cudaMemcpyAsync(L.p, d_Kuu, sizeof(double) * (size_t)M * M,
                           cudaMemcpyDeviceToDevice, st));
  k_add_diag<<<ceil_div(M, 256), 256, 0, st>>>(M, L.as<double>(), jitter);
  FGB_LAUNCH_CHECK("k_add_diag");
  if ((rc = dense::cholesky(M, L.as<double>(), M, st)) ||
      (rc = dense::trtri_lower(M, L.as<double>(), M, d_L_inv, M, st)) ||
      (rc = dense::build_At(M, n_labels, d_Kuf, d_noise, d_y, L.as<double>(),
                            At.as<double>(), b.as<double>(), st)) ||
      (rc = dense::cholqr_solve(M, rows, At.as<double>(), b.as<double>(),
                                R_inv, Qtb.as<double>(), st)))
    return rc;
  k_upper_gemv<<<ceil_div((long long)M * 32, 256), 256, 0, st>>>(
      M, R_inv, Qtb.as<double>(), d_alpha);
  FGB_LAUNCH_CHECK("k_upper_gemv");
  FGB_CUDA(cudaStreamSynchronize(st));
  return FGB_OK;
}

// Thin Q of a Householder QR (cuSOLVER geqrf + orgqr): A and Q column-major
// rows x cols (rows >= cols).  The varmap coefficients of a power-1 model
// (normalized_dot_product.cpp:769-830) are the leading rows of such a Q.
extern "C" int fgb_qr_thin_q(int rows, int cols, const double *d_A,
                             double *d_Q, void *stream) {
  if (rows <= 0 || cols <= 0 || rows < cols || !d_A || !d_Q) {
    set_error("fgb_qr_thin_q: invalid arguments (rows >= cols > 0)");
    return FGB_EINVAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int rc = FGB_OK;
  cusolverDnHandle_t sol = nullptr;
  DevBuf tau, work, info;
  int lwork = 0, lw2 = 0, hinfo = 0;
  if ((rc = tau.ensure(sizeof(double) * (size_t)cols)) ||
      (rc = info.ensure(sizeof(int))))
    return rc;
  FGB_SOLVER(cusolverDnCreate(&sol), "cusolverDnCreate");
  FGB_SOLVER(cusolverDnSetStream(sol, st), "cusolverDnSetStream");
  FGB_SOLVER(cudaMemcpyAsync(d_Q, d_A, sizeof(double) * (size_t)rows * cols,
                             cudaMemcpyDeviceToDevice, st), "copy A");
  FGB_SOLVER(cusolverDnDgeqrf_bufferSize(sol, rows, cols, d_Q, rows, &lwork),
             "geqrf_bufferSize");
  FGB_SOLVER(cusolverDnDorgqr_bufferSize(sol, rows, cols, cols, d_Q, rows,
                                         tau.as<double>(), &lw2),
             "orgqr_bufferSize");
  lwork = std::max(lwork, lw2);
  if ((rc = work.ensure(sizeof(double) * ((size_t)lwork + 1)))) goto done;
  FGB_SOLVER(cusolverDnDgeqrf(sol, rows, cols, d_Q, rows, tau.as<double>(),
                              work.as<double>(), lwork, info.as<int>()),
             "geqrf");
  FGB_SOLVER(cusolverDnDorgqr(sol, rows, cols, cols, d_Q, rows,
                              tau.as<double>(), work.as<double>(), lwork,
                              info.as<int>()),
             "orgqr");
  FGB_SOLVER(cudaMemcpyAsync(&hinfo, info.p, sizeof(int),
                             cudaMemcpyDeviceToHost, st), "info");
  FGB_SOLVER(cudaStreamSynchronize(st), "sync");
  if (hinfo != 0) {
    set_error("fgb_qr_thin_q: QR failed (info %d)", hinfo);
    rc = FGB_ECUDA;
  }
done:
  if (sol) cusolverDnDestroy(sol);
  return rc;
}
