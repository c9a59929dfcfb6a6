// The stored-gradient form, the reference's algorithm on the GPU (forward-mode
// descriptor gradients, envs_struc as exact-slice products and sums over the
// pairs), envs_envs, and the FP64 QR solve.
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
// Kernels over the flat pair list, bound by FP64 instructions (64 cycles each
// per warp on an SM quarter), so the pairs are spread over all SMs.  One
// block per atom that walked its pairs in series, one thread evaluating each
// pair's basis, took 913 us for 108 FCC atoms (3,456 pairs, n_d 144) and a
// thread per descriptor over eight pairs' rows 78 us (lanes of different l
// and species blocks); these take 64 us (k_pair_basis 14, k_b2_dervs 38,
// k_row_dots 12).
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

// Radial pairs (n1 <= n2) ordered for a neighbour of species s = blockIdx.x:
// first those with both in its block of n_max (two products), then one in it
// (one product), then none (zero rows); tab[s npair + rank] = n1 | n2 << 16.
__global__ void k_derv_items(int nr, int nm, int npair, int *__restrict__ tab) {
  const int s = blockIdx.x, lo = s * nm, hi = lo + nm, out = nr - nm;
  const int two = nm * (nm + 1) / 2, one = nm * out;
  int n1 = 0, first = 0;   // pairs of rows before n1
  for (int pi = threadIdx.x; pi < npair; pi += blockDim.x) {
    while (pi - first >= nr - n1) { first += nr - n1; n1++; }
    const int n2 = n1 + pi - first;
    const bool i1 = n1 >= lo && n1 < hi, i2 = n2 >= lo && n2 < hi;
    // index among the columns outside the block
    const int o1 = n1 < lo ? n1 : n1 - nm, o2 = n2 < lo ? n2 : n2 - nm;
    int r;
    if (i1 && i2) r = (n1 - lo) * nm - (n1 - lo) * (n1 - lo - 1) / 2 + n2 - n1;
    else if (i1) r = two + (n1 - lo) * out + o2;
    else if (i2) r = two + (n2 - lo) * out + o1;
    else r = two + one + o1 * out - o1 * (o1 - 1) / 2 + o2 - o1;
    tab[s * npair + r] = n1 | n2 << 16;
  }
}

// dB2 rows of PP consecutive pairs: their dA and their centres' A in shared
// memory (rows of odd length, so that the lanes' rows fall into different
// banks), then a thread per (pair, radial pair) for its l_max + 1 values of
// the three components, in k_derv_items' order so that a warp's threads do
// the same number of products.
constexpr int kDTmax = 256;
template <int PP, int LC>
__global__ void __launch_bounds__(kDTmax)
k_b2_dervs(B2Params p, long long P, const int *__restrict__ center,
           const int *__restrict__ nbr_j, const double4_16a *__restrict__ rel,
           const int *__restrict__ species, const double *__restrict__ basis,
           const int *__restrict__ tab, int npair,
           const double *__restrict__ A_in, double *__restrict__ dB2) {
  extern __shared__ double sm[];   // dA: PP x 3 x nm x ld | A: PP x nr x ld
  const int L = LC > 0 ? LC : p.l_max, L1 = L + 1;
  const int nh = L1 * L1, ld = nh | 1;
  const int nm = p.n_max, nr = p.n_rad, nd = p.n_d, nmh = nm * nh;
  const long long p0 = (long long)blockIdx.x * PP;
  const int np = (int)min((long long)PP, P - p0);
  const int t = threadIdx.x, nt = blockDim.x;
  double *dA = sm, *As = sm + PP * 3 * nm * ld;
  __shared__ int s_slot[PP], s_sj[PP];
  if (t < np) {
    // pairs of one centre share the slot of the first
    const int c = center[p0 + t];
    int k = t;
    while (k > 0 && center[p0 + k - 1] == c) k--;
    s_slot[t] = k;
    s_sj[t] = species[nbr_j[p0 + t]];
  }
  __syncthreads();
  for (int k = 0; k < np; k++) {
    const double4_16a r = rel[p0 + k];
    const double ir = 1.0 / r.x;
    for (int e = t; e < nmh; e += nt) {
      const int n = e / nh, lm = e - n * nh;
      const double *bn = basis + n * P + p0 + k;
      const double *by = basis + (2 * nm + lm) * P + p0 + k;
      const double g = bn[0], dgy = bn[nm * P] * ir * by[0];
      double *d = dA + (k * 3 * nm + n) * ld + lm;
      d[0] = fma(dgy, r.y, g * by[nh * P]);
      d[nm * ld] = fma(dgy, r.z, g * by[2 * nh * P]);
      d[2 * nm * ld] = fma(dgy, r.w, g * by[3 * nh * P]);
    }
    if (s_slot[k] == k) {
      const double *A = A_in + (long long)center[p0 + k] * p.n_A;
      for (int e = t; e < nr * nh; e += nt)
        As[(k * nr + e / nh) * ld + e % nh] = A[e];
    }
  }
  __syncthreads();
  const int two = nm * (nm + 1) / 2, one = nm * (nr - nm);
  int k = 0;
  for (int f = t;; f += nt) {
    while (k < np && f - k * npair >= npair) k++;
    if (k >= np) break;
    const int it = f - k * npair, sj = s_sj[k];
    const int n12 = tab[sj * npair + it], n1 = n12 & 0xFFFF, n2 = n12 >> 16;
    const int pidx = n1 * nr - n1 * (n1 - 1) / 2 + n2 - n1;
    double *out = dB2 + 3 * (p0 + k) * nd + pidx * L1;
    // product 1: dA of the column in the block, A of the other
    const bool in1 = it < two || (n1 >= sj * nm && n1 < (sj + 1) * nm);
    const int cin = in1 ? n1 : n2, cot = in1 ? n2 : n1;
    const double *a = As + (s_slot[k] * nr + cot) * ld;
    const double *d = dA + (k * 3 * nm + cin - sj * nm) * ld;
    const double *b = As + (s_slot[k] * nr + cin) * ld;
    const double *e = dA + (k * 3 * nm + cot - sj * nm) * ld;
#pragma unroll
    for (int l = 0; l <= L; l++) {
      double v0 = 0.0, v1 = 0.0, v2 = 0.0;
      if (it < two + one) {
#pragma unroll
        for (int m = l * l; m < (l + 1) * (l + 1); m++) {
          const double x = a[m];
          v0 = fma(x, d[m], v0);
          v1 = fma(x, d[nm * ld + m], v1);
          v2 = fma(x, d[2 * nm * ld + m], v2);
        }
        if (it < two)
#pragma unroll
          for (int m = l * l; m < (l + 1) * (l + 1); m++) {
            const double x = b[m];
            v0 = fma(x, e[m], v0);
            v1 = fma(x, e[nm * ld + m], v1);
            v2 = fma(x, e[2 * nm * ld + m], v2);
          }
      }
      out[l] = v0;
      out[nd + l] = v1;
      out[2 * (long long)nd + l] = v2;
    }
  }
}

// Each gradient row's dot with its centre's B2 and its largest magnitude (the
// tensor-core row scales): a warp per row.
__global__ void __launch_bounds__(256)
k_row_dots(long long rows, int nd, const int *__restrict__ center,
           const double *__restrict__ dB2, const double *__restrict__ B2,
           double *__restrict__ fdots, double *__restrict__ rowmax) {
  const long long m = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (m >= rows) return;
  const double *a = dB2 + m * nd, *b = B2 + (long long)center[m / 3] * nd;
  double x = 0.0;
  unsigned long long mx = 0;
  for (int q = lane; q < nd; q += 32) {
    const double v = a[q];
    x = fma(v, b[q], x);
    mx = max(mx, (unsigned long long)__double_as_longlong(v) &
                     0x7FFFFFFFFFFFFFFFULL);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    x += __shfl_down_sync(0xffffffffu, x, off);
    mx = max(mx, (unsigned long long)__shfl_down_sync(0xffffffffu,
                                                      (long long)mx, off));
  }
  if (lane == 0) {
    fdots[m] = x;
    if (rowmax) rowmax[m] = __longlong_as_double((long long)mx);
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

// The energy and stress columns are sums over all atoms or pairs for every
// sparse row: block (32 sparse rows x 8 groups) x chunk of atoms or pairs,
// then k_col_final adds the chunks in order.  A thread per sparse row that
// walked every pair alone took 1,751 us (108 FCC atoms, 3,456 pairs, 200
// sparse rows) and every atom 406 us; the three kernels here take 15, 3 and
// 3 us, the stress part at 1.1 TB/s of FK (16.6 MB, partly in L2).
constexpr int kColRows = 32, kColGroups = 8;

// part[ch][i] = sum over the chunk's atoms j of sig2 c_ij^power (c zero for
// empty rows, which add nothing)
__global__ void __launch_bounds__(kColRows * kColGroups)
k_energy_part(int Ns, int Ms, int per, const double *__restrict__ cosine,
              const int *__restrict__ perm, const double *__restrict__ dnorm,
              const double *__restrict__ snorm, double sig2, double power,
              double *__restrict__ part, int ldp) {
  __shared__ double red[kColGroups][kColRows + 1];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int i = blockIdx.x * kColRows + x, ch = blockIdx.y;
  double acc = 0.0;
  if (i < Ms && snorm[i] >= kEmptyThresh) {
    const int j1 = min(Ns, (ch + 1) * per);
    for (int j = ch * per + g; j < j1; j += kColGroups)
      if (dnorm[perm[j]] >= kEmptyThresh)
        acc += sig2 * powx(cosine[(long long)j * Ms + i], power);
  }
  red[g][x] = acc;
  __syncthreads();
  if (g == 0 && i < Ms) {
    for (int q = 1; q < kColGroups; q++) acc += red[q][x];
    part[(long long)ch * ldp + i] = acc;
  }
}

// First sparse row of each species: FK[gr][i] is written only where row i
// and the centre of pair gr / 3 have one species; elsewhere it is zero by
// definition and not read.
struct SparseOffsets {
  int o[kMaxSpecies + 1];
  int n;
  __device__ int species(int i) const {
    int s = 0;
    while (s + 1 < n && i >= o[s + 1]) s++;
    return s;
  }
};

// part[ch][k][i] = sum over the chunk's pairs of fk_a r_b (b >= a, flare order)
__global__ void __launch_bounds__(kColRows * kColGroups)
k_stress_part(int M, long long P, long long per, SparseOffsets so,
              const double4_16a *__restrict__ rel,
              const int *__restrict__ center, const int *__restrict__ species,
              const double *__restrict__ FK, double *__restrict__ part) {
  __shared__ double red[6][kColGroups][kColRows + 1];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int i = blockIdx.x * kColRows + x;
  const long long ch = blockIdx.y;
  double s[6] = {0, 0, 0, 0, 0, 0};
  if (i < M) {
    const int si = so.species(i);
    const long long p1 = min(P, (ch + 1) * per);
    for (long long p = ch * per + g; p < p1; p += kColGroups) {
      if (species[center[p]] != si) continue;
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

// Energy row (k = 0) and stress rows (k = 1..6, times -1/V) of K^T from the
// chunks' partial sums: block of 32 sparse rows, 8 groups of chunks.
__global__ void __launch_bounds__(kColRows * kColGroups)
k_col_final(int M, int nce, int ncs, const double *__restrict__ epart,
            const double *__restrict__ spart, double vol_inv, int n_atoms,
            double *__restrict__ kt) {
  __shared__ double red[kColGroups][kColRows + 1];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int i = blockIdx.x * kColRows + x, k = blockIdx.y;
  const int nc = k ? ncs : nce;
  const double *src = k ? spart + (long long)(k - 1) * M : epart;
  const long long step = k ? 6LL * M : M;
  double s = 0.0;
  if (i < M)
    for (int c = g; c < nc; c += kColGroups) s += src[c * step + i];
  red[g][x] = s;
  __syncthreads();
  if (g || i >= M) return;
  for (int q = 1; q < kColGroups; q++) s += red[q][x];
  if (k == 0) kt[i] = s;
  else kt[(3LL * n_atoms + k) * M + i] = -s * vol_inv;
}

// Force rows of K^T by owner-computes: K^T[1+3a+c][i] = sum_{p in out(a)}
// FK[3p+c][i] - FK[3 twin(p)+c][i].  Block: an atom x 32 sparse rows x 8
// groups of its pairs (one group that walked all of them waited on each
// twin: 37 us against 13, 108 FCC atoms, 200 sparse rows).
__global__ void __launch_bounds__(kColRows * kColGroups)
k_force_cols(int M, int N, SparseOffsets so, const long long *__restrict__ off,
             const int *__restrict__ nbr_j, const long long *__restrict__ twin,
             const int *__restrict__ species, const double *__restrict__ FK,
             double *__restrict__ kt) {
  __shared__ double red[3][kColGroups][kColRows + 1];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int i = blockIdx.y * kColRows + x, a = blockIdx.x;
  double f[3] = {0.0, 0.0, 0.0};
  if (i < M) {
    const int si = so.species(i);
    const bool own = species[a] == si;
    for (long long q = off[a] + g; q < off[a + 1]; q += kColGroups) {
      const long long tw = twin[q];
      if (own)
        for (int c = 0; c < 3; c++) f[c] += FK[(3 * q + c) * M + i];
      if (tw >= 0 && species[nbr_j[q]] == si)
        for (int c = 0; c < 3; c++) f[c] -= FK[(3 * tw + c) * M + i];
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++) red[c][g][x] = f[c];
  __syncthreads();
  if (g < 3 && i < M) {
    double s = 0.0;
    for (int q = 0; q < kColGroups; q++) s += red[g][q][x];
    kt[(1 + 3LL * a + g) * M + i] = s;
  }
}

// The pairs grouped by their centre's species: with the atoms in species
// order (perm), start[k] is the first place of atom perm[k]'s pairs,
// inv[perm[k]] = k and spairs[s] the first place of species s (spairs[S] =
// all pairs).  One block.
__global__ void __launch_bounds__(1024)
k_group_scan(int N, const int *__restrict__ perm, const int *__restrict__ species,
             const long long *__restrict__ off, int S, int *__restrict__ start,
             int *__restrict__ inv, int *__restrict__ spairs) {
  __shared__ int wsum[32], cnt[kMaxSpecies], carry;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t < kMaxSpecies) cnt[t] = 0;
  if (t == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < N; base += 1024) {
    const int k = base + t;
    int n = 0;
    if (k < N) {
      const int a = perm[k];
      n = (int)(off[a + 1] - off[a]);
      inv[a] = k;
      atomicAdd(&cnt[species[a]], n);
    }
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    int before = carry;
    for (int q = 0; q < w; q++) before += wsum[q];
    if (k < N) start[k] = before + x - n;
    __syncthreads();
    if (t == 1023) carry = before + x;
    __syncthreads();
  }
  if (t == 0) {
    int acc = 0;
    for (int s = 0; s < S; s++) {
      spairs[s] = acc;
      acc += cnt[s];
    }
    spairs[S] = acc;
  }
}

// rows[3 r + c] = 3 q + c for the pair q at place r of the grouped order: a
// warp per atom.
__global__ void k_group_rows(int N, const int *__restrict__ perm,
                             const long long *__restrict__ off,
                             const int *__restrict__ start,
                             int *__restrict__ rows) {
  const int k = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (k >= N) return;
  const int a = perm[k];
  const int q0 = (int)off[a], n = (int)(off[a + 1] - off[a]);
  for (int e = threadIdx.x & 31; e < 3 * n; e += 32)
    rows[3 * start[k] + e] = 3 * q0 + e;
}

// out (C x R) = in^T (in: R x C), 32 x 32 tiles.
__global__ void k_transpose32(long long R, int C, const double *__restrict__ in,
                              double *__restrict__ out) {
  __shared__ double t[32][33];
  const long long r0 = (long long)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y)
    if (r0 + k < R && c0 + (int)threadIdx.x < C)
      t[k][threadIdx.x] = in[(r0 + k) * C + c0 + threadIdx.x];
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y)
    if (c0 + k < C && r0 + threadIdx.x < R)
      out[(c0 + k) * R + r0 + threadIdx.x] = t[threadIdx.x][k];
}

// The products' bounded waits: a kernel matrix of which a tile is missing
// becomes NaN as a whole, in the order of the stream (the host does not wait).
__global__ void k_nan_on_flag(long long n, const int *__restrict__ flag,
                              double *__restrict__ out) {
  if (*flag == 0) return;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = __longlong_as_double(0x7FF8000000000000LL);
}

int envs_envs_sliced(const double *d1, const double *norm1, int n1,
                     const double *d2, const double *norm2, int n2, int nd,
                     double sig2, double power, double *d_kern,
                     cudaStream_t st) {
  oz::Sliced A(st), B(st);
  DevBuf err(st);
  const int v = oz::tile64(n1, n2);
  int rc;
  if ((rc = err.ensure(sizeof(int)))) return rc;
  FGB_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), st));
  if ((rc = oz::slice({n1, nd, oz::kTM, d1, nd, nullptr, nullptr}, A, st,
                      oz::kS64)) ||
      (rc = oz::slice({n2, nd, oz::kTN64v[v], d2, nd, nullptr, nullptr}, B, st,
                      oz::kS64)) ||
      (rc = oz::gemm_envs(A, B, norm1, norm2, sig2, power, d_kern,
                          err.as<int>(), st)))
    return rc;
  k_nan_on_flag<<<32, 256, 0, st>>>((long long)n1 * n2, err.as<int>(), d_kern);
  FGB_LAUNCH_CHECK("k_nan_on_flag");
  return FGB_OK;
}

}  // namespace

int launch_b2_dervs(const B2Params &p, const fgb_nlist_s *nl,
                    const int *d_species, const double *d_A, const double *d_B2,
                    double *d_dB2, double *d_force_dots, DevBuf &center,
                    DevBuf &basis, cudaStream_t st, double *d_rowmax) {
  const int N = nl->n_atoms;
  const long long P = nl->n_pairs;
  if (N == 0 || P == 0) return FGB_OK;
  // descriptors whose A, B2 row and pair basis together exceed 200 KB are
  // refused by every stored-gradient entry point
  const size_t lim = sizeof(double) *
                     ((size_t)p.n_A + p.n_d + 2 * p.n_max + 4 * p.n_harm + 192 +
                      3 * (size_t)p.n_max * p.n_harm);
  if (lim > 200 * 1024) {
    set_error("stored-gradient form needs %zu bytes of shared memory", lim);
    return FGB_EINVAL;
  }
  // dA and A of a pair: 4 pairs a block while that leaves room for four
  // blocks on an SM, else one
  const size_t per = sizeof(double) * (3 * (size_t)p.n_max + p.n_rad) *
                     (p.n_harm | 1);
  const int PP = 4 * per <= 48 * 1024 ? 4 : 1;
  const int npair = p.n_rad * (p.n_rad + 1) / 2;
  const size_t nbasis = (size_t)(2 * p.n_max + 4 * p.n_harm) * (size_t)P;
  int rc;
  if ((rc = center.ensure(sizeof(int) * P)) ||
      (rc = basis.ensure(sizeof(double) * nbasis +
                         sizeof(int) * (size_t)p.n_species * npair)))
    return rc;
  int *tab = reinterpret_cast<int *>(basis.as<double>() + nbasis);
  k_pair_center<<<ceil_div((long long)N * 32, 128), 128, 0, st>>>(
      N, nl->offsets.as<long long>(), center.as<int>());
  FGB_LAUNCH_CHECK("k_pair_center");
  k_derv_items<<<p.n_species, 128, 0, st>>>(p.n_rad, p.n_max, npair, tab);
  FGB_LAUNCH_CHECK("k_derv_items");
  // threads: whole warps, the block's items split evenly over the fewest
  // passes
  const int items = PP * npair, passes = ceil_div(items, kDTmax);
  const int nt = 32 * ceil_div(ceil_div(items, passes), 32);
  const auto run = [&](auto pp, auto lc) -> int {
    constexpr int K = decltype(pp)::value, LC = decltype(lc)::value;
    k_pair_basis<LC><<<ceil_div(P, kBT), kBT, 0, st>>>(
        p, P, center.as<int>(), nl->nbr_j.as<int>(),
        nl->nbr_rel.as<double4_16a>(), d_species, basis.as<double>());
    FGB_LAUNCH_CHECK("k_pair_basis");
    FGB_CUDA(cudaFuncSetAttribute(k_b2_dervs<K, LC>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(K * per)));
    k_b2_dervs<K, LC><<<ceil_div(P, K), nt, K * per, st>>>(
        p, P, center.as<int>(), nl->nbr_j.as<int>(),
        nl->nbr_rel.as<double4_16a>(), d_species, basis.as<double>(), tab,
        npair, d_A, d_dB2);
    FGB_LAUNCH_CHECK("k_b2_dervs");
    return FGB_OK;
  };
  const auto with_l = [&](auto pp) -> int {
    switch (p.l_max) {
      case 1: return run(pp, std::integral_constant<int, 1>());
      case 2: return run(pp, std::integral_constant<int, 2>());
      case 3: return run(pp, std::integral_constant<int, 3>());
      case 4: return run(pp, std::integral_constant<int, 4>());
      default: return run(pp, std::integral_constant<int, 0>());
    }
  };
  if ((rc = PP == 4 ? with_l(std::integral_constant<int, 4>())
                    : with_l(std::integral_constant<int, 1>())))
    return rc;
  k_row_dots<<<ceil_div(3 * P * 32, 256), 256, 0, st>>>(
      3 * P, p.n_d, center.as<int>(), d_dB2, d_B2, d_force_dots, d_rowmax);
  FGB_LAUNCH_CHECK("k_row_dots");
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
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
    cudaGetLastError();
    cs = cudaStreamCaptureStatusActive;   // unknown: allocate nothing
  }
  if (cs == cudaStreamCaptureStatusNone) {
    const int rc = envs_envs_sliced(d_desc1, d_norm1, n1, d_desc2, d_norm2, n2,
                                    n_desc, sig2, power, d_kern, st);
    if (rc != FGB_ENOMEM) return rc;
  }
  // a call being captured, whose graph then holds no allocation, or without
  // room for the slices
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
// envs_struc for one structure, transposed: d_kt [(1 + 3N + 6) x M]; B2,
// norms and stored gradients of the structure are left in ws.  The dots with
// the sparse rows are exact kS64-slice products (ozaki.cu), whose epilogues
// write the cosines and the force-kernel values.
int envs_struc_impl(const B2Params &p, double sigma, double power,
                    const int *h_counts, const double *d_sparse,
                    fgb_nlist_s *nl, const int *d_species, double *d_kt,
                    fgb_workspace &ws, cudaStream_t st) {
  if (nl->n_struc != 1) {
    set_error("envs_struc needs a single-structure neighbour list");
    return FGB_EINVAL;
  }
  const int N = nl->n_atoms, S = p.n_species, nd = p.n_d;
  const long long P = nl->n_pairs;
  int rc;
  SparseOffsets so;
  so.n = S;
  so.o[0] = 0;
  for (int s = 0; s < S; s++) so.o[s + 1] = so.o[s] + h_counts[s];
  const int M = so.o[S];
  const long long ncol = 1 + 3LL * N + 6;
  if ((rc = ws.ozerr.ensure(sizeof(int)))) return rc;
  FGB_CUDA(cudaMemsetAsync(ws.ozerr.p, 0, sizeof(int), st));
  if (M == 0) return check_species(d_species, N, S, ws.flag, st);
  if (N == 0) {
    FGB_CUDA(cudaMemsetAsync(d_kt, 0, sizeof(double) * M * ncol, st));
    return FGB_OK;
  }
  std::vector<int> counts;
  bool pending = false;
  if ((rc = species_permutation_start(S, ws, d_species, N, counts, st, nullptr,
                                      pending)) ||
      (rc = ws.start.ensure(sizeof(int) * (2 * (size_t)N + S + 1))) ||
      (rc = ws.rows.ensure(sizeof(int) * (3 * (size_t)P + 1))) ||
      (rc = ws.A.ensure(sizeof(double) * ((size_t)N * p.n_A + 1))) ||
      (rc = ws.B2.ensure(sizeof(double) * ((size_t)N * nd + 1))) ||
      (rc = ws.norms.ensure(sizeof(double) * (N + 1))) ||
      (rc = ws.rowmax.ensure(sizeof(double) * (N + 1))) ||
      (rc = ws.dB2.ensure(sizeof(double) * ((size_t)3 * P * nd + 1))) ||
      (rc = ws.fdots.ensure(sizeof(double) * (6 * P + 1))) ||
      (rc = ws.kern.ensure(sizeof(double) * ((size_t)3 * P * M + 1))) ||
      (rc = ws.snorm.ensure(sizeof(double) * (3 * (size_t)M + 1))))
    return rc;
  double *snorm = ws.snorm.as<double>();
  double2 *sinv = reinterpret_cast<double2 *>(snorm + M + (M & 1));
  // the forward takes any species value; a species out of range is found
  // next, before anything is indexed by it
  if ((rc = launch_b2_forward(p, nl, d_species, ws.A.as<double>(),
                              ws.B2.as<double>(), ws.norms.as<double>(), st,
                              false, ws.rowmax.as<double>())) ||
      (rc = oz::row_inverse(M, nd, d_sparse, snorm, sinv, st)) ||
      (pending && (rc = species_permutation_finish(S, ws, counts))))
    return rc;
  const long long *off = nl->offsets.as<long long>();
  const int *perm = ws.perm.as<int>();
  int *start = ws.start.as<int>(), *inv = start + N, *dsp = inv + N;
  k_group_scan<<<1, 1024, 0, st>>>(N, perm, d_species, off, S, start, inv, dsp);
  FGB_LAUNCH_CHECK("k_group_scan");
  int *spairs = ws.counts.h + kMaxSpecies + 1;
  FGB_CUDA(cudaMemcpyAsync(spairs, dsp, sizeof(int) * (S + 1),
                           cudaMemcpyDeviceToHost, st));
  if ((rc = ws.counts.queued(st))) return rc;
  k_group_rows<<<ceil_div((long long)N * 32, 128), 128, 0, st>>>(
      N, perm, off, start, ws.rows.as<int>());
  FGB_LAUNCH_CHECK("k_group_rows");
  if ((rc = launch_b2_dervs(p, nl, d_species, ws.A.as<double>(),
                            ws.B2.as<double>(), ws.dB2.as<double>(),
                            ws.fdots.as<double>(), ws.pos, ws.basis, st,
                            ws.fdots.as<double>() + 3 * P)))
    return rc;
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
  if ((rc = ws.counts.wait())) return rc;
  constexpr int kRows = 65536;   // gradient rows sliced at a time
  int base = 0;
  for (int s = 0; s < S; s++) {
    const int Ns = counts[s], Ms = h_counts[s], k0 = base;
    base += Ns;
    if (Ns == 0 || Ms == 0) continue;
    const int *perm_s = perm + k0;
    const int R = 3 * (spairs[s + 1] - spairs[s]);
    const int vc = oz::tile64(Ns, Ms);
    const int vf = oz::tile64(std::min(std::max(R, 1), kRows), Ms);
    for (int v = 0; v < oz::kTiles64; v++)
      if ((v == vc || (v == vf && R > 0)) &&
          (rc = oz::slice({Ms, nd, oz::kTN64v[v],
                           d_sparse + (size_t)so.o[s] * nd, nd, nullptr,
                           nullptr},
                          ws.ozSp[v], st, oz::kS64)))
        return rc;
    if ((rc = ws.dots.ensure(sizeof(double) * (size_t)Ns * Ms)) ||
        (rc = oz::slice({Ns, nd, oz::kTM, ws.B2.as<double>(), nd, perm_s,
                         nullptr, ws.rowmax.as<double>()},
                        ws.ozA, st, oz::kS64)) ||
        (rc = oz::gemm_cosine(ws.ozA, ws.ozSp[vc], perm_s,
                              ws.norms.as<double>(), sinv + so.o[s],
                              snorm + so.o[s], ws.dots.as<double>(),
                              ws.ozerr.as<int>(), st)))
      return rc;
    k_energy_part<<<dim3(ceil_div(Ms, kColRows), ceil_div(Ns, eper)),
                    kColRows * kColGroups, 0, st>>>(
        Ns, Ms, eper, ws.dots.as<double>(), perm_s, ws.norms.as<double>(),
        snorm + so.o[s], sig2, power, ws.part.as<double>() + so.o[s], M);
    FGB_LAUNCH_CHECK("k_energy_part");
    for (int r0 = 0; r0 < R; r0 += kRows) {
      const int Rc = std::min(kRows, R - r0);
      const int *rows = ws.rows.as<int>() + 3LL * spairs[s] + r0;
      oz::ForceKernelArgs fk;
      fk.rows = rows;
      fk.center = ws.pos.as<int>();
      fk.crow = inv;
      fk.crow0 = k0;   // inv is the place among all species
      fk.cosine = ws.dots.as<double>();
      fk.d_norm = ws.norms.as<double>();
      fk.fdots = ws.fdots.as<double>();
      fk.s_norm = snorm + so.o[s];
      fk.s_inv = sinv + so.o[s];
      fk.sig2 = sig2;
      fk.power = power;
      fk.FK = ws.kern.as<double>();
      fk.c_s = so.o[s];
      fk.M = M;
      if ((rc = oz::slice({Rc, nd, oz::kTM, ws.dB2.as<double>(), nd, rows,
                           nullptr, ws.fdots.as<double>() + 3 * P},
                          ws.ozK, st, oz::kS64)) ||
          (rc = oz::gemm_force_kernel(ws.ozK, ws.ozSp[vf], fk,
                                      ws.ozerr.as<int>(), st)))
        return rc;
    }
  }
  k_force_cols<<<dim3(N, ceil_div(M, kColRows)), kColRows * kColGroups, 0,
                 st>>>(
      M, N, so, off, nl->nbr_j.as<int>(), nl->nbr_twin.as<long long>(),
      d_species, ws.kern.as<double>(), d_kt);
  FGB_LAUNCH_CHECK("k_force_cols");
  if (P > 0) {
    k_stress_part<<<dim3(ceil_div(M, kColRows), ncs), kColRows * kColGroups, 0,
                    st>>>(M, P, sper, so, nl->nbr_rel.as<double4_16a>(),
                          ws.pos.as<int>(), d_species, ws.kern.as<double>(),
                          spart);
    FGB_LAUNCH_CHECK("k_stress_part");
  }
  k_col_final<<<dim3(ceil_div(M, kColRows), 7), kColRows * kColGroups, 0, st>>>(
      M, nce, ncs, ws.part.as<double>(), spart, 1.0 / nl->h_volume[0], N, d_kt);
  FGB_LAUNCH_CHECK("k_col_final");
  return FGB_OK;
}

// The tensor-core time-out flag of the products above, after the stream's
// work (synchronises).
int sliced_finish(fgb_workspace &ws, cudaStream_t st, const char *what) {
  int h = 0;
  if (ws.ozerr.p)
    FGB_CUDA(cudaMemcpyAsync(&h, ws.ozerr.p, sizeof(int),
                             cudaMemcpyDeviceToHost, st));
  FGB_CUDA(cudaStreamSynchronize(st));
  if (h) {
    set_error("%s: a bounded device wait ran out", what);
    return FGB_ETIMEOUT;
  }
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
  cudaStream_t st = (cudaStream_t)stream;
  fgb_workspace ws;
  ws.scratch_on(st);
  long long M = 0;
  for (int s = 0; s < b2->p.n_species; s++) M += h_counts[s];
  const long long ncol = 1 + 3LL * nl->n_atoms + 6;
  DevBuf kt(st);
  int rc;
  if ((rc = kt.ensure(sizeof(double) * ((size_t)M * ncol + 1))) ||
      (rc = envs_struc_impl(b2->p, sigma, power, h_counts, d_sparse, nl,
                            d_species, kt.as<double>(), ws, st)))
    return rc;
  if (M > 0) {
    k_transpose32<<<dim3(ceil_div(ncol, 32), ceil_div(M, 32)), dim3(32, 8), 0,
                    st>>>(ncol, (int)M, kt.as<double>(), d_kern);
    FGB_LAUNCH_CHECK("k_transpose32");
  }
  return sliced_finish(ws, st, "envs_struc");
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
  DevBuf kt(st);
  if ((rc = kt.ensure(sizeof(double) * ((size_t)M * ncol + 1)))) return rc;
  if ((rc = envs_struc_impl(m->b2, m->sigma, m->power, m->h_counts.data(),
                            m->Sraw.as<double>(), nl, d_species,
                            kt.as<double>(), m->ws, st)) ||
      (rc = launch_kt_alpha(M, ncol, kt.as<double>(), m->alpha.as<double>(),
                            d_mean_efs, st)))
    return rc;
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
  return sliced_finish(m->ws, st, "fgb_predict_plain");
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
  DevBuf L(st), At(st), b(st), Qtb(st), Rinv(st);
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
  if ((rc = dense::cholesky_inverse(M, L.as<double>(), d_L_inv, st)) ||
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
