// The device-resident model and the fgb_predict pipeline, and K3/K4 (kernel
// against the sparse set, adjoint GEMM and local variance) as FP64 SIMT
// kernels: for powers other than 1 and 2 and for non-finite weights.  The
// others take the exact-slice products of ozaki.cu.
//
// For the atoms of species s (rows gathered through a species permutation):
//   GEMM1 (NT)  C = B2_s S^_s^T;  epilogue c = C/|d|, k = sigma^2 c^xi,
//               w = sigma^2 xi alpha c^(xi-1)   (normalized_dot_product.cpp:171-181)
//   E_i = sum_t alpha_t k_it                     (sparse_gp.cpp:751 mean = K^T alpha)
//   GEMM2 (NN)  G = W S^_s;  epilogue dE/dB2 = (G - xi E d^)/|d|
//   GEMM3 (NT, lower-triangular)  Z = K L_s^T;  epilogue row sums of Z^2
//   var_i = k_self - sum_r Z_ir^2                (sparse_gp.cpp:116-133)
// L_inv of a single-kernel model is block-diagonal by species (cross-species
// Kuu blocks are exactly zero), so species s only needs its panel of L_inv.
#include <cstring>
#include <vector>

#include "fgb_internal.h"
#include "fgb_kernels.h"
#include "fgb_model.h"
#include "fgb_gemm64.cuh"
#include "fgb_profile.h"

namespace fgb {

namespace {

constexpr int kRowChunk = 32768;
using namespace gemm64;

// GEMM1: rows = atoms of one species (through perm), cols = sparse envs.
__global__ void __launch_bounds__(GT)
k_kernel_gemm(int M, int N, int K, const double *__restrict__ B2,
              const int *__restrict__ perm, const double *__restrict__ norms,
              const double *__restrict__ S, const double *__restrict__ alpha,
              const unsigned char *__restrict__ svalid, double sig2, double xi,
              double *__restrict__ Kmat, double *__restrict__ Wmat) {
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  double acc[4][4];
  gemm_mainloop<true>(acc, m0, n0, M, N, K, B2, K, perm, S, K);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    int m = m0 + ty + 16 * i;
    if (m >= M) continue;
    double nd = norms[perm[m]];
    bool dok = nd >= kEmptyThresh;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int n = n0 + tx + 16 * j;
      if (n >= N) continue;
      double kv = 0.0, wv = 0.0;
      if (dok && svalid[n]) {
        double c = acc[i][j] / nd;
        kv = sig2 * powx(c, xi);
        wv = sig2 * xi * powx(c, xi - 1.0) * alpha[n];
      }
      Kmat[(long long)m * N + n] = kv;
      Wmat[(long long)m * N + n] = wv;
    }
  }
}

// E_m = sum_n alpha_n K[m][n]: warp per row, fixed-order shuffle tree.
__global__ void k_row_energy(int M, int N, const double *__restrict__ Kmat,
                             const double *__restrict__ alpha,
                             const int *__restrict__ perm,
                             double *__restrict__ e_rows,
                             double *__restrict__ e_atom) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (warp >= M) return;
  const double *row = Kmat + (long long)warp * N;
  double acc = 0.0;
  for (int n = lane; n < N; n += 32) acc += alpha[n] * row[n];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
    acc += __shfl_down_sync(0xffffffffu, acc, off);
  if (lane == 0) {
    e_rows[warp] = acc;
    if (e_atom) e_atom[perm[warp]] = acc;
  }
}

// GEMM2: G = W S (NN); epilogue dE/dB2 rows in atom order.
__global__ void __launch_bounds__(GT)
k_adjoint_gemm(int M, int N, int K, const double *__restrict__ Wmat,
               const double *__restrict__ S, const int *__restrict__ perm,
               const double *__restrict__ norms, const double *__restrict__ B2,
               const double *__restrict__ e_rows, double xi,
               double *__restrict__ gB2) {
  // M rows (atoms), N = n_d columns, K = M_s
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  double acc[4][4];
  gemm_mainloop<false>(acc, m0, n0, M, N, K, Wmat, K, nullptr, S, N);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    int m = m0 + ty + 16 * i;
    if (m >= M) continue;
    int atom = perm[m];
    double nd = norms[atom];
    bool dok = nd >= kEmptyThresh;
    double inv = dok ? 1.0 / nd : 0.0;
    double xe = xi * e_rows[m];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int n = n0 + tx + 16 * j;
      if (n >= N) continue;
      double v = 0.0;
      if (dok) {
        double dh = B2[(long long)atom * N + n] * inv;
        v = (acc[i][j] - xe * dh) * inv;
      }
      gB2[(long long)atom * N + n] = v;
    }
  }
}

// GEMM3: Z = K L^T over the lower-triangular panel; row sums of Z^2 per
// column tile.
__global__ void __launch_bounds__(GT)
k_variance_gemm(int M, int R, int Ms, const double *__restrict__ Kmat,
                const double *__restrict__ Lp, double *__restrict__ part,
                int ntiles) {
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int kmax = min(Ms, n0 + BN);
  double acc[4][4];
  gemm_mainloop<true>(acc, m0, n0, M, R, kmax, Kmat, Ms, nullptr, Lp, Ms);
  __shared__ double red[16][BM + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int n = n0 + tx + 16 * j;
      if (n < R) s += acc[i][j] * acc[i][j];
    }
    red[tx][ty + 16 * i] = s;
  }
  __syncthreads();
  if (threadIdx.x < BM) {
    int mm = threadIdx.x;
    double s = 0.0;
    for (int q = 0; q < 16; q++) s += red[q][mm];
    int m = m0 + mm;
    if (m < M) part[(long long)m * ntiles + blockIdx.x] = s;
  }
}

__global__ void k_variance_final(int M, int ntiles, const double *__restrict__ part,
                                 const int *__restrict__ perm,
                                 const double *__restrict__ norms, double sig2,
                                 double xi, double scale,
                                 double *__restrict__ var) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int m = (int)(gt / kRowLanes), q = (int)(gt % kRowLanes);
  if (m >= M) return;   // whole lane groups
  const double s = row_slots_sum(part, m, ntiles, q);
  if (q) return;
  int atom = perm[m];
  double nd = norms[atom];
  // K_self = sig^2 (d.d/(|d||d|))^xi, zero for an empty environment.
  double kself = nd >= kEmptyThresh ? sig2 * powx((nd * nd) / (nd * nd), xi)
                                    : 0.0;
  var[atom] = kself - s * scale;
}

// The kernel matrix and GEMM3 above for models of few sparse environments
// (small_variance), a thread an element, the same operations in the same
// order: the same bits.  8 x 16 elements a block, four warps, which the FP64
// unit of an SM serves in the 64 cycles of one instruction.
constexpr int kSmT = 128, kSmR = 8, kSmC = 16, kSmK = 48;
__global__ void __launch_bounds__(kSmT)
k_kernel_small(int M, int N, int K, const double *__restrict__ B2,
               const int *__restrict__ perm, const double *__restrict__ norms,
               const double *__restrict__ S,
               const unsigned char *__restrict__ svalid, double sig2, double xi,
               double *__restrict__ Kmat) {
  __shared__ double As[kSmR][kSmK + 1], Bs[kSmC][kSmK + 1];
  const int t = threadIdx.x, r = t / kSmC, c = t % kSmC;
  const int m0 = blockIdx.y * kSmR, n0 = blockIdx.x * kSmC;
  const int m = m0 + r, n = n0 + c;
  double acc = 0.0;
  for (int k0 = 0; k0 < K; k0 += kSmK) {
    const int kc = min(kSmK, K - k0);
    for (int e = t; e < (kSmR + kSmC) * kSmK; e += kSmT) {
      const int row = e / kSmK, k = e % kSmK;
      double v = 0.0;
      if (row < kSmR) {
        if (m0 + row < M && k < kc)
          v = B2[(long long)perm[m0 + row] * K + k0 + k];
        As[row][k] = v;
      } else {
        if (n0 + row - kSmR < N && k < kc)
          v = S[(long long)(n0 + row - kSmR) * K + k0 + k];
        Bs[row - kSmR][k] = v;
      }
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < kc; k++) acc = fma(As[r][k], Bs[c][k], acc);
    __syncthreads();
  }
  if (m >= M || n >= N) return;
  const double nd = norms[perm[m]];
  double kv = 0.0;
  if (nd >= kEmptyThresh && svalid[n]) {
    const double x = acc / nd;
    kv = sig2 * powx(x, xi);
  }
  Kmat[(long long)m * N + n] = kv;
}
// Two rows and BN columns a block.
__global__ void __launch_bounds__(kSmT)
k_variance_small(int M, int R, int Ms, const double *__restrict__ Kmat,
                 const double *__restrict__ Lp, double *__restrict__ part,
                 int ntiles) {
  static_assert(kSmT == 2 * BN, "two rows of a column tile");
  __shared__ double Ks[2][32], Ls[BN][33], red[2][BN];
  const int t = threadIdx.x, r = t / BN, c = t % BN;
  const int m0 = blockIdx.y * 2, n0 = blockIdx.x * BN;
  const int kmax = min(Ms, n0 + BN);
  double acc = 0.0;
  for (int k0 = 0; k0 < kmax; k0 += 32) {
    const int kc = min(32, kmax - k0);
    if (t < 64) {
      const int row = t / 32, k = t % 32;
      Ks[row][k] = m0 + row < M && k < kc
                       ? Kmat[(long long)(m0 + row) * Ms + k0 + k] : 0.0;
    }
    for (int e = t; e < BN * 32; e += kSmT) {
      const int row = e / 32, k = e % 32;
      Ls[row][k] = n0 + row < R && k < kc
                       ? Lp[(long long)(n0 + row) * Ms + k0 + k] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < kc; k++) acc = fma(Ks[r][k], Ls[c][k], acc);
    __syncthreads();
  }
  red[r][c] = acc;
  __syncthreads();
  double s = 0.0;
  if (c < 16)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const double z = red[r][c + 16 * j];
      if (n0 + c + 16 * j < R) s += z * z;
    }
  __syncthreads();
  if (c < 16) red[r][c] = s;
  __syncthreads();
  if (c == 0 && m0 + r < M) {
    double v = 0.0;
    for (int q = 0; q < 16; q++) v += red[r][q];
    part[(long long)(m0 + r) * ntiles + blockIdx.x] = v;
  }
}

// out[m] = sum of the row's partial slots (fixed order, row_slots_sum)
__global__ void k_sum_parts(int M, int nslots, const double *__restrict__ part,
                            double *__restrict__ out) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int m = (int)(gt / kRowLanes), q = (int)(gt % kRowLanes);
  if (m >= M) return;   // whole lane groups
  const double s = row_slots_sum(part, m, nslots, q);
  if (q == 0) out[m] = s;
}

// variance_efs = K_self - Q_self + V_SOR (sparse_gp.cpp:726)
__global__ void k_dtc_combine(long long n, const double *__restrict__ kself,
                              const double *__restrict__ q,
                              double *__restrict__ v) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = kself[i] - q[i] + v[i];
}

// out[o] = K^T row o . alpha: a warp per output.  The terms cancel (|alpha|
// up to 1e6 against energies of eV), so products and sums keep their errors
// in a second word.
__global__ void k_kt_alpha(int M, long long ncol, const double *__restrict__ KT,
                           const double *__restrict__ alpha,
                           double *__restrict__ out) {
  const long long o = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (o >= ncol) return;
  double acc = 0.0, err = 0.0;
  const auto add = [&](double b, double b_err) {
    const double s = __dadd_rn(acc, b), bb = __dadd_rn(s, -acc);
    const double e = __dadd_rn(__dadd_rn(acc, -__dadd_rn(s, -bb)),
                               __dadd_rn(b, -bb));
    acc = s;
    err = __dadd_rn(err, __dadd_rn(e, b_err));
  };
  for (int i = lane; i < M; i += 32) {
    const double x = KT[o * M + i], a = alpha[i], p = __dmul_rn(x, a);
    add(p, __fma_rn(x, a, -p));
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double b = __shfl_down_sync(0xffffffffu, acc, off);
    const double b_err = __shfl_down_sync(0xffffffffu, err, off);
    add(b, b_err);
  }
  if (lane == 0) out[o] = acc + err;
}

__global__ void k_check_species(int n, const int *__restrict__ species, int ns,
                                int *__restrict__ flag) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && (species[i] < 0 || species[i] >= ns)) atomicExch(flag, 1);
}

// Species permutation as a counting sort over blocks of kPermBlock atoms
// (n_species <= kMaxSpecies): per-block histograms, one block of offsets,
// then a stable scatter (atoms of a species keep their index order).
constexpr int kPermBlock = 1024;

// hist[s * nb + b] = atoms of species s in block b; flag: a species out of
// [0, ns)
__global__ void __launch_bounds__(kPermBlock)
k_species_hist(int n, const int *__restrict__ species, int ns,
               int *__restrict__ hist, int *__restrict__ flag) {
  __shared__ int cnt[kMaxSpecies];
  const int t = threadIdx.x, b = blockIdx.x, nb = gridDim.x;
  if (t < kMaxSpecies) cnt[t] = 0;
  __syncthreads();
  const int i = b * kPermBlock + t;
  if (i < n) {
    const int sp = species[i];
    if (sp < 0 || sp >= ns) atomicExch(flag, 1);
    else atomicAdd(&cnt[sp], 1);
  }
  __syncthreads();
  if (t < ns) hist[t * nb + b] = cnt[t];
}

// In place: hist becomes the exclusive prefix over (species, block) in
// species-major order, i.e. the first perm slot of each (species, block);
// totals[s] = atoms of species s.  One block; each thread scans a
// contiguous run, then the runs' sums are scanned (by warps: one thread that
// added the 1,024 sums made this kernel 6.8 us).
__global__ void __launch_bounds__(kPermBlock)
k_species_offsets(int nb, int ns, int *__restrict__ hist,
                  int *__restrict__ totals) {
  __shared__ int wsum[32];
  __shared__ int grand;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, L = ns * nb;
  const int per = (L + kPermBlock - 1) / kPermBlock;
  const int lo = min(L, t * per), hi = min(L, lo + per);
  int sum = 0;
  for (int k = lo; k < hi; k++) sum += hist[k];
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  int before = 0;
  for (int q = 0; q < w; q++) before += wsum[q];
  if (t == kPermBlock - 1) grand = before + x;
  int acc = before + x - sum;
  for (int k = lo; k < hi; k++) {
    const int v = hist[k];
    hist[k] = acc;
    acc += v;
  }
  __syncthreads();
  if (t < ns) totals[t] = (t + 1 < ns ? hist[(t + 1) * nb] : grand) - hist[t * nb];
}

// The three kernels' work in one block, for up to kPermOne atoms (three
// launches of 1.5 to 7 us against one of 2.9 at 256 atoms, 7.8 at 5,500).  Rounds of kPermBlock atoms:
// per species, the atoms of earlier warps and rounds come first.
constexpr int kPermOne = 8 * kPermBlock;
__global__ void __launch_bounds__(kPermBlock)
k_species_perm_one(int n, const int *__restrict__ species, int ns,
                   int *__restrict__ perm, int *__restrict__ totals,
                   int *__restrict__ flag) {
  __shared__ int wc[kPermBlock / 32][kMaxSpecies];
  __shared__ int cnt[kMaxSpecies], first[kMaxSpecies];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  if (t < kMaxSpecies) cnt[t] = 0;
  __syncthreads();
  bool bad = false;
  for (int i = t; i < n; i += kPermBlock) {
    const int sp = species[i];
    if (sp < 0 || sp >= ns) bad = true;
    else atomicAdd(&cnt[sp], 1);
  }
  const int any_bad = __syncthreads_or(bad);
  if (t == 0) {
    int acc = 0;
    for (int s = 0; s < ns; s++) {
      first[s] = acc;
      acc += cnt[s];
      totals[s] = cnt[s];
    }
    *flag = any_bad ? 1 : 0;
  }
  __syncthreads();
  for (int i0 = 0; i0 < n; i0 += kPermBlock) {
    const int i = i0 + t;
    int sp = i < n ? species[i] : -1;
    if (sp >= ns || sp < 0) sp = -1;
    const unsigned same = __match_any_sync(0xffffffffu, sp);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (lane < kMaxSpecies) wc[w][lane] = 0;
    __syncwarp();
    if (sp >= 0 && rank == 0) wc[w][sp] = __popc(same);
    __syncthreads();
    if (sp >= 0) {
      int before = first[sp];
      for (int q = 0; q < w; q++) before += wc[q][sp];
      perm[before + rank] = i;
    }
    __syncthreads();
    if (t < ns)
      for (int q = 0; q < kPermBlock / 32; q++) first[t] += wc[q][t];
    __syncthreads();
  }
}

// perm[first(s, b) + rank of atom i among block b's species-s atoms] = i
__global__ void __launch_bounds__(kPermBlock)
k_species_scatter(int n, const int *__restrict__ species, int ns,
                  const int *__restrict__ first, int *__restrict__ perm) {
  __shared__ int wc[kPermBlock / 32][kMaxSpecies];   // per-warp counts
  const int t = threadIdx.x, b = blockIdx.x, nb = gridDim.x;
  const int w = t >> 5, lane = t & 31;
  const int i = b * kPermBlock + t;
  int sp = i < n ? species[i] : -1;
  if (sp >= ns) sp = -1;
  const unsigned same = __match_any_sync(0xffffffffu, sp);
  const int rank = __popc(same & ((1u << lane) - 1u));
  if (lane < kMaxSpecies) wc[w][lane] = 0;
  __syncwarp();
  if (sp >= 0 && rank == 0) wc[w][sp] = __popc(same);
  __syncthreads();
  if (sp >= 0) {
    int before = 0;
    for (int q = 0; q < w; q++) before += wc[q][sp];
    perm[first[sp * nb + b] + before + rank] = i;
  }
}

}  // namespace

int launch_kt_alpha(int M, long long ncol, const double *KT,
                    const double *alpha, double *out, cudaStream_t st) {
  k_kt_alpha<<<ceil_div(ncol * 32, 128), 128, 0, st>>>(M, ncol, KT, alpha, out);
  FGB_LAUNCH_CHECK("k_kt_alpha");
  return FGB_OK;
}

// Local variances of Mr rows of species s by k_kernel_small and
// k_variance_small, from ws.B2 and ws.norms.
int variance_small(fgb_model_s *m, int s, int Mr, const int *perm,
                   double *d_var, cudaStream_t st) {
  const int Ms = m->h_counts[s], R = m->h_panel_rows[s], nd = m->b2.n_d;
  const int off = m->h_offsets[s], nt = ceil_div(R, BN);
  const double sig2 = m->sigma * m->sigma;
  int rc;
  if ((rc = m->ws.kmat.ensure(sizeof(double) * (size_t)Mr * Ms)) ||
      (rc = m->ws.vpart.ensure(sizeof(double) * (size_t)Mr * nt)))
    return rc;
  {
    StageTimer _pt(kStVarianceGemm, st, 2);
    k_kernel_small<<<dim3(ceil_div(Ms, kSmC), ceil_div(Mr, kSmR)), kSmT, 0,
                     st>>>(Mr, Ms, nd, m->ws.B2.as<double>(), perm,
                           m->ws.norms.as<double>(),
                           m->S.as<double>() + (size_t)off * nd,
                           m->svalid.as<unsigned char>() + off, sig2, m->power,
                           m->ws.kmat.as<double>());
    FGB_LAUNCH_CHECK("k_kernel_small");
    k_variance_small<<<dim3(nt, ceil_div(Mr, 2)), kSmT, 0, st>>>(
        Mr, R, Ms, m->ws.kmat.as<double>(),
        m->Lp.as<double>() + m->h_panel_off[s], m->ws.vpart.as<double>(), nt);
    FGB_LAUNCH_CHECK("k_variance_small");
  }
  return launch_variance_final(Mr, nt, m->ws.vpart.as<double>(), perm,
                               m->ws.norms.as<double>(), sig2, m->power, d_var,
                               st);
}

int launch_variance_final(int Mr, int ntiles, const double *part,
                          const int *perm, const double *norms, double sig2,
                          double xi, double *var, cudaStream_t st,
                          double scale) {
  StageTimer _pt(kStVarianceFinal, st);
  k_variance_final<<<
      ceil_div((long long)Mr * kRowLanes, 128), 128, 0, st>>>(
      Mr, ntiles, part, perm, norms, sig2, xi, scale, var);
  FGB_LAUNCH_CHECK("k_variance_final");
  return FGB_OK;
}

int check_species(const int *d_species, int n, int n_species, DevBuf &flag,
                  cudaStream_t st) {
  if (n == 0) return FGB_OK;
  int rc = flag.ensure(sizeof(int));
  if (rc) return rc;
  FGB_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
  k_check_species<<<ceil_div(n, 256), 256, 0, st>>>(n, d_species, n_species,
                                                    flag.as<int>());
  FGB_LAUNCH_CHECK("k_check_species");
  int h = 0;
  FGB_CUDA(cudaMemcpyAsync(&h, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  FGB_CUDA(cudaStreamSynchronize(st));
  if (h) {
    set_error("species must lie in [0, %d)", n_species);
    return FGB_EINVAL;
  }
  return FGB_OK;
}

// Species permutation: perm = atoms of species 0 (ascending), then 1, ...
// The species range check and every species count come back to the host in
// one read (a single wait).
int species_permutation(fgb_model_s *m, const int *d_species, int N,
                        std::vector<int> &counts, cudaStream_t st,
                        const int *h_species) {
  return species_permutation(m->b2.n_species, m->ws, d_species, N, counts, st,
                             h_species);
}

int species_permutation(int S, fgb_workspace &ws, const int *d_species, int N,
                        std::vector<int> &counts, cudaStream_t st,
                        const int *h_species) {
  bool pending = false;
  int rc = species_permutation_start(S, ws, d_species, N, counts, st,
                                     h_species, pending);
  if (rc || !pending) return rc;
  return species_permutation_finish(S, ws, counts);
}

int species_permutation_start(int S, fgb_workspace &ws, const int *d_species,
                              int N, std::vector<int> &counts, cudaStream_t st,
                              const int *h_species, bool &pending) {
  pending = false;
  counts.assign(S, 0);
  if (S < 1 || S > kMaxSpecies) {
    set_error("species permutation: %d species (at most %d)", S, kMaxSpecies);
    return FGB_EINVAL;
  }
  if (h_species) {
    for (int i = 0; i < N; i++) {
      const int q = h_species[i];
      if (q < 0 || q >= S) {
        set_error("species must lie in [0, %d)", S);
        return FGB_EINVAL;
      }
      counts[q]++;
    }
  }
  const int nb = ceil_div(std::max(N, 1), kPermBlock);
  int rc;
  if ((rc = ws.perm.ensure(sizeof(int) * (N + 1))) ||
      (rc = ws.flags.ensure(sizeof(int) * ((size_t)S * nb + 1))) ||
      (rc = ws.scal.ensure(sizeof(int) * (S + 2))))
    return rc;
  if (N == 0) return FGB_OK;
  int *tot = ws.scal.as<int>();   // [0, S): counts; [S]: range flag
  int *hist = ws.flags.as<int>();
  if (N <= kPermOne) {
    k_species_perm_one<<<1, kPermBlock, 0, st>>>(N, d_species, S,
                                                 ws.perm.as<int>(), tot,
                                                 tot + S);
    FGB_LAUNCH_CHECK("k_species_perm_one");
  } else {
    FGB_CUDA(cudaMemsetAsync(tot + S, 0, sizeof(int), st));
    k_species_hist<<<nb, kPermBlock, 0, st>>>(N, d_species, S, hist, tot + S);
    FGB_LAUNCH_CHECK("k_species_hist");
    k_species_offsets<<<1, kPermBlock, 0, st>>>(nb, S, hist, tot);
    FGB_LAUNCH_CHECK("k_species_offsets");
    k_species_scatter<<<nb, kPermBlock, 0, st>>>(N, d_species, S, hist,
                                                 ws.perm.as<int>());
    FGB_LAUNCH_CHECK("k_species_scatter");
  }
  if (h_species) return FGB_OK;   // counted and checked above
  fgb_pinned_counts &pc = ws.counts;
  if (!pc.h && pc.pageable) pc.h = pc.host;
  if (!pc.h)
    FGB_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&pc.h),
                           sizeof(int) * fgb_pinned_counts::kInts,
                           cudaHostAllocDefault));
  if (!pc.ev && !pc.pageable)
    FGB_CUDA(cudaEventCreateWithFlags(&pc.ev, cudaEventDisableTiming));
  FGB_CUDA(cudaMemcpyAsync(pc.h, tot, sizeof(int) * (S + 1),
                           cudaMemcpyDeviceToHost, st));
  if ((rc = pc.queued(st))) return rc;
  pending = true;
  return FGB_OK;
}

int species_permutation_finish(int S, fgb_workspace &ws,
                               std::vector<int> &counts) {
  const fgb_pinned_counts &pc = ws.counts;
  const int rc = pc.wait();
  if (rc) return rc;
  if (pc.h[S]) {
    set_error("species must lie in [0, %d)", S);
    return FGB_EINVAL;
  }
  counts.assign(pc.h, pc.h + S);
  return FGB_OK;
}

// Kernel, energy, adjoint GEMM and variance for all species (FP64).
int kernel_stage_fp64(fgb_model_s *m, int N, const std::vector<int> &counts,
                      bool want_grad, bool want_var, double *d_e_atom,
                      double *d_gB2, double *d_var, cudaStream_t st) {
  const B2Params &p = m->b2;
  const int nd = p.n_d;
  const double sig2 = m->sigma * m->sigma;
  int base = 0;
  for (int s = 0; s < p.n_species; s++) {
    const int Ns = counts[s];
    const int Ms = m->h_counts[s];
    const int *perm_s = m->ws.perm.as<int>() + base;
    if (Ns > 0 && Ms == 0 && want_var) {
      // No sparse environments of this species: k = 0 and E = 0 (zero
      // filled), var = k_self.
      k_variance_final<<<
          ceil_div((long long)Ns * kRowLanes, 128), 128, 0, st>>>(
          Ns, 0, nullptr, perm_s, m->ws.norms.as<double>(), sig2, m->power,
          1.0, d_var);
      FGB_LAUNCH_CHECK("k_variance_final");
    }
    for (int r0 = 0; r0 < Ns && Ms > 0; r0 += kRowChunk) {
      const int Mr = std::min(kRowChunk, Ns - r0);
      const int *perm = perm_s + r0;
      int rc;
      if ((rc = m->ws.kmat.ensure(sizeof(double) * (size_t)Mr * Ms)) ||
          (rc = m->ws.wmat.ensure(sizeof(double) * (size_t)Mr * Ms)) ||
          (rc = m->ws.erows.ensure(sizeof(double) * (size_t)Mr)))
        return rc;
      dim3 g1(ceil_div(Ms, BN), ceil_div(Mr, BM));
      {
        StageTimer _pt(kStKernelGemm, st, 1);
        k_kernel_gemm<<<g1, GT, 0, st>>>(
            Mr, Ms, nd, m->ws.B2.as<double>(), perm, m->ws.norms.as<double>(),
            m->S.as<double>() + (size_t)m->h_offsets[s] * nd,
            m->alpha.as<double>() + m->h_offsets[s],
            m->svalid.as<unsigned char>() + m->h_offsets[s], sig2, m->power,
            m->ws.kmat.as<double>(), m->ws.wmat.as<double>());
        FGB_LAUNCH_CHECK("k_kernel_gemm");
      }
      {
        StageTimer _pt(kStRowEnergy, st, 1);
        k_row_energy<<<ceil_div((long long)Mr * 32, 256), 256, 0, st>>>(
            Mr, Ms, m->ws.kmat.as<double>(),
            m->alpha.as<double>() + m->h_offsets[s], perm,
            m->ws.erows.as<double>(), d_e_atom);
        FGB_LAUNCH_CHECK("k_row_energy");
      }
      if (want_grad) {
        dim3 g2(ceil_div(nd, BN), ceil_div(Mr, BM));
        {
          StageTimer _pt(kStAdjointGemm, st, 1);
          k_adjoint_gemm<<<g2, GT, 0, st>>>(
              Mr, nd, Ms, m->ws.wmat.as<double>(),
              m->S.as<double>() + (size_t)m->h_offsets[s] * nd, perm,
              m->ws.norms.as<double>(), m->ws.B2.as<double>(),
              m->ws.erows.as<double>(), m->power, d_gB2);
          FGB_LAUNCH_CHECK("k_adjoint_gemm");
        }
      }
      if (want_var) {
        const int R = m->h_panel_rows[s];
        const int ntiles = ceil_div(R, BN);
        if ((rc = m->ws.part.ensure(sizeof(double) * (size_t)Mr * ntiles)))
          return rc;
        dim3 g3(ntiles, ceil_div(Mr, BM));
        {
          StageTimer _pt(kStVarianceGemm, st, 1);
          k_variance_gemm<<<g3, GT, 0, st>>>(
              Mr, R, Ms, m->ws.kmat.as<double>(),
              m->Lp.as<double>() + m->h_panel_off[s], m->ws.part.as<double>(),
              ntiles);
          FGB_LAUNCH_CHECK("k_variance_gemm");
        }
        {
          StageTimer _pt(kStVarianceFinal, st, 1);
          k_variance_final<<<
              ceil_div((long long)Mr * kRowLanes, 128), 128, 0, st>>>(
              Mr, ntiles, m->ws.part.as<double>(), perm,
              m->ws.norms.as<double>(), sig2, m->power, 1.0, d_var);
          FGB_LAUNCH_CHECK("k_variance_final");
        }
      }
    }
    base += Ns;
  }
  return FGB_OK;
}

}  // namespace fgb

using namespace fgb;

// ----------------------------------------------------------------- model
extern "C" int fgb_model_create(fgb_model_t *out, fgb_b2_t b2, double sigma,
                                double power) {
  if (!out || !b2) { set_error("fgb_model_create: invalid arguments"); return FGB_EINVAL; }
  if (!std::isfinite(sigma) || !std::isfinite(power)) {
    set_error("fgb_model_create: non-finite hyperparameters");
    return FGB_EINVAL;
  }
  fgb_model_s *m = new fgb_model_s();
  m->b2 = b2->p;
  m->sigma = sigma;
  m->power = power;
  *out = m;
  return FGB_OK;
}

extern "C" int fgb_model_destroy(fgb_model_t m) {
  delete m;
  return FGB_OK;
}

// On the bits, without a branch: 4 M entries of L_inv one by one with
// std::isfinite took 2 of the 10 ms of a call.
static bool all_finite(const double *x, int n) {
  unsigned bad = 0;
  for (int i = 0; i < n; i++) {
    unsigned long long b;
    std::memcpy(&b, x + i, sizeof(b));
    bad |= (b << 1) >= 0xFFE0000000000000ULL;
  }
  return !bad;
}

extern "C" int fgb_model_set(fgb_model_t m, const int *h_counts,
                             const double *h_desc, const double *h_alpha,
                             const double *h_L_inv) {
  if (!m || !h_counts) { set_error("fgb_model_set: invalid arguments"); return FGB_EINVAL; }
  const int S = m->b2.n_species, nd = m->b2.n_d;
  int M = 0;
  for (int s = 0; s < S; s++) {
    if (h_counts[s] < 0) { set_error("fgb_model_set: negative count"); return FGB_EINVAL; }
    M += h_counts[s];
  }
  if (M > 0 && !h_desc) { set_error("fgb_model_set: descriptors required"); return FGB_EINVAL; }
  // nothing of the weights before stays in use, also if this call fails on
  // the way: neither R_inv (of another Sigma, perhaps of another size) nor
  // any sliced operand
  m->solved = false;
  m->has_rinv = false;
  m->bmap_ready = false;
  m->lfull_ready = false;
  m->slices_chosen = false;
  m->oz_S = oz::kS;
  m->oz_Sv = oz::kS;
  m->oz_err_est = 0.0;
  m->oz_var_err_est = 0.0;
  m->force_f64 = false;
  m->fold_max = 0.0;
  for (bool &r : m->ozS_ready) r = false;
  for (bool &r : m->ozL_ready) r = false;
  for (bool &r : m->ozB_ready) r = false;
  for (int v = 0; v < oz::kTiles64; v++)
    m->oz64S_ready[v] = m->oz64ST_ready[v] = m->oz64L_ready[v] =
        m->oz64R_ready[v] = m->oz64Lfull_ready[v] = false;
  m->h_counts.assign(h_counts, h_counts + S);
  m->h_offsets.assign(S + 1, 0);
  for (int s = 0; s < S; s++)
    m->h_offsets[s + 1] = m->h_offsets[s] + h_counts[s];
  m->M = M;
  // normalised sparse descriptors, validity flags (norm >= 1e-8)
  std::vector<double> Sh((size_t)M * nd);
  std::vector<unsigned char> valid(M);
  std::vector<double> snorm(M);
  for (int t = 0; t < M; t++) {
    const double *row = h_desc + (size_t)t * nd;
    double nn = 0;
    for (int q = 0; q < nd; q++) nn += row[q] * row[q];
    double n = std::sqrt(nn);
    snorm[t] = n;
    valid[t] = n >= kEmptyThresh;
    for (int q = 0; q < nd; q++) Sh[(size_t)t * nd + q] = valid[t] ? row[q] / n : 0.0;
  }
  m->h_snorm = snorm;
  m->h_desc.assign(h_desc, h_desc + (size_t)M * nd);
  int rc;
  if ((rc = m->S.ensure(sizeof(double) * (size_t)M * nd)) ||
      (rc = m->svalid.ensure(M + 1)) ||
      (rc = m->Sraw.ensure(sizeof(double) * (size_t)M * nd)) ||
      (rc = m->snorm.ensure(sizeof(double) * (M + 1))))
    return rc;
  if (M > 0) {
    FGB_CUDA(cudaMemcpy(m->S.p, Sh.data(), sizeof(double) * (size_t)M * nd,
                        cudaMemcpyHostToDevice));
    FGB_CUDA(cudaMemcpy(m->Sraw.p, h_desc, sizeof(double) * (size_t)M * nd,
                        cudaMemcpyHostToDevice));
    FGB_CUDA(cudaMemcpy(m->svalid.p, valid.data(), M, cudaMemcpyHostToDevice));
    FGB_CUDA(cudaMemcpy(m->snorm.p, snorm.data(), sizeof(double) * M,
                        cudaMemcpyHostToDevice));
  }
  m->finite = true;
  for (int t = 0; t < M; t++) m->finite &= std::isfinite(snorm[t]);
  if (!h_alpha || !h_L_inv) return FGB_OK;
  if ((rc = m->alpha.ensure(sizeof(double) * (M + 1)))) return rc;
  if (M > 0)
    FGB_CUDA(cudaMemcpy(m->alpha.p, h_alpha, sizeof(double) * M,
                        cudaMemcpyHostToDevice));
  m->h_alpha.assign(h_alpha, h_alpha + M);
  m->alpha_max.assign(S, 0.0);
  for (int s = 0; s < S; s++)
    for (int t = m->h_offsets[s]; t < m->h_offsets[s + 1]; t++) {
      m->finite &= std::isfinite(h_alpha[t]);
      m->alpha_max[s] = std::max(m->alpha_max[s], std::fabs(h_alpha[t]));
    }
  m->h_L_inv.assign(h_L_inv, h_L_inv + (size_t)M * M);
  // L_inv panels: species s uses rows [c_s, c_s + R_s) and columns
  // [c_s, c_s + M_s); R_s = M_s when everything below the diagonal block is
  // exactly zero (the single-kernel case), else M - c_s.
  std::vector<double> panels;
  bool finite = true;
  m->h_panel_rows.assign(S, 0);
  m->h_panel_off.assign(S, 0);
  for (int s = 0; s < S; s++) {
    const int cs = m->h_offsets[s], Ms = h_counts[s];
    bool below_zero = true;
    for (int r = cs + Ms; r < M && below_zero; r++)
      for (int c = cs; c < cs + Ms; c++)
        if (h_L_inv[(size_t)r * M + c] != 0.0) { below_zero = false; break; }
    const int R = below_zero ? Ms : M - cs;
    m->h_panel_rows[s] = R;
    m->h_panel_off[s] = (long long)panels.size();
    for (int r = 0; r < R; r++) {
      const double *row = h_L_inv + (size_t)(cs + r) * M + cs;
      panels.insert(panels.end(), row, row + Ms);
      finite &= all_finite(row, Ms);   // while it is in the cache
    }
  }
  m->finite &= finite;
  if ((rc = m->Lp.ensure(sizeof(double) * (panels.size() + 1)))) return rc;
  if (!panels.empty())
    FGB_CUDA(cudaMemcpy(m->Lp.p, panels.data(), sizeof(double) * panels.size(),
                        cudaMemcpyHostToDevice));
  m->solved = true;
  return FGB_OK;
}

// A model with the same weights and its own device workspace.
fgb_model_s *model_replicate(const fgb_model_s *src, int &rc) {
  fgb_model_s *m = new fgb_model_s();
  m->b2 = src->b2;
  m->sigma = src->sigma;
  m->power = src->power;
  rc = fgb_model_set(m, src->h_counts.data(), src->h_desc.data(),
                     src->solved ? src->h_alpha.data() : nullptr,
                     src->solved ? src->h_L_inv.data() : nullptr);
  if (rc) { delete m; return nullptr; }
  if (src->has_rinv) {
    if ((rc = m->RinvT.ensure(src->RinvT.bytes))) { delete m; return nullptr; }
    cudaError_t e = cudaMemcpy(m->RinvT.p, src->RinvT.p, src->RinvT.bytes,
                               cudaMemcpyDeviceToDevice);
    if (e != cudaSuccess) {
      rc = cuda_status(e, "model_replicate");
      delete m;
      return nullptr;
    }
    m->has_rinv = true;
  }
  return m;
}

// ------------------------------------------------------------- predict
int predict_impl(fgb_model_s *m, int n_struc, const int *h_atom_offsets,
                 const double *h_cells, const double *d_positions,
                 const int *d_species, double cutoff, int want, int precision,
                 double *d_energy, double *d_forces, double *d_stress,
                 double *d_local_var, cudaStream_t st, const FixedPlan *fixed,
                 const PredictHostIO *hio) {
  if (!m->solved) {
    set_error("L_inv must be up to date to make predictions. Please call "
              "update_matrices_QR and try again.");
    return FGB_ESTALE;
  }
  if (precision != FGB_PREC_FP64 && precision != FGB_PREC_MIXED) {
    set_error("fgb_predict: unknown precision %d", precision);
    return FGB_EINVAL;
  }
  int rc;
  if (fixed && (m->nl.n_struc != n_struc || m->nl.n_atoms !=
                    h_atom_offsets[n_struc] ||
                (int)fixed->counts.size() != m->b2.n_species)) {
    set_error("fgb_predict: fixed call on a different batch than the last");
    return FGB_EINVAL;
  }
  {
    StageTimer _pt(kStNeighbors, st);
    rc = fixed ? nlist_rebuild_fixed(&m->nl, d_positions, cutoff,
                                     fixed->pair_cap, st)
               : nlist_build(&m->nl, n_struc, h_atom_offsets, h_cells,
                             d_positions, cutoff, st, false);
    _pt.set_launches(m->nl.last_launches);
    if (rc) return rc;
  }
  const B2Params &p = m->b2;
  const int N = m->nl.n_atoms;
  const long long P = m->nl.n_pairs;
  const bool mixed = precision == FGB_PREC_MIXED;
  // the bounded tensor-core waits report into ws.ozerr, read at the end (a
  // fixed call's caller clears and reads it)
  if ((rc = m->ws.ozerr.ensure(sizeof(int)))) return rc;
  const bool sliced = mixed || fp64_stage_sliced(m);
  if (!fixed && sliced)
    FGB_CUDA(cudaMemsetAsync(m->ws.ozerr.p, 0, sizeof(int), st));
  const bool want_e = want & FGB_WANT_ENERGY, want_f = want & FGB_WANT_FORCES,
             want_s = want & FGB_WANT_STRESS, want_v = want & FGB_WANT_LOCAL_VAR;
  const bool want_grad = want_f || want_s;
  // forces and local variances go straight to the caller's buffers when
  // given (no device-to-device copy at the end)
  const bool f_direct = want_f && d_forces, v_direct = want_v && d_local_var;
  if ((rc = m->ws.A.ensure(sizeof(float) * ((size_t)N * p.n_A + 2))) ||
      (rc = m->ws.B2.ensure(sizeof(double) * ((size_t)N * p.n_d + 1))) ||
      (rc = m->ws.norms.ensure(sizeof(double) * (N + 1))) ||
      (rc = m->ws.e_atom.ensure(sizeof(double) * (N + 1))) ||
      (rc = m->ws.var.ensure(sizeof(double) * (N + 1))) ||
      (rc = m->ws.rowmax.ensure(sizeof(double) * (N + 1))))
    return rc;
  if (want_grad &&
      ((rc = m->ws.gB2.ensure(sizeof(double) * ((size_t)N * p.n_d + 1))) ||
       (rc = m->ws.pair_grad.ensure(sizeof(double3) * (P + 1))) ||
       (rc = m->ws.forces.ensure(sizeof(double) * (3 * (size_t)N + 1))) ||
       (rc = m->ws.virial.ensure(sizeof(double) * (6 * (size_t)N + 1)))))
    return rc;
  // the kernel stages write every atom of a species with sparse environments
  bool unwritten = false;
  for (int s = 0; s < p.n_species; s++) unwritten |= m->h_counts[s] == 0;
  if (N > 0 && unwritten) {
    FGB_CUDA(cudaMemsetAsync(m->ws.e_atom.p, 0, sizeof(double) * N, st));
    FGB_CUDA(cudaMemsetAsync(v_direct ? d_local_var : m->ws.var.as<double>(),
                             0, sizeof(double) * N, st));
  }
  // the fold guard is known before the descriptor: models with large folded
  // coefficients take the descriptor, force product and adjoint at FP64
  // level (a fixed call reuses the full call's fold)
  if (mixed && !fixed && (rc = prepare_mixed(m, st))) return rc;
  // FP32 adjoint (and FP32 pair gradients and force sums) in the mixed
  // path (dE/dB2 written in FP32 by the mapped gradient), unless the fold
  // guard asked for FP64-level forces or the power has no folded form
  // (FP64 kernel stage); its A is written in FP32 by the forward
  const bool adj32 = mixed && !m->force_f64 &&
                     (m->power == 2.0 || m->power == 1.0);
  if (!adj32 &&
      (rc = m->ws.A.ensure(sizeof(double) * ((size_t)N * p.n_A + 1))))
    return rc;
  // species counts: queued before the descriptor and waited for after it,
  // so the GPU runs the descriptor while the host waits (on device species)
  std::vector<int> counts;
  bool counts_pending = false;
  if (fixed) {
    counts = fixed->counts;
  } else {
    StageTimer _pt(kStSpeciesPerm, st, N <= kPermOne ? 1 : 3);
    if ((rc = species_permutation_start(p.n_species, m->ws, d_species, N,
                                        counts, st,
                                        hio ? hio->species : nullptr,
                                        counts_pending)))
      return rc;
  }
  {
    StageTimer _pt(kStB2Forward, st);
    // mixed precision: the descriptor in double-float (about 46 bits)
    if ((rc = launch_b2_forward(p, &m->nl, d_species,
                                adj32 ? nullptr : m->ws.A.as<double>(),
                                m->ws.B2.as<double>(), m->ws.norms.as<double>(),
                                st, mixed && !m->force_f64,
                                sliced ? m->ws.rowmax.as<double>() : nullptr,
                                adj32 ? m->ws.A.as<float>() : nullptr)))
      return rc;
  }
  if (counts_pending &&
      (rc = species_permutation_finish(p.n_species, m->ws, counts)))
    return rc;
  if (!fixed) m->last_species_counts = counts;
  // dE/dB2 rows: the kernel stages write every row of a species with sparse
  // environments; rows of species without any stay zero
  if (want_grad && N > 0) {
    bool zero = false;
    for (int s = 0; s < p.n_species; s++)
      zero |= counts[s] > 0 && m->h_counts[s] == 0;
    if (zero)
      FGB_CUDA(cudaMemsetAsync(m->ws.gB2.p, 0,
                               sizeof(double) * (size_t)N * p.n_d, st));
  }
  if (precision == FGB_PREC_MIXED) {
    if ((rc = kernel_stage_mixed(m, N, counts, want_grad, want_v,
                                 m->ws.e_atom.as<double>(),
                                 m->ws.gB2.as<double>(),
                                 v_direct ? d_local_var : m->ws.var.as<double>(),
                                 st, fixed != nullptr)))
      return rc;
  } else if (sliced) {
    if ((rc = kernel_stage_fp64_oz(m, counts, want_grad, want_v,
                                   m->ws.e_atom.as<double>(),
                                   m->ws.gB2.as<double>(),
                                   v_direct ? d_local_var : m->ws.var.as<double>(),
                                   st, fixed != nullptr, true)))
      return rc;
  } else {
    if ((rc = kernel_stage_fp64(m, N, counts, want_grad, want_v,
                                m->ws.e_atom.as<double>(),
                                m->ws.gB2.as<double>(),
                                v_direct ? d_local_var : m->ws.var.as<double>(),
                                st)))
      return rc;
  }
  if (want_grad) {
    {
      StageTimer _pt(kStB2Adjoint, st);
      if ((rc = launch_b2_adjoint(p, &m->nl, d_species,
                                  adj32 ? nullptr : m->ws.A.as<double>(),
                                  m->ws.gB2.p, m->ws.pair_grad.p, st, adj32,
                                  adj32 ? m->ws.A.as<float>() : nullptr)))
        return rc;
    }
    {
      StageTimer _pt(kStForces, st);
      if ((rc = launch_forces(&m->nl, m->ws.pair_grad.p, adj32,
                              f_direct ? d_forces : m->ws.forces.as<double>(),
                              m->ws.virial.as<double>(), st)))
        return rc;
    }
  }
  if ((want_e && d_energy) || (want_s && d_stress)) {
    StageTimer _ptr(kStStructReduce, st);
    if ((rc = launch_struct_reduce(
             &m->nl, m->ws.e_atom.as<double>(),
             want_grad ? m->ws.virial.as<double>() : nullptr,
             want_e ? d_energy : nullptr, want_s ? d_stress : nullptr,
             m->ws.redpart, st)))
      return rc;
  }
  if (fixed) return FGB_OK;
  // results to the host ahead of the one synchronisation below
  if (hio && hio->stage) {
    FGB_CUDA(cudaMemcpyAsync(hio->stage, hio->block, hio->bytes,
                             cudaMemcpyDeviceToHost, st));
  } else if (hio) {
    if (hio->energy && want_e)
      FGB_CUDA(cudaMemcpyAsync(hio->energy, d_energy, sizeof(double) * n_struc,
                               cudaMemcpyDeviceToHost, st));
    if (hio->forces && want_f && N > 0)
      FGB_CUDA(cudaMemcpyAsync(hio->forces, d_forces, sizeof(double) * 3 * N,
                               cudaMemcpyDeviceToHost, st));
    if (hio->stress && want_s)
      FGB_CUDA(cudaMemcpyAsync(hio->stress, d_stress, sizeof(double) * 6 * n_struc,
                               cudaMemcpyDeviceToHost, st));
    if (hio->local_var && want_v && N > 0)
      FGB_CUDA(cudaMemcpyAsync(hio->local_var, d_local_var,
                               sizeof(double) * N, cudaMemcpyDeviceToHost, st));
  }
  // deferred checks: neighbour-list consistency, tensor-core waits
  if (!m->ws.counts.status)
    FGB_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&m->ws.counts.status),
                           sizeof(int) * 8, cudaHostAllocDefault));
  int *h = m->ws.counts.status;
  h[4] = 0;
  FGB_CUDA(cudaMemcpyAsync(h, m->nl.flag.p, sizeof(int) * 4,
                           cudaMemcpyDeviceToHost, st));
  if (sliced)
    FGB_CUDA(cudaMemcpyAsync(h + 4, m->ws.ozerr.p, sizeof(int),
                             cudaMemcpyDeviceToHost, st));
  FGB_CUDA(cudaStreamSynchronize(st));
  rc = nlist_finish(&m->nl, h);
  if (rc == kNlistRetry) {
    // an atom had more pairs than its single-pass slots: the whole call
    // again, its list built with a count pass
    m->nl.count_pass = true;
    rc = predict_impl(m, n_struc, h_atom_offsets, h_cells, d_positions,
                      d_species, cutoff, want, precision, d_energy, d_forces,
                      d_stress, d_local_var, st, nullptr, hio);
    m->nl.count_pass = false;
    return rc;
  }
  if (rc) return rc;
  if (h[4]) {
    set_error("tensor-core stage: a bounded device wait ran out");
    return FGB_ETIMEOUT;
  }
  return FGB_OK;
}

extern "C" int fgb_predict(fgb_model_t m, int n_struc, const int *h_atom_offsets,
                           const double *h_cells, const double *d_positions,
                           const int *d_species, double cutoff, int want,
                           int precision, double *d_energy, double *d_forces,
                           double *d_stress, double *d_local_var, void *stream) {
  if (!m) { set_error("fgb_predict: null model"); return FGB_EINVAL; }
  return predict_impl(m, n_struc, h_atom_offsets, h_cells, d_positions,
                      d_species, cutoff, want, precision, d_energy, d_forces,
                      d_stress, d_local_var, (cudaStream_t)stream);
}

extern "C" int fgb_predict_host(fgb_model_t m, int n_struc,
                                const int *h_atom_offsets, const double *h_cells,
                                const double *h_positions, const int *h_species,
                                double cutoff, int want, int precision,
                                double *h_energy, double *h_forces,
                                double *h_stress, double *h_local_var,
                                void *stream) {
  if (!m || n_struc <= 0 || !h_atom_offsets) {
    set_error("fgb_predict_host: invalid arguments");
    return FGB_EINVAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int N = h_atom_offsets[n_struc];
  int rc;
  const size_t in_pos = sizeof(double) * 3 * (size_t)N;
  const size_t in_bytes = in_pos + sizeof(int) * (size_t)N;
  const size_t S = n_struc;
  const size_t out_bytes = sizeof(double) * (7 * S + 4 * (size_t)N);
  fgb_io &io = m->io;
  if ((rc = io.in.ensure(in_bytes + 16)) || (rc = io.out.ensure(out_bytes + 16)))
    return rc;
  const bool stage_in = in_bytes <= fgb_io::kStage,
             stage_out = out_bytes <= fgb_io::kStage;
  if ((stage_in || stage_out) && !io.stage)
    FGB_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&io.stage),
                           2 * fgb_io::kStage, cudaHostAllocDefault));
  double *d_pos = io.in.as<double>();
  int *d_species = reinterpret_cast<int *>(d_pos + 3 * (size_t)N);
  if (N > 0 && stage_in) {
    std::memcpy(io.stage, h_positions, in_pos);
    std::memcpy(io.stage + in_pos, h_species, in_bytes - in_pos);
    FGB_CUDA(cudaMemcpyAsync(d_pos, io.stage, in_bytes, cudaMemcpyHostToDevice,
                             st));
  } else if (N > 0) {
    FGB_CUDA(cudaMemcpyAsync(d_pos, h_positions, in_pos,
                             cudaMemcpyHostToDevice, st));
    FGB_CUDA(cudaMemcpyAsync(d_species, h_species, in_bytes - in_pos,
                             cudaMemcpyHostToDevice, st));
  }
  double *d_e = io.out.as<double>(), *d_s = d_e + S, *d_v = d_s + 6 * S,
         *d_f = d_v + N;
  // species counted on the host (no read-back) and results copied back
  // before the prediction's final synchronisation
  PredictHostIO hio;
  hio.species = h_species;
  hio.energy = h_energy;
  hio.forces = h_forces;
  hio.stress = h_stress;
  hio.local_var = h_local_var;
  unsigned char *out = io.stage + fgb_io::kStage;
  if (stage_out) {
    hio.block = d_e;
    hio.stage = out;
    hio.bytes = out_bytes;
  }
  if ((rc = predict_impl(m, n_struc, h_atom_offsets, h_cells, d_pos, d_species,
                         cutoff, want, precision, d_e, d_f, d_s, d_v, st,
                         nullptr, &hio)))
    return rc;
  if (stage_out) {
    const double *r = reinterpret_cast<const double *>(out);
    if (h_energy && (want & FGB_WANT_ENERGY))
      std::memcpy(h_energy, r, sizeof(double) * S);
    if (h_stress && (want & FGB_WANT_STRESS))
      std::memcpy(h_stress, r + S, sizeof(double) * 6 * S);
    if (h_local_var && (want & FGB_WANT_LOCAL_VAR))
      std::memcpy(h_local_var, r + 7 * S, sizeof(double) * N);
    if (h_forces && (want & FGB_WANT_FORCES))
      std::memcpy(h_forces, r + 7 * S + N, sizeof(double) * 3 * N);
  }
  return FGB_OK;
}

extern "C" int fgb_model_set_R_inv(fgb_model_t m, const double *h_R_inv) {
  if (!m || !h_R_inv) { set_error("fgb_model_set_R_inv: invalid arguments"); return FGB_EINVAL; }
  const int M = m->M;
  std::vector<double> t((size_t)M * M);
  for (int r = 0; r < M; r++)
    for (int c = 0; c < M; c++) t[(size_t)c * M + r] = h_R_inv[(size_t)r * M + c];
  int rc;
  if ((rc = m->RinvT.ensure(sizeof(double) * ((size_t)M * M + 1)))) return rc;
  if (M > 0)
    FGB_CUDA(cudaMemcpy(m->RinvT.p, t.data(), sizeof(double) * (size_t)M * M,
                        cudaMemcpyHostToDevice));
  m->has_rinv = true;
  for (bool &r : m->oz64R_ready) r = false;
  return FGB_OK;
}

// out[o] = |row o of K^T T|^2 for K^T (ncol x M, sliced in kt) and the lower
// triangular B operand (row-major, M x M; its slices kept in `B` per model).
static int solved_variance(fgb_model_s *m, const oz::Sliced &kt,
                           const oz::Sliced &B, long long ncol, DevBuf &part,
                           double *out, cudaStream_t st) {
  int rc;
  const int slots = B.RP / 16;
  if ((rc = part.ensure(sizeof(double) * ((size_t)ncol * slots + 1))) ||
      (rc = oz::gemm_rowsq(kt, B, true, part.as<double>(),
                           m->ws.ozerr.as<int>(), st)))
    return rc;
  k_sum_parts<<<ceil_div(ncol * kRowLanes, 128), 128, 0, st>>>(
      (int)ncol, slots, part.as<double>(), out);
  FGB_LAUNCH_CHECK("k_sum_parts");
  return FGB_OK;
}

// The M x M lower-triangular matrix `src` of the model as a kS64-slice B
// operand for products with ncol rows, sliced once per tile height.
static int solved_operand(const DevBuf &src, int M, int v, oz::Sliced *out,
                          bool *ready, cudaStream_t st) {
  if (ready[v]) return FGB_OK;
  const int rc = oz::slice({M, M, oz::kTN64v[v], src.as<double>(), M, nullptr,
                            nullptr, nullptr, true},
                           out[v], st, oz::kS64);
  if (rc == FGB_OK) ready[v] = true;
  return rc;
}

// Mean and, with `dtc`, the DTC (else the SOR) variances of one structure.
static int predict_solved(fgb_model_s *m, fgb_nlist_s *nl, const int *d_species,
                          double *d_mean_efs, double *d_variance_efs, bool dtc,
                          const char *what, cudaStream_t st) {
  if (!m->solved || !m->has_rinv) {
    set_error("L_inv must be up to date to make predictions. Please call "
              "update_matrices_QR and try again.");
    return FGB_ESTALE;
  }
  const int N = nl->n_atoms, M = m->M;
  const long long ncol = 1 + 3LL * N + 6;
  if (ncol > (1LL << 30)) { set_error("%s: structure too large", what); return FGB_EINVAL; }
  int rc;
  DevBuf kt(st), part(st), kself(st), q(st);
  oz::Sliced kts(st);
  if ((rc = kt.ensure(sizeof(double) * ((size_t)M * ncol + 1)))) return rc;
  if (dtc && !m->lfull_ready && M > 0) {
    if ((rc = m->Lfull.ensure(sizeof(double) * (size_t)M * M))) return rc;
    FGB_CUDA(cudaMemcpy(m->Lfull.p, m->h_L_inv.data(),
                        sizeof(double) * (size_t)M * M, cudaMemcpyHostToDevice));
    m->lfull_ready = true;
    for (bool &r : m->oz64Lfull_ready) r = false;
  }
  if ((rc = envs_struc_impl(m->b2, m->sigma, m->power, m->h_counts.data(),
                            m->Sraw.as<double>(), nl, d_species,
                            kt.as<double>(), m->ws, st)))
    return rc;
  if (dtc) {
    // K_self from the descriptors and stored gradients envs_struc left in
    // the workspace (it computes them only when M > 0 and N > 0)
    if ((rc = kself.ensure(sizeof(double) * ncol)) ||
        (rc = q.ensure(sizeof(double) * ncol)) ||
        (rc = self_kernel_impl(m->b2, m->sigma, m->power, nl, d_species,
                               kself.as<double>(), m->ws, st, M > 0)))
      return rc;
  }
  if (M == 0) {
    FGB_CUDA(cudaMemsetAsync(d_mean_efs, 0, sizeof(double) * ncol, st));
    if (dtc)
      FGB_CUDA(cudaMemcpyAsync(d_variance_efs, kself.p, sizeof(double) * ncol,
                               cudaMemcpyDeviceToDevice, st));
    else
      FGB_CUDA(cudaMemsetAsync(d_variance_efs, 0, sizeof(double) * ncol, st));
    FGB_CUDA(cudaStreamSynchronize(st));
    return FGB_OK;
  }
  const int v = oz::tile64((int)ncol, M);
  if ((rc = launch_kt_alpha(M, ncol, kt.as<double>(), m->alpha.as<double>(),
                            d_mean_efs, st)) ||
      (rc = oz::slice({(int)ncol, M, oz::kTM, kt.as<double>(), M, nullptr,
                       nullptr},
                      kts, st, oz::kS64)) ||
      // diag(K^T Sigma K) = column sums of (R_inv^T K)^2, with the lower
      // factor R_inv^T (sparse_gp.cpp:689-691, 724)
      (rc = solved_operand(m->RinvT, M, v, m->oz64R, m->oz64R_ready, st)) ||
      (rc = solved_variance(m, kts, m->oz64R[v], ncol, part, d_variance_efs,
                            st)))
    return rc;
  if (dtc) {
    // diag(K^T Kuu^-1 K) = column sums of (L_inv K)^2 (sparse_gp.cpp:723)
    if ((rc = solved_operand(m->Lfull, M, v, m->oz64Lfull, m->oz64Lfull_ready,
                             st)) ||
        (rc = solved_variance(m, kts, m->oz64Lfull[v], ncol, part,
                              q.as<double>(), st)))
      return rc;
    k_dtc_combine<<<ceil_div(ncol, 256), 256, 0, st>>>(
        ncol, kself.as<double>(), q.as<double>(), d_variance_efs);
    FGB_LAUNCH_CHECK("k_dtc_combine");
  }
  return sliced_finish(m->ws, st, what);
}

extern "C" int fgb_predict_sor(fgb_model_t m, fgb_nlist_t nl,
                               const int *d_species, double *d_mean_efs,
                               double *d_variance_efs, void *stream) {
  if (!m || !nl || !d_mean_efs || !d_variance_efs) {
    set_error("fgb_predict_sor: invalid arguments");
    return FGB_EINVAL;
  }
  return predict_solved(m, nl, d_species, d_mean_efs, d_variance_efs, false,
                        "fgb_predict_sor", (cudaStream_t)stream);
}

extern "C" int fgb_predict_dtc(fgb_model_t m, fgb_nlist_t nl,
                               const int *d_species, double *d_mean_efs,
                               double *d_variance_efs, void *stream) {
  if (!m || !nl || !d_mean_efs || !d_variance_efs) {
    set_error("fgb_predict_dtc: invalid arguments");
    return FGB_EINVAL;
  }
  return predict_solved(m, nl, d_species, d_mean_efs, d_variance_efs, true,
                        "fgb_predict_dtc", (cudaStream_t)stream);
}
