// Launchers shared between libflaregb translation units.
#pragma once
#include "fgb_internal.h"

namespace fgb {

size_t b2_forward_smem(const B2Params &p, bool regA = false,
                       bool half = false);
// dfloat: compute in double-float (mixed-precision path) instead of FP64;
// d_rowmax (optional): each row's largest |B2| as written
// d_A32 (double-float forward only): A written in FP32 instead of d_A, for
// the FP32 adjoint
int launch_b2_forward(const B2Params &p, const fgb_nlist_s *nl,
                      const int *d_species, double *d_A, double *d_B2,
                      double *d_norms, cudaStream_t st, bool dfloat = false,
                      double *d_rowmax = nullptr, float *d_A32 = nullptr);
// d_gB2: dE/dB2 rows [N, n_d] and d_pair_grad: pair gradients [P], both in
// the compute type (float / float3 when fp32, else double / double3)
// d_A32 (fp32 only): A read in FP32 instead of from d_A
int launch_b2_adjoint(const B2Params &p, const fgb_nlist_s *nl,
                      const int *d_species, const double *d_A,
                      const void *d_gB2, void *d_pair_grad,
                      cudaStream_t st, bool fp32 = false,
                      const float *d_A32 = nullptr);
// d_pair_grad as the adjoint wrote it (fp32: float3)
int launch_forces(const fgb_nlist_s *nl, const void *d_pair_grad, bool fp32,
                  double *d_forces, double *d_virial, cudaStream_t st);
// Energies and stresses of the list's structures from per-atom energies and
// virials; `part`: scratch for structures of more than one chunk of atoms.
int launch_struct_reduce(const fgb_nlist_s *nl, const double *d_e_atom,
                         const double *d_virial, double *d_energy,
                         double *d_stress, DevBuf &part, cudaStream_t st);

// Stored forward-mode gradients (the reference's algorithm); scratch: each
// pair's centre atom (left for the caller) and the pairs' basis values;
// d_rowmax (optional): each gradient row's largest magnitude.
int launch_b2_dervs(const B2Params &p, const fgb_nlist_s *nl,
                    const int *d_species, const double *d_A, const double *d_B2,
                    double *d_dB2, double *d_force_dots, DevBuf &center,
                    DevBuf &basis, cudaStream_t st,
                    double *d_rowmax = nullptr);

// The local-variance finish var = k_self - scale sum(part) (predict.cu).
int launch_variance_final(int Mr, int ntiles, const double *part,
                          const int *perm, const double *norms, double sig2,
                          double xi, double *var, cudaStream_t st,
                          double scale = 1.0);

// mean_efs = K^T alpha from K^T (ncol x M).
int launch_kt_alpha(int M, long long ncol, const double *KT,
                    const double *alpha, double *out, cudaStream_t st);

// Validate coded species in [0, n_species); returns FGB_EINVAL otherwise.
int check_species(const int *d_species, int n, int n_species, DevBuf &flag,
                  cudaStream_t st);

}  // namespace fgb
