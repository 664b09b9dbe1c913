// FP64 vector kernels of the device Krylov solver (see kernels.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cmps {

// Device-resident coefficients of a Lanczos cycle: the local projection a (2),
// the Gram-Schmidt products h (2 per basis vector), beta_j and the scale s_j
// of basis vector j (V_j = s_j U_j), and |U_{j+1}|^2.
struct LanczosCoef {
  double *a, *h, *beta, *scale, *nrm2;
};

// Planar FP64 complex vectors of a fixed length n.  Reductions add one partial
// sum per CTA in a fixed order, in a second launch or in the CTA that finishes
// last, so results are deterministic run to run.
struct VecOps {
  int64_t n = 0;
  int nb = 0;
  double* d_partial = nullptr;
  double* d_small = nullptr;
  int64_t* d_pidx = nullptr;
  int init(int64_t n, cudaStream_t st);
  void release();
  // h[j] = <V_j, w> (conjugate-linear in V), k vectors with stride ldv; h_host gets 2k doubles.
  int multidot(const double* Vr, const double* Vi, int64_t ldv, int k, const double* wr, const double* wi,
               double* h_host, cudaStream_t st);
  int norm2(const double* xr, const double* xi, double* out, cudaStream_t st);
  int random(double* re, double* im, uint64_t seed, cudaStream_t st);
  // y = sum_j c_j V_j, c real
  int combine(const double* Vr, const double* Vi, int64_t ldv, int k, const double* c_host, double* yr,
              double* yi, cudaStream_t st);
  int absmax(const double* re, const double* im, double* val_sq, int64_t* idx, cudaStream_t st);

  // Krylov steps whose coefficients stay on the device (no host round trip).
  double* d_coef = nullptr;  // coefficient scratch, kCoefDoubles
  static constexpr int kCoefDoubles = 2048;
  // d_out[2j], d_out[2j+1] = <V_j, w> for j < k (k <= 128); d_out[2k] = |w|^2.
  int mdot_dev(const double* Vr, const double* Vi, int64_t ldv, int k, const double* wr, const double* wi,
               double* d_out, cudaStream_t st);
  // w -= sum_j h_j V_j with h = d_h (2k doubles); *d_nrm2 = |w|^2 afterwards.
  int maxpy_norm_dev(const double* Vr, const double* Vi, int64_t ldv, int k, const double* d_h, double* wr,
                     double* wi, double* d_nrm2, cudaStream_t st);
  // Step j of a Lanczos cycle with full re-orthogonalisation (kernels.cu):
  // basis vectors U_0 .. U_j at U + i ldv (real plane, imaginary plane n
  // further), y = H U_j, or H V_j where `unit` is set; the next vector into
  // (outr, outi) unless they are null, alpha_j and beta_j into host[0..1] (pinned
  // memory) once the stream has come this far.  The cycle's first scale, lanczos_coef().scale[0], is the caller's.
  int lanczos(const double* U, int64_t ldv, const double* yr, const double* yi, bool unit, int j, double* outr,
              double* outi, double* host, cudaStream_t st);
  LanczosCoef lanczos_coef() const;
  unsigned* d_count = nullptr;  // CTAs of the current launch that have finished
  // y = x / sqrt(*d_sq)
  int scale_dev(const double* xr, const double* xi, const double* d_sq, double* yr, double* yi, cudaStream_t st);
  int phase_drop(double* re, double* im, double pr, double pi, double thr, cudaStream_t st);
};

}  // namespace cmps
