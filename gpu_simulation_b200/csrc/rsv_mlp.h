// Launchers of the warm-start network kernels (rsv_mlp.cu), used by the host
// side (rsv_mlp_host.cpp).
#pragma once

#include <cuda_runtime.h>

namespace rsv {

// One product C[m][n] = sum_k A[m*sam + k*sak] * B[k*sbk + n*sbn] (C is M x N,
// row-major) and what follows it: + bias[n], the sum itself to Z, GELU, times
// GELU's derivative at gelu_of[m][n] (each where not null / set).  row_sums[m]
// receives sum_k A(m, k) where not null.
struct MlpGemm {
  int M, N, K;
  const float *A;
  long long sam, sak;
  const float *B;
  long long sbk, sbn;
  float *C;
  const float *bias;
  float *Z;
  const float *gelu_of;
  float *row_sums;
  bool gelu;
};
// One or two independent products in one launch.
cudaError_t mlp_gemm(const MlpGemm *g, int count, cudaStream_t s);
// partials: 256 floats
cudaError_t mlp_mse(long long count, const float *out, const float *target, float *dout, float *partials,
                    float *loss, cudaStream_t s);
cudaError_t gd_step(long long count, double *p, const double *g, double stepsize, const double *energy,
                    double *energy_hist, double *gnorm_hist, int *counter, cudaStream_t s);
cudaError_t adam_vqe_step(long long count, double *p, const double *g, double *m, double *v, double lr,
                          double beta1, double beta2, double eps, const double *energy, double *energy_hist,
                          int *counter, cudaStream_t s);
template <typename T>
cudaError_t adam_step(long long count, T *p, const T *g, T *m, T *v, T lr, T beta1, T beta2, T eps,
                      int step, cudaStream_t s);

}  // namespace rsv
