// Energy and gradient of a shallow circuit by contraction along the ring
// (rsv_ring.cu): host-callable launchers.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace rsv {

// Layers up to which the ring kernels are built (bond 2^(L-1) <= 16).
constexpr int kRingMaxLayers = 5;

struct RingParams {
  int n, L;
  double field;
  const double4 *coef;   // [L * n] (cos t/2, sin t/2, cos p/2, sin p/2)
  double2 *left;         // [n][chains][5][D * D] left components of every site before its last layer
  double2 *right;        // [n][chains][5][D * D] right components after every site
  double *energy_parts;  // [chains], then the energy itself
  unsigned int *counter; // finished left sweeps; 0 between calls
  double *energy_out;    // [1], or null
  double *grad_out;      // [2 n L]
};

// Bond vectors are padded to 8 (L <= 4) or 16 (L = 5) values a side.
constexpr int ring_padded_bond(int L) { return L <= 4 ? 8 : 16; }
constexpr int ring_chains(int L) { return 1 << (2 * (L - 1)); }
inline size_t ring_component_values(int n, int L) {
  const size_t d = static_cast<size_t>(ring_padded_bond(L));
  return static_cast<size_t>(n) * ring_chains(L) * 5 * d * d;
}

// The sweeps: left (energy; components kept for the gradient when `keep`),
// right, or both at once; then the gradient from the kept components.
cudaError_t launch_ring_sweeps(const RingParams &P, bool left, bool right, bool keep, cudaStream_t s);
cudaError_t launch_ring_gradient(const RingParams &P, cudaStream_t s);

}  // namespace rsv
