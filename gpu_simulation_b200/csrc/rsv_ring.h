// Energy and gradient of a shallow circuit by contraction along the ring
// (rsv_ring.cu): host-callable launchers.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace rsv {

// Layers up to which the ring kernels are built (bond 2^(L-1) <= 16).
constexpr int kRingMaxLayers = 5;
constexpr int kRingDerivs = 2 * kRingMaxLayers;

struct RingParams {
  int n, L;
  double field;
  const double *params;  // angles [2 L n] on the device, or null: coef is given
  double4 *coef;         // [L * n] (cos t/2, sin t/2, cos p/2, sin p/2); written by the sweeps from params
  double2 *left;         // [n][chains][5][D * D] left components of every site before its last layer
  double2 *right;        // [n][chains][5][D * D] right components after every site
  double *energy_parts;  // [chains], then the energy itself (kRingMaxParts values at most)
  double *grad_parts;    // [n][8][kRingDerivs]
  unsigned int *counter; // [1 + n] finished left sweeps, finished CTAs of every site; 0 between calls
  double *energy_out;    // [1], or null
  double *grad_out;      // [2 n L]
};

// Bond vectors are padded to 8 (L <= 4) or 16 (L = 5) values a side.
constexpr int ring_padded_bond(int L) { return L <= 4 ? 8 : 16; }
// Chains: pairs a <= abar of the bits that enter wire 0.
constexpr int ring_chains(int L) { return (1 << (L - 1)) * ((1 << (L - 1)) + 1) / 2; }
constexpr int kRingMaxParts = ring_chains(kRingMaxLayers) + 1;
inline size_t ring_component_values(int n, int L) {
  const size_t d = static_cast<size_t>(ring_padded_bond(L));
  return static_cast<size_t>(n) * ring_chains(L) * 5 * d * d;
}

// Warps of a gradient CTA, and the chains it takes at a time.
constexpr int kRingGradWarps = 10;
constexpr int ring_chains_a_step(int L) { return L <= 4 ? 4 : 1; }
// CTAs a site of the gradient: at most eight, no more than its chains need, and no
// more (one CTA an SM) than fill the SMs once.  Wire 0 needs a warp for every one of
// its 2^(L-1) columns whatever the device has: two CTAs at L = 5 (with one, its ten
// warps would leave the sixteen columns' gradient zero).
constexpr int ring_gradient_ctas(int n, int L, int sms) {
  const int steps = (ring_chains(L) + ring_chains_a_step(L) - 1) / ring_chains_a_step(L);
  const int least = ((1 << (L - 1)) + kRingGradWarps - 1) / kRingGradWarps;
  int ctas = steps < 8 ? steps : 8;
  while (ctas > least && ctas * n > sms) --ctas;
  return ctas;
}

// The sweeps: left (energy; components kept for the gradient when `keep`),
// right, or both at once; then the gradient from the kept components.
cudaError_t launch_ring_sweeps(const RingParams &P, bool left, bool right, bool keep, cudaStream_t s);
cudaError_t launch_ring_gradient(const RingParams &P, cudaStream_t s);

}  // namespace rsv
