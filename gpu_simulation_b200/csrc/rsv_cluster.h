// Circuits whose state lives in the registers and shared memory of one
// thread-block cluster (rsv_cluster.cu): host-callable launchers.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace rsv {

constexpr int kClusterMaxQubits = 16;
constexpr int kClusterMaxLayers = 64;

// One circuit of a launch; every circuit of a launch has n qubits.
struct ClusterItem {
  int L;
  int index;              // energy_out[index]
  long long param_off;    // params, grad_out: + param_off
  double h;
};

// How a launch spreads a circuit: 2^log_ctas CTAs, 2^register_bits amplitudes a
// thread; with checkpoints the backward reads psi from memory.  Tiled: psi and
// lambda are in memory, and the CTAs work through them tile by tile.
struct ClusterShape {
  int log_ctas, register_bits;
  bool checkpoints;
  bool tiled = false;
};

struct ClusterArgs {
  int n;
  ClusterShape shape;
  int count;                   // circuits
  int clusters;                // with a counter (tiled): clusters that take them in turn
  int *counter;                // 0 at the launch, or null: one cluster a circuit
  double2 *memory;             // clusters * cluster_memory_values(n, shape, max_layers)
  const ClusterItem *items;    // [count], or null: the one circuit `item`
  ClusterItem item;
  int max_layers;              // largest L of the circuits
  const double *params;        // angles, or null: `coef` (one circuit)
  const double4 *coef;         // [L * n] (cos t/2, sin t/2, cos p/2, sin p/2)
  double4 *coef_out;           // or null: the one circuit's are written here
  double *energy_out;          // or null
  double *grad_out;            // or null: no backward
  // One circuit only: the forward call leaves psi (without checkpoints) and
  // H psi here (tiled: in `memory`), and with `resume` a later call starts from them (and the
  // checkpoints) and runs the backward alone.
  double2 *psi, *lam;
  int resume;
  int polls;                   // whole device: how often a CTA polls a barrier before it gives up
};

// Polls of a whole-device barrier: about a second.
constexpr int kGridPolls = 1 << 21;

// Global memory of a cluster: psi's checkpoints, or a tiled circuit's vectors.
size_t cluster_memory_values(int n, ClusterShape h, int max_layers);
cudaError_t launch_cluster(const ClusterArgs &A, cudaStream_t s);
// Clusters of that shape that fit the device at once (0: none).
cudaError_t cluster_capacity(int n, ClusterShape h, int max_layers, int *clusters);

// Tiled circuits (rsv_tiles.cu); the functions above go there.
cudaError_t launch_tiles(const ClusterArgs &A, cudaStream_t s);
cudaError_t tile_capacity(int n, ClusterShape h, int max_layers, int *clusters);

// One circuit of more than kClusterMaxQubits (rsv_grid.cu): tiled on the whole
// device; the functions above go there.
constexpr int kGridMaxQubits = 20;
size_t grid_memory_values(int n, int max_layers);
cudaError_t launch_grid(const ClusterArgs &A, cudaStream_t s);
cudaError_t grid_capacity(int n, int max_layers, int *circuits);
// On the device: non-zero where the circuit's last call gave up; all of its results are NaN.
const unsigned *grid_lost_flag(const ClusterArgs &A);

}  // namespace rsv
