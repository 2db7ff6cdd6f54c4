// Energy and adjoint gradient of circuits of 13 to 16 qubits whose state passes
// through a cluster of 1 to 2^(n-12) CTAs in tiles of 4096 amplitudes, 16 a
// thread: two passes over psi (and lambda) a layer and direction, and a barrier
// of the circuit's CTAs between them.  The vectors are in global memory, where
// they mostly stay in L2.
//
// A low pass takes tiles of the index bits 0..11 and the wires 0..n-5 in three
// register layouts (bits 4..7, then 0..3 within a warp, then 8..11 across the CTA,
// through shared memory), in place.  A high pass takes the wires n-4..n-1, whose
// bits are the registers, with the threads on bits 0..7: no exchange at all; the
// forward applies the RZ phases there and stores through the CNOT ring, the
// backward loads through it, into the circuit's second pair of vectors.  Every
// load and store of a warp covers whole lines.  Gates, phases, sums and their
// corrections are those of the cluster-resident kernel (rsv_cluster.cu), but that
// a theta sum is taken behind its own step's rotations (rotating both vectors
// leaves it but for 1 + k^2, so the wires of the step are no longer pending): psi
// is rotated and on its way through shared memory while lambda still arrives.
//
// With several tiles a CTA the next tile's loads run ahead: into registers in the
// forward, by cp.async into the thread's own slots in the backward (a high pass
// uses the exchange buffers, a low pass a third one for psi, where the tables of
// a deep circuit leave room).
//
// What bounds it: FP64, the loads and stores from L2 and the exchanges follow each
// other more than they overlap, since two vectors of 16 amplitudes leave a SM 8
// warps: 15 to 18 us a tile and layer on one CTA a circuit.  128 circuits of n = 16,
// L = 6 keep the FP64 pipe busy 26 % of the time, L2 30 %, L1 and shared memory 39 %,
// and the warps wait for loads first (2.2 for each that issues).  Keeping the state in registers instead costs 25 (n = 13) to 47 us (n =
// 16), bound by the stores into other CTAs.  148 circuits of L = 8, before
// (registers) and now: n = 13 0.39 -> 0.26 ms, n = 14 1.13 -> 0.59, n = 15 2.61 ->
// 1.23, n = 16 6.25 -> 2.64; 4096 mixed circuits 23.6 -> 12.2 ms; one of n = 16, L =
// 8 258 -> 184 us.  Without the loads ahead 128 of n = 16, L = 6 on one CTA each
// took 2.04 ms (1.90).
#include <cuda_runtime.h>

#include <atomic>

#include "rsv_resident.cuh"

namespace rsv {
namespace {

template <int n_>
struct Tiled {
  static constexpr int n = n_, N = n_, R = 4, threads = 256, warps = 8;
  static constexpr int tables = (N - R + 3) / 4 + 1;
  static constexpr int H = n - 4;            // first wire of the high pass
  static constexpr int tiles = 1 << (n - 12);
  static constexpr int low_wires = n - 4;    // wires of the low pass
};

constexpr size_t kTileBuf = size_t{16} << 12;  // one exchange buffer
constexpr size_t kMostTileSmem = kMostSmem - 256;  // beside the static part
// A layer's record: theta sums of 16 wires, then register bits (4), total, lane bits (5), tile bits (4)
constexpr int kRecTile = 26;

// Barrier of the circuit's CTAs; what they stored to global memory is there for
// loads that go to L2.
__device__ __forceinline__ void sync_circuit(unsigned ctas) {
  if (ctas > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
}

// `ahead`: a tile's loads go out while the one before is worked on (for several
// tiles a CTA, and room for a third buffer).
template <int n, bool ahead>
__device__ __forceinline__ void run_tiles(const ClusterArgs &A, const ClusterItem &item, unsigned char *smem,
                                          double2 *scratch, unsigned rank, unsigned ctas) {
  using G = Tiled<n>;
  constexpr int H = G::H, nt = G::tables, LW = G::low_wires;
  constexpr unsigned size = 1u << n, hi = 1u << H;
  const int L = item.L;
  const unsigned t = threadIdx.x;
  const int lane = t & 31, warp = t >> 5;
  unsigned char *bufP = smem, *bufL = smem + kTileBuf;
  unsigned char *bufN = smem + 2 * kTileBuf;
  const Tables T =
      build_tables<G>(A.params ? A.params + item.param_off : nullptr, A.coef, rank == 0 ? A.coef_out : nullptr, L, smem,
                      (ahead ? 3 : 2) * kTileBuf);
  __syncthreads();
  // the forward ends on the first vector after an odd number of layers
  double2 *psi0 = scratch, *psi1 = scratch + size, *lam0 = scratch + 2 * size, *lam1 = scratch + 3 * size;
  auto swap = [](double2 *&a, double2 *&b) {
    double2 *s = a;
    a = b;
    b = s;
  };

  // low-pass layouts: register bits 4..7 (B), 0..3 (C), 8..11 (A); the thread's
  // amplitude of register 0 in a tile, and its exchange slots
  const unsigned idx_b = spread(t, 4, 4), idx_c = t << 4, idx_a = t;
  const unsigned slot_b = slot(idx_b), slot_c = slot(idx_c), slot_a = slot(idx_a);
  auto bit_b = [](int j) { return slot(1u << (4 + j)); };
  auto bit_c = [](int j) { return slot(1u << j); };
  auto bit_a = [](int j) { return slot(1u << (8 + j)); };
  // J swaps of four wires as register numbers
  auto swaps = [](unsigned flip, int first) { return (flip >> first) & 15u; };
  auto put = [&](const double2 (&a)[16], unsigned char *buf, unsigned base, auto &&bit) {
    for_registers<4>(base, bit, [&](int r, unsigned p) { *reinterpret_cast<double2 *>(buf + p) = a[r]; });
  };
  auto get = [&](double2 (&a)[16], const unsigned char *buf, unsigned base, auto &&bit) {
    for_registers<4>(base, bit, [&](int r, unsigned p) { a[r] = *reinterpret_cast<const double2 *>(buf + p); });
  };
  auto swapped = [](unsigned base, unsigned x, auto &&bit) {
#pragma unroll
    for (int j = 0; j < 4; ++j) base ^= (0u - ((x >> j) & 1u)) & bit(j);
    return base;
  };
  // high pass: thread t holds x = tile << 8 | t with register r << H
  auto ring_bit = [](int j) { return ring_map(1u << (H + j), n); };
  // phase of the thread's low eight bits, and of a tile's bits 8..H-1
  auto phase_low = [&](const double2 *tab) { return cmul(tab[t & 15], tab[16 + ((t >> 4) & 15)]); };
  auto phase_tile = [&](const double2 *tab, unsigned tile) {
    double2 z = tab[32 + (tile & 15)];
    if constexpr (nt > 4) z = cmul(z, tab[48 + (tile >> 4)]);
    return z;
  };

  if (A.resume) {
    if (L % 2 == 0) swap(psi0, psi1);
  } else {
  // ---- forward
  {
    const double2 z0 = phase_low(T.prod);
    for (unsigned tile = rank; tile < G::tiles; tile += ctas) {  // layer 0: the product state
      const double2 z = cmul(z0, phase_tile(T.prod, tile));
      for_registers<4>(ring_map(tile << 8 | t, n), ring_bit,
                       [&](int r, unsigned y) { psi0[y] = cmul(z, T.prod[16 * (nt - 1) + r]); });
    }
  }
  for (int l = 1; l < L; ++l) {
    const unsigned flip = T.flip[l];
    const double *rot = T.rot + l * n;
    sync_circuit(ctas);  // the state is there
    {
      double2 a[16], next[16];
      auto load = [&](double2 (&v)[16], unsigned tile) {
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = __ldcg(psi0 + (tile << 12 | idx_b | r << 4));
      };
      if constexpr (ahead) load(next, rank);
      for (unsigned tile = rank; tile < G::tiles; tile += ctas) {
        if constexpr (ahead) {
#pragma unroll
          for (int r = 0; r < 16; ++r) a[r] = next[r];
          if (tile + ctas < G::tiles) load(next, tile + ctas);
        } else {
          load(a, tile);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) rotate<4>(a, j, rot[4 + j]);
        put(a, bufP, swapped(slot_b, swaps(flip, 4), bit_b), bit_b);
        __syncwarp();
        get(a, bufP, slot_c, bit_c);
#pragma unroll
        for (int j = 0; j < 4; ++j) rotate<4>(a, j, rot[j]);
        put(a, bufP, swapped(slot_c, swaps(flip, 0), bit_c), bit_c);
        __syncthreads();
        get(a, bufP, slot_a, bit_a);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (8 + j < LW) rotate<4>(a, j, rot[8 + j]);
        const unsigned x = swaps(flip & ((1u << LW) - 1), 8);
#pragma unroll
        for (int r = 0; r < 16; ++r) psi0[tile << 12 | idx_a | (static_cast<unsigned>(r) ^ x) << 8] = a[r];
        __syncthreads();  // the buffer is read
      }
    }
    sync_circuit(ctas);
    {
      const double2 *tab = T.phase + static_cast<size_t>(l) * nt * 16;
      double2 z0 = phase_low(tab);
      z0.x *= T.scale[l];
      z0.y *= T.scale[l];
      const unsigned x = swaps(flip, H);
      double2 a[16], next[16];
      auto load = [&](double2 (&v)[16], unsigned tile) {
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = __ldcg(psi0 + (tile << 8 | t | static_cast<unsigned>(r) * hi));
      };
      if constexpr (ahead) load(next, rank);
      for (unsigned tile = rank; tile < G::tiles; tile += ctas) {
        if constexpr (ahead) {
#pragma unroll
          for (int r = 0; r < 16; ++r) a[r] = next[r];
          if (tile + ctas < G::tiles) load(next, tile + ctas);
        } else {
          load(a, tile);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) rotate<4>(a, j, rot[H + j]);
        const double2 z = cmul(z0, phase_tile(tab, tile));
        for_registers<4>(swapped(ring_map(tile << 8 | t, n), x, ring_bit), ring_bit, [&](int r, unsigned y) {
          psi1[y] = cmul(a[r], cmul(z, tab[16 * (nt - 1) + r]));
        });
      }
    }
    swap(psi0, psi1);
  }
  sync_circuit(ctas);
  // ---- lambda = H psi and the energy, on low tiles
  double energy = 0.0;
  const bool keep = A.grad_out != nullptr || A.lam != nullptr;
  for (unsigned tile = rank; tile < G::tiles; tile += ctas) {
    __syncthreads();  // the buffer is read
    double2 a[16], b[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) a[r] = __ldcg(psi0 + (tile << 12 | idx_a | r << 8));
    put(a, bufP, slot_a, bit_a);
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      b[r] = make_double2(0.0, 0.0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b[r].x += a[r ^ (1 << j)].x;
        b[r].y += a[r ^ (1 << j)].y;
      }
    }
#pragma unroll
    for (int w = 12; w < n; ++w)
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const double2 q = __ldcg(psi0 + ((tile << 12 | idx_a | r << 8) ^ (1u << w)));
        b[r].x += q.x;
        b[r].y += q.y;
      }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w)
      for_registers<4>(slot_a ^ slot(1u << w), bit_a, [&](int r, unsigned p) {
        const double2 q = *reinterpret_cast<const double2 *>(bufP + p);
        b[r].x += q.x;
        b[r].y += q.y;
      });
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const unsigned x = tile << 12 | idx_a | r << 8;
      const unsigned turn = ((x << 1) & (size - 1)) | (x >> (n - 1));
      const double d = static_cast<double>(2 * __popc(x ^ turn) - n);
      b[r] = make_double2(fma(d, a[r].x, -item.h * b[r].x), fma(d, a[r].y, -item.h * b[r].y));
      energy = fma(a[r].x, b[r].x, energy);
      energy = fma(a[r].y, b[r].y, energy);
      if (keep) lam0[x] = b[r];
    }
  }
  energy = warp_sum(energy);
  if (lane == 0) T.red[warp] = energy;
  __syncthreads();
  double *sum = T.red + 64 * G::warps;
  if (t == 0) {
    double s = 0.0;
    for (int k = 0; k < G::warps; ++k) s += T.red[k];
    *sum = s;
  }
  sync_circuit(ctas);  // the sums and H psi are there
  if (rank == 0 && t == 0 && A.energy_out != nullptr) {
    double s = *sum;
    for (unsigned k = 1; k < ctas; ++k) s += load_cluster(cluster_address(shared_address(sum), k));
    A.energy_out[item.index] = s;
  }
  }
  if (A.grad_out == nullptr) {
    sync_circuit(ctas);  // the first CTA has read the others' sums: their shared memory may go
    return;
  }

  // ---- backward
  for (int l = L - 1; l >= 0; --l) {
    const unsigned flip = T.flip[l];
    const double *rot = T.rot + l * n;
    {  // high pass: through P^-1, phi sums, D^+ K, the wires H..n-1
      const double2 *tab = T.phase + static_cast<size_t>(l) * nt * 16;
      double2 z0 = phase_low(tab);
      z0.x *= T.scale[l];
      z0.y *= T.scale[l];
      const unsigned x = swaps(flip, H);
      double theta[4] = {0.0, 0.0, 0.0, 0.0}, one[4] = {0.0, 0.0, 0.0, 0.0}, tot = 0.0;
      double part[4] = {0.0, 0.0, 0.0, 0.0};  // totals of the tiles with bit 8 + j
      auto start = [&](unsigned tile) {
        for_registers<4>(swapped(ring_map(tile << 8 | t, n), x, ring_bit), ring_bit, [&](int r, unsigned y) {
          fetch(bufP, r, psi0 + y);
          fetch(bufL, r, lam0 + y);
        });
      };
      if constexpr (ahead) start(rank);
      for (unsigned tile = rank; tile < G::tiles; tile += ctas) {
        double2 p[16], q[16];
        if constexpr (ahead) {
          fetched();
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            p[r] = take(bufP, r);
            q[r] = take(bufL, r);
          }
          if (tile + ctas < G::tiles) start(tile + ctas);
        } else {
          for_registers<4>(swapped(ring_map(tile << 8 | t, n), x, ring_bit), ring_bit, [&](int r, unsigned y) {
            p[r] = __ldcg(psi0 + y);
            q[r] = __ldcg(lam0 + y);
          });
        }
        double sum = 0.0;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const double v = fma(q[r].x, p[r].y, -q[r].y * p[r].x);
          sum += v;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((r >> j) & 1) one[j] += v;
        }
        tot += sum;
#pragma unroll
        for (int j = 0; j < n - 12; ++j) part[j] += ((tile >> j) & 1) ? sum : 0.0;
        const double2 z = cmul(z0, phase_tile(tab, tile));
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const double2 f = cmul(z, tab[16 * (nt - 1) + r]);
          p[r] = cmul_conj(p[r], f);
          q[r] = cmul_conj(q[r], f);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          rotate<4>(p, j, -rot[H + j]);
          rotate<4>(q, j, -rot[H + j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) theta[j] += theta_sum<4>(p, q, j);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const unsigned at = tile << 8 | t | static_cast<unsigned>(r) * hi;
          psi1[at] = p[r];
          lam1[at] = q[r];
        }
      }
      double sums[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) sums[i] = 0.0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sums[H + j] = theta[j];
        sums[kRecPhi + j] = one[j];
        sums[kRecTile + j] = part[j];
      }
      sums[kRecTotal] = tot;
#pragma unroll
      for (int j = 0; j < 5; ++j) sums[kRecLane + j] = ((lane >> j) & 1) ? tot : 0.0;
      const double s = warp_sums32(sums, lane);
      T.red[32 * warp + lane] = s;
      if (lane == kRecTotal) T.tot[l * 8 + warp] = s;
    }
    swap(psi0, psi1);
    swap(lam0, lam1);
    sync_circuit(ctas);  // the vectors and the warps' sums are there
    if (warp == 0) {
      double sum = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += T.red[32 * k + lane];
      T.rec[l * kRec + lane] = sum;
    }
    {  // low pass, in place
      double theta[12];
#pragma unroll
      for (int i = 0; i < 12; ++i) theta[i] = 0.0;
      const unsigned xb = swaps(flip, 4), xc = swaps(flip, 0), xa = swaps(flip & ((1u << LW) - 1), 8);
      auto start = [&](unsigned tile) {
#pragma unroll
        for (int r = 0; r < 16; ++r) fetch(bufN, r, psi0 + (tile << 12 | idx_b | (static_cast<unsigned>(r) ^ xb) << 4));
      };
      if constexpr (ahead) start(rank);
      for (unsigned tile = rank; tile < G::tiles; tile += ctas) {
        double2 p[16], q[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) q[r] = __ldcg(lam0 + (tile << 12 | idx_b | (static_cast<unsigned>(r) ^ xb) << 4));
        if constexpr (ahead) {
          fetched();
#pragma unroll
          for (int r = 0; r < 16; ++r) p[r] = take(bufN, r);
          if (tile + ctas < G::tiles) {
            start(tile + ctas);
            if (t == 0)
              asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lam0 + ((tile + ctas) << 12)), "r"(65536)
                           : "memory");
          }
        } else {
#pragma unroll
          for (int r = 0; r < 16; ++r) p[r] = __ldcg(psi0 + (tile << 12 | idx_b | (static_cast<unsigned>(r) ^ xb) << 4));
        }
        // psi's part of a step first: lambda may still be on its way
        auto undo = [&](double2 (&a)[16], int first) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (first + j < LW) rotate<4>(a, j, -rot[first + j]);
        };
        auto sums = [&](int first) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (first + j < LW) theta[first + j] += theta_sum<4>(p, q, j);
        };
        undo(p, 4);
        put(p, bufP, slot_b, bit_b);
        undo(q, 4);
        put(q, bufL, slot_b, bit_b);
        sums(4);
        __syncwarp();
        get(p, bufP, swapped(slot_c, xc, bit_c), bit_c);
        get(q, bufL, swapped(slot_c, xc, bit_c), bit_c);
        undo(p, 0);
        put(p, bufP, slot_c, bit_c);
        undo(q, 0);
        put(q, bufL, slot_c, bit_c);
        sums(0);
        __syncthreads();
        get(p, bufP, swapped(slot_a, xa, bit_a), bit_a);
        get(q, bufL, swapped(slot_a, xa, bit_a), bit_a);
        undo(p, 8);
        undo(q, 8);
        if (l > 0) {
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            psi0[tile << 12 | idx_a | r << 8] = p[r];
            lam0[tile << 12 | idx_a | r << 8] = q[r];
          }
        }
        sums(8);
        __syncthreads();  // the buffers are read
      }
      double all[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) all[i] = i < LW ? theta[i < 12 ? i : 0] : 0.0;
      const double v = warp_sums32(all, lane);
      T.red[32 * (8 + warp) + lane] = v;
    }
    sync_circuit(ctas);  // the vectors and the warps' sums are there
    if (warp == 0) {
      double sum = 0.0;
#pragma unroll
      for (int k = 8; k < 16; ++k) sum += T.red[32 * k + lane];
      T.rec[l * kRec + lane] += sum;
    }
  }
  sync_circuit(ctas);
  auto total = [&](const double *p) {  // over the CTAs
    double s = 0.0;
    if (ctas == 1) return *p;
    for (unsigned k = 0; k < ctas; ++k) s += load_cluster(cluster_address(shared_address(p), k));
    return s;
  };
  for (int e = rank * 256 + t; e < L * n * 2; e += ctas * 256) {
    const int l = e / (2 * n), w = e % (2 * n) / 2;
    const double *rec = T.rec + l * kRec;
    double out;
    if ((e & 1) == 0) {
      // prod (1 + k^2) over the wires still pending behind the step: those of the
      // low pass, then without 4..7, without 0..3, none
      const unsigned low = (1u << LW) - 1;
      const unsigned pending = w >= H ? low : (w >= 8 ? 0u : (w < 4 ? low & ~0xffu : low & ~0xf0u));
      double s = 1.0;
      for (int v = 0; v < n; ++v)
        if ((pending >> v) & 1) s *= fma(T.rot[l * n + v], T.rot[l * n + v], 1.0);
      out = total(rec + w) * s;
    } else {
      double b = 0.0;
      if (w < 5) {
        b = total(rec + kRecLane + w);
      } else if (w < 8) {
        for (int k = 0; k < 8; ++k)
          if ((k >> (w - 5)) & 1) b += total(T.tot + l * 8 + k);
      } else if (w < H) {
        b = total(rec + kRecTile + w - 8);
      } else {
        b = total(rec + kRecPhi + w - H);
      }
      out = total(rec + kRecTotal) - 2.0 * b;
      if (w >= H && ((T.flip[l] >> w) & 1)) out = -out;  // its register bit is 1 where the wire is 0
    }
    A.grad_out[item.param_off + e] = out;
  }
  sync_circuit(ctas);  // the tables are read
}

template <int n, bool ahead>
__global__ void __launch_bounds__(256, 1) tile_circuit_kernel(const __grid_constant__ ClusterArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int next;
  const unsigned ctas = 1u << A.shape.log_ctas, cluster = blockIdx.x >> A.shape.log_ctas, rank = blockIdx.x & (ctas - 1);
  double2 *scratch = A.memory + (static_cast<size_t>(cluster) << (n + 2));
  if (A.counter == nullptr) {
    run_tiles<n, ahead>(A, A.items ? A.items[cluster] : A.item, smem, scratch, rank, ctas);
    return;
  }
  sync_circuit(ctas);  // every CTA of the cluster runs
  for (;;) {           // as many clusters as fit take the circuits in order
    if (rank == 0 && threadIdx.x == 0) {
      const int i = atomicAdd(A.counter, 1);
      next = i;
      for (unsigned k = 1; k < ctas; ++k) store_cluster_u32(cluster_address(shared_address(&next), k), i);
    }
    sync_circuit(ctas);
    const int i = next;
    if (i >= A.count) return;
    run_tiles<n, ahead>(A, A.items[i], smem, scratch, rank, ctas);  // (ends in a barrier: everyone has read `next`)
  }
}

template <int n>
struct TileShape {
  // A third buffer where the deepest circuit leaves room and a CTA has several tiles.
  static bool ahead(int log_ctas, int max_layers) {
    return (1 << (n - 12 - log_ctas)) >= 4 && smem(max_layers, true) <= kMostTileSmem;
  }
  static size_t smem(int max_layers, bool third) {
    return (third ? 3 : 2) * kTileBuf + table_bytes<Tiled<n>>(max_layers);
  }
  template <bool third>
  static cudaError_t configure(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at, int log_ctas, int max_layers, int count) {
    static std::atomic<unsigned long long> smem_done{0}, size_done{0};
    cudaError_t e = set_smem_limit_once(tile_circuit_kernel<n, third>, kMostTileSmem, smem_done);
    if (e == cudaSuccess && log_ctas > 3) e = allow_any_cluster_once(tile_circuit_kernel<n, third>, size_done);
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(static_cast<unsigned>(count) << log_ctas);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem(max_layers, third);
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1u << log_ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return e;
  }
  template <bool third>
  static cudaError_t launch(const ClusterArgs &A, cudaStream_t s) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    const cudaError_t e =
        configure<third>(cfg, at, A.shape.log_ctas, A.max_layers, A.counter ? A.clusters : A.count);
    if (e != cudaSuccess) return e;
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, tile_circuit_kernel<n, third>, A);
  }
  template <bool third>
  static cudaError_t capacity(int log_ctas, int max_layers, int *clusters) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    const cudaError_t e = configure<third>(cfg, at, log_ctas, max_layers, 1);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveClusters(clusters, tile_circuit_kernel<n, third>, &cfg);
  }
};

template <typename F>
bool with_tiles(int n, int log_ctas, F &&f) {
  if (log_ctas < 0 || log_ctas > n - 12) return false;
  switch (n) {
    case 13: f(TileShape<13>{}); return true;
    case 14: f(TileShape<14>{}); return true;
    case 15: f(TileShape<15>{}); return true;
    case 16: f(TileShape<16>{}); return true;
    default: return false;
  }
}

}  // namespace

cudaError_t launch_tiles(const ClusterArgs &A, cudaStream_t s) {
  cudaError_t e = cudaErrorInvalidValue;
  with_tiles(A.n, A.shape.log_ctas, [&](auto shape) {
    using S = decltype(shape);
    e = S::ahead(A.shape.log_ctas, A.max_layers) ? S::template launch<true>(A, s) : S::template launch<false>(A, s);
  });
  return e;
}

cudaError_t tile_capacity(int n, ClusterShape h, int max_layers, int *clusters) {
  cudaError_t e = cudaSuccess;
  with_tiles(n, h.log_ctas, [&](auto shape) {
    using S = decltype(shape);
    if (S::smem(max_layers, false) > kMostTileSmem) return;
    e = S::ahead(h.log_ctas, max_layers) ? S::template capacity<true>(h.log_ctas, max_layers, clusters)
                                         : S::template capacity<false>(h.log_ctas, max_layers, clusters);
  });
  return e;
}

}  // namespace rsv
