// Energy and adjoint gradient of one circuit of 17 to 20 qubits in one launch:
// the tiled kernel (rsv_tiles.cu) on one CTA a SM, with a barrier of the whole
// grid between passes.
//
// Tiles have 4096 amplitudes, 16 a thread, q = 24 - n.  A low pass takes the index bits
// 0..11 and their wires as there.  A high pass takes the bits 0..q-1 (so that
// loads and stores are whole lines) and 12..n-1: as local bits u = 0..q-1 and
// q..11.  Its wires are n-4..n-1 in one register layout (u = 8..11) and what is
// left of 12..n-5 in another (u = q..q+3), an exchange through shared memory
// between them.
//
// Before, every pass was a launch of the general tile-pass kernels (two passes a
// layer and direction, 20 qubits: forward 12 to 13.5 us, backward 25 to 31),
// with the first three layers as matrix products.  A layer now takes 27 to 29 us from
// 17 to 19 qubits, a tile or less a CTA, and 50 us with 20 qubits: 108 of 148 CTAs
// have a second tile, which the others wait for (issuing its loads ahead, as
// rsv_tiles.cu does, made L = 8 456 us instead of the 422 of that time).  More warps
// wait at a barrier than for anything else (n = 20: 3.7 for each that issues; next are
// loads with 2.3); FP64 and L2 are each busy a fifth of the time.  Energy and gradient
// at L = 8: n = 17 330 -> 219 us, n = 18 331 -> 220, n = 19 349 -> 245, n = 20 493 -> 415.
#include <cuda_runtime.h>

#include <atomic>

#include "rsv_resident.cuh"

namespace rsv {
namespace {

template <int n_>
struct Grid {
  static constexpr int n = n_, N = n_, R = 4, threads = 256, warps = 8;
  static constexpr int tables = (N - R + 3) / 4 + 1;
  static constexpr int q = 24 - n, tiles = 1 << (n - 12), top = n - 4;
};

constexpr size_t kGridBuf = size_t{16} << 12;  // one exchange buffer
constexpr size_t kMostGridSmem = kMostSmem - 256;
constexpr int kMostGridCtas = 256;
// A layer's record of a CTA: theta sums of the wires top..n-1, 12..15, then phi
// values of register bits, total, lane bits, tile bits, warp bits; theta sums of 0..11
constexpr int kGridRec = 48, kGridHigh = 4, kGridPhi = 8, kGridTotal = 12, kGridLane = 13, kGridTile = 18, kGridWarp = 26,
              kGridLow = 32;
// Behind the four vectors: records [layer][value][CTA], energies [CTA], then
struct GridState {
  unsigned arrived;  // CTAs that came to a barrier, all barriers; 0 at the launch
  unsigned lost;     // set by a launch that gave up; 0 at a call's first launch
};
constexpr unsigned kGridVoid = 1u << 31;  // of `arrived`: a CTA gave up waiting

// Barrier of the grid: what its CTAs stored is there for loads that go to L2.
// A CTA looks `polls` times whether the others have arrived, then it gives up for
// all of them.  It does so in the word that counts them, and only while that is
// still short: so either no CTA passes a barrier or every one does, and none is
// left with results that the others void.
__device__ __forceinline__ bool sync_grid(GridState *S, unsigned &target, int polls) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    unsigned seen = atomicAdd(&S->arrived, 1u) + 1;
    // (a void word is above every target)
#pragma unroll 1
    for (int k = 0; seen < target && k < polls; ++k) {
      // (the second load spaces the polls out: n = 20, L = 8 418 us against 434 without it, n = 17 166 at
      // L = 6 against 171)
      unsigned spare;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&S->arrived) : "memory");
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(spare) : "l"(&S->lost) : "memory");
    }
#pragma unroll 1
    while (seen < target) {  // (no more turns than CTAs: each one that fails found another arrival)
      const unsigned was = atomicCAS(&S->arrived, seen, seen | kGridVoid);
      seen = was == seen ? seen | kGridVoid : was;
    }
    __threadfence();
    ok = seen < kGridVoid;
  }
  __syncthreads();
  return ok != 0;
}

__host__ __device__ inline size_t grid_doubles(int max_layers) {  // behind the vectors, without the state
  return static_cast<size_t>(max_layers) * kGridRec * kMostGridCtas + kMostGridCtas;
}
__host__ __device__ inline GridState *grid_state(const ClusterArgs &A, int n) {
  return reinterpret_cast<GridState *>(reinterpret_cast<double *>(A.memory + (size_t{4} << n)) + grid_doubles(A.max_layers));
}

template <int n>
__device__ __forceinline__ bool run_grid(const ClusterArgs &A, unsigned char *smem) {
  using G = Grid<n>;
  constexpr int q = G::q, top = G::top, nt = G::tables;
  constexpr unsigned size = 1u << n;
  const ClusterItem &item = A.item;
  const int L = item.L;
  const unsigned t = threadIdx.x, cta = blockIdx.x, ctas = gridDim.x;
  const int lane = t & 31, warp = t >> 5;
  unsigned char *bufP = smem, *bufL = smem + kGridBuf;
  double *recs = reinterpret_cast<double *>(A.memory + (size_t{4} << n));
  double *energies = recs + static_cast<size_t>(A.max_layers) * kGridRec * kMostGridCtas;
  GridState *S = grid_state(A, n);
  unsigned arrivals = 0;
  const Tables T = build_tables<G>(A.params ? A.params + item.param_off : nullptr, A.coef, cta == 0 ? A.coef_out : nullptr,
                                   L, smem, 2 * kGridBuf);
  __syncthreads();
  // the forward ends on the first vector after an odd number of layers
  double2 *psi0 = A.memory, *psi1 = psi0 + size, *lam0 = psi1 + size, *lam1 = lam0 + size;
  auto swap = [](double2 *&a, double2 *&b) {
    double2 *s = a;
    a = b;
    b = s;
  };

  // layouts of a tile: the thread's local amplitude of register 0 and its slots
  const unsigned u_b = spread(t, 4, 4), u_c = t << 4, u_a = t, u_h = spread(t, q, 4);
  const unsigned slot_b = slot(u_b), slot_c = slot(u_c), slot_a = slot(u_a), slot_h = slot(u_h);
  auto bit_b = [](int j) { return slot(1u << (4 + j)); };
  auto bit_c = [](int j) { return slot(1u << j); };
  auto bit_a = [](int j) { return slot(1u << (8 + j)); };
  auto bit_h = [](int j) { return slot(1u << (q + j)); };
  auto ring_bit = [](int j) { return ring_map(1u << (top + j), n); };
  // index of a high tile's local amplitude
  auto index = [](unsigned tile, unsigned u) { return (u & ((1u << q) - 1)) | tile << q | (u >> q) << 12; };
  // J swaps of four wires as register numbers; of the second high layout's
  auto swaps = [](unsigned flip, int first) { return (flip >> first) & 15u; };
  auto swaps_h = [](unsigned flip) { return ((flip & ((1u << top) - 1)) >> 12) & 15u; };
  auto swapped = [](unsigned base, unsigned x, auto &&bit) {
#pragma unroll
    for (int j = 0; j < 4; ++j) base ^= (0u - ((x >> j) & 1u)) & bit(j);
    return base;
  };
  auto put = [&](const double2 (&a)[16], unsigned char *buf, unsigned base, auto &&bit) {
    for_registers<4>(base, bit, [&](int r, unsigned p) { *reinterpret_cast<double2 *>(buf + p) = a[r]; });
  };
  auto get = [&](double2 (&a)[16], const unsigned char *buf, unsigned base, auto &&bit) {
    for_registers<4>(base, bit, [&](int r, unsigned p) { a[r] = *reinterpret_cast<const double2 *>(buf + p); });
  };
  auto phase = [&](const double2 *tab, unsigned x) {  // of the bits below the registers
    double2 z = tab[x & 15];
#pragma unroll
    for (int g = 1; g < nt - 1; ++g) z = cmul(z, tab[16 * g + ((x >> (4 * g)) & 15)]);
    return z;
  };

  if (A.resume) {
    if (L % 2 == 0) swap(psi0, psi1);
  } else {
    // ---- forward
    for (unsigned tile = cta; tile < G::tiles; tile += ctas) {  // layer 0: the product state
      const unsigned x = index(tile, u_a);
      const double2 z = phase(T.prod, x);
      for_registers<4>(ring_map(x, n), ring_bit,
                       [&](int r, unsigned y) { psi0[y] = cmul(z, T.prod[16 * (nt - 1) + r]); });
    }
    for (int l = 1; l < L; ++l) {
      const unsigned flip = T.flip[l];
      const double *rot = T.rot + l * n;
      double2 a[16];
      if (!sync_grid(S, arrivals, A.polls)) return false;
      for (unsigned tile = cta; tile < G::tiles; tile += ctas) {
#pragma unroll
        for (int r = 0; r < 16; ++r) a[r] = __ldcg(psi0 + (tile << 12 | u_b | r << 4));
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
        for (int j = 0; j < 4; ++j) rotate<4>(a, j, rot[8 + j]);
        const unsigned x = swaps(flip, 8);
#pragma unroll
        for (int r = 0; r < 16; ++r) psi0[tile << 12 | u_a | (static_cast<unsigned>(r) ^ x) << 8] = a[r];
        __syncthreads();  // the buffer is read
      }
      if (!sync_grid(S, arrivals, A.polls)) return false;
      const double2 *tab = T.phase + static_cast<size_t>(l) * nt * 16;
      const double scale = T.scale[l];
      for (unsigned tile = cta; tile < G::tiles; tile += ctas) {
#pragma unroll
        for (int r = 0; r < 16; ++r) a[r] = __ldcg(psi0 + (index(tile, u_h) | static_cast<unsigned>(r) << 12));
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (12 + j < top) rotate<4>(a, j, rot[12 + j]);
        put(a, bufP, swapped(slot_h, swaps_h(flip), bit_h), bit_h);
        __syncthreads();
        get(a, bufP, slot_a, bit_a);
#pragma unroll
        for (int j = 0; j < 4; ++j) rotate<4>(a, j, rot[top + j]);
        const unsigned x = index(tile, u_a);
        double2 z = phase(tab, x);
        z.x *= scale;
        z.y *= scale;
        for_registers<4>(swapped(ring_map(x, n), swaps(flip, top), ring_bit), ring_bit, [&](int r, unsigned y) {
          psi1[y] = cmul(a[r], cmul(z, tab[16 * (nt - 1) + r]));
        });
        __syncthreads();  // the buffer is read
      }
      swap(psi0, psi1);
    }
    if (!sync_grid(S, arrivals, A.polls)) return false;
    // ---- lambda = H psi and the energy, on low tiles
    const bool keep = A.grad_out != nullptr || A.lam != nullptr;
    double energy = 0.0;
    for (unsigned tile = cta; tile < G::tiles; tile += ctas) {
      __syncthreads();  // the buffer is read
      double2 a[16], b[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) a[r] = __ldcg(psi0 + (tile << 12 | u_a | r << 8));
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
          const double2 v = __ldcg(psi0 + ((tile << 12 | u_a | r << 8) ^ (1u << w)));
          b[r].x += v.x;
          b[r].y += v.y;
        }
      __syncthreads();
#pragma unroll
      for (int w = 0; w < 8; ++w)
        for_registers<4>(slot_a ^ slot(1u << w), bit_a, [&](int r, unsigned p) {
          const double2 v = *reinterpret_cast<const double2 *>(bufP + p);
          b[r].x += v.x;
          b[r].y += v.y;
        });
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const unsigned x = tile << 12 | u_a | r << 8;
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
    if (t == 0) {
      double s = 0.0;
      for (int k = 0; k < G::warps; ++k) s += T.red[k];
      energies[cta] = s;
    }
    if (!sync_grid(S, arrivals, A.polls)) return false;  // the energies and H psi are there
    if (cta == 0 && warp == 0 && A.energy_out != nullptr) {
      double s = 0.0;
      for (unsigned k = lane; k < ctas; k += 32) s += __ldcg(energies + k);
      s = warp_sum(s);
      if (lane == 0) A.energy_out[item.index] = s;
    }
  }
  if (A.grad_out == nullptr) return true;

  // ---- backward
  for (int l = L - 1; l >= 0; --l) {
    const unsigned flip = T.flip[l];
    const double *rot = T.rot + l * n;
    double *rec = recs + static_cast<size_t>(l) * kGridRec * ctas + cta;
    {  // high pass: through P^-1, phi sums, D^+ K, the wires 12..n-1
      const double2 *tab = T.phase + static_cast<size_t>(l) * nt * 16;
      const double scale = T.scale[l];
      double theta[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, one[4] = {0.0, 0.0, 0.0, 0.0}, tot = 0.0;
      double part = 0.0;  // lane j: total of the tiles with bit j
      for (unsigned tile = cta; tile < G::tiles; tile += ctas) {
        double2 p[16], v[16];
        const unsigned x = index(tile, u_a);
        for_registers<4>(swapped(ring_map(x, n), swaps(flip, top), ring_bit), ring_bit, [&](int r, unsigned y) {
          p[r] = __ldcg(psi0 + y);
          v[r] = __ldcg(lam0 + y);
        });
        double sum = 0.0;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const double s = fma(v[r].x, p[r].y, -v[r].y * p[r].x);
          sum += s;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((r >> j) & 1) one[j] += s;
        }
        tot += sum;
        sum = warp_sum(sum);
        if ((tile >> lane) & 1) part += sum;
        double2 z = phase(tab, x);
        z.x *= scale;
        z.y *= scale;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const double2 f = cmul(z, tab[16 * (nt - 1) + r]);
          p[r] = cmul_conj(p[r], f);
          v[r] = cmul_conj(v[r], f);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          rotate<4>(p, j, -rot[top + j]);
          rotate<4>(v, j, -rot[top + j]);
        }
        put(p, bufP, slot_a, bit_a);
        put(v, bufL, slot_a, bit_a);
#pragma unroll
        for (int j = 0; j < 4; ++j) theta[j] += theta_sum<4>(p, v, j);
        __syncthreads();
        get(p, bufP, swapped(slot_h, swaps_h(flip), bit_h), bit_h);
        get(v, bufL, swapped(slot_h, swaps_h(flip), bit_h), bit_h);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (12 + j < top) {
            rotate<4>(p, j, -rot[12 + j]);
            rotate<4>(v, j, -rot[12 + j]);
          }
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const unsigned at = index(tile, u_h) | static_cast<unsigned>(r) << 12;
          psi1[at] = p[r];
          lam1[at] = v[r];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (12 + j < top) theta[4 + j] += theta_sum<4>(p, v, j);
        __syncthreads();  // the buffers are read
      }
      double sums[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) sums[i] = 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) sums[j] = theta[j];
#pragma unroll
      for (int j = 0; j < 4; ++j) sums[kGridPhi + j] = one[j];
      sums[kGridTotal] = tot;
#pragma unroll
      for (int j = 0; j < 5; ++j) sums[kGridLane + j] = ((lane >> j) & 1) ? tot : 0.0;
#pragma unroll
      for (int j = 0; j < n - 12; ++j) sums[kGridTile + j] = lane == j ? part : 0.0;
      T.red[32 * warp + lane] = warp_sums32(sums, lane);
      __syncthreads();
      if (warp == 0) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (lane < kGridWarp) s += T.red[32 * k + lane];
          else if (lane < kGridWarp + 3 && ((k >> (lane - kGridWarp)) & 1)) s += T.red[32 * k + kGridTotal];
        }
        rec[static_cast<size_t>(lane) * ctas] = s;
      }
    }
    swap(psi0, psi1);
    swap(lam0, lam1);
    if (!sync_grid(S, arrivals, A.polls)) return false;
    {  // low pass, in place
      double theta[12];
#pragma unroll
      for (int i = 0; i < 12; ++i) theta[i] = 0.0;
      const unsigned xb = swaps(flip, 4), xc = swaps(flip, 0), xa = swaps(flip, 8);
      for (unsigned tile = cta; tile < G::tiles; tile += ctas) {
        double2 p[16], v[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const unsigned at = tile << 12 | u_b | (static_cast<unsigned>(r) ^ xb) << 4;
          p[r] = __ldcg(psi0 + at);
          v[r] = __ldcg(lam0 + at);
        }
        auto undo = [&](double2 (&a)[16], int first) {
#pragma unroll
          for (int j = 0; j < 4; ++j) rotate<4>(a, j, -rot[first + j]);
        };
        auto sums = [&](int first) {
#pragma unroll
          for (int j = 0; j < 4; ++j) theta[first + j] += theta_sum<4>(p, v, j);
        };
        undo(p, 4);
        put(p, bufP, slot_b, bit_b);
        undo(v, 4);
        put(v, bufL, slot_b, bit_b);
        sums(4);
        __syncwarp();
        get(p, bufP, swapped(slot_c, xc, bit_c), bit_c);
        get(v, bufL, swapped(slot_c, xc, bit_c), bit_c);
        undo(p, 0);
        put(p, bufP, slot_c, bit_c);
        undo(v, 0);
        put(v, bufL, slot_c, bit_c);
        sums(0);
        __syncthreads();
        get(p, bufP, swapped(slot_a, xa, bit_a), bit_a);
        get(v, bufL, swapped(slot_a, xa, bit_a), bit_a);
        undo(p, 8);
        undo(v, 8);
        if (l > 0) {
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            psi0[tile << 12 | u_a | r << 8] = p[r];
            lam0[tile << 12 | u_a | r << 8] = v[r];
          }
        }
        sums(8);
        __syncthreads();  // the buffers are read
      }
      double all[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) all[i] = i < 12 ? theta[i < 12 ? i : 0] : 0.0;
      T.red[32 * (8 + warp) + lane] = warp_sums32(all, lane);
      __syncthreads();
      if (warp == 0 && lane < 12) {
        double s = 0.0;
#pragma unroll
        for (int k = 8; k < 16; ++k) s += T.red[32 * k + lane];
        rec[static_cast<size_t>(kGridLow + lane) * ctas] = s;
      }
    }
    if (!sync_grid(S, arrivals, A.polls)) return false;
  }
  // ---- the gradient, a warp an angle
  for (int e = static_cast<int>(cta * G::warps) + warp; e < L * n * 2; e += static_cast<int>(ctas) * G::warps) {
    const int l = e / (2 * n), w = e % (2 * n) / 2;
    const double *rec = recs + static_cast<size_t>(l) * kGridRec * ctas;
    auto total = [&](int i) {  // over the CTAs
      double s = 0.0;
      for (unsigned k = lane; k < ctas; k += 32) s += __ldcg(rec + static_cast<size_t>(i) * ctas + k);
      return warp_sum(s);
    };
    double out;
    if ((e & 1) == 0) {
      // prod (1 + k^2) over the wires still pending behind the step
      const unsigned pending = w >= top ? (1u << top) - 1 : w >= 12 ? 0xfffu : w >= 8 ? 0u : w < 4 ? 0xf00u : 0xf0fu;
      double s = 1.0;
      for (int k = 0; k < n; ++k)
        if ((pending >> k) & 1) s *= fma(T.rot[l * n + k], T.rot[l * n + k], 1.0);
      out = total(w >= top ? w - top : w >= 12 ? kGridHigh + w - 12 : kGridLow + w) * s;
    } else {
      int i;
      if (w >= top) {
        i = kGridPhi + w - top;
      } else if (w >= q && w < 12) {
        i = kGridTile + w - q;
      } else {  // a bit of the thread's number
        const int b = w < q ? w : q + w - 12;
        i = b < 5 ? kGridLane + b : kGridWarp + b - 5;
      }
      out = total(kGridTotal) - 2.0 * total(i);
      if (w >= top && ((T.flip[l] >> w) & 1)) out = -out;  // its register bit is 1 where the wire is 0
    }
    if (lane == 0) A.grad_out[item.param_off + e] = out;
  }
  return true;
}

template <int n>
__global__ void __launch_bounds__(256, 1) grid_circuit_kernel(const __grid_constant__ ClusterArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  if (run_grid<n>(A, smem)) return;
  if (threadIdx.x == 0)
    *static_cast<volatile unsigned *>(&grid_state(A, n)->lost) = 1u;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);  // a CTA did not arrive
  if (A.energy_out && blockIdx.x == 0 && threadIdx.x == 0) A.energy_out[A.item.index] = nan;
  if (A.grad_out)
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 2 * n * A.item.L; e += gridDim.x * blockDim.x)
      A.grad_out[A.item.param_off + e] = nan;
}

template <int n>
struct GridShape {
  static size_t smem(int max_layers) { return 2 * kGridBuf + table_bytes<Grid<n>>(max_layers); }
  static cudaError_t configure() {
    static std::atomic<unsigned long long> done{0};
    return set_smem_limit_once(grid_circuit_kernel<n>, kMostGridSmem, done);
  }
  // CTAs of a launch: one a SM, no more than there are tiles; 0 where none fits
  static cudaError_t ctas(int max_layers, int *count) {
    *count = 0;
    if (smem(max_layers) > kMostGridSmem) return cudaSuccess;
    cudaError_t e = configure();
    int dev = 0, sms = 0, fit = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, grid_circuit_kernel<n>, 256, smem(max_layers));
    if (e != cudaSuccess || fit < 1) return e;
    *count = sms < Grid<n>::tiles ? sms : Grid<n>::tiles;
    if (*count > kMostGridCtas) *count = kMostGridCtas;
    return e;
  }
  static cudaError_t launch(const ClusterArgs &A, cudaStream_t s) {
    int count = 0;
    cudaError_t e = ctas(A.max_layers, &count);
    if (e != cudaSuccess) return e;
    if (count < 1 || A.count != 1 || A.items != nullptr) return cudaErrorInvalidValue;
    // (a backward that resumes a forward leaves what that one lost)
    const size_t bytes = A.resume ? sizeof(unsigned) : sizeof(GridState);
    if ((e = cudaMemsetAsync(grid_state(A, n), 0, bytes, s)) != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at;
    cfg.gridDim = dim3(static_cast<unsigned>(count));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem(A.max_layers);
    cfg.stream = s;
    at.id = cudaLaunchAttributeCooperative;  // all CTAs run at the same time
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, grid_circuit_kernel<n>, A);
  }
};

template <typename F>
bool with_grid(int n, F &&f) {
  switch (n) {
    case 17: f(GridShape<17>{}); return true;
    case 18: f(GridShape<18>{}); return true;
    case 19: f(GridShape<19>{}); return true;
    case 20: f(GridShape<20>{}); return true;
    default: return false;
  }
}

}  // namespace

const unsigned *grid_lost_flag(const ClusterArgs &A) { return &grid_state(A, A.n)->lost; }

size_t grid_memory_values(int n, int max_layers) {
  return (size_t{4} << n) + grid_doubles(max_layers) / 2 + 1 + sizeof(GridState) / sizeof(double2) + 1;
}

cudaError_t launch_grid(const ClusterArgs &A, cudaStream_t s) {
  cudaError_t e = cudaErrorInvalidValue;
  with_grid(A.n, [&](auto shape) { e = decltype(shape)::launch(A, s); });
  return e;
}

cudaError_t grid_capacity(int n, int max_layers, int *circuits) {
  cudaError_t e = cudaSuccess;
  int ctas = 0;
  with_grid(n, [&](auto shape) { e = decltype(shape)::ctas(max_layers, &ctas); });
  *circuits = e == cudaSuccess && ctas > 0;
  return e;
}

}  // namespace rsv
