// Energy and adjoint gradient of a shallow circuit, contracted along the ring
// instead of along the layers.
//
// In a layer every wire meets its neighbours only through the CNOT ring, and
// CNOT(w, w+1) carries one bit: wire w's value after its rotations and the bit
// it received itself.  So the circuit's amplitude is a sum over the bits
// s_1 .. s_{L-1} that cross each gap between neighbouring wires in layers
// 1 .. L-1 (the last ring only relabels the basis and is moved into H): a trace of
// n matrices of size D = 2^(L-1),
//   T_w[s; s'] = prod_l U_{l,w}[s_l ^ s'_l, s_{l-1}]    (s_0 = 0; wire 0: T_0[s; a] =
//                prod_l U_{l,0}[s_l, s_{l-1} ^ a_{l-1}], a the bits arriving at wire 0),
// with U = RZ RY of the wire in that layer, s' the bits arriving and s the bits
// leaving (l = 1 .. L-1 here; s_{L-1} is also the wire's value before the last
// layer).  <psi|O|psi> of a product operator is the same sum for bra and ket
// with the 2x2 matrix M_O = U_L^+ O U_L between them at every wire.
// P^T H P (P the last ring) is a sum of such operators:
//   - sum_{w != 1} Z_w - (Z on every wire but 1) - h sum_{w < n-1} X_w X_{w+1} - h X_{n-1} X_0 X_1,
// so one pass over the wires carrying five components does all of it:
//   I identity so far, X an open X on the last wire, H complete terms,
//   W an open X_0 X_1, S the Z string.
// The ring is closed by fixing the bits (a, abar) that enter wire 0: D^2
// independent chains, each a D x D matrix (ket bits x bra bits) per component.
// Exact, and the cost is n 16^(L-1) L instead of 2^n n L; every entry is a
// transition amplitude between projected states, at most 1 in magnitude, so
// nothing grows along the chain.
//
// Kernels:
//   ring_sweep_kernel: one CTA per chain and direction.  Left sweeps apply the
//     sites 1 .. n-1 in order and end in the energy; right sweeps apply the
//     transposes from the closed end.  Warp c holds component c in registers
//     (m8n8k4 accumulator layout) and applies T . V . T^+ as two products on
//     the FP64 tensor cores: contracting the columns of an accumulator needs no
//     shuffle (element j of a lane is k = 2 (lane % 4) + j of the operand), and
//     the second product's accumulator is again ket x bra.  A sixth warp
//     builds the next site's T.  One barrier per site.
//   ring_grad_kernel: one cluster per site.  From the left components before
//     and the right components after the site: dE/dT[s; s'] summed over chains
//     and components on the tensor cores, then the site's 2 L derivatives.
// Both are bound by latency (n dependent sites of two small products), not by
// memory or arithmetic throughput.
// energy_and_grad at L = 4: n = 16 33 us (tile passes 141), n = 24 40 us (1598),
// n = 28 42 us (21 400).  L = 5 (16 x 16 matrices): n = 22 427 us (807), n = 24
// 445 us (2631); n = 20 410 us against 322.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>

#include "rsv_device.cuh"
#include "rsv_launch.h"
#include "rsv_ring.h"

namespace rsv {
namespace {

namespace cg = cooperative_groups;

constexpr int kComps = 5;  // I, X, H, W, S
constexpr int kI = 0, kX = 1, kH = 2, kW = 3, kS = 4;
constexpr int kSweepThreads = 32 * (kComps + 1);
constexpr int kGradWarps = 8;
constexpr int kMaxDerivs = 2 * kRingMaxLayers;

struct SiteM {  // cos, sin of the full angles of a wire's last layer
  double ct, st, cp, sp;
};

// A D x D complex matrix in a warp's registers: tile (i, j), element e of lane
// l is row 8 i + l / 4, column 8 j + 2 (l % 4) + e.
template <int DB>
struct Mat {
  double re[DB][DB][2], im[DB][DB][2];
};

template <int DB>
__device__ __forceinline__ int frag_row(int i, int lane) {
  return 8 * i + lane / 4;
}
template <int DB>
__device__ __forceinline__ int frag_col(int j, int lane, int e) {
  return 8 * j + 2 * (lane % 4) + e;
}

template <int DB>
__device__ __forceinline__ Mat<DB> zero_mat() {
  Mat<DB> m;
#pragma unroll
  for (int i = 0; i < DB; ++i)
#pragma unroll
    for (int j = 0; j < DB; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) m.re[i][j][e] = m.im[i][j][e] = 0.0;
  return m;
}

// Matrices in memory keep that order: [tile][lane][element].
template <int DB>
__device__ __forceinline__ void store_mat(double2 *p, const Mat<DB> &m, int lane) {
#pragma unroll
  for (int i = 0; i < DB; ++i)
#pragma unroll
    for (int j = 0; j < DB; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        p[(i * DB + j) * 64 + 2 * lane + e] = make_double2(m.re[i][j][e], m.im[i][j][e]);
}
template <int DB>
__device__ __forceinline__ Mat<DB> load_mat(const double2 *p, int lane) {
  Mat<DB> m;
#pragma unroll
  for (int i = 0; i < DB; ++i)
#pragma unroll
    for (int j = 0; j < DB; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double2 v = p[(i * DB + j) * 64 + 2 * lane + e];
        m.re[i][j][e] = v.x;
        m.im[i][j][e] = v.y;
      }
  return m;
}

// Z[m][n] += sum_k A[m][k] B[n][k] (no conjugation of B; A conjugated when CONJ).
template <int DB, bool CONJ>
__device__ __forceinline__ void mma_rows(Mat<DB> &Z, const Mat<DB> &A, const Mat<DB> &B) {
#pragma unroll
  for (int i = 0; i < DB; ++i)
#pragma unroll
    for (int j = 0; j < DB; ++j) {
      double r0 = Z.re[i][j][0], r1 = Z.re[i][j][1], q0 = 0.0, q1 = 0.0;
      double s0 = Z.im[i][j][0], s1 = Z.im[i][j][1], t0 = 0.0, t1 = 0.0;
#pragma unroll
      for (int k = 0; k < DB; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          mma_f64(r0, r1, A.re[i][k][e], B.re[j][k][e]);
          mma_f64(q0, q1, A.im[i][k][e], B.im[j][k][e]);
          mma_f64(s0, s1, A.re[i][k][e], B.im[j][k][e]);
          mma_f64(t0, t1, A.im[i][k][e], B.re[j][k][e]);
        }
      Z.re[i][j][0] = CONJ ? r0 + q0 : r0 - q0;
      Z.re[i][j][1] = CONJ ? r1 + q1 : r1 - q1;
      Z.im[i][j][0] = CONJ ? s0 - t0 : s0 + t0;
      Z.im[i][j][1] = CONJ ? s1 - t1 : s1 + t1;
    }
}

// T . V . T^+ for T given as rows of the result's side: first the bra columns
// (conj T), then the ket rows; `T` is in shared memory in matrix order.
template <int DB>
__device__ __forceinline__ Mat<DB> sandwich(const double2 *T, const Mat<DB> &V, int lane) {
  const Mat<DB> t = load_mat<DB>(T, lane);
  Mat<DB> z = zero_mat<DB>();
  mma_rows<DB, true>(z, t, V);   // z[bra][ket]
  Mat<DB> y = zero_mat<DB>();
  mma_rows<DB, false>(y, t, z);  // y[ket][bra]
  return y;
}

__device__ __forceinline__ SiteM site_m(double4 c) {
  SiteM m;
  m.ct = c.x * c.x - c.y * c.y;
  m.st = 2.0 * c.x * c.y;
  m.cp = c.z * c.z - c.w * c.w;
  m.sp = 2.0 * c.z * c.w;
  return m;
}

// U[q][c] = (RZ RY)[q][c] at u[2 q + c]
__device__ __forceinline__ void site_u(double4 c, double2 *u) {
  u[0] = make_double2(c.x * c.z, -c.x * c.w);
  u[1] = make_double2(-c.y * c.z, c.y * c.w);
  u[2] = make_double2(c.y * c.z, c.y * c.w);
  u[3] = make_double2(c.x * c.z, c.x * c.w);
}

// M_Z and M_X of a site at (bra bit, ket bit)
__device__ __forceinline__ double m_z(const SiteM &m, int bra, int ket) {
  return bra == ket ? (ket ? -m.ct : m.ct) : -m.st;
}
__device__ __forceinline__ double2 m_x(const SiteM &m, int bra, int ket) {
  if (bra == ket) return make_double2(ket ? -m.cp * m.st : m.cp * m.st, 0.0);
  return make_double2(m.cp * m.ct, ket ? m.sp : -m.sp);
}

// T_w[s; s'] of a wire w >= 1; U of layer l at U[l * stride]
__device__ __forceinline__ double2 t_entry(const double2 *U, int stride, int nb, int s, int sp) {
  if (((s | sp) >> nb) != 0) return make_double2(0.0, 0.0);
  double2 v = make_double2(1.0, 0.0);
  int prev = 0;
  for (int l = 0; l < nb; ++l) {
    const int q = ((s ^ sp) >> l) & 1;
    v = cmul(v, U[l * stride + 2 * q + prev]);
    prev = (s >> l) & 1;
  }
  return v;
}

// T_0[s; a]
__device__ __forceinline__ double2 t0_entry(const double2 *U, int stride, int nb, int s, int a) {
  if (((s | a) >> nb) != 0) return make_double2(0.0, 0.0);
  double2 v = make_double2(1.0, 0.0);
  int prev = 0;
  for (int l = 0; l < nb; ++l) {
    const int q = (s >> l) & 1;
    v = cmul(v, U[l * stride + 2 * q + prev]);
    prev = ((s ^ a) >> l) & 1;
  }
  return v;
}

// Element e of a matrix in memory order is row r, column c of it.
template <int DB>
__device__ __forceinline__ void order_rc(int e, int &r, int &c) {
  const int tile = e / 64, lane = (e % 64) / 2;
  r = frag_row<DB>(tile / DB, lane);
  c = frag_col<DB>(tile % DB, lane, e & 1);
}

// The bit of a bond index that is the wire's value before the last layer.
__device__ __forceinline__ int last_bit(int v, int nb) { return nb > 0 ? (v >> (nb - 1)) & 1 : 0; }

template <int DB>
constexpr size_t sweep_smem_bytes(int n, int L) {
  return sizeof(double2) * (static_cast<size_t>(L > 1 ? L - 1 : 0) * n * 4 + (2 + 6) * 64 * DB * DB) +
         sizeof(SiteM) * static_cast<size_t>(n);
}

// Applies f(i, j, e, bra bit, ket bit) to every element of a lane; the bits are
// those before the last layer, flipped by fb / fk (wire 0: the arriving bits).
template <int DB, typename F>
__device__ __forceinline__ void each(int lane, int nb, int fk, int fb, F &&f) {
#pragma unroll
  for (int i = 0; i < DB; ++i)
#pragma unroll
    for (int j = 0; j < DB; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        f(i, j, e, last_bit(frag_col<DB>(j, lane, e), nb) ^ fb, last_bit(frag_row<DB>(i, lane), nb) ^ fk);
}

// Left components after a site from those before its last layer (t*), for
// component c of wire w (1 <= w < n - 1) or, at the last wire, the energy share
// of every component.
template <int DB>
__global__ void __launch_bounds__(kSweepThreads) ring_sweep_kernel(const RingParams P, int first_dir, int keep) {
  constexpr int D = 8 * DB, DD = D * D;
  extern __shared__ double2 smem[];
  const int n = P.n, L = P.L, nb = L - 1;
  const int chains = gridDim.x, chain = blockIdx.x;
  const bool rightward = first_dir + static_cast<int>(blockIdx.y) == 0;
  const int a = chain >> nb, ab = chain & ((1 << nb) - 1);
  double2 *U = smem;                       // [nb][n][4]
  double2 *T = U + nb * n * 4;             // [2][DD]
  double2 *ex = T + 2 * DD;                // [2][3][DD]
  SiteM *M = reinterpret_cast<SiteM *>(ex + 6 * DD);  // [n]
  const int tid = threadIdx.x, lane = tid & 31, comp = tid >> 5;
  for (int k = tid; k < nb * n; k += kSweepThreads) site_u(P.coef[k], U + 4 * k);
  for (int k = tid; k < n; k += kSweepThreads) M[k] = site_m(P.coef[nb * n + k]);
  __syncthreads();
  const int ustride = 4 * n;
  auto build = [&](int w, double2 *out, int first, int step) {
    for (int e = first; e < DD; e += step) {
      int r, c;
      order_rc<DB>(e, r, c);
      out[e] = rightward ? t_entry(U + 4 * w, ustride, nb, r, c) : t_entry(U + 4 * w, ustride, nb, c, r);
    }
  };
  build(rightward ? 1 : n - 1, T, tid, kSweepThreads);
  const double h = P.field;

  if (rightward) {
    Mat<DB> v;
    if (comp < kComps) {
      const SiteM m = M[0];
      each<DB>(lane, nb, last_bit(a, nb), last_bit(ab, nb), [&](int i, int j, int e, int bra, int ket) {
        const double2 uk = t0_entry(U, ustride, nb, frag_row<DB>(i, lane), a);
        const double2 ub = t0_entry(U, ustride, nb, frag_col<DB>(j, lane, e), ab);
        double2 x = cmul_conj(uk, ub);
        if (comp == kI) {
          if (bra != ket) x = make_double2(0.0, 0.0);
        } else if (comp == kX) {
          x = cmul(m_x(m, bra, ket), x);
        } else if (comp == kW) {
          x = make_double2(0.0, 0.0);
        } else {
          const double z = -m_z(m, bra, ket);
          x = make_double2(z * x.x, z * x.y);
        }
        v.re[i][j][e] = x.x;
        v.im[i][j][e] = x.y;
      });
    }
    __syncthreads();
    for (int w = 1; w < n; ++w) {
      const int p = (w - 1) & 1;
      double2 *xI = ex + p * 3 * DD, *xX = xI + DD;
      if (comp < kComps) {
        v = sandwich<DB>(T + p * DD, v, lane);
        if (keep) store_mat<DB>(P.left + ((static_cast<size_t>(w) * chains + chain) * kComps + comp) * DD, v, lane);
        if (comp == kI) store_mat<DB>(xI, v, lane);
        if (comp == kX) store_mat<DB>(xX, v, lane);
      } else if (w + 1 < n) {
        build(w + 1, T + (p ^ 1) * DD, lane, 32);
      }
      __syncthreads();
      if (w == n - 1) break;
      const SiteM m = M[w];
      if (comp == kI || (comp == kW && w > 1) || (comp == kS && w == 1)) {
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          if (bra != ket) v.re[i][j][e] = v.im[i][j][e] = 0.0;
        });
      } else if (comp == kX || comp == kW) {
        const double2 *src = comp == kX ? xI : xX;
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          const double2 x = cmul(m_x(m, bra, ket), src[(i * DB + j) * 64 + 2 * lane + e]);
          v.re[i][j][e] = x.x;
          v.im[i][j][e] = x.y;
        });
      } else if (comp == kH) {
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          const int at = (i * DB + j) * 64 + 2 * lane + e;
          const double2 x = cmul(m_x(m, bra, ket), xX[at]);
          const double z = w == 1 ? 0.0 : m_z(m, bra, ket);
          const double2 t = xI[at];
          const double keep_re = bra == ket ? v.re[i][j][e] : 0.0, keep_im = bra == ket ? v.im[i][j][e] : 0.0;
          v.re[i][j][e] = keep_re - z * t.x - h * x.x;
          v.im[i][j][e] = keep_im - z * t.y - h * x.y;
        });
      } else if (comp == kS) {
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          const double z = m_z(m, bra, ket);
          v.re[i][j][e] *= z;
          v.im[i][j][e] *= z;
        });
      }
    }
    // the ring closes on the bits (a, ab): Re of each component's share
    __shared__ double share[kComps];
    if (comp < kComps) {
      const SiteM m = M[n - 1];
      each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
        if (frag_row<DB>(i, lane) != a || frag_col<DB>(j, lane, e) != ab) return;
        const double re = v.re[i][j][e], im = v.im[i][j][e];
        double x;
        if (comp == kH) {
          x = bra == ket ? re : 0.0;
        } else if (comp == kI || comp == kS) {
          x = (comp == kI ? -1.0 : 1.0) * m_z(m, bra, ket) * re;
        } else {
          const double2 q = m_x(m, bra, ket);
          x = -h * (q.x * re - q.y * im);
        }
        share[comp] = x;
      });
    }
    __syncthreads();
    __shared__ bool last;
    if (tid == 0) {
      P.energy_parts[chain] = ((share[kI] + share[kX]) + (share[kH] + share[kW])) + share[kS];
      __threadfence();
      last = atomicInc(P.counter, static_cast<unsigned>(chains - 1)) == static_cast<unsigned>(chains - 1);
    }
    __syncthreads();
    if (last && comp == 0) {  // every share is written: add them in a fixed order
      __threadfence();
      double s = 0.0;
      for (int k = lane; k < chains; k += 32) s += __ldcg(P.energy_parts + k);
      s = warp_sum(s);
      if (lane == 0) {
        P.energy_parts[chains] = s;
        if (P.energy_out) *P.energy_out = s;
      }
    }
    return;
  }

  // Right sweep: components after site n - 1 are the closed end.
  Mat<DB> v = zero_mat<DB>();
  if (comp == kH || comp == kS)
    each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int, int) {
      if (frag_row<DB>(i, lane) == a && frag_col<DB>(j, lane, e) == ab) v.re[i][j][e] = 1.0;
    });
  for (int w = n - 1; w >= 1; --w) {
    const int p = (n - 1 - w) & 1;
    double2 *xH = ex + p * 3 * DD, *xX = xH + DD, *xW = xX + DD;
    if (comp == kH) store_mat<DB>(xH, v, lane);
    if (comp == kX) store_mat<DB>(xX, v, lane);
    if (comp == kW && w == 1) store_mat<DB>(xW, v, lane);
    if (comp < kComps && w < n - 1)
      store_mat<DB>(P.right + ((static_cast<size_t>(w) * chains + chain) * kComps + comp) * DD, v, lane);
    __syncthreads();
    const SiteM m = M[w];
    if (comp == kComps) {
      if (w > 1) build(w - 1, T + (p ^ 1) * DD, lane, 32);
      continue;
    }
    each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
      const int at = (i * DB + j) * 64 + 2 * lane + e;
      double re = v.re[i][j][e], im = v.im[i][j][e];
      const double z = m_z(m, bra, ket);
      if (comp == kI) {
        const double2 x = cmul(m_x(m, bra, ket), xX[at]);
        const double zz = w == 1 ? 0.0 : z;
        if (bra != ket) re = im = 0.0;
        re += x.x - zz * xH[at].x;
        im += x.y - zz * xH[at].y;
      } else if (comp == kX || (comp == kW && w == n - 1)) {
        double2 t = make_double2(-h * xH[at].x, -h * xH[at].y);
        if (w == 1) {
          t.x += xW[at].x;
          t.y += xW[at].y;
        }
        t = cmul(m_x(m, bra, ket), t);
        re = t.x;
        im = t.y;
      } else if (comp == kH || (comp == kW && w > 1) || (comp == kS && w == 1)) {
        if (bra != ket) re = im = 0.0;
      } else if (comp == kW) {
        re = im = 0.0;
      } else {
        re *= z;
        im *= z;
      }
      v.re[i][j][e] = re;
      v.im[i][j][e] = im;
    });
    v = sandwich<DB>(T + p * DD, v, lane);
  }
  if (comp < kComps)
    store_mat<DB>(P.right + (static_cast<size_t>(chain) * kComps + comp) * DD, v, lane);
}

// One cluster per site; its warps share the chains.
template <int DB>
__global__ void __launch_bounds__(32 * kGradWarps) ring_grad_kernel(const RingParams P) {
  constexpr int D = 8 * DB, DD = D * D;
  extern __shared__ double2 smem[];
  __shared__ double2 Uw[4 * (kRingMaxLayers - 1)], U0[4 * (kRingMaxLayers - 1)];
  __shared__ double red[kGradWarps][kMaxDerivs];
  __shared__ double total[kMaxDerivs];
  double2 *T = smem;              // [DD] T_w, or T_0 for sites 0 and 1 behind it
  double2 *T0 = T + DD;           // [DD]
  double2 *G = T0 + DD;           // [kGradWarps][DD]
  cg::cluster_group cluster = cg::this_cluster();
  const int G_ctas = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int w = static_cast<int>(blockIdx.x) / G_ctas;
  const int n = P.n, L = P.L, nb = L - 1, chains = 1 << (2 * nb), bond = 1 << nb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < nb) {
    site_u(P.coef[tid * n + w], Uw + 4 * tid);
    site_u(P.coef[tid * n], U0 + 4 * tid);
  }
  __syncthreads();
  for (int e = tid; e < DD; e += 32 * kGradWarps) {
    int r, c;
    order_rc<DB>(e, r, c);
    T[e] = t_entry(Uw, 4, nb, r, c);
    T0[e] = t0_entry(U0, 4, nb, r, c);
  }
  for (int e = tid; e < kGradWarps * DD; e += 32 * kGradWarps) G[e] = make_double2(0.0, 0.0);
  __syncthreads();
  const double h = P.field;
  const SiteM m = site_m(P.coef[nb * n + w]);
  // d/dtheta and d/dphi of M_X and M_Z of this site
  const SiteM mt{-m.st, m.ct, m.cp, 0.0};  // theta: M_X keeps its cos(phi) part
  const SiteM mp{m.ct, m.st, -m.sp, m.cp}; // phi
  double g_theta = 0.0, g_phi = 0.0;
  auto right_of = [&](int c, int chain) {
    return load_mat<DB>(P.right + ((static_cast<size_t>(w) * chains + chain) * kComps + c) * DD, lane);
  };
  auto last_layer = [&](int bra, int ket, double2 qx, double2 qz) {
    const double2 xt = m_x(mt, bra, ket), xp = m_x(mp, bra, ket);
    g_theta += xt.x * qx.x - xt.y * qx.y + m_z(mt, bra, ket) * qz.x;
    g_phi += xp.x * qx.x - xp.y * qx.y;
  };
  if (w == 0) {
    // T_0's column a from the chains (a, .): sum over the bra bits and over ab
    for (int a = rank * kGradWarps + warp; a < bond; a += G_ctas * kGradWarps) {
      double gr[DB], gi[DB];
#pragma unroll
      for (int i = 0; i < DB; ++i) gr[i] = gi[i] = 0.0;
      for (int ab = 0; ab < bond; ++ab) {
        const int chain = (a << nb) | ab;
        const Mat<DB> rI = right_of(kI, chain), rX = right_of(kX, chain), rH = right_of(kH, chain),
                      rS = right_of(kS, chain);
        each<DB>(lane, nb, last_bit(a, nb), last_bit(ab, nb), [&](int i, int j, int e, int bra, int ket) {
          const double2 uk = t0_entry(U0, 4, nb, frag_row<DB>(i, lane), a);
          const double2 ub = t0_entry(U0, 4, nb, frag_col<DB>(j, lane, e), ab);
          const double2 x = make_double2(rX.re[i][j][e], rX.im[i][j][e]);
          const double2 s = make_double2(-(rH.re[i][j][e] + rS.re[i][j][e]), -(rH.im[i][j][e] + rS.im[i][j][e]));
          const double z = m_z(m, bra, ket);
          double2 r = cmul(m_x(m, bra, ket), x);
          r.x += z * s.x;
          r.y += z * s.y;
          if (bra == ket) {
            r.x += rI.re[i][j][e];
            r.y += rI.im[i][j][e];
          }
          r = cmul_conj(r, ub);
          gr[i] += r.x;
          gi[i] += r.y;
          const double2 v = cmul_conj(uk, ub);
          last_layer(bra, ket, cmul(v, x), cmul(v, s));
        });
      }
#pragma unroll
      for (int i = 0; i < DB; ++i) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          gr[i] += __shfl_xor_sync(0xffffffffu, gr[i], o);
          gi[i] += __shfl_xor_sync(0xffffffffu, gi[i], o);
        }
        // element (row, a) in matrix order, in this warp's slice
        if (lane % 4 == 0)
          G[warp * DD + (i * DB + a / 8) * 64 + 2 * ((lane / 4) * 4 + (a % 8) / 2) + (a & 1)] =
              make_double2(gr[i], gi[i]);
      }
    }
  } else {
    Mat<DB> g = zero_mat<DB>();
    const Mat<DB> t = load_mat<DB>(T, lane);
    const SiteM m1 = site_m(P.coef[nb * n + w - 1]);
    for (int chain = rank * kGradWarps + warp; chain < chains; chain += G_ctas * kGradWarps) {
      const int a = chain >> nb, ab = chain & (bond - 1);
      const double2 *before = P.left + (static_cast<size_t>(w - 1) * chains + chain) * kComps * DD;
      const double2 *here = P.left + (static_cast<size_t>(w) * chains + chain) * kComps * DD;
      Mat<DB> rH, rX = zero_mat<DB>();
      if (w == n - 1) {
        rH = zero_mat<DB>();
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int, int) {
          if (frag_row<DB>(i, lane) == a && frag_col<DB>(j, lane, e) == ab) rH.re[i][j][e] = 1.0;
        });
      } else {
        rH = right_of(kH, chain);
        rX = right_of(kX, chain);
      }
#pragma unroll
      for (int c = 0; c < kComps; ++c) {
        if (c == kW && w == 1) continue;  // no open X_0 X_1 before wire 1
        // left component before the site, from the previous site's
        Mat<DB> v;
        if (w == 1) {
          each<DB>(lane, nb, last_bit(a, nb), last_bit(ab, nb), [&](int i, int j, int e, int bra, int ket) {
            const int col = frag_col<DB>(j, lane, e);
            // rows a / ab of T_0 (column index in matrix order)
            const double2 uk = T0[(i * DB + a / 8) * 64 + 2 * ((lane / 4) * 4 + (a % 8) / 2) + (a & 1)];
            const double2 ub = T0[(col / 8 * DB + ab / 8) * 64 + 2 * ((col % 8) * 4 + (ab % 8) / 2) + (ab & 1)];
            double2 x = cmul_conj(uk, ub);
            if (c == kI) {
              if (bra != ket) x = make_double2(0.0, 0.0);
            } else if (c == kX) {
              x = cmul(m_x(m1, bra, ket), x);
            } else {
              const double z = -m_z(m1, bra, ket);
              x = make_double2(z * x.x, z * x.y);
            }
            v.re[i][j][e] = x.x;
            v.im[i][j][e] = x.y;
          });
        } else {
          const bool first = w - 1 == 1;
          const int src = c == kX ? kI : (c == kW && first ? kX : c);
          v = load_mat<DB>(before + src * DD, lane);
          if (c == kX || (c == kW && first)) {
            each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
              const double2 x = cmul(m_x(m1, bra, ket), make_double2(v.re[i][j][e], v.im[i][j][e]));
              v.re[i][j][e] = x.x;
              v.im[i][j][e] = x.y;
            });
          } else if (c == kS && !first) {
            each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
              const double z = m_z(m1, bra, ket);
              v.re[i][j][e] *= z;
              v.im[i][j][e] *= z;
            });
          } else {
            each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
              if (bra != ket) v.re[i][j][e] = v.im[i][j][e] = 0.0;
            });
            if (c == kH)
              each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
                const int at = (i * DB + j) * 64 + 2 * lane + e;
                const double2 x = cmul(m_x(m1, bra, ket), before[kX * DD + at]);
                const double z = first ? 0.0 : m_z(m1, bra, ket);
                const double2 ti = before[kI * DD + at];
                v.re[i][j][e] += -z * ti.x - h * x.x;
                v.im[i][j][e] += -z * ti.y - h * x.y;
              });
          }
        }
        // right component behind the site's last layer, and that layer's sums
        Mat<DB> r = zero_mat<DB>(), q = zero_mat<DB>();
        if (w < n - 1 && (c == kI || c == kS || c == kW)) {
          if (c != kW || w > 1) r = right_of(c, chain);
        }
        if (c == kS && w == n - 1) r = rH;
        Mat<DB> rW1;
        if (c == kX && w == 1) rW1 = right_of(kW, chain);
        if (c != kH) q = load_mat<DB>(here + c * DD, lane);
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          const double2 H = make_double2(rH.re[i][j][e], rH.im[i][j][e]);
          const double2 X = make_double2(rX.re[i][j][e], rX.im[i][j][e]);
          const double2 mx = m_x(m, bra, ket);
          const double z = m_z(m, bra, ket);
          const double2 tq = make_double2(q.re[i][j][e], q.im[i][j][e]);
          double2 o = make_double2(r.re[i][j][e], r.im[i][j][e]);
          if (c == kI) {
            const double zz = w == 1 ? 0.0 : z;
            const double2 x = cmul(mx, X);
            last_layer(bra, ket, cmul(tq, X),
                       w == 1 ? make_double2(0.0, 0.0) : cmul(tq, make_double2(-H.x, -H.y)));
            if (bra != ket) o = make_double2(0.0, 0.0);
            o.x += x.x - zz * H.x;
            o.y += x.y - zz * H.y;
          } else if (c == kX || (c == kW && w == n - 1)) {
            double2 x = make_double2(-h * H.x, -h * H.y);
            if (c == kX && w == 1) {
              x.x += rW1.re[i][j][e];
              x.y += rW1.im[i][j][e];
            }
            last_layer(bra, ket, cmul(tq, x), make_double2(0.0, 0.0));
            o = cmul(mx, x);
          } else if (c == kH) {
            o = bra == ket ? H : make_double2(0.0, 0.0);
          } else if (c == kW || w == 1) {
            if (bra != ket) o = make_double2(0.0, 0.0);
          } else {
            last_layer(bra, ket, make_double2(0.0, 0.0), cmul(tq, o));
            o = make_double2(z * o.x, z * o.y);
          }
          r.re[i][j][e] = o.x;
          r.im[i][j][e] = o.y;
        });
        // y[s'][bra] = sum v[s'][.] conj(T[bra][.]); g[s][s'] += sum r[s][bra] y[s'][bra]
        Mat<DB> vc = v;
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int, int) { vc.im[i][j][e] = -vc.im[i][j][e]; });
        Mat<DB> y = zero_mat<DB>();
        mma_rows<DB, false>(y, vc, t);  // conj(v) T: the conjugate of y
        each<DB>(lane, nb, 0, 0, [&](int i, int j, int e, int, int) { y.im[i][j][e] = -y.im[i][j][e]; });
        mma_rows<DB, false>(g, r, y);
      }
    }
    store_mat<DB>(G + warp * DD, g, lane);
  }
  __syncthreads();
  // The site's derivatives from dE/dT = 2 Re sum G dT (linear: every CTA its part)
  double d[kMaxDerivs];
#pragma unroll
  for (int k = 0; k < kMaxDerivs; ++k) d[k] = 0.0;
  for (int e = tid; e < DD; e += 32 * kGradWarps) {
    double2 g = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < kGradWarps; ++k) {
      g.x += G[k * DD + e].x;
      g.y += G[k * DD + e].y;
    }
    int r, c;
    order_rc<DB>(e, r, c);
    if (((r | c) >> nb) != 0) continue;
    // factor index 2 q + prev of every layer
    int f[kRingMaxLayers - 1];
    int prev = 0;
#pragma unroll
    for (int l = 0; l < kRingMaxLayers - 1; ++l) {
      if (l >= nb) break;
      const int s = (r >> l) & 1, o = (c >> l) & 1;
      f[l] = 2 * (w == 0 ? s : s ^ o) + prev;
      prev = w == 0 ? s ^ o : s;
    }
#pragma unroll
    for (int l = 0; l < kRingMaxLayers - 1; ++l) {
      if (l >= nb) break;
      double2 rest = g;
#pragma unroll
      for (int k = 0; k < kRingMaxLayers - 1; ++k)
        if (k < nb && k != l) rest = cmul(rest, Uw[4 * k + f[k]]);
      // dU/dtheta[q][c]: half of U with its columns (c, s) -> (-s, c); dU/dphi: -+ i/2 U
      const double2 u = Uw[4 * l + f[l]], v = Uw[4 * l + (f[l] ^ 1)];
      const double sign = (f[l] & 1) ? -1.0 : 1.0;  // d(column 0) = column 1, d(column 1) = -column 0
      const double2 t = cmul(rest, v);
      const double2 ph = cmul(rest, u);
      d[2 * l] += sign * t.x;                            // 2 Re(rest (sign v / 2))
      d[2 * l + 1] += (f[l] & 2) ? -ph.y : ph.y;         // 2 Re(-+ i/2 rest u)
    }
  }
  // (the last layer's sums are complete: every lane its own elements)
#pragma unroll
  for (int l = 0; l < kRingMaxLayers; ++l)
    if (l == nb) {
      d[2 * l] = g_theta;
      d[2 * l + 1] = g_phi;
    }
#pragma unroll
  for (int k = 0; k < kMaxDerivs; ++k) {
    const double s = warp_sum(d[k]);
    if (lane == 0) red[warp][k] = s;
  }
  __syncthreads();
  if (tid < kMaxDerivs) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kGradWarps; ++k) s += red[k][tid];
    total[tid] = s;
  }
  cluster.sync();
  if (rank == 0 && tid < 2 * L) {
    double s = 0.0;
    for (int k = 0; k < G_ctas; ++k) s += *cluster.map_shared_rank(total + tid, k);
    // a NaN energy (a non-finite angle) voids the whole gradient
    const double energy = P.energy_parts[chains];
    if (energy != energy) s = energy;
    P.grad_out[static_cast<size_t>(tid / 2 * n + w) * 2 + (tid & 1)] = s;
  }
  cluster.sync();  // peers' shared memory stays until it is read
}

template <int DB>
cudaError_t sweeps(const RingParams &P, int first, int dirs, bool keep, cudaStream_t s) {
  static std::atomic<unsigned long long> done{0};
  const size_t smem = sweep_smem_bytes<DB>(P.n, P.L);
  const cudaError_t e = set_smem_limit_once(ring_sweep_kernel<DB>, sweep_smem_bytes<DB>(kMaxQubits, kRingMaxLayers), done);
  if (e != cudaSuccess) return e;
  const dim3 grid(static_cast<unsigned>(ring_chains(P.L)), static_cast<unsigned>(dirs));
  ring_sweep_kernel<DB><<<grid, kSweepThreads, smem, s>>>(P, first, keep ? 1 : 0);
  return cudaGetLastError();
}

template <int DB>
cudaError_t gradient(const RingParams &P, cudaStream_t s) {
  static std::atomic<unsigned long long> done{0};
  constexpr size_t smem = sizeof(double2) * (2 + kGradWarps) * 64 * DB * DB;
  cudaError_t e = set_smem_limit_once(ring_grad_kernel<DB>, smem, done);
  if (e != cudaSuccess) return e;
  // two chains a warp, four CTAs a site at 64 chains, at most eight
  int ctas = 1;
  while (ctas < 8 && ctas * 2 * kGradWarps < ring_chains(P.L)) ctas *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(P.n * ctas));
  cfg.blockDim = dim3(32 * kGradWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = static_cast<unsigned>(ctas);
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, ring_grad_kernel<DB>, P);
}

}  // namespace

cudaError_t launch_ring_sweeps(const RingParams &P, bool left, bool right, bool keep, cudaStream_t s) {
  const int first = left ? 0 : 1, dirs = (left ? 1 : 0) + (right ? 1 : 0);
  return P.L <= 4 ? sweeps<1>(P, first, dirs, keep, s) : sweeps<2>(P, first, dirs, keep, s);
}

cudaError_t launch_ring_gradient(const RingParams &P, cudaStream_t s) {
  return P.L <= 4 ? gradient<1>(P, s) : gradient<2>(P, s);
}

}  // namespace rsv
