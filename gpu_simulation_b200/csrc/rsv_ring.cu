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
// independent chains, each a D x D matrix (ket bits x bra bits) per component;
// (abar, a) has the conjugate transposes of (a, abar), so D (D + 1) / 2 are carried.
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
//   ring_grad_kernel: up to eight CTAs a site.  From the left components before
//     and the right components after the site: dE/dT[s; s'] summed over chains
//     and components on the tensor cores, then the site's 2 L derivatives.
// Both are bound by latency (n dependent sites of two small products), not by
// memory or arithmetic throughput.
//
// energy_and_grad at L = 4: n = 12 27 us (tile passes 142), n = 16 29 us (144),
// n = 24 37 us (1590), n = 28 38 us (21 400).  L = 5 (16 x 16 matrices): n = 16
// 180 us (194), n = 20 220 us (325), n = 24 254 us (2630).  At L = 4 a site of a
// sweep takes about 0.6 us: two products of dependent MMAs, the elementwise step
// and a barrier; at L = 5 ten component warps share an SM's FP64 tensor pipe, so
// the products' zero tiles are left out.
#include <cuda_runtime.h>

#include <atomic>

#include "rsv_device.cuh"
#include "rsv_launch.h"
#include "rsv_ring.h"

namespace rsv {
namespace {

constexpr int kComps = 5;  // I, X, H, W, S
constexpr int kI = 0, kX = 1, kH = 2, kW = 3, kS = 4;
constexpr int kSweepThreads = 32 * (kComps + 1);
constexpr int kGradWarps = kRingGradWarps;
static_assert(kGradWarps == 2 * kComps, "two warps a component");
constexpr int kMaxDerivs = kRingDerivs;

struct SiteM {  // cos, sin of the full angles of a wire's last layer
  double ct, st, cp, sp;
};

// An 8 R x 8 C complex matrix in a warp's registers: tile (i, j), element e of
// lane l is row 8 i + l / 4, column 8 j + 2 (l % 4) + e.
template <int R, int C>
struct Mat {
  double re[R][C][2], im[R][C][2];
};

__device__ __forceinline__ int frag_row(int i, int lane) { return 8 * i + lane / 4; }
__device__ __forceinline__ int frag_col(int j, int lane, int e) { return 8 * j + 2 * (lane % 4) + e; }
// D x D matrices in memory keep that order, [tile][element][lane] (D = 8 DB):
// where element (row, col) is.
template <int DB>
__device__ __forceinline__ int frag_at(int row, int col) {
  return (row / 8 * DB + col / 8) * 64 + 32 * (col & 1) + (row % 8) * 4 + (col % 8) / 2;
}

template <int R, int C, typename F>
__device__ __forceinline__ void elements(F &&f) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) f(i, j, e);
}

template <int R, int C>
__device__ __forceinline__ Mat<R, C> zero_mat() {
  Mat<R, C> m;
  elements<R, C>([&](int i, int j, int e) { m.re[i][j][e] = m.im[i][j][e] = 0.0; });
  return m;
}
template <int DB>
__device__ __forceinline__ void store_mat(double2 *p, const Mat<DB, DB> &m, int lane) {
  elements<DB, DB>([&](int i, int j, int e) {
    p[(i * DB + j) * 64 + 32 * e + lane] = make_double2(m.re[i][j][e], m.im[i][j][e]);
  });
}
template <int DB>
__device__ __forceinline__ Mat<DB, DB> load_mat(const double2 *p, int lane) {
  Mat<DB, DB> m;
  elements<DB, DB>([&](int i, int j, int e) {
    const double2 v = p[(i * DB + j) * 64 + 32 * e + lane];
    m.re[i][j][e] = v.x;
    m.im[i][j][e] = v.y;
  });
  return m;
}

// Z[m][n] += sum_k A[m][k] B[n][k], A conjugated when CONJ; of Z's tiles only
// those with m == n when OUTD, and only B's tiles with n == k when BD, A's
// with m == k when AD (the others are zero).  `n0`: the tile row of B that its
// first one is.
template <bool CONJ, bool OUTD, bool BD, bool AD, int R, int C, int K>
__device__ __forceinline__ void mma_rows(Mat<R, C> &Z, const Mat<R, K> &A, const Mat<C, K> &B, int n0 = 0) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) {
      if (OUTD && i != j) continue;
      double r0 = Z.re[i][j][0], r1 = Z.re[i][j][1], q0 = 0.0, q1 = 0.0;
      double s0 = Z.im[i][j][0], s1 = Z.im[i][j][1], t0 = 0.0, t1 = 0.0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (BD && j + n0 != k) continue;
        if (AD && i != k) continue;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          mma_f64(r0, r1, A.re[i][k][e], B.re[j][k][e]);
          mma_f64(q0, q1, A.im[i][k][e], B.im[j][k][e]);
          mma_f64(s0, s1, A.re[i][k][e], B.im[j][k][e]);
          mma_f64(t0, t1, A.im[i][k][e], B.re[j][k][e]);
        }
      }
      Z.re[i][j][0] = CONJ ? r0 + q0 : r0 - q0;
      Z.re[i][j][1] = CONJ ? r1 + q1 : r1 - q1;
      Z.im[i][j][0] = CONJ ? s0 - t0 : s0 + t0;
      Z.im[i][j][1] = CONJ ? s1 - t1 : s1 + t1;
    }
}

// T . V . T^+: first the bra columns (conj T), then the ket rows; `T` is in
// shared memory in matrix order.  IND: V's off-diagonal tiles are zero; OUTD:
// only the result's diagonal tiles are wanted (the others come back zero).
template <int DB, bool IND, bool OUTD>
__device__ __forceinline__ Mat<DB, DB> sandwich(const double2 *T, const Mat<DB, DB> &V, int lane) {
  const Mat<DB, DB> t = load_mat<DB>(T, lane);
  Mat<DB, DB> z = zero_mat<DB, DB>();
  mma_rows<true, false, IND, false>(z, t, V);   // z[bra][ket]
  Mat<DB, DB> y = zero_mat<DB, DB>();
  mma_rows<false, OUTD, false, false>(y, t, z);  // y[ket][bra]
  return y;
}
template <int DB>
__device__ __forceinline__ Mat<DB, DB> sandwich(const double2 *T, const Mat<DB, DB> &V, bool ind, bool outd, int lane) {
  if constexpr (DB > 1) {
    if (ind && outd) return sandwich<DB, true, true>(T, V, lane);
    if (ind) return sandwich<DB, true, false>(T, V, lane);
    if (outd) return sandwich<DB, false, true>(T, V, lane);
  }
  return sandwich<DB, false, false>(T, V, lane);
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
  const int tile = e / 64, lane = e % 32;
  r = frag_row(tile / DB, lane);
  c = frag_col(tile % DB, lane, (e / 32) & 1);
}

// Chain k is the k-th pair a <= ab (by ab, then a); the pair (ab, a) has the
// conjugate transposes of its matrices and is not carried.
__device__ __forceinline__ void chain_pair(int k, int &a, int &ab) {
  ab = 0;
  while ((ab + 1) * (ab + 2) / 2 <= k) ++ab;
  a = k - ab * (ab + 1) / 2;
}

// The bit of a bond index that is the wire's value before the last layer.
__device__ __forceinline__ int last_bit(int v, int nb) { return nb > 0 ? (v >> (nb - 1)) & 1 : 0; }

template <int DB>
constexpr size_t sweep_smem_bytes(int n, int L) {
  return sizeof(double2) * (static_cast<size_t>(L > 1 ? L - 1 : 0) * n * 4 + (2 + 6) * 64 * DB * DB) +
         sizeof(SiteM) * static_cast<size_t>(n);
}

// Applies f(i, j, e, bra bit, ket bit) to every element of a lane (tile rows
// from i0); the bits are those before the last layer, flipped by fb / fk (wire
// 0: the arriving bits).
template <int R, int C, typename F>
__device__ __forceinline__ void each(int lane, int nb, int fk, int fb, F &&f, int i0 = 0) {
  elements<R, C>([&](int i, int j, int e) {
    f(i, j, e, last_bit(frag_col(j, lane, e), nb) ^ fb, last_bit(frag_row(i0 + i, lane), nb) ^ fk);
  });
}

// Left components after a site from those before its last layer (t*), for
// component c of wire w (1 <= w < n - 1) or, at the last wire, the energy share
// of every component.
template <int DB>
__global__ void __launch_bounds__(kSweepThreads) ring_sweep_kernel(const RingParams P, int first_dir, int keep) {
  constexpr int D = 8 * DB, DD = D * D;
  extern __shared__ double2 smem[];
  const int n = P.n, L = P.L, nb = L - 1;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int chains = gridDim.x, chain = blockIdx.x;
  const bool rightward = first_dir + static_cast<int>(blockIdx.y) == 0;
  int a, ab;
  chain_pair(chain, a, ab);
  double2 *U = smem;                       // [nb][n][4]
  double2 *T = U + nb * n * 4;             // [2][DD]
  double2 *ex = T + 2 * DD;                // [2][3][DD]
  SiteM *M = reinterpret_cast<SiteM *>(ex + 6 * DD);  // [n]
  const int tid = threadIdx.x, lane = tid & 31;
  // W and I, the components with the fewest products, share a scheduler
  constexpr int kCompOf[kComps + 1] = {kW, kH, kX, kS, kI, kComps};
  const int comp = kCompOf[tid >> 5];
  for (int k = tid; k < L * n; k += kSweepThreads) {
    double4 v;
    if (P.params) {
      sincos(P.params[2 * k] * 0.5, &v.y, &v.x);
      sincos(P.params[2 * k + 1] * 0.5, &v.w, &v.z);
      if (blockIdx.x == 0 && blockIdx.y == 0) P.coef[k] = v;  // for the gradient kernel
    } else {
      v = P.coef[k];
    }
    if (k < nb * n) site_u(v, U + 4 * k);
    else M[k - nb * n] = site_m(v);
  }
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
    Mat<DB, DB> v;
    if (comp < kComps) {
      const SiteM m = M[0];
      each<DB, DB>(lane, nb, last_bit(a, nb), last_bit(ab, nb), [&](int i, int j, int e, int bra, int ket) {
        const double2 uk = t0_entry(U, ustride, nb, frag_row(i, lane), a);
        const double2 ub = t0_entry(U, ustride, nb, frag_col(j, lane, e), ab);
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
      const SiteM m = M[w];
      if (comp < kComps) {
        // behind an identity the bra and ket bits agree (at L = 5 the
        // off-diagonal tiles are zero), and of H and W only what the next
        // identity keeps is used
        v = sandwich<DB>(T + p * DD, v, (comp == kI && w > 1) || (comp == kW && w > 2),
                         comp == kH || (comp == kW && w < n - 1), lane);
        if (keep) store_mat<DB>(P.left + ((static_cast<size_t>(w) * chains + chain) * kComps + comp) * DD, v, lane);
        if (comp == kI) store_mat<DB>(xI, v, lane);
        if (comp == kX) store_mat<DB>(xX, v, lane);
      } else if (w + 1 < n) {
        build(w + 1, T + (p ^ 1) * DD, lane, 32);
      }
      __syncthreads();
      if (w == n - 1) break;
      if (comp == kI || (comp == kW && w > 1) || (comp == kS && w == 1)) {
        each<DB, DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          if (bra != ket) v.re[i][j][e] = v.im[i][j][e] = 0.0;
        });
      } else if (comp == kX || comp == kW) {
        const double2 *src = comp == kX ? xI : xX;
        each<DB, DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          const double2 x = cmul(m_x(m, bra, ket), src[(i * DB + j) * 64 + 32 * e + lane]);
          v.re[i][j][e] = x.x;
          v.im[i][j][e] = x.y;
        });
      } else if (comp == kH) {
        each<DB, DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
          const int at = (i * DB + j) * 64 + 32 * e + lane;
          const double2 x = cmul(m_x(m, bra, ket), xX[at]);
          const double z = w == 1 ? 0.0 : m_z(m, bra, ket);
          const double2 t = xI[at];
          const double keep_re = bra == ket ? v.re[i][j][e] : 0.0, keep_im = bra == ket ? v.im[i][j][e] : 0.0;
          v.re[i][j][e] = keep_re - z * t.x - h * x.x;
          v.im[i][j][e] = keep_im - z * t.y - h * x.y;
        });
      } else if (comp == kS) {
        each<DB, DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
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
      each<DB, DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
        if (frag_row(i, lane) != a || frag_col(j, lane, e) != ab) return;
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
      const double s = ((share[kI] + share[kX]) + (share[kH] + share[kW])) + share[kS];
      P.energy_parts[chain] = a == ab ? s : 2.0 * s;
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
  Mat<DB, DB> v = zero_mat<DB, DB>();
  if (comp == kH || comp == kS)
    each<DB, DB>(lane, nb, 0, 0, [&](int i, int j, int e, int, int) {
      if (frag_row(i, lane) == a && frag_col(j, lane, e) == ab) v.re[i][j][e] = 1.0;
    });
  for (int w = n - 1; w >= 1; --w) {
    const int p = (n - 1 - w) & 1;
    double2 *xH = ex + p * 3 * DD, *xX = xH + DD, *xW = xX + DD;
    if (comp == kH) store_mat<DB>(xH, v, lane);
    if (comp == kX) store_mat<DB>(xX, v, lane);
    if (comp == kW && w == 1) store_mat<DB>(xW, v, lane);
    if (comp < kComps && w < n - 1)
      store_mat<DB>(P.right + ((static_cast<size_t>(w) * chains + chain) * kComps + comp) * DD, v, lane);
    const SiteM m = M[w];
    __syncthreads();
    if (comp == kComps) {
      if (w > 1) build(w - 1, T + (p ^ 1) * DD, lane, 32);
      continue;
    }
    each<DB, DB>(lane, nb, 0, 0, [&](int i, int j, int e, int bra, int ket) {
      const int at = (i * DB + j) * 64 + 32 * e + lane;
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
    v = sandwich<DB>(T + p * DD, v, comp == kH || (comp == kW && w < n - 1),
                     (comp == kI && w > 1) || (comp == kW && w > 2), lane);
  }
  if (comp < kComps)
    store_mat<DB>(P.right + (static_cast<size_t>(chain) * kComps + comp) * DD, v, lane);
}

// Rows [8 i0, ...) of a D x D matrix in shared memory (matrix order), or of its
// conjugate transpose; conjugated once more when `conj`.
template <int DB, int R>
__device__ __forceinline__ Mat<R, DB> load_rows(const double2 *p, bool mirror, int i0, bool conj, int lane) {
  Mat<R, DB> m;
  const int base = mirror ? 32 * ((lane / 4) & 1) + 8 * (lane % 4) + lane / 8 : lane;
  const int di = mirror ? 64 : 64 * DB, dj = mirror ? 64 * DB : 64, de = mirror ? 4 : 32;
  const double sign = mirror != conj ? -1.0 : 1.0;
  elements<R, DB>([&](int i, int j, int e) {
    const double2 v = p[base + (i0 + i) * di + j * dj + e * de];
    m.re[i][j][e] = v.x;
    m.im[i][j][e] = sign * v.y;
  });
  return m;
}

// Chains of one step of ring_grad_kernel: 256 elements of each matrix kind.
template <int DB>
__host__ __device__ constexpr int chains_a_step() {
  return ring_chains_a_step(DB == 1 ? 4 : 5);
}

__device__ __forceinline__ void copy16(double2 *to, const double2 *from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(to))),
               "l"(from)
               : "memory");
}

// A site's CTAs share the chains, NC at a time.  The chains'
// left components before and at the site and their right components are staged
// in shared memory (cp.async, one step ahead); all threads turn them into the
// products' operands V_c (left, before the site) and R_c (right, behind the
// site's last layer) and take that layer's sums; then the warps form
//   y[s'][bra] = sum V[s'][.] conj(T[bra][.]),  dE/dT[s][s'] += sum R[s][bra] y[s'][bra]
// on the tensor cores: a warp has one component, and at L <= 4 the chain's pair
// (a, ab) or its mirror (ab, a), at L = 5 both and one of the two tile rows of s'.
// (Operands formed by every warp for itself: 480 us at n = 20, L = 5.)
template <int DB>
__global__ void __launch_bounds__(32 * kGradWarps, 1) ring_grad_kernel(const RingParams P) {
  constexpr int D = 8 * DB, DD = D * D, kSlices = kGradWarps / DB;
  extern __shared__ double2 smem[];
  __shared__ double2 Uw[4 * (kRingMaxLayers - 1)], U0[4 * (kRingMaxLayers - 1)];
  __shared__ double red[kGradWarps][kMaxDerivs];
  double2 *T = smem;              // [DD] T_w
  double2 *T0 = T + DD;           // [DD] T_0
  double2 *G = T0 + DD;           // [kSlices][DD]
  constexpr int NC = chains_a_step<DB>(), kSet = kComps * DD;
  double2 *stages = G + kSlices * DD;   // [2][NC][3][kComps][DD]
  double2 *ops = stages + 6 * NC * kSet;  // [NC][2][kComps][DD]
  const int G_ctas = static_cast<int>(gridDim.x), rank = static_cast<int>(blockIdx.x), w = static_cast<int>(blockIdx.y);
  const int n = P.n, L = P.L, nb = L - 1, bond = 1 << nb, chains = bond * (bond + 1) / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < kSlices * DD; e += 32 * kGradWarps) G[e] = make_double2(0.0, 0.0);
  // launched while the sweeps end: their results from here on
  asm volatile("griddepcontrol.wait;" ::: "memory");
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
  __syncthreads();
  const double h = P.field;
  const SiteM m = site_m(P.coef[nb * n + w]), m1 = site_m(P.coef[nb * n + (w > 0 ? w - 1 : 0)]);
  // d/dtheta and d/dphi of M_X and M_Z of this site
  const SiteM mt{-m.st, m.ct, m.cp, 0.0};   // theta: M_X keeps its cos(phi) part
  const SiteM mp{m.ct, m.st, -m.sp, m.cp};  // phi
  double g_theta = 0.0, g_phi = 0.0;
  const int worker = rank * kGradWarps + warp, workers = G_ctas * kGradWarps;
  if (w == 0) {
    // T_0's column a from the pairs (a, .): sum over the bra bits and over ab
    const int share = workers / bond;  // warps a column (one at least: ring_gradient_ctas)
    if (worker < share * bond) {
      const int a = worker % bond;
      double gr[DB], gi[DB];
#pragma unroll
      for (int i = 0; i < DB; ++i) gr[i] = gi[i] = 0.0;
      for (int ab = worker / bond; ab < bond; ab += share) {
        const int lo = a < ab ? a : ab, hi = a < ab ? ab : a;
        const double2 *right = P.right + static_cast<size_t>(hi * (hi + 1) / 2 + lo) * kSet;
        const Mat<DB, DB> rI = load_rows<DB, DB>(right + kI * DD, a > ab, 0, false, lane);
        const Mat<DB, DB> rX = load_rows<DB, DB>(right + kX * DD, a > ab, 0, false, lane);
        const Mat<DB, DB> rH = load_rows<DB, DB>(right + kH * DD, a > ab, 0, false, lane);
        const Mat<DB, DB> rS = load_rows<DB, DB>(right + kS * DD, a > ab, 0, false, lane);
        each<DB, DB>(lane, nb, last_bit(a, nb), last_bit(ab, nb), [&](int i, int j, int e, int bra, int ket) {
          const double2 uk = T0[frag_at<DB>(frag_row(i, lane), a)];
          const double2 ub = T0[frag_at<DB>(frag_col(j, lane, e), ab)];
          const double2 x = make_double2(rX.re[i][j][e], rX.im[i][j][e]);
          const double2 q = make_double2(-(rH.re[i][j][e] + rS.re[i][j][e]), -(rH.im[i][j][e] + rS.im[i][j][e]));
          const double z = m_z(m, bra, ket);
          double2 r = cmul(m_x(m, bra, ket), x);
          r.x += z * q.x;
          r.y += z * q.y;
          if (bra == ket) {
            r.x += rI.re[i][j][e];
            r.y += rI.im[i][j][e];
          }
          r = cmul_conj(r, ub);
          gr[i] += r.x;
          gi[i] += r.y;
          const double2 v = cmul_conj(uk, ub);
          const double2 qx = cmul(v, x), qz = cmul(v, q);
          const double2 xt = m_x(mt, bra, ket), xp = m_x(mp, bra, ket);
          g_theta += xt.x * qx.x - xt.y * qx.y + m_z(mt, bra, ket) * qz.x;
          g_phi += xp.x * qx.x - xp.y * qx.y;
        });
      }
#pragma unroll
      for (int i = 0; i < DB; ++i) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          gr[i] += __shfl_xor_sync(0xffffffffu, gr[i], o);
          gi[i] += __shfl_xor_sync(0xffffffffu, gi[i], o);
        }
        // element (row, a); the warps of a slice have different columns
        if (lane % 4 == 0) G[(warp / DB) * DD + frag_at<DB>(frag_row(i, lane), a)] = make_double2(gr[i], gi[i]);
      }
    }
  } else {
    const int c = warp / 2, js = DB == 1 ? 0 : warp % 2;
    const bool end = w == n - 1, first = w == 1, second = w == 2;
    auto fetch = [&](int chain0, double2 *to) {
      for (int k = 0; k < NC && chain0 + k < chains; ++k, to += 3 * kSet) {
        const size_t chain = static_cast<size_t>(chain0 + k);
        const double2 *before = P.left + (static_cast<size_t>(w - 1) * chains + chain) * kSet;
        const double2 *here = P.left + (static_cast<size_t>(w) * chains + chain) * kSet;
        const double2 *right = P.right + (static_cast<size_t>(w) * chains + chain) * kSet;
        for (int e = tid; e < kSet; e += 32 * kGradWarps) {
          if (!first) copy16(to + e, before + e);  // (site 0's are formed from T_0)
          copy16(to + kSet + e, here + e);
          if (!end) copy16(to + 2 * kSet + e, right + e);  // (the closed end's are 0 or 1)
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int step = G_ctas * NC;
    Mat<DB, 1> g = zero_mat<DB, 1>();
    fetch(rank * NC, stages);
    for (int chain0 = rank * NC, k = 0; chain0 < chains; chain0 += step, ++k) {
      const double2 *stage = stages + (k & 1) * 3 * NC * kSet;
      fetch(chain0 + step, stages + ((k & 1) ^ 1) * 3 * NC * kSet);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      for (int q = tid; q < NC * DD; q += 32 * kGradWarps) {
        const int sub = q / DD, e = q % DD;
        if (chain0 + sub >= chains) break;
        int a, ab, row, col;
        chain_pair(chain0 + sub, a, ab);
        order_rc<DB>(e, row, col);
        const double2 *B = stage + sub * 3 * kSet + e, *S = B + kSet, *R = S + kSet;
        double2 *V = ops + sub * 2 * kSet + e, *O = V + kSet;
        const double2 zero = make_double2(0.0, 0.0);
        auto scaled = [](double f, double2 x) { return make_double2(f * x.x, f * x.y); };
        auto plus = [](double2 x, double2 y) { return make_double2(x.x + y.x, x.y + y.y); };
        int bra = last_bit(col, nb), ket = last_bit(row, nb);
        if (first) {
          const int b0 = bra ^ last_bit(ab, nb), k0 = ket ^ last_bit(a, nb);
          const double2 v = cmul_conj(T0[frag_at<DB>(row, a)], T0[frag_at<DB>(col, ab)]);
          const double2 zv = scaled(-m_z(m1, b0, k0), v);
          V[kI * DD] = b0 == k0 ? v : zero;
          V[kX * DD] = cmul(m_x(m1, b0, k0), v);
          V[kH * DD] = zv;
          V[kW * DD] = zero;
          V[kS * DD] = zv;
        } else {
          const double2 x1 = m_x(m1, bra, ket), tI = B[kI * DD], tX = cmul(x1, B[kX * DD]);
          const double z1 = m_z(m1, bra, ket);
          double2 hh = scaled(-h, tX);
          if (!second) hh = plus(hh, scaled(-z1, tI));
          if (bra == ket) hh = plus(hh, B[kH * DD]);
          V[kI * DD] = bra == ket ? tI : zero;
          V[kX * DD] = cmul(x1, tI);
          V[kH * DD] = hh;
          V[kW * DD] = second ? tX : (bra == ket ? B[kW * DD] : zero);
          V[kS * DD] = second ? (bra == ket ? B[kS * DD] : zero) : scaled(z1, B[kS * DD]);
        }
        const double2 x = m_x(m, bra, ket);
        const double z = m_z(m, bra, ket);
        const double2 one = make_double2(row == a && col == ab ? 1.0 : 0.0, 0.0);
        const double2 rI = end ? zero : R[kI * DD], rX = end ? zero : R[kX * DD], rH = end ? one : R[kH * DD];
        const double2 rW = end ? zero : R[kW * DD], rS = end ? one : R[kS * DD];
        const double2 hH = scaled(-h, rH);
        double2 o = cmul(x, rX);
        if (bra == ket) o = plus(o, rI);
        O[kI * DD] = first ? o : plus(o, scaled(-z, rH));
        const double2 xx = first ? plus(hH, rW) : hH;
        O[kX * DD] = cmul(x, xx);
        O[kH * DD] = bra == ket ? rH : zero;
        O[kW * DD] = end ? cmul(x, hH) : (first || bra != ket ? zero : rW);
        O[kS * DD] = first ? (bra == ket ? rS : zero) : scaled(z, rS);
        // the last layer's sums; the mirrored pair's are their conjugates
        double2 qx = plus(cmul(S[kI * DD], rX), cmul(S[kX * DD], xx));
        if (end) qx = plus(qx, cmul(S[kW * DD], hH));
        const double twice = a == ab ? 1.0 : 2.0;
        const double2 xt = m_x(mt, bra, ket), xp = m_x(mp, bra, ket);
        double dt = xt.x * qx.x - xt.y * qx.y;
        if (!first) dt += m_z(mt, bra, ket) * (cmul(S[kS * DD], rS).x - cmul(S[kI * DD], rH).x);
        g_theta += twice * dt;
        g_phi += twice * (xp.x * qx.x - xp.y * qx.y);
      }
      __syncthreads();
      const Mat<DB, DB> t = load_mat<DB>(T, lane);
#pragma unroll 1
      for (int sub = 0; sub < NC && chain0 + sub < chains; ++sub) {
        int a, ab;
        chain_pair(chain0 + sub, a, ab);
        const double2 *V = ops + sub * 2 * kSet + c * DD, *O = V + kSet;
#pragma unroll 1
        for (int mirror = DB == 1 ? warp % 2 : 0; mirror < (a == ab ? 1 : 2); mirror += DB == 1 ? 2 : 1) {
          const Mat<1, DB> v = load_rows<DB, 1>(V, mirror != 0, js, true, lane);
          Mat<1, DB> y = zero_mat<1, DB>();
          mma_rows<false, false, false, false>(y, v, t);  // conj(V) T: the conjugate of y
          elements<1, DB>([&](int i, int j, int e) { y.im[i][j][e] = -y.im[i][j][e]; });
          const Mat<DB, DB> r = load_rows<DB, DB>(O, mirror != 0, 0, false, lane);
          // (an identity's R: at L = 5 its off-diagonal tiles are zero)
          if (DB > 1 && (c == kH || (c == kW && !end))) mma_rows<false, false, false, true>(g, r, y);
          else mma_rows<false, false, false, false>(g, r, y);
        }
      }
      __syncthreads();  // the operands are read
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    elements<DB, 1>([&](int i, int, int e) {
      G[(warp / DB) * DD + (i * DB + js) * 64 + 32 * e + lane] = make_double2(g.re[i][0][e], g.im[i][0][e]);
    });
  }
  __syncthreads();
  // The site's derivatives from dE/dT = 2 Re sum G dT (linear: every CTA its part)
  double d[kMaxDerivs];
#pragma unroll
  for (int k = 0; k < kMaxDerivs; ++k) d[k] = 0.0;
  for (int e = tid; e < DD; e += 32 * kGradWarps) {
    double2 g = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < kSlices; ++k) {
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
  // this CTA's part; the site's last CTA to finish adds them in order
  double *parts = P.grad_parts + static_cast<size_t>(w) * G_ctas * kMaxDerivs;
  if (tid < kMaxDerivs) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kGradWarps; ++k) s += red[k][tid];
    parts[rank * kMaxDerivs + tid] = s;
    __threadfence();
  }
  __shared__ bool last;
  __syncthreads();
  if (tid == 0)
    last = atomicInc(P.counter + 1 + w, static_cast<unsigned>(G_ctas - 1)) == static_cast<unsigned>(G_ctas - 1);
  __syncthreads();
  if (last && tid < 2 * L) {
    __threadfence();
    double s = 0.0;
    for (int k = 0; k < G_ctas; ++k) s += __ldcg(parts + k * kMaxDerivs + tid);
    // a NaN energy (a non-finite angle) voids the whole gradient
    const double energy = P.energy_parts[chains];
    if (energy != energy) s = energy;
    P.grad_out[static_cast<size_t>(tid / 2 * n + w) * 2 + (tid & 1)] = s;
  }
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
  constexpr size_t smem = sizeof(double2) * (2 + kGradWarps / DB + 8 * chains_a_step<DB>() * kComps) * 64 * DB * DB;
  cudaError_t e = set_smem_limit_once(ring_grad_kernel<DB>, smem, done);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  const int ctas = ring_gradient_ctas(P.n, P.L, sms);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas), static_cast<unsigned>(P.n));
  cfg.blockDim = dim3(32 * kGradWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
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
