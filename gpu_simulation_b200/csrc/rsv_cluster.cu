// Energy and adjoint gradient of circuits whose whole state stays in one
// thread-block cluster: psi and lambda in registers, exchanged through the
// shared memory of the cluster's CTAs.  One launch does every layer, forward,
// energy and backward; circuits of one launch share their qubit count.
//
// A state of N qubits (n padded to at least 7 with wires that do nothing) is
// spread over 2^c CTAs with 2^(N-c-R) threads each; a thread holds the 2^R
// amplitudes of R index bits, its register bits.  K layouts cover the wires:
//   layout k < K-1: register bits [lo_k, lo_k + R), lo_k = min(R k, N - 2R);
//                   the CTA holds the index bits [N-c, N) ("top" class);
//   layout K-1:     register bits [N-R, N); the CTA holds the bits [0, c)
//                   ("low" class), so the top c wires are in registers.
// A change of layout writes every amplitude where its next owner reads it:
// within the CTA between the first layouts, into the other CTAs' shared memory
// (st.shared::cluster) into and out of the last one.  The CNOT ring is such a
// change: after a layer's last layout the amplitude x goes to P(x) of the next
// layer's layout 0, and the backward sends it from layout 0 to P^-1(x) of the
// last layout.  So a layer costs K exchanges of each vector, two of them across
// CTAs, and no memory traffic.  All exchange addresses are linear in the index
// over GF(2) (the bank swizzle too): a base per thread and one XOR with a
// constant per amplitude.  In layouts 0 and K-1, whose register bits decide the
// next CTA, register r holds the index bits r ^ rank: the CTAs then write to
// different CTAs at any time instead of all to the same one.
//
// Gates are applied in tangent form: RY / f = [[1, -k], [k, 1]] with k = tan t/2
// where |cos| >= |sin|, else J [[1, -k], [k, 1]] with k = -cot t/2 and J = [[0, -1],
// [1, 0]]; 1 + k^2 = 1 / f^2 <= 2.  J costs nothing: its swap is an XOR on the
// address that the registers are stored to (or, backward, loaded from), its
// sign and the layer's product K_l of the f ride on the RZ phase.  (J commutes
// with RY's generator, so a theta sum may be taken after J is undone.)  Backward, D^+ K_l is applied first, so a layer
// starts and ends with true vectors, and a theta sum taken while the wires S
// are still to undo is K_S^2 times the true one (prod (1 + k^2) undoes that).  The
// gates of a layout commute, so their sums are taken together before any of
// them is undone.  phi sums are taken on the true vectors at the layer's start:
// sum_i z_w(i) Im(conj(lambda_i) psi_i).
//
// With checkpoints (CK) the forward writes psi behind every layout's rotations
// to memory, 2^R amplitudes a thread in the thread's own order, and the backward
// reads them back instead of un-computing psi: only lambda is rotated and
// exchanged, and a theta or phi sum with a checkpoint needs no correction (psi
// there is 1 / K_S of what un-computing gives, which is what the sum lacks).
// Layer 0's psi is the product state and is un-computed.
//
// Sums go through fixed orders (lanes, warps, CTAs): equal inputs give equal bits.
//
// Bound by latency up to 12 qubits (one launch against one a layer and pass:
// energy and gradient at L = 8, n = 8 246 -> 18.7 us, n = 10 256 -> 31, n = 12
// 269 -> 64) and by the stores into other CTAs above (about 9 to 12 bytes a clock
// and SM; n = 14 327 -> 120 us, n = 16 336 -> 293).  Every shape is its own
// instantiation: with the layouts' arithmetic at run time n = 8 took 58 us and
// n = 12 118, most of it integer and address latency.
#include <cuda_runtime.h>

#include <atomic>

#include "rsv_cluster.h"
#include "rsv_device.cuh"
#include "rsv_launch.h"

namespace rsv {
namespace {

constexpr size_t kMostSmem = 227 * 1024;
// A layer's record: theta sums of 16 wires, then phi values: register bits (4), total, lane bits (5)
constexpr int kRec = 32;
constexpr int kRecPhi = 16, kRecTotal = 20, kRecLane = 21;

#define RSV_HD __host__ __device__ __forceinline__ constexpr

RSV_HD unsigned ring_map(unsigned x, int n) {  // P (rsv_device.cuh, at most 16 bits)
  const unsigned mask = (1u << n) - 1;
  unsigned p = x & mask;
  p ^= p << 1;
  p ^= p << 2;
  p ^= p << 4;
  p ^= p << 8;
  p &= mask;
  return (x & ~mask) | (p & ~1u) | (((p >> (n - 1)) ^ x) & 1u);
}
RSV_HD unsigned ring_unmap(unsigned x, int n) {  // P^-1
  const unsigned mask = (1u << n) - 1;
  return (x & ~mask) | ((((x & mask) ^ ((x & mask) << 1)) & mask) ^ (((x >> (n - 1)) & 1u) * 3u));
}

// Where the amplitude x of an N-qubit state lies in a class: CTA << 24 | byte
// offset of its 16-byte slot, swizzled so that any three neighbouring local
// bits select the bank group.  Linear over GF(2).
RSV_HD unsigned slot(unsigned p) { return (p ^ (((p >> 3) ^ (p >> 6) ^ (p >> 9)) & 7u)) << 4; }
RSV_HD unsigned place_top(unsigned x, int m) { return ((x >> m) << 24) | slot(x & ((1u << m) - 1)); }
RSV_HD unsigned place_low(unsigned x, int c) { return ((x & ((1u << c) - 1)) << 24) | slot(x >> c); }
// t with R zero bits inserted at bit `at`
RSV_HD unsigned spread(unsigned t, int at, int R) { return (t & ((1u << at) - 1)) | ((t >> at) << (at + R)); }

// n qubits on 2^C CTAs, 2^R amplitudes a thread.
template <int n_, int R_, int C_>
struct Geo {
  static constexpr int n = n_, R = R_, C = C_, N = n < 7 ? 7 : n, m = N - C, NR = 1 << R, ctas = 1 << C;
  static constexpr int bits = m - R, threads = 1 << bits, warps = threads / 32;
  static constexpr int K = (N - 1) / R + 1;         // layouts
  static constexpr int tables = (N - R + 3) / 4 + 1;  // phase tables of four index bits, the last of the register bits
  static_assert(C <= R && bits >= 5 && m <= 12 && threads <= 1024, "cluster shape");

  RSV_HD static int lo(int k) { return k == K - 1 ? N - R : (R * k < N - 2 * R ? R * k : N - 2 * R); }
  // wire of register bit j in layout k, or -1 where an earlier layout has it
  RSV_HD static int wire(int k, int j) {
    return k == K - 1 || (lo(k) + j >= R * k && lo(k) + j < N - R) ? lo(k) + j : -1;
  }
  // wires still to undo when the backward is in layout k
  RSV_HD static int pending(int w) { return w >= N - R ? n : (w / R * R + R < N - R ? w / R * R + R : N - R); }
  // Local index (of its class) of a thread's register 0.  In layout K-2 the last
  // bits of the thread number are the low C index bits, which name the CTA of
  // the layout that follows: a warp's stores into it go to as few CTAs as possible.
  RSV_HD static unsigned local(int k, unsigned tid) {
    if (k == K - 1) return tid;
    if (k == K - 2) tid = ((tid << C) | (tid >> (bits - C))) & (threads - 1u);
    return spread(tid, lo(k), R);
  }
  RSV_HD static unsigned index(int k, unsigned rank, unsigned tid) {
    const unsigned p = local(k, tid);
    const unsigned x = k == K - 1 ? (p << C) | rank : (rank << m) | p;
    return k == 0 || k == K - 1 ? x ^ (rank << lo(k)) : x;
  }
  RSV_HD static unsigned own(int k, unsigned x) {  // own slot of amplitude x in layout k
    return (k == K - 1 ? place_low(x, C) : place_top(x, m)) & 0xffffffu;
  }
  // what register bit j adds to the addresses: own slots, the ring (to the top
  // class, or the low one), its inverse, the changes K-1 -> K-2 and K-2 -> K-1
  RSV_HD static unsigned own_bit(int k, int j) { return own(k, 1u << (lo(k) + j)); }
  RSV_HD static unsigned ring_bit(int j) { return place_top(ring_map(1u << (N - R + j), n), m); }
  RSV_HD static unsigned ring_low_bit(int j) { return place_low(ring_map(1u << (N - R + j), n), C); }
  RSV_HD static unsigned unring_bit(int j) { return place_low(ring_unmap(1u << j, n), C); }
  RSV_HD static unsigned down_bit(int j) { return place_top(1u << (N - R + j), m); }
  RSV_HD static unsigned up_bit(int j) { return place_low(1u << (lo(K - 2) + j), C); }
};

// Shared memory of a CTA: two exchange buffers (16 * 2^m bytes each), then
struct Tables {
  double2 *phase;        // [L][tables][16]: K_l e^{+-i phi / 2} products with J's signs
  double2 *prod;         // [tables][16]: the same for layer 0's product state
  double *rot;           // [L][N] k
  double *rec;           // [L][kRec]
  double *tot;           // [L][warps] phi totals
  double *red;           // [2][warps][32], then 4 scalars
  double *scale;         // [L] K_l
  unsigned *flip;        // [L] wires with a J
};
template <typename G>
RSV_HD size_t doubles_of(int L) {  // everything behind `prod` but `flip`
  return (static_cast<size_t>(L) * (G::N + kRec + G::warps + 1) + 64 * G::warps + 4 + 1) & ~size_t{1};
}
template <typename G>
RSV_HD size_t table_bytes(int L) {
  return 256 * static_cast<size_t>(G::tables) * (static_cast<size_t>(L) + 1) + 8 * doubles_of<G>(L) +
         4 * ((static_cast<size_t>(L) + 3) & ~size_t{3});
}
RSV_HD size_t trig_bytes(int n, int L) { return size_t{16} * n * (L + 1); }

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_address(unsigned addr, unsigned cta) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(cta));
  return a;
}
__device__ __forceinline__ void store_cluster(unsigned addr, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ double load_cluster(unsigned addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}

// Barrier of the CTA, and of the cluster in two halves: arrive() when this
// thread has read its slots, wait() before the next write into them.
template <typename G>
__device__ __forceinline__ void sync_cta() {
  if constexpr (G::threads == 32) __syncwarp();
  else __syncthreads();
}
template <typename G>
__device__ __forceinline__ void arrive() {
  if constexpr (G::C > 0) cluster_arrive();
}
template <typename G>
__device__ __forceinline__ void wait() {
  if constexpr (G::C > 0) cluster_wait();
  else sync_cta<G>();
}
template <typename G>
__device__ __forceinline__ void sync_all() {
  arrive<G>();
  wait<G>();
}

// Calls f(r, address of register r) for every register, in Gray-code order;
// bit(j) is what register bit j adds.
template <int R, typename B, typename F>
__device__ __forceinline__ void for_registers(unsigned base, B &&bit, F &&f) {
  unsigned at = base;
#pragma unroll
  for (int g = 0; g < (1 << R); ++g) {
    if (g > 0) {
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (((g ^ (g >> 1)) ^ ((g - 1) ^ ((g - 1) >> 1))) == (1 << j)) at ^= bit(j);
    }
    f(g ^ (g >> 1), at);
  }
}
template <typename G, typename B>
__device__ __forceinline__ void push(const double2 (&a)[G::NR], unsigned smem, unsigned base, B &&bit) {
  for_registers<G::R>(base, bit, [&](int r, unsigned p) {
    if constexpr (G::C > 0) store_cluster(cluster_address(smem + (p & 0xffffffu), p >> 24), a[r]);
    else store_cluster(smem + p, a[r]);
  });
}
template <typename G>
__device__ __forceinline__ void store_own(const double2 (&a)[G::NR], unsigned char *buf, int k, unsigned base) {
  for_registers<G::R>(base, [&](int j) { return G::own_bit(k, j); },
                      [&](int r, unsigned p) { *reinterpret_cast<double2 *>(buf + p) = a[r]; });
}
template <typename G>
__device__ __forceinline__ void load_own(double2 (&a)[G::NR], const unsigned char *buf, int k, unsigned base) {
  for_registers<G::R>(base, [&](int j) { return G::own_bit(k, j); },
                      [&](int r, unsigned p) { a[r] = *reinterpret_cast<const double2 *>(buf + p); });
}

// [[1, -k], [k, 1]] on register bit j
template <int R>
__device__ __forceinline__ void rotate(double2 (&a)[1 << R], int j, double k) {
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if ((r >> j) & 1) continue;
    const double2 x = a[r], y = a[r | (1 << j)];
    a[r] = make_double2(fma(-k, y.x, x.x), fma(-k, y.y, x.y));
    a[r | (1 << j)] = make_double2(fma(k, x.x, y.x), fma(k, x.y, y.y));
  }
}

// sum over the pairs of register bit j: Re(conj(l1) p0) - Re(conj(l0) p1)
template <int R>
__device__ __forceinline__ double theta_sum(const double2 (&p)[1 << R], const double2 (&l)[1 << R], int j) {
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if ((r >> j) & 1) continue;
    const int q = r | (1 << j);
    s0 = fma(l[q].x, p[r].x, s0);
    s1 = fma(l[r].x, p[q].x, s1);
    s0 = fma(l[q].y, p[r].y, s0);
    s1 = fma(l[r].y, p[q].y, s1);
  }
  return s0 - s1;
}

// The sums of 32 values over a warp: lane l returns that of v[l].
__device__ __forceinline__ double warp_sums32(double (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const double keep = up ? v[i + o] : v[i], send = up ? v[i] : v[i + o];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

template <bool V>
struct Flag {
  static constexpr bool value = V;
};

// One circuit on this cluster; `ck`: this CTA's checkpoints.
template <typename G, bool CK>
__device__ __forceinline__ void run_circuit(const ClusterArgs &A, const ClusterItem item, unsigned char *smem,
                                            double2 *ck) {
  constexpr int n = G::n, N = G::N, R = G::R, C = G::C, m = G::m, K = G::K, NR = G::NR, nt = G::tables;
  constexpr int threads = G::threads, warps = G::warps;
  const int L = item.L;
  const unsigned rank = blockIdx.x & ((1u << C) - 1), tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  unsigned char *bufP = smem, *bufL = smem + (size_t{16} << m);
  const unsigned smP = static_cast<unsigned>(__cvta_generic_to_shared(bufP));
  const unsigned smL = smP + (16u << m);
  Tables T;
  T.phase = reinterpret_cast<double2 *>(bufL + (size_t{16} << m));
  T.prod = T.phase + static_cast<size_t>(L) * nt * 16;
  T.rot = reinterpret_cast<double *>(T.prod + nt * 16);
  T.rec = T.rot + L * N;
  T.tot = T.rec + L * kRec;
  T.red = T.tot + L * warps;
  T.scale = T.red + 64 * warps + 4;
  T.flip = reinterpret_cast<unsigned *>(T.rot + doubles_of<G>(L));

  // ---- tables: tangent forms, then phases and the first layer's product state
  const double *params = A.params ? A.params + item.param_off : nullptr;
  // (cos, sin) of the half angles: phi of every wire, then theta of layer 0, in
  // the exchange buffers until the first exchange where they fit
  double2 *trig = trig_bytes(n, L) <= (size_t{32} << m) ? reinterpret_cast<double2 *>(smem)
                                                        : reinterpret_cast<double2 *>(T.flip + ((L + 3) & ~3));
  for (int l = tid; l < L; l += threads) T.flip[l] = 0;
  sync_cta<G>();
  for (int k = tid; k < L * n; k += threads) {
    double4 v;
    if (params) {
      sincos(params[2 * k] * 0.5, &v.y, &v.x);
      sincos(params[2 * k + 1] * 0.5, &v.w, &v.z);
    } else {
      v = A.coef[k];
    }
    if (A.coef_out && rank == 0) A.coef_out[k] = v;
    trig[k] = make_double2(v.z, v.w);
    if (k < n) trig[L * n + k] = make_double2(v.x, v.y);
    const bool cot = fabs(v.y) > fabs(v.x);
    T.rot[k / n * N + k % n] = cot ? -v.x / v.y : v.y / v.x;
    if (cot) atomicOr(T.flip + k / n, 1u << (k % n));
  }
  if constexpr (N > n)
    for (int k = tid; k < L * (N - n); k += threads) T.rot[k / (N - n) * N + n + k % (N - n)] = 0.0;
  sync_cta<G>();
  for (int l = tid; l < L; l += threads) {  // K_l = prod 1 / sqrt(1 + k^2)
    double s[4] = {1.0, 1.0, 1.0, 1.0};
#pragma unroll
    for (int w = 0; w < n; ++w) {
      const double k = T.rot[l * N + w];
      s[w & 3] *= fma(k, k, 1.0);
    }
    T.scale[l] = 1.0 / sqrt((s[0] * s[1]) * (s[2] * s[3]));
  }
  for (int e = tid; e < (L + 1) * nt * 16; e += threads) {
    const int l = e / (nt * 16), t = e / 16 % nt, v = e & 15;
    const int first = t == nt - 1 ? N - R : 4 * t, end = t == nt - 1 ? N : (4 * t + 4 < N - R ? 4 * t + 4 : N - R);
    double2 z = make_double2(1.0, 0.0);
    const unsigned flip = l < L ? T.flip[l] : 0u;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int w = first + b;
      if (w >= end) break;
      const bool swapped = (flip >> w) & 1;  // a J on this wire; registers are numbered before its swap
      const bool one = (((v >> b) & 1) != 0) != (swapped && t == nt - 1);
      if (w >= n) {  // a padding wire stays |0>
        if (l == L && one) z = make_double2(0.0, 0.0);
        continue;
      }
      const double2 q = trig[(l == L ? 0 : l * n) + w];
      double2 f = make_double2(q.x, one ? q.y : -q.y);
      if (swapped && !one) f = make_double2(-f.x, -f.y);
      if (l == L) {
        const double a = one ? trig[L * n + w].y : trig[L * n + w].x;
        f.x *= a;
        f.y *= a;
      }
      z = cmul(z, f);
    }
    T.phase[e] = z;
  }
  sync_all<G>();  // the tables are ready, and every CTA is done with its (cos, sin) pairs

  // amplitudes of register 0, and where the exchanges send them
  const unsigned last = G::index(K - 1, rank, tid), x0 = G::index(0, rank, tid);
  const unsigned xb = G::index(K - 2, rank, tid);
  const unsigned ring = place_top(ring_map(last, n), m), unring = place_low(ring_unmap(x0, n), C);
  const unsigned down = place_top(last, m), up = place_low(xb, C);
  unsigned own[K];
#pragma unroll
  for (int k = 0; k < K; ++k) own[k] = G::own(k, G::index(k, rank, tid));
  auto ring_bit = [](int j) { return G::ring_bit(j); };
  auto unring_bit = [](int j) { return G::unring_bit(j); };
  auto down_bit = [](int j) { return G::down_bit(j); };
  auto up_bit = [](int j) { return G::up_bit(j); };
  // register bit j of layout k holds the index bit, or (layouts 0 and K-1) its
  // complement where the rank says so: the rotation's sign follows
  auto turned = [&](int k, int j) { return C > 0 && (k == 0 || k == K - 1) && ((rank >> j) & 1); };
  auto factor = [&](const double *rot, int k, int j) {
    const double v = rot[G::wire(k, j)];
    return turned(k, j) ? -v : v;
  };
  // what the J swaps of layout k's wires add to an address
  auto swaps = [&](unsigned flip, int k, auto &&bit) {
    unsigned x = 0;
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (G::wire(k, j) >= 0) x ^= (0u - ((flip >> G::wire(k, j)) & 1u)) & bit(j);
    return x;
  };
  auto phase_base = [&](const double2 *tab) {
    double2 z = tab[last & 15 & ((1u << (N - R)) - 1)];
#pragma unroll
    for (int t = 1; t < nt - 1; ++t) z = cmul(z, tab[16 * t + (((last & ((1u << (N - R)) - 1)) >> (4 * t)) & 15)]);
    return z;
  };
  const unsigned top_turn = C > 0 ? rank : 0u;

  double2 psi[NR], lam[NR];
  // a thread's amplitudes behind layout k of layer l (l >= 1)
  auto checkpoint = [&](int l, int k) { return ck + (static_cast<size_t>(l) * K + k) * (NR * threads) + tid; };
  auto save = [&](int l, int k) {
    double2 *p = checkpoint(l, k);
#pragma unroll
    for (int r = 0; r < NR; ++r) p[r * threads] = psi[r];
  };
  auto restore = [&](int l, int k) {
    const double2 *p = checkpoint(l, k);
#pragma unroll
    for (int r = 0; r < NR; ++r) psi[r] = p[r * threads];
  };
  const bool keep = A.grad_out != nullptr || A.lam != nullptr;
  if (!A.resume) {
    // ---- layer 0: the product state, in layout K-1
    {
      const double2 z = phase_base(T.prod);
#pragma unroll
      for (int r = 0; r < NR; ++r) psi[r] = cmul(z, T.prod[16 * (nt - 1) + (r ^ top_turn)]);
    }
    unsigned swap = 0;
#pragma unroll 1
    for (int l = 1; l < L; ++l) {
      push<G>(psi, smP, ring ^ swap, ring_bit);
      sync_all<G>();
      load_own<G>(psi, bufP, 0, own[0]);
      const unsigned flip = T.flip[l];
      const double *rot = T.rot + l * N;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k >= K - 2) arrive<G>();  // this thread has read its slots
#pragma unroll
        for (int j = 0; j < R; ++j)
          if (G::wire(k, j) >= 0) rotate<R>(psi, j, factor(rot, k, j));
        if (CK && keep) save(l, k);
        if (k == K - 1) break;
        if (k + 1 < K - 1) {
          store_own<G>(psi, bufP, k, own[k] ^ swaps(flip, k, [&](int j) { return G::own_bit(k, j); }));
          sync_cta<G>();
        } else {
          wait<G>();
          push<G>(psi, smP, up ^ swaps(flip, k, up_bit), up_bit);
          sync_all<G>();
        }
        load_own<G>(psi, bufP, k + 1, own[k + 1]);
      }
      const double2 *tab = T.phase + static_cast<size_t>(l) * nt * 16;
      double2 z = phase_base(tab);
      z.x *= T.scale[l];
      z.y *= T.scale[l];
#pragma unroll
      for (int r = 0; r < NR; ++r) psi[r] = cmul(psi[r], cmul(z, tab[16 * (nt - 1) + (r ^ top_turn)]));
      swap = swaps(flip, K - 1, ring_bit);
      wait<G>();
    }
    // ---- lambda = H psi and the energy, in layout 0.  With several CTAs the
    // state passes through layout K-1 once more, where the top wires'
    // neighbours are in registers; everything else is in the CTA's own slots.
    if constexpr (C > 0) {
      const unsigned low = place_low(ring_map(last, n), C);
      // (the swap of the last layer's J in this exchange's terms)
      unsigned s = 0;
      if (L > 1) s = swaps(T.flip[L - 1], K - 1, [](int j) { return G::ring_low_bit(j); });
      push<G>(psi, smP, low ^ s, [](int j) { return G::ring_low_bit(j); });
      sync_all<G>();
      load_own<G>(psi, bufP, K - 1, own[K - 1]);
      arrive<G>();
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        lam[r] = make_double2(0.0, 0.0);
#pragma unroll
        for (int j = 0; j < R; ++j) {
          lam[r].x += psi[r ^ (1 << j)].x;
          lam[r].y += psi[r ^ (1 << j)].y;
        }
      }
      wait<G>();
      push<G>(psi, smP, down, down_bit);
      push<G>(lam, smL, down, down_bit);
      sync_all<G>();
      load_own<G>(psi, bufP, 0, own[0]);
      load_own<G>(lam, bufL, 0, own[0]);
    } else {
      push<G>(psi, smP, ring ^ swap, ring_bit);
      sync_all<G>();
      load_own<G>(psi, bufP, 0, own[0]);
#pragma unroll
      for (int r = 0; r < NR; ++r) lam[r] = make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int w = 0; w < (C > 0 ? N - R : n); ++w) {
      if (w < R) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          lam[r].x += psi[r ^ (1 << w)].x;
          lam[r].y += psi[r ^ (1 << w)].y;
        }
      } else {
        for_registers<R>(own[0] ^ G::own(0, 1u << w), [&](int j) { return G::own_bit(0, j); }, [&](int r, unsigned p) {
          const double2 q = *reinterpret_cast<const double2 *>(bufP + p);
          lam[r].x += q.x;
          lam[r].y += q.y;
        });
      }
    }
    double energy = 0.0;
    constexpr unsigned mask = (1u << n) - 1;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const unsigned x = x0 ^ static_cast<unsigned>(r), p = x & mask;
      const unsigned next = ((p << 1) & mask) | (p >> (n - 1));
      const double d = static_cast<double>(2 * __popc(p ^ next) - n);
      // (a padding index has a zero amplitude and keeps a zero lambda)
      lam[r] = x > mask ? make_double2(0.0, 0.0)
                        : make_double2(fma(d, psi[r].x, -item.h * lam[r].x), fma(d, psi[r].y, -item.h * lam[r].y));
      energy = fma(psi[r].x, lam[r].x, energy);
      energy = fma(psi[r].y, lam[r].y, energy);
    }
    energy = warp_sum(energy);
    if (lane == 0) T.red[warp] = energy;
    if (A.lam) {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        if (!CK) A.psi[x0 ^ static_cast<unsigned>(r)] = psi[r];
        A.lam[x0 ^ static_cast<unsigned>(r)] = lam[r];
      }
    }
    sync_all<G>();  // every CTA's shares are there, and every slot is read
    if (rank == 0 && warp == 0 && A.energy_out) {
      double s = 0.0;
      const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(T.red));
      for (int k = lane; k < warps * G::ctas; k += 32) {
        const unsigned a = at + 8u * (k % warps);
        s += load_cluster(C > 0 ? cluster_address(a, k / warps) : a);
      }
      s = warp_sum(s);
      if (lane == 0) A.energy_out[item.index] = s;
    }
    sync_all<G>();  // the shares stay until they are read
  } else {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      if (!CK) psi[r] = A.psi[x0 ^ static_cast<unsigned>(r)];
      lam[r] = A.lam[x0 ^ static_cast<unsigned>(r)];
    }
  }
  if (A.grad_out == nullptr) return;

  // the record of layer l from its warps' sums, behind a barrier after them
  auto gather = [&](int l) {
    if constexpr (warps > 1) {
      if (warp == l % warps) {
        const double *red = T.red + (l & 1) * 32 * warps;
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < warps; ++k) sum += red[32 * k + lane];
        T.rec[l * kRec + lane] = sum;
      }
    }
  };

  // ---- backward (the slots are free at the start of every layer)
  auto undo_layer = [&](int l, auto mode) {
    constexpr bool uncompute = decltype(mode)::value;
    const unsigned flip = T.flip[l];
    const unsigned swap = swaps(flip, K - 1, [](int j) { return G::own_bit(K - 1, j); });
    if (!CK) push<G>(psi, smP, unring, unring_bit);
    push<G>(lam, smL, unring, unring_bit);
    if constexpr (!uncompute) {
      restore(l, K - 1);
    } else if constexpr (CK) {
      {  // the product state; registers are numbered before J's swap
        const double2 z = phase_base(T.prod);
        const unsigned turn = top_turn ^ ((flip >> (N - R)) & (NR - 1));
#pragma unroll
        for (int r = 0; r < NR; ++r) psi[r] = cmul(z, T.prod[16 * (nt - 1) + (r ^ turn)]);
      }
    }
    sync_all<G>();
    if (l < L - 1) gather(l + 1);
    if (!CK) load_own<G>(psi, bufP, K - 1, own[K - 1] ^ swap);
    load_own<G>(lam, bufL, K - 1, own[K - 1] ^ swap);
    arrive<G>();
    // D^+ K on lambda, and on a psi that is un-computed; phi sums on the true
    // vectors, or on lambda behind D^+ K and the checkpoint before D
    double tot = 0.0, one[R];
#pragma unroll
    for (int j = 0; j < R; ++j) one[j] = 0.0;
    auto phi_sum = [&](int r) {
      const double q = fma(lam[r].x, psi[r].y, -lam[r].y * psi[r].x);
      tot += q;
#pragma unroll
      for (int j = 0; j < R; ++j)
        if ((r >> j) & 1) one[j] += q;
    };
    {
      const double2 *tab = T.phase + static_cast<size_t>(l) * nt * 16;
      double2 z = phase_base(tab);
      z.x *= T.scale[l];
      z.y *= T.scale[l];
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const double2 f = cmul(z, tab[16 * (nt - 1) + (r ^ top_turn)]);
        if constexpr (uncompute) {
          phi_sum(r);
          psi[r] = cmul_conj(psi[r], f);
        }
        lam[r] = cmul_conj(lam[r], f);
        if constexpr (!uncompute) phi_sum(r);
      }
    }
    double sums[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) sums[i] = 0.0;
    const double *rot = T.rot + l * N;
#pragma unroll
    for (int k = K - 1; k >= 0; --k) {
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (G::wire(k, j) >= 0) {
          const double s = theta_sum<R>(psi, lam, j);
          sums[G::wire(k, j) & 15] = turned(k, j) ? -s : s;
        }
      if (!uncompute && k > 0) restore(l, k - 1);  // in flight during lambda's exchange
      if (k > 0 || l > 0) {
#pragma unroll
        for (int j = 0; j < R; ++j)
          if (G::wire(k, j) >= 0) {
            const double f = -factor(rot, k, j);
            if (uncompute) rotate<R>(psi, j, f);
            rotate<R>(lam, j, f);
          }
      }
      if (k == 0) break;
      if (k == K - 1) {
        wait<G>();
        if (uncompute) push<G>(psi, smP, down, down_bit);
        push<G>(lam, smL, down, down_bit);
        sync_all<G>();
      } else {
        if (uncompute) store_own<G>(psi, bufP, k, own[k]);
        store_own<G>(lam, bufL, k, own[k]);
        sync_cta<G>();
      }
      const unsigned next = own[k - 1] ^ swaps(flip, k - 1, [&](int j) { return G::own_bit(k - 1, j); });
      if (uncompute) load_own<G>(psi, bufP, k - 1, next);
      load_own<G>(lam, bufL, k - 1, next);
    }
    arrive<G>();
#pragma unroll
    for (int j = 0; j < R; ++j) sums[kRecPhi + j] = one[j];
    sums[kRecTotal] = tot;
#pragma unroll
    for (int j = 0; j < 5; ++j) sums[kRecLane + j] = ((lane >> j) & 1) ? tot : 0.0;
    const double s = warp_sums32(sums, lane);
    if constexpr (warps == 1) T.rec[l * kRec + lane] = s;
    else T.red[(l & 1) * 32 * warps + 32 * warp + lane] = s;  // (read while the next layer fills the other half)
    if (lane == kRecTotal) T.tot[l * warps + warp] = s;
    wait<G>();  // every slot is read
  };
  if constexpr (CK) {
#pragma unroll 1
    for (int l = L - 1; l > 0; --l) undo_layer(l, Flag<false>{});
    undo_layer(0, Flag<true>{});
  } else {
#pragma unroll 1
    for (int l = L - 1; l >= 0; --l) undo_layer(l, Flag<true>{});
  }
  sync_all<G>();
  gather(0);
  sync_all<G>();  // every CTA's records are there
  const unsigned rec0 = static_cast<unsigned>(__cvta_generic_to_shared(T.rec));
  const unsigned tot0 = static_cast<unsigned>(__cvta_generic_to_shared(T.tot));
  for (int e = static_cast<int>(rank) * threads + static_cast<int>(tid); e < L * n * 2; e += G::ctas * threads) {
    const int l = e / (2 * n), w = e % (2 * n) / 2;
    double out = 0.0;
    if ((e & 1) == 0) {
      for (int k = 0; k < G::ctas; ++k) {
        const unsigned at = rec0 + 8u * (l * kRec + w);
        out += load_cluster(C > 0 ? cluster_address(at, k) : at);
      }
      double s[2] = {1.0, 1.0};  // prod (1 + k^2) over the wires still pending there
      const int pending = G::pending(w);
      for (int v = 0; v < pending && v < n; ++v) s[v & 1] *= fma(T.rot[l * N + v], T.rot[l * N + v], 1.0);
      if (!CK || l == 0) out *= s[0] * s[1];
    } else {
      // sum of z_w: the total less twice the sum over the amplitudes with bit w
      double tot = 0.0, b = 0.0;
      for (int k = 0; k < G::ctas; ++k) {
        const unsigned at = rec0 + 8u * (l * kRec);
        const unsigned base = C > 0 ? cluster_address(at, k) : at;
        const double t = load_cluster(base + 8u * kRecTotal);
        tot += t;
        if (w < C) {
          b += ((k >> w) & 1) ? t : 0.0;
        } else if (w >= N - R) {  // a register bit, complemented where the rank says so
          const double v = load_cluster(base + 8u * (kRecPhi + w - (N - R)));
          b += C > 0 && ((k >> (w - (N - R))) & 1) ? t - v : v;
        } else if (w < C + 5) {
          b += load_cluster(base + 8u * (kRecLane + w - C));
        } else {
          const unsigned tb = tot0 + 8u * (l * warps);
          const unsigned tk = C > 0 ? cluster_address(tb, k) : tb;
          for (int v = 0; v < warps; ++v)
            if ((v >> (w - C - 5)) & 1) b += load_cluster(tk + 8u * v);
        }
      }
      out = tot - 2.0 * b;
      if (w >= N - R && ((T.flip[l] >> w) & 1)) out = -out;  // its register bit is 1 where the wire is 0
    }
    A.grad_out[item.param_off + e] = out;
  }
  sync_all<G>();  // records stay until they are read
}

__device__ __forceinline__ void store_cluster_u32(unsigned addr, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <int n, int R, int C, bool CK>
__global__ void __launch_bounds__(Geo<n, R, C>::threads, 1) cluster_kernel(const __grid_constant__ ClusterArgs A) {
  using G = Geo<n, R, C>;
  extern __shared__ __align__(128) unsigned char smem[];
  const unsigned cluster = blockIdx.x >> C, rank = blockIdx.x & ((1u << C) - 1);
  double2 *ck = CK ? A.checkpoints + (static_cast<size_t>(cluster) * G::ctas + rank) * A.max_layers *
                                         (static_cast<size_t>(G::K) * G::NR * G::threads)
                   : nullptr;
  unsigned size;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(size));
  int *next = reinterpret_cast<int *>(smem + size - 16);
  const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(next));
  for (;;) {
    int i = static_cast<int>(cluster);
    if (A.counter != nullptr) {  // as many clusters as fit take the circuits in order
      if (rank == 0 && threadIdx.x == 0) {
        i = atomicAdd(A.counter, 1);
        for (int k = 0; k < G::ctas; ++k) store_cluster_u32(C > 0 ? cluster_address(at, k) : at, i);
      }
      sync_all<G>();
      i = *reinterpret_cast<volatile int *>(next);
      if (i >= A.count) return;
    }
    run_circuit<G, CK>(A, A.items ? A.items[i] : A.item, smem, ck);
    if (A.counter == nullptr) return;
    sync_all<G>();  // (an energy-only circuit's last reads; everyone has read `next`)
  }
}

template <int n, int R, int C, bool CK>
struct Shape {
  using G = Geo<n, R, C>;
  static bool is(int qubits, ClusterShape h) {
    return qubits == n && h.register_bits == R && h.log_ctas == C && h.checkpoints == CK;
  }
  static size_t checkpoint_values(int max_layers) {
    return CK ? (static_cast<size_t>(max_layers) * G::K) << G::N : 0;
  }
  static size_t smem(int max_layers) {
    const size_t bufs = size_t{32} << G::m;
    size_t most = 0;  // (a circuit of fewer layers may be the one whose pairs need room of their own)
    for (int L = 1; L <= max_layers; ++L) {
      const size_t b = bufs + table_bytes<G>(L) + (trig_bytes(n, L) <= bufs ? 0 : trig_bytes(n, L));
      if (b > most) most = b;
    }
    return most + 16;  // (the next circuit's number)
  }
  static void fill(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at, int max_layers, int clusters) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters) << C);
    cfg.blockDim = dim3(static_cast<unsigned>(G::threads));
    cfg.dynamicSmemBytes = smem(max_layers);
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1u << C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
  }
  // both attributes belong to the device: set once on each
  static cudaError_t configure() {
    static std::atomic<unsigned long long> smem_done{0}, size_done{0};
    cudaError_t e = set_smem_limit_once(cluster_kernel<n, R, C, CK>, kMostSmem, smem_done);
    if (e != cudaSuccess || C < 4) return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? (1ull << dev) : 0ull;
    if (bit != 0 && (size_done.load(std::memory_order_acquire) & bit) != 0) return cudaSuccess;
    e = cudaFuncSetAttribute(cluster_kernel<n, R, C, CK>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess && bit != 0) size_done.fetch_or(bit, std::memory_order_acq_rel);
    return e;
  }
  static cudaError_t launch(const ClusterArgs &A, cudaStream_t s) {
    const cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    fill(cfg, at, A.max_layers, A.counter ? A.clusters : A.count);
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, cluster_kernel<n, R, C, CK>, A);
  }
  static cudaError_t capacity(int max_layers, int *clusters) {
    if (smem(max_layers) > kMostSmem) return cudaSuccess;
    const cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    fill(cfg, at, max_layers, 1);
    return cudaOccupancyMaxActiveClusters(clusters, cluster_kernel<n, R, C, CK>, &cfg);
  }
};

// f(shape) for the built shape of n qubits; false where there is none
template <typename F>
bool with_shape(int n, ClusterShape h, F &&f) {
  bool found = false;
  auto one = [&](auto shape) {
    if (!found && decltype(shape)::is(n, h)) {
      found = true;
      f(shape);
    }
  };
  one(Shape<2, 2, 0, false>{});
  one(Shape<3, 2, 0, false>{});
  one(Shape<4, 2, 0, false>{});
  one(Shape<5, 2, 0, false>{});
  one(Shape<6, 2, 0, false>{});
  one(Shape<7, 2, 0, false>{});
  one(Shape<8, 2, 0, false>{});
  one(Shape<9, 2, 0, false>{});
  one(Shape<9, 3, 0, false>{});
  one(Shape<10, 3, 0, false>{});
  one(Shape<10, 4, 0, false>{});
  one(Shape<11, 3, 0, false>{});
  one(Shape<11, 4, 0, false>{});
  one(Shape<12, 3, 3, false>{});
  one(Shape<12, 4, 0, false>{});
  one(Shape<13, 3, 3, false>{});
  one(Shape<13, 4, 1, false>{});
  one(Shape<13, 4, 1, true>{});
  one(Shape<14, 4, 4, false>{});
  one(Shape<14, 4, 2, false>{});
  one(Shape<14, 4, 2, true>{});
  one(Shape<15, 4, 4, true>{});
  one(Shape<15, 4, 3, false>{});
  one(Shape<15, 4, 3, true>{});
  one(Shape<16, 4, 4, false>{});
  one(Shape<16, 4, 4, true>{});
  return found;
}

}  // namespace

bool cluster_shape_built(int n, ClusterShape h) {
  return with_shape(n, h, [](auto) {});
}

cudaError_t launch_cluster(const ClusterArgs &A, cudaStream_t s) {
  if (A.count < 1) return cudaSuccess;
  cudaError_t e = cudaErrorInvalidValue;
  with_shape(A.n, A.shape, [&](auto shape) { e = decltype(shape)::launch(A, s); });
  return e;
}

cudaError_t cluster_capacity(int n, ClusterShape h, int max_layers, int *clusters) {
  *clusters = 0;
  cudaError_t e = cudaSuccess;
  with_shape(n, h, [&](auto shape) { e = decltype(shape)::capacity(max_layers, clusters); });
  return e;
}

size_t cluster_checkpoint_values(int n, ClusterShape h, int max_layers) {
  size_t v = 0;
  with_shape(n, h, [&](auto shape) { v = decltype(shape)::checkpoint_values(max_layers); });
  return v;
}

}  // namespace rsv
