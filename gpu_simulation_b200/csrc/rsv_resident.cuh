// Building blocks of the kernels that keep psi and lambda in registers
// (rsv_cluster.cu, rsv_tiles.cu): index arithmetic, layouts, tangent-form gates,
// per-circuit tables.
#pragma once

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

RSV_HD unsigned ring_map(unsigned x, int n) {  // P (rsv_device.cuh, at most 32 bits)
  const unsigned mask = (1u << n) - 1;
  unsigned p = x & mask;
  p ^= p << 1;
  p ^= p << 2;
  p ^= p << 4;
  p ^= p << 8;
  if (n > 16) p ^= p << 16;
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

__device__ __forceinline__ void store_cluster_u32(unsigned addr, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned shared_address(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// Clusters of 16 CTAs: an attribute of the kernel on a device, set once on each.
template <typename K>
cudaError_t allow_any_cluster_once(K *kernel, std::atomic<unsigned long long> &done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? (1ull << dev) : 0ull;
  if (bit != 0 && (done.load(std::memory_order_acquire) & bit) != 0) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess && bit != 0) done.fetch_or(bit, std::memory_order_acq_rel);
  return e;
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

// The tables of a circuit of L layers behind `bufs` (buf_bytes of exchange
// buffers, which hold the (cos, sin) pairs meanwhile): tangent forms, then phases
// and the first layer's product state.  From the angles, or from `coef`.
template <typename G>
__device__ __forceinline__ Tables build_tables(const double *params, const double4 *coef, double4 *coef_out, int L,
                                               unsigned char *bufs, size_t buf_bytes) {
  constexpr int n = G::n, N = G::N, R = G::R, nt = G::tables, threads = G::threads, warps = G::warps;
  const unsigned tid = threadIdx.x;
  Tables T;
  T.phase = reinterpret_cast<double2 *>(bufs + buf_bytes);
  T.prod = T.phase + static_cast<size_t>(L) * nt * 16;
  T.rot = reinterpret_cast<double *>(T.prod + nt * 16);
  T.rec = T.rot + L * N;
  T.tot = T.rec + L * kRec;
  T.red = T.tot + L * warps;
  T.scale = T.red + 64 * warps + 4;
  T.flip = reinterpret_cast<unsigned *>(T.rot + doubles_of<G>(L));
  // (cos, sin) of the half angles: phi of every wire, then theta of layer 0
  double2 *trig = trig_bytes(n, L) <= buf_bytes ? reinterpret_cast<double2 *>(bufs)
                                                : reinterpret_cast<double2 *>(T.flip + ((L + 3) & ~3));
  for (int l = tid; l < L; l += threads) T.flip[l] = 0;
  sync_cta<G>();
  for (int k = tid; k < L * n; k += threads) {
    double4 v;
    if (params) {
      sincos(params[2 * k] * 0.5, &v.y, &v.x);
      sincos(params[2 * k + 1] * 0.5, &v.w, &v.z);
    } else {
      v = coef[k];
    }
    if (coef_out) coef_out[k] = v;
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
  return T;
}

// A thread's amplitudes of the next tile on their way into its own 16 slots of a
// buffer ([register][thread]); only that thread reads them.
__device__ __forceinline__ void fetch(unsigned char *buf, int r, const double2 *from) {
  const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(buf)) + ((r << 8) + threadIdx.x) * 16;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
__device__ __forceinline__ void fetched() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ double2 take(const unsigned char *buf, int r) {
  return reinterpret_cast<const double2 *>(buf)[(r << 8) + threadIdx.x];
}

template <bool V>
struct Flag {
  static constexpr bool value = V;
};

}  // namespace
}  // namespace rsv
