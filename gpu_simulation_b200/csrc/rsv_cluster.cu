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
// and SM; n = 14 327 -> 120 us, n = 15 331 -> 163; from there on the tiled
// kernel is the faster one).  Every shape is its own
// instantiation: with the layouts' arithmetic at run time n = 8 took 58 us and
// n = 12 118, most of it integer and address latency.
#include <cuda_runtime.h>

#include <atomic>

#include "rsv_resident.cuh"

namespace rsv {
namespace {

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
  const Tables T = build_tables<G>(A.params ? A.params + item.param_off : nullptr, A.coef,
                                   rank == 0 ? A.coef_out : nullptr, L, smem, size_t{32} << m);
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


template <int n, int R, int C, bool CK>
__global__ void __launch_bounds__(Geo<n, R, C>::threads, 1) cluster_kernel(const __grid_constant__ ClusterArgs A) {
  using G = Geo<n, R, C>;
  extern __shared__ __align__(128) unsigned char smem[];
  const unsigned cluster = blockIdx.x >> C, rank = blockIdx.x & ((1u << C) - 1);
  double2 *ck = CK ? A.memory + (static_cast<size_t>(cluster) * G::ctas + rank) * A.max_layers *
                                    (static_cast<size_t>(G::K) * G::NR * G::threads)
                   : nullptr;
  run_circuit<G, CK>(A, A.items ? A.items[cluster] : A.item, smem, ck);
}

template <int n, int R, int C, bool CK>
struct Shape {
  using G = Geo<n, R, C>;
  static bool is(int qubits, ClusterShape h) {
    return qubits == n && h.register_bits == R && h.log_ctas == C && h.checkpoints == CK;
  }
  static size_t memory_values(int max_layers) {
    return CK ? (static_cast<size_t>(max_layers) * G::K) << G::N : 0;
  }
  static size_t smem(int max_layers) {
    const size_t bufs = size_t{32} << G::m;
    size_t most = 0;  // (a circuit of fewer layers may be the one whose pairs need room of their own)
    for (int L = 1; L <= max_layers; ++L) {
      const size_t b = bufs + table_bytes<G>(L) + (trig_bytes(n, L) <= bufs ? 0 : trig_bytes(n, L));
      if (b > most) most = b;
    }
    return most;
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
    const cudaError_t e = set_smem_limit_once(cluster_kernel<n, R, C, CK>, kMostSmem, smem_done);
    if (e != cudaSuccess || C < 4) return e;
    return allow_any_cluster_once(cluster_kernel<n, R, C, CK>, size_done);
  }
  static cudaError_t launch(const ClusterArgs &A, cudaStream_t s) {
    const cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    fill(cfg, at, A.max_layers, A.count);
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
  one(Shape<14, 4, 4, false>{});
  one(Shape<15, 4, 4, true>{});
  return found;
}

}  // namespace

cudaError_t launch_cluster(const ClusterArgs &A, cudaStream_t s) {
  if (A.count < 1) return cudaSuccess;
  if (A.n > kClusterMaxQubits) return launch_grid(A, s);
  if (A.shape.tiled) return launch_tiles(A, s);
  cudaError_t e = cudaErrorInvalidValue;
  with_shape(A.n, A.shape, [&](auto shape) { e = decltype(shape)::launch(A, s); });
  return e;
}

cudaError_t cluster_capacity(int n, ClusterShape h, int max_layers, int *clusters) {
  *clusters = 0;
  if (n > kClusterMaxQubits) return grid_capacity(n, max_layers, clusters);
  if (h.tiled) return tile_capacity(n, h, max_layers, clusters);
  cudaError_t e = cudaSuccess;
  with_shape(n, h, [&](auto shape) { e = decltype(shape)::capacity(max_layers, clusters); });
  return e;
}

size_t cluster_memory_values(int n, ClusterShape h, int max_layers) {
  if (n > kClusterMaxQubits) return grid_memory_values(n, max_layers);
  if (h.tiled) return size_t{4} << n;
  size_t v = 0;
  with_shape(n, h, [&](auto shape) { v = decltype(shape)::memory_values(max_layers); });
  return v;
}

}  // namespace rsv
