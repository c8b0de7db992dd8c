// Correlators of one sector state: the one-body density matrix
// rho[i][j] = <psi| a_i^dagger a_j |psi> (off_diagonal_long_range_order,
// observables/off_diagonal_long_range_order.py:43-140) and the orbit-summed
// density pairs behind the static structure factor
// (_build_density_correlation_matrix, observables/static_structure_factor.py:54-149).
//
// Both reduce into an N x N matrix whose entries are owned by threads of a
// block and accumulated in a fixed order (no atomics); one wave of blocks
// walks its chunks with a grid stride, writes one partial matrix per block,
// and a final pass adds the block partials in a fixed order -- the same sums
// on every run of a device.
#include "rsed_internal.cuh"

namespace {

constexpr int kCT = 256;

int one_wave(const void* fn, size_t smem) {
  int dev = 0, n_sm = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kCT, smem) != cudaSuccess) return -1;
  return n_sm * (per_sm > 0 ? per_sm : 1);
}

// ---- one-body density matrix ------------------------------------------------
//
// A basis state m (table entry rep, g, alpha; coefficient c of its orbit,
// stabilizer S) carries the ket amplitude
//   ket(m) = c / sqrt(|G| |S|) * sum over g with g(rep) = m of conj(chi(g)) phase_g(rep)
// and, when rep is in the sector, the bra coefficient of the reference
//   bra(m) = c * sqrt(|S| / |G|) * conj(alpha conj(chi(g))).
// For i != j, rho[i][j] = sum over m with j occupied and i empty of
// conj(bra(m - j + i)) * ket(m) * (Jordan-Wigner sign), and rho[j][j] gains
// |c|^2 |S| / |G| from every m with j occupied.  Every hop goes through the
// state n = m - j with one particle less, and the sign is s_i(n) s_j(n) with
// s_i(n) = (-1)^(particles of n below i), so with
//   B(n, i) = s_i(n) bra(n + i),  K(n, j) = s_j(n) ket(n + j)   (0 if occupied)
// the matrix is the contraction rho[i][j] = sum_n conj(B(n, i)) K(n, j) over
// the C(N, k-1) states n: N - k + 1 table lookups per n instead of one per hop
// (25 instead of 200 for 8 of 32 sites).  A tile of TN states n is looked up
// with lane = site, four lookups in flight per lane, into shared memory; then
// the 256 threads add the tile's outer products, each owning RT x RT entries.
// Two-species bases run the particle taken from species A and from species B
// as two sets of states n; hops between the species stay zero.
//
// With scratch for it (32 B a state) K and B of every state are written once
// (k_obdm_states) and a lookup is one 32-B read (DENSE); otherwise each lookup
// evaluates its state from the table, the representative's mask, coefficient,
// stabilizer and membership.  The diagonal comes from the orbits alone
// (k_obdm_diag).
// 32 sites, 8 bosons, 10.5 million states: 120.6 ms with one rank, table and
// coefficient chain per hop and thread; 6.5 ms evaluating each lookup (a state
// k times; 24 % occupancy, latency of the dependent loads); 2.62 ms plus 0.25 for
// the states with the states written first.
template <int NP>
struct ObdmTile {
  static constexpr int TN = NP == 32 ? 32 : 16;       // states n of one tile
  static constexpr int NW = TN / (kCT / 32);          // of which one warp looks up NW
  static constexpr int U = NW * (NP / 32);            // lookups per lane
  static constexpr int RT = NP / 16;                  // outputs per thread and dimension
};

// Launches that need more than 48 KB allow the kernel what the largest group
// takes, not what they take themselves: host threads share the attribute.
struct ObdmLayout {
  size_t binom, eta, chi, perm, tile, total;
};

ObdmLayout obdm_layout(int n_site, int n_filled, int n_group) {
  ObdmLayout l{};
  size_t off = 0;
  l.tile = off;  // K then B: TN * NP = 1024 entries each
  off += 2 * sizeof(double2) * 1024;
  l.eta = off;
  off += sizeof(double2) * (size_t)n_group * n_site;
  l.chi = off;
  off += sizeof(double2) * (size_t)n_group;
  l.binom = off;
  off += sizeof(int64_t) * (size_t)(n_site + 1) * (n_filled + 1);
  l.perm = off;
  off += align_up((size_t)n_group * n_site, 16);
  l.total = off;
  return l;
}

// Rank of n + site i for one species: the particles of n above i move up one
// place in the colex sum.
__device__ __forceinline__ int64_t rank_with(uint64_t n, int i, const int64_t* __restrict__ binom, int kp1) {
  int64_t r = binom[i * kp1 + __popcll(n & ((1ull << i) - 1ull)) + 1];
  int l = 1;
  while (n) {
    const int b = __ffsll((long long)n) - 1;
    r += binom[b * kp1 + l + (b > i ? 1 : 0)];
    ++l;
    n &= n - 1;
  }
  return r;
}

struct KetBra {
  double2 ket, bra;
};

// Ket amplitude and bra coefficient of the state m with table entry e.
__device__ __forceinline__ KetBra ket_bra(const int4 e, uint64_t s, uint64_t m, double2 c, double2 ph, uint64_t stab,
                                          bool member, const rsed_group_t& grp, const uint8_t* perm,
                                          const double2* eta, const double2* chi) {
  KetBra o;
  o.ket = o.bra = make_double2(0.0, 0.0);
  if (c.x == 0.0 && c.y == 0.0) return o;
  const double S = (double)__popcll(stab);
  const double norm = 1.0 / sqrt((double)grp.n_group * S);
  o.ket = rsed_state_amplitude(s, m, e.y, ph, stab, grp, perm, eta, chi, make_double2(c.x * norm, c.y * norm));
  if (member) {
    const double2 ch = chi[e.y];
    const double2 pc = cmul(make_double2((double)__int_as_float(e.z), (double)__int_as_float(e.w)),
                            make_double2(ch.x, -ch.y));
    const double sr = S * norm;  // sqrt(S / |G|)
    o.bra = cmul(c, make_double2(sr * pc.x, -sr * pc.y));
  }
  return o;
}

__device__ __forceinline__ bool stage_phases(const rsed_group_t& grp, const double2* chi_g, double2* eta, uint8_t* perm,
                                             double2* chi) {
  bool twisted = false;
  for (int i = threadIdx.x; i < grp.n_group * grp.n_site; i += kCT) {
    const double2 v = reinterpret_cast<const double2*>(grp.eta)[i];
    twisted |= v.x != 1.0 || v.y != 0.0;
    eta[i] = v;
    perm[i] = grp.perm[i];
  }
  for (int i = threadIdx.x; i < grp.n_group; i += kCT) chi[i] = chi_g[i];
  return __syncthreads_or(twisted) == 0;  // all site phases exactly 1
}

// K and B of every state, in rank order.
__global__ void __launch_bounds__(kCT) k_obdm_states(rsed_group_t grp, const int4* __restrict__ table,
                                                     const uint64_t* __restrict__ repr_masks,
                                                     const uint64_t* __restrict__ stab_mask,
                                                     const uint64_t* __restrict__ member, int sector,
                                                     const double2* __restrict__ chi_g, const double2* __restrict__ x,
                                                     ObdmLayout lay, KetBra* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* eta = reinterpret_cast<double2*>(smem + lay.eta);
  double2* chi = reinterpret_cast<double2*>(smem + lay.chi);
  uint8_t* perm = smem + lay.perm;
  const bool unit = stage_phases(grp, chi_g, eta, perm, chi);
  const int N = grp.n_site;
  for (int64_t r = (int64_t)blockIdx.x * kCT + threadIdx.x; r < grp.n_states; r += (int64_t)gridDim.x * kCT) {
    const int4 e = __ldg(table + r);
    KetBra o;
    o.ket = o.bra = make_double2(0.0, 0.0);
    if (e.x >= 0) {
      const double2 c = __ldg(x + e.x);
      const uint64_t s[1] = {__ldg(repr_masks + e.x)};
      const uint64_t stab = __ldg(stab_mask + e.x);
      const bool mem = (__ldg(member + e.x) >> sector) & 1ull;
      const int g[1] = {e.y};
      double2 ph[1];
      rsed_phases<1>(s, g, N, grp.n_filled, perm, eta, grp.fermionic, unit, ph);
      const uint64_t m = __popcll(stab) > 1 ? rsed_permute(s[0], perm + e.y * N) : 0;
      o = ket_bra(e, s[0], m, c, ph[0], stab, mem, grp, perm, eta, chi);
    }
    out[r] = o;
  }
}

// Sum over the orbits of |c|^2 per occupied site of the representative, lane =
// site (and site + 32); one partial per block.
__global__ void __launch_bounds__(kCT) k_obdm_diag(int64_t n_orbits, const uint64_t* __restrict__ repr_masks,
                                                   const double2* __restrict__ x, double* __restrict__ part) {
  __shared__ double sums[kCT / 32][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double lo = 0.0, hi = 0.0;
  for (int64_t o0 = ((int64_t)blockIdx.x * (kCT / 32) + warp) * 32; o0 < n_orbits;
       o0 += (int64_t)gridDim.x * kCT) {
    const int64_t o = o0 + lane;
    uint64_t m = 0;
    double w = 0.0;
    if (o < n_orbits) {
      const double2 c = __ldg(x + o);
      m = __ldg(repr_masks + o);
      w = c.x * c.x + c.y * c.y;
    }
    for (int q = 0; q < 32; ++q) {
      const uint64_t mq = __shfl_sync(0xffffffffu, m, q);
      const double wq = __shfl_sync(0xffffffffu, w, q);
      if ((mq >> lane) & 1ull) lo += wq;
      if ((mq >> (lane + 32)) & 1ull) hi += wq;
    }
  }
  sums[warp][lane] = lo;
  sums[warp][lane + 32] = hi;
  __syncthreads();
  if (threadIdx.x < 64) {
    double s = 0.0;
    for (int w = 0; w < kCT / 32; ++w) s += sums[w][threadIdx.x];
    part[blockIdx.x * 64 + threadIdx.x] = s;
  }
}

// rho[j][j] = (1/|G|) sum_g D[a] with g(a) = j, D the block partials' sum; one
// block, 16 lanes per site.
__global__ void __launch_bounds__(1024) k_obdm_rotate(rsed_group_t grp, const double* __restrict__ part, int n_blocks,
                                                      double2* __restrict__ rho) {
  __shared__ double D[64];
  const int t = threadIdx.x / 16, h = threadIdx.x % 16, N = grp.n_site;
  double s = 0.0;
  for (int b = h; b < n_blocks; b += 16) s += part[b * 64 + t];
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (h == 0) D[t] = s;
  __syncthreads();
  double d = 0.0;
  if (t < N)
    for (int e = h; e < grp.n_group * N; e += 16)
      if (grp.perm[e] == t) d += D[e % N];
  for (int o = 8; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
  if (t < N && h == 0) rho[t * N + t] = make_double2(d / (double)grp.n_group, 0.0);
}

template <int NP, bool DENSE>
__global__ void __launch_bounds__(kCT, DENSE && NP == 32 ? 3 : 2) k_obdm_part(rsed_group_t grp, const int4* __restrict__ table,
                                                      const uint64_t* __restrict__ repr_masks,
                                                      const uint64_t* __restrict__ stab_mask,
                                                      const uint64_t* __restrict__ member, int sector,
                                                      const double2* __restrict__ chi_g,
                                                      const double2* __restrict__ x, int per_warp,
                                                      int64_t n_a, int64_t n_b, ObdmLayout lay,
                                                      const KetBra* __restrict__ states,
                                                      double2* __restrict__ part) {
  using T = ObdmTile<NP>;
  extern __shared__ __align__(16) unsigned char smem[];
  double2* Kt = reinterpret_cast<double2*>(smem + lay.tile);  // [TN][NP]
  double2* Bt = Kt + T::TN * NP;
  double2* eta = reinterpret_cast<double2*>(smem + lay.eta);
  double2* chi = reinterpret_cast<double2*>(smem + lay.chi);
  int64_t* binom = reinterpret_cast<int64_t*>(smem + lay.binom);
  uint8_t* perm = smem + lay.perm;
  const int N = grp.n_site, kp1 = grp.n_filled + 1;
  for (int i = threadIdx.x; i < (N + 1) * kp1; i += kCT) binom[i] = grp.binom[i];
  bool unit = false;
  if constexpr (DENSE)
    __syncthreads();
  else
    unit = stage_phases(grp, chi_g, eta, perm, chi);
  const uint64_t first = (1ull << grp.n_filled) - 1ull;  // stands in for missing states (N <= 63)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const bool fermion = grp.fermionic != 0;
  const uint64_t sb = grp.species_b;
  const int64_t cb = sb ? binom[__popcll(sb) * kp1 + grp.n_filled_b] : 1;
  const uint64_t all = (1ull << N) - 1ull;
  double2 acc[T::RT][T::RT];
#pragma unroll
  for (int a = 0; a < T::RT; ++a)
#pragma unroll
    for (int b = 0; b < T::RT; ++b) acc[a][b] = make_double2(0.0, 0.0);
  const int64_t per_chunk = (int64_t)(kCT / 32) * per_warp;
  const int64_t chunks_a = (n_a + per_chunk - 1) / per_chunk, chunks_b = (n_b + per_chunk - 1) / per_chunk;
  for (int64_t ch = blockIdx.x; ch < chunks_a + chunks_b; ch += gridDim.x) {
    const bool in_b = ch >= chunks_a;  // the particle is taken from species B
    rsed_group_t red = grp;            // the basis of the states n
    red.n_filled -= 1;
    if (in_b) red.n_filled_b -= 1;
    const uint64_t allowed = sb ? (in_b ? sb : all & ~sb) : all;
    const int64_t n_red = in_b ? n_b : n_a;
    const int64_t r0 = (in_b ? ch - chunks_a : ch) * per_chunk + (int64_t)warp * per_warp;
    RankWalker walk;
    if (r0 < n_red) walk.init(r0, red, binom, kp1);
    for (int t = 0; t < per_warp; t += T::NW) {
      uint64_t n[T::NW];
#pragma unroll
      for (int w = 0; w < T::NW; ++w) {
        const int64_t r = r0 + t + w;
        n[w] = r < n_red ? walk.m : ~0ull;  // all sites taken: no lookups
        if (r + 1 < n_red) walk.next();
      }
      int64_t idx[T::U];
      bool ok[T::U];
#pragma unroll
      for (int u = 0; u < T::U; ++u) {
        const int i = lane + 32 * (u % (NP / 32));
        const uint64_t nn = n[u / (NP / 32)];
        ok[u] = i < N && ((allowed >> i) & 1ull) && !((nn >> i) & 1ull);
        idx[u] = 0;
        if (ok[u]) idx[u] = sb ? rsed_rank2(nn | (1ull << i), binom, kp1, sb, cb) : rank_with(nn, i, binom, kp1);
        ok[u] = ok[u] && idx[u] >= 0 && idx[u] < grp.n_states;
      }
      KetBra kb[T::U];
      if constexpr (DENSE) {
#pragma unroll
        for (int u = 0; u < T::U; ++u) {
          kb[u].ket = kb[u].bra = make_double2(0.0, 0.0);
          if (ok[u])
            asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                : "=d"(kb[u].ket.x), "=d"(kb[u].ket.y), "=d"(kb[u].bra.x), "=d"(kb[u].bra.y)
                : "l"(states + idx[u]));
        }
      } else {
        int4 e[T::U];
#pragma unroll
        for (int u = 0; u < T::U; ++u) e[u] = ok[u] ? __ldg(table + idx[u]) : make_int4(-1, 0, 0, 0);
        double2 c[T::U], ph[T::U];
        uint64_t s[T::U], st[T::U], mem[T::U];
        int ge[T::U];
#pragma unroll
        for (int u = 0; u < T::U; ++u) {
          c[u] = make_double2(0.0, 0.0);
          s[u] = first;
          st[u] = mem[u] = 0;
          ge[u] = e[u].y;
          if (e[u].x >= 0) {
            c[u] = __ldg(x + e[u].x);
            s[u] = __ldg(repr_masks + e[u].x);
            st[u] = __ldg(stab_mask + e[u].x);
            mem[u] = __ldg(member + e[u].x);
          }
        }
        rsed_phases<T::U>(s, ge, N, grp.n_filled, perm, eta, fermion, unit, ph);
#pragma unroll
        for (int u = 0; u < T::U; ++u)
          kb[u] = ket_bra(e[u], s[u], n[u / (NP / 32)] | (1ull << ((lane + 32 * (u % (NP / 32))) & 63)), c[u], ph[u], st[u],
                          (mem[u] >> sector) & 1ull, grp, perm, eta, chi);
      }
#pragma unroll
      for (int u = 0; u < T::U; ++u) {
        const int i = lane + 32 * (u % (NP / 32)), q = warp * T::NW + u / (NP / 32);
        const bool flip = fermion && (__popcll(n[u / (NP / 32)] & ((1ull << i) - 1ull)) & 1);
        Kt[q * NP + i] = flip ? make_double2(-kb[u].ket.x, -kb[u].ket.y) : kb[u].ket;
        Bt[q * NP + i] = flip ? make_double2(-kb[u].bra.x, -kb[u].bra.y) : kb[u].bra;
      }
      __syncthreads();
#pragma unroll 4
      for (int q = 0; q < T::TN; ++q) {
        double2 bv[T::RT], kv[T::RT];
#pragma unroll
        for (int a = 0; a < T::RT; ++a) bv[a] = Bt[q * NP + ty + 16 * a];
#pragma unroll
        for (int b = 0; b < T::RT; ++b) kv[b] = Kt[q * NP + tx + 16 * b];
#pragma unroll
        for (int a = 0; a < T::RT; ++a)
#pragma unroll
          for (int b = 0; b < T::RT; ++b) {
            acc[a][b].x = fma(bv[a].x, kv[b].x, fma(bv[a].y, kv[b].y, acc[a][b].x));
            acc[a][b].y = fma(bv[a].x, kv[b].y, fma(-bv[a].y, kv[b].x, acc[a][b].y));
          }
      }
      __syncthreads();
    }
  }
  double2* out = part + (int64_t)blockIdx.x * N * N;  // the diagonal is overwritten later
#pragma unroll
  for (int a = 0; a < T::RT; ++a)
#pragma unroll
    for (int b = 0; b < T::RT; ++b) {
      const int i = ty + 16 * a, j = tx + 16 * b;
      if (i < N && j < N) out[i * N + j] = acc[a][b];
    }
}

// ---- density pairs --------------------------------------------------------------
//
// D[a][b] = sum_o |x_o|^2 n_a(s_o) n_b(s_o) over the representatives s_o; the
// structure factor's C[i][j] = (1/|G|) sum_g D[a][b] at i = g(a), j = g(b)
// follows from it on the host.  A warp takes 32 orbits at a time and adds each
// to the 32 rows a of its half (blockIdx.y) that are occupied, lane = b (and
// b + 32), all sums in registers: two instructions per row, no atomics.
// 657,756 orbits of 8 bosons on 32 sites: 185 us with every thread testing its
// pairs against every orbit, 255 us with the rows in shared memory (a chain of
// read-modify-writes), 117 us in this form.
template <int NH>
__global__ void __launch_bounds__(NH == 1 ? 256 : 128, NH == 1 ? 2 : 3)
    k_pairs_part(int n_site, int64_t n_orbits, const uint64_t* __restrict__ repr_masks,
                 const double2* __restrict__ x, double* __restrict__ part) {
  constexpr int W = 32 * NH;
  extern __shared__ double dacc[];  // [warp][32][W]
  const int N = n_site, warps = blockDim.x >> 5, a0 = 32 * blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double acc[NH][32];
#pragma unroll
  for (int h = 0; h < NH; ++h)
#pragma unroll
    for (int a = 0; a < 32; ++a) acc[h][a] = 0.0;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t o0 = (int64_t)blockIdx.x * blockDim.x + warp * 32; o0 < n_orbits; o0 += step) {
    const int64_t o = o0 + lane;
    uint64_t m = 0;
    double w = 0.0;
    if (o < n_orbits) {
      const double2 c = __ldg(x + o);
      m = __ldg(repr_masks + o);
      w = c.x * c.x + c.y * c.y;
    }
    for (int q = 0; q < 32; ++q) {
      const uint64_t mq = __shfl_sync(0xffffffffu, m, q);
      const double wq = __shfl_sync(0xffffffffu, w, q);
      const uint32_t rows = (uint32_t)(mq >> a0);
      double wl[NH];
#pragma unroll
      for (int h = 0; h < NH; ++h) wl[h] = (mq >> (lane + 32 * h)) & 1ull ? wq : 0.0;
#pragma unroll
      for (int a = 0; a < 32; ++a)
        if (rows & (1u << a)) {
#pragma unroll
          for (int h = 0; h < NH; ++h) acc[h][a] += wl[h];
        }
    }
  }
  double* D = dacc + (size_t)warp * 32 * W + lane;
#pragma unroll
  for (int a = 0; a < 32; ++a)
#pragma unroll
    for (int h = 0; h < NH; ++h) D[a * W + 32 * h] = acc[h][a];
  __syncthreads();
  const int rows = min(32, N - a0);
  for (int p = threadIdx.x; p < rows * N; p += blockDim.x) {
    double s = 0.0;
    for (int v = 0; v < warps; ++v) s += dacc[((size_t)v * 32 + p / N) * W + p % N];
    part[((int64_t)blockIdx.x * N + a0) * N + p] = s;
  }
}

// out[p] = sum over the blocks' partials, one warp per entry: lane l adds
// blocks l, l + 32, ... in order, then a fixed butterfly combines the lanes.
// C = doubles per entry.  (One thread per entry walked every block alone:
// 99 us for 1024 complex entries of 1184 blocks.)
template <int C>
__global__ void k_sum_blocks(const double* __restrict__ part, int n_blocks, int nn, double* __restrict__ out) {
  const int p = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (p >= nn) return;  // whole warps leave together
  double s[C];
#pragma unroll
  for (int k = 0; k < C; ++k) s[k] = 0.0;
  for (int b = lane; b < n_blocks; b += 32)
#pragma unroll
    for (int k = 0; k < C; ++k) s[k] += part[((int64_t)b * nn + p) * C + k];
#pragma unroll
  for (int k = 0; k < C; ++k)
    for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < C; ++k) out[(int64_t)p * C + k] = s[k];
}

constexpr int kObdmBlocksPerSm = 4;  // partial matrices per SM at most

int sm_count() {
  int dev = 0, n_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  return n_sm;
}

int64_t choose(int n, int k) {
  if (k < 0 || k > n) return 0;
  __int128 c = 1;
  for (int i = 1; i <= k; ++i) c = c * (n - k + i) / i;
  return (int64_t)c;
}

template <int NP, bool DENSE>
int obdm_launch(const rsed_group_t& grp, const int4* table, const uint64_t* repr_masks, const uint64_t* stab_mask,
                const uint64_t* member, int sector, const double2* chi, const double2* x, int64_t n_a, int64_t n_b,
                const KetBra* states, double2* part, int* grid_out, cudaStream_t stream) {
  auto kern = k_obdm_part<NP, DENSE>;
  const ObdmLayout lay = obdm_layout(grp.n_site, grp.n_filled, DENSE ? 0 : grp.n_group);
  if (lay.total > 48 * 1024)
    RSED_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)obdm_layout(RSED_MAX_SITES, RSED_MAX_SITES, DENSE ? 0 : RSED_MAX_GROUP).total));
  const int n_sm = sm_count();
  const int wave = one_wave((const void*)kern, lay.total);
  RSED_REQUIRE(n_sm > 0 && wave > 0, RSED_ECUDA, "no occupancy for the one-body density kernel");
  int64_t grid = wave < n_sm * kObdmBlocksPerSm ? wave : n_sm * kObdmBlocksPerSm;
  // states n per warp: 32 amortise the unranking; fewer when the blocks of one
  // wave would not all have a chunk
  int per_warp = 32;
  while (per_warp > 4 && (n_a + n_b) / (8 * per_warp) < 2 * grid) per_warp /= 2;
  const int64_t pc = 8 * per_warp;
  const int64_t chunks = (n_a + pc - 1) / pc + (n_b + pc - 1) / pc;
  if (grid > chunks) grid = chunks;
  kern<<<(unsigned)grid, kCT, lay.total, stream>>>(grp, table, repr_masks, stab_mask, member, sector, chi, x, per_warp,
                                                   n_a, n_b, lay, states, part);
  RSED_CHECK_LAUNCH();
  *grid_out = (int)grid;
  return RSED_OK;
}

// Partial matrices, then the diagonal's partials (64 per SM).
size_t obdm_part_bytes(int n_site, int n_sm) {
  return align_up(sizeof(double2) * (size_t)n_sm * kObdmBlocksPerSm * n_site * n_site, 256);
}
size_t obdm_diag_bytes(int n_sm) { return align_up(sizeof(double) * 64 * (size_t)n_sm, 256); }

}  // namespace

extern "C" size_t rsed_obdm_scratch_bytes(int32_t n_site) {
  const int n_sm = sm_count();
  if (n_sm <= 0) return 0;
  return obdm_part_bytes(n_site, n_sm) + obdm_diag_bytes(n_sm);
}

extern "C" size_t rsed_obdm_states_bytes(int64_t n_states) {
  return n_states < 1 ? 0 : sizeof(KetBra) * (size_t)n_states;
}

extern "C" int rsed_one_body_density(const rsed_group_t* grp, const rsed_entry_t* table, int64_t n_orbits,
                                     const uint64_t* repr_masks, const uint64_t* stab_mask, const uint64_t* member,
                                     int32_t sector, const double* chi, const double* x_orbit, double* rho,
                                     void* scratch, size_t scratch_bytes, void* stream_) {
  int rc = check_group(grp);
  if (rc) return rc;
  RSED_REQUIRE(table && repr_masks && stab_mask && member && chi && x_orbit && rho && scratch && n_orbits >= 1,
               RSED_EINVAL, "bad one-body density arguments");
  RSED_REQUIRE(grp->eta != nullptr, RSED_EINVAL, "one-body density needs the group's eta phases");
  RSED_REQUIRE(sector >= 0 && sector < 64, RSED_EINVAL, "sector index %d outside [0, 64)", sector);
  RSED_REQUIRE(scratch_bytes >= rsed_obdm_scratch_bytes(grp->n_site), RSED_ESCRATCH,
               "one-body density scratch too small");
  cudaStream_t stream = as_stream(stream_);
  const int N = grp->n_site, nn = N * N;
  // states with one particle less: taken from species A (or the only one), from B
  int64_t n_a, n_b = 0;
  if (grp->species_b) {
    const int nb = __builtin_popcountll(grp->species_b), kb = grp->n_filled_b, ka = grp->n_filled - kb;
    n_a = choose(N - nb, ka - 1) * choose(nb, kb);
    n_b = choose(N - nb, ka) * choose(nb, kb - 1);
  } else {
    n_a = choose(N, grp->n_filled - 1);
  }
  if (n_a + n_b == 0) {  // no particles
    RSED_TRY_CUDA(cudaMemsetAsync(rho, 0, sizeof(double2) * (size_t)nn, stream));
    return RSED_OK;
  }
  const int n_sm = sm_count();
  RSED_REQUIRE(n_sm > 0, RSED_ECUDA, "no device");
  char* base = reinterpret_cast<char*>(scratch);
  double2* part = reinterpret_cast<double2*>(base);
  double* dpart = reinterpret_cast<double*>(base + obdm_part_bytes(N, n_sm));
  const int4* tb = reinterpret_cast<const int4*>(table);
  const double2* ch = reinterpret_cast<const double2*>(chi);
  const double2* xo = reinterpret_cast<const double2*>(x_orbit);
  // the caller's scratch decides: the states written once if they fit (32-B
  // aligned), else evaluated at every lookup
  KetBra* states = reinterpret_cast<KetBra*>(base + rsed_obdm_scratch_bytes(N));
  const bool dense = scratch_bytes >= rsed_obdm_scratch_bytes(N) + rsed_obdm_states_bytes(grp->n_states) &&
                     (reinterpret_cast<uintptr_t>(states) & 31) == 0;
  if (dense) {
    const ObdmLayout lay = obdm_layout(N, grp->n_filled, grp->n_group);
    if (lay.total > 48 * 1024)
      RSED_TRY_CUDA(cudaFuncSetAttribute(k_obdm_states, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)obdm_layout(RSED_MAX_SITES, RSED_MAX_SITES, RSED_MAX_GROUP).total));
    const int wave = one_wave((const void*)k_obdm_states, lay.total);
    RSED_REQUIRE(wave > 0, RSED_ECUDA, "no occupancy for the state kernel");
    const int64_t blocks = (grp->n_states + kCT - 1) / kCT;
    k_obdm_states<<<(unsigned)(blocks < wave ? blocks : wave), kCT, lay.total, stream>>>(
        *grp, tb, repr_masks, stab_mask, member, sector, ch, xo, lay, states);
    RSED_CHECK_LAUNCH();
  }
  int grid = 0;
  auto launch = N <= 32 ? (dense ? obdm_launch<32, true> : obdm_launch<32, false>)
                        : (dense ? obdm_launch<64, true> : obdm_launch<64, false>);
  rc = launch(*grp, tb, repr_masks, stab_mask, member, sector, ch, xo, n_a, n_b, states, part, &grid, stream);
  if (rc) return rc;
  k_sum_blocks<2><<<(nn + 3) / 4, 128, 0, stream>>>(reinterpret_cast<const double*>(part), grid, nn, rho);
  RSED_CHECK_LAUNCH();
  const int64_t dblocks = (n_orbits + kCT - 1) / kCT;
  const int dgrid = (int)(dblocks < n_sm ? dblocks : n_sm);
  k_obdm_diag<<<dgrid, kCT, 0, stream>>>(n_orbits, repr_masks, xo, dpart);
  RSED_CHECK_LAUNCH();
  k_obdm_rotate<<<1, 1024, 0, stream>>>(*grp, dpart, dgrid, reinterpret_cast<double2*>(rho));
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

extern "C" size_t rsed_density_pairs_scratch_bytes(int32_t n_site) {
  const int n_sm = sm_count();
  if (n_sm <= 0) return 0;
  return sizeof(double) * (size_t)(2 * n_sm) * n_site * n_site;
}

extern "C" int rsed_density_pairs(int32_t n_site, int64_t n_orbits, const uint64_t* repr_masks,
                                  const double* x_orbit, double* pairs, void* scratch, size_t scratch_bytes,
                                  void* stream_) {
  RSED_REQUIRE(n_site >= 1 && n_site <= RSED_MAX_SITES, RSED_ERANGE, "n_site = %d outside [1, %d]", n_site,
               RSED_MAX_SITES);
  RSED_REQUIRE(repr_masks && x_orbit && pairs && scratch && n_orbits >= 1, RSED_EINVAL,
               "bad density-pair arguments");
  RSED_REQUIRE(scratch_bytes >= rsed_density_pairs_scratch_bytes(n_site), RSED_ESCRATCH,
               "density-pair scratch too small");
  cudaStream_t stream = as_stream(stream_);
  double* part = reinterpret_cast<double*>(scratch);
  const bool wide = n_site > 32;
  const int threads = wide ? 128 : 256;
  const size_t smem = sizeof(double) * (size_t)(threads / 32) * 32 * (wide ? 64 : 32);  // 64 KB
  auto kern = wide ? k_pairs_part<2> : k_pairs_part<1>;
  RSED_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int n_sm = sm_count();
  RSED_REQUIRE(n_sm > 0, RSED_ECUDA, "no device");
  const int64_t blocks = (n_orbits + threads - 1) / threads;
  const int grid = (int)(blocks < 2 * n_sm ? blocks : 2 * n_sm);
  kern<<<dim3(grid, wide ? 2 : 1), threads, smem, stream>>>(n_site, n_orbits, repr_masks,
                                                           reinterpret_cast<const double2*>(x_orbit), part);
  RSED_CHECK_LAUNCH();
  const int nn = n_site * n_site;
  k_sum_blocks<1><<<(nn + 3) / 4, 128, 0, stream>>>(part, grid, nn, pairs);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}
