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
// 32 sites, 8 bosons, 10.5 million states: 120.6 ms with one rank, table and
// coefficient chain per hop and thread, 7.0 ms in this form.
template <int NP>
struct ObdmTile {
  static constexpr int TN = NP == 32 ? 32 : 16;       // states n of one tile
  static constexpr int NW = TN / (kCT / 32);          // of which one warp looks up NW
  static constexpr int U = NW * (NP / 32);            // lookups per lane
  static constexpr int RT = NP / 16;                  // outputs per thread and dimension
};

struct ObdmLayout {
  size_t binom, eta, chi, perm, tile, diag, total;
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
  l.diag = off;
  off += sizeof(double) * (kCT / 32) * 64;
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

template <int NP>
__global__ void __launch_bounds__(kCT, 2) k_obdm_part(rsed_group_t grp, const int4* __restrict__ table,
                                                      const uint64_t* __restrict__ repr_masks,
                                                      const uint64_t* __restrict__ stab_mask,
                                                      const uint64_t* __restrict__ member, int sector,
                                                      const double2* __restrict__ chi_g,
                                                      const double2* __restrict__ x, int per_warp,
                                                      int64_t n_a, int64_t n_b, ObdmLayout lay,
                                                      double2* __restrict__ part) {
  using T = ObdmTile<NP>;
  extern __shared__ __align__(16) unsigned char smem[];
  double2* Kt = reinterpret_cast<double2*>(smem + lay.tile);  // [TN][NP]
  double2* Bt = Kt + T::TN * NP;
  double2* eta = reinterpret_cast<double2*>(smem + lay.eta);
  double2* chi = reinterpret_cast<double2*>(smem + lay.chi);
  int64_t* binom = reinterpret_cast<int64_t*>(smem + lay.binom);
  double* diag = reinterpret_cast<double*>(smem + lay.diag);
  uint8_t* perm = smem + lay.perm;
  const int N = grp.n_site, ng = grp.n_group, kp1 = grp.n_filled + 1;
  for (int i = threadIdx.x; i < (N + 1) * kp1; i += kCT) binom[i] = grp.binom[i];
  bool twisted = false;
  for (int i = threadIdx.x; i < ng * N; i += kCT) {
    const double2 v = reinterpret_cast<const double2*>(grp.eta)[i];
    twisted |= v.x != 1.0 || v.y != 0.0;
    eta[i] = v;
    perm[i] = grp.perm[i];
  }
  for (int i = threadIdx.x; i < ng; i += kCT) chi[i] = chi_g[i];
  const bool unit = __syncthreads_or(twisted) == 0;
  const uint64_t first = (1ull << grp.n_filled) - 1ull;  // stands in for missing states (N <= 63)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const bool fermion = grp.fermionic != 0;
  const uint64_t sb = grp.species_b;
  const int64_t cb = sb ? binom[__popcll(sb) * kp1 + grp.n_filled_b] : 1;
  const double inv_ng = 1.0 / (double)ng;
  const uint64_t all = (1ull << N) - 1ull;
  double2 acc[T::RT][T::RT];
#pragma unroll
  for (int a = 0; a < T::RT; ++a)
#pragma unroll
    for (int b = 0; b < T::RT; ++b) acc[a][b] = make_double2(0.0, 0.0);
  double dacc[NP / 32];
#pragma unroll
  for (int h = 0; h < NP / 32; ++h) dacc[h] = 0.0;
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
      for (int u = 0; u < T::U; ++u) {
        const int i = lane + 32 * (u % (NP / 32));
        const uint64_t nn = n[u / (NP / 32)];
        double2 K = make_double2(0.0, 0.0), B = make_double2(0.0, 0.0);
        if (e[u].x >= 0 && (c[u].x != 0.0 || c[u].y != 0.0)) {
          const double S = (double)__popcll(st[u]);
          const double norm = 1.0 / sqrt((double)ng * S);
          K = rsed_state_amplitude(s[u], nn | (1ull << i), e[u].y, ph[u], st[u], grp, perm, eta, chi,
                                   make_double2(c[u].x * norm, c[u].y * norm));
          if ((mem[u] >> sector) & 1ull) {
            const double2 ch = chi[e[u].y];
            const double2 pc = cmul(make_double2((double)__int_as_float(e[u].z), (double)__int_as_float(e[u].w)),
                                    make_double2(ch.x, -ch.y));
            const double sr = S * norm;  // sqrt(S / |G|)
            B = cmul(c[u], make_double2(sr * pc.x, -sr * pc.y));
          }
          if (fermion && (__popcll(nn & ((1ull << i) - 1ull)) & 1)) {
            K = make_double2(-K.x, -K.y);
            B = make_double2(-B.x, -B.y);
          }
          dacc[u % (NP / 32)] += (c[u].x * c[u].x + c[u].y * c[u].y) * S * inv_ng;
        }
        const int q = warp * T::NW + u / (NP / 32);
        Kt[q * NP + i] = K;
        Bt[q * NP + i] = B;
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
#pragma unroll
  for (int h = 0; h < NP / 32; ++h) diag[warp * 64 + lane + 32 * h] = dacc[h];
  __syncthreads();
  double2* out = part + (int64_t)blockIdx.x * N * N;
#pragma unroll
  for (int a = 0; a < T::RT; ++a)
#pragma unroll
    for (int b = 0; b < T::RT; ++b) {
      const int i = ty + 16 * a, j = tx + 16 * b;
      if (i >= N || j >= N) continue;
      double2 v = acc[a][b];
      if (i == j) {
        v = make_double2(0.0, 0.0);
        for (int w = 0; w < kCT / 32; ++w) v.x += diag[w * 64 + i];
      }
      out[i * N + j] = v;
    }
}

// ---- density pairs --------------------------------------------------------------
//
// D[a][b] = sum_o |x_o|^2 n_a(s_o) n_b(s_o) over the representatives s_o; the
// structure factor's C[i][j] = (1/|G|) sum_g D[a][b] at i = g(a), j = g(b)
// follows from it on the host.
__global__ void __launch_bounds__(kCT) k_pairs_part(int n_site, int64_t n_orbits,
                                                    const uint64_t* __restrict__ repr_masks,
                                                    const double2* __restrict__ x, double* __restrict__ part) {
  extern __shared__ double dacc[];
  __shared__ uint64_t sm[kCT];
  __shared__ double sw[kCT];
  const int N = n_site, NN = N * N;
  const int64_t n_chunks = (n_orbits + kCT - 1) / kCT;
  for (int p = threadIdx.x; p < NN; p += kCT) dacc[p] = 0.0;
  for (int64_t ch = blockIdx.x; ch < n_chunks; ch += gridDim.x) {
    __syncthreads();
    const int64_t o = ch * kCT + threadIdx.x;
    if (o < n_orbits) {
      const double2 c = x[o];
      sm[threadIdx.x] = repr_masks[o];
      sw[threadIdx.x] = c.x * c.x + c.y * c.y;
    } else {
      sm[threadIdx.x] = 0;
      sw[threadIdx.x] = 0.0;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < NN; p += kCT) {
      const uint64_t both = (1ull << (p / N)) | (1ull << (p % N));
      double d = dacc[p];
      for (int q = 0; q < kCT; ++q)
        if ((sm[q] & both) == both) d += sw[q];
      dacc[p] = d;
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < NN; p += kCT) part[(int64_t)blockIdx.x * NN + p] = dacc[p];
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

template <int NP>
int obdm_launch(const rsed_group_t& grp, const int4* table, const uint64_t* repr_masks, const uint64_t* stab_mask,
                const uint64_t* member, int sector, const double2* chi, const double2* x, int64_t n_a, int64_t n_b,
                double2* part, int* grid_out, cudaStream_t stream) {
  const ObdmLayout lay = obdm_layout(grp.n_site, grp.n_filled, grp.n_group);
  if (lay.total > 48 * 1024)
    RSED_TRY_CUDA(cudaFuncSetAttribute(k_obdm_part<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lay.total));
  const int n_sm = sm_count();
  const int wave = one_wave((const void*)k_obdm_part<NP>, lay.total);
  RSED_REQUIRE(n_sm > 0 && wave > 0, RSED_ECUDA, "no occupancy for the one-body density kernel");
  int64_t grid = wave < n_sm * kObdmBlocksPerSm ? wave : n_sm * kObdmBlocksPerSm;
  // states n per warp: 32 amortise the unranking; fewer when the blocks of one
  // wave would not all have a chunk
  int per_warp = 32;
  while (per_warp > 4 && (n_a + n_b) / (8 * per_warp) < 2 * grid) per_warp /= 2;
  const int64_t pc = 8 * per_warp;
  const int64_t chunks = (n_a + pc - 1) / pc + (n_b + pc - 1) / pc;
  if (grid > chunks) grid = chunks;
  k_obdm_part<NP><<<(unsigned)grid, kCT, lay.total, stream>>>(grp, table, repr_masks, stab_mask, member, sector, chi,
                                                              x, per_warp, n_a, n_b, lay, part);
  RSED_CHECK_LAUNCH();
  *grid_out = (int)grid;
  return RSED_OK;
}

int pairs_grid(int n_site, size_t* smem) {
  *smem = sizeof(double) * (size_t)n_site * n_site;
  return one_wave((const void*)k_pairs_part, *smem);
}

}  // namespace

extern "C" size_t rsed_obdm_scratch_bytes(int32_t n_site) {
  const int n_sm = sm_count();
  if (n_sm <= 0) return 0;
  return sizeof(double2) * (size_t)n_sm * kObdmBlocksPerSm * n_site * n_site;
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
  double2* part = reinterpret_cast<double2*>(scratch);
  const int4* tb = reinterpret_cast<const int4*>(table);
  const double2* ch = reinterpret_cast<const double2*>(chi);
  const double2* xo = reinterpret_cast<const double2*>(x_orbit);
  int grid = 0;
  rc = N <= 32 ? obdm_launch<32>(*grp, tb, repr_masks, stab_mask, member, sector, ch, xo, n_a, n_b, part, &grid, stream)
               : obdm_launch<64>(*grp, tb, repr_masks, stab_mask, member, sector, ch, xo, n_a, n_b, part, &grid, stream);
  if (rc) return rc;
  k_sum_blocks<2><<<(nn + 3) / 4, 128, 0, stream>>>(reinterpret_cast<const double*>(part), grid, nn, rho);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

extern "C" size_t rsed_density_pairs_scratch_bytes(int32_t n_site) {
  size_t smem = 0;
  const int grid = pairs_grid(n_site, &smem);
  if (grid <= 0) return 0;
  return sizeof(double) * (size_t)grid * n_site * n_site;
}

extern "C" int rsed_density_pairs(int32_t n_site, int64_t n_orbits, const uint64_t* repr_masks,
                                  const double* x_orbit, double* pairs, void* scratch, size_t scratch_bytes,
                                  void* stream_) {
  RSED_REQUIRE(n_site >= 1 && n_site <= RSED_MAX_SITES, RSED_ERANGE, "n_site = %d outside [1, %d]", n_site,
               RSED_MAX_SITES);
  RSED_REQUIRE(repr_masks && x_orbit && pairs && scratch && n_orbits >= 1, RSED_EINVAL,
               "bad density-pair arguments");
  size_t smem = 0;
  const int grid = pairs_grid(n_site, &smem);
  RSED_REQUIRE(grid > 0, RSED_ECUDA, "no occupancy for the density-pair kernel");
  RSED_REQUIRE(scratch_bytes >= sizeof(double) * (size_t)grid * n_site * n_site, RSED_ESCRATCH,
               "density-pair scratch too small");
  cudaStream_t stream = as_stream(stream_);
  double* part = reinterpret_cast<double*>(scratch);
  k_pairs_part<<<grid, kCT, smem, stream>>>(n_site, n_orbits, repr_masks, reinterpret_cast<const double2*>(x_orbit),
                                           part);
  RSED_CHECK_LAUNCH();
  const int nn = n_site * n_site;
  k_sum_blocks<1><<<(nn + 3) / 4, 128, 0, stream>>>(part, grid, nn, pairs);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}
