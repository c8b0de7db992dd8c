// K1-K5: combinadic enumeration, orbit-stabilizer catalog, flux phase update
// and sector membership.
//
// Layout in HBM (one catalog):
//   table       C(N,k) x 16 B   rsed_entry_t, indexed by combinadic rank
//   repr_masks  n_orb  x 8 B    representative masks, ascending (= rank order)
//   stab_mask   n_orb  x 8 B    bit g set iff g(rep) == rep
//   stab_off    n_orb+1 x 8 B   exclusive offsets into stab_phase
//   stab_phase  sum|Stab| x 16 B complex128 alpha_h(rep), ascending h
#include <cstring>
#include <mutex>
#include "rsed_internal.cuh"

namespace {

constexpr int kFlagThreads = 256;           // threads per block in the flag pass
constexpr int kRanksPerWord = 32;           // one uint32 bitmap word
// Ranks of one block of the flag and list passes: large bases amortise the
// block's tables over 8192 ranks; below 2^20 states 256 ranks a block (one
// rank per thread) spread the little work over the SMs (12,870 states: two
// blocks of 8192 took 329 us).
int ranks_per_block(int64_t n_states) { return n_states >= (1ll << 20) ? 8192 : 256; }

struct GroupView {
  const int64_t* binom;
  const uint8_t* perm;
  const double* angle;
  const double2* eta;
};

// Stage the group tables into dynamic shared memory.
__device__ GroupView stage_group(const rsed_group_t& g, unsigned char* smem, size_t binom_off,
                                 size_t perm_off, size_t angle_off, size_t eta_off,
                                 bool with_angle, bool with_eta) {
  const int kp1 = g.n_filled + 1;
  const int nb = (g.n_site + 1) * kp1;
  int64_t* sb = reinterpret_cast<int64_t*>(smem + binom_off);
  for (int i = threadIdx.x; i < nb; i += blockDim.x) sb[i] = g.binom[i];
  const int np = g.n_group * g.n_site;
  uint8_t* sp = smem + perm_off;
  for (int i = threadIdx.x; i < np; i += blockDim.x) sp[i] = g.perm[i];
  GroupView v{sb, sp, nullptr, nullptr};
  if (with_angle) {
    double* sa = reinterpret_cast<double*>(smem + angle_off);
    for (int i = threadIdx.x; i < np; i += blockDim.x) sa[i] = g.angle[i];
    v.angle = sa;
  }
  if (with_eta) {
    double2* se = reinterpret_cast<double2*>(smem + eta_off);
    const double2* ge = reinterpret_cast<const double2*>(g.eta);
    for (int i = threadIdx.x; i < np; i += blockDim.x) se[i] = ge[i];
    v.eta = se;
  }
  __syncthreads();
  return v;
}

// A site permutation as rotations: the sites that move by the same distance
// form a class, and the image of a mask is the union of its classes, each
// rotated by its distance.  A translation of a periodic lattice has two classes
// per wrapped direction at most (4 in two dimensions), so an image takes 4
// and-rotate-or steps instead of one table step per occupied site.  Elements of
// more than kClasses distances (reflections, rotations) take the image bit by bit.
constexpr int kClasses = 8;

template <typename M>
struct MoveClass {
  M mask;
  M rot;
};
template <typename M>
struct GroupMoves {
  MoveClass<M> cls[RSED_MAX_GROUP][kClasses];
  int n[RSED_MAX_GROUP];
};

__device__ __forceinline__ uint32_t rotl(uint32_t x, uint32_t d) { return __funnelshift_l(x, x, d); }
__device__ __forceinline__ uint64_t rotl(uint64_t x, uint64_t d) {
  const int s = (int)d & 63;
  return (x << s) | (x >> ((64 - s) & 63));
}

__device__ __forceinline__ int low_bit(uint32_t m) { return __ffs((int)m) - 1; }
__device__ __forceinline__ int low_bit(uint64_t m) { return __ffsll((long long)m) - 1; }
__device__ __forceinline__ int count_bits(uint32_t m) { return __popc(m); }
__device__ __forceinline__ int count_bits(uint64_t m) { return __popcll(m); }

// rsed_rank_any on masks and ranks of the width of M (up to 32 sites every rank
// is below C(32, 16) < 2^31).
template <typename M, typename I>
__device__ __forceinline__ I rank_of(M m, const I* binom, int kp1, M sb, I cb) {
  I ra = 0, rb = 0;
  int ja = 1, jb = 1;
  while (m) {
    const int b = low_bit(m);
    m &= m - 1;
    if (sb == 0) {
      ra += binom[b * kp1 + ja];
      ++ja;
    } else {
      const int below_b = count_bits((M)(sb & (((M)1 << b) - 1)));
      if ((sb >> b) & 1) {
        rb += binom[below_b * kp1 + jb];
        ++jb;
      } else {
        ra += binom[(b - below_b) * kp1 + ja];
        ++ja;
      }
    }
  }
  return sb ? ra * cb + rb : ra;
}

// Image of m under the site permutation perm, bit by bit.
template <typename M>
__device__ __forceinline__ M permuted(M m, const uint8_t* perm) {
  M img = 0;
  for (; m; m &= m - 1) img |= (M)1 << perm[low_bit(m)];
  return img;
}

// Fills `mv` from the staged permutations; the elements with more than kClasses
// classes (theirs are incomplete), as a bitmask.  All threads of the block call it.
template <typename M>
__device__ uint64_t stage_moves(const rsed_group_t& grp, const uint8_t* perm, GroupMoves<M>& mv) {
  constexpr int W = 8 * sizeof(M) - 1;
  __shared__ unsigned long long many;
  if (threadIdx.x == 0) many = 0;
  for (int g = threadIdx.x; g < grp.n_group; g += blockDim.x) mv.n[g] = 0;
  __syncthreads();
  for (int t = threadIdx.x; t < grp.n_group * grp.n_site; t += blockDim.x) {
    const int g = t / grp.n_site, i = t % grp.n_site;
    const uint8_t* pg = perm + g * grp.n_site;
    const int d = (pg[i] - i) & W;
    bool first = true;
    for (int k = 0; k < i && first; ++k) first = ((pg[k] - k) & W) != d;
    if (!first) continue;
    M mask = 0;
    for (int k = i; k < grp.n_site; ++k)
      if (((pg[k] - k) & W) == d) mask |= (M)1 << k;
    const int at = atomicAdd(&mv.n[g], 1);  // the order of the classes does not matter
    if (at < kClasses)
      mv.cls[g][at] = MoveClass<M>{mask, (M)d};
    else
      atomicOr(&many, 1ull << g);
  }
  __syncthreads();
  return many;
}

// Pass 1: representative flags as a bitmap (symmetry_resolved_ed.py:519-528).
// A thread tests R consecutive ranks (32 / R lanes share a bitmap word), first
// against the images by move classes, each class loaded once for the R masks.
// Bound by integer issue: some lane of a warp nearly always holds a
// representative, so leaving that loop at the first smaller image saved nothing,
// and the images themselves are the cost.  The elements without few classes come
// after, for the ranks that are left, up to the first smaller image: their images
// cost a step per occupied site.  M = uint32_t up to 32 sites.
// 10.5 million states, 32 sites, |G| = 16: 865 us with one image per occupied
// site step and 32 ranks per thread, 139 us in this form.  Dihedral group of 26
// sites, 10.4 million states, half of 52 elements bit by bit: 2.46 ms with 32
// ranks per thread and an exit at the first smaller image, 7.0 ms with every
// element of the group bit by bit and no exit, 0.67 ms as here.
template <typename M, int R>
__global__ void __launch_bounds__(kFlagThreads) k_rep_flags(rsed_group_t grp, uint32_t* bitmap, int64_t* block_count,
                                                            int per_block, GroupSmemLayout lay) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ GroupMoves<M> mv;
  __shared__ int warp_sums[kFlagThreads / 32];
  GroupView gv = stage_group(grp, smem, lay.binom_off, lay.perm_off, 0, 0, false, false);
  const uint64_t many = stage_moves<M>(grp, gv.perm, mv);
  const int kp1 = grp.n_filled + 1;
  int count = 0;
  for (int t = 0; t < per_block; t += kFlagThreads * R) {
    const int64_t r0 = (int64_t)blockIdx.x * per_block + t + (int64_t)threadIdx.x * R;
    M m[R];
    uint32_t bits = 0;
    RankWalker w;
    if (r0 < grp.n_states) w.init(r0, grp, gv.binom, kp1);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      m[i] = 0;
      if (r0 + i < grp.n_states) {
        m[i] = (M)w.m;
        bits |= 1u << i;
      }
      if (i + 1 < R && r0 + i + 1 < grp.n_states) w.next();
    }
    for (int g = 0; g < grp.n_group; ++g) {
      if ((many >> g) & 1ull) continue;
      M img[R];
#pragma unroll
      for (int i = 0; i < R; ++i) img[i] = 0;
      for (int c = 0; c < mv.n[g]; ++c) {
        const MoveClass<M> cl = mv.cls[g][c];
#pragma unroll
        for (int i = 0; i < R; ++i) img[i] |= rotl(m[i] & cl.mask, cl.rot);
      }
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (img[i] < m[i]) bits &= ~(1u << i);
    }
    if (many) {
#pragma unroll
      for (int i = 0; i < R; ++i)
        for (uint64_t h = (bits >> i) & 1u ? many : 0; h; h &= h - 1)
          if (permuted(m[i], gv.perm + (__ffsll((long long)h) - 1) * grp.n_site) < m[i]) {
            bits &= ~(1u << i);
            break;
          }
    }
    count += __popc(bits);
    // the 32 / R lanes of a word put their bits together
    if (R < 32) {
      bits <<= (threadIdx.x & (32 / R - 1)) * R;
#pragma unroll
      for (int o = 1; o < 32 / R; o <<= 1) bits |= __shfl_xor_sync(0xffffffffu, bits, o);
    }
    if ((threadIdx.x & (32 / R - 1)) == 0 && r0 < grp.n_states) bitmap[r0 / kRanksPerWord] = bits;
  }
  for (int o = 16; o > 0; o >>= 1) count += __shfl_down_sync(0xffffffffu, count, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = count;
  __syncthreads();
  if (threadIdx.x == 0) {
    int64_t s = 0;
    for (int k = 0; k < kFlagThreads / 32; ++k) s += warp_sums[k];
    block_count[blockIdx.x] = s;
  }
}

// Pass 2a: representative masks in rank order; rep index = exclusive scan of
// the flags (symmetry_resolved_ed.py:531-532).  The block also sets its ranks'
// entries to (rep -1, g 0, alpha 0), the reference's initial table
// (symmetry_resolved_ed.py:1359-1361); every state of a group's catalog is
// overwritten by k_expand.
__global__ void k_rep_list(rsed_group_t grp, const uint32_t* bitmap, const int64_t* block_off, int per_block,
                           uint64_t* repr_masks, RsedEntry* table, GroupSmemLayout lay) {
  extern __shared__ __align__(16) unsigned char smem[];
  GroupView gv = stage_group(grp, smem, lay.binom_off, lay.perm_off, 0, 0, false, false);
  __shared__ int warp_tot[kFlagThreads / 32];
  const int kp1 = grp.n_filled + 1;
  const int64_t first = (int64_t)blockIdx.x * per_block;
  for (int64_t r = first + threadIdx.x; r < min(grp.n_states, first + per_block); r += blockDim.x)
    reinterpret_cast<int4*>(table)[r] = make_int4(-1, 0, 0, 0);
  const int64_t r0 = first + (int64_t)threadIdx.x * kRanksPerWord;
  uint32_t bits = ((int)threadIdx.x * kRanksPerWord < per_block && r0 < grp.n_states) ? bitmap[r0 / kRanksPerWord] : 0u;
  // block-exclusive prefix of popcounts
  int c = __popc(bits);
  int incl = c;
  const int lane = threadIdx.x & 31;
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[threadIdx.x >> 5] = incl;
  __syncthreads();
  int warp_prefix = 0;
  for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) warp_prefix += warp_tot[w];
  int64_t off = block_off[blockIdx.x] + warp_prefix + (incl - c);
  if (bits) {
    RankWalker w;
    w.init(r0, grp, gv.binom, kp1);
    for (int i = 0; i < kRanksPerWord; ++i) {
      if ((bits >> i) & 1u) repr_masks[off++] = w.m;
      const uint32_t rest = (i < kRanksPerWord - 1) ? (bits >> (i + 1)) : 0u;
      if (rest == 0u) break;
      w.next();
    }
  }
}

// Canonicalisation amplitude of U_g on the representative m as the catalog
// computes it: exp(i * angle-sum) with the fermionic flip
// (symmetry_resolved_ed.py:536-551), except at n_filled in {0, n_site} where
// the reference takes the product form (:483-508).
__device__ __forceinline__ double2 catalog_alpha(uint64_t m, int g, const rsed_group_t& grp,
                                                 const GroupView& gv, bool product_form,
                                                 uint64_t* img) {
  const uint8_t* pg = gv.perm + g * grp.n_site;
  if (product_form) return rsed_phase_product(m, pg, gv.eta + g * grp.n_site, grp.fermionic, img);
  *img = rsed_permute(m, pg);
  double ang = rsed_angle_sum(m, gv.angle + g * grp.n_site, grp.n_site);
  double s, c;
  sincos(ang, &s, &c);
  double2 a = make_double2(c, s);
  if (grp.fermionic && rsed_perm_parity(m, pg)) a = rsed_cmul_exact(a, make_double2(-1.0, 0.0));
  return a;
}

// Pass 2b: orbit expansion into the representative table (g ascending, the last
// writer wins for stabilizer cosets, symmetry_resolved_ed.py:553-560) and the
// stabilizer bitmask (:563).  One thread per (orbit, group element), the group
// tables transposed to [site][g] so that the lanes of an orbit read consecutive
// words; the image, the byte-ordered angle sum and the parity come out of one
// walk over the occupied sites.  In an orbit with a stabilizer several elements
// reach the same state and only the largest of them writes.
// Bound by integer issue and the shared-memory lookups of the two walks (with
// sincos or the scattered writes taken out it ran as long); masks and ranks are
// 32-bit up to 32 sites.  657,756 orbits of 16 elements: 267 us with one thread
// per orbit walking its images, 309 us with 64-bit masks, 224 us in this form.
// 81,712 orbits of 60 elements on 36 sites, three quarters symmetric: 522 us with
// the later elements' images walked again for the last writer, 149 us with the
// images of the step in shared memory.
template <typename M, typename I>
__global__ void __launch_bounds__(256) k_expand(rsed_group_t grp, int64_t n_orb, const uint64_t* repr_masks,
                                                RsedEntry* table, uint64_t* stab_mask, GroupSmemLayout lay, int* err) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_stab[256];
  __shared__ M s_img[256];
  const bool product_form = (grp.n_filled == 0 || grp.n_filled == grp.n_site);
  const int N = grp.n_site, ng = grp.n_group, kp1 = grp.n_filled + 1;
  I* binom = reinterpret_cast<I*>(smem + lay.binom_off);
  double* angle = reinterpret_cast<double*>(smem + lay.angle_off);   // [site][g]
  uint8_t* perm = smem + lay.perm_off;                               // [site][g]
  for (int i = threadIdx.x; i < (N + 1) * kp1; i += blockDim.x) binom[i] = (I)grp.binom[i];
  for (int i = threadIdx.x; i < ng * N; i += blockDim.x) {
    const int g = i / N, b = i % N;
    perm[b * ng + g] = grp.perm[i];
    angle[b * ng + g] = grp.angle[i];
  }
  const int per_block = 256 / ng;  // orbits of one block and step
  const int lo = threadIdx.x / ng, g = threadIdx.x % ng;
  const I cb = grp.species_b ? (I)grp.binom[__popcll(grp.species_b) * kp1 + grp.n_filled_b] : 1;
  for (int64_t o0 = (int64_t)blockIdx.x * per_block; o0 < n_orb; o0 += (int64_t)gridDim.x * per_block) {
    __syncthreads();  // the tables are staged, the previous step's stabilizers read
    if (threadIdx.x < per_block) s_stab[threadIdx.x] = 0ull;
    __syncthreads();
    const int64_t o = o0 + lo;
    const bool act = lo < per_block && o < n_orb;
    M m = 0, img = 0;
    double2 a = make_double2(1.0, 0.0);
    if (act) {
      m = (M)repr_masks[o];
      if (product_form) {
        uint64_t placed;
        a = rsed_phase_product(m, grp.perm + g * N, reinterpret_cast<const double2*>(grp.eta) + g * N, grp.fermionic,
                               &placed);
        img = (M)placed;
      } else {
        // rsed_angle_sum's order: partial sums per byte, bytes ascending
        double total = 0.0, part = 0.0;
        int byte = 0, par = 0;
        for (M t = m; t; t &= t - 1) {
          const int b = low_bit(t);
          const int p = perm[b * ng + g];
          // placed images above p (the shift by p + 1 in two steps: p + 1 can be the width)
          if (grp.fermionic) par ^= count_bits((M)((img >> p) >> 1)) & 1;
          img |= (M)1 << p;
          if ((b >> 3) != byte) {
            total = __dadd_rn(total, part);
            part = 0.0;
            byte = b >> 3;
          }
          part = __dadd_rn(part, angle[b * ng + g]);
        }
        total = __dadd_rn(total, part);
        if (total != 0.0) sincos(total, &a.y, &a.x);  // sincos(0) = (0, 1)
        if (par) a = rsed_cmul_exact(a, make_double2(-1.0, 0.0));
      }
      if (img == m) atomicOr(&s_stab[lo], 1ull << g);
      s_img[threadIdx.x] = img;
    }
    __syncthreads();
    if (!act) continue;
    const uint64_t stab = s_stab[lo];
    if (g == 0) stab_mask[o] = stab;
    bool last = true;
    if (__popcll(stab) > 1)
      for (int h = g + 1; h < ng && last; ++h) last = s_img[lo * ng + h] != img;
    if (!last) continue;
    const int64_t idx = rank_of<M, I>(img, binom, kp1, (M)grp.species_b, cb);
    if (idx < 0 || idx >= grp.n_states) {
      rsed_flag_error(err, 1);
      continue;
    }
    int4 e;
    e.x = (int32_t)o;
    e.y = g;
    e.z = __float_as_int(__double2float_rn(a.x));
    e.w = __float_as_int(__double2float_rn(a.y));
    reinterpret_cast<int4*>(table)[idx] = e;
  }
}

__global__ void k_stab_counts(int64_t n_orb, const uint64_t* stab_mask, int64_t* counts) {
  int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o < n_orb) counts[o] = __popcll(stab_mask[o]);
}

// Stabilizer phases (complex128), ascending g (symmetry_resolved_ed.py:563-571).
__global__ void k_stab_phases(rsed_group_t grp, int64_t n_orb, const uint64_t* repr_masks,
                              const uint64_t* stab_mask, const int64_t* stab_off,
                              double2* stab_phase, GroupSmemLayout lay) {
  extern __shared__ __align__(16) unsigned char smem[];
  const bool product_form = (grp.n_filled == 0 || grp.n_filled == grp.n_site);
  GroupView gv = stage_group(grp, smem, lay.binom_off, lay.perm_off, lay.angle_off, lay.eta_off,
                             true, product_form);
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n_orb) return;
  const uint64_t m = repr_masks[o];
  uint64_t s = stab_mask[o];
  int64_t off = stab_off[o];
  while (s) {
    int g = __ffsll((long long)s) - 1;
    uint64_t img;
    stab_phase[off++] = catalog_alpha(m, g, grp, gv, product_form, &img);
    s &= s - 1;
  }
}

// K4: flux phase update in product form (symmetry_resolved_ed.py:1248-1268),
// stabilizer phases of every orbit, ascending g (:1248-1257).
__global__ void k_phase_stab(rsed_group_t grp, int64_t n_orb, const uint64_t* repr_masks, const uint64_t* stab_mask,
                             const int64_t* stab_off, double2* stab_phase, GroupSmemLayout lay) {
  extern __shared__ __align__(16) unsigned char smem[];
  GroupView gv = stage_group(grp, smem, lay.binom_off, lay.perm_off, 0, lay.eta_off, false, true);
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n_orb) return;
  const uint64_t m = repr_masks[o];
  uint64_t s = stab_mask[o];
  int64_t off = stab_off[o];
  while (s) {
    int g = __ffsll((long long)s) - 1;
    uint64_t img;
    stab_phase[off++] =
        rsed_phase_product(m, gv.perm + g * grp.n_site, gv.eta + g * grp.n_site, grp.fermionic, &img);
    s &= s - 1;
  }
}

// The amplitudes of the representative table.  The permutations are those the
// table was built with, so every state keeps its orbit and its (last) group
// element and only the phase is new: one thread per table entry, read and
// written in rank order.  The entry is checked against the group: its element
// has to map the representative to the state of this rank.
// Bound by the walk over the occupied sites (a 16-B lookup and an unfused
// complex product per site, a lookup per site of the image's rank).  10.5
// million states, 32 sites: 247 us with one thread per orbit, its |G| entries
// read and rewritten at random, 145 us in this form (135 without the products).
template <typename M, typename I>
__global__ void __launch_bounds__(256) k_phase_table(rsed_group_t grp, int64_t n_orb, const uint64_t* repr_masks,
                                                     int4* table, GroupSmemLayout lay, int* err) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int N = grp.n_site, ng = grp.n_group, kp1 = grp.n_filled + 1;
  I* binom = reinterpret_cast<I*>(smem + lay.binom_off);
  double2* eta = reinterpret_cast<double2*>(smem + lay.eta_off);
  uint8_t* perm = smem + lay.perm_off;
  for (int i = threadIdx.x; i < (N + 1) * kp1; i += blockDim.x) binom[i] = (I)grp.binom[i];
  bool twisted = false;
  for (int i = threadIdx.x; i < ng * N; i += blockDim.x) {
    const double2 v = reinterpret_cast<const double2*>(grp.eta)[i];
    twisted |= v.x != 1.0 || v.y != 0.0;
    eta[i] = v;
    perm[i] = grp.perm[i];
  }
  const bool unit = __syncthreads_or(twisted) == 0;  // products of exact ones are left out
  const I cb = grp.species_b ? binom[__popcll(grp.species_b) * kp1 + grp.n_filled_b] : 1;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < grp.n_states; r += stride) {
    int4 e = table[r];
    if (e.x < 0 || e.x >= n_orb || e.y < 0 || e.y >= ng) {
      rsed_flag_error(err, 2);
      continue;
    }
    const int base = e.y * N;
    M img = 0;
    int par = 0;
    double2 a = make_double2(1.0, 0.0);
    for (M t = (M)__ldg(repr_masks + e.x); t; t &= t - 1) {
      const int b = low_bit(t);
      const int p = perm[base + b];
      if (grp.fermionic) par ^= count_bits((M)((img >> p) >> 1)) & 1;
      img |= (M)1 << p;
      if (!unit) a = rsed_cmul_exact(a, eta[base + b]);
    }
    if (grp.fermionic) a = rsed_cmul_exact(a, make_double2(par ? -1.0 : 1.0, 0.0));
    if ((int64_t)rank_of<M, I>(img, binom, kp1, (M)grp.species_b, cb) != r) {
      rsed_flag_error(err, 2);
      continue;
    }
    e.z = __float_as_int(__double2float_rn(a.x));
    e.w = __float_as_int(__double2float_rn(a.y));
    table[r] = e;
  }
}

// K5: sector membership for many irreps at once (symmetry_resolved_ed.py:1484-1512).
__global__ void k_sector_members(int64_t n_orb, int n_group, int n_sec, const uint64_t* stab_mask,
                                 const int64_t* stab_off, const double2* stab_phase,
                                 const double2* chi, double atol, uint64_t* member,
                                 double* sqrt_stab, unsigned long long* dims) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* schi = reinterpret_cast<double2*>(smem);
  for (int i = threadIdx.x; i < n_sec * n_group; i += blockDim.x) schi[i] = chi[i];
  __shared__ unsigned int bcount[64];
  for (int i = threadIdx.x; i < 64; i += blockDim.x) bcount[i] = 0;
  __syncthreads();
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o < n_orb) {
    const uint64_t sm = stab_mask[o];
    const int64_t off = stab_off[o];
    uint64_t bits = 0;
    for (int s = 0; s < n_sec; ++s) {
      bool ok = true;
      uint64_t t = sm;
      int64_t j = off;
      while (t) {
        int g = __ffsll((long long)t) - 1;
        double2 a = stab_phase[j++];
        double2 c = schi[s * n_group + g];
        if (!(hypot(c.x - a.x, c.y - a.y) <= atol)) {
          ok = false;
          break;
        }
        t &= t - 1;
      }
      if (ok) {
        bits |= 1ull << s;
        atomicAdd(&bcount[s], 1u);
      }
    }
    member[o] = bits;
    sqrt_stab[o] = sqrt((double)__popcll(sm));
  }
  __syncthreads();
  for (int s = threadIdx.x; s < n_sec; s += blockDim.x)
    if (bcount[s]) atomicAdd(&dims[s], (unsigned long long)bcount[s]);
}

__global__ void k_member_bit(int64_t n, const uint64_t* member, int sector, int64_t* out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (member[i] >> sector) & 1ull;
}

__global__ void k_sector_rows(int64_t n, const uint64_t* member, int sector, const int64_t* pos,
                              int32_t* orbit_of_row, int32_t* row_of_orbit) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if ((member[i] >> sector) & 1ull) {
    int64_t r = pos[i];
    if (orbit_of_row) orbit_of_row[r] = (int32_t)i;
    if (row_of_orbit) row_of_orbit[i] = (int32_t)r;
  } else if (row_of_orbit) {
    row_of_orbit[i] = -1;
  }
}

// Density-density diagonal per orbit in term order (symmetry_resolved_ed.py:641-646).
__global__ void k_density_diag(int64_t n_orb, const uint64_t* repr_masks, int nd, const uint8_t* di,
                               const uint8_t* dj, const double2* dv, double2* hdiag) {
  int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n_orb) return;
  uint64_t m = repr_masks[o];
  double2 h = make_double2(0.0, 0.0);
  for (int d = 0; d < nd; ++d) {
    if (((m >> di[d]) & 1ull) && ((m >> dj[d]) & 1ull)) {
      h.x = __dadd_rn(h.x, dv[d].x);
      h.y = __dadd_rn(h.y, dv[d].y);
    }
  }
  hdiag[o] = h;
}

// ---- generic exclusive scan -------------------------------------------------
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ int64_t block_exclusive_scan(int64_t v, int64_t* total) {
  __shared__ int64_t ws[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nw = (int)(blockDim.x >> 5);
  int64_t incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    int64_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  if (w == 0) {
    int64_t x = (lane < nw) ? ws[lane] : 0;
    int64_t xi = x;
    for (int o = 1; o < 32; o <<= 1) {
      int64_t t = __shfl_up_sync(0xffffffffu, xi, o);
      if (lane >= o) xi += t;
    }
    ws[lane] = xi - x;
    if (lane == nw - 1) *total = xi;
  }
  __syncthreads();
  int64_t r = ws[w] + (incl - v);
  __syncthreads();
  return r;
}

__global__ void k_tile_sums(const int64_t* in, int64_t n, int64_t* tile_sum) {
  __shared__ int64_t tot;
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  int64_t s = 0;
  for (int j = 0; j < kScanItems; ++j) {
    int64_t i = base + (int64_t)threadIdx.x * kScanItems + j;
    if (i < n) s += in[i];
  }
  block_exclusive_scan(s, &tot);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

__global__ void k_scan_tiles(int64_t* tile_sum, int64_t n_tiles, int64_t* total_out) {
  __shared__ int64_t tot;
  int64_t carry = 0;
  for (int64_t base = 0; base < n_tiles; base += kScanThreads) {
    int64_t i = base + threadIdx.x;
    int64_t v = i < n_tiles ? tile_sum[i] : 0;
    int64_t ex = block_exclusive_scan(v, &tot);
    if (i < n_tiles) tile_sum[i] = carry + ex;
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total_out = carry;
}

__global__ void k_tile_scan(const int64_t* in, int64_t n, const int64_t* tile_off,
                            const int64_t* total, int64_t* out) {
  __shared__ int64_t tot;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t v[kScanItems];
  int64_t s = 0;
  for (int j = 0; j < kScanItems; ++j) {
    int64_t i = base + j;
    v[j] = i < n ? in[i] : 0;
    s += v[j];
  }
  int64_t ex = block_exclusive_scan(s, &tot) + tile_off[blockIdx.x];
  for (int j = 0; j < kScanItems; ++j) {
    int64_t i = base + j;
    if (i < n) out[i] = ex;
    ex += v[j];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = *total;
}

}  // namespace

// ---- host ------------------------------------------------------------------

size_t rsed_scan_scratch_bytes(int64_t n) {
  int64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles < 1) tiles = 1;
  return align_up((size_t)(tiles + 1) * sizeof(int64_t), 256);
}

int rsed_exclusive_scan_i64(const int64_t* in, int64_t* out, int64_t n, void* scratch,
                            size_t scratch_bytes, cudaStream_t stream) {
  int64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles < 1) tiles = 1;
  RSED_REQUIRE(scratch_bytes >= rsed_scan_scratch_bytes(n), RSED_ESCRATCH, "scan scratch too small");
  int64_t* tile_sum = reinterpret_cast<int64_t*>(scratch);
  int64_t* total = tile_sum + tiles;
  if (n == 0) {
    RSED_TRY_CUDA(cudaMemsetAsync(out, 0, sizeof(int64_t), stream));
    return RSED_OK;
  }
  k_tile_sums<<<(unsigned)tiles, kScanThreads, 0, stream>>>(in, n, tile_sum);
  RSED_CHECK_LAUNCH();
  k_scan_tiles<<<1, kScanThreads, 0, stream>>>(tile_sum, tiles, total);
  RSED_CHECK_LAUNCH();
  k_tile_scan<<<(unsigned)tiles, kScanThreads, 0, stream>>>(in, n, tile_sum, total, out);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

GroupSmemLayout group_smem_layout(int n_site, int n_filled, int n_group, bool with_eta,
                                  bool with_angle) {
  GroupSmemLayout l{};
  size_t off = 0;
  l.binom_off = off;
  off = align_up(off + sizeof(int64_t) * (size_t)(n_site + 1) * (size_t)(n_filled + 1), 16);
  l.angle_off = off;
  if (with_angle) off = align_up(off + sizeof(double) * (size_t)n_group * n_site, 16);
  l.eta_off = off;
  if (with_eta) off = align_up(off + 2 * sizeof(double) * (size_t)n_group * n_site, 16);
  l.perm_off = off;
  off = align_up(off + (size_t)n_group * n_site, 16);
  l.total = off;
  return l;
}

// Worst-case staged group (63 sites, 31 particles, |G| = 64) needs ~115 KB.
static int set_catalog_smem_limits() {
  static bool done = false;
  if (done) return RSED_OK;
  const int big = 160 * 1024;
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_rep_flags<uint32_t, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_rep_flags<uint32_t, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_rep_flags<uint64_t, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_rep_flags<uint64_t, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_rep_list, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_expand<uint32_t, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_expand<uint64_t, int64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_stab_phases, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_phase_stab, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_phase_table<uint32_t, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_phase_table<uint64_t, int64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  RSED_TRY_CUDA(cudaFuncSetAttribute(k_sector_members, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  done = true;
  return RSED_OK;
}

// Blocks of `threads` that the device holds at once.
static int blocks_of_one_wave(const void* kern, int threads, size_t smem, int64_t* out) {
  int dev = 0, n_sm = 0, per_sm = 0;
  RSED_TRY_CUDA(cudaGetDevice(&dev));
  RSED_TRY_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  RSED_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
  *out = (int64_t)n_sm * (per_sm > 0 ? per_sm : 1);
  return RSED_OK;
}

int check_group(const rsed_group_t* g) {
  RSED_REQUIRE(g != nullptr, RSED_EINVAL, "group descriptor is NULL");
  RSED_REQUIRE(g->n_site >= 1 && g->n_site <= RSED_MAX_SITES, RSED_ERANGE,
               "n_site = %d outside [1, %d]", g->n_site, RSED_MAX_SITES);
  RSED_REQUIRE(g->n_filled >= 0 && g->n_filled <= g->n_site, RSED_EINVAL,
               "n_filled = %d outside [0, n_site]", g->n_filled);
  RSED_REQUIRE(g->n_group >= 1 && g->n_group <= RSED_MAX_GROUP, RSED_ERANGE,
               "|G| = %d outside [1, %d]", g->n_group, RSED_MAX_GROUP);
  RSED_REQUIRE(g->n_states >= 1, RSED_EINVAL, "n_states must be >= 1");
  RSED_REQUIRE(g->binom && g->perm, RSED_EINVAL, "group tables missing");
  if (g->species_b) {
    const uint64_t all = (g->n_site >= 64) ? ~0ull : ((1ull << g->n_site) - 1ull);
    const int nb = __builtin_popcountll(g->species_b);
    RSED_REQUIRE((g->species_b & ~all) == 0ull && nb < g->n_site, RSED_EINVAL,
                 "species_b must mark a proper subset of the sites");
    RSED_REQUIRE(g->n_filled_b >= 0 && g->n_filled_b <= nb && g->n_filled_b <= g->n_filled &&
                     g->n_filled - g->n_filled_b <= g->n_site - nb,
                 RSED_EINVAL, "n_filled_b = %d does not fit the two species", g->n_filled_b);
  }
  return RSED_OK;
}

namespace {
struct CatalogScratch {
  uint32_t* bitmap;
  int64_t* block_count;
  int64_t* block_off;  // n_blocks + 1
  void* scan;
  size_t scan_bytes;
  int64_t n_blocks;
  int per_block;  // ranks of one block
};

CatalogScratch carve_catalog_scratch(const rsed_group_t* g, void* base) {
  CatalogScratch s{};
  s.per_block = ranks_per_block(g->n_states);
  s.n_blocks = (g->n_states + s.per_block - 1) / s.per_block;
  char* p = reinterpret_cast<char*>(base);
  size_t off = 0;
  s.bitmap = reinterpret_cast<uint32_t*>(p + off);
  off = align_up(off + sizeof(uint32_t) * (size_t)(s.n_blocks * (s.per_block / kRanksPerWord)), 256);
  s.block_count = reinterpret_cast<int64_t*>(p + off);
  off = align_up(off + sizeof(int64_t) * (size_t)s.n_blocks, 256);
  s.block_off = reinterpret_cast<int64_t*>(p + off);
  off = align_up(off + sizeof(int64_t) * (size_t)(s.n_blocks + 1), 256);
  s.scan = p + off;
  s.scan_bytes = rsed_scan_scratch_bytes(s.n_blocks);
  return s;
}
}  // namespace

extern "C" size_t rsed_catalog_scratch_bytes(const rsed_group_t* g) {
  if (!g || g->n_states < 1) return 0;
  const int per_block = ranks_per_block(g->n_states);
  int64_t n_blocks = (g->n_states + per_block - 1) / per_block;
  size_t b = align_up(sizeof(uint32_t) * (size_t)(n_blocks * (per_block / kRanksPerWord)), 256);
  b += align_up(sizeof(int64_t) * (size_t)n_blocks, 256);
  b += align_up(sizeof(int64_t) * (size_t)(n_blocks + 1), 256);
  b += rsed_scan_scratch_bytes(n_blocks);
  return b;
}

extern "C" int rsed_catalog_count(const rsed_group_t* g, void* scratch, size_t scratch_bytes,
                                  int64_t* n_orbits_out, void* stream_) {
  int rc = check_group(g);
  if (rc) return rc;
  RSED_REQUIRE(scratch_bytes >= rsed_catalog_scratch_bytes(g), RSED_ESCRATCH,
               "catalog scratch too small (%zu < %zu)", scratch_bytes, rsed_catalog_scratch_bytes(g));
  RSED_REQUIRE(n_orbits_out != nullptr, RSED_EINVAL, "n_orbits_out is NULL");
  cudaStream_t stream = as_stream(stream_);
  rc = set_catalog_smem_limits();
  if (rc) return rc;
  CatalogScratch s = carve_catalog_scratch(g, scratch);
  GroupSmemLayout lay = group_smem_layout(g->n_site, g->n_filled, g->n_group, false, false);
  const bool wide = g->n_site > 32;
  auto flags = s.per_block == 8192 ? (wide ? k_rep_flags<uint64_t, 8> : k_rep_flags<uint32_t, 8>)
                                   : (wide ? k_rep_flags<uint64_t, 1> : k_rep_flags<uint32_t, 1>);
  flags<<<(unsigned)s.n_blocks, kFlagThreads, lay.total, stream>>>(*g, s.bitmap, s.block_count, s.per_block, lay);
  RSED_CHECK_LAUNCH();
  rc = rsed_exclusive_scan_i64(s.block_count, s.block_off, s.n_blocks, s.scan, s.scan_bytes, stream);
  if (rc) return rc;
  int64_t n_orb = 0;
  RSED_TRY_CUDA(cudaMemcpyAsync(&n_orb, s.block_off + s.n_blocks, sizeof(int64_t),
                                cudaMemcpyDeviceToHost, stream));
  RSED_TRY_CUDA(cudaStreamSynchronize(stream));
  RSED_REQUIRE(n_orb < (int64_t)INT32_MAX, RSED_ERANGE, "more than 2^31-1 orbits");
  *n_orbits_out = n_orb;
  return RSED_OK;
}

extern "C" int rsed_catalog_fill(const rsed_group_t* g, const void* scratch, size_t scratch_bytes,
                                 int64_t n_orbits, uint64_t* repr_masks, rsed_entry_t* table,
                                 uint64_t* stab_mask, void* stream_) {
  int rc = check_group(g);
  if (rc) return rc;
  RSED_REQUIRE(scratch_bytes >= rsed_catalog_scratch_bytes(g), RSED_ESCRATCH,
               "catalog scratch too small");
  RSED_REQUIRE(g->angle != nullptr && g->eta != nullptr, RSED_EINVAL, "group phases missing");
  RSED_REQUIRE(n_orbits >= 1 && repr_masks && table && stab_mask, RSED_EINVAL,
               "catalog outputs missing");
  cudaStream_t stream = as_stream(stream_);
  CatalogScratch s = carve_catalog_scratch(g, const_cast<void*>(scratch));
  GroupSmemLayout lay0 = group_smem_layout(g->n_site, g->n_filled, g->n_group, false, false);
  k_rep_list<<<(unsigned)s.n_blocks, kFlagThreads, lay0.total, stream>>>(
      *g, s.bitmap, s.block_off, s.per_block, repr_masks, reinterpret_cast<RsedEntry*>(table), lay0);
  RSED_CHECK_LAUNCH();
  GroupSmemLayout lay = group_smem_layout(g->n_site, g->n_filled, g->n_group, true, true);
  int* err = reinterpret_cast<int*>(s.block_count);  // block counts are consumed by now
  RSED_TRY_CUDA(cudaMemsetAsync(err, 0, sizeof(int), stream));
  const int per_block = 256 / g->n_group;
  const int64_t steps = (n_orbits + per_block - 1) / per_block;
  // one wave of blocks walks the orbits: the tables are staged once per block
  // (one step per block measured 20 us slower on 657,756 orbits)
  auto expand = g->n_site > 32 ? k_expand<uint64_t, int64_t> : k_expand<uint32_t, int32_t>;
  int64_t wave = 0;
  rc = blocks_of_one_wave((const void*)expand, 256, lay.total, &wave);
  if (rc) return rc;
  expand<<<(unsigned)(steps < wave ? steps : wave), 256, lay.total, stream>>>(
      *g, n_orbits, repr_masks, reinterpret_cast<RsedEntry*>(table), stab_mask, lay, err);
  RSED_CHECK_LAUNCH();
  int herr = 0;
  RSED_TRY_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, stream));
  RSED_TRY_CUDA(cudaStreamSynchronize(stream));
  RSED_REQUIRE(herr == 0, RSED_EINVAL, "catalog expansion produced an out-of-range rank");
  return RSED_OK;
}

extern "C" size_t rsed_stab_scratch_bytes(int64_t n_orbits) {
  return align_up(sizeof(int64_t) * (size_t)(n_orbits + 1), 256) + rsed_scan_scratch_bytes(n_orbits);
}

extern "C" int rsed_catalog_stab_count(int64_t n_orbits, const uint64_t* stab_mask, int64_t* stab_off,
                                       int64_t* n_stab_out, void* scratch, size_t scratch_bytes,
                                       void* stream_) {
  RSED_REQUIRE(n_orbits >= 1 && stab_mask && stab_off && n_stab_out, RSED_EINVAL,
               "bad stabilizer-count arguments");
  RSED_REQUIRE(scratch_bytes >= rsed_stab_scratch_bytes(n_orbits), RSED_ESCRATCH,
               "stabilizer scratch too small");
  cudaStream_t stream = as_stream(stream_);
  int64_t* counts = reinterpret_cast<int64_t*>(scratch);
  char* scan = reinterpret_cast<char*>(scratch) + align_up(sizeof(int64_t) * (size_t)(n_orbits + 1), 256);
  k_stab_counts<<<(unsigned)((n_orbits + 255) / 256), 256, 0, stream>>>(n_orbits, stab_mask, counts);
  RSED_CHECK_LAUNCH();
  int rc = rsed_exclusive_scan_i64(counts, stab_off, n_orbits, scan, rsed_scan_scratch_bytes(n_orbits),
                                   stream);
  if (rc) return rc;
  RSED_TRY_CUDA(cudaMemcpyAsync(n_stab_out, stab_off + n_orbits, sizeof(int64_t),
                                cudaMemcpyDeviceToHost, stream));
  RSED_TRY_CUDA(cudaStreamSynchronize(stream));
  return RSED_OK;
}

extern "C" int rsed_catalog_stab(const rsed_group_t* g, int64_t n_orbits, const uint64_t* repr_masks,
                                 const uint64_t* stab_mask, const int64_t* stab_off,
                                 double* stab_phase, void* stream_) {
  int rc = check_group(g);
  if (rc) return rc;
  RSED_REQUIRE(g->angle != nullptr && g->eta != nullptr, RSED_EINVAL, "group phases missing");
  RSED_REQUIRE(n_orbits >= 1 && repr_masks && stab_mask && stab_off && stab_phase, RSED_EINVAL,
               "bad stabilizer arguments");
  cudaStream_t stream = as_stream(stream_);
  rc = set_catalog_smem_limits();
  if (rc) return rc;
  GroupSmemLayout lay = group_smem_layout(g->n_site, g->n_filled, g->n_group, true, true);
  k_stab_phases<<<(unsigned)((n_orbits + 255) / 256), 256, lay.total, stream>>>(
      *g, n_orbits, repr_masks, stab_mask, stab_off, reinterpret_cast<double2*>(stab_phase), lay);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

extern "C" int rsed_phase_update(const rsed_group_t* g, int64_t n_orbits, const uint64_t* repr_masks,
                                 const uint64_t* stab_mask, const int64_t* stab_off,
                                 double* stab_phase, rsed_entry_t* table, int* err_dev,
                                 void* stream_) {
  int rc = check_group(g);
  if (rc) return rc;
  RSED_REQUIRE(g->eta != nullptr, RSED_EINVAL, "group phases missing");
  RSED_REQUIRE(n_orbits >= 1 && repr_masks && stab_mask && stab_off && stab_phase && table && err_dev,
               RSED_EINVAL, "bad phase-update arguments");
  cudaStream_t stream = as_stream(stream_);
  rc = set_catalog_smem_limits();
  if (rc) return rc;
  GroupSmemLayout lay = group_smem_layout(g->n_site, g->n_filled, g->n_group, true, false);
  RSED_TRY_CUDA(cudaMemsetAsync(err_dev, 0, sizeof(int), stream));
  k_phase_stab<<<(unsigned)((n_orbits + 255) / 256), 256, lay.total, stream>>>(
      *g, n_orbits, repr_masks, stab_mask, stab_off, reinterpret_cast<double2*>(stab_phase), lay);
  RSED_CHECK_LAUNCH();
  auto kern = g->n_site > 32 ? k_phase_table<uint64_t, int64_t> : k_phase_table<uint32_t, int32_t>;
  int64_t wave = 0;
  rc = blocks_of_one_wave((const void*)kern, 256, lay.total, &wave);
  if (rc) return rc;
  const int64_t blocks = (g->n_states + 255) / 256;
  kern<<<(unsigned)(blocks < wave ? blocks : wave), 256, lay.total, stream>>>(*g, n_orbits, repr_masks,
                                                                            reinterpret_cast<int4*>(table), lay, err_dev);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

extern "C" size_t rsed_sector_scratch_bytes(int64_t n_orbits, int32_t n_sectors) {
  (void)n_sectors;
  return align_up(sizeof(int64_t) * (size_t)(n_orbits + 1), 256) * 2 +
         rsed_scan_scratch_bytes(n_orbits);
}

extern "C" int rsed_sector_members(int64_t n_orbits, int32_t n_group, int32_t n_sectors,
                                   const uint64_t* stab_mask, const int64_t* stab_off,
                                   const double* stab_phase, const double* chi, double atol,
                                   uint64_t* member, double* sqrt_stab, int64_t* sector_dims,
                                   void* stream_) {
  RSED_REQUIRE(n_orbits >= 1 && n_group >= 1 && n_group <= RSED_MAX_GROUP, RSED_EINVAL,
               "bad sector arguments");
  RSED_REQUIRE(n_sectors >= 1 && n_sectors <= 64, RSED_ERANGE, "n_sectors = %d outside [1, 64]",
               n_sectors);
  RSED_REQUIRE(stab_mask && stab_off && stab_phase && chi && member && sqrt_stab && sector_dims,
               RSED_EINVAL, "sector buffers missing");
  cudaStream_t stream = as_stream(stream_);
  int rc = set_catalog_smem_limits();
  if (rc) return rc;
  RSED_TRY_CUDA(cudaMemsetAsync(sector_dims, 0, sizeof(int64_t) * n_sectors, stream));
  size_t smem = sizeof(double2) * (size_t)n_sectors * n_group;
  k_sector_members<<<(unsigned)((n_orbits + 255) / 256), 256, smem, stream>>>(
      n_orbits, n_group, n_sectors, stab_mask, stab_off, reinterpret_cast<const double2*>(stab_phase),
      reinterpret_cast<const double2*>(chi), atol, member, sqrt_stab,
      reinterpret_cast<unsigned long long*>(sector_dims));
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

extern "C" int rsed_sector_rows(int64_t n_orbits, const uint64_t* member, int32_t sector,
                                int32_t* orbit_of_row, int32_t* row_of_orbit, void* scratch,
                                size_t scratch_bytes, void* stream_) {
  RSED_REQUIRE(n_orbits >= 1 && member && sector >= 0 && sector < 64, RSED_EINVAL,
               "bad sector-rows arguments");
  RSED_REQUIRE(scratch_bytes >= rsed_sector_scratch_bytes(n_orbits, 1), RSED_ESCRATCH,
               "sector scratch too small");
  cudaStream_t stream = as_stream(stream_);
  char* p = reinterpret_cast<char*>(scratch);
  size_t a = align_up(sizeof(int64_t) * (size_t)(n_orbits + 1), 256);
  int64_t* flags = reinterpret_cast<int64_t*>(p);
  int64_t* pos = reinterpret_cast<int64_t*>(p + a);
  const unsigned nb = (unsigned)((n_orbits + 255) / 256);
  k_member_bit<<<nb, 256, 0, stream>>>(n_orbits, member, sector, flags);
  RSED_CHECK_LAUNCH();
  int rc = rsed_exclusive_scan_i64(flags, pos, n_orbits, p + 2 * a, rsed_scan_scratch_bytes(n_orbits),
                                   stream);
  if (rc) return rc;
  k_sector_rows<<<nb, 256, 0, stream>>>(n_orbits, member, sector, pos, orbit_of_row, row_of_orbit);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

extern "C" int rsed_density_diag(int64_t n_orbits, const uint64_t* repr_masks, int32_t n_density,
                                 const uint8_t* dens_i, const uint8_t* dens_j, const double* dens_v,
                                 double* hdiag, void* stream_) {
  RSED_REQUIRE(n_orbits >= 1 && repr_masks && hdiag && n_density >= 0, RSED_EINVAL,
               "bad density arguments");
  RSED_REQUIRE(n_density == 0 || (dens_i && dens_j && dens_v), RSED_EINVAL, "density terms missing");
  cudaStream_t stream = as_stream(stream_);
  k_density_diag<<<(unsigned)((n_orbits + 255) / 256), 256, 0, stream>>>(
      n_orbits, repr_masks, n_density, dens_i, dens_j, reinterpret_cast<const double2*>(dens_v),
      reinterpret_cast<double2*>(hdiag));
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

// ---- sector rows without device allocation ----------------------------------
// rsed_sector_rows_noalloc: the same result as rsed_sector_rows, for callers
// that cannot hand the library a scratch buffer.  Its only scratch is the
// per-tile sums of the scan, held in this file-scope device array (one copy
// on every GPU that loads the library, kept until the process exits).  The
// member bit is re-derived from `member` in both passes instead of being
// stored, so no buffer proportional to n_orbits is needed.
namespace {

constexpr int64_t kNoAllocMaxTiles = 16384;  // 16384 tiles x 8192 orbits = 2^27 orbits
constexpr int64_t kNoAllocMaxOrbits = kNoAllocMaxTiles * kScanTile;

// tile sums (kNoAllocMaxTiles) followed by the total
static __device__ __align__(256) int64_t g_rows_scan_scratch[kNoAllocMaxTiles + 1];

__global__ void k_nb_tile_counts(int64_t n, const uint64_t* member, int sector, int64_t* tile_sum) {
  __shared__ int64_t tot;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t c = 0;
  for (int j = 0; j < kScanItems; ++j) {
    const int64_t i = base + j;
    if (i < n) c += (member[i] >> sector) & 1ull;
  }
  block_exclusive_scan(c, &tot);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

__global__ void k_nb_tile_rows(int64_t n, const uint64_t* member, int sector, const int64_t* tile_off,
                               int32_t* orbit_of_row, int32_t* row_of_orbit) {
  __shared__ int64_t tot;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int flag[kScanItems];
  int64_t c = 0;
  for (int j = 0; j < kScanItems; ++j) {
    const int64_t i = base + j;
    flag[j] = (i < n) ? (int)((member[i] >> sector) & 1ull) : 0;
    c += flag[j];
  }
  int64_t pos = block_exclusive_scan(c, &tot) + tile_off[blockIdx.x];
  for (int j = 0; j < kScanItems; ++j) {
    const int64_t i = base + j;
    if (i >= n) break;
    if (flag[j]) {
      if (orbit_of_row) orbit_of_row[pos] = (int32_t)i;
      if (row_of_orbit) row_of_orbit[i] = (int32_t)pos;
      ++pos;
    } else if (row_of_orbit) {
      row_of_orbit[i] = -1;
    }
  }
}

// Device address of the scratch array, looked up once per device.
std::mutex g_noalloc_mu;
int64_t* g_noalloc_ptr[64] = {nullptr};

int noalloc_scratch(int64_t** out) {
  int dev = -1;
  RSED_TRY_CUDA(cudaGetDevice(&dev));
  RSED_REQUIRE(dev >= 0 && dev < 64, RSED_ERANGE, "device ordinal %d outside [0, 64)", dev);
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    RSED_TRY_CUDA(cudaGetSymbolAddress(&p, g_rows_scan_scratch));
    g_noalloc_ptr[dev] = reinterpret_cast<int64_t*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return RSED_OK;
}

}  // namespace

extern "C" int rsed_sector_rows_noalloc(int64_t n_orbits, const uint64_t* member, int32_t sector,
                                        int32_t* orbit_of_row, int32_t* row_of_orbit, void* stream_) {
  RSED_REQUIRE(n_orbits >= 1 && member && sector >= 0 && sector < 64, RSED_EINVAL,
               "bad sector-rows arguments");
  RSED_REQUIRE(orbit_of_row || row_of_orbit, RSED_EINVAL, "no output buffer");
  RSED_REQUIRE(n_orbits <= kNoAllocMaxOrbits, RSED_ERANGE,
               "rsed_sector_rows_noalloc handles at most %lld orbits (got %lld); "
               "use rsed_sector_rows with a caller-owned scratch buffer",
               (long long)kNoAllocMaxOrbits, (long long)n_orbits);
  int64_t* scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  cudaStream_t stream = as_stream(stream_);
  const int64_t tiles = (n_orbits + kScanTile - 1) / kScanTile;
  int64_t* tile_sum = scratch;
  int64_t* total = scratch + kNoAllocMaxTiles;
  // every tile sum and the total are rewritten below, so the contents left
  // by an earlier call need no clearing
  k_nb_tile_counts<<<(unsigned)tiles, kScanThreads, 0, stream>>>(n_orbits, member, sector, tile_sum);
  RSED_CHECK_LAUNCH();
  k_scan_tiles<<<1, kScanThreads, 0, stream>>>(tile_sum, tiles, total);
  RSED_CHECK_LAUNCH();
  k_nb_tile_rows<<<(unsigned)tiles, kScanThreads, 0, stream>>>(n_orbits, member, sector, tile_sum,
                                                               orbit_of_row, row_of_orbit);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}

extern "C" int64_t rsed_sector_rows_noalloc_max_orbits(void) { return kNoAllocMaxOrbits; }
