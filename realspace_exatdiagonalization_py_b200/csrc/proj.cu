// K6b: orbit-space projection table and its streaming SpMV.
//
// The on-the-fly apply (apply.cu) re-derives every hop on every call: gate
// test, combinadic rank, a random 16-B gather from the C(N,k)-sized table.
// Across the ~100 matvecs of one eigen-solve those hops never change, so this
// file builds them once per catalog state into a CSR over orbit rows whose
// entries carry only what does not depend on the sector:
//   cg = c | g << 26   (target orbit, group element)
//   w  = conj(t * s_JW * alpha) * sqrt(S_c) / sqrt(S_r)
// A matvec then streams the table from HBM once per column chunk and gathers
// x[c][chunk] rows; chunks are sized by the caller so that x[:, chunk] stays
// resident in L2 while the table streams past it.
#include <type_traits>
#include "rsed_internal.cuh"
#include "rsed_apply.cuh"

using namespace rsed_apply;

namespace {

constexpr int kOrbitBits = 26;
constexpr uint32_t kOrbitMask = (1u << kOrbitBits) - 1u;

// Hops of row r in the order of the on-the-fly apply: occupied source site
// ascending, then the terms of that site in order, skipping occupied targets.
__global__ void __launch_bounds__(256) k_proj_count(rsed_model_t md, int64_t* counts, ApplySmemLayout lay) {
  extern __shared__ __align__(16) unsigned char smem[];
  rsed_sectors_t none{};
  ApplyView v = stage_apply(md, none, lay, smem);
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= md.n_orbits) return;
  const uint64_t m = md.repr_masks[r];
  int64_t n = 0;
  uint64_t occ = m;
  while (occ) {
    const int i = __ffsll((long long)occ) - 1;
    occ &= occ - 1;
    for (int t = v.tbeg[i]; t < v.tbeg[i + 1]; ++t) n += ((m >> v.tto[t]) & 1ull) ? 0 : 1;
  }
  counts[r] = n;
}

// Table entries are gathered HB hops at a time so each thread keeps several
// random 16-B loads in flight.
template <int HB>
__global__ void __launch_bounds__(256) k_proj_fill(rsed_model_t md, const double* __restrict__ sqrt_stab,
                                                   const int64_t* __restrict__ rowptr, uint32_t* __restrict__ cg,
                                                   double2* __restrict__ w64, float2* __restrict__ w32,
                                                   ApplySmemLayout lay) {
  extern __shared__ __align__(16) unsigned char smem[];
  rsed_sectors_t none{};
  ApplyView v = stage_apply(md, none, lay, smem);
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= md.n_orbits) return;
  const int kp1 = md.n_filled + 1;
  const int64_t cbs = md.species_b ? v.binom[__popcll(md.species_b) * kp1 + md.n_filled_b] : 1;
  const uint64_t m = md.repr_masks[r];
  const double sr = sqrt_stab[r];
  int64_t pos = rowptr[r];
  int bt[HB];
  int64_t bidx[HB];
  int nh = 0;
  auto flush = [&](int cnt) {
    RsedEntry e[HB];
#pragma unroll
    for (int h = 0; h < HB; ++h)
      if (h < cnt) e[h] = load_entry(reinterpret_cast<const RsedEntry*>(md.table), bidx[h]);
    double sq[HB];
#pragma unroll
    for (int h = 0; h < HB; ++h)
      if (h < cnt) sq[h] = __ldg(sqrt_stab + e[h].rep);
#pragma unroll
    for (int h = 0; h < HB; ++h) {
      if (h >= cnt) continue;
      const int t = bt[h];
      double2 ta = cmul(v.tamp[t], make_double2(e[h].re, e[h].im));
      if (md.fermionic && (__popcll(m & v.tjw[t]) & 1)) {
        ta.x = -ta.x;
        ta.y = -ta.y;
      }
      const double ratio = sq[h] / sr;
      const double2 w = make_double2(ta.x * ratio, -ta.y * ratio);
      if (cg) cg[pos] = (uint32_t)e[h].rep | ((uint32_t)e[h].g << kOrbitBits);
      if (w64) w64[pos] = w;
      if (w32) w32[pos] = make_float2((float)w.x, (float)w.y);
      ++pos;
    }
  };
  uint64_t occ = m;
  while (occ) {
    const int i = __ffsll((long long)occ) - 1;
    occ &= occ - 1;
    for (int t = v.tbeg[i]; t < v.tbeg[i + 1]; ++t) {
      const int jj = v.tto[t];
      if ((m >> jj) & 1ull) continue;
      bt[nh] = t;
      bidx[nh] = rsed_rank_any(m ^ (1ull << i) ^ (1ull << jj), v.binom, kp1, md.species_b, cbs);
      if (++nh == HB) {
        flush(HB);
        nh = 0;
      }
    }
  }
  if (nh) flush(nh);
}

// ---- streaming SpMV --------------------------------------------------------
// One warp per orbit row (grid-stride).  The warp's lanes form EPW = 32/L
// entry slots of L lanes; the L lanes of a slot cover the NC = L*CPL columns
// of the chunk, CPL contiguous columns each (one 16-B gather per lane and
// hop).  Entry slots walk the row's hops EPW at a time, U hops per batch
// (all U table entries, then all U x rows, then the arithmetic), and are
// summed with xor-shuffles at the end of the row.
template <int PREC>
struct ProjTypes;
template <>
struct ProjTypes<64> {
  using W = double2;
  using Real = double;
};
template <>
struct ProjTypes<32> {
  using W = float2;
  using Real = float;
};

// CPL contiguous columns of one x row, loaded as 16-B vectors (two FP32 or one
// FP64 complex value each); vectors at or beyond the row's leading dimension
// read as zero, so a lane's segment never leaves its row.
template <int PREC, int CPL>
struct XVec {
  using W = typename ProjTypes<PREC>::W;
  static constexpr int kPer = (PREC == 64) ? 1 : 2;  // columns per 16-B vector
  static constexpr int kVec = CPL / kPer;
  W v[CPL];
  __device__ __forceinline__ void load(const char* base, int avail) {
#pragma unroll
    for (int k = 0; k < kVec; ++k) {
      if (k * kPer < avail) {
        if constexpr (PREC == 64) {
          v[k] = __ldg(reinterpret_cast<const double2*>(base) + k);
        } else {
          const float4 q = __ldg(reinterpret_cast<const float4*>(base) + k);
          v[2 * k] = make_float2(q.x, q.y);
          v[2 * k + 1] = make_float2(q.z, q.w);
        }
      } else {
#pragma unroll
        for (int j = 0; j < kPer; ++j) v[k * kPer + j].x = v[k * kPer + j].y = 0;
      }
    }
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int j = 0; j < CPL; ++j) v[j].x = v[j].y = 0;
  }
};

template <typename T>
__device__ __forceinline__ T ld_stream(const T* p) {
  return __ldcs(p);
}

// A lane's 32-B segment of an x row (4 FP32 or 2 FP64 complex values) in one
// 256-bit load.
__device__ __forceinline__ void load_segment(const char* p, float2 (&v)[4]) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y), "=f"(v[3].x), "=f"(v[3].y)
      : "l"(p));
}
__device__ __forceinline__ void load_segment(const char* p, double2 (&v)[2]) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(v[0].x), "=d"(v[0].y), "=d"(v[1].x), "=d"(v[1].y)
      : "l"(p));
}

// The rows r0, r0 + step, ... of lanes whose 32-B segments hold pairs of columns
// of one sector each (blocks of 2 or 4: FP32 two pairs, FP64 one), as long as
// they belong to every sector of the warp (`need`); returns the first row that
// does not (the caller takes it column by column and comes back) or one past
// the end.
//
// The loop is bound by instruction issue and load latency as much as by the
// gathers (with every target in one L1-sized window the FP32 form ran only 13 %
// faster), so it is written for few instructions: entries at constant offsets
// from per-lane pointers, a lane's characters in one shared-memory word
// chp[g*L], one weight-character product per pair, no per-column tests, missing
// entries past the row's end as (the row itself, weight 0) -- its x is read for
// the diagonal anyway, so a non-finite value spreads no further than H takes it --
// and the slots' sums combined by halving exchanges, so that every lane finishes
// its share of the row.  The entries of the next batch -- of
// this row or the next one, whose offsets are loaded a row ahead -- are fetched
// while the current batch gathers.  U = 2 hops per lane and batch at 4 blocks
// per SM: more warps hide the gathers better than deeper batches.
// 36.7 million hops, 32 columns: FP32 1228 us in the per-row form with U = 4 at
// 3 blocks per SM, 1103 us as here with U = 4, 1017 us with U = 2 (U = 3 at 3
// blocks: 1035; U = 2 at 5 blocks spills: 1528); FP64 2637 us with per-column
// tests, 2051 us in this form.
template <int PREC, int L, int U>
__device__ __forceinline__ int64_t spmv_rows_pairs(const rsed_model_t& md, const rsed_sectors_t& sc, int64_t r0,
                                                   int64_t step, uint64_t need, int c0, bool live,
                                                   const char* __restrict__ xl,
                                                   const typename ProjTypes<PREC>::W* chp,
                                                   const typename ProjTypes<PREC>::W* __restrict__ x,
                                                   double2* __restrict__ y) {
  using W = typename ProjTypes<PREC>::W;
  using Real = typename ProjTypes<PREC>::Real;
  constexpr int CPL = PREC == 32 ? 4 : 2;    // columns of a lane
  constexpr int EPW = 32 / L;
  constexpr int B = EPW * U;                 // hops per batch and warp
  const int lane = threadIdx.x & 31, eslot = lane / L;
  const uint32_t* __restrict__ cgt = md.proj_cg + eslot;
  const W* __restrict__ wt =
      reinterpret_cast<const W*>(PREC == 64 ? (const void*)md.proj_w64 : (const void*)md.proj_w32) + eslot;
  const int64_t* __restrict__ rp = md.proj_rowptr;
  const uint32_t rowb = (uint32_t)(sc.ld * sizeof(W));
  if (r0 >= md.n_orbits || (sc.member[r0] & need) != need) return r0;
  int64_t e0 = rp[r0];
  int left = (int)(rp[r0 + 1] - e0);
  uint32_t cgn[U];
  W wn[U];
  auto fetch = [&](int64_t row, int64_t e, int n) {  // the batch at e, n entries of its row left
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool ok = u * EPW + eslot < n;
      cgn[u] = ok ? ld_stream(cgt + e + u * EPW) : (uint32_t)row;
      if (ok) {
        wn[u] = ld_stream(wt + e + u * EPW);
      } else {
        wn[u].x = 0;
        wn[u].y = 0;
      }
    }
  };
  fetch(r0, e0, left);
  for (int64_t r = r0;;) {
    const int64_t rn = r + step;
    const bool more = rn < md.n_orbits;
    const uint64_t memn = more ? __ldg(sc.member + rn) : 0ull;
    const int64_t en = more ? __ldg(rp + rn) : 0;
    const int leftn = more ? (int)(__ldg(rp + rn + 1) - en) : 0;
    W a[CPL];
#pragma unroll
    for (int j = 0; j < CPL; ++j) a[j].x = a[j].y = 0;
    do {
      uint32_t cgc[U];
      W wc[U], xs[U][CPL];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        cgc[u] = cgn[u];
        wc[u] = wn[u];
        load_segment(xl + (uint64_t)(cgc[u] & kOrbitMask) * rowb, xs[u]);
      }
      e0 += B;
      left -= B;
      if (left > 0)
        fetch(r, e0, left);
      else
        fetch(rn, en, leftn);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const W* ch = chp + (cgc[u] >> kOrbitBits) * (L * CPL / 2);
#pragma unroll
        for (int h = 0; h < CPL / 2; ++h) {
          const W k = ch[h], w = wc[u];
          const Real px = w.x * k.x - w.y * k.y, py = w.x * k.y + w.y * k.x;
#pragma unroll
          for (int j = 2 * h; j < 2 * h + 2; ++j) {
            a[j].x += px * xs[u][j].x - py * xs[u][j].y;
            a[j].y += px * xs[u][j].y + py * xs[u][j].x;
          }
        }
      }
    } while (left > 0);
    // the slots' sums: halve the columns while there are two, then plain exchanges
    constexpr int H1 = EPW >= 2, H2 = PREC == 32 && EPW >= 4;
    if constexpr (H1) {
      const bool up = lane & 16;
#pragma unroll
      for (int j = 0; j < CPL / 2; ++j) {
        const W lo = a[j], hi = a[j + CPL / 2];
        a[j].x = (up ? hi.x : lo.x) + __shfl_xor_sync(0xffffffffu, up ? lo.x : hi.x, 16);
        a[j].y = (up ? hi.y : lo.y) + __shfl_xor_sync(0xffffffffu, up ? lo.y : hi.y, 16);
      }
    }
    if constexpr (H2) {
      const bool up = lane & 8;
      const W lo = a[0], hi = a[1];
      a[0].x = (up ? hi.x : lo.x) + __shfl_xor_sync(0xffffffffu, up ? lo.x : hi.x, 8);
      a[0].y = (up ? hi.y : lo.y) + __shfl_xor_sync(0xffffffffu, up ? lo.y : hi.y, 8);
    }
    constexpr int OWN = CPL >> (H1 + H2);        // columns a lane finishes
    constexpr int REST = 32 >> (H1 + H2);        // lanes that hold the same columns' parts
#pragma unroll
    for (int off = REST / 2; off >= L; off >>= 1) {
#pragma unroll
      for (int j = 0; j < OWN; ++j) {
        a[j].x += __shfl_xor_sync(0xffffffffu, a[j].x, off);
        a[j].y += __shfl_xor_sync(0xffffffffu, a[j].y, off);
      }
    }
    const int col = c0 + (H1 ? (lane >> 4 & 1) * (CPL / 2) : 0) + (H2 ? (lane >> 3 & 1) : 0);
    if (live && (lane & (REST - 1)) < L) {
      const double2 hd = __ldg(reinterpret_cast<const double2*>(md.hdiag) + r);
      const int64_t at = r * sc.ld + col;
#pragma unroll
      for (int j = 0; j < OWN; ++j) {
        const W xr = __ldg(x + at + j);
        const double xx = (double)xr.x, xy = (double)xr.y;
        y[at + j] = make_double2((double)a[j].x + (hd.x * xx + hd.y * xy), (double)a[j].y + (hd.x * xy - hd.y * xx));
      }
    }
    if (!more || (memn & need) != need) return rn;
    r = rn;
    e0 = en;
    left = leftn;
  }
}

// Byte offset of the pair table behind a character table of `bytes`.
__host__ __device__ constexpr size_t pair_table_offset(size_t bytes) { return (bytes + 15) & ~(size_t)15; }

// Whether a lane's segment is 32 B: the form with the pair loop.
template <int PREC, int CPL>
constexpr bool kWide = CPL * (PREC == 32 ? 8 : 16) == 32;

template <int PREC, int L, int CPL, int U>
__global__ void __launch_bounds__(256, kWide<PREC, CPL> ? 4 : 3) k_proj_spmv(rsed_model_t md, rsed_sectors_t sc, const void* __restrict__ xin,
                                                   double2* __restrict__ y, int chunk0, int guard) {
  if (guard) {  // run only if the columns are (1) or are not (2) pairs of one sector each
    bool same = true;
    for (int c = 2 * (int)threadIdx.x; c < sc.n_cols; c += 2 * (int)blockDim.x)
      same = same && c + 1 < sc.n_cols && sc.col_sector[c] == sc.col_sector[c + 1];
    if ((__syncthreads_and(same) != 0) != (guard == 1)) return;
  }
  using W = typename ProjTypes<PREC>::W;
  using Real = typename ProjTypes<PREC>::Real;
  constexpr int EPW = 32 / L;
  constexpr int NC = L * CPL;
  extern __shared__ __align__(16) unsigned char smem[];
  // characters transposed to [g][sector]: the L lanes of an entry slot share
  // g and read consecutive words
  W* chi = reinterpret_cast<W*>(smem);
  const double2* gchi = reinterpret_cast<const double2*>(sc.chi);
  const int nsec = sc.n_sectors;
  const int nchi = nsec * md.n_group;
  for (int i = threadIdx.x; i < nchi; i += blockDim.x) {
    const int s = i / md.n_group, g = i % md.n_group;
    const double2 c = gchi[i];
    chi[g * nsec + s].x = (Real)c.x;
    chi[g * nsec + s].y = (Real)c.y;
  }
  // the characters of a lane's sector pairs side by side, [g][lane of the slot][pair]
  W* chpair = reinterpret_cast<W*>(smem + pair_table_offset(sizeof(W) * (size_t)nchi));
  if constexpr (kWide<PREC, CPL>) {
    const int cfirst = (chunk0 + (int)blockIdx.y) * NC;
    for (int i = threadIdx.x; i < md.n_group * (NC / 2); i += blockDim.x) {
      const int g = i / (NC / 2), c = cfirst + i % (NC / 2) * 2;
      const double2 k = gchi[(c < sc.n_cols ? sc.col_sector[c] : 0) * md.n_group + g];
      chpair[i].x = (Real)k.x;
      chpair[i].y = (Real)k.y;
    }
  }
  __syncthreads();
  const W* __restrict__ wt = reinterpret_cast<const W*>(PREC == 64 ? (const void*)md.proj_w64
                                                                    : (const void*)md.proj_w32);
  const uint32_t* __restrict__ cgt = md.proj_cg;
  const int64_t* __restrict__ rp = md.proj_rowptr;
  const int lane = threadIdx.x & 31;
  const int eslot = lane / L;
  const int c0 = (chunk0 + (int)blockIdx.y) * NC + (lane % L) * CPL;
  const int64_t ld = sc.ld;
  const int avail = (int)ld - c0;
  int sec[CPL];
  bool colv[CPL], fresh[CPL];
#pragma unroll
  for (int j = 0; j < CPL; ++j) {
    colv[j] = c0 + j < sc.n_cols;
    sec[j] = colv[j] ? sc.col_sector[c0 + j] : -1;
    // the block vectors of one sector sit in adjacent columns, so a lane's
    // columns usually share the hop weight
    fresh[j] = (j == 0) || sec[j] != sec[j - 1];
  }
  const char* xb = reinterpret_cast<const char*>(xin) + (size_t)c0 * sizeof(W);
  // 32-B segments of sector pairs (blocks of 2 or 4 columns): the pair loop over
  // the rows that are in all of the warp's sectors.  Lanes past the last column
  // run it too, on column 0 of x (in bounds), and their sums are dropped.
  bool pairs = false;
  const char* xfast = xb;
  uint64_t need = 0;  // the sectors of the warp's columns
  if constexpr (kWide<PREC, CPL>) {
    // a lane's segment starts at a multiple of CPL columns: with ld a multiple of
    // CPL too (and x 32-B aligned) it is 32-B aligned for one 256-bit load
    bool lane_ok = !colv[0];
    if (colv[CPL - 1]) {
      lane_ok = true;
#pragma unroll
      for (int j = 0; j < CPL; j += 2) lane_ok = lane_ok && sec[j + 1] == sec[j];
    }
    pairs = __all_sync(0xffffffffu, lane_ok) && (ld % CPL) == 0 && (reinterpret_cast<uintptr_t>(xin) & 31) == 0;
    if (!colv[0]) xfast = reinterpret_cast<const char*>(xin);
    if (colv[0] && lane_ok)
#pragma unroll
      for (int j = 0; j < CPL; j += 2) need |= 1ull << sec[j];
    for (int o = 16; o > 0; o >>= 1) need |= __shfl_xor_sync(0xffffffffu, need, o);
  }
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < md.n_orbits; r += warps) {
    if constexpr (kWide<PREC, CPL>) {
      if (pairs) {
        r = spmv_rows_pairs<PREC, L, U>(md, sc, r, warps, need, c0, colv[0], xfast, chpair + lane % L * (CPL / 2),
                                        reinterpret_cast<const W*>(xin), y);
        if (r >= md.n_orbits) break;
      }
    }
    const uint64_t memr = sc.member[r];
    bool on[CPL];
    bool any = false;
#pragma unroll
    for (int j = 0; j < CPL; ++j) {
      on[j] = colv[j] && ((memr >> sec[j]) & 1ull);
      any |= on[j];
    }
    W acc[CPL];
#pragma unroll
    for (int j = 0; j < CPL; ++j) acc[j].x = acc[j].y = (Real)0;
    if (__any_sync(0xffffffffu, any)) {
      const int64_t e0 = rp[r], e1 = rp[r + 1];
      for (int64_t base = e0; base < e1; base += EPW * U) {
        uint32_t cgv[U];
        W wv[U];
        XVec<PREC, CPL> xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int64_t idx = base + u * EPW + eslot;
          if (idx < e1) {
            cgv[u] = ld_stream(cgt + idx);
            wv[u] = ld_stream(wt + idx);
          } else {
            cgv[u] = 0xffffffffu;
            wv[u].x = wv[u].y = (Real)0;
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (cgv[u] != 0xffffffffu && any)
            xv[u].load(xb + (size_t)(cgv[u] & kOrbitMask) * ld * sizeof(W), avail);
          else
            xv[u].zero();
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (cgv[u] == 0xffffffffu) continue;
          const W* chg = chi + (int)(cgv[u] >> kOrbitBits) * nsec;
          Real wcx = 0, wcy = 0;
#pragma unroll
          for (int j = 0; j < CPL; ++j) {
            if (!on[j]) continue;
            if (fresh[j] || !on[j - (j > 0)]) {
              const W ch = chg[sec[j]];
              wcx = wv[u].x * ch.x - wv[u].y * ch.y;
              wcy = wv[u].x * ch.y + wv[u].y * ch.x;
            }
            const W xx = xv[u].v[j];
            acc[j].x += wcx * xx.x - wcy * xx.y;
            acc[j].y += wcx * xx.y + wcy * xx.x;
          }
        }
      }
    }
#pragma unroll
    for (int off = L; off < 32; off <<= 1) {
#pragma unroll
      for (int j = 0; j < CPL; ++j) {
        acc[j].x += __shfl_xor_sync(0xffffffffu, acc[j].x, off);
        acc[j].y += __shfl_xor_sync(0xffffffffu, acc[j].y, off);
      }
    }
    if (eslot == 0) {
      const double2 hd = reinterpret_cast<const double2*>(md.hdiag)[r];
#pragma unroll
      for (int j = 0; j < CPL; ++j) {
        if (!colv[j]) continue;
        double2 o = make_double2(0.0, 0.0);
        if (on[j]) {
          const W xr = reinterpret_cast<const W*>(xin)[r * ld + c0 + j];
          const double xx = (double)xr.x, xy = (double)xr.y;
          o.x = (double)acc[j].x + (hd.x * xx + hd.y * xy);
          o.y = (double)acc[j].y + (hd.x * xy - hd.y * xx);
        }
        y[r * ld + c0 + j] = o;
      }
    }
  }
}

template <int PREC, int L, int CPL>
int launch_spmv(const rsed_model_t& md, const rsed_sectors_t& sc, const void* x, double2* y, bool sequential,
                int guard, cudaStream_t stream) {
  using W = typename ProjTypes<PREC>::W;
  constexpr int U = kWide<PREC, CPL> ? 2 : 4;
  constexpr int NC = L * CPL;
  auto kern = k_proj_spmv<PREC, L, CPL, U>;
  size_t smem = sizeof(W) * (size_t)sc.n_sectors * md.n_group;
  if (kWide<PREC, CPL>) smem = pair_table_offset(smem) + sizeof(W) * (size_t)md.n_group * (NC / 2);
  static int blocks_per_sm[16] = {0};  // per device, computed once
  int dev = 0;
  RSED_TRY_CUDA(cudaGetDevice(&dev));
  int& bps = blocks_per_sm[dev & 15];
  if (smem > 48 * 1024) {
    // the limit of every model, not this call's size: host threads share the attribute
    constexpr size_t chars = sizeof(W) * 64 * RSED_MAX_GROUP;
    constexpr size_t most = kWide<PREC, CPL> ? pair_table_offset(chars) + sizeof(W) * RSED_MAX_GROUP * (NC / 2) : chars;
    RSED_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
  }
  if (bps == 0) {
    RSED_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, 256, smem));
    if (bps < 1) bps = 1;
  }
  static int n_sm = 0;
  if (n_sm == 0) RSED_TRY_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  const int n_chunks = (sc.n_cols + NC - 1) / NC;
  const int64_t row_blocks = (md.n_orbits + 7) / 8;
  const int64_t gx = row_blocks < (int64_t)n_sm * bps ? row_blocks : (int64_t)n_sm * bps;
  if (sequential) {
    for (int c = 0; c < n_chunks; ++c) {
      kern<<<dim3((unsigned)gx, 1), 256, smem, stream>>>(md, sc, x, y, c, guard);
      RSED_CHECK_LAUNCH();
    }
  } else {
    kern<<<dim3((unsigned)gx, (unsigned)n_chunks), 256, smem, stream>>>(md, sc, x, y, 0, guard);
    RSED_CHECK_LAUNCH();
  }
  return RSED_OK;
}

int check_proj_model(const rsed_model_t* md) {
  RSED_REQUIRE(md != nullptr, RSED_EINVAL, "model descriptor is NULL");
  RSED_REQUIRE(md->n_site >= 1 && md->n_site <= RSED_MAX_SITES, RSED_ERANGE, "bad n_site");
  RSED_REQUIRE(md->n_group >= 1 && md->n_group <= RSED_MAX_GROUP, RSED_ERANGE, "bad |G|");
  RSED_REQUIRE(md->n_orbits >= 1 && md->table && md->repr_masks && md->binom && md->hdiag, RSED_EINVAL,
               "model tables missing");
  RSED_REQUIRE(md->n_terms >= 0 && md->term_begin, RSED_EINVAL, "terms missing");
  RSED_REQUIRE(md->n_orbits <= (int64_t)kOrbitMask, RSED_ERANGE,
               "projection table holds at most 2^26 - 1 orbits");
  return RSED_OK;
}

int launch_variant(const rsed_model_t& md, const rsed_sectors_t& sc, const void* x, double2* y, int precision,
                   int variant, int guard, cudaStream_t stream) {
  const int family = variant / 100;  // 3/4: 16-B segment per lane, 5/6: 32-B segment
  const bool seq = family == 3 || family == 5;
  const bool wide = family >= 5;
  const int nc = variant % 100 + (variant % 100 == 28 ? 100 : 0);  // 528 / 628 = 128 columns
  if (family >= 3 && family <= 6) {
    if (precision == 64) {
      if (!wide) {
        switch (nc) {
          case 2: return launch_spmv<64, 2, 1>(md, sc, x, y, seq, guard, stream);
          case 4: return launch_spmv<64, 4, 1>(md, sc, x, y, seq, guard, stream);
          case 8: return launch_spmv<64, 8, 1>(md, sc, x, y, seq, guard, stream);
          case 16: return launch_spmv<64, 16, 1>(md, sc, x, y, seq, guard, stream);
          case 32: return launch_spmv<64, 32, 1>(md, sc, x, y, seq, guard, stream);
          default: break;
        }
      } else {
        switch (nc) {
          case 4: return launch_spmv<64, 2, 2>(md, sc, x, y, seq, guard, stream);
          case 8: return launch_spmv<64, 4, 2>(md, sc, x, y, seq, guard, stream);
          case 16: return launch_spmv<64, 8, 2>(md, sc, x, y, seq, guard, stream);
          case 32: return launch_spmv<64, 16, 2>(md, sc, x, y, seq, guard, stream);
          case 64: return launch_spmv<64, 32, 2>(md, sc, x, y, seq, guard, stream);
          default: break;
        }
      }
    } else {
      if (!wide) {
        switch (nc) {
          case 4: return launch_spmv<32, 2, 2>(md, sc, x, y, seq, guard, stream);
          case 8: return launch_spmv<32, 4, 2>(md, sc, x, y, seq, guard, stream);
          case 16: return launch_spmv<32, 8, 2>(md, sc, x, y, seq, guard, stream);
          case 32: return launch_spmv<32, 16, 2>(md, sc, x, y, seq, guard, stream);
          case 64: return launch_spmv<32, 32, 2>(md, sc, x, y, seq, guard, stream);
          default: break;
        }
      } else {
        switch (nc) {
          case 8: return launch_spmv<32, 2, 4>(md, sc, x, y, seq, guard, stream);
          case 16: return launch_spmv<32, 4, 4>(md, sc, x, y, seq, guard, stream);
          case 32: return launch_spmv<32, 8, 4>(md, sc, x, y, seq, guard, stream);
          case 64: return launch_spmv<32, 16, 4>(md, sc, x, y, seq, guard, stream);
          case 128: return launch_spmv<32, 32, 4>(md, sc, x, y, seq, guard, stream);
          default: break;
        }
      }
    }
  }
  return rsed_set_error(RSED_EINVAL, "projection apply variant %d invalid at precision %d", variant, precision);
}

// Hops of a row on average: occupied sites times the terms of a site with an
// empty target.
double mean_hops(const rsed_model_t& md) {
  const double N = md.n_site, k = md.n_filled;
  return N > 1 ? md.n_terms * k * (N - k) / (N * (N - 1)) : 0.0;
}

// The variant for columns that do not pair up: 16-B segments, in the chunks that
// leave the fewest columns of the last one empty, the wider ones first (each chunk
// reads the table again and pays a row's fixed cost).  Rings, 13 hops a row, us:
//   112,720 orbits, 24 columns: chunks of 16 / 32 167 / 133 FP64, 125 / 98 FP32
//   400,024 orbits, 64 columns: 1248 / 961 FP64, chunks of 16 / 32 / 64 1059 / 750 / 605 FP32
//   657,756 orbits of 56 hops: 24 columns 2925 / 2890 FP64, 2140 / 1890 FP32
// 11,240 orbits of 56 hops lack the warps for it (24 columns: 55 / 57 FP64).  With a
// third of a chunk empty the table counts against the padding: FP32, 18 columns,
// chunks of 16 / 32: 56,742 orbits of 60 hops 178 / 183; 40 columns, chunks of 16 / 64: 291 / 288 with 25 hops a row, 383 / 412 with 37
// (112,720 orbits), 1147 / 1079 with 27 and 1501 / 1563 with 41 (400,024 orbits).
// Several FP64 chunks go one after another, so that a chunk of x stays in L2, only
// on the largest bases (48 columns: 657,756 orbits 4434 against 4750 in one
// launch, 400,024 orbits 1456 against 1430, 112,720 orbits 255 against 241).
int narrow_variant(const rsed_model_t& md, int n_cols, int precision) {
  const auto last = [&](int nc) { return (n_cols - 1) % nc + 1; };  // columns of the last chunk
  const bool few_hops = mean_hops(md) < 28.0;
  int nc = 2;
  while (nc < n_cols && nc < 16) nc *= 2;
  if (md.n_orbits >= (1 << 14) && n_cols > 16) {
    if (last(32) > (precision == 32 && !few_hops ? 21 : 16)) nc = 32;
    if (precision == 32 && n_cols > 32 && last(64) > (few_hops ? 32 : 48)) nc = 64;
  }
  if (precision == 32 || md.n_orbits < 65536) return 400 + (nc < 4 ? 4 : nc);
  return (md.n_orbits < (1 << 19) ? 400 : 300) + nc;
}

}  // namespace

// Called by rsed_apply_h for variants 0 (with a table present), 3NN-6NN.
// pairs: 1 = the caller knows that columns 2i and 2i + 1 share a sector, 0 = it
// knows that they do not, -1 = unknown.
int rsed_proj_apply(const rsed_model_t& md, const rsed_sectors_t& sc, const void* x, double2* y, int precision,
                    int variant, int pairs, cudaStream_t stream) {
  RSED_REQUIRE(md.proj_rowptr && md.proj_cg, RSED_EINVAL, "no projection table in the model");
  RSED_REQUIRE(precision == 64 ? md.proj_w64 != nullptr : md.proj_w32 != nullptr, RSED_EINVAL,
               "projection table has no weights for precision %d", precision);
  RSED_REQUIRE((sc.ld & 1) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0, RSED_EINVAL,
               "projection apply needs an even leading dimension and a 16-byte aligned x");
  if (variant != 0) return launch_variant(md, sc, x, y, precision, variant, 0, stream);
  // Pairs of columns of one sector run the pair loop on 32-B segments, one launch
  // of up to 64 columns per chunk (B200, us, against 16-B segments in chunks of 16;
  // 657,756 orbits: FP64 32 columns 2051 and 3009, 64 columns 4269 and 5931, 8
  // columns 671 and 838, FP32 32 columns 995 and 1892; 11,240 orbits, 24 columns:
  // FP64 31 and 40, FP32 22 and 27).  Few columns fill no 32-B segments of enough
  // lanes, which pays only where the gathers miss L2 (FP64 4 columns: 657,756
  // orbits 482 and 521, 112,720 orbits 52 and 47; 2 columns: 445 and 330; FP32 4
  // columns 385 and 367, 8 columns 415 and 580).  80 columns go in chunks of 32, not
  // of 64 (84,576 orbits: FP64 567 and 628, FP32 291 and 335).  A table of fewer than
  // 2^16 hops has too few rows or hops for it (48 columns, FP64: 892 orbits of 42
  // hops 17 and 8.6, 2,704 of 10 hops 10.2 and 8.2, 3,542 of 37 hops 16 and 21).
  // Other columns run best on 16-B segments (16 columns of 16 sectors: FP64 1470 and 1610, FP32 1062 and 1082; 48
  // columns, FP64 4470 and 6456), as do the smallest bases, which want the warps of
  // more chunks: see narrow_variant.  Where the caller does not know, a large basis
  // launches both forms and the kernel that does not fit the columns leaves at once:
  // 4 us, FP64 from 2^25 hops of all columns on (about 250 us; ring of 400,024
  // orbits, 12 columns: pairs 291 instead of 320 us, single columns 327 instead of
  // 323; ring of 112,720 orbits, 36 columns: pairs 173 instead of 240).
  const int cpl = precision == 64 ? 2 : 4;
  const bool fits = sc.ld % cpl == 0 && (reinterpret_cast<uintptr_t>(x) & 31) == 0 && sc.n_cols % 2 == 0;
  const int64_t elems = md.n_orbits * (int64_t)sc.n_cols;
  const bool small = md.n_orbits < 65536;
  const bool gains = precision == 32 ? sc.n_cols >= 8 : sc.n_cols > 16 || (sc.n_cols >= 4 && elems >= (1 << 21));
  int wide = precision == 64 ? 4 : 8;
  while (wide < sc.n_cols && wide < 64) wide *= 2;
  if (sc.n_cols > 64 && (sc.n_cols - 1) % 64 < 32) wide = 32;  // half of the last chunk empty
  wide += 600;
  const int narrow = narrow_variant(md, sc.n_cols, precision);
  if (!fits || !gains || pairs == 0 || md.n_orbits * mean_hops(md) < (1 << 16) ||
      (pairs < 0 && (small || (precision == 64 && elems * mean_hops(md) < (1 << 25)))))
    return launch_variant(md, sc, x, y, precision, narrow, 0, stream);
  const int rc = launch_variant(md, sc, x, y, precision, wide, pairs < 0 ? 1 : 0, stream);
  if (rc || pairs > 0) return rc;
  return launch_variant(md, sc, x, y, precision, narrow, 2, stream);
}

extern "C" size_t rsed_proj_scratch_bytes(int64_t n_orbits) {
  return align_up(sizeof(int64_t) * (size_t)(n_orbits + 1), 256) + rsed_scan_scratch_bytes(n_orbits);
}

extern "C" int rsed_proj_count(const rsed_model_t* md, int64_t* rowptr, int64_t* n_hops_out, void* scratch,
                               size_t scratch_bytes, void* stream_) {
  int rc = check_proj_model(md);
  if (rc) return rc;
  RSED_REQUIRE(rowptr && n_hops_out && scratch, RSED_EINVAL, "bad projection count arguments");
  RSED_REQUIRE(scratch_bytes >= rsed_proj_scratch_bytes(md->n_orbits), RSED_ESCRATCH,
               "projection scratch too small");
  cudaStream_t stream = as_stream(stream_);
  int64_t* counts = reinterpret_cast<int64_t*>(scratch);
  char* scan = reinterpret_cast<char*>(scratch) + align_up(sizeof(int64_t) * (size_t)(md->n_orbits + 1), 256);
  rsed_sectors_t none{};
  ApplySmemLayout lay = apply_layout(*md, none);
  RSED_REQUIRE(lay.total <= 48 * 1024, RSED_ERANGE, "term tables exceed 48 KB of shared memory");
  k_proj_count<<<(unsigned)((md->n_orbits + 255) / 256), 256, lay.total, stream>>>(*md, counts, lay);
  RSED_CHECK_LAUNCH();
  rc = rsed_exclusive_scan_i64(counts, rowptr, md->n_orbits, scan, rsed_scan_scratch_bytes(md->n_orbits),
                               stream);
  if (rc) return rc;
  RSED_TRY_CUDA(cudaMemcpyAsync(n_hops_out, rowptr + md->n_orbits, sizeof(int64_t), cudaMemcpyDeviceToHost,
                                stream));
  RSED_TRY_CUDA(cudaStreamSynchronize(stream));
  return RSED_OK;
}

extern "C" int rsed_proj_fill(const rsed_model_t* md, const double* sqrt_stab, const int64_t* rowptr,
                              uint32_t* cg, double* w64, float* w32, void* stream_) {
  int rc = check_proj_model(md);
  if (rc) return rc;
  RSED_REQUIRE(sqrt_stab && rowptr && (cg || w64 || w32), RSED_EINVAL, "bad projection fill arguments");
  cudaStream_t stream = as_stream(stream_);
  rsed_sectors_t none{};
  ApplySmemLayout lay = apply_layout(*md, none);
  RSED_REQUIRE(lay.total <= 48 * 1024, RSED_ERANGE, "term tables exceed 48 KB of shared memory");
  k_proj_fill<4><<<(unsigned)((md->n_orbits + 255) / 256), 256, lay.total, stream>>>(
      *md, sqrt_stab, rowptr, cg, reinterpret_cast<double2*>(w64), reinterpret_cast<float2*>(w32), lay);
  RSED_CHECK_LAUNCH();
  return RSED_OK;
}
