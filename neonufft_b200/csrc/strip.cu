// 1D and 2D ES spreading and interpolation on points sorted along narrow strips (method 1 with
// the automatic tile, BinGeom::strip).
//
// Replaces the reference's 1D / 2D spreading (src/neonufft/gpu/kernels/spreading_kernel.cu:477-715,
// one global float atomic per cell and point) and interpolation
// (src/neonufft/gpu/kernels/interpolation_kernel.cu).
//
// The points are sorted by (x strip of TX cells, row y), rows fastest (1D: by cell), and every
// record carries its absolute first cell, so any range of consecutive records can be worked on
// without looking its bin up: both kernels cut the sorted array into equal runs, whatever the
// distribution of the points, and need no work list.
//
// Spreading: a run is walked by RY = W lanes (a warp walks 32 / W runs side by side; with windows
// rounded up to 8 or 16 rows it walked 4 runs instead of 5 at w = 6, 2 instead of 3 at w = 10).
// Lane b holds in registers the strip's row y = b (mod RY) of a window of RY rows, P0 =
// TX + W - 1 cells as pairs of neighbours, and applies each point with packed FMAs: no lane
// touches another's row, so there are neither atomics nor shared-memory updates per cell. When
// the next point starts on a later row (or strip) the rows left behind are added to the grid,
// one 16-byte vector atomic per pair of cells in single precision. The RY points of a batch are
// staged in shared memory by one lane each: kx placed over the strip's cells and ky over the
// window, zero elsewhere, so that the register indices are fixed.
//
// 2D points that are sparse on average are added to the grid directly, but for the places where
// they crowd (spread_sparse_unit, spread_mixed_kernel). Bins may hold several cells (1D) or rows of a
// strip (2D, direct spreading and interpolation only) where rows would outnumber the points by far.
//
// Interpolation: one thread per point reads its W^d cells through the L1. Neighbouring threads
// hold neighbouring points, so a warp's load of one (dx, dy) falls on a few rows of one strip.
//
// The kernels that these replace as the default (spread.cu, interp.cu) give a warp to one point
// at a time with the region in shared memory and are bound by the chain of shared-memory accesses
// and shuffles from point to point. Measured, before -> now: 3e6 radial points on a 1554 x 1280
// grid, w = 6, single: spreading 579 -> 150 us, interpolation 901 -> 63 us; 5e6 points on 4e5
// cells in 1D, w = 10, double: 888 -> 155 us and 1476 -> 135 us. Interpolation is now bound by the
// L1 (83 % of its throughput), spreading by latency (40 % of the issue slots at 24 warps per SM).
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "packed.cuh"

namespace nnb {

namespace {

constexpr int kStripWarps = 4;          // warps per CTA (spreading)
constexpr int kStripInterpThreads = 128;
static_assert(32 * kStripWarps == kStripUnit, "direct spreading: one CTA per unit of points");

template <typename T, int DIM, int W>
struct StripShape {
  static constexpr int RY = W;       // window rows, lanes per run
  static constexpr int NG = 32 / RY;  // runs per warp
  // Distance of the row held by lane r of a run from the first row of its window.
  static __device__ __forceinline__ int offset(int r, int cur) {
    const int d = r - int(unsigned(cur) % unsigned(RY));
    return d < 0 ? d + RY : d;
  }
  static constexpr int TX = DIM == 1 ? 1 : strip_width(sizeof(T), W);
  static constexpr int P0 = DIM == 1 ? 1 : TX + W - 1;  // region cells per row
  static constexpr int NP = (P0 + 1) / 2;               // cell pairs per row
  static constexpr int KXN = DIM == 1 ? 0 : 4 * ((NP + 1) / 2);  // staged kx values
};

// One staged point. `row`: absolute first window row (2D: y, 1D: the cell); `strip`: x strip.
template <typename T, int DIM, int W>
struct alignas(16) StripSlotFields {
  using S = StripShape<T, DIM, W>;
  T kx[S::KXN > 0 ? S::KXN : 4];  // over the strip's cells (1D: unused)
  T ky[S::RY];                    // over the window
  cplx_t<T> v;
  int row, strip;
};
template <bool ODD>
struct StripSlotPad {
  int pad[4];
};
template <>
struct StripSlotPad<true> {};
// An odd number of 16-byte units per slot: 16-byte accesses of consecutive slots fall in
// different banks.
template <typename T, int DIM, int W>
struct alignas(16) StripSlot
    : StripSlotFields<T, DIM, W>, StripSlotPad<(sizeof(StripSlotFields<T, DIM, W>) / 16) % 2 == 1> {
};

// Absolute first cell of a strip-sorted record.
template <int DIM, typename T>
__device__ __forceinline__ void strip_cell(const PointRec<T>& r, int& x0, int& y0) {
  x0 = int(r.local);
  y0 = DIM == 2 ? strip_row(r) : 0;
}

// Spreads the runs of CTA `block`. UNITS: of the points in the units flagged as crowded only.
template <typename T, int DIM, int W, bool UNITS = false>
__device__ __forceinline__ void spread_strip_runs(const SpreadArgs<T>& a, u32 chunk, u32 block,
                                                  StripSlot<T, DIM, W> (*slots)[32]) {
  using S = StripShape<T, DIM, W>;
  using Ops = Packed<T>;
  using P = typename Ops::P;
  using C = cplx_t<T>;
  constexpr int RY = S::RY;

  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int grp = lane / RY;
  const int rb = lane % RY;
  const i64 M = a.pts.M;
  const i64 first = (i64(block) * kStripWarps + warp) * S::NG * chunk;  // of the warp
  if (first >= M) return;
  const i64 beg = first + i64(grp) * chunk;
  // lanes left over by the runs have no points
  int count = grp < S::NG ? int(max(i64(0), min(i64(chunk), M - beg))) : 0;
  if constexpr (UNITS) {  // chunk divides the unit
    if (count > 0 && a.pts.crowded[beg / kStripUnit] == 0) count = 0;
    if (!__any_sync(kFull, count > 0)) return;
  }
  // run 0 of a warp is its longest
  const int iters = (int(min(i64(chunk), M - first)) + RY - 1) / RY;

  const C* __restrict__ in = a.in + i64(blockIdx.y) * a.in_bdist;
  C* grid = a.grid + i64(blockIdx.y) * a.grid_bdist;
  const i64 nfx = a.g.nf[0];
  const i64 nrows = DIM == 1 ? a.g.nf[0] : a.g.nf[1];
  [[maybe_unused]] const i64 cells = a.g.nf[0] * a.g.nf[1];
  const bool vec = (nfx % 2) == 0 && (reinterpret_cast<size_t>(grid) % 16) == 0;

  P are[S::NP], aim[S::NP];
#pragma unroll
  for (int q = 0; q < S::NP; ++q) are[q] = aim[q] = Ops::zero();
  int cur = 0, strip = -1;
  int dz = 0;
  bool dirty = false;

  // Adds this lane's row (absolute; may exceed the grid by less than a window) and clears it.
  auto flush = [&](i64 p) {
    if (!dirty) return;
    dirty = false;
    if (p >= nrows) p -= nrows;
    if constexpr (DIM == 1) {
      if (NNB_CHECK_INDEX(p, cells)) atomic_add_cplx(&grid[p], C{Ops::lo(are[0]), Ops::lo(aim[0])});
    } else {
      const i64 base = p * nfx;
      const i64 gx0 = i64(strip) * S::TX;
      C* row = grid + base;
      if (vec && gx0 + S::P0 <= nfx) {
#pragma unroll
        for (int q = 0; q < S::NP; ++q) {
          if (2 * q + 1 < S::P0) {
            if (NNB_CHECK_INDEX(base + gx0 + 2 * q + 1, cells)) {
              atomic_add_pair(row + gx0 + 2 * q, Ops::lo(are[q]), Ops::lo(aim[q]), Ops::hi(are[q]),
                              Ops::hi(aim[q]));
            }
          } else if (NNB_CHECK_INDEX(base + gx0 + 2 * q, cells)) {
            atomic_add_cplx(row + gx0 + 2 * q, C{Ops::lo(are[q]), Ops::lo(aim[q])});
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < S::NP; ++q) {
          i64 x = gx0 + 2 * q;
          while (x >= nfx) x -= nfx;
          if (NNB_CHECK_INDEX(base + x, cells)) {
            atomic_add_cplx(&row[x], C{Ops::lo(are[q]), Ops::lo(aim[q])});
          }
          x = gx0 + 2 * q + 1;
          while (x >= nfx) x -= nfx;
          if (2 * q + 1 < S::P0 && NNB_CHECK_INDEX(base + x, cells)) {
            atomic_add_cplx(&row[x], C{Ops::hi(are[q]), Ops::hi(aim[q])});
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < S::NP; ++q) are[q] = aim[q] = Ops::zero();
  };

  // The record is loaded two batches ahead and its strength one batch ahead.
  auto load_rec = [&](int k) {
    PointRec<T> r;
    r.perm = 0;
    r.local = 0;
    r.frac[0] = r.frac[1] = r.frac[2] = T(0);
    const int j = k * RY + rb;
    if (j < count && NNB_CHECK_INDEX(beg + j, M)) r = a.pts.rec[beg + j];
    return r;
  };
  auto load_val = [&](const PointRec<T>& r, int k) {
    C v{T(0), T(0)};
    if (k * RY + rb < count && NNB_CHECK_INDEX(r.perm, M)) {
      v = in[r.perm];
      if (a.prephase) v = cmul(v, a.prephase[r.perm]);
    }
    return v;
  };
  PointRec<T> rec = load_rec(0);
  PointRec<T> next = load_rec(1);
  C val = load_val(rec, 0);
  auto& sl = slots[warp][lane];
  for (int k = 0; k < iters; ++k) {
    const PointRec<T> next2 = load_rec(k + 2);
    const C next_val = load_val(next, k + 1);
    {
      int x0, y0;
      strip_cell<DIM>(rec, x0, y0);
      if constexpr (DIM == 2) {
        float4* z = reinterpret_cast<float4*>(sl.kx);
#pragma unroll
        for (int i = 0; i < int(S::KXN * sizeof(T) / 16); ++i) z[i] = make_float4(0, 0, 0, 0);
        T* dst = sl.kx + unsigned(x0) % unsigned(S::TX);
        T wt[W];
        es_weights<W>(rec.frac[0], a.es, a.beta, a.c, wt);
#pragma unroll
        for (int i = 0; i < W; ++i) dst[i] = wt[i];
      }
      T wt[W];
      es_weights<W>(rec.frac[DIM - 1], a.es, a.beta, a.c, wt);
#pragma unroll
      for (int i = 0; i < W; ++i) sl.ky[i] = wt[i];
      sl.v = val;
      sl.row = DIM == 2 ? y0 : x0;
      sl.strip = DIM == 2 ? int(unsigned(x0) / unsigned(S::TX)) : 0;
    }
    __syncwarp();
    const int nb = min(RY, count - k * RY);
#pragma unroll 2
    for (int j = 0; j < nb; ++j) {
      const auto& pt = slots[warp][grp * RY + j];
      const int tp = pt.row, ts = pt.strip;
      if (tp != cur || ts != strip) {  // rows [cur, tp), or the whole window, are complete
        // (1D bins may hold several cells in any order: an earlier cell counts as far ahead)
        if (unsigned(dz) < (ts == strip ? unsigned(tp - cur) : unsigned(RY))) flush(i64(cur) + dz);
        cur = tp;
        strip = ts;
        dz = S::offset(rb, cur);
      }
      dirty = true;
      const T kw = pt.ky[dz];
      const P wre = Ops::splat(pt.v.x * kw);
      const P wim = Ops::splat(pt.v.y * kw);
      if constexpr (DIM == 1) {
        are[0] = Ops::add(are[0], wre);
        aim[0] = Ops::add(aim[0], wim);
      } else {
#pragma unroll
        for (int q = 0; q < S::NP; q += 2) {
          P kk[2];
          load_pairs<T>(&pt.kx[2 * q], kk);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (q + u < S::NP) {
              are[q + u] = Ops::fma(kk[u], wre, are[q + u]);
              aim[q + u] = Ops::fma(kk[u], wim, aim[q + u]);
            }
          }
        }
      }
    }
    __syncwarp();
    rec = next;
    next = next2;
    val = next_val;
  }
  // Runs of a warp that end in the same window are added up before they go to the grid: points that
  // crowd into a few cells are many runs long, and each addition to a cell rounds its sum (over
  // the CTA's warps, with a barrier: walking the points gets 4 % slower).
  if (S::NG > 1) {
    const int cur0 = __shfl_sync(kFull, cur, 0);  // (not in the test: every lane takes part)
    const int strip0 = __shfl_sync(kFull, strip, 0);
    const bool same = cur == cur0 && strip == strip0;
    if (__all_sync(kFull, same || count <= 0)) {
#pragma unroll
      for (int q = 0; q < S::NP; ++q) {
        const P re = are[q], im = aim[q];
#pragma unroll
        for (int g = 1; g < S::NG; ++g) {
          are[q] = Ops::add(are[q], Ops::shfl(re, rb + g * RY));
          aim[q] = Ops::add(aim[q], Ops::shfl(im, rb + g * RY));
        }
      }
      if (grp > 0) dirty = false;
    }
  }
  flush(i64(cur) + dz);
}

template <typename T, int DIM, int W>
__global__ void __launch_bounds__(32 * kStripWarps)
    spread_strip_kernel(const __grid_constant__ SpreadArgs<T> a, u32 chunk) {
  __shared__ StripSlot<T, DIM, W> slots[kStripWarps][32];
  spread_strip_runs<T, DIM, W>(a, chunk, blockIdx.x, slots);
}

// 2D spreading of points so sparse that a window's rows would be flushed after a point or two: the
// warp's lanes add a point's footprint to the grid directly, neighbouring lanes neighbouring
// cells, so that one atomic instruction covers whole sectors of several rows. An element is an
// aligned pair of cells (16 bytes) in single precision, a real or imaginary part in double (there
// are no vector atomics for doubles). A CTA takes one unit of points.
template <typename T, int W>
struct SparseShape {
  static constexpr bool SINGLE = sizeof(T) == 4;
  static constexpr int PER_ROW = SINGLE ? W / 2 + 1 : 2 * W;  // elements per footprint row
  static constexpr int ELEMS = W * PER_ROW;
  static constexpr int KXN = SINGLE ? 2 * PER_ROW : W;        // staged kx values
};
template <typename T, int W>
struct SparseSlot {
  T kx[SparseShape<T, W>::KXN];  // single: from the aligned pair that holds the first cell
  T ky[W];
  cplx_t<T> v;
  int x0, y0;
};

template <typename T, int W>
__device__ __forceinline__ void spread_sparse_unit(const SpreadArgs<T>& a, bool aligned, u32 unit,
                                                   SparseSlot<T, W> (*slots)[32]) {
  using S = SparseShape<T, W>;
  using C = cplx_t<T>;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const i64 M = a.pts.M;
  const i64 first = i64(unit) * kStripUnit + warp * 32;
  if (first >= M) return;
  const int count = int(min(i64(32), M - first));
  const C* __restrict__ in = a.in + i64(blockIdx.y) * a.in_bdist;
  C* grid = a.grid + i64(blockIdx.y) * a.grid_bdist;
  const int nfx = int(a.g.nf[0]), nfy = int(a.g.nf[1]);
  [[maybe_unused]] const i64 cells = a.g.nf[0] * a.g.nf[1];
  if (lane < count && NNB_CHECK_INDEX(first + lane, M)) {
    const PointRec<T> rec = a.pts.rec[first + lane];
    auto& sl = slots[warp][lane];
    C v{T(0), T(0)};
    if (NNB_CHECK_INDEX(rec.perm, M)) {
      v = in[rec.perm];
      if (a.prephase) v = cmul(v, a.prephase[rec.perm]);
    }
    strip_cell<2>(rec, sl.x0, sl.y0);
    T wt[W];
    es_weights<W>(rec.frac[0], a.es, a.beta, a.c, wt);
    const int odd = S::SINGLE ? sl.x0 & 1 : 0;
    if constexpr (S::SINGLE) sl.kx[0] = sl.kx[S::KXN - 1] = sl.kx[S::KXN - 2] = T(0);
#pragma unroll
    for (int i = 0; i < W; ++i) sl.kx[odd + i] = wt[i];
    es_weights<W>(rec.frac[1], a.es, a.beta, a.c, wt);
#pragma unroll
    for (int i = 0; i < W; ++i) sl.ky[i] = wt[i];
    sl.v = v;
  }
  __syncwarp();
  constexpr int PASSES = (S::ELEMS + 31) / 32;
  int row[PASSES], col[PASSES];
#pragma unroll
  for (int p = 0; p < PASSES; ++p) {
    row[p] = (lane + 32 * p) / S::PER_ROW;
    col[p] = (lane + 32 * p) % S::PER_ROW;
  }
  for (int j = 0; j < count; ++j) {
    const auto& pt = slots[warp][j];
    const C v = pt.v;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
      if (row[p] >= W) continue;
      int y = pt.y0 + row[p];
      if (y >= nfy) y -= nfy;
      const i64 base = i64(y) * nfx;
      const T ky = pt.ky[row[p]];
      if constexpr (S::SINGLE) {
        const int x = (pt.x0 & ~1) + 2 * col[p];
        const T k0 = pt.kx[2 * col[p]] * ky, k1 = pt.kx[2 * col[p] + 1] * ky;
        if (aligned && (pt.x0 & ~1) + 2 * S::PER_ROW <= nfx) {
          // an even first cell leaves the last pair without weights
          if (2 * col[p] < W + (pt.x0 & 1) && NNB_CHECK_INDEX(base + x + 1, cells)) {
            atomic_add_pair(grid + base + x, k0 * v.x, k0 * v.y, k1 * v.x, k1 * v.y);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int off = 2 * col[p] + i - (pt.x0 & 1);  // cell of the footprint
            int xi = x + i;
            if (xi >= nfx) xi -= nfx;
            if (off >= 0 && off < W && NNB_CHECK_INDEX(base + xi, cells)) {
              const T k = i ? k1 : k0;
              atomic_add_cplx(grid + base + xi, C{k * v.x, k * v.y});
            }
          }
        }
      } else {
        int x = pt.x0 + col[p] / 2;
        if (x >= nfx) x -= nfx;
        const T k = pt.kx[col[p] / 2] * ky;
        if (NNB_CHECK_INDEX(base + x, cells)) {
          T* cell = reinterpret_cast<T*>(grid + base + x);
          atomicAdd(cell + (col[p] & 1), k * ((col[p] & 1) ? v.y : v.x));
        }
      }
    }
  }
}

template <typename T, int W>
__global__ void __launch_bounds__(32 * kStripWarps)
    spread_sparse_kernel(const __grid_constant__ SpreadArgs<T> a, bool aligned) {
  __shared__ SparseSlot<T, W> slots[kStripWarps][32];
  spread_sparse_unit<T, W>(a, aligned, blockIdx.x, slots);
}

// Sparse points with crowded units: the first `nwindow` CTAs walk the crowded ones through windows
// in runs of `chunk` points, the others add the points of the rest directly. (One launch, so that
// the latency of a few runs hides behind the direct additions: 1e6 radial points on 3000^2 cells,
// w = 7, 97 us; 127 in two launches, 106 with all points added directly.)
template <typename T, int W>
__global__ void __launch_bounds__(32 * kStripWarps)
    spread_mixed_kernel(const __grid_constant__ SpreadArgs<T> a, bool aligned, u32 chunk,
                        u32 nwindow) {
  __shared__ union Slots {
    __device__ Slots() {}
    StripSlot<T, 2, W> window[kStripWarps][32];
    SparseSlot<T, W> direct[kStripWarps][32];
  } sh;
  if (blockIdx.x < nwindow) {
    spread_strip_runs<T, 2, W, true>(a, chunk, blockIdx.x, sh.window);
  } else if (a.pts.crowded[blockIdx.x - nwindow] == 0) {
    spread_sparse_unit<T, W>(a, aligned, blockIdx.x - nwindow, sh.direct);
  }
}

template <typename T, int DIM, int W>
__global__ void __launch_bounds__(kStripInterpThreads)
    interp_strip_kernel(const __grid_constant__ InterpArgs<T> a) {
  using C = cplx_t<T>;
  const i64 i = i64(blockIdx.x) * kStripInterpThreads + threadIdx.x;
  if (i >= a.pts.M) return;
  const PointRec<T> rec = a.pts.rec[i];
  const u32 idx = rec.perm;
  int x0, y0;
  strip_cell<DIM>(rec, x0, y0);
  const i64 nfx = a.g.nf[0];
  [[maybe_unused]] const i64 cells = a.g.nf[0] * a.g.nf[1];
  const C* __restrict__ grid = a.grid;
  constexpr int NR = DIM == 1 ? 1 : W;
  T kx[W], ky[NR];
  es_weights<W>(rec.frac[0], a.es, a.beta, a.c, kx);
  if constexpr (DIM == 2) es_weights<W>(rec.frac[1], a.es, a.beta, a.c, ky);
  T sx = 0, sy = 0;
  const int ny = int(a.g.nf[1]);
  const bool inside = i64(x0) + W <= nfx;  // the cells of a row are consecutive
#pragma unroll
  for (int dy = 0; dy < NR; ++dy) {
    int y = y0 + dy;
    if (DIM == 2 && y >= ny) y -= ny;
    const i64 base = DIM == 2 ? i64(y) * nfx : 0;
    const C* __restrict__ row = grid + base;
    T rx = 0, ry = 0;
    if (inside) {
      const C* __restrict__ p = row + x0;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        if (NNB_CHECK_INDEX(base + x0 + k, cells)) {
          const C v = p[k];
          rx += kx[k] * v.x;
          ry += kx[k] * v.y;
        }
      }
    } else {
#pragma unroll
      for (int k = 0; k < W; ++k) {
        i64 x = i64(x0) + k;
        if (x >= nfx) x -= nfx;
        if (NNB_CHECK_INDEX(base + x, cells)) {
          const C v = row[x];
          rx += kx[k] * v.x;
          ry += kx[k] * v.y;
        }
      }
    }
    if constexpr (DIM == 2) {
      sx += ky[dy] * rx;
      sy += ky[dy] * ry;
    } else {
      sx = rx;
      sy = ry;
    }
  }
  C res{sx, sy};
  if (!NNB_CHECK_INDEX(idx, a.pts.M)) return;
  if (a.postphase) res = cmul(res, a.postphase[idx]);
  a.out[idx] = res;
}

// Points per run: enough runs to fill the GPU, but not so short that the rows flushed at a run's
// end outweigh its points, and no longer than balances the load. Where points crowd into single
// bins runs are as long as the work items of the shared-memory kernels, so that a cell's sum is
// rounded no more often (2e7 strengths of one sign on 200 cells, a dozen of which hold all, w = 7:
// a relative error of 7e-7 in 403 us, with runs of 512 points 6e-6 in 383 us, and 5e-5 with these
// added one by one; 2e7 on 4e4 cells 453 and 406 us).
u32 strip_chunk(i64 M, bool crowded, int runs_per_warp, int ry) {
  const i64 runs = i64(148) * 24 * runs_per_warp;
  i64 c = (M + runs - 1) / runs;
  c = (c + ry - 1) / ry * ry;
  const i64 lo = 2 * ry, hi = crowded ? i64(kWorkItemPoints) : 512;
  return u32(c < lo ? lo : (c > hi ? hi : c));
}

// Whether a unit of points is crowded: four or more of its points to every bin that it touches.
// (Uniform points at the limit to sparse sets come 1.2 to 1.8 to an occupied bin.)
template <typename T>
__global__ void __launch_bounds__(kStripUnit)
    strip_crowded_kernel(const PointRec<T>* __restrict__ rec, i64 M, int tx,
                         unsigned char* crowded) {
  const i64 i = i64(blockIdx.x) * kStripUnit + threadIdx.x;
  bool first = false;
  if (i < M) {
    int x0, y0;
    strip_cell<2>(rec[i], x0, y0);
    first = threadIdx.x == 0;
    if (!first) {
      int px, py;
      strip_cell<2>(rec[i - 1], px, py);
      first = py != y0 || px / tx != x0 / tx;
    }
  }
  const int bins = __syncthreads_count(first);
  if (threadIdx.x == 0) {
    const int n = int(min(i64(kStripUnit), M - i64(blockIdx.x) * kStripUnit));
    crowded[blockIdx.x] = 4 * bins <= n ? 1 : 0;
  }
}

template <typename T, int DIM, int W>
void launch_spread_strip_w(const SpreadArgs<T>& a, cudaStream_t stream) {
  using S = StripShape<T, DIM, W>;
  if constexpr (DIM == 2) {
    const i64 ctas = (a.pts.M + kStripUnit - 1) / kStripUnit;  // units
    if (strip_sparse(a.g, a.pts.M)) {
      const bool aligned = a.g.nf[0] % 2 == 0 && a.grid_bdist % 2 == 0 &&
                           reinterpret_cast<uintptr_t>(a.grid) % 16 == 0;
      dim3 grid{unsigned(ctas), unsigned(a.batch), 1u};
      // The crowded units go to windows: added directly, the points of a cluster queue up for a
      // few sectors, and a cell's sum is rounded once per point (1.2e6 points of one sign, sigma
      // 0.01 rad, 3000^2 cells, w = 7: 1669 us and a relative error of 2e-4 against 66 us and
      // 5e-7).
      if (a.pts.crowded_points == 0) {
        spread_sparse_kernel<T, W><<<grid, 32 * kStripWarps, 0, stream>>>(a, aligned);
      } else {
        // runs of a unit; of a half or a quarter while there are few
        u32 chunk = kStripUnit;
        while (chunk > 32 && a.pts.crowded_points / chunk < 148 * 24) chunk /= 2;
        const i64 per_cta = i64(chunk) * S::NG * kStripWarps;
        const unsigned nwindow = unsigned((a.pts.M + per_cta - 1) / per_cta);
        grid.x += nwindow;
        spread_mixed_kernel<T, W><<<grid, 32 * kStripWarps, 0, stream>>>(a, aligned, chunk,
                                                                         nwindow);
      }
      NNB_LAUNCH_CHECK();
      return;
    }
  }
  const u32 chunk = strip_chunk(a.pts.M, a.pts.crowded_points > 0, S::NG, S::RY);
  const i64 per_cta = i64(chunk) * S::NG * kStripWarps;
  const i64 ctas = (a.pts.M + per_cta - 1) / per_cta;
  if (ctas > 0x7fffffffll) throw_input("grid too large");
  dim3 grid{unsigned(ctas), unsigned(a.batch), 1u};
  spread_strip_kernel<T, DIM, W><<<grid, 32 * kStripWarps, 0, stream>>>(a, chunk);
  NNB_LAUNCH_CHECK();
}

template <typename T, int DIM, int W>
void launch_interp_strip_w(const InterpArgs<T>& a, cudaStream_t stream) {
  const i64 ctas = (a.pts.M + kStripInterpThreads - 1) / kStripInterpThreads;
  interp_strip_kernel<T, DIM, W><<<unsigned(ctas), kStripInterpThreads, 0, stream>>>(a);
  NNB_LAUNCH_CHECK();
}

// Calls f(std::integral_constant<int, w>) for 2 <= w <= 16.
template <int W, typename F>
void with_strip_width(int w, F&& f) {
  if constexpr (W > 16) {
    throw_internal("n_spread not in [2, 16]");
  } else {
    if (w == W) return f(std::integral_constant<int, W>{});
    with_strip_width<W + 1>(w, f);
  }
}

void check_strip_geom(const BinGeom& g) {
  if (!g.strip || (g.dim != 1 && g.dim != 2)) {
    throw_internal("strip kernels need a 1D or 2D strip-ordered tiling");
  }
}

}  // namespace

// w cells per point or more, at least 6. Uniform points on 4096^2 cells (2048^2 in double
// precision), windows / direct, in us, at 20, 10 and 5 cells per point: w = 4 133 / 75, 173 / 119,
// 209 / 223; w = 8 193 / 126, 232 / 212, 344 / 405; double w = 10 138 / 79, 174 / 147, 249 / 290;
// w = 13 177 / 123, 218 / 239, 303 / 495. The type-3 spread of 5e6 points on 12740^2 cells, w = 6:
// 2176 / 827 (shared-memory slabs 1335).
bool strip_sparse(const BinGeom& g, i64 M) {
  return g.dim == 2 && g.strip && double(M) * std::max(6, g.w) < double(g.nf[0]) * double(g.nf[1]);
}

template <typename T>
void launch_strip_crowded(const BinGeom& g, const PointRec<T>* rec, i64 M, unsigned char* crowded,
                          cudaStream_t stream) {
  const i64 units = (M + kStripUnit - 1) / kStripUnit;
  strip_crowded_kernel<T><<<unsigned(units), kStripUnit, 0, stream>>>(rec, M, g.tile[0], crowded);
  NNB_LAUNCH_CHECK();
}

template <typename T>
void launch_spread_strip(const SpreadArgs<T>& a, cudaStream_t stream) {
  check_strip_geom(a.g);
  // 2D windows need the points of a strip row by row
  if (a.g.dim == 2 && (a.g.tile[0] != strip_width(sizeof(T), a.g.w) ||
                       (a.g.tile[1] != 1 && !strip_sparse(a.g, a.pts.M)))) {
    throw_internal("strip spreading needs bins of one row");
  }
  if (a.batch > 65535) throw_input("batch size above 65535");
  if (a.pts.M <= 0) return;
  with_strip_width<2>(a.g.w, [&](auto wc) {
    constexpr int W = decltype(wc)::value;
    if (a.g.dim == 1) {
      launch_spread_strip_w<T, 1, W>(a, stream);
    } else {
      launch_spread_strip_w<T, 2, W>(a, stream);
    }
  });
}

template <typename T>
void launch_interp_strip(const InterpArgs<T>& a, cudaStream_t stream) {
  check_strip_geom(a.g);
  if (a.pts.M <= 0) return;
  with_strip_width<2>(a.g.w, [&](auto wc) {
    constexpr int W = decltype(wc)::value;
    if (a.g.dim == 1) {
      launch_interp_strip_w<T, 1, W>(a, stream);
    } else {
      launch_interp_strip_w<T, 2, W>(a, stream);
    }
  });
}

template void launch_spread_strip<float>(const SpreadArgs<float>&, cudaStream_t);
template void launch_spread_strip<double>(const SpreadArgs<double>&, cudaStream_t);
template void launch_strip_crowded<float>(const BinGeom&, const PointRec<float>*, i64,
                                          unsigned char*, cudaStream_t);
template void launch_strip_crowded<double>(const BinGeom&, const PointRec<double>*, i64,
                                           unsigned char*, cudaStream_t);
template void launch_interp_strip<float>(const InterpArgs<float>&, cudaStream_t);
template void launch_interp_strip<double>(const InterpArgs<double>&, cudaStream_t);

}  // namespace nnb
