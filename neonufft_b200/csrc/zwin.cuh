// 3D ES spreading and interpolation with a sliding z-window held in registers (method 3).
//
// Replaces, for 3D plans, the reference's spreading
// (src/neonufft/gpu/kernels/spreading_kernel.cu:477-715, one global float atomic per cell and
// point) and interpolation (src/neonufft/gpu/kernels/interpolation_kernel.cu, one thread per
// point reading w^3 cells from global memory).
//
// Points are binned by (x tile of TX cells, y tile of TY cells, single z plane), and the bins of
// one (x, y) column are consecutive in plane order (BinGeom::zmajor), so the points of a column
// and range of planes are one contiguous run of records. One CTA walks one column over a chunk
// of planes. Its region is P0 x P1 cells in (x, y), P0 = TX + w - 1 and P1 = TY + w - 1, times a
// window of RZ >= w consecutive planes [t, t + RZ): 4 or 8 planes up to w = 8, exactly w above.
//  * thread (a, b) keeps in registers the whole region row y = a (P0 cells, as pairs of
//    neighbouring cells) of the window plane p = b (mod RZ), or of two planes, RZ / 2 apart
//    (ZShape::PZ). The RY >= P1 rows are split over the warps, LA rows per warp (as many as its
//    32 lanes hold with RZ / PZ lanes each), so for a point whose footprint covers rows
//    [ly, ly + w) a warp either owns some of them or skips the point with a warp-uniform
//    branch; no thread holds a cell that another thread updates, so there are no atomics and
//    no shared-memory traffic per cell;
//  * the run of points is staged in shared memory 32 to 64 at a time (ZShape::BATCH;
//    double-buffered, one barrier per batch, spread over all warps): kx over the region's x
//    range, ky over the rows and kz over the RZ planes, each zero outside the footprint, so that
//    every thread applies them with fixed register indices and no range tests;
//  * each owning thread updates its row with packed two-float FMAs (fma.rn.f32x2 on sm_100a),
//    one for the real and one for the imaginary parts of two neighbouring cells;
//  * when the next point starts on a later plane, the window advances: spreading adds each
//    completed plane to the fine grid (float2 / double2 atomics: neighbouring columns and
//    chunks overlap by the halo); interpolation reloads the threads that held it with the
//    plane RZ further on (plain loads: a cp.async prefetch one plane ahead measured no faster);
//  * interpolation reduces the row sums of eight points at a time (four of wide kernels) through
//    a per-warp shared-memory transpose, then over warps.
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "packed.cuh"

namespace nnb {

namespace {

// ---- geometry ----------------------------------------------------------------------------------
// PZ: window planes per thread. With two, a warp holds 8 rows instead of 4, so a point is visited
// by fewer warps (1.9 of 2 instead of 2.75 of 4 at w = 8, 8-row tiles) and each visit's loads,
// weights and bookkeeping serve twice the FMAs. 1e7 points on 256^3 cells, w = 8, single precision:
// spreading 2.03 -> 1.86 ms, interpolation 2.58 -> 2.43 ms (with one plane the polynomial weights
// had already taken interpolation from 2.73 to 2.58 ms). Spreading on 4-row tiles keeps one plane
// (1e8 points on 480^3 cells: 16.5 against 18.2 ms with two), and so does double precision (3e6
// clustered points, w = 7: spreading 1.19 against 1.26 ms, interpolation 1.30 against 1.29).
template <typename T, int W, int TX, int TY_ = 8, int PZ_ = 1>
struct ZShape {
  static constexpr int PZ = PZ_;
  static constexpr bool WIDE = W > 8;
  // Window planes = z residues (>= W). Wide kernels take exactly W: rounded up to 16, half of the
  // FMAs of w = 10 would be on planes outside the footprint.
  static constexpr int RZ = W <= 4 ? 4 : (W <= 8 ? 8 : W);
  static constexpr int ZL = RZ / PZ;                // lanes along z
  static constexpr int LA = 32 / ZL;                // rows per warp
  static constexpr int TY = TY_;                    // tile y (4, 8 or 16)
  static constexpr int P1 = TY + W - 1;             // region y extent
  // region rows (>= P1, a multiple of the rows per warp)
  static constexpr int RY = TY == 4 || WIDE || PZ > 1 ? (P1 + LA - 1) / LA * LA : TY + 8;
  static constexpr int NWARP = RY / LA;
  static constexpr int NT = 32 * NWARP;             // threads per CTA
  static constexpr int P0 = TX + W - 1;             // region x extent (cells)
  static constexpr int NP = (P0 + 1) / 2;           // cell pairs per row
  static constexpr int KXN = 4 * ((NP + 1) / 2);    // staged kx values (16-byte multiple)
  static constexpr int RYS = (RY + 3) / 4 * 4;      // staged ky values (16-byte multiple)
  static constexpr int RZS = (RZ + 3) / 4 * 4;      // staged kz values (16-byte multiple)
  // points staged at a time, each warp its share
  static constexpr int BATCH =
      sizeof(T) == 4 && !WIDE && PZ == 1 ? (NWARP == 1 ? 32 : (NWARP % 3 == 0 ? 48 : 64)) : 32;
  static constexpr int PW = (BATCH + NWARP - 1) / NWARP;  // points staged per warp
  static constexpr int G = WIDE ? 4 : 8;            // points reduced together (interpolation)
  // CTAs per SM the interpolation kernel is compiled for: 6 in single precision (78 registers,
  // no spills; 86 uncapped, which allows only 5 CTAs and measured 6 % slower), 5 in double.
  // Two planes per thread: 96 registers (interpolation), 92 (spreading).
  static constexpr int PZ_INTERP_CTAS = 65536 / (NT * 96);
  static constexpr int SPREAD_CTAS = 65536 / (NT * 92);
  // The wide kernels have a budget of 112 registers (3 CTAs of 192 threads at w = 10 in double
  // precision, a few spills; uncapped, ptxas takes 157 and 2 CTAs fit: spreading 5e5 points
  // 512 -> 453 us, interpolation 628 -> 567 us).
  static constexpr int WIDE_CTAS = 65536 / (NT * 112) > 0 ? 65536 / (NT * 112) : 1;
  static constexpr int INTERP_CTAS =
      WIDE ? WIDE_CTAS : (PZ > 1 ? PZ_INTERP_CTAS : (sizeof(T) == 4 ? 6 : 5));
  // CTAs per SM the two-vector spreading kernel is compiled for: a budget of about 88 registers
  // a thread (7 CTAs of 96 threads; ptxas then allocates 80 registers and spills 24 bytes for
  // w = 8). Uncapped, the allocator takes 158 registers for w = 8, which leaves 2 CTAs per SM.
  static constexpr int SPREAD2_CTAS = 65536 / (NT * 88) > 0 ? 65536 / (NT * 88) : 1;
  static_assert(W <= RZ && P1 <= RY, "window smaller than the kernel footprint");
  static_assert(RZ % PZ == 0 && (PZ == 1 || !WIDE), "planes per thread");
  static_assert(PW <= 32 && BATCH % G == 0, "staging threads");
  // Residue of a plane (>= 0), and its distance from residue r of a window starting at cur.
  static __device__ __forceinline__ int offset(int r, int cur) {
    if constexpr (!WIDE) return (r - cur) & (RZ - 1);
    const int d = r - int(unsigned(cur) % unsigned(RZ));
    return d < 0 ? d + RZ : d;
  }
};

// CTAs per SM the persistent kernels are compiled for: without the cap, their loop over items
// lets the register allocator grow far past the per-transform kernels (166 against 72).
template <typename T>
constexpr int kSpreadFusedCtas = sizeof(T) == 4 ? 7 : 4;
template <typename T>
constexpr int kInterpFusedCtas = sizeof(T) == 4 ? 6 : 4;

// Per-point data staged in shared memory (one slot per point of a batch).
template <typename T, int W, int TX, int TY = 8, int PZ = 1>
struct alignas(16) ZSlotFields {
  using S = ZShape<T, W, TX, TY, PZ>;
  T kx[S::KXN];    // kx over the region's x range, zero outside the footprint
  T ky[S::RYS];    // ky over the region rows, zero outside the footprint
  T kz[S::RZS];    // kz per window offset, zero beyond w
  cplx_t<T> v;     // strength (spreading)
  int lyp;         // first footprint row | first footprint plane << 4
  u32 perm;        // original point index
};
// 16 bytes of padding when the fields span an even number of 16-byte units: with an odd slot
// stride, consecutive lanes staging consecutive slots store to different banks.
template <bool ODD>
struct ZSlotPad {
  int pad[4];
};
template <>
struct ZSlotPad<true> {};
template <typename T, int W, int TX, int TY = 8, int PZ = 1>
struct alignas(16) ZSlot
    : ZSlotFields<T, W, TX, TY, PZ>,
      ZSlotPad<(sizeof(ZSlotFields<T, W, TX, TY, PZ>) / 16) % 2 == 1> {};

// Stages `count` (<= 16) bin-sorted records `recs` into slots[0 .. count), one warp: lanes
// 0 .. count - 1 load the records (and, for spreading, the strengths; with `v2_out`, also the
// second vector's strengths from `in2`, or zeros where in2 is null, into v2_out[0 .. count), so
// that both gathers are in flight together); then lane pair
// (2p, 2p + 1) fills point p's slot with the same instruction stream: the even lane kx and the
// first half of kz, the odd lane ky and the second half, each zeroing half of the contiguous
// kx / ky arrays first, so all 32 lanes evaluate kernel values.
//
// POLY: kernel values by the polynomials of the pieces; double precision gives each lane of the
// pair its half of kz (single precision measured slower that way: 1.98 against 1.86 ms per 1e7
// points) while both evaluate all of kz in single.
template <typename T, int W, int TX, bool SPREAD, int TY = 8, int PZ = 1, bool POLY = true>
__device__ __forceinline__ void stage_warp(ZSlot<T, W, TX, TY, PZ>* slots, const PointRec<T>* recs,
                                           int count, const cplx_t<T>* in,
                                           const cplx_t<T>* prephase,
                                           const EsPoly<T>& es, T beta, T c, int lane, i64 num,
                                           const cplx_t<T>* in2 = nullptr,
                                           cplx_t<T>* v2_out = nullptr) {
  using S = ZShape<T, W, TX, TY, PZ>;
  using C = cplx_t<T>;
  constexpr unsigned kFull = 0xffffffffu;
  PointRec<T> rec;
  rec.perm = 0;
  rec.local = 0;
  rec.frac[0] = rec.frac[1] = rec.frac[2] = T(0);
  C v{T(0), T(0)};
  if (lane < count) {
    rec = recs[lane];
    if constexpr (SPREAD) {
      C v2{T(0), T(0)};
      if (NNB_CHECK_INDEX(rec.perm, num)) {
        v = in[rec.perm];
        if (in2) v2 = in2[rec.perm];
        if (prephase) {
          const C ph = prephase[rec.perm];
          v = cmul(v, ph);
          v2 = cmul(v2, ph);
        }
      }
      if (v2_out) v2_out[lane] = v2;
    }
  }
  const int p = lane >> 1;
  const int h = lane & 1;
  const u32 loc = __shfl_sync(kFull, rec.local, p);
  const u32 perm = __shfl_sync(kFull, rec.perm, p);
  const T fx = __shfl_sync(kFull, rec.frac[0], p);
  const T fy = __shfl_sync(kFull, rec.frac[1], p);
  const T fz = __shfl_sync(kFull, rec.frac[2], p);
  const T vx = __shfl_sync(kFull, v.x, p);
  const T vy = __shfl_sync(kFull, v.y, p);
  ZSlot<T, W, TX, TY, PZ>& sl = slots[p < count ? p : 0];
  constexpr int kZero16 = int((S::KXN + S::RYS) * sizeof(T) / 16);  // kx and ky are contiguous
  constexpr int kHalf = (kZero16 + 1) / 2;
  if (p < count) {
    float4* z = reinterpret_cast<float4*>(sl.kx);
#pragma unroll
    for (int i = 0; i < kHalf; ++i) {
      if (h * kHalf + i < kZero16) z[h * kHalf + i] = make_float4(0, 0, 0, 0);
    }
  }
  __syncwarp();
  if (p < count) {
    const int lx = int(loc & 0xFu);
    const int ly = int((loc >> 4) & 0xFu);
    T* dst = h ? sl.ky + ly : sl.kx + lx;
    if constexpr (POLY) {
      T wt[W];
      es_weights<W>(h ? fy : fx, es, beta, c, wt);
#pragma unroll
      for (int k = 0; k < W; ++k) dst[k] = wt[k];
      if constexpr (sizeof(T) == 8) {
        es_half<W>(fz, h, es, beta, c, [&](int k, T v) { sl.kz[k] = v; });
        if (h) {
#pragma unroll
          for (int k = W; k < S::RZS; ++k) sl.kz[k] = T(0);
        }
      } else {
        es_weights<W>(fz, es, beta, c, wt);
#pragma unroll
        for (int i = 0; i < S::RZS / 2; ++i) {
          constexpr int H = S::RZS / 2;
          const T lo = i < W ? wt[i < W ? i : 0] : T(0);
          const T hi = H + i < W ? wt[H + i < W ? H + i : 0] : T(0);
          sl.kz[h * H + i] = h ? hi : lo;
        }
      }
    } else {
      const T f = h ? fy : fx;
#pragma unroll
      for (int k = 0; k < W; ++k) dst[k] = es_eval_fast<T>(f + T(k), beta, c);
#pragma unroll
      for (int i = 0; i < S::RZS / 2; ++i) {
        const int k = h * (S::RZS / 2) + i;
        sl.kz[k] = k < W ? es_eval_fast<T>(fz + T(k), beta, c) : T(0);
      }
    }
    if (h == 0) {
      sl.v = C{vx, vy};
      sl.lyp = ly | int((loc >> 8) << 4);
      sl.perm = perm;
    }
  }
}

// base + off wrapped to [0, n) for 0 <= base < n, 0 <= off.
__device__ __forceinline__ i64 wrap_add(i64 base, int off, i64 n) {
  i64 i = base + off;
  while (i >= n) i -= n;
  return i;
}

// Column gx0 + i wrapped to the grid; `narrow` when the grid is narrower than the region.
__device__ __forceinline__ i64 wrap_x(i64 gx0, int i, i64 nfx, bool narrow) {
  i64 x = gx0 + i;
  if (narrow) {
    while (x >= nfx) x -= nfx;
  } else if (x >= nfx) {
    x -= nfx;
  }
  return x;
}

// Plane p (p >= 0, below nfz plus a window) wrapped into the grid.
__device__ __forceinline__ i64 wrap_plane(int p, i64 nfz) {
  i64 z = p;
  while (z >= nfz) z -= nfz;
  return z;
}

// CTA coordinates: column (tx, ty), plane range [z0, z1) and its run of points [pbeg, pend).
struct ZCta {
  int tx, ty, z0, z1;
  u32 pbeg, pend;
};
__device__ __forceinline__ bool zcta(const BinGeom& g, const u32* bin_start, ZChunks ch,
                                     const WorkList& wl, u32 item, ZCta& c) {
  u32 unit, slice;
  if (!work_item_at(wl, item, unit, slice)) return false;
  const i64 ncols = i64(g.ntiles[0]) * g.ntiles[1];
  const int chunk = int(unit / ncols);
  const i64 col = unit - i64(chunk) * ncols;
  c.tx = int(col % g.ntiles[0]);
  c.ty = int(col / g.ntiles[0]);
  const int nz = g.ntiles[2];  // == nf[2]: single-plane tiles
  c.z0 = chunk * ch.len;
  c.z1 = min(c.z0 + ch.len, nz);
  const u32* bs = bin_start + col * nz;
  work_slice(bs[c.z0], bs[c.z1], slice, wl.cap, c.pbeg, c.pend);
  return c.pbeg < c.pend;
}

// Thread layout shared by both kernels.
template <typename T, int W, int TX, int TY = 8, int PZ = 1>
struct ZThread {
  using S = ZShape<T, W, TX, TY, PZ>;
  int tid, warp, lane, ra, rb, a_lo;
  bool active;  // the lane holds a row (with LA RZ < 32 lanes per warp, some do not)
  int stage_j;  // batch slot this thread stages (< BATCH), or -1
  __device__ __forceinline__ ZThread() {
    tid = threadIdx.x;
    warp = tid >> 5;
    lane = tid & 31;
    active = S::LA * S::ZL == 32 || lane < S::LA * S::ZL;
    ra = warp * S::LA + lane % S::LA;  // region row
    rb = active ? lane / S::LA : 0;     // z residue of the first plane, the next ZL further on
    a_lo = warp * S::LA;                // first row of this warp
    // consecutive lanes stage consecutive slots (the slot stride is 4 words times an odd
    // number, so their shared-memory stores fall in different banks)
    stage_j = lane < S::PW ? warp * S::PW + lane : -1;
  }
  // Whether this warp owns rows of a footprint starting at row ly.
  __device__ __forceinline__ bool owns(int ly) const { return ly < a_lo + S::LA && ly + W > a_lo; }
};

// ---- spreading ---------------------------------------------------------------------------------
// NV strength vectors on the same points (NV = 2: the second vector's staged strengths).
template <typename T, int W, int TX, int TY = 8, int NV = 1, int PZ = 1>
struct ZSpreadShared {
  ZSlot<T, W, TX, TY, PZ> slots[2][ZShape<T, W, TX, TY, PZ>::BATCH];
  cplx_t<T> v2[2][NV > 1 ? ZShape<T, W, TX, TY, PZ>::BATCH : 1];
};

// Whether spreading takes kernel values from the polynomials.
//
// One vector and one plane per thread in single precision keeps the formula: with the
// polynomials ptxas takes 96 instead of 55 registers and 1e8 points on 480^3 cells 23.5 instead
// of 16.5 ms (20.2 capped at 64). With two planes they take 1e7 points from 2.32 to 1.86 ms.
// Two vectors take what the single vector of the same tile and width takes: on points clustered
// in a few cells the formula's rounding (5e-7 per dimension) does not average out, and the
// vectors of transform_type_1_many would differ from single transforms by more than 1e-6.
template <typename T, int W, int TY, int NV, int PZ>
constexpr bool zspread_poly =
    sizeof(T) == 8 || W > 8 || PZ > 1 || (NV > 1 && W >= 5 && TY == 8);

// Spreads work item `item` of batch entries batch .. batch + NV - 1 (one CTA; every thread
// calls it). With NV = 2 each staged point, its kernel values and the window's bookkeeping
// serve two strength vectors on the same points (type-3 batches, repeated type-1 transforms):
// the second vector's row sums sit in their own registers and go to the next grid (at
// grid_bdist); a missing second entry (an odd batch) is skipped.
template <typename T, int W, int TX, int TY = 8, int NV = 1, int PZ = 1,
          bool POLY = zspread_poly<T, W, TY, NV, PZ>>
__device__ __forceinline__ void spread_zwin_item(const SpreadArgs<T>& a, ZChunks ch,
                                                 const WorkList& wl, u32 item, int batch,
                                                 ZSpreadShared<T, W, TX, TY, NV, PZ>& sh) {
  static_assert(NV == 1 || NV == 2, "one or two strength vectors per pass");
  static_assert(NV == 1 || (PZ == 1 && !ZShape<T, W, TX, TY, PZ>::WIDE),
                "two vectors use one plane per thread, widths up to 8");
  using S = ZShape<T, W, TX, TY, PZ>;
  using Ops = Packed<T>;
  using P = typename Ops::P;
  using C = cplx_t<T>;
  using Slot = ZSlot<T, W, TX, TY, PZ>;
  auto& slots = sh.slots;

  const BinGeom& g = a.g;
  ZCta cta;
  if (!zcta(g, a.pts.bin_start, ch, wl, item, cta)) return;
  const ZThread<T, W, TX, TY, PZ> th;
  const C* in = a.in + batch * a.in_bdist;
  C* grid = a.grid + batch * a.grid_bdist;
  const bool has2 = NV > 1 && batch + 1 < a.batch;  // the second vector exists
  const i64 nfx = g.nf[0], nfy = g.nf[1], nfz = g.nf[2];
  [[maybe_unused]] const i64 cells = nfx * nfy * nfz;
  const bool narrow = nfx < S::P0;
  const bool has_row = th.active && th.ra < S::P1;
  const i64 row_y = has_row ? wrap_add(i64(cta.ty) * S::TY, th.ra, nfy) : 0;
  const i64 gx0 = i64(cta.tx) * TX;

  // real / imaginary parts of cell pairs (2q, 2q + 1) of the row, per strength vector or plane
  constexpr int NA = NV * PZ;
  P are[NA][S::NP], aim[NA][S::NP];
#pragma unroll
  for (int v = 0; v < NA; ++v) {
#pragma unroll
    for (int q = 0; q < S::NP; ++q) are[v][q] = aim[v][q] = Ops::zero();
  }
  bool dirty = false;

  // Adds this thread's row of plane p (absolute; may exceed nfz; the thread's z-th plane, a
  // constant) to the grid(s) and clears it.
  // The region's x range lies inside the grid and its rows start 16-byte aligned (the usual
  // case): whole cell pairs are added with one vector atomic each.
  const bool pairs = !narrow && gx0 + S::P0 <= nfx && (nfx % 2) == 0 &&
                     (reinterpret_cast<size_t>(grid) % 16) == 0 &&
                     (NV == 1 || (a.grid_bdist % 2) == 0);
  auto flush = [&](auto zc, int p) {
    constexpr int z = decltype(zc)::value;
    if (has_row && dirty) {
      const i64 base = (wrap_plane(p, nfz) * nfy + row_y) * nfx;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int k = v + z;
        if (v == 1 && !has2) break;
        C* row = grid + v * a.grid_bdist + base;
        if (pairs) {
          C* r = row + gx0;
#pragma unroll
          for (int q = 0; q < S::NP; ++q) {
            if (2 * q + 1 < S::P0) {
              if (NNB_CHECK_INDEX(base + gx0 + 2 * q + 1, cells)) {
                atomic_add_pair(r + 2 * q, Ops::lo(are[k][q]), Ops::lo(aim[k][q]),
                                Ops::hi(are[k][q]), Ops::hi(aim[k][q]));
              }
            } else if (NNB_CHECK_INDEX(base + gx0 + 2 * q, cells)) {
              atomic_add_cplx(r + 2 * q, C{Ops::lo(are[k][q]), Ops::lo(aim[k][q])});
            }
          }
        } else {
#pragma unroll
          for (int q = 0; q < S::NP; ++q) {
            const i64 x0 = wrap_x(gx0, 2 * q, nfx, narrow);
            if (NNB_CHECK_INDEX(base + x0, cells)) {
              atomic_add_cplx(&row[x0], C{Ops::lo(are[k][q]), Ops::lo(aim[k][q])});
            }
            const i64 x1 = wrap_x(gx0, 2 * q + 1, nfx, narrow);
            if (2 * q + 1 < S::P0 && NNB_CHECK_INDEX(base + x1, cells)) {
              atomic_add_cplx(&row[x1], C{Ops::hi(are[k][q]), Ops::hi(aim[k][q])});
            }
          }
        }
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) {
#pragma unroll
        for (int q = 0; q < S::NP; ++q) are[v + z][q] = aim[v + z][q] = Ops::zero();
      }
    }
    if (PZ == 1) dirty = false;
  };
  using Z0 = std::integral_constant<int, 0>;
  using Z1 = std::integral_constant<int, PZ - 1>;

  const u32 npts = cta.pend - cta.pbeg;
  const int nbatch = int((npts + S::BATCH - 1) / S::BATCH);
  auto stage = [&](int k) {
    const u32 off = u32(k) * S::BATCH;
    const int nb = int(min(npts - off, u32(S::BATCH)));
    constexpr int PW = S::PW;
    const int count = min(nb - th.warp * PW, PW);
    for (int c0 = 0; c0 < count; c0 += 16) {
      if (!NNB_CHECK_INDEX(i64(cta.pbeg) + off + th.warp * PW + c0 + min(count - c0, 16) - 1,
                           a.pts.M)) {
        break;
      }
      // NV = 2: the second vector's strengths at the same points (zeros when it is missing)
      stage_warp<T, W, TX, true, TY, PZ, POLY>(slots[k & 1] + th.warp * PW + c0,
                                 a.pts.rec + cta.pbeg + off + th.warp * PW + c0,
                                 min(count - c0, 16), in, a.prephase, a.es, a.beta, a.c, th.lane,
                                 a.pts.M, NV > 1 && has2 ? in + a.in_bdist : nullptr,
                                 NV > 1 ? sh.v2[k & 1] + th.warp * PW + c0 : nullptr);
    }
  };

  stage(0);
  __syncthreads();
  int cur = slots[0][0].lyp >> 4;  // window start: the first point's plane
  int dz = S::offset(th.rb, cur);
  for (int k = 0; k < nbatch; ++k) {
    const int nb = int(min(npts - u32(k) * S::BATCH, u32(S::BATCH)));
    const Slot* sb = slots[k & 1];
    constexpr int NH = (S::BATCH + 31) / 32;
    if constexpr (NV == 1) {
      // The points of this batch whose footprint covers rows of this warp, one bit per slot:
      // the warp visits only those, with a window of its own (no other warp touches its rows).
      u32 own[NH];
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        const int j = h * 32 + th.lane;
        own[h] = __ballot_sync(0xffffffffu, j < nb && th.owns(sb[j < nb ? j : 0].lyp & 15));
      }
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        for (u32 m = own[h]; m != 0u; m &= m - 1u) {
          const int si = h * 32 + __ffs(int(m)) - 1;
          const Slot& sl = sb[si];
          const int tp = sl.lyp >> 4;
          if (tp != cur) {  // advance the window: planes [cur, tp) are complete
            if constexpr (S::WIDE) {
              if (dz < tp - cur) flush(Z0{}, cur + dz);
            } else {  // (by dz < tp - cur as above: 4 % slower)
              const int n = min(tp - cur, S::RZ);
              for (int i = 0; i < n; ++i) {
                const int r = (cur + i) & (S::RZ - 1);
                if (th.rb == r) flush(Z0{}, cur + i);
                if (PZ > 1 && th.rb + S::ZL == r) flush(Z1{}, cur + i);
              }
            }
            cur = tp;
            dz = S::offset(th.rb, cur);
          }
          dirty = true;
          const T ky = sl.ky[th.ra];
          const C v = sl.v;
          P wre[PZ], wim[PZ];
#pragma unroll
          for (int z = 0; z < PZ; ++z) {  // planes rb and rb + ZL = RZ / 2: offsets dz, dz ^ ZL
            const T kw = ky * sl.kz[z ? dz ^ S::ZL : dz];
            wre[z] = Ops::splat(v.x * kw);
            wim[z] = Ops::splat(v.y * kw);
          }
#pragma unroll
          for (int q = 0; q < S::NP; q += 2) {
            P kk[2];
            load_pairs<T>(&sl.kx[2 * q], kk);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              if (q + u < S::NP) {
#pragma unroll
                for (int z = 0; z < PZ; ++z) {
                  are[z][q + u] = Ops::fma(kk[u], wre[z], are[z][q + u]);
                  aim[z][q + u] = Ops::fma(kk[u], wim[z], aim[z][q + u]);
                }
              }
            }
          }
        }
      }
    } else {
      // Two vectors: the owned points are visited one plane at a time (the slots are in plane
      // order), so that the window moves once per plane and the loop over a plane's points
      // holds only the loads and the FMAs. (Measured at 1e8 points on a 512^3 grid, w = 8,
      // tiles 4 x 4 x 1: 28.8 ms per two-vector pass against 32.7 ms with the single-vector
      // loop; that loop stays the faster one for one vector, 17.3 against 17.7 ms.)
      u32 own[NH];
      int pl[NH];  // plane of slot 32 h + lane
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        const int j = h * 32 + th.lane;
        const int lyp = sb[j < nb ? j : 0].lyp;
        pl[h] = lyp >> 4;
        own[h] = __ballot_sync(0xffffffffu, j < nb && th.owns(lyp & 15));
      }
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        u32 m = own[h];
        while (m != 0u) {
          const int tp = __shfl_sync(0xffffffffu, pl[h], __ffs(int(m)) - 1);
          const u32 run = m & __ballot_sync(0xffffffffu, pl[h] == tp);
          m &= ~run;
          if (tp != cur) {  // advance the window: planes [cur, tp) are complete
            const int n = min(tp - cur, S::RZ);  // (by dz < tp - cur as for wide kernels: 4 % slower)
            for (int i = 0; i < n; ++i) {
              if (th.rb == ((cur + i) & (S::RZ - 1))) flush(Z0{}, cur + i);
            }
            cur = tp;
            dz = S::offset(th.rb, cur);
          }
          dirty = true;
          for (u32 r = run; r != 0u; r &= r - 1u) {
            const int si = h * 32 + __ffs(int(r)) - 1;
            const Slot& sl = sb[si];
            const T kw = sl.ky[th.ra] * sl.kz[dz];
            P wre[NV], wim[NV];
            {
              const C v = sl.v;
              wre[0] = Ops::splat(v.x * kw);
              wim[0] = Ops::splat(v.y * kw);
              const C v2 = sh.v2[k & 1][si];
              wre[1] = Ops::splat(v2.x * kw);
              wim[1] = Ops::splat(v2.y * kw);
            }
#pragma unroll
            for (int q = 0; q < S::NP; q += 2) {
              P kk[2];
              load_pairs<T>(&sl.kx[2 * q], kk);
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                if (q + u < S::NP) {
#pragma unroll
                  for (int v = 0; v < NV; ++v) {
                    are[v][q + u] = Ops::fma(kk[u], wre[v], are[v][q + u]);
                    aim[v][q + u] = Ops::fma(kk[u], wim[v], aim[v][q + u]);
                  }
                }
              }
            }
          }
        }
      }
    }
    if (k + 1 < nbatch) stage(k + 1);
    __syncthreads();
  }
  flush(Z0{}, cur + dz);  // the rest of the window
  if (PZ > 1) flush(Z1{}, cur + (dz ^ S::ZL));
}

// Double precision is held to 100 registers (5 CTAs of 128 threads): uncapped, ptxas takes 106
// and 3e6 clustered points spread in 1.59 instead of 1.19 ms.
template <typename T, int W, int TX, int TY>
__global__ void __launch_bounds__(ZShape<T, W, TX, TY>::NT,
                                  sizeof(T) == 8 && TX == 4 ? 65536 / (ZShape<T, W, TX, TY>::NT * 100) : 0)
    spread_zwin_kernel(const __grid_constant__ SpreadArgs<T> a, ZChunks ch,
                       const __grid_constant__ WorkList wl) {
  __shared__ ZSpreadShared<T, W, TX, TY> sh;
  spread_zwin_item<T, W, TX, TY>(a, ch, wl, blockIdx.x, int(blockIdx.y), sh);
}

// Kernel widths above 8.
template <typename T, int W, int TX, int TY>
__global__ void __launch_bounds__(ZShape<T, W, TX, TY>::NT, ZShape<T, W, TX, TY>::WIDE_CTAS)
    spread_zwin_wide_kernel(const __grid_constant__ SpreadArgs<T> a, ZChunks ch,
                            const __grid_constant__ WorkList wl) {
  __shared__ ZSpreadShared<T, W, TX, TY> sh;
  spread_zwin_item<T, W, TX, TY>(a, ch, wl, blockIdx.x, int(blockIdx.y), sh);
}

// Two planes per thread.
template <typename T, int W, int TX, int TY>
__global__ void __launch_bounds__(ZShape<T, W, TX, TY, 2>::NT,
                                  ZShape<T, W, TX, TY, 2>::SPREAD_CTAS)
    spread_zwin_planes_kernel(const __grid_constant__ SpreadArgs<T> a, ZChunks ch,
                              const __grid_constant__ WorkList wl) {
  __shared__ ZSpreadShared<T, W, TX, TY, 1, 2> sh;
  spread_zwin_item<T, W, TX, TY, 1, 2>(a, ch, wl, blockIdx.x, int(blockIdx.y), sh);
}

// Two strength vectors per CTA: batch entries 2 blockIdx.y and 2 blockIdx.y + 1.
template <typename T, int W, int TX, int TY>
__global__ void __launch_bounds__(ZShape<T, W, TX, TY>::NT, ZShape<T, W, TX, TY>::SPREAD2_CTAS)
    spread_zwin2_kernel(const __grid_constant__ SpreadArgs<T> a, ZChunks ch,
                        const __grid_constant__ WorkList wl) {
  __shared__ ZSpreadShared<T, W, TX, TY, 2> sh;
  spread_zwin_item<T, W, TX, TY, 2>(a, ch, wl, blockIdx.x, 2 * int(blockIdx.y), sh);
}

// ---- interpolation -----------------------------------------------------------------------------
template <typename T, int W, int TX, int TY = 8, int PZ = 1>
struct ZInterpShared {
  using S = ZShape<T, W, TX, TY, PZ>;
  static constexpr int RS = 33;  // odd row stride of the transpose buffer: conflict-free reads
  ZSlot<T, W, TX, TY, PZ> slots[2][S::BATCH];
  cplx_t<T> red[S::NWARP][S::G][RS];
  cplx_t<T> res[2][S::NWARP][S::BATCH];
};

// Interpolates work item `item` (one CTA; every thread calls it).
template <typename T, int W, int TX, int TY = 8, int PZ = 1>
__device__ __forceinline__ void interp_zwin_item(const InterpArgs<T>& a, ZChunks ch,
                                                 const WorkList& wl, u32 item,
                                                 ZInterpShared<T, W, TX, TY, PZ>& sh) {
  using S = ZShape<T, W, TX, TY, PZ>;
  using Ops = Packed<T>;
  using P = typename Ops::P;
  using C = cplx_t<T>;
  using Slot = ZSlot<T, W, TX, TY, PZ>;
  constexpr int G = S::G;
  auto& slots = sh.slots;
  auto& red = sh.red;
  auto& res = sh.res;

  const BinGeom& g = a.g;
  ZCta cta;
  if (!zcta(g, a.pts.bin_start, ch, wl, item, cta)) return;
  const ZThread<T, W, TX, TY, PZ> th;
  const C* grid = a.grid;
  const i64 nfx = g.nf[0], nfy = g.nf[1], nfz = g.nf[2];
  [[maybe_unused]] const i64 cells = nfx * nfy * nfz;
  const bool narrow = nfx < S::P0;
  const bool has_row = th.active && th.ra < S::P1;
  const i64 row_y = has_row ? wrap_add(i64(cta.ty) * S::TY, th.ra, nfy) : 0;
  const i64 gx0 = i64(cta.tx) * TX;

  // Row values of the window plane: real / imaginary parts of cell pairs (2q, 2q + 1); rows
  // outside the region stay zero.
  P gre[PZ][S::NP], gim[PZ][S::NP];
#pragma unroll
  for (int z = 0; z < PZ; ++z) {
#pragma unroll
    for (int q = 0; q < S::NP; ++q) gre[z][q] = gim[z][q] = Ops::zero();
  }
  // The region's x range lies inside the grid (the usual case): contiguous row segments.
  const bool contiguous = !narrow && gx0 + S::P0 <= nfx;
  // ... and its cell pairs start 16-byte aligned (single precision): one 16-byte load per pair
  const bool pairs16 = sizeof(T) == 4 && contiguous && (nfx % 2) == 0 &&
                       (reinterpret_cast<size_t>(grid) % 16) == 0;
  auto load_row = [&](auto zc, int p) {
    constexpr int z = decltype(zc)::value;
    if (!has_row) return;
    const i64 base = (wrap_plane(p, nfz) * nfy + row_y) * nfx;
    const C* row = grid + base;
    if constexpr (sizeof(T) == 4) {
      if (pairs16) {
#pragma unroll
        for (int q = 0; q < S::NP; ++q) {
          if (2 * q + 1 < S::P0) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (NNB_CHECK_INDEX(base + gx0 + 2 * q + 1, cells)) {
              v = *reinterpret_cast<const float4*>(row + gx0 + 2 * q);
            }
            gre[z][q] = Ops::pack(v.x, v.z);
            gim[z][q] = Ops::pack(v.y, v.w);
          } else {
            C c0{T(0), T(0)};
            if (NNB_CHECK_INDEX(base + gx0 + 2 * q, cells)) c0 = row[gx0 + 2 * q];
            gre[z][q] = Ops::pack(c0.x, T(0));
            gim[z][q] = Ops::pack(c0.y, T(0));
          }
        }
        return;
      }
    }
#pragma unroll
    for (int q = 0; q < S::NP; ++q) {
      C c0{T(0), T(0)}, c1{T(0), T(0)};
      const i64 x0 = contiguous ? gx0 + 2 * q : wrap_x(gx0, 2 * q, nfx, narrow);
      const i64 x1 = contiguous ? gx0 + 2 * q + 1 : wrap_x(gx0, 2 * q + 1, nfx, narrow);
      if (NNB_CHECK_INDEX(base + x0, cells)) c0 = row[x0];
      if (2 * q + 1 < S::P0 && NNB_CHECK_INDEX(base + x1, cells)) c1 = row[x1];
      gre[z][q] = Ops::pack(c0.x, c1.x);
      gim[z][q] = Ops::pack(c0.y, c1.y);
    }
  };
  const u32 npts = cta.pend - cta.pbeg;
  const int nbatch = int((npts + S::BATCH - 1) / S::BATCH);
  auto stage = [&](int k) {
    const u32 off = u32(k) * S::BATCH;
    const int nb = int(min(npts - off, u32(S::BATCH)));
    constexpr int PW = S::PW;
    const int count = min(nb - th.warp * PW, PW);
    for (int c0 = 0; c0 < count; c0 += 16) {
      if (!NNB_CHECK_INDEX(i64(cta.pbeg) + off + th.warp * PW + c0 + min(count - c0, 16) - 1,
                           a.pts.M)) {
        break;
      }
      stage_warp<T, W, TX, false, TY, PZ>(slots[k & 1] + th.warp * PW + c0,
                                  a.pts.rec + cta.pbeg + off + th.warp * PW + c0,
                                  min(count - c0, 16), nullptr, nullptr, a.es, a.beta, a.c, th.lane,
                                  a.pts.M);
    }
  };
  // Writes the outputs of batch k: this thread's staged point, whose slot only this thread's
  // next staging rewrites.
  auto output = [&](int k) {
    const int nb = int(min(npts - u32(k) * S::BATCH, u32(S::BATCH)));
    const int j = th.stage_j;
    if (j >= 0 && j < nb) {
      C r = res[k & 1][0][j];
#pragma unroll
      for (int w = 1; w < S::NWARP; ++w) {
        r.x += res[k & 1][w][j].x;
        r.y += res[k & 1][w][j].y;
      }
      const u32 perm = slots[k & 1][j].perm;
      if (NNB_CHECK_INDEX(perm, a.pts.M)) {
        if (a.postphase) r = cmul(r, a.postphase[perm]);
        a.out[perm] = r;
      }
    }
  };

  stage(0);
  __syncthreads();
  int cur = slots[0][0].lyp >> 4;  // window start: the first point's plane
  int dz = S::offset(th.rb, cur);
  using Z0 = std::integral_constant<int, 0>;
  using Z1 = std::integral_constant<int, PZ - 1>;
  load_row(Z0{}, cur + dz);
  if (PZ > 1) load_row(Z1{}, cur + (dz ^ S::ZL));

  for (int k = 0; k < nbatch; ++k) {
    const int nb = int(min(npts - u32(k) * S::BATCH, u32(S::BATCH)));
    const Slot* sb = slots[k & 1];
    // The points of this batch whose footprint covers rows of this warp (bit j: slot j).
    unsigned long long own = 0ull;
#pragma unroll
    for (int h = 0; h < (S::BATCH + 31) / 32; ++h) {
      const int j = h * 32 + th.lane;
      const u32 bits = __ballot_sync(0xffffffffu, j < nb && th.owns(sb[j < nb ? j : 0].lyp & 15));
      own |= (unsigned long long)bits << (32 * h);
    }
    // Row sum of an owned point over this thread's row, times ky kz.
    auto partial = [&](const Slot& sl) -> C {
      // one plane: two chains, over the even and the odd pairs; two planes: a chain each
      P sr[2], si[2];
      sr[0] = sr[1] = si[0] = si[1] = Ops::zero();
#pragma unroll
      for (int q = 0; q < S::NP; q += 2) {
        P kp[2];
        load_pairs<T>(&sl.kx[2 * q], kp);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (q + u >= S::NP) continue;
#pragma unroll
          for (int z = 0; z < PZ; ++z) {
            const int k = PZ > 1 ? z : u;
            sr[k] = Ops::fma(kp[u], gre[z][q + u], sr[k]);
            si[k] = Ops::fma(kp[u], gim[z][q + u], si[k]);
          }
        }
      }
      const T ky = sl.ky[th.ra];
      if constexpr (PZ > 1) {
        const P k0 = Ops::splat(sl.kz[dz]), k1 = Ops::splat(sl.kz[dz ^ S::ZL]);
        const P r = Ops::fma(k0, sr[0], Ops::fma(k1, sr[1], Ops::zero()));
        const P i = Ops::fma(k0, si[0], Ops::fma(k1, si[1], Ops::zero()));
        return C{ky * (Ops::lo(r) + Ops::hi(r)), ky * (Ops::lo(i) + Ops::hi(i))};
      } else {
        const T kw = ky * sl.kz[dz];
        const P r = Ops::add(sr[0], sr[1]);
        const P i = Ops::add(si[0], si[1]);
        return C{kw * (Ops::lo(r) + Ops::hi(r)), kw * (Ops::lo(i) + Ops::hi(i))};
      }
    };
    for (int j0 = 0; j0 < nb; j0 += G) {
      // Points are plane-sorted: if the group's last point is on the window's first plane, so
      // are all of them and the window does not move inside the group.
      // ownership bits of the group (bit kk: slot j0 + kk); zero past the batch's points
      const u32 ob = u32(own >> j0);
      if ((sb[min(j0 + G, nb) - 1].lyp >> 4) == cur) {
        const Slot* g0 = sb + j0;
#pragma unroll
        for (int kk = 0; kk < G; ++kk) {
          red[th.warp][kk][th.lane] = ((ob >> kk) & 1u) ? partial(g0[kk]) : C{T(0), T(0)};
        }
      } else {
#pragma unroll 1
        for (int kk = 0; kk < G; ++kk) {
          C part{T(0), T(0)};
          const int j = j0 + kk;
          if (j < nb) {
            const Slot& sl = sb[j];
            const int lyp = sl.lyp;
            const int tp = lyp >> 4;
            if (tp != cur) {  // advance the window: rows of planes [cur, tp) move on by RZ
              if constexpr (S::WIDE) {
                if (dz < tp - cur) load_row(Z0{}, tp + S::offset(th.rb, tp));
              } else if (tp - cur >= S::RZ) {
                const int nz = S::offset(th.rb, tp);
                load_row(Z0{}, tp + nz);
                if (PZ > 1) load_row(Z1{}, tp + (nz ^ S::ZL));
              } else {
                for (int i = 0; i < tp - cur; ++i) {
                  const int r = (cur + i) & (S::RZ - 1);
                  if (th.rb == r) load_row(Z0{}, cur + i + S::RZ);
                  if (PZ > 1 && th.rb + S::ZL == r) load_row(Z1{}, cur + i + S::RZ);
                }
              }
              cur = tp;
              dz = S::offset(th.rb, cur);
            }
            if ((ob >> kk) & 1u) part = partial(sl);
          }
          red[th.warp][kk][th.lane] = part;
        }
      }
      __syncwarp();
      {
        // lane (k8, q4): sum of G lanes' partials of point j0 + k8, then over the 32 / G parts
        const int k8 = th.lane & (G - 1);
        const int q4 = th.lane / G;
        C sum{T(0), T(0)};
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const C v = red[th.warp][k8][q4 * G + i];
          sum.x += v.x;
          sum.y += v.y;
        }
#pragma unroll
        for (int o = G; o < 32; o <<= 1) {
          sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o);
          sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
        }
        if (q4 == 0) res[k & 1][th.warp][j0 + k8] = sum;
      }
      __syncwarp();
    }
    if (k > 0) output(k - 1);
    if (k + 1 < nbatch) stage(k + 1);
    __syncthreads();
  }
  output(nbatch - 1);
}

template <typename T, int W, int TX, int TY, int PZ = 1>
__global__ void __launch_bounds__(ZShape<T, W, TX, TY, PZ>::NT,
                                  ZShape<T, W, TX, TY, PZ>::INTERP_CTAS)
    interp_zwin_kernel(const __grid_constant__ InterpArgs<T> a, ZChunks ch,
                       const __grid_constant__ WorkList wl) {
  if constexpr (ZShape<T, W, TX, TY>::WIDE) {  // more than the 48 KB of static shared memory
    extern __shared__ __align__(16) unsigned char smem_raw[];
    interp_zwin_item<T, W, TX, TY>(a, ch, wl, blockIdx.x,
                                   *reinterpret_cast<ZInterpShared<T, W, TX, TY>*>(smem_raw));
  } else {
    __shared__ ZInterpShared<T, W, TX, TY, PZ> sh;
    interp_zwin_item<T, W, TX, TY, PZ>(a, ch, wl, blockIdx.x, sh);
  }
}

}  // namespace

}  // namespace nnb
