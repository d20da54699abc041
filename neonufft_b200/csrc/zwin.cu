// Launchers of the z-window kernels (zwin.cuh) for kernel widths up to 8, the persistent kernels
// over many transforms, and the spreading on tensor cores (method 4).
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "zwin.cuh"

namespace nnb {

namespace {

// Takes the next item of the queue spanning all jobs; every thread returns the same values.
// The job's record is copied to shared memory once per item.
template <typename Job>
__device__ __forceinline__ bool next_fused_item(const Job* jobs, const i64* item_end, int njobs,
                                                i64 total, u32* queue, Job& job, u32& local) {
  __shared__ i64 s_item;
  __shared__ int s_job;
  if (threadIdx.x == 0) {
    const i64 it = i64(atomicAdd(queue, 1u));
    int lo = 0, hi = njobs;  // first job whose cumulative item count exceeds it
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (item_end[mid] > it) {
        hi = mid;
      } else {
        lo = mid + 1;
      }
    }
    s_item = it;
    s_job = lo;
  }
  __syncthreads();
  const i64 it = s_item;
  const int j = s_job;
  if (it >= total || j >= njobs) return false;
  static_assert(sizeof(Job) % 4 == 0, "job records are copied in words");
  const int* src = reinterpret_cast<const int*>(jobs + j);
  int* dst = reinterpret_cast<int*>(&job);
  for (int k = int(threadIdx.x); k < int(sizeof(Job) / 4); k += int(blockDim.x)) dst[k] = src[k];
  local = u32(it - (j > 0 ? item_end[j - 1] : 0));
  __syncthreads();
  return true;
}

// Window planes per thread (ZShape::PZ) of the kernels of one transform.
template <typename T, int W, int TX, int TY>
constexpr int zwin_planes = sizeof(T) == 4 && W >= 5 && TX == 4 && TY <= 8 ? 2 : 1;

// Kernel values as the launches of one transform take them, but one plane per thread: 24 type-1
// transforms of 1e4 to 3e6 points, w = 8, single precision, in 6.36 ms (one plane, 5 CTAs per SM;
// 6.45 and 6.49 with 6 and 7) against 7.10 to 7.40 (two planes, 8 to 11 CTAs) and 7.00 (the
// formula, 7 CTAs).
template <typename T, int W, int TX>
constexpr bool fused_poly = zspread_poly<T, W, 8, 1, zwin_planes<T, W, TX, 8>>;

template <typename T, int W, int TX>
__global__ void __launch_bounds__(ZShape<T, W, TX>::NT,
                                  sizeof(T) == 4 && fused_poly<T, W, TX> ? 5 : kSpreadFusedCtas<T>)
    spread_zwin_fused_kernel(const ZSpreadJob<T>* jobs, const i64* item_end, int njobs,
                             i64 total, u32* queue) {
  __shared__ ZSpreadShared<T, W, TX> sh;
  __shared__ ZSpreadJob<T> job;
  u32 local;
  while (next_fused_item(jobs, item_end, njobs, total, queue, job, local)) {
    spread_zwin_item<T, W, TX, 8, 1, 1, fused_poly<T, W, TX>>(job.a, job.ch, job.wl, local, 0, sh);
    __syncthreads();  // the job record and the slots are rewritten for the next item
  }
}

// ---- spreading on the tensor cores (method 4, single precision, 5 <= w <= 8) ---------------------
//
// The same window, staging and flushes as spread_zwin_kernel, with the per-point row updates
// replaced by TF32 tensor-core products. For a chunk of up to 8 points of the current plane,
//   region[x, (plane, y)] += sum_p kx_p[x] * (v_p ky_p[y] kz_p[plane])
// is, for each tile of one plane and 8 rows, a 16 x 8 x 8 matrix product (mma.sync m16n8k8:
// M = the 16 x cells of the region, K = the points, N = the rows). Both operands are split into
// a TF32 value and a TF32 remainder and the product accumulated as hi*hi + hi*lo + lo*hi in FP32
// (about 2^-21 of each product). Warp w owns window planes 2w, 2w + 1 (mod 8) and both 8-row y
// groups: four tiles, real and imaginary accumulators in registers; in the m16n8k8 fragment
// layout thread (q, t) = (lane / 4, lane % 4) holds x = q, q + 8 and rows 2t, 2t + 1 of a tile.
// A completed plane is added to the grid by its owning warp (all 32 lanes, float2 atomics).

__device__ __forceinline__ unsigned to_tf32(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void tf32_split(float x, unsigned& hi, unsigned& lo) {
  hi = to_tf32(x);
  lo = to_tf32(x - __uint_as_float(hi));
}
// c += a * b for one m16n8k8 TF32 tile (FP32 accumulation)
__device__ __forceinline__ void mma_tf32(float* c, const unsigned* a, unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += a * b with both operands split (3 products). The products of one chunk are summed on the
// tensor core into a fresh tile and added to the accumulator with ordinary FP32 adds: chaining
// the accumulator through every MMA of a long run of points loses accuracy.
__device__ __forceinline__ void mma_tf32x3(float* c, const unsigned* ahi, const unsigned* alo,
                                           float b0, float b1) {
  unsigned b0h, b0l, b1h, b1l;
  tf32_split(b0, b0h, b0l);
  tf32_split(b1, b1h, b1l);
  float t[4] = {0.f, 0.f, 0.f, 0.f};
  mma_tf32(t, alo, b0h, b1h);
  mma_tf32(t, ahi, b0l, b1l);
  mma_tf32(t, ahi, b0h, b1h);
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] += t[e];
}

template <int W>
__global__ void __launch_bounds__(128) spread_zmma_kernel(SpreadArgs<float> a, ZChunks ch,
                                                          WorkList wl) {
  constexpr int TX = 8;
  using S = ZShape<float, W, TX>;
  static_assert(S::RZ == 8 && S::NWARP == 4 && S::P0 <= 16, "tile shapes");
  using C = float2;
  using Slot = ZSlot<float, W, TX>;
  __shared__ Slot slots[2][S::BATCH];

  const BinGeom& g = a.g;
  ZCta cta;
  if (!zcta(g, a.pts.bin_start, ch, wl, blockIdx.x, cta)) return;
  const ZThread<float, W, TX> th;
  const int gq = th.lane >> 2;  // fragment row group
  const int tq = th.lane & 3;   // thread in group
  const bool hi8 = gq + 8 < S::KXN;  // staged kx covers x = gq + 8 (cells beyond it are zero)
  const int batch = blockIdx.y;
  const C* in = a.in + batch * a.in_bdist;
  C* grid = a.grid + batch * a.grid_bdist;
  const i64 nfx = g.nf[0], nfy = g.nf[1], nfz = g.nf[2];
  const bool narrow = nfx < S::P0;
  const i64 gx0 = i64(cta.tx) * TX;
  const i64 gy0 = i64(cta.ty) * S::TY;

  float cre[2][2][4], cim[2][2][4];  // [plane of the warp][y group][fragment element]
#pragma unroll
  for (int pl = 0; pl < 2; ++pl) {
#pragma unroll
    for (int yg = 0; yg < 2; ++yg) {
#pragma unroll
      for (int e = 0; e < 4; ++e) cre[pl][yg][e] = cim[pl][yg][e] = 0.f;
    }
  }
  unsigned dirty = 0;  // plane residues with contributions since their last flush

  // Adds the warp's tiles of window plane p (residue 2 warp + pl) to the grid and clears them.
  auto flush = [&](int pl, int p) {
    const unsigned bit = 1u << (2 * th.warp + pl);
    if (dirty & bit) {
      const i64 plane = wrap_plane(p, nfz);
#pragma unroll
      for (int yg = 0; yg < 2; ++yg) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int x = gq + 8 * (e >> 1);
          const int y = 8 * yg + 2 * tq + (e & 1);
          if (x < S::P0 && y < S::P1) {
            const i64 gy = wrap_add(gy0, y, nfy);
            const i64 idx = (plane * nfy + gy) * nfx + wrap_x(gx0, x, nfx, narrow);
            if (NNB_CHECK_INDEX(idx, nfx * nfy * nfz)) {
              atomic_add_cplx(&grid[idx], C{cre[pl][yg][e], cim[pl][yg][e]});
            }
          }
          cre[pl][yg][e] = cim[pl][yg][e] = 0.f;
        }
      }
      dirty &= ~bit;
    }
  };
  auto flush_plane = [&](int p) {
    const int b = p & 7;
    if ((b >> 1) == th.warp) flush(b & 1, p);
  };

  const u32 npts = cta.pend - cta.pbeg;
  const int nbatch = int((npts + S::BATCH - 1) / S::BATCH);
  auto stage = [&](int k) {
    const u32 off = u32(k) * S::BATCH;
    const int nb = int(min(npts - off, u32(S::BATCH)));
    constexpr int PW = S::BATCH / S::NWARP;
    const int count = min(nb - th.warp * PW, PW);
    for (int c0 = 0; c0 < count; c0 += 16) {
      if (!NNB_CHECK_INDEX(i64(cta.pbeg) + off + th.warp * PW + c0 + min(count - c0, 16) - 1,
                           a.pts.M)) {
        break;
      }
      stage_warp<float, W, TX, true>(slots[k & 1] + th.warp * PW + c0,
                                     a.pts.rec + cta.pbeg + off + th.warp * PW + c0,
                                     min(count - c0, 16), in, a.prephase, a.es, a.beta, a.c, th.lane,
                                     a.pts.M);
    }
  };

  stage(0);
  __syncthreads();
  int cur = slots[0][0].lyp >> 4;
  int dz0 = (2 * th.warp - cur) & 7, dz1 = (2 * th.warp + 1 - cur) & 7;
  for (int k = 0; k < nbatch; ++k) {
    const int nb = int(min(npts - u32(k) * S::BATCH, u32(S::BATCH)));
    const Slot* sb = slots[k & 1];
    int j = 0;
    while (j < nb) {
      const int tp = sb[j].lyp >> 4;
      if (tp != cur) {  // advance the window: planes [cur, tp) are complete
        const int n = min(tp - cur, S::RZ);
        for (int i = 0; i < n; ++i) flush_plane(cur + i);
        cur = tp;
        dz0 = (2 * th.warp - cur) & 7;
        dz1 = (2 * th.warp + 1 - cur) & 7;
      }
      // the chunk: points j .. j + n - 1 of plane cur (a prefix, the points are plane-sorted)
      const bool on = th.lane < 8 && j + th.lane < nb && (sb[min(j + th.lane, nb - 1)].lyp >> 4) == cur;
      const int n = __popc(__ballot_sync(0xffffffffu, on));
      const bool h0 = tq < n, h1 = tq + 4 < n;
      const Slot& s0 = sb[h0 ? j + tq : j];
      const Slot& s1 = sb[h1 ? j + tq + 4 : j];
      // A: kx of points tq, tq + 4 at x = gq, gq + 8
      unsigned ahi[4], alo[4];
      tf32_split(h0 ? s0.kx[gq] : 0.f, ahi[0], alo[0]);
      tf32_split(h0 && hi8 ? s0.kx[gq + 8] : 0.f, ahi[1], alo[1]);
      tf32_split(h1 ? s1.kx[gq] : 0.f, ahi[2], alo[2]);
      tf32_split(h1 && hi8 ? s1.kx[gq + 8] : 0.f, ahi[3], alo[3]);
      // B: v ky kz of points tq, tq + 4 at row gq of each tile
      const C v0 = h0 ? s0.v : C{0.f, 0.f};
      const C v1 = h1 ? s1.v : C{0.f, 0.f};
      const float y00 = s0.ky[gq], y01 = s0.ky[gq + 8], z00 = s0.kz[dz0], z01 = s0.kz[dz1];
      const float y10 = s1.ky[gq], y11 = s1.ky[gq + 8], z10 = s1.kz[dz0], z11 = s1.kz[dz1];
#pragma unroll
      for (int pl = 0; pl < 2; ++pl) {
#pragma unroll
        for (int yg = 0; yg < 2; ++yg) {
          const float w0 = (yg ? y01 : y00) * (pl ? z01 : z00);
          const float w1 = (yg ? y11 : y10) * (pl ? z11 : z10);
          mma_tf32x3(cre[pl][yg], ahi, alo, v0.x * w0, v1.x * w1);
          mma_tf32x3(cim[pl][yg], ahi, alo, v0.y * w0, v1.y * w1);
        }
      }
      dirty = 0xffu;
      j += n;
    }
    if (k + 1 < nbatch) stage(k + 1);
    __syncthreads();
  }
  for (int i = 0; i < S::RZ; ++i) flush_plane(cur + i);  // the rest of the window
}

template <typename T, int W, int TX>
__global__ void __launch_bounds__(ZShape<T, W, TX>::NT, kInterpFusedCtas<T>)
    interp_zwin_fused_kernel(const ZInterpJob<T>* jobs, const i64* item_end, int njobs,
                             i64 total, u32* queue) {
  __shared__ ZInterpShared<T, W, TX> sh;
  __shared__ ZInterpJob<T> job;
  u32 local;
  while (next_fused_item(jobs, item_end, njobs, total, queue, job, local)) {
    interp_zwin_item<T, W, TX>(job.a, job.ch, job.wl, local, sh);
    __syncthreads();  // the job record and the shared buffers are rewritten for the next item
  }
}

}  // namespace

ZChunks make_chunks(i64 ncols, int nz, int w) {
  // About four waves of 8 CTAs per SM; chunks of at least 4 w planes bound the window
  // overhead (w - 1 extra planes flushed, or RZ planes loaded, per chunk).
  const i64 target = 148 * 8 * 4;
  i64 count = (target + ncols - 1) / ncols;
  int min_len = 4 * w;
  // A wide point takes a CTA long: on grids of few columns shorter chunks, until there are two for
  // each SM (3e4 uniform points on 32^3 cells, w = 10, double precision: spreading 209 us with
  // chunks of 4 w planes, 47 with 4; shared-memory slabs 173; interpolation 230, 52 and 121).
  while (w > 8 && min_len > 4 && ncols * ((nz + min_len - 1) / min_len) < 2 * 148) {
    min_len = std::max(4, min_len / 2);
  }
  const i64 max_count = (nz + min_len - 1) / min_len;
  if (count > max_count) count = max_count;
  if (count < 1) count = 1;
  ZChunks ch;
  ch.len = int((nz + count - 1) / count);
  ch.count = (nz + ch.len - 1) / ch.len;
  return ch;
}

// Launch units of a plane-major point set: (column, chunk) pairs.
UnitMap zwin_unit_map(const BinGeom& g, ZChunks ch) {
  UnitMap m{};
  m.kind = UnitMap::kZwin;
  m.ncols = i64(g.ntiles[0]) * g.ntiles[1];
  m.units = m.ncols * ch.count;
  m.nz = g.ntiles[2];
  m.zlen = ch.len;
  return m;
}

ZChunks zwin_chunks(const BinGeom& g) {
  return make_chunks(i64(g.ntiles[0]) * g.ntiles[1], g.ntiles[2], g.w);
}

// Work list of (column, chunk) units split into items of at most kWorkItemPoints points.
template <typename T>
WorkList zwin_work_list(const BinGeom& g, const SortedPoints<T>& pts, ZChunks ch) {
  const WorkList wl = describe_work_list(zwin_unit_map(g, ch), pts.M, pts.work);
  if (wl.grid > 0x7fffffffll) throw_input("grid too large");
  return wl;
}
template WorkList zwin_work_list<float>(const BinGeom&, const SortedPoints<float>&, ZChunks);
template WorkList zwin_work_list<double>(const BinGeom&, const SortedPoints<double>&, ZChunks);

namespace {

template <typename T, int W, int TX, int TY>
void launch_spread_zwin_tw(const SpreadArgs<T>& a, cudaStream_t stream) {
  using S = ZShape<T, W, TX, TY>;
  const i64 ncols = i64(a.g.ntiles[0]) * a.g.ntiles[1];
  const ZChunks ch = make_chunks(ncols, a.g.ntiles[2], W);
  const WorkList wl = zwin_work_list(a.g, a.pts, ch);
  // Single precision with the default or 4-row tiles spreads two strength vectors per pass
  // when there are several (the second vector costs its FMAs only).
  constexpr bool kPairs = std::is_same<T, float>::value && TX == 4 && (TY == 8 || TY == 4);
  if constexpr (kPairs) {
    if (a.batch > 1) {
      dim3 grid{unsigned(wl.grid), unsigned((a.batch + 1) / 2), 1u};
      spread_zwin2_kernel<T, W, TX, TY><<<grid, S::NT, 0, stream>>>(a, ch, wl);
      NNB_LAUNCH_CHECK();
      return;
    }
  }
  dim3 grid{unsigned(wl.grid), unsigned(a.batch), 1u};
  if constexpr (zwin_planes<T, W, TX, TY> == 2 && TY == 8) {
    spread_zwin_planes_kernel<T, W, TX, TY>
        <<<grid, ZShape<T, W, TX, TY, 2>::NT, 0, stream>>>(a, ch, wl);
  } else {
    spread_zwin_kernel<T, W, TX, TY><<<grid, S::NT, 0, stream>>>(a, ch, wl);
  }
  NNB_LAUNCH_CHECK();
}

template <typename T, int W, int TX, int TY>
void launch_interp_zwin_tw(const InterpArgs<T>& a, cudaStream_t stream) {
  const i64 ncols = i64(a.g.ntiles[0]) * a.g.ntiles[1];
  const ZChunks ch = make_chunks(ncols, a.g.ntiles[2], W);
  const WorkList wl = zwin_work_list(a.g, a.pts, ch);
  constexpr int PZ = zwin_planes<T, W, TX, TY>;
  interp_zwin_kernel<T, W, TX, TY, PZ>
      <<<unsigned(wl.grid), ZShape<T, W, TX, TY, PZ>::NT, 0, stream>>>(a, ch, wl);
  NNB_LAUNCH_CHECK();
}

template <typename T, int TX, int TY>
void spread_zwin_tx(const SpreadArgs<T>& a, cudaStream_t stream) {
  switch (a.g.w) {
    case 2: return launch_spread_zwin_tw<T, 2, TX, TY>(a, stream);
    case 3: return launch_spread_zwin_tw<T, 3, TX, TY>(a, stream);
    case 4: return launch_spread_zwin_tw<T, 4, TX, TY>(a, stream);
    case 5: return launch_spread_zwin_tw<T, 5, TX, TY>(a, stream);
    case 6: return launch_spread_zwin_tw<T, 6, TX, TY>(a, stream);
    case 7: return launch_spread_zwin_tw<T, 7, TX, TY>(a, stream);
    case 8: return launch_spread_zwin_tw<T, 8, TX, TY>(a, stream);
    default: throw_internal("z-window kernels need n_spread <= 8");
  }
}

template <typename T, int TX, int TY>
void interp_zwin_tx(const InterpArgs<T>& a, cudaStream_t stream) {
  switch (a.g.w) {
    case 2: return launch_interp_zwin_tw<T, 2, TX, TY>(a, stream);
    case 3: return launch_interp_zwin_tw<T, 3, TX, TY>(a, stream);
    case 4: return launch_interp_zwin_tw<T, 4, TX, TY>(a, stream);
    case 5: return launch_interp_zwin_tw<T, 5, TX, TY>(a, stream);
    case 6: return launch_interp_zwin_tw<T, 6, TX, TY>(a, stream);
    case 7: return launch_interp_zwin_tw<T, 7, TX, TY>(a, stream);
    case 8: return launch_interp_zwin_tw<T, 8, TX, TY>(a, stream);
    default: throw_internal("z-window kernels need n_spread <= 8");
  }
}

void check_zwin_geom(const BinGeom& g) {
  if (g.dim != 3 || !g.zmajor || (g.tile[1] != 4 && g.tile[1] != 8 && g.tile[1] != 16) ||
      g.tile[2] != 1 ||
      (g.tile[0] != 2 && g.tile[0] != 4 && g.tile[0] != 8) || g.w > 8) {
    throw_internal("z-window kernels need a 3D plane-major (2|4|8, 4|8|16, 1) tiling and n_spread <= 8");
  }
}


// Persistent launches: as many CTAs as fit on the GPU at once, or fewer when there are fewer
// items; each takes items from the shared queue until it is empty.
template <typename K>
unsigned persistent_grid(K kernel, int threads, i64 total) {
  int dev = 0, sms = 0, per_sm = 0;
  NNB_CUDA(cudaGetDevice(&dev));
  NNB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  NNB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0));
  i64 g = i64(sms) * (per_sm > 0 ? per_sm : 1);
  if (g > total) g = total;
  return unsigned(g < 1 ? 1 : g);
}

template <typename T, int W, int TX>
void spread_fused_tw(const ZSpreadJob<T>* jobs, const i64* item_end, int njobs, i64 total,
                     u32* queue, cudaStream_t stream) {
  constexpr int NT = ZShape<T, W, TX>::NT;
  const unsigned grid = persistent_grid(spread_zwin_fused_kernel<T, W, TX>, NT, total);
  spread_zwin_fused_kernel<T, W, TX><<<grid, NT, 0, stream>>>(jobs, item_end, njobs, total,
                                                              queue);
  NNB_LAUNCH_CHECK();
}

template <typename T, int W, int TX>
void interp_fused_tw(const ZInterpJob<T>* jobs, const i64* item_end, int njobs, i64 total,
                     u32* queue, cudaStream_t stream) {
  constexpr int NT = ZShape<T, W, TX>::NT;
  const unsigned grid = persistent_grid(interp_zwin_fused_kernel<T, W, TX>, NT, total);
  interp_zwin_fused_kernel<T, W, TX><<<grid, NT, 0, stream>>>(jobs, item_end, njobs, total,
                                                              queue);
  NNB_LAUNCH_CHECK();
}

// Calls f(std::integral_constant<int, w>) for 2 <= w <= 8.
template <typename F>
void with_width(int w, F&& f) {
  switch (w) {
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 5: return f(std::integral_constant<int, 5>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 7: return f(std::integral_constant<int, 7>{});
    case 8: return f(std::integral_constant<int, 8>{});
    default: throw_internal("z-window kernels need n_spread <= 8");
  }
}

void check_fused(int njobs, i64 total, int tile_x) {
  if (njobs < 1) throw_internal("a persistent launch needs at least one job");
  if (total < 1 || total > 0x7fffffffll) throw_internal("persistent launch item count out of range");
  if (tile_x != 2 && tile_x != 4 && tile_x != 8) {
    throw_internal("z-window kernels need tiles of 2, 4 or 8 in x");
  }
}
}  // namespace

template <int W>
void launch_spread_zmma_w(const SpreadArgs<float>& a, cudaStream_t stream) {
  const i64 ncols = i64(a.g.ntiles[0]) * a.g.ntiles[1];
  const ZChunks ch = make_chunks(ncols, a.g.ntiles[2], W);
  const WorkList wl = zwin_work_list(a.g, a.pts, ch);
  dim3 grid{unsigned(wl.grid), unsigned(a.batch), 1u};
  spread_zmma_kernel<W><<<grid, 128, 0, stream>>>(a, ch, wl);
  NNB_LAUNCH_CHECK();
}

template <typename T>
void launch_spread_zwin(const SpreadArgs<T>& a, cudaStream_t stream) {
  if (a.g.w > 8 && a.method == 3) return launch_spread_zwin_wide<T>(a, stream);
  check_zwin_geom(a.g);
  if (a.batch > 65535) throw_input("batch size above 65535");
  if (a.method == 4) {
    if constexpr (std::is_same<T, float>::value) {
      if (a.g.tile[0] != 8) throw_internal("tensor-core spreading needs tiles of 8 cells in x");
      switch (a.g.w) {
        case 5: return launch_spread_zmma_w<5>(a, stream);
        case 6: return launch_spread_zmma_w<6>(a, stream);
        case 7: return launch_spread_zmma_w<7>(a, stream);
        case 8: return launch_spread_zmma_w<8>(a, stream);
        default: throw_internal("tensor-core spreading needs 5 <= n_spread <= 8");
      }
    }
    throw_internal("tensor-core spreading is single precision");
  }
  if (a.g.tile[1] == 16) {
    if constexpr (std::is_same<T, float>::value) {
      if (a.g.tile[0] == 8) return spread_zwin_tx<T, 8, 16>(a, stream);
      if (a.g.tile[0] == 2) return spread_zwin_tx<T, 2, 16>(a, stream);
      return spread_zwin_tx<T, 4, 16>(a, stream);
    }
    throw_internal("z-window tiles of 16 rows are single precision");
  }
  if (a.g.tile[1] == 4) {
    if constexpr (std::is_same<T, float>::value) {
      if (a.g.tile[0] == 4) return spread_zwin_tx<T, 4, 4>(a, stream);
    }
    throw_internal("z-window tiles of 4 rows are single precision, 4 cells in x");
  }
  if (a.g.tile[0] == 8) return spread_zwin_tx<T, 8, 8>(a, stream);
  if (a.g.tile[0] == 2) return spread_zwin_tx<T, 2, 8>(a, stream);
  return spread_zwin_tx<T, 4, 8>(a, stream);
}

template <typename T>
void launch_interp_zwin(const InterpArgs<T>& a, cudaStream_t stream) {
  if (a.g.w > 8 && a.method == 3) return launch_interp_zwin_wide<T>(a, stream);
  check_zwin_geom(a.g);
  if (a.g.tile[1] == 16) {
    if constexpr (std::is_same<T, float>::value) {
      if (a.g.tile[0] == 8) return interp_zwin_tx<T, 8, 16>(a, stream);
      if (a.g.tile[0] == 2) return interp_zwin_tx<T, 2, 16>(a, stream);
      return interp_zwin_tx<T, 4, 16>(a, stream);
    }
    throw_internal("z-window tiles of 16 rows are single precision");
  }
  if (a.g.tile[1] == 4) {
    if constexpr (std::is_same<T, float>::value) {
      if (a.g.tile[0] == 4) return interp_zwin_tx<T, 4, 4>(a, stream);
    }
    throw_internal("z-window tiles of 4 rows are single precision, 4 cells in x");
  }
  if (a.g.tile[0] == 8) return interp_zwin_tx<T, 8, 8>(a, stream);
  if (a.g.tile[0] == 2) return interp_zwin_tx<T, 2, 8>(a, stream);
  return interp_zwin_tx<T, 4, 8>(a, stream);
}

template <typename T>
ZSpreadJob<T> zwin_spread_job(const SpreadArgs<T>& a) {
  check_zwin_geom(a.g);
  if (a.g.tile[1] != 8) throw_internal("persistent z-window kernels use tiles of 8 rows");
  if (a.method != 3 || a.batch != 1) throw_internal("persistent spreading is method 3, batch 1");
  ZSpreadJob<T> j;
  j.a = a;
  j.ch = zwin_chunks(a.g);
  j.wl = describe_work_list(zwin_unit_map(a.g, j.ch), a.pts.M, a.pts.work);
  return j;
}

template <typename T>
ZInterpJob<T> zwin_interp_job(const InterpArgs<T>& a) {
  check_zwin_geom(a.g);
  if (a.g.tile[1] != 8) throw_internal("persistent z-window kernels use tiles of 8 rows");
  if (a.method != 3) throw_internal("persistent interpolation is method 3");
  ZInterpJob<T> j;
  j.a = a;
  j.ch = zwin_chunks(a.g);
  j.wl = describe_work_list(zwin_unit_map(a.g, j.ch), a.pts.M, a.pts.work);
  return j;
}

template <typename T>
void zwin_build_work_list(const BinGeom& g, const SortedPoints<T>& pts, cudaStream_t stream) {
  if (g.dim != 3 || !g.zmajor) throw_internal("z-window work lists need plane-major points");
  (void)build_work_list(zwin_unit_map(g, zwin_chunks(g)), g, pts.bin_start, pts.M, pts.work,
                        stream);
}

template <typename T>
void launch_spread_zwin_fused(const ZSpreadJob<T>* jobs, const i64* item_end, int njobs,
                              i64 total, int w, int tile_x, u32* queue, cudaStream_t stream) {
  check_fused(njobs, total, tile_x);
  with_width(w, [&](auto wc) {
    constexpr int W = decltype(wc)::value;
    if (tile_x == 8) {
      spread_fused_tw<T, W, 8>(jobs, item_end, njobs, total, queue, stream);
    } else if (tile_x == 2) {
      spread_fused_tw<T, W, 2>(jobs, item_end, njobs, total, queue, stream);
    } else {
      spread_fused_tw<T, W, 4>(jobs, item_end, njobs, total, queue, stream);
    }
  });
}

template <typename T>
void launch_interp_zwin_fused(const ZInterpJob<T>* jobs, const i64* item_end, int njobs,
                              i64 total, int w, int tile_x, u32* queue, cudaStream_t stream) {
  check_fused(njobs, total, tile_x);
  with_width(w, [&](auto wc) {
    constexpr int W = decltype(wc)::value;
    if (tile_x == 8) {
      interp_fused_tw<T, W, 8>(jobs, item_end, njobs, total, queue, stream);
    } else if (tile_x == 2) {
      interp_fused_tw<T, W, 2>(jobs, item_end, njobs, total, queue, stream);
    } else {
      interp_fused_tw<T, W, 4>(jobs, item_end, njobs, total, queue, stream);
    }
  });
}

template ZSpreadJob<float> zwin_spread_job<float>(const SpreadArgs<float>&);
template ZSpreadJob<double> zwin_spread_job<double>(const SpreadArgs<double>&);
template ZInterpJob<float> zwin_interp_job<float>(const InterpArgs<float>&);
template ZInterpJob<double> zwin_interp_job<double>(const InterpArgs<double>&);
template void zwin_build_work_list<float>(const BinGeom&, const SortedPoints<float>&,
                                          cudaStream_t);
template void zwin_build_work_list<double>(const BinGeom&, const SortedPoints<double>&,
                                           cudaStream_t);
template void launch_spread_zwin_fused<float>(const ZSpreadJob<float>*, const i64*, int, i64,
                                              int, int, u32*, cudaStream_t);
template void launch_spread_zwin_fused<double>(const ZSpreadJob<double>*, const i64*, int, i64,
                                               int, int, u32*, cudaStream_t);
template void launch_interp_zwin_fused<float>(const ZInterpJob<float>*, const i64*, int, i64,
                                              int, int, u32*, cudaStream_t);
template void launch_interp_zwin_fused<double>(const ZInterpJob<double>*, const i64*, int, i64,
                                               int, int, u32*, cudaStream_t);
template void launch_spread_zwin<float>(const SpreadArgs<float>&, cudaStream_t);
template void launch_spread_zwin<double>(const SpreadArgs<double>&, cudaStream_t);
template void launch_interp_zwin<float>(const InterpArgs<float>&, cudaStream_t);
template void launch_interp_zwin<double>(const InterpArgs<double>&, cudaStream_t);

}  // namespace nnb
