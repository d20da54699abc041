// 3D spreading and interpolation of wide kernels (n_spread 9 to 16) with the z-window kernels of
// zwin.cuh: windows of exactly w planes, tiles of 4 x 8 x 1 cells.
//
// The shared-memory slabs that took these widths (spread.cu, interp.cu) are bound by the chain of
// shared-memory accesses from point to point: 5e5 points on 128 x 120 x 128 cells, w = 10, double
// precision, spread in 2.87 ms and interpolated in 1.56 ms; here 0.45 and 0.57 ms, bound by the
// FP64 pipe and, at a quarter of a point per cell, by the latency of the planes that enter and
// leave the window.
#include "kernels.cuh"
#include "zwin.cuh"

namespace nnb {

namespace {

constexpr int kWideTx = 4;
constexpr int kWideTy = 8;

template <typename T, int W>
void spread_wide_w(const SpreadArgs<T>& a, cudaStream_t stream) {
  using S = ZShape<T, W, kWideTx, kWideTy>;
  const ZChunks ch = make_chunks(i64(a.g.ntiles[0]) * a.g.ntiles[1], a.g.ntiles[2], W);
  const WorkList wl = zwin_work_list(a.g, a.pts, ch);
  dim3 grid{unsigned(wl.grid), unsigned(a.batch), 1u};
  spread_zwin_wide_kernel<T, W, kWideTx, kWideTy><<<grid, S::NT, 0, stream>>>(a, ch, wl);
  NNB_LAUNCH_CHECK();
}

template <typename T, int W>
void interp_wide_w(const InterpArgs<T>& a, cudaStream_t stream) {
  using S = ZShape<T, W, kWideTx, kWideTy>;
  constexpr int smem = int(sizeof(ZInterpShared<T, W, kWideTx, kWideTy>));
  auto kern = interp_zwin_kernel<T, W, kWideTx, kWideTy>;
  // Per device and cheap; set on every launch so that multi-device processes stay correct.
  NNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const ZChunks ch = make_chunks(i64(a.g.ntiles[0]) * a.g.ntiles[1], a.g.ntiles[2], W);
  const WorkList wl = zwin_work_list(a.g, a.pts, ch);
  kern<<<unsigned(wl.grid), S::NT, smem, stream>>>(a, ch, wl);
  NNB_LAUNCH_CHECK();
}

void check_wide_geom(const BinGeom& g) {
  if (g.dim != 3 || !g.zmajor || g.tile[0] != kWideTx || g.tile[1] != kWideTy || g.tile[2] != 1) {
    throw_internal("wide z-window kernels need a 3D plane-major (4, 8, 1) tiling");
  }
}

}  // namespace

template <typename T>
void launch_spread_zwin_wide(const SpreadArgs<T>& a, cudaStream_t stream) {
  check_wide_geom(a.g);
  if (a.batch > 65535) throw_input("batch size above 65535");
  switch (a.g.w) {
    case 9: return spread_wide_w<T, 9>(a, stream);
    case 10: return spread_wide_w<T, 10>(a, stream);
    case 11: return spread_wide_w<T, 11>(a, stream);
    case 12: return spread_wide_w<T, 12>(a, stream);
    case 13: return spread_wide_w<T, 13>(a, stream);
    case 14: return spread_wide_w<T, 14>(a, stream);
    case 15: return spread_wide_w<T, 15>(a, stream);
    case 16: return spread_wide_w<T, 16>(a, stream);
    default: throw_internal("wide z-window kernels need n_spread in [9, 16]");
  }
}

template <typename T>
void launch_interp_zwin_wide(const InterpArgs<T>& a, cudaStream_t stream) {
  check_wide_geom(a.g);
  switch (a.g.w) {
    case 9: return interp_wide_w<T, 9>(a, stream);
    case 10: return interp_wide_w<T, 10>(a, stream);
    case 11: return interp_wide_w<T, 11>(a, stream);
    case 12: return interp_wide_w<T, 12>(a, stream);
    case 13: return interp_wide_w<T, 13>(a, stream);
    case 14: return interp_wide_w<T, 14>(a, stream);
    case 15: return interp_wide_w<T, 15>(a, stream);
    case 16: return interp_wide_w<T, 16>(a, stream);
    default: throw_internal("wide z-window kernels need n_spread in [9, 16]");
  }
}

template void launch_spread_zwin_wide<float>(const SpreadArgs<float>&, cudaStream_t);
template void launch_spread_zwin_wide<double>(const SpreadArgs<double>&, cudaStream_t);
template void launch_interp_zwin_wide<float>(const InterpArgs<float>&, cudaStream_t);
template void launch_interp_zwin_wide<double>(const InterpArgs<double>&, cudaStream_t);

}  // namespace nnb
