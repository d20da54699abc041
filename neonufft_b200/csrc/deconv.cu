// Deconvolution by the kernel's Fourier transform, with mode reordering.
//
// downsample (type 1) follows the reference's downsample_{1,2,3}d_kernel
// (src/neonufft/gpu/kernels/downsample_kernel.cu:18-191): mode k of the user's box (CMCL order
// k = i - N/2, or FFT order) is read from fine cell k mod nf and scaled by prod_d corr_d[|k_d|].
// upsample (type 2, type-3 stage 2) is the inverse (reference upsample_kernel.cu:18-196), but
// here one kernel writes every fine cell -- zero outside the mode box -- so the separate grid
// memset of the reference (src/neonufft/gpu/plan_impl.hpp:117) is fused away.
#include "kernels.cuh"

namespace nnb {

namespace {

constexpr int kDeconvThreads = 256;

__device__ __forceinline__ i64 mode_of_index(i64 i, i64 n, int order) {
  const i64 n_neg = n / 2;
  if (order == NEONUFFT_MODE_ORDER_CMCL) return i - n_neg;
  const i64 n_nonneg = n - n_neg;
  return i < n_nonneg ? i : i - n;
}

__device__ __forceinline__ i64 index_of_mode(i64 k, i64 n, int order) {
  const i64 n_neg = n / 2;
  if (order == NEONUFFT_MODE_ORDER_CMCL) return k + n_neg;
  return k >= 0 ? k : k + n;
}

// Elements spanned by the user's strided mode array: 1 + sum_d (modes_d - 1) stride_d.
template <typename T>
__device__ __forceinline__ i64 mode_array_extent(const DeconvArgs<T>& a) {
  i64 e = 1;
  for (int d = 0; d < a.dim; ++d) e += (a.modes[d] - 1) * a.stride[d];
  return e;
}

// Both kernels give a warp one segment of a row, so that the row's coordinates, factors and
// addresses are worked out once per warp and short rows do not leave most of a block idle. They
// are bound by memory. Measured against one thread per cell of a 256-thread block of a row:
// upsampling 12740^2 modes to 25600^2 cells (single precision, 6.5 GB) 2.03 -> 1.00 ms, 136^3 to
// 270^3 99 -> 33 us; downsampling a 480^3 grid to 256^3 modes 92 -> 56 us.
constexpr int kDeconvWarps = kDeconvThreads / 32;

struct RowTasks {
  i64 tasks;  // rows * segs
  u32 segs;   // segments per row
  u32 len;    // cells per segment
  u32 n1;     // rows per plane
};
// Segments of up to 1024 cells, shorter while there are fewer than 24 warps per SM (one long row:
// 1D grids of 2000 and 4e5 cells took 5.7 and 17.7 us with segments of 1024).
RowTasks row_tasks(i64 n0, i64 n1, i64 n2) {
  RowTasks t;
  t.n1 = u32(n1);
  for (t.len = 1024;; t.len /= 2) {
    t.segs = u32((n0 + t.len - 1) / t.len);
    t.tasks = n1 * n2 * t.segs;
    if (t.len == 64 || t.tasks >= 148 * 24) break;
  }
  return t;
}
// Row (i1, i2) and cells [begin, end) of the calling warp's task; false past the last task.
__device__ __forceinline__ bool row_task(const RowTasks& t, i64 n0, int& i1, int& i2, i64& begin,
                                         i64& end) {
  const i64 task = i64(blockIdx.x) * kDeconvWarps + (threadIdx.x >> 5);
  if (task >= t.tasks) return false;
  const i64 row = t.segs == 1 ? task : task / t.segs;
  begin = (task - row * t.segs) * t.len;
  end = min(begin + t.len, n0);
  if (row < i64(0x7fffffff)) {
    i2 = int(u32(row) / t.n1);
  } else {
    i2 = int(row / t.n1);
  }
  i1 = int(row - i64(i2) * t.n1);
  return true;
}

template <typename T>
__global__ void __launch_bounds__(kDeconvThreads)
    downsample_kernel(const __grid_constant__ DeconvArgs<T> a, RowTasks t,
                      const cplx_t<T>* __restrict__ fine, cplx_t<T>* __restrict__ out) {
  int i1, i2;
  i64 begin, end;
  if (!row_task(t, a.modes[0], i1, i2, begin, end)) return;
  T c12 = 1;
  i64 f12 = 0, o12 = 0;
  if (a.dim > 1) {
    const i64 k1 = mode_of_index(i1, a.modes[1], a.order);
    c12 = a.corr[1][k1 < 0 ? -k1 : k1];
    f12 = (k1 >= 0 ? k1 : a.nf[1] + k1) * a.nf[0];
    o12 = i1 * a.stride[1];
  }
  T c2 = 1;
  if (a.dim > 2) {
    const i64 k2 = mode_of_index(i2, a.modes[2], a.order);
    c2 = a.corr[2][k2 < 0 ? -k2 : k2];
    f12 += (k2 >= 0 ? k2 : a.nf[2] + k2) * a.nf[0] * a.nf[1];
    o12 += i2 * a.stride[2];
  }
#pragma unroll 4
  for (i64 i0 = begin + (threadIdx.x & 31); i0 < end; i0 += 32) {
    const i64 k0 = mode_of_index(i0, a.modes[0], a.order);
    T c = a.corr[0][k0 < 0 ? -k0 : k0];
    if (a.dim > 1) c *= c12;
    if (a.dim > 2) c *= c2;
    const i64 f = f12 + (k0 >= 0 ? k0 : a.nf[0] + k0);
    const i64 o = o12 + i0 * a.stride[0];
    if (NNB_CHECK_INDEX(f, a.nf[0] * a.nf[1] * a.nf[2]) &&
        NNB_CHECK_INDEX(o, mode_array_extent(a))) {
      const cplx_t<T> v = fine[f];
      out[o] = cplx_t<T>{v.x * c, v.y * c};
    }
  }
}

// Fine cell j holds mode k = j (j < n_nonneg) or k = j - nf (j >= nf - n_neg); none between.
__device__ __forceinline__ bool mode_of_cell(i64 j, i64 n, i64 nf, i64& k) {
  const i64 n_neg = n / 2;
  if (j < n - n_neg) {
    k = j;
    return true;
  }
  k = j - nf;
  return k >= -n_neg;
}

__device__ __forceinline__ void store_pair(float2* p, float2 u, float2 v) {
  *reinterpret_cast<float4*>(p) = make_float4(u.x, u.y, v.x, v.y);
}
__device__ __forceinline__ void store_pair(double2* p, double2 u, double2 v) {
  p[0] = u;
  p[1] = v;
}

template <typename T>
__global__ void __launch_bounds__(kDeconvThreads)
    upsample_kernel(const __grid_constant__ DeconvArgs<T> a, RowTasks t,
                    const cplx_t<T>* __restrict__ in, cplx_t<T>* __restrict__ fine, bool vec) {
  using C = cplx_t<T>;
  int j1, j2;
  i64 begin, end;
  if (!row_task(t, a.nf[0], j1, j2, begin, end)) return;
  const i64 row = (j1 + j2 * a.nf[1]) * a.nf[0];
  [[maybe_unused]] const i64 cells = a.nf[0] * a.nf[1] * a.nf[2];
  bool inside = true;  // the row holds modes
  T c1 = 1, c2 = 1;
  i64 src12 = 0, k;
  if (a.dim > 1) {
    inside = mode_of_cell(j1, a.modes[1], a.nf[1], k);
    if (inside) {
      c1 = a.corr[1][k < 0 ? -k : k];
      src12 = index_of_mode(k, a.modes[1], a.order) * a.stride[1];
    }
  }
  if (a.dim > 2 && inside) {
    inside = mode_of_cell(j2, a.modes[2], a.nf[2], k);
    if (inside) {
      c2 = a.corr[2][k < 0 ? -k : k];
      src12 += index_of_mode(k, a.modes[2], a.order) * a.stride[2];
    }
  }
  auto value = [&](i64 j0) -> C {
    i64 k0;
    if (!inside || !mode_of_cell(j0, a.modes[0], a.nf[0], k0)) return C{T(0), T(0)};
    T c = a.corr[0][k0 < 0 ? -k0 : k0];
    if (a.dim > 1) c *= c1;
    if (a.dim > 2) c *= c2;
    const i64 src = src12 + index_of_mode(k0, a.modes[0], a.order) * a.stride[0];
    if (!NNB_CHECK_INDEX(src, mode_array_extent(a))) return C{T(0), T(0)};
    const C v = in[src];
    return C{v.x * c, v.y * c};
  };
  const int lane = threadIdx.x & 31;
  if (vec) {  // even rows from a 16-byte boundary: two cells per lane and store
#pragma unroll 4
    for (i64 j0 = begin + 2 * lane; j0 < end; j0 += 64) {
      const C u = value(j0), v = value(j0 + 1);
      if (NNB_CHECK_INDEX(row + j0 + 1, cells)) store_pair(fine + row + j0, u, v);
    }
  } else {
#pragma unroll 4
    for (i64 j0 = begin + lane; j0 < end; j0 += 32) {
      const C u = value(j0);
      if (NNB_CHECK_INDEX(row + j0, cells)) fine[row + j0] = u;
    }
  }
}

unsigned deconv_grid(const RowTasks& t) {
  const i64 ctas = (t.tasks + kDeconvWarps - 1) / kDeconvWarps;
  if (ctas > 0x7fffffffll) throw_input("grid too large");
  return unsigned(ctas);
}

}  // namespace

template <typename T>
void launch_downsample(const DeconvArgs<T>& a, const cplx_t<T>* fine, cplx_t<T>* out,
                       cudaStream_t stream) {
  const i64 m1 = a.dim > 1 ? a.modes[1] : 1;
  const i64 m2 = a.dim > 2 ? a.modes[2] : 1;
  // (the public limits of the interface; the launch itself has none)
  if (m1 > 65535 || m2 > 65535) throw_input("mode count above 65535 in dimension 1 or 2");
  const RowTasks t = row_tasks(a.modes[0], m1, m2);
  downsample_kernel<T><<<deconv_grid(t), kDeconvThreads, 0, stream>>>(a, t, fine, out);
  NNB_LAUNCH_CHECK();
}

template <typename T>
void launch_upsample(const DeconvArgs<T>& a, const cplx_t<T>* in, cplx_t<T>* fine,
                     cudaStream_t stream) {
  const i64 n1 = a.dim > 1 ? a.nf[1] : 1;
  const i64 n2 = a.dim > 2 ? a.nf[2] : 1;
  // (the public limits of the interface; the launch itself has none)
  if (n1 > 65535 || n2 > 65535) throw_input("fine grid above 65535 in dimension 1 or 2");
  const RowTasks t = row_tasks(a.nf[0], n1, n2);
  const bool vec = a.nf[0] % 2 == 0 && reinterpret_cast<uintptr_t>(fine) % 16 == 0;
  upsample_kernel<T><<<deconv_grid(t), kDeconvThreads, 0, stream>>>(a, t, in, fine, vec);
  NNB_LAUNCH_CHECK();
}

template void launch_downsample<float>(const DeconvArgs<float>&, const float2*, float2*, cudaStream_t);
template void launch_downsample<double>(const DeconvArgs<double>&, const double2*, double2*, cudaStream_t);
template void launch_upsample<float>(const DeconvArgs<float>&, const float2*, float2*, cudaStream_t);
template void launch_upsample<double>(const DeconvArgs<double>&, const double2*, double2*, cudaStream_t);

}  // namespace nnb
