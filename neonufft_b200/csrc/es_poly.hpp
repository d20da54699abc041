// Piecewise polynomials of the ES kernel.
//
// A point's w kernel values are phi(frac + k), k = 0 .. w - 1, with frac in [-w/2, -w/2 + 1]: the
// k-th value is a smooth function of t = 2 frac + w - 1 in [-1, 1], except at the outer edge of
// the first and the last piece, where phi has a square-root end. The kernel is even, so pieces k
// and w - 1 - k are mirror images: one even and one odd polynomial in t give both. (Piecewise
// polynomial evaluation of this kernel: Barnett, Magland, af Klinteberg, SIAM J. Sci. Comput. 41,
// 2019, section 5.3; here from Chebyshev interpolation of each piece.)
#pragma once

namespace nnb {

template <typename T>
struct EsPoly {
  // degree 9 in single, 16 in double precision: below the rounding of the direct formula where they
  // are used (es_poly in params.hpp; at w = 8 and upsampling 2 the inner pieces are off by 1e-10
  // and up to 8e-16 of the kernel's peak, the edge piece by 1.6e-8 in single precision)
  static constexpr int NE = sizeof(T) == 4 ? 5 : 9;
  static constexpr int NO = sizeof(T) == 4 ? 5 : 8;
  T e[8][NE];  // coefficients of t^0, t^2, ... of piece k
  T o[8][NO];  // coefficients of t^1, t^3, ...
  int mode;    // which pieces the polynomials serve
};
enum EsPolyMode { kEsAllPoly = 0, kEsExactEdges = 1, kEsAllExact = 2 };

}  // namespace nnb
