// Gather and scatter of the sphere's z columns for the register-FFT z passes
// (qx_fftplane_kern.cuh, qx_fftplane64_kern.cuh).
#pragma once
#include "qx_fftplane.h"
#include "qx_regfft.cuh"

namespace qx {

// The z samples of a line from the sphere coefficients of two bands: code =
// +-(ig + 1) of the sample, 0 for none.  U samples at a time: their codes, then
// their coefficients, without a branch, so that the dependent loads of U
// samples are in flight together (sample by sample they were a chain of U
// memory latencies, which bounded these passes: Si512, 96 points, 1100 bands,
// 727 -> 472 us backward and 822 -> 462 us forward; Si64, 54 points, 160 bands,
// 15.6 -> 12.8 us backward).  Sample i of 0 .. CNT - 1:
// code_at(IC<i>) and put(IC<i>, z), for the i with HAS::at(i).
template <typename T, int CNT, class HAS, class CODE, class PUT>
__device__ __forceinline__ void z_gather(const T *__restrict__ cA, const T *__restrict__ cB, bool two, CODE code_at,
                                         PUT put) {
  constexpr int U = 8;
  rf::static_for<0, (CNT + U - 1) / U>([&](auto bc) {
    constexpr int b = decltype(bc)::value * U, e = b + U < CNT ? b + U : CNT;
    int code[U];
    T ra[U], ia[U], rb[U], ib[U];
    rf::static_for<b, e>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      if constexpr (HAS::at(i)) code[i - b] = code_at(ic);
    });
    rf::static_for<b, e>([&](auto ic) {
      constexpr int i = decltype(ic)::value, u = i - b;
      if constexpr (HAS::at(i)) {
        const int ig = max(abs(code[u]), 1) - 1;
        ra[u] = __ldg(cA + 2 * ig);
        ia[u] = __ldg(cA + 2 * ig + 1);
        rb[u] = __ldg(cB + 2 * ig);
        ib[u] = __ldg(cB + 2 * ig + 1);
      }
    });
    rf::static_for<b, e>([&](auto ic) {
      constexpr int i = decltype(ic)::value, u = i - b;
      if constexpr (HAS::at(i)) {
        const bool in = code[u] != 0, im = abs(code[u]) > 1;   // the G = 0 coefficient is real
        const T ar = in ? ra[u] : T(0), ai = im ? ia[u] : T(0);
        const T br = in && two ? rb[u] : T(0), bi = im && two ? ib[u] : T(0);
        put(ic, code[u] > 0 ? ar - bi : ar + bi, code[u] > 0 ? ai + br : br - ai);
      }
    });
  });
}
// The scatter of the forward passes: the codes of U rows first.
template <typename T, int CNT, class HAS, class CODE, class GET>
__device__ __forceinline__ void z_scatter(typename c2t<T>::type *__restrict__ Z, T s, CODE code_at, GET get) {
  constexpr int U = 8;
  rf::static_for<0, (CNT + U - 1) / U>([&](auto bc) {
    constexpr int b = decltype(bc)::value * U, e = b + U < CNT ? b + U : CNT;
    int code[U];
    rf::static_for<b, e>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      if constexpr (HAS::at(i)) code[i - b] = code_at(ic);
    });
    rf::static_for<b, e>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      if constexpr (HAS::at(i)) {
        const int c = code[i - b];
        if (c != 0) {
          typename c2t<T>::type z = get(ic);
          z.x *= s;
          z.y *= s;
          Z[c > 0 ? 2 * (c - 1) : 2 * (-c - 1) + 1] = z;
          if (c == 1) Z[1] = z;
        }
      }
    });
  });
}
// rows of a one-lane line of N samples, of a two-lane line's N / 2 (either
// lane's), that may be inside a sphere of half width MB
template <int N, int MB> struct ZRows1 { static constexpr bool at(int i) { return i <= MB || i >= N - MB; } };
template <int N, int MB> struct ZIn2 { static constexpr bool at(int j) { return z2_kind<N, MB>(j) != Z2_NONE; } };
template <int N, int MB> struct ZOut2 { static constexpr bool at(int k) { return k <= MB || N / 2 - k <= MB; } };

}  // namespace qx
