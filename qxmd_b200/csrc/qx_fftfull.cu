// Full-grid FP64 transforms of the density side (rfft3/fft3 drop-in, the
// passes of launch_full_fft) with the lines in registers (compile-time-length
// FFTs, twiddles exact to double rounding): one lane a line for odd lengths,
// two adjacent lanes for even ones (pl64::Line).  In the z and y passes
// consecutive lines are consecutive i1, so a warp reads and writes runs of
// 16-byte elements of every plane it crosses; in the x pass each line is
// contiguous.
// A pass is one chain per line, a few thousand threads on the whole GPU:
// latency bounds it, so a thread holds as little of a line as divides evenly.
// Against the shared-memory stages at 54^3: 20.5 -> 6.1 us a pass, an SCF
// iteration of Si64 (12 passes) 1399 -> 1352 us.
#include "qx_internal.h"
#include "qx_fftplane64_kern.cuh"

namespace qx {

constexpr int FL_T = 64;

// axis 2: lines along z (i3), one per (i1, i2); axis 1: along y (i2), one per
// (i1, i3); axis 0: along x (i1), one per (i2, i3).  g[(i3 k2 + i2) k1 + i1],
// in place, times scale.
template <int N, int SIGN>
__global__ void __launch_bounds__(FL_T) k_full_lines(double2 *__restrict__ g, int k1, int k2, int k3, int axis,
                                                     double scale) {
  using Z = pl64::Line<N>;
  const long nlines = axis == 0 ? (long)k2 * k3 : (long)k1 * (axis == 2 ? k2 : k3);
  long t = (blockIdx.x * (long)FL_T + threadIdx.x) / Z::L;
  const int h = threadIdx.x % Z::L;
  const bool on = t < nlines;   // whole warps run: lanes past the last line work on zeros and store nothing
  t = on ? t : nlines - 1;
  long stride;
  double2 *base;
  if (axis == 0) {
    stride = 1;
    base = g + t * k1;
  } else {
    const int i1 = (int)(t % k1), o = (int)(t / k1);
    stride = axis == 2 ? (long)k1 * k2 : (long)k1;
    base = g + (axis == 2 ? (long)o * k1 + i1 : (long)o * k2 * k1 + i1);
  }
  double2 x[Z::M];
#pragma unroll
  for (int j = 0; j < Z::M; ++j) x[j] = on ? base[(Z::L * j + h) * stride] : make_double2(0.0, 0.0);
  Z::template dit<SIGN>(x, h);   // every output needs every sample of both lanes: in place is safe
  if (!on) return;
  rf::static_for<0, Z::M>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    double2 z = x[rf::out_pos(Z::M, k)];
    z.x *= scale;
    z.y *= scale;
    base[(k + h * Z::M) * stride] = z;
  });
}

template <int N>
static void full_lines_go(double2 *g, int k1, int k2, int k3, int axis, int sign, double scale, cudaStream_t st) {
  const long nl = pl64::lanes(N) * (axis == 0 ? (long)k2 * k3 : (long)k1 * (axis == 2 ? k2 : k3));
  const int blocks = (int)((nl + FL_T - 1) / FL_T);
  if (axis != 0) scale = 1.0;
  if (sign > 0) k_full_lines<N, +1><<<blocks, FL_T, 0, st>>>(g, k1, k2, k3, axis, scale);
  else k_full_lines<N, -1><<<blocks, FL_T, 0, st>>>(g, k1, k2, k3, axis, scale);
  note_launch();
}

// QX_FULL_LINES=0 keeps every pass on the shared-memory kernels (read at
// every call).
static bool full_lines_enabled() {
  const char *e = getenv("QX_FULL_LINES");
  return !(e && e[0] == '0');
}

int launch_full_lines_f64(double2 *g, int k1, int k2, int k3, int axis, int sign, double scale, cudaStream_t st) {
  if (!full_lines_enabled() || axis < 0 || axis > 2) return -1;
  switch (axis == 2 ? k3 : axis == 1 ? k2 : k1) {
#define QX_CASE(N) \
  case N: full_lines_go<N>(g, k1, k2, k3, axis, sign, scale, st); return 0;
    QX_ZCOLS64_LENGTHS(QX_CASE)
#undef QX_CASE
    default: return -1;
  }
}

}  // namespace qx
