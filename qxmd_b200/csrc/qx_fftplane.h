// Launchers of the fused FFT plane kernels (qx_fftplane_kern.cuh), one per
// specialised plane shape or z length, explicitly instantiated in the
// qx_fftplane_*.cu files.  Each returns 0 after queuing its kernels on st,
// or -1 if the plane does not fit the kernel (the caller then takes the
// generic passes).
#pragma once
#include "qx_internal.h"

namespace qx {

// One grid line per thread: planes of NX = k1 by NY = k2 points (each at
// most 64), z columns of N = k3 points.
template <int NX, int NY>
int plane_launch(const PipeParams &P, int npl, float2 *bufA, const float *vloct, cudaStream_t st);
// the passes around the real-space projectors: backward into R (nl null),
// forward from R with the projectors' part (nl)
template <int NX, int NY>
int plane_r_launch(const PipeParams &P, int npl, float2 *bufA, float2 *R, const float *vloc,
                   const NlPoints<float> *nl, cudaStream_t st);
template <int NX, int NY>
int rho_launch(const PipeParams &P, int npl, const float2 *bufA, const double *wocc, double *part, double *rho,
               int accumulate, cudaStream_t st);
template <int N>
int zcols_launch(const PipeParams &P, int npl, const float *cin, long ldc, float2 *bufA, const float2 *src,
                 float2 *zsph, bool inv, cudaStream_t st);

// Two lanes a line (N = 96).
template <int N>
int plane2_launch(const PipeParams &P, int npl, float2 *bufA, const float *vloct, cudaStream_t st);
template <int N>
int rho2_launch(const PipeParams &P, int npl, const float2 *bufA, const double *wocc, double *part, double *rho,
                int accumulate, cudaStream_t st);
template <int N>
int zcols2_launch(const PipeParams &P, int npl, const float *cin, long ldc, float2 *bufA, const float2 *src,
                  float2 *zsph, bool inv, cudaStream_t st);

// The k1 x k2 plane shapes with register kernels, X(k1, k2): sixteen square
// ones of 20 to 64 points (36 and 64 for callers with grids of their own; of the
// lengths that cells give, 35, 56 and 63 have none), and the elongated cells of
// the 48-cell batch (two or three unit cells along x).  Other planes, 48 x 24 or 49 x 54 say, take the
// shared-memory stages.  The same list drives the dispatch and the
// instantiation files.
#define QX_PLANE_GRIDS(X)                                                                              \
  X(20, 20) X(21, 21) X(24, 24) X(25, 25) X(27, 27) X(30, 30) X(32, 32) X(36, 36) X(40, 40) X(42, 42) \
  X(45, 45) X(48, 48) X(49, 49) X(54, 54) X(60, 60) X(64, 64)                                         \
  X(24, 25) X(25, 24) X(25, 27) X(27, 25) X(42, 21) X(45, 24) X(45, 42) X(48, 45) X(49, 25) X(54, 24) \
  X(54, 25) X(54, 27)
// The z lengths with register column kernels.
#define QX_ZCOLS_LENGTHS(X) \
  X(20) X(21) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(42) X(45) X(48) X(49) X(54) X(60) X(64)

// FP64 (qx_fftplane64_kern.cuh): those of the FP32 shapes above whose lines are
// even, or odd and at most 32 points (not 45 and 49).
#define QX_PLANE64_GRIDS(X)                                                                            \
  X(20, 20) X(21, 21) X(24, 24) X(25, 25) X(27, 27) X(30, 30) X(32, 32) X(36, 36) X(40, 40) X(42, 42) \
  X(48, 48) X(54, 54) X(60, 60) X(64, 64)                                                             \
  X(24, 25) X(25, 24) X(25, 27) X(27, 25) X(42, 21) X(54, 24) X(54, 25) X(54, 27)
#define QX_ZCOLS64_LENGTHS(X) X(20) X(21) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(42) X(48) X(54) X(60) X(64)
// cin: the backward pass into bufA; null: the forward pass into zsph
template <int N>
int zcols64_launch(const PipeParams &P, int npl, const double *cin, long ldc, double2 *bufA, double2 *zsph,
                   cudaStream_t st);
template <int NX, int NY>
int plane64_launch(const PipeParams &P, int npl, double2 *bufA, const double *vloct, cudaStream_t st);

constexpr int plane_grid_key(int k1, int k2) { return k1 * 1024 + k2; }

// The line of N points whose samples MB < i < N - MB are zero: MB = (N - 1) / 4
// wherever the density cutoff is at least four times the wavefunction's
// (then the wavefunction sphere spans half the grid), (N - 1) / 2 otherwise.
template <int N, bool HALF> constexpr int line_mb() { return HALF ? (N - 1) / 4 : (N - 1) / 2; }

// Which samples i = 2 j + h of a two-lane line may be nonzero when those at
// MB < i < N - MB are zero: nothing for either lane, one lane, or both, at
// the start (sample i) or the end (sample i - N) of the line.
enum { Z2_NONE, Z2_POS, Z2_POS0, Z2_NEG, Z2_NEG1 };
template <int N, int MB> constexpr int z2_kind(int j) {
  return 2 * j + 1 <= MB ? Z2_POS : 2 * j <= MB ? Z2_POS0 : 2 * j >= N - MB ? Z2_NEG : 2 * j + 1 >= N - MB ? Z2_NEG1 : Z2_NONE;
}
// the bound of rf::fft_nz on a lane's N / 2 samples
template <int N, int MB> constexpr int z2_bound() {
  const int lo = MB / 2, hi = N / 2 - (N - MB) / 2;
  return lo > hi ? lo : hi;
}

// QX_PLANE_PAIRS=0 keeps one z plane a CTA (read at every call).
bool plane_pairs_enabled();

// rho = [rho +] the sum of the RHO_GROUPS partial planes in part, in group order.
void rho_groups_launch(const double *part, long n, double *rho, int accumulate, cudaStream_t st);

}  // namespace qx
