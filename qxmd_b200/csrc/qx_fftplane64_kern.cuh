// The FP64 H|psi> plane pass with the lines in registers: the fused y-x-y pass
// of qx_fftplane_kern.cuh for double, one lane a line up to 32 odd points and
// two lanes a line for even lengths up to 64 (each then transforms the even or
// the odd samples, N / 2 points, and one butterfly exchange by shuffles
// completes the line), so that a line is at most 32 complex doubles of
// registers.  Between the phases a plane lives in shared memory as NY rows of
// LD complex values, LD = 2 modulo 4 so that the four rows of a quarter warp
// start in different banks.
// It replaces the shared-memory stage kernels k_ypass, k_xvx and k_ypass, whose
// two passes per stage through shared memory and the round trips of bufB bound
// them.  Whole pipeline, 160 / 16 / 2 bands: 24^3 81 / 37 / 35 -> 42 / 27 / 27
// us, 40^3 192 / 49 / 38 -> 124 / 37 / 33, 54^3 392 / 63 / 45 -> 342 / 52 / 45,
// 60^3 598 / 90 / 51 -> 440 / 77 / 49.  At 54 points registers allow three
// CTAs of 128 threads a SM; the FP64 chains and instruction fetches bound it.
// The z passes in the same form measured slower than the stage kernels (54^3,
// 16 bands: 63 -> 69 us) and were left out.
#pragma once
#include "qx_fftplane.h"
#include "qx_regfft.cuh"

namespace qx {
namespace pl64 {

constexpr int lanes(int n) { return n % 2 == 0 ? 2 : 1; }
constexpr int plane_threads(int nx, int ny) { return (ny * lanes(nx) + 31) / 32 * 32; }
// resident CTAs asked of the register allocator: 128 registers a thread up to
// 16 points a lane, 168 beyond
constexpr int plane_ctas(int nx, int ny) {
  const int mx = nx / lanes(nx), my = ny / lanes(ny), m = mx > my ? mx : my;
  const int c = 65536 / (plane_threads(nx, ny) * (m <= 16 ? 128 : 168));
  return c > 16 ? 16 : (c < 1 ? 1 : c);
}

__device__ __forceinline__ double2 swap1(double2 v) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, 1), __shfl_xor_sync(0xffffffffu, v.y, 1));
}

// A line of N points over L = lanes(N) adjacent lanes, M = N / L points each.
template <int N>
struct Line {
  static constexpr int L = lanes(N), M = N / L;
  // x[j] = sample L j + h in; sample k + h M at x[out_pos(M, k)] out
  template <int SIGN>
  static __device__ __forceinline__ void dit(double2 (&x)[M], int h) {
    rf::fft<double, SIGN, M>(x);
    if constexpr (L == 2) {
      rf::static_for<0, M>([&](auto kc) {
        constexpr int k = decltype(kc)::value, pk = rf::out_pos(M, k);
        const double2 mine = x[pk], other = swap1(mine);
        const double2 e = h ? other : mine;
        const double2 t = rf::twiddle<double, SIGN, k, N>(h ? mine : other);
        x[pk] = h ? rf::sub(e, t) : rf::add(e, t);
      });
    }
  }
  // x[out_pos(M, k)] = sample k + h M in; output L j + h at u[out_pos(M, j)]
  template <int SIGN>
  static __device__ __forceinline__ void dif(const double2 (&x)[M], double2 (&u)[M], int h) {
    rf::static_for<0, M>([&](auto kc) {
      constexpr int k = decltype(kc)::value, pk = rf::out_pos(M, k);
      if constexpr (L == 2) {
        const double2 mine = x[pk], other = swap1(mine);
        const double2 lo = h ? other : mine, hi = h ? mine : other;
        u[k] = h ? rf::twiddle<double, SIGN, k, N>(rf::sub(lo, hi)) : rf::add(lo, hi);
      } else {
        u[k] = x[pk];
      }
    });
    rf::fft<double, SIGN, M>(u);
  }
};

constexpr int plane_ld(int p1) { return p1 + (6 - p1 % 4) % 4; }

}  // namespace pl64

// One band pair's z plane a CTA; whole warps run each phase (lanes without a
// line work on zeros and store nothing), so every shuffle has its full mask.
template <int NX, int NY>
__global__ void __launch_bounds__(pl64::plane_threads(NX, NY), pl64::plane_ctas(NX, NY))
    k_plane64(PipeParams P, double2 *__restrict__ bufA, const double *__restrict__ vloc) {
  using rf::out_pos;
  using X = pl64::Line<NX>;
  using Y = pl64::Line<NY>;
  constexpr int NT = pl64::plane_threads(NX, NY);
  const int i3 = blockIdx.x;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair)) return;
  const int P1 = P.P1, P2 = P.P2, m1 = P.m1, m2 = P.m2, LD = pl64::plane_ld(P1);
  extern __shared__ double2 T64[];   // [NY][LD]
  double2 *T = T64;
  double2 *A = bufA + ((long)pl * P.k3 + i3) * P2 * P1;
  const int t = threadIdx.x;
  const double2 zero = make_double2(0.0, 0.0);

  // (1) y backward, line = sphere column a
  for (int a0 = 0; a0 < P1; a0 += NT / Y::L) {
    const int a = a0 + t / Y::L, h = t % Y::L;
    if (a0 + (t & ~31) / Y::L >= P1) continue;   // uniform in the warp
    const bool on = a < P1;
    double2 x[Y::M];
#pragma unroll
    for (int j = 0; j < Y::M; ++j) {
      const int i2 = Y::L * j + h;
      const int j2 = (i2 <= m2) ? i2 + m2 : ((i2 >= NY - m2) ? i2 - NY + m2 : -1);
      double2 v = zero;
      if (on && j2 >= 0 && a >= P.row_lo[j2] && a <= P.row_hi[j2]) v = A[j2 * P1 + a];
      x[j] = v;
    }
    Y::template dit<+1>(x, h);
    if (on) {
      rf::static_for<0, Y::M>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        T[(k + h * Y::M) * LD + a] = x[out_pos(Y::M, k)];
      });
    }
  }
  __syncthreads();
  // (2) x backward, * V, x forward; line = grid row
  if ((t & ~31) / X::L < NY) {
    const int r = t / X::L, h = t % X::L;
    const bool on = r < NY;
    double2 *row = T + (on ? r : NY - 1) * LD;
    double2 x[X::M], u[X::M];
#pragma unroll
    for (int j = 0; j < X::M; ++j) {
      const int i1 = X::L * j + h;
      double2 v = zero;
      if (i1 <= m1) v = row[i1 + m1];
      else if (i1 >= NX - m1) v = row[i1 - NX + m1];
      x[j] = v;
    }
    X::template dit<+1>(x, h);
    const double *V = vloc + ((long)i3 * NY + (on ? r : NY - 1)) * NX + h * X::M;
    rf::static_for<0, X::M>([&](auto kc) {
      constexpr int k = decltype(kc)::value, pk = out_pos(X::M, k);
      const double vv = V[k];
      x[pk] = make_double2(x[pk].x * vv, x[pk].y * vv);
    });
    X::template dif<-1>(x, u, h);
    __syncwarp();   // a row's lanes, in one warp, have read it before either rewrites it
    if (on) {
      rf::static_for<0, X::M>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        const int i1 = X::L * j + h;
        if (i1 <= m1) row[i1 + m1] = u[out_pos(X::M, j)];
        else if (i1 >= NX - m1) row[i1 - NX + m1] = u[out_pos(X::M, j)];
      });
    }
  }
  __syncthreads();
  // (3) y forward, line = sphere column a; only rows inside the sphere are kept
  for (int a0 = 0; a0 < P1; a0 += NT / Y::L) {
    const int a = a0 + t / Y::L, h = t % Y::L;
    if (a0 + (t & ~31) / Y::L >= P1) continue;
    const bool on = a < P1;
    double2 x[Y::M];
#pragma unroll
    for (int j = 0; j < Y::M; ++j) x[j] = on ? T[(Y::L * j + h) * LD + a] : zero;
    Y::template dit<-1>(x, h);
    if (on) {
      rf::static_for<0, Y::M>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        const int i2 = k + h * Y::M;
        const int j2 = (i2 <= m2) ? i2 + m2 : ((i2 >= NY - m2) ? i2 - NY + m2 : -1);
        if (j2 >= 0 && a >= P.row_lo[j2] && a <= P.row_hi[j2]) A[j2 * P1 + a] = x[out_pos(Y::M, k)];
      });
    }
  }
}

template <int NX, int NY>
int plane64_launch(const PipeParams &P, int npl, double2 *bufA, const double *vloc, cudaStream_t st) {
  const size_t sm = sizeof(double2) * (size_t)NY * pl64::plane_ld(P.P1);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_plane64<NX, NY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(double2) * NY * pl64::plane_ld(NX)));
    attr = true;
  }
  k_plane64<NX, NY><<<dim3(P.k3, npl), pl64::plane_threads(NX, NY), sm, st>>>(P, bufA, vloc);
  note_launch();
  return 0;
}

#define QX_PLANE64_GRID(NX, NY) \
  template int plane64_launch<NX, NY>(const PipeParams &, int, double2 *, const double *, cudaStream_t);

}  // namespace qx
