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
// 60^3 598 / 90 / 51 -> 440 / 77 / 49 with whole lines; leaving out what a
// sphere of half the grid has zero (HALF) took H|psi> of Si64 (54^3, 160 bands,
// both projector contractions included) from 410 to 292 us, and the z passes in
// the same form to 267.  At 54 points registers allow three CTAs of 128 threads
// a SM; with the FP64 pipe active for 41 % and an instruction issued in 39 % of
// the cycles, dependent chains, barriers and loads at 12 warps bound it.  The
// 168 registers spill 4 to 64 bytes a thread at 42 to 54 points, 88 at 60 and 224
// at 64.
#pragma once
#include "qx_fftplane.h"
#include "qx_regfft.cuh"
#include "qx_zlines.cuh"

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
  // (ZM: rf::fft_nz's bound on the lane's samples, (M - 1) / 2 for none zero)
  template <int SIGN, int ZM = M / 2>
  static __device__ __forceinline__ void dit(double2 (&x)[M], int h) {
    rf::fft_nz<double, SIGN, M, ZM>(x);
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

constexpr int z_ctas(int n) { return n / lanes(n) <= 16 ? 8 : 6; }   // of 64 threads

constexpr int plane_ld(int p1) { return p1 + (6 - p1 % 4) % 4; }

// z2_kind and z2_bound for a line over one or two lanes
template <int N, int MB> constexpr int kind(int j) {
  return lanes(N) == 2 ? z2_kind<N, MB>(j) : (j <= MB ? Z2_POS : j >= N - MB ? Z2_NEG : Z2_NONE);
}
template <int N, int MB> constexpr int bound() {
  return lanes(N) == 2 ? z2_bound<N, MB>() : (2 * MB + 1 < N ? MB : N / 2);
}

}  // namespace pl64

// One band pair's z plane a CTA; whole warps run each phase (lanes without a
// line work on zeros and store nothing), so every shuffle has its full mask.
// HALF, the tile's columns and the sphere's rows as in k_plane.
template <int NX, int NY, bool HALF>
__global__ void __launch_bounds__(pl64::plane_threads(NX, NY), pl64::plane_ctas(NX, NY))
    k_plane64(PipeParams P, double2 *__restrict__ bufA, const double *__restrict__ vloct) {
  using rf::out_pos;
  using X = pl64::Line<NX>;
  using Y = pl64::Line<NY>;
  constexpr int NT = pl64::plane_threads(NX, NY), MBX = line_mb<NX, HALF>(), MBY = line_mb<NY, HALF>();
  constexpr int PC = 2 * MBX + 1, LD = pl64::plane_ld(PC);
  const int i3 = blockIdx.x;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair)) return;
  const int P1 = P.P1, m1 = P.m1;
  extern __shared__ double2 T64[];   // [NY][LD]
  double2 *T = T64;
  double2 *A = bufA + ((long)pl * P.k3 + i3) * P.P2 * P1 + P.m2 * P1;   // row m2
  const int t = threadIdx.x;
  const double2 zero = make_double2(0.0, 0.0);

  // (1) y backward, line = tile column c (sphere column c - (MBX - m1))
  for (int c0 = 0; c0 < PC; c0 += NT / Y::L) {
    const int c = c0 + t / Y::L, h = t % Y::L, a = c - (MBX - m1);
    if (c0 + (t & ~31) / Y::L >= PC) continue;   // uniform in the warp
    const bool in = c < PC && a >= 0 && a < P1;
    const ulonglong2 m = in ? P.col_mask[a] : make_ulonglong2(0ull, 0ull);
    const unsigned px = (unsigned)m.x >> h, nx = (unsigned)m.y << h;   // bit L j: row L j + h; bit NY - L j: row -(NY - L j - h)
    double2 x[Y::M];
    rf::static_for<0, Y::M>([&](auto jc) {
      constexpr int j = decltype(jc)::value, kind = pl64::kind<NY, MBY>(j);
      double2 v = zero;
      if constexpr (kind == Z2_POS || kind == Z2_POS0) {
        if ((px >> (Y::L * j)) & 1u) v = A[(Y::L * j + h) * P1 + a];
      } else if constexpr (kind == Z2_NEG || kind == Z2_NEG1) {
        if ((nx >> (NY - Y::L * j)) & 1u) v = A[-(NY - Y::L * j - h) * P1 + a];
      }
      x[j] = v;
    });
    Y::template dit<+1, pl64::bound<NY, MBY>()>(x, h);
    if (c < PC) {
      rf::static_for<0, Y::M>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        T[(k + h * Y::M) * LD + c] = x[out_pos(Y::M, k)];
      });
    }
  }
  __syncthreads();
  // (2) x backward, * V, x forward; line = grid row
  if ((t & ~31) / X::L < NY) {
    const int r = t / X::L, h = t % X::L;
    const bool on = r < NY;
    double2 *row = T + (on ? r : NY - 1) * LD + MBX;   // sample k at row[k]
    double2 x[X::M], u[X::M];
    rf::static_for<0, X::M>([&](auto jc) {
      constexpr int j = decltype(jc)::value, kind = pl64::kind<NX, MBX>(j);
      double2 v = zero;
      if constexpr (kind == Z2_POS) v = row[X::L * j + h];
      else if constexpr (kind == Z2_POS0) v = h ? zero : row[2 * j];
      else if constexpr (kind == Z2_NEG) v = row[X::L * j - NX + h];
      else if constexpr (kind == Z2_NEG1) v = h ? row[2 * j + 1 - NX] : zero;
      x[j] = v;
    });
    X::template dit<+1, pl64::bound<NX, MBX>()>(x, h);
    const double *V = vloct + ((long)i3 * NX + h * X::M) * NY + (on ? r : NY - 1);   // y fastest (see k_plane)
    rf::static_for<0, X::M>([&](auto kc) {
      constexpr int k = decltype(kc)::value, pk = out_pos(X::M, k);
      const double vv = V[k * NY];
      x[pk] = make_double2(x[pk].x * vv, x[pk].y * vv);
    });
    X::template dif<-1>(x, u, h);
    __syncwarp();   // a row's lanes, in one warp, have read it before either rewrites it
    if (on) {
      rf::static_for<0, X::M>([&](auto jc) {
        constexpr int j = decltype(jc)::value, kind = pl64::kind<NX, MBX>(j), q = out_pos(X::M, j);
        if constexpr (kind == Z2_POS) row[X::L * j + h] = u[q];
        else if constexpr (kind == Z2_POS0) { if (!h) row[2 * j] = u[q]; }
        else if constexpr (kind == Z2_NEG) row[X::L * j - NX + h] = u[q];
        else if constexpr (kind == Z2_NEG1) { if (h) row[2 * j + 1 - NX] = u[q]; }
      });
    }
  }
  __syncthreads();
  // (3) y forward, line = tile column c; only rows inside the sphere are kept
  for (int c0 = 0; c0 < PC; c0 += NT / Y::L) {
    const int c = c0 + t / Y::L, h = t % Y::L, a = c - (MBX - m1);
    if (c0 + (t & ~31) / Y::L >= PC) continue;
    const bool in = c < PC && a >= 0 && a < P1;
    const ulonglong2 m = in ? P.col_mask[a] : make_ulonglong2(0ull, 0ull);
    const unsigned inx = (unsigned)m.x, iny = (unsigned)m.y;
    double2 x[Y::M];
#pragma unroll
    for (int j = 0; j < Y::M; ++j) x[j] = c < PC ? T[(Y::L * j + h) * LD + c] : zero;
    Y::template dit<-1>(x, h);
    if constexpr (Y::L == 2) {
      // lane 0 holds rows k < M, lane 1 rows k - M
      rf::static_for<0, Y::M>([&](auto kc) {
        constexpr int k = decltype(kc)::value, kn = Y::M - k;
        if constexpr (k <= MBY || kn <= MBY) {
          const bool keep = h ? (kn <= MBY && ((iny >> (kn < 32 ? kn : 0)) & 1u)) : (k <= MBY && ((inx >> k) & 1u));
          if (keep) A[(k - h * Y::M) * P1 + a] = x[out_pos(Y::M, k)];
        }
      });
    } else {
      rf::static_for<0, MBY + 1>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        if ((inx >> k) & 1u) A[k * P1 + a] = x[out_pos(NY, k)];
        if constexpr (k > 0)
          if ((iny >> k) & 1u) A[-k * P1 + a] = x[out_pos(NY, NY - k)];
      });
    }
  }
}

// The z passes, one sphere column a line (see k_zcols_inv, k_zcols_fwd).
constexpr int ZC64_T = 64;

template <int N, bool HALF>
__global__ void __launch_bounds__(ZC64_T, pl64::z_ctas(N)) k_zcols64_inv(PipeParams P, const double *__restrict__ cin,
                                                                        long ldc, double2 *__restrict__ bufA) {
  using Z = pl64::Line<N>;
  int q = (int)((blockIdx.x * ZC64_T + threadIdx.x) / Z::L);
  const int h = threadIdx.x % Z::L;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair)) return;   // uniform in the block
  const bool on = q < P.ncol;
  q = min(q, P.ncol - 1);
  const int bA = P.pairs[2 * p], bB = P.pairs[2 * p + 1];
  const double *cA = cin + (long)bA * ldc;
  const double *cB = bB >= 0 ? cin + (long)bB * ldc : cA;
  constexpr int MB = line_mb<N, HALF>();
  double2 x[Z::M] = {};
  z_gather<double, Z::M, std::conditional_t<Z::L == 2, ZIn2<N, MB>, ZRows1<N, MB>>>(
      cA, cB, bB >= 0, [&](auto ic) { return __ldg(P.col_ig + (Z::L * decltype(ic)::value + h) * P.ncol + q); },
      [&](auto ic, double re, double im) { x[decltype(ic)::value] = make_double2(re, im); });
  Z::template dit<+1, pl64::bound<N, MB>()>(x, h);
  if (on) {
    double2 *dst = bufA + (long)pl * N * P.P2 * P.P1 + P.col_ja[q];
    rf::static_for<0, Z::M>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      dst[(long)(k + h * Z::M) * P.P2 * P.P1] = x[rf::out_pos(Z::M, k)];
    });
  }
}

template <int N, bool HALF>
__global__ void __launch_bounds__(ZC64_T, pl64::z_ctas(N)) k_zcols64_fwd(PipeParams P,
                                                                        const double2 *__restrict__ bufA,
                                                                        double2 *__restrict__ zsph) {
  using Z = pl64::Line<N>;
  int q = (int)((blockIdx.x * ZC64_T + threadIdx.x) / Z::L);
  const int h = threadIdx.x % Z::L;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair)) return;   // uniform in the block
  const bool on = q < P.ncol;
  q = min(q, P.ncol - 1);
  const double2 *src = bufA + (long)pl * N * P.P2 * P.P1 + P.col_ja[q];
  double2 x[Z::M];
#pragma unroll
  for (int j = 0; j < Z::M; ++j) x[j] = src[(long)(Z::L * j + h) * P.P2 * P.P1];
  Z::template dit<-1>(x, h);
  if (!on) return;
  constexpr int MB = line_mb<N, HALF>(), M = Z::M;
  z_scatter<double, M, std::conditional_t<Z::L == 2, ZOut2<N, MB>, ZRows1<N, MB>>>(
      zsph + (long)pl * (P.nplw + 1) * 2, P.inv_n,
      [&](auto ic) { return __ldg(P.col_ig + (decltype(ic)::value + h * M) * P.ncol + q); },
      [&](auto ic) { return x[rf::out_pos(M, decltype(ic)::value)]; });
}

template <int NX, int NY, bool HALF>
static void plane64_go(const PipeParams &P, int npl, double2 *bufA, const double *vloct, cudaStream_t st) {
  constexpr size_t sm = sizeof(double2) * (size_t)NY * pl64::plane_ld(2 * line_mb<NX, HALF>() + 1);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_plane64<NX, NY, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attr = true;
  }
  k_plane64<NX, NY, HALF><<<dim3(P.k3, npl), pl64::plane_threads(NX, NY), sm, st>>>(P, bufA, vloct);
}

// Spheres beyond half the grid (a density cutoff below four times the
// wavefunction's) take the stage kernels.
template <int NX, int NY>
int plane64_launch(const PipeParams &P, int npl, double2 *bufA, const double *vloct, cudaStream_t st) {
  if (P.m1 > line_mb<NX, true>() || P.m2 > line_mb<NY, true>()) return -1;
  plane64_go<NX, NY, true>(P, npl, bufA, vloct, st);
  note_launch();
  return 0;
}

template <int N>
int zcols64_launch(const PipeParams &P, int npl, const double *cin, long ldc, double2 *bufA, double2 *zsph,
                   cudaStream_t st) {
  if (P.m3 > line_mb<N, true>()) return -1;
  dim3 g((pl64::lanes(N) * P.ncol + ZC64_T - 1) / ZC64_T, npl);
  if (cin) k_zcols64_inv<N, true><<<g, ZC64_T, 0, st>>>(P, cin, ldc, bufA);
  else k_zcols64_fwd<N, true><<<g, ZC64_T, 0, st>>>(P, bufA, zsph);
  note_launch();
  return 0;
}

#define QX_PLANE64_GRID(NX, NY) \
  template int plane64_launch<NX, NY>(const PipeParams &, int, double2 *, const double *, cudaStream_t);

#define QX_ZCOLS64_LENGTH(N) \
  template int zcols64_launch<N>(const PipeParams &, int, const double *, long, double2 *, double2 *, cudaStream_t);

}  // namespace qx
