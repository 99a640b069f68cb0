// Fused y-x-y pass of the FP32 H|psi> pipeline for k1 x k2 planes of the
// specialised shapes (x length NX = k1, y length NY = k2), one CTA per (band
// pair, z plane or two), one grid line per thread with the whole line in
// registers (compile-time-length FFTs of qx_regfft.cuh):
//   (1) backward y-FFT of each of the P1 sphere columns, read straight from
//       the z-transformed plane in bufA (rows outside the sphere are zero);
//   (2) per grid row: backward x-FFT (P1 non-zero inputs), times V_loc(r),
//       forward x-FFT, keep the P1 sphere columns;
//   (3) forward y-FFT of each column, the sphere rows written back to bufA.
// Between the steps the plane lives in shared memory as NY x P1 complex
// values.  This replaces k_ypass<+1>, k_xvx and k_ypass<-1> (hcnonloc's
// c2r -> V_loc * psi -> r2c, engrad.f90:484-571) and removes the two round
// trips of bufB through L2/HBM.
//
// This header holds the kernel templates and their per-shape launchers; each
// qx_fftplane_*.cu file instantiates a group of shapes and z lengths (so the
// groups compile in parallel), and qx_fftplane.cu dispatches on the grid.
#pragma once
#include "qx_fftplane.h"
#include "qx_regfft.cuh"
#include "qx_zlines.cuh"

namespace qx {

// Resident CTAs per SM asked of the register allocator: 8 (128 registers) up
// to 54 points, where that spills nothing or 4 to 32 bytes a thread.
constexpr int plane_minb(int n) { return n <= 54 ? 8 : 1; }

// Grid rows of the x phase, thread t of a 64-thread CTA: with two planes of
// at most 32 rows, warp w takes plane w's rows (both planes at once);
// otherwise thread t takes row t of each plane in turn.
template <int NY, int PL>
struct PlaneRows {
  static constexpr bool both = PL == 2 && NY <= 32;
  static constexpr int passes = both ? 1 : PL;
  __device__ static int plane(int t, int pass) { return both ? (t >> 5) : pass; }
  __device__ static int row(int t) { return both ? (t & 31) : t; }
};

// the rows of sphere column a as P.col_mask, at most 32 either way
__device__ __forceinline__ uint2 col_rows(const PipeParams &P, int a) {
  const ulonglong2 m = P.col_mask[a];
  return make_uint2((unsigned)m.x, (unsigned)m.y);
}

// Backward y transform of sphere column a of a plane (A: its [P2][P1] rows)
// into column c of a tile with `ld` columns.
template <int NY, int MB>
__device__ __forceinline__ void plane_y_back(const PipeParams &P, const float2 *A, int a, float2 *Tc, int ld) {
  const uint2 in = col_rows(P, a);
  const int P1 = P.P1;
  const float2 *A0 = A + P.m2 * P1 + a;
  const float2 zero = make_float2(0.f, 0.f);
  float2 x[NY];
  rf::static_for<0, MB + 1>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    x[k] = (in.x >> k) & 1u ? A0[k * P1] : zero;
    if constexpr (k > 0) x[NY - k] = (in.y >> k) & 1u ? A0[-k * P1] : zero;
  });
  if constexpr (2 * MB + 1 < NY) rf::fft_nz<float, +1, NY, MB>(x);
  else {
    if constexpr (2 * MB + 2 == NY) x[MB + 1] = zero;
    rf::fft<float, +1, NY>(x);
  }
  rf::static_for<0, NY>([&](auto ic) {
    constexpr int i2 = decltype(ic)::value, q = rf::out_pos(NY, i2);
    Tc[i2 * ld] = x[q];
  });
}

// Backward x transform of a tile row: column MB + k holds sample k (|k| <= MB).
template <int NX, int MB>
__device__ __forceinline__ void plane_x_back(const float2 *row, float2 (&x)[NX]) {
  rf::static_for<0, MB + 1>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    x[k] = row[MB + k];
    if constexpr (k > 0) x[NX - k] = row[MB - k];
  });
  if constexpr (2 * MB + 1 < NX && 2 * MB + 2 != NX) rf::fft_nz<float, +1, NX, MB>(x);
  else {
    if constexpr (2 * MB + 2 == NX) x[MB + 1] = make_float2(0.f, 0.f);
    rf::fft<float, +1, NX>(x);
  }
}

// U units a CTA: U band pairs of the same planes on 64 threads each, whose
// phases the CTA's barriers keep together.  The unrolled transforms are some
// tens of kilobytes of code that every unit runs once, so units in step share
// its instruction fetches: two at 54 x 54 (Si64, 160 bands, whole H|psi>) 163
// -> 147 us, four the same, eight 158 us.
// HALF: the sphere spans at most half of either axis (line_mb), so that the
// zero samples' loads and butterflies and the outputs beyond the sphere are
// left out at compile time; the tile then has 2 MBX + 1 columns, those beyond
// the sphere zero.  At Si64 (54 x 54, 160 bands): 88 -> 49 us the pass, and the
// outputs are the same bit for bit.  The FMA pipe is active for 66 % of it, at
// 16 warps a SM (the registers' limit); stalls on instruction fetches are few.
template <int NX, int NY, int PL, int U, bool HALF>
__global__ void __launch_bounds__(64 * U, (plane_minb(NX > NY ? NX : NY) + U - 1) / U)
    k_plane(PipeParams P, float2 *__restrict__ bufA, const float *__restrict__ vloct, int npl) {
  using rf::out_pos;
  using Rows = PlaneRows<NY, PL>;
  constexpr int MBX = line_mb<NX, HALF>(), MBY = line_mb<NY, HALF>(), PB = 2 * MBX + 1;
  // PL = 2: the unit takes planes i3 and i3 + 1; the y phases give warp w the
  // columns of plane w (PB <= 32).  PL = 1: one plane, the columns on
  // threads 0 .. PB - 1.  NX = k1 (x, the sphere's P1 columns), NY = k2.
  const int i3b = blockIdx.x * PL;
  const int np = P.npair_dev ? *P.npair_dev : P.npair;
  if (P.pair0 + (int)blockIdx.y * U >= np) return;
  const int pl = blockIdx.y * U + (threadIdx.x >> 6);
  const bool live = pl < npl && P.pair0 + pl < np;
  const int P1 = P.P1, P2 = P.P2, m1 = P.m1;
  const int npl_here = live ? min(PL, P.k3 - i3b) : 0;   // planes of this unit
  extern __shared__ float2 Tu[];   // [U][PL][NY][PB]
  float2 *T = Tu + (threadIdx.x >> 6) * (PL * NY * PB);
  const int t = threadIdx.x & 63;
  // column phases: plane and tile column of this thread
  const int cpl = (PL == 2) ? (t >> 5) : 0, col = (PL == 2) ? (t & 31) : t;
  const bool col_on = col < PB && cpl < npl_here;
  const int a = col - (MBX - m1);   // sphere column
  const bool in_sphere = a >= 0 && a < P1;
  float2 *A = bufA + ((long)pl * P.k3 + i3b + cpl) * P2 * P1;
  float2 *Tc = T + cpl * (NY * PB) + col;

  // (1) y backward, thread = column of its plane
  if (col_on) {
    if (in_sphere) {
      plane_y_back<NY, MBY>(P, A, a, Tc, PB);
    } else {
      for (int i = 0; i < NY; ++i) Tc[i * PB] = make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
  // (2) x backward, * V, x forward; thread = grid row r of plane rp
  const int r = Rows::row(t);
  for (int pass = 0; pass < Rows::passes; ++pass) {
    const int rp = Rows::plane(t, pass);
    if (r < NY && rp < npl_here) {
      float2 x[NX];
      float2 *row = T + (rp * NY + r) * PB;
      plane_x_back<NX, MBX>(row, x);
      // y fastest, so that the threads of a warp, one row each, read runs: in
      // the grid's order every load touched 32 lines of cache, 8 cycles each
      // (H|psi> of Si64: 104.9 -> 101.6 us)
      const float *V = vloct + (long)(i3b + rp) * NX * NY + r;
      float2 y[NX];
      rf::static_for<0, NX>([&](auto ic) {
        constexpr int i1 = decltype(ic)::value, q = out_pos(NX, i1);
        const float vv = V[i1 * NY];
        y[i1] = make_float2(x[q].x * vv, x[q].y * vv);
      });
      rf::fft<float, -1, NX>(y);
      rf::static_for<0, MBX + 1>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        row[MBX + k] = y[out_pos(NX, k)];
        if constexpr (k > 0) row[MBX - k] = y[out_pos(NX, NX - k)];
      });
    }
  }
  __syncthreads();
  // (3) y forward, thread = column of its plane; only rows inside the sphere are kept
  if (col_on && in_sphere) {
    const uint2 in = col_rows(P, a);
    float2 x[NY];
#pragma unroll
    for (int i2 = 0; i2 < NY; ++i2) x[i2] = Tc[i2 * PB];
    rf::fft<float, -1, NY>(x);
    float2 *A0 = A + P.m2 * P1 + a;
    rf::static_for<0, MBY + 1>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      if ((in.x >> k) & 1u) A0[k * P1] = x[out_pos(NY, k)];
      if constexpr (k > 0)
        if ((in.y >> k) & 1u) A0[-k * P1] = x[out_pos(NY, NY - k)];
    });
  }
}

// ---------------------------------------------------------------------------
// The same fused y-x-y pass for longer lines (N = 2H, H a register-FFT length,
// N > 64), two threads per line: lanes 2l and 2l + 1 of a warp own line l.
// Backward transforms and the forward y transform by decimation in time:
// thread h holds the samples x[2j + h], transforms them (H points), and one
// butterfly exchange with its partner (shfl_xor 1) leaves it the outputs
// X[k + hH], k < H, at positions out_pos(H, k).  The forward x transform
// follows the potential multiply, when thread h holds the second half of the
// line (y[k + hH]), so it runs by decimation in frequency: the exchange
// stage first (a = y[k] + y[k+H] kept by h = 0, b = (y[k] - y[k+H]) w^k by
// h = 1), then the H-point transform gives the outputs Y[2j + h].  Whole
// warps run each phase (lanes without a line work on zeros and store
// nothing), so every shuffle has its full mask.
namespace pl2 {
template <int SIGN, int N>
__device__ __forceinline__ void dit_combine(float2 (&v)[N / 2], int h) {
  constexpr int H = N / 2;
  rf::static_for<0, H>([&](auto kc) {
    constexpr int k = decltype(kc)::value, pk = rf::out_pos(H, k);
    const float2 mine = v[pk];
    float2 other;
    other.x = __shfl_xor_sync(0xffffffffu, mine.x, 1);
    other.y = __shfl_xor_sync(0xffffffffu, mine.y, 1);
    const float2 e = h ? other : mine;
    const float2 t = rf::twiddle<float, SIGN, k, N>(h ? mine : other);
    v[pk] = h ? rf::sub(e, t) : rf::add(e, t);
  });
}
// v[out_pos(H, k)] = y[k + hH] in; u[k] (natural order) = a[k] (h = 0) or
// b[k] (h = 1) out, ready for the H-point transform.
template <int SIGN, int N>
__device__ __forceinline__ void dif_split(const float2 (&v)[N / 2], float2 (&u)[N / 2], int h) {
  constexpr int H = N / 2;
  rf::static_for<0, H>([&](auto kc) {
    constexpr int k = decltype(kc)::value, pk = rf::out_pos(H, k);
    const float2 mine = v[pk];
    float2 other;
    other.x = __shfl_xor_sync(0xffffffffu, mine.x, 1);
    other.y = __shfl_xor_sync(0xffffffffu, mine.y, 1);
    const float2 lo = h ? other : mine, hi = h ? mine : other;   // y[k], y[k + H]
    u[k] = h ? rf::twiddle<float, SIGN, k, N>(rf::sub(lo, hi)) : rf::add(lo, hi);
  });
}
}  // namespace pl2

// The tile holds the sphere's columns only: at Si512 (96^3, 1100 bands) the pass
// took 5950 us with whole lines, 2920 us with HALF (and 2 MB + 1 = 47 columns).
template <int N, bool HALF> constexpr int plane2_pitch() { return (2 * line_mb<N, HALF>() + 1 + 14) / 16 * 16 + 2; }

template <int N, bool HALF>
__global__ void __launch_bounds__(2 * N) k_plane2(PipeParams P, float2 *__restrict__ bufA,
                                                 const float *__restrict__ vloct) {
  using rf::out_pos;
  constexpr int H = N / 2;
  const int i3 = blockIdx.x;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair)) return;
  // tile columns: sample k of x at column MB + k (zero beyond the sphere); the
  // pitch PB = 2 modulo 16 puts the eight lines of a half warp, two adjacent
  // samples each, in different banks
  constexpr int MB = line_mb<N, HALF>(), PC = 2 * MB + 1, PB = plane2_pitch<N, HALF>();
  const int P1 = P.P1, m1 = P.m1;
  extern __shared__ float2 T[];   // [N][PB]
  float2 *A = bufA + ((long)pl * P.k3 + i3) * P.P2 * P1;
  const int t = threadIdx.x, l = t >> 1, h = t & 1;
  const bool warp_on_cols = (t & ~31) < 2 * PC;   // some lane of this warp owns a column
  const float2 zero = make_float2(0.f, 0.f);
  const int a = l - (MB - m1);                    // sphere column of tile column l
  const bool in_sphere = l < PC && a >= 0 && a < P1;
  typedef typename std::conditional<(MB < 31), unsigned, unsigned long long>::type Mask;
  const ulonglong2 in2 = in_sphere ? P.col_mask[a] : make_ulonglong2(0ull, 0ull);
  const Mask inx = (Mask)in2.x, iny = (Mask)in2.y;
  float2 *A0 = A + P.m2 * P1 + a;

  // (1) y backward, line = tile column l
  if (warp_on_cols) {
    const Mask px = inx >> h, nx = iny << h;   // bit 2j: row 2j + h; bit N - 2j: row -(N - 2j - h)
    float2 x[H];
    rf::static_for<0, H>([&](auto jc) {
      constexpr int j = decltype(jc)::value, kind = z2_kind<N, MB>(j);
      float2 v = zero;
      if constexpr (kind == Z2_POS || kind == Z2_POS0) {
        if ((px >> (2 * j)) & 1) v = A0[(2 * j + h) * P1];
      } else if constexpr (kind == Z2_NEG || kind == Z2_NEG1) {
        if ((nx >> (N - 2 * j)) & 1) v = A0[-(N - 2 * j - h) * P1];
      }
      x[j] = v;
    });
    rf::fft_nz<float, +1, H, z2_bound<N, MB>()>(x);
    pl2::dit_combine<+1, N>(x, h);
    if (l < PC) {
      rf::static_for<0, H>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        T[(k + h * H) * PB + l] = x[out_pos(H, k)];
      });
    }
  }
  __syncthreads();
  // (2) x backward, * V, x forward; line = grid row i2 = l (every thread has one)
  {
    float2 x[H];
    float2 *row = T + l * PB + MB;   // sample k at row[k]
    rf::static_for<0, H>([&](auto jc) {
      constexpr int j = decltype(jc)::value, kind = z2_kind<N, MB>(j);
      float2 v = zero;
      if constexpr (kind == Z2_POS) v = row[2 * j + h];
      else if constexpr (kind == Z2_POS0) v = h ? zero : row[2 * j];
      else if constexpr (kind == Z2_NEG) v = row[2 * j - N + h];
      else if constexpr (kind == Z2_NEG1) v = h ? row[2 * j + 1 - N] : zero;
      x[j] = v;
    });
    rf::fft_nz<float, +1, H, z2_bound<N, MB>()>(x);
    pl2::dit_combine<+1, N>(x, h);
    // y fastest (see k_plane); in the grid's order, value by value, these loads
    // were a seventh of the pass (Si512: 2885 -> 2480 us)
    const float *V = vloct + ((long)i3 * N + h * H) * N + l;
    rf::static_for<0, H>([&](auto kc) {
      constexpr int k = decltype(kc)::value, pk = out_pos(H, k);
      const float vv = V[k * N];
      x[pk] = make_float2(x[pk].x * vv, x[pk].y * vv);
    });
    float2 u[H];
    pl2::dif_split<-1, N>(x, u, h);
    rf::fft<float, -1, H>(u);
    __syncwarp();   // a row's two lanes have read it before either rewrites it
    rf::static_for<0, H>([&](auto jc) {
      constexpr int j = decltype(jc)::value, kind = z2_kind<N, MB>(j), q = out_pos(H, j);
      if constexpr (kind == Z2_POS) row[2 * j + h] = u[q];
      else if constexpr (kind == Z2_POS0) { if (!h) row[2 * j] = u[q]; }
      else if constexpr (kind == Z2_NEG) row[2 * j - N + h] = u[q];
      else if constexpr (kind == Z2_NEG1) { if (h) row[2 * j + 1 - N] = u[q]; }
    });
  }
  __syncthreads();
  // (3) y forward, line = tile column l; only rows inside the sphere are kept
  if (warp_on_cols) {
    float2 x[H];
#pragma unroll
    for (int j = 0; j < H; ++j) x[j] = l < PC ? T[(2 * j + h) * PB + l] : zero;
    rf::fft<float, -1, H>(x);
    pl2::dit_combine<-1, N>(x, h);
    // lane 0 holds rows k < H, lane 1 rows k - H
    rf::static_for<0, H>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      if constexpr (k <= MB || H - k <= MB) {
        constexpr int kp = k <= MB ? k : 0, kn = H - k <= MB ? H - k : 0;
        const bool keep = h ? (H - k <= MB && ((iny >> kn) & 1)) : (k <= MB && ((inx >> kp) & 1));
        if (keep) A0[(k - h * H) * P1] = x[out_pos(H, k)];
      }
    });
  }
}

// ---------------------------------------------------------------------------
// The y and x passes around the real-space projectors, which need psi(r) of
// the whole cell between the backward and the forward transforms: two band
// pairs of one z plane a CTA, 64 threads a pair, the planes in shared memory
// as NY x (NX | 1) complex values.
//   k_plane_inv_r: backward y and x, the planes stored to R (coalesced);
//   k_plane_fwd_r: V psi plus the projectors' part, forward x and y back to
//     bufA.  A grid point's projector points come in grid-point order
//     (NlPoints), so each thread sums its own points in a fixed order,
//     for both pairs of the CTA from one read of the projector values.
// The L1 path (70 % busy) and the latency of the projector values' gathers
// bound the second (24 bytes an entry and CTA, 313 k entries at Si64), hence
// two pairs a CTA and four grid points in flight a thread.  Against the shared-memory stage
// kernels and the scatter by float atomics in shared memory that these
// replace, per 160-band pass at Si64: y and x backward 118 -> 55 us, forward
// 366 -> 145 us.
template <int NX, int NY, bool HALF>
__global__ void __launch_bounds__(128, plane_minb(NX > NY ? NX : NY) > 1 ? 4 : 1)
    k_plane_inv_r(PipeParams P, const float2 *__restrict__ bufA, float2 *__restrict__ R, int npl) {
  using rf::out_pos;
  constexpr int LD = NX | 1, MBX = line_mb<NX, HALF>(), MBY = line_mb<NY, HALF>();
  const int i3 = blockIdx.x, h = threadIdx.x >> 6, u = threadIdx.x & 63;
  const int pl = blockIdx.y * 2 + h, np = P.npair_dev ? *P.npair_dev : P.npair;
  if (P.pair0 + (int)blockIdx.y * 2 >= np) return;
  const bool on = pl < npl && P.pair0 + pl < np;
  extern __shared__ float2 T[];
  float2 *Tp = T + h * (NY * LD);
  if (on && u < 2 * MBX + 1) {   // x sample k = u - MBX, at position k or NX + k of the rows
    const int k = u - MBX, a = k + P.m1;
    float2 *Tc = Tp + (k >= 0 ? k : NX + k);
    if (a >= 0 && a < P.P1) {
      plane_y_back<NY, MBY>(P, bufA + ((long)pl * P.k3 + i3) * P.P2 * P.P1, a, Tc, LD);
    } else {
      for (int i = 0; i < NY; ++i) Tc[i * LD] = make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
  if (on && u < NY) {
    float2 x[NX];
    float2 *row = Tp + u * LD;
    rf::static_for<0, MBX + 1>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      x[k] = row[k];
      if constexpr (k > 0) x[NX - k] = row[NX - k];
    });
    rf::fft_nz<float, +1, NX, MBX>(x);
    rf::static_for<0, NX>([&](auto ic) {
      constexpr int i1 = decltype(ic)::value, q = out_pos(NX, i1);
      row[i1] = x[q];
    });
  }
  __syncthreads();
  if (on) {
    float2 *dst = R + ((long)pl * P.k3 + i3) * (NX * NY);
#pragma unroll 4
    for (int i = u; i < NX * NY; i += 64) dst[i] = Tp[(i / NX) * LD + i % NX];
  }
}

template <int NX, int NY, bool HALF>
__global__ void __launch_bounds__(128, plane_minb(NX > NY ? NX : NY) > 1 ? 4 : 1)
    k_plane_fwd_r(PipeParams P, const float2 *__restrict__ R, float2 *__restrict__ bufA,
                  const float *__restrict__ vloc, NlPoints<float> nl, int npl) {
  using rf::out_pos;
  constexpr int LD = NX | 1, NP = NX * NY, UN = 4, MBX = line_mb<NX, HALF>(), MBY = line_mb<NY, HALF>();
  const int i3 = blockIdx.x, t = threadIdx.x, h = t >> 6, u = t & 63;
  const int pl0 = blockIdx.y * 2, np = P.npair_dev ? *P.npair_dev : P.npair;
  if (P.pair0 + pl0 >= np) return;
  const bool two = pl0 + 1 < npl && P.pair0 + pl0 + 1 < np;
  const int P1 = P.P1;
  extern __shared__ float2 T[];
  {
    const long g0 = (long)i3 * NP;
    const float2 *R0 = R + (long)pl0 * P.k3 * NP + g0, *R1 = two ? R0 + (long)P.k3 * NP : R0;
    const float *V = vloc + g0;
    const int *off = nl.off + g0;
    const float2 *S0 = nl.sumr + (long)pl0 * nl.natom * nl.lmx, *S1 = two ? S0 + (long)nl.natom * nl.lmx : S0;
    for (int ib = t; ib < NP; ib += 128 * UN) {
      float2 z0[UN], z1[UN];
      int e0[UN], e1[UN];
#pragma unroll
      for (int q = 0; q < UN; ++q) {
        const int i = min(ib + 128 * q, NP - 1);
        e0[q] = off[i];
        e1[q] = off[i + 1];
        const float v = V[i];
        const float2 a = R0[i], b = R1[i];
        z0[q] = make_float2(a.x * v, a.y * v);
        z1[q] = make_float2(b.x * v, b.y * v);
      }
      if (nl.lmx == 4) {
        // the UN points' entries side by side, so that their loads overlap
        int more = 0;
#pragma unroll
        for (int q = 0; q < UN; ++q) more = max(more, e1[q] - e0[q]);
        for (int k = 0; k < more; ++k) {
          int at[UN];
          float4 v[UN];
#pragma unroll
          for (int q = 0; q < UN; ++q) {
            const bool in = e0[q] + k < e1[q];
            at[q] = in ? nl.atom[e0[q] + k] : -1;
            v[q] = in ? *reinterpret_cast<const float4 *>(nl.vnl + 4L * (e0[q] + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int q = 0; q < UN; ++q) {
            if (at[q] < 0) continue;
            const float4 *a = reinterpret_cast<const float4 *>(S0 + 4L * at[q]);
            const float4 *b = reinterpret_cast<const float4 *>(S1 + 4L * at[q]);
            const float4 a0 = a[0], a1 = a[1], b0 = b[0], b1 = b[1], w = v[q];
            z0[q].x += w.x * a0.x + w.y * a0.z + w.z * a1.x + w.w * a1.z;
            z0[q].y += w.x * a0.y + w.y * a0.w + w.z * a1.y + w.w * a1.w;
            z1[q].x += w.x * b0.x + w.y * b0.z + w.z * b1.x + w.w * b1.z;
            z1[q].y += w.x * b0.y + w.y * b0.w + w.z * b1.y + w.w * b1.w;
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < UN; ++q)
          for (int e = e0[q]; e < e1[q]; ++e) {
            const long at = (long)nl.lmx * nl.atom[e];
            for (int l = 0; l < nl.lmx; ++l) {
              const float v = nl.vnl[(long)nl.lmx * e + l];
              const float2 a = S0[at + l], b = S1[at + l];
              z0[q].x += v * a.x;
              z0[q].y += v * a.y;
              z1[q].x += v * b.x;
              z1[q].y += v * b.y;
            }
          }
      }
#pragma unroll
      for (int q = 0; q < UN; ++q) {
        const int i = ib + 128 * q;
        if (i >= NP) break;
        const int o = (i / NX) * LD + i % NX;
        T[o] = z0[q];
        T[NY * LD + o] = z1[q];
      }
    }
  }
  __syncthreads();
  float2 *Tp = T + h * (NY * LD);
  const bool on = h == 0 || two;
  if (on && u < NY) {
    float2 x[NX];
    float2 *row = Tp + u * LD;
#pragma unroll
    for (int i1 = 0; i1 < NX; ++i1) x[i1] = row[i1];
    rf::fft<float, -1, NX>(x);
    rf::static_for<0, MBX + 1>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      row[k] = x[out_pos(NX, k)];
      if constexpr (k > 0) row[NX - k] = x[out_pos(NX, NX - k)];
    });
  }
  __syncthreads();
  if (on && u < P1) {
    const int k1 = u - P.m1;
    const uint2 in = col_rows(P, u);
    const float2 *Tc = Tp + (k1 >= 0 ? k1 : NX + k1);
    float2 *A0 = bufA + ((long)(pl0 + h) * P.k3 + i3) * P.P2 * P1 + P.m2 * P1 + u;
    float2 x[NY];
#pragma unroll
    for (int i2 = 0; i2 < NY; ++i2) x[i2] = Tc[i2 * LD];
    rf::fft<float, -1, NY>(x);
    rf::static_for<0, MBY + 1>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      if ((in.x >> k) & 1u) A0[k * P1] = x[out_pos(NY, k)];
      if constexpr (k > 0)
        if ((in.y >> k) & 1u) A0[-k * P1] = x[out_pos(NY, NY - k)];
    });
  }
}

// ---------------------------------------------------------------------------
// The z transforms of the FP32 pipeline, one sphere z-column (j2, a) of one
// band pair per thread with the whole line in registers (replacing the
// shared-memory k_zinv / k_zfwd for the specialised lengths).  The column's
// coefficients come from the z-column table (col_ig, i3-major, so a warp's
// lookups are one row); positions without a sphere entry are zero.
//   inverse: two real bands packed as c_A + i c_B (their +G and -G halves),
//            backward z-FFT, written to bufA[pair][i3][j2][a];
//   forward: read the column from bufA, forward z-FFT, scale by 1/N and
//            scatter to zsph as k_zfwd does.
constexpr int ZC_T = 64;

template <int N, bool HALF>
__global__ void __launch_bounds__(ZC_T) k_zcols_inv(PipeParams P, const float *__restrict__ cin, long ldc,
                                                     float2 *__restrict__ bufA) {
  using rf::out_pos;
  const int q = blockIdx.x * ZC_T + threadIdx.x;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair) || q >= P.ncol) return;
  const int bA = P.pairs[2 * p], bB = P.pairs[2 * p + 1];
  const float *cA = cin + (long)bA * ldc;
  const float *cB = bB >= 0 ? cin + (long)bB * ldc : cA;
  constexpr int MB = line_mb<N, HALF>();   // samples beyond it are zero
  float2 x[N];
  z_gather<float, N, ZRows1<N, MB>>(
      cA, cB, bB >= 0, [&](auto ic) { return __ldg(P.col_ig + decltype(ic)::value * P.ncol + q); },
      [&](auto ic, float re, float im) { x[decltype(ic)::value] = make_float2(re, im); });
  rf::fft_nz<float, +1, N, MB>(x);
  float2 *dst = bufA + (long)pl * N * P.P2 * P.P1 + P.col_ja[q];
  rf::static_for<0, N>([&](auto ic) {
    constexpr int i3 = decltype(ic)::value;
    dst[(long)i3 * P.P2 * P.P1] = x[out_pos(N, i3)];
  });
}

template <int N, bool HALF>
__global__ void __launch_bounds__(ZC_T) k_zcols_fwd(PipeParams P, const float2 *__restrict__ bufA,
                                                     float2 *__restrict__ zsph) {
  using rf::out_pos;
  const int q = blockIdx.x * ZC_T + threadIdx.x;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair) || q >= P.ncol) return;
  const float2 *src = bufA + (long)pl * N * P.P2 * P.P1 + P.col_ja[q];
  float2 x[N];
#pragma unroll
  for (int i3 = 0; i3 < N; ++i3) x[i3] = src[(long)i3 * P.P2 * P.P1];
  rf::fft<float, -1, N>(x);
  z_scatter<float, N, ZRows1<N, line_mb<N, HALF>()>>(
      zsph + (long)pl * (P.nplw + 1) * 2, (float)P.inv_n,
      [&](auto ic) { return __ldg(P.col_ig + decltype(ic)::value * P.ncol + q); },
      [&](auto ic) { return x[out_pos(N, decltype(ic)::value)]; });
}


// The inverse z pass for the two-lanes-a-line lengths (N = 2H > 64): lanes
// 2c and 2c + 1 own sphere z-column c, each gathers the coefficients of the
// even or odd i3 and transforms them (H points), and the butterfly exchange
// of k_plane2 completes the N-point transform.  Whole warps run (lanes past
// the last column repeat it and store nothing).
template <int N, bool HALF>
__global__ void __launch_bounds__(ZC_T) k_zcols_inv2(PipeParams P, const float *__restrict__ cin, long ldc,
                                                      float2 *__restrict__ bufA) {
  using rf::out_pos;
  constexpr int H = N / 2;
  int q = (int)((blockIdx.x * ZC_T + threadIdx.x) >> 1);
  const int h = threadIdx.x & 1;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair)) return;   // uniform in the block
  const bool on = q < P.ncol;
  q = min(q, P.ncol - 1);
  const int bA = P.pairs[2 * p], bB = P.pairs[2 * p + 1];
  const float *cA = cin + (long)bA * ldc;
  const float *cB = bB >= 0 ? cin + (long)bB * ldc : cA;
  constexpr int MB = line_mb<N, HALF>();   // samples beyond it are zero
  float2 x[H] = {};
  z_gather<float, H, ZIn2<N, MB>>(
      cA, cB, bB >= 0, [&](auto ic) { return __ldg(P.col_ig + (2 * decltype(ic)::value + h) * P.ncol + q); },
      [&](auto ic, float re, float im) { x[decltype(ic)::value] = make_float2(re, im); });
  rf::fft_nz<float, +1, H, z2_bound<N, MB>()>(x);
  pl2::dit_combine<+1, N>(x, h);
  if (on) {
    float2 *dst = bufA + (long)pl * N * P.P2 * P.P1 + P.col_ja[q];
    rf::static_for<0, H>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      dst[(long)(k + h * H) * P.P2 * P.P1] = x[out_pos(H, k)];
    });
  }
}

// The forward z pass the same way: lane h of a column loads the samples 2j + h
// of bufA and, after the exchange, scatters the rows k + h H inside the sphere
// to zsph as k_zfwd does.
template <int N, bool HALF>
__global__ void __launch_bounds__(ZC_T) k_zcols_fwd2(PipeParams P, const float2 *__restrict__ bufA,
                                                     float2 *__restrict__ zsph) {
  using rf::out_pos;
  constexpr int H = N / 2, MB = line_mb<N, HALF>();
  int q = (int)((blockIdx.x * ZC_T + threadIdx.x) >> 1);
  const int h = threadIdx.x & 1;
  const int pl = blockIdx.y, p = P.pair0 + pl;
  if (p >= (P.npair_dev ? *P.npair_dev : P.npair)) return;   // uniform in the block
  const bool on = q < P.ncol;
  q = min(q, P.ncol - 1);
  const float2 *src = bufA + (long)pl * N * P.P2 * P.P1 + P.col_ja[q];
  float2 x[H];
#pragma unroll
  for (int j = 0; j < H; ++j) x[j] = src[(long)(2 * j + h) * P.P2 * P.P1];
  rf::fft<float, -1, H>(x);
  pl2::dit_combine<-1, N>(x, h);
  if (!on) return;
  z_scatter<float, H, ZOut2<N, MB>>(
      zsph + (long)pl * (P.nplw + 1) * 2, (float)P.inv_n,
      [&](auto ic) { return __ldg(P.col_ig + (decltype(ic)::value + h * H) * P.ncol + q); },
      [&](auto ic) { return x[out_pos(H, decltype(ic)::value)]; });
}

template <int N>
int zcols2_launch(const PipeParams &P, int npl, const float *cin, long ldc, float2 *bufA, const float2 *src,
                  float2 *zsph, bool inv, cudaStream_t st) {
  dim3 g((2 * P.ncol + ZC_T - 1) / ZC_T, npl);
  if (P.m3 <= line_mb<N, true>()) {
    if (inv) k_zcols_inv2<N, true><<<g, ZC_T, 0, st>>>(P, cin, ldc, bufA);
    else k_zcols_fwd2<N, true><<<g, ZC_T, 0, st>>>(P, src, zsph);
  } else {
    if (inv) k_zcols_inv2<N, false><<<g, ZC_T, 0, st>>>(P, cin, ldc, bufA);
    else k_zcols_fwd2<N, false><<<g, ZC_T, 0, st>>>(P, src, zsph);
  }
  note_launch();
  return 0;
}

template <int N>
int zcols_launch(const PipeParams &P, int npl, const float *cin, long ldc, float2 *bufA, const float2 *src,
                        float2 *zsph, bool inv, cudaStream_t st) {
  dim3 g((P.ncol + ZC_T - 1) / ZC_T, npl);
  if (P.m3 <= line_mb<N, true>()) {
    if (inv) k_zcols_inv<N, true><<<g, ZC_T, 0, st>>>(P, cin, ldc, bufA);
    else k_zcols_fwd<N, true><<<g, ZC_T, 0, st>>>(P, src, zsph);
  } else {
    if (inv) k_zcols_inv<N, false><<<g, ZC_T, 0, st>>>(P, cin, ldc, bufA);
    else k_zcols_fwd<N, false><<<g, ZC_T, 0, st>>>(P, src, zsph);
  }
  note_launch();
  return 0;
}

// Density for the same grids (softchg, chgdns.f90:388-454): per CTA one z
// plane and one group of band pairs; for each pair the backward y- and
// x-FFTs of the plane as above, then rho += occ_A/Omega psi_A(r)^2 +
// occ_B/Omega psi_B(r)^2 accumulated in FP64 in shared memory (each thread
// owns one grid row).  The group's partial plane goes to part[group]; a
// second kernel sums the groups in a fixed order, so the result is the same
// from run to run.
template <int NX, int NY, int PL, bool HALF>
__global__ void __launch_bounds__(64) k_rho_plane(PipeParams P, const float2 *__restrict__ bufA,
                                                  const double *__restrict__ wocc, double *__restrict__ part,
                                                  int npl, int per_group) {
  using rf::out_pos;
  using Rows = PlaneRows<NY, PL>;
  // PL = 2: planes i3 and i3 + 1, warp w taking plane w's columns in the y
  // phase (P1 <= 32); the x phase as in k_plane.
  const int i3b = blockIdx.x * PL, grp = blockIdx.y;
  constexpr int MBX = line_mb<NX, HALF>(), MBY = line_mb<NY, HALF>(), PB = 2 * MBX + 1, LA = NX | 1;
  const int npl_here = min(PL, P.k3 - i3b);
  constexpr int NP = NX * NY;
  // [PL][NY][LA] FP64 (a row's pitch keeps the rows of a warp in different
  // banks), then the [PL][NY][PB] complex tiles
  extern __shared__ double accs[];
  float2 *T = reinterpret_cast<float2 *>(accs + PL * NY * LA);
  const int t = threadIdx.x;
  const int cpl = (PL == 2) ? (t >> 5) : 0, col = (PL == 2) ? (t & 31) : t;
  const bool col_on = col < PB && cpl < npl_here;
  const int a0 = col - (MBX - P.m1);   // sphere column
  float2 *Tc = T + cpl * (NY * PB) + col;
  for (int i = t; i < PL * NY * LA; i += blockDim.x) accs[i] = 0.0;
  if (col_on && (a0 < 0 || a0 >= P.P1))
    for (int i = 0; i < NY; ++i) Tc[i * PB] = make_float2(0.f, 0.f);
  const int np = min(npl, (P.npair_dev ? *P.npair_dev : P.npair) - P.pair0);
  const int pl0 = grp * per_group, pl1 = min(np, pl0 + per_group);
  const int r = Rows::row(t);
  for (int pl = pl0; pl < pl1; ++pl) {
    const int p = P.pair0 + pl;
    if (col_on && a0 >= 0 && a0 < P.P1)
      plane_y_back<NY, MBY>(P, bufA + ((long)pl * P.k3 + i3b + cpl) * P.P2 * P.P1, a0, Tc, PB);
    __syncthreads();
    const int bA = P.pairs[2 * p], bB = P.pairs[2 * p + 1];
    const double fa = wocc[bA], fb = bB >= 0 ? wocc[bB] : 0.0;
    for (int pass = 0; pass < Rows::passes; ++pass) {
      const int rp = Rows::plane(t, pass);
      if (r < NY && rp < npl_here) {
        float2 x[NX];
        plane_x_back<NX, MBX>(T + (rp * NY + r) * PB, x);
        double *a = accs + (rp * NY + r) * LA;
        rf::static_for<0, NX>([&](auto ic) {
          constexpr int i1 = decltype(ic)::value, q = out_pos(NX, i1);
          const double re = x[q].x, im = x[q].y;
          a[i1] += fa * re * re + fb * im * im;
        });
      }
    }
    __syncthreads();
  }
  __syncthreads();
  for (int rp = 0; rp < npl_here; ++rp) {
    double *dst = part + ((long)grp * P.k3 + i3b + rp) * NP;
    for (int i = t; i < NP; i += blockDim.x) dst[i] = accs[(rp * NY + i / NX) * LA + i % NX];
  }
}

// The density pass for the two-threads-a-line lengths (see k_plane2): the
// y and x backward transforms by decimation in time, thread h of row l then
// adds the columns k + hH, k < H, of the row to the FP64 accumulation plane.
template <int N>
__global__ void __launch_bounds__(2 * N) k_rho_plane2(PipeParams P, const float2 *__restrict__ bufA,
                                                     const double *__restrict__ wocc, double *__restrict__ part,
                                                     int npl, int per_group) {
  using rf::out_pos;
  constexpr int H = N / 2;
  const int i3 = blockIdx.x, grp = blockIdx.y;
  const int P1 = P.P1, P2 = P.P2, m1 = P.m1, m2 = P.m2;
  extern __shared__ double accs[];            // [N][N] FP64, then the [N][P1] complex tile
  float2 *T = reinterpret_cast<float2 *>(accs + N * N);
  const int t = threadIdx.x, l = t >> 1, h = t & 1;
  const bool warp_on_cols = (t & ~31) < 2 * P1;
  const float2 zero = make_float2(0.f, 0.f);
  for (int i = t; i < N * N; i += 2 * N) accs[i] = 0.0;
  const int np = min(npl, (P.npair_dev ? *P.npair_dev : P.npair) - P.pair0);
  const int pl0 = grp * per_group, pl1 = min(np, pl0 + per_group);
  for (int pl = pl0; pl < pl1; ++pl) {
    const int p = P.pair0 + pl;
    const float2 *A = bufA + ((long)pl * P.k3 + i3) * P2 * P1;
    if (warp_on_cols) {
      const bool on = l < P1;
      float2 x[H];
#pragma unroll
      for (int j = 0; j < H; ++j) {
        const int i2 = 2 * j + h;
        const int j2 = (i2 <= m2) ? i2 + m2 : ((i2 >= N - m2) ? i2 - N + m2 : -1);
        float2 v = zero;
        if (on && j2 >= 0 && l >= P.row_lo[j2] && l <= P.row_hi[j2]) v = A[j2 * P1 + l];
        x[j] = v;
      }
      rf::fft<float, +1, H>(x);
      pl2::dit_combine<+1, N>(x, h);
      if (on) {
        rf::static_for<0, H>([&](auto kc) {
          constexpr int k = decltype(kc)::value;
          T[(k + h * H) * P1 + l] = x[out_pos(H, k)];
        });
      }
    }
    __syncthreads();
    {
      float2 x[H];
      const float2 *row = T + l * P1;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        const int i1 = 2 * j + h;
        float2 v = zero;
        if (i1 <= m1) v = row[i1 + m1];
        else if (i1 >= N - m1) v = row[i1 - N + m1];
        x[j] = v;
      }
      rf::fft<float, +1, H>(x);
      pl2::dit_combine<+1, N>(x, h);
      const int bA = P.pairs[2 * p], bB = P.pairs[2 * p + 1];
      const double fa = wocc[bA], fb = bB >= 0 ? wocc[bB] : 0.0;
      double *a = accs + l * N + h * H;
      rf::static_for<0, H>([&](auto kc) {
        constexpr int k = decltype(kc)::value, q = out_pos(H, k);
        const double re = x[q].x, im = x[q].y;
        a[k] += fa * re * re + fb * im * im;
      });
    }
    __syncthreads();
  }
  __syncthreads();
  double *dst = part + ((long)grp * P.k3 + i3) * N * N;
  for (int i = t; i < N * N; i += 2 * N) dst[i] = accs[i];
}

template <int NX, int NY, int PL, bool HALF>
static void rho_go(const PipeParams &P, int npl, const float2 *bufA, const double *wocc, double *part,
                   cudaStream_t st) {
  constexpr size_t sm = PL * NY * (sizeof(double) * (NX | 1) + sizeof(float2) * (2 * line_mb<NX, HALF>() + 1));
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_rho_plane<NX, NY, PL, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attr = true;
  }
  const int per_group = (npl + RHO_GROUPS - 1) / RHO_GROUPS;
  k_rho_plane<NX, NY, PL, HALF>
      <<<dim3((P.k3 + PL - 1) / PL, RHO_GROUPS), 64, sm, st>>>(P, bufA, wocc, part, npl, per_group);
}

template <int NX, int NY>
int rho_launch(const PipeParams &P, int npl, const float2 *bufA, const double *wocc, double *part, double *rho,
               int accumulate, cudaStream_t st) {
  // two planes a CTA where the half sphere fits 32 lanes
  if (P.m1 <= line_mb<NX, true>() && P.m2 <= line_mb<NY, true>()) {
    if (plane_pairs_enabled()) rho_go<NX, NY, 2, true>(P, npl, bufA, wocc, part, st);
    else rho_go<NX, NY, 1, true>(P, npl, bufA, wocc, part, st);
  } else {
    rho_go<NX, NY, 1, false>(P, npl, bufA, wocc, part, st);
  }
  note_launch();
  rho_groups_launch(part, (long)P.k1 * P.k2 * P.k3, rho, accumulate, st);
  return 0;
}

template <int N>
int rho2_launch(const PipeParams &P, int npl, const float2 *bufA, const double *wocc, double *part, double *rho,
                       int accumulate, cudaStream_t st) {
  const size_t sm = sizeof(double) * (size_t)N * N + sizeof(float2) * (size_t)N * P.P1;
  if (sm > 200 * 1024) return -1;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_rho_plane2<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    attr = true;
  }
  const int per_group = (npl + RHO_GROUPS - 1) / RHO_GROUPS;
  dim3 g(P.k3, RHO_GROUPS);
  k_rho_plane2<N><<<g, 2 * N, sm, st>>>(P, bufA, wocc, part, npl, per_group);
  note_launch();
  const long n = (long)P.k1 * P.k2 * P.k3;
  rho_groups_launch(part, n, rho, accumulate, st);
  return 0;
}

template <int NX, int NY, int PL, int U, bool HALF>
static void plane_go(const PipeParams &P, int npl, float2 *bufA, const float *vloct, cudaStream_t st) {
  constexpr size_t sm = sizeof(float2) * U * PL * NY * (2 * line_mb<NX, HALF>() + 1);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_plane<NX, NY, PL, U, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attr = true;
  }
  k_plane<NX, NY, PL, U, HALF>
      <<<dim3((P.k3 + PL - 1) / PL, (npl + U - 1) / U), 64 * U, sm, st>>>(P, bufA, vloct, npl);
}

template <int NX, int NY>
int plane_launch(const PipeParams &P, int npl, float2 *bufA, const float *vloct, cudaStream_t st) {
  const bool half = P.m1 <= line_mb<NX, true>() && P.m2 <= line_mb<NY, true>();
  if (half) {
    // two planes a unit (warp w takes plane w's columns) where 32 lanes hold the columns
    if constexpr (2 * line_mb<NX, true>() + 1 <= 32) {
      if (plane_pairs_enabled()) plane_go<NX, NY, 2, 2, true>(P, npl, bufA, vloct, st);
      else plane_go<NX, NY, 1, 1, true>(P, npl, bufA, vloct, st);
    } else {
      plane_go<NX, NY, 1, 1, true>(P, npl, bufA, vloct, st);
    }
  } else {
    plane_go<NX, NY, 1, 1, false>(P, npl, bufA, vloct, st);
  }
  note_launch();
  return 0;
}

template <int NX, int NY, bool HALF>
static void plane_r_go(const PipeParams &P, int npl, float2 *bufA, float2 *R, const float *vloc,
                       const NlPoints<float> *nl, cudaStream_t st) {
  constexpr size_t sm = sizeof(float2) * 2 * (size_t)NY * (NX | 1);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_plane_inv_r<NX, NY, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k_plane_fwd_r<NX, NY, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attr = true;
  }
  dim3 g(P.k3, (npl + 1) / 2);
  if (nl) k_plane_fwd_r<NX, NY, HALF><<<g, 128, sm, st>>>(P, R, bufA, vloc, *nl, npl);
  else k_plane_inv_r<NX, NY, HALF><<<g, 128, sm, st>>>(P, bufA, R, npl);
}

template <int NX, int NY>
int plane_r_launch(const PipeParams &P, int npl, float2 *bufA, float2 *R, const float *vloc,
                   const NlPoints<float> *nl, cudaStream_t st) {
  if (P.m1 <= line_mb<NX, true>() && P.m2 <= line_mb<NY, true>()) plane_r_go<NX, NY, true>(P, npl, bufA, R, vloc, nl, st);
  else plane_r_go<NX, NY, false>(P, npl, bufA, R, vloc, nl, st);
  note_launch();
  return 0;
}

template <int N, bool HALF>
static void plane2_go(const PipeParams &P, int npl, float2 *bufA, const float *vloct, cudaStream_t st) {
  constexpr size_t sm = sizeof(float2) * (size_t)N * plane2_pitch<N, HALF>();
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_plane2<N, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attr = true;
  }
  k_plane2<N, HALF><<<dim3(P.k3, npl), 2 * N, sm, st>>>(P, bufA, vloct);
}
template <int N>
int plane2_launch(const PipeParams &P, int npl, float2 *bufA, const float *vloct, cudaStream_t st) {
  if (P.m1 <= line_mb<N, true>() && P.m2 <= line_mb<N, true>()) plane2_go<N, true>(P, npl, bufA, vloct, st);
  else plane2_go<N, false>(P, npl, bufA, vloct, st);
  note_launch();
  return 0;
}

// Explicit instantiation of the launchers of one k1 x k2 plane shape.
#define QX_PLANE_GRID(NX, NY)                                                                                    \
  template int plane_launch<NX, NY>(const PipeParams &, int, float2 *, const float *, cudaStream_t);             \
  template int plane_r_launch<NX, NY>(const PipeParams &, int, float2 *, float2 *, const float *,                \
                                      const NlPoints<float> *, cudaStream_t);                                    \
  template int rho_launch<NX, NY>(const PipeParams &, int, const float2 *, const double *, double *, double *,   \
                                  int, cudaStream_t);
// ... and of the z-column launcher of one k3.
#define QX_ZCOLS_LENGTH(N)                                                                                      \
  template int zcols_launch<N>(const PipeParams &, int, const float *, long, float2 *, const float2 *, float2 *, \
                               bool, cudaStream_t);
// The same for the two-lanes-a-line kernels.
#define QX_PLANE_LENGTH2(N)                                                                                     \
  template int plane2_launch<N>(const PipeParams &, int, float2 *, const float *, cudaStream_t);                \
  template int rho2_launch<N>(const PipeParams &, int, const float2 *, const double *, double *, double *, int,  \
                              cudaStream_t);                                                                    \
  template int zcols2_launch<N>(const PipeParams &, int, const float *, long, float2 *, const float2 *, float2 *, \
                                bool, cudaStream_t);

}  // namespace qx
