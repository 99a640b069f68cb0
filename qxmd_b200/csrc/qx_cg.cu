// Batched BKL conjugate-gradient band update (eigen_BKL, eigen.f90:199-938,
// preconditioner prpcg eigen.f90:1093-1113, subgs4 engrad.f90:1196-1248).
// All bands iterate together; band ib is projected against the entry
// snapshot of bands < ib (subgs3, done as two GEMMs by the caller), which is
// the reference's result with one band per rank.  A cluster of CTAs a band (one
// CTA in k_cg_init); every reduction is accumulated in FP64.  Per-band state lives on the device, so a
// CG sweep needs no host round trip.
#include <cooperative_groups.h>

#include "qx_internal.h"
#include "qx_cg.h"

namespace qx {
namespace cg = cooperative_groups;

// One CTA per band; 1024 threads give each SM enough loads in flight for
// these bandwidth-bound sweeps over a band.
constexpr int CGT = 1024;

template <typename T>
__device__ __forceinline__ double ld(const T *p, long i) { return (double)p[i]; }

// Gamma-point inner product of two bands, block-wide.
template <typename T>
__device__ double bdot(const T *x, const T *y, int ne, double *red) {
  double s = 0.0;
  for (int i = threadIdx.x; i < ne; i += blockDim.x) s += ld(x, i) * ld(y, i);
  s = block_sum(s, red);
  return 2.0 * s - ld(x, 0) * ld(y, 0);
}

template <typename T>
__global__ void __launch_bounds__(CGT) k_cg_init(int ne, long ldx, const T *__restrict__ x,
                                                         const T *__restrict__ hx, T *__restrict__ g, CgState s) {
  __shared__ double red[CGT / 32];
  const int b = blockIdx.x;
  const T *xb = x + b * ldx, *hb = hx + b * ldx;
  T *gb = g + b * ldx;
  const double e = bdot(xb, hb, ne, red);
  double z = 0.0;
  for (int i = threadIdx.x; i < ne; i += blockDim.x) {
    const T v = (T)e * xb[i] - hb[i];
    gb[i] = v;
    z += (double)v * (double)v;
  }
  z = block_sum(z, red);
  z = 2.0 * z - ld(gb, 0) * ld(gb, 0);
  if (threadIdx.x == 0) {
    s.eig[b] = e;
    s.zansa[b] = z;
    s.zansab[b] = z;
    s.z000re[b] = z;
    s.x000re[b] = 1.0e10;
    s.eigb[b] = e;
    s.dinnerx[b] = 0.0;
    s.betk[b] = 0.0;
    s.izcnt[b] = 0;
    s.lreset[b] = 1;
    s.iter[b] = 0;
    s.active[b] = 1;
  }
}

// prpcg (eigen.f90:1093-1113), e15 = 1.5 ekib.
__device__ __forceinline__ double prpcg(double dk, double e15) {
  // t / (t + 16 x^4) * 2 / e15 at x = dk / e15, numerator and denominator
  // times e15^4: one division
  const double a = dk, e = e15, e2 = e * e;
  const double t = e * (27.0 * e2 + a * (18.0 * e + 12.0 * a)) + 8.0 * (a * a) * a;   // e15^3 t
  const double a2 = a * a;
  return 2.0 * t / (e * t + 16.0 * a2 * a2);
}

// The batched sweeps run a cluster of CGC CTAs of CGB threads a band, CGU
// elements a thread at a time with the loads first.  L2 latency bounds them
// (a band of Si64 is nine elements a thread), so loads in flight and the
// spread over the SMs matter: one CTA of 1024 threads a band left 160 CTAs on
// 148 SMs and one load a thread in flight; in CTAs of 256 threads at most 48
// registers keep five a SM, and 160 bands fit one wave.  At Si64, FP32: update
// 17.4 -> 13.7 us, preconditioner 15.2 -> 10.6 us, projection 12.4 -> 6.4 us.
constexpr int CGC = 4, CGB = 256, CGS = CGC * CGB;
template <typename T> constexpr int cgu() { return sizeof(T) == 4 ? 5 : 3; }

// Sums of NV values over the C CTAs of a cluster, the same in every thread:
// each CTA leaves its sums in its own shared memory (slot, of its own for
// each use), and after the cluster barrier every warp reads them rank by rank.
template <int NV, int C>
__device__ __forceinline__ void cluster_sums(double (&v)[NV], double (*red)[32], double *slot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0) red[k][warp] = v[k];
  }
  __syncthreads();
  if (warp < NV) {
    double r = lane < nw ? red[warp][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (lane == 0) slot[warp] = r;
  }
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double r = cl.map_shared_rank(slot, lane & (C - 1))[k];
#pragma unroll
    for (int o = C / 2; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    v[k] = r;
  }
}

// The active-band list and the band pairs of the FFT pipeline, by one warp: 32
// bands a round with a ballot and a population-count prefix.
__device__ __forceinline__ void cg_list(int nb, const CgState &s) {
  const int lane = threadIdx.x;
  int n = 0;
  for (int b0 = 0; b0 < nb; b0 += 32) {
    const int b = b0 + lane;
    const bool act = (b < nb) && s.active[b];
    const unsigned m = __ballot_sync(0xffffffffu, act);
    if (act) s.list[n + __popc(m & ((1u << lane) - 1u))] = b;
    n += __popc(m);
  }
  __syncwarp();
  for (int p = lane; p < (n + 1) / 2; p += 32) {
    s.pairs[2 * p] = s.list[2 * p];
    s.pairs[2 * p + 1] = (2 * p + 1 < n) ? s.list[2 * p + 1] : -1;
  }
  if (lane == 0) {
    *s.nact = n;
    *s.npair = (n + 1) / 2;
  }
}

// g <- prcd * g; zansap = <g|g>; h <- g + beta*h (h <- g on reset).  One more
// cluster after those of the bands writes the active-band list (the sweep
// leaves `active` alone), which the H|h> that follows reads.
template <typename T>
__global__ void __cluster_dims__(CGC, 1, 1) __launch_bounds__(CGB, 5) k_cg_prec(int nb, int ne, long ldx, T *__restrict__ g, T *__restrict__ h,
                                                         const double *__restrict__ dk, CgState s) {
  constexpr int U = cgu<T>();
  __shared__ double red[1][32], slot[1];
  const int b = blockIdx.x / CGC;
  if (b == nb) {
    if (blockIdx.x % CGC == 0 && threadIdx.x < 32) cg_list(nb, s);
    return;
  }
  if (!s.active[b]) return;
  T *gb = g + b * ldx, *hb = h + b * ldx;
  const double e15 = 1.5 * s.ekib[b];
  const int reset = s.lreset[b], i00 = (blockIdx.x % CGC) * CGB + threadIdx.x;
  const double zold = s.betk[b];
  double z[1] = {0.0};
  for (int i0 = i00; i0 < ne; i0 += U * CGS) {
    T gv[U];
    double d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u * CGS, ne - 1);
      gv[u] = gb[i];
      d[u] = dk[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * CGS;
      if (i >= ne) break;
      const T v = (T)((double)gv[u] * prpcg(d[u], e15));
      gb[i] = v;
      z[0] += (i == 0 ? 1.0 : 2.0) * (double)v * (double)v;
    }
  }
  cluster_sums<1, CGC>(z, red, slot);
  const T beta = reset ? (T)0 : (T)(z[0] / zold);
  for (int i0 = i00; i0 < ne; i0 += U * CGS) {
    T gv[U], hv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u * CGS, ne - 1);
      gv[u] = gb[i];
      hv[u] = reset ? (T)0 : hb[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * CGS;
      if (i < ne) hb[i] = gv[u] + beta * hv[u];
    }
  }
  cg::this_cluster().sync();   // no CTA leaves, and no state changes, while another still reads
  if (blockIdx.x % CGC == 0 && threadIdx.x == 0) {
    s.lreset[b] = 0;
    s.betk[b] = z[0];
    s.iter[b] += 1;
  }
}

// subgs4: h -= <x|h> x.
template <typename T>
__global__ void __cluster_dims__(CGC, 1, 1) __launch_bounds__(CGB, 5) k_cg_orth(int ne, long ldx, const T *__restrict__ x, T *__restrict__ h,
                                                 CgState s) {
  constexpr int U = cgu<T>();
  __shared__ double red[1][32], slot[1];
  const int b = blockIdx.x / CGC, i00 = (blockIdx.x % CGC) * CGB + threadIdx.x;
  if (!s.active[b]) return;
  const T *xb = x + b * ldx;
  T *hb = h + b * ldx;
  double d[1] = {0.0};
  for (int i0 = i00; i0 < ne; i0 += U * CGS) {
    T xv[U], hv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u * CGS, ne - 1);
      xv[u] = xb[i];
      hv[u] = hb[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * CGS;
      if (i < ne) d[0] += (i == 0 ? 1.0 : 2.0) * (double)xv[u] * (double)hv[u];
    }
  }
  cluster_sums<1, CGC>(d, red, slot);
  const T hhx = (T)d[0];
  for (int i0 = i00; i0 < ne; i0 += U * CGS) {
    T xv[U], hv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u * CGS, ne - 1);
      xv[u] = xb[i];
      hv[u] = hb[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * CGS;
      if (i < ne) hb[i] = hv[u] - hhx * xv[u];
    }
  }
  cg::this_cluster().sync();   // no CTA leaves while another still reads its sum
}

// BKL 2x2 step (eigen.f90:593-622): the new eigenvalue e, the step dtnew
// along h and the normalisation alpsq, from cai = <h|hx>, cbi = <h|gh>,
// hhi = <h|h> > 0.
__device__ __forceinline__ void bkl_step(double cai, double cbi, double hhi, double &e, double &dtnew,
                                         double &alpsq) {
  const double h11 = e, h12 = cai / sqrt(hhi), h21 = h12, h22 = cbi / hhi;
  const double enew = 0.5 * (h11 + h22 - sqrt((h11 + h22) * (h11 + h22) - 4.0 * (h11 * h22 - h12 * h21)));
  dtnew = (enew - h11) / h12 / sqrt(hhi);
  alpsq = sqrt(1.0 / (1.0 + dtnew * (0.0 + dtnew * hhi)));
  e = enew;
}

// Line minimisation (eigen.f90:624-695) for hhi = 0, with hhx = <h|x>; *dmax
// receives a larger inner product than dinx.
__device__ __forceinline__ void bkl_line(double cai, double cbi, double hhi, double hhx, double dinx,
                                         const CgParm &pm, double *dmax, bool writer, double &e, double &dtnew,
                                         double &alpsq) {
  const double c0 = e, c1 = cai, c2 = cbi, c3 = hhi, c4 = 2.0 * hhx;
  const double s0 = c0 * c4 - c1, s1 = c0 * c3 - c2, s2 = c1 * c3 - c2 * c4;
  const double sr = s1 * s1 - s2 * s0;
  dtnew = (sr > 0.0) ? (-s1 - sqrt(sr)) / s2 : -1.0;
  if (dtnew > 0.0) {
    const double dinner = sqrt(1.0 / (1.0 + dtnew * dtnew * hhi));
    if (dinner < pm.threinn) dtnew = 0.0;
    if (dinner < dinx * pm.wdinner) dtnew = 0.0;
    if (writer && dinner > dinx) *dmax = dinner;
  }
  const double d2 = dtnew * dtnew;
  const double alpsq2 = 1.0 / (1.0 + dtnew * c4 + d2 * c3);
  e = (c0 + dtnew * c1 + d2 * c2) * alpsq2;
  alpsq = sqrt(alpsq2);
}

// Convergence test of band b after step `iter` (eigen.f90:731-764) and its
// state for the next one; true when the band stops.
__device__ __forceinline__ bool bkl_stop(const CgState &s, const CgParm &pm, int b, int iter, double e,
                                         double zansa) {
  const double de = fabs(s.eigb[b] - e);
  const bool stop = (b < pm.noband && iter >= pm.itermx) || (b >= pm.noband && iter >= pm.iteremx) ||
                    zansa < pm.tolera || de < pm.tolera || zansa < s.z000re[b] * pm.roughfzan ||
                    (iter > 1 && de < s.x000re[b] * pm.roughfeig);
  s.eig[b] = e;
  s.zansa[b] = zansa;
  if (stop) {
    s.active[b] = 0;
  } else {
    if (iter == 1) s.x000re[b] = de;
    if (zansa > s.zansab[b]) {
      if (++s.izcnt[b] > 20) { s.izcnt[b] = 0; s.lreset[b] = 1; }
    }
    s.zansab[b] = zansa;
    s.eigb[b] = e;
  }
  return stop;
}

// x/hx update (eigen.f90:698-709), residual and convergence test of every
// active band.
template <typename T>
__global__ void __cluster_dims__(CGC, 1, 1) __launch_bounds__(CGB, 5) k_cg_update(int ne, long ldx, T *__restrict__ x, T *__restrict__ hx,
                                                      T *__restrict__ g, const T *__restrict__ h,
                                                      const T *__restrict__ gh, CgState s, CgParm pm) {
  constexpr int U = cgu<T>();
  __shared__ double red[3][32], slot[3][4];
  const int b = blockIdx.x / CGC, i00 = (blockIdx.x % CGC) * CGB + threadIdx.x;
  const bool first = blockIdx.x % CGC == 0 && threadIdx.x == 0;
  if (!s.active[b]) return;
  T *xb = x + b * ldx, *hxb = hx + b * ldx, *gb = g + b * ldx;
  const T *hb = h + b * ldx, *ghb = gh + b * ldx;
  const double dinx = s.dinnerx[b];   // the state is read before the first cluster barrier
  double e = s.eig[b];
  double v[3] = {0.0, 0.0, 0.0};      // <h|hx>, <h|gh>, <h|h>
  for (int i0 = i00; i0 < ne; i0 += U * CGS) {
    T a[U], c[U], d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u * CGS, ne - 1);
      a[u] = hb[i];
      c[u] = hxb[i];
      d[u] = ghb[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * CGS;
      if (i >= ne) break;
      const double hv = (double)a[u], hf = (i == 0 ? 1.0 : 2.0) * hv;
      v[0] += hf * (double)c[u];
      v[1] += hf * (double)d[u];
      v[2] += hf * hv;
    }
  }
  cluster_sums<3, CGC>(v, red, slot[0]);
  double dtnew, alpsq;
  if (v[2] > 0.0) {
    bkl_step(v[0], v[1], v[2], e, dtnew, alpsq);
  } else {
    double w[1] = {0.0};
    for (int i = i00; i < ne; i += CGS) w[0] += (i == 0 ? 1.0 : 2.0) * (double)hb[i] * (double)xb[i];
    __syncthreads();
    cluster_sums<1, CGC>(w, red, slot[1]);
    bkl_line(v[0], v[1], v[2], w[0], dinx, pm, &s.dinnerx[b], first, e, dtnew, alpsq);
  }
  const T al = (T)alpsq, dt = (T)dtnew, et = (T)e;
  double z[1] = {0.0};
  for (int i0 = i00; i0 < ne; i0 += U * CGS) {
    T a[U], c[U], d[U], f[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u * CGS, ne - 1);
      a[u] = hb[i];
      c[u] = hxb[i];
      d[u] = ghb[i];
      f[u] = xb[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * CGS;
      if (i >= ne) break;
      const T xn = al * (f[u] + dt * a[u]);
      const T hn = al * (c[u] + dt * d[u]);
      xb[i] = xn;
      hxb[i] = hn;
      const T gv = et * xn - hn;
      gb[i] = gv;
      z[0] += (i == 0 ? 1.0 : 2.0) * (double)gv * (double)gv;
    }
  }
  __syncthreads();
  cluster_sums<1, CGC>(z, red, slot[2]);
  cg::this_cluster().sync();   // no CTA leaves while another still reads its sums
  if (first) bkl_stop(s, pm, b, s.iter[b], e, z[0]);
}

// ---- the one-rank band order ------------------------------------------------
// A CG step of band *cur is a chain of kernels in a graph loop, so its length
// in kernels and the slowest of them bound it.  The step is arranged so that
// every sweep over the band runs on many CTAs and every reduction ends in the
// kernel that needs it:
//   * g is kept preconditioned (g <- prcd (e x - hx), with zp = <g|g>), so
//     h = g + beta h (beta = zp / zp of the previous step) is formed where it
//     is read;
//   * k_seq_dots: p_j = <s_j|h> and q_j = <s_j|x> for the snapshot columns
//     s_j of the bands below, and <x|h>;
//   * k_seq_axpy_h: subgs3 and subgs4 in one pass, h <- h - sum_j p_j s_j -
//     hhx x with hhx = <x|h> - sum_j p_j q_j = <x|h - sum_j p_j s_j>;
//   * H|h>: the FFT pipeline beside the two KB kernels;
//   * k_seq_update, one cluster of CTAs: <h|hx>, <h|gh>, <h|h>, the BKL step,
//     x, hx, g, the residual and the next band.
// Before this the step ran thirteen kernels in a row, four of them (g and h,
// the projection on x, the update) sweeping the band on one SM.
// One sweep at Si64 (FP64, 160 bands): 25.6 -> 16.2 ms.

// g = prcd (e x - hx) of every band at entry, with its <g|g> before (z) and
// after (zp, in s.cai) the preconditioner.
template <typename T>
__global__ void __launch_bounds__(CGT) k_seq_init(int ne, long ldx, const T *__restrict__ x,
                                                  const T *__restrict__ hx, T *__restrict__ g,
                                                  const double *__restrict__ dk, CgState s) {
  __shared__ double red[CGT / 32];
  const int b = blockIdx.x;
  const T *xb = x + b * ldx, *hb = hx + b * ldx;
  T *gb = g + b * ldx;
  const double e = bdot(xb, hb, ne, red), e15 = 1.5 * s.ekib[b];
  double z = 0.0, zp = 0.0;
  for (int i = threadIdx.x; i < ne; i += blockDim.x) {
    const T v = (T)e * xb[i] - hb[i];
    const T w = (T)((double)v * prpcg(dk[i], e15));
    gb[i] = w;
    const double f = i == 0 ? 1.0 : 2.0;
    z += f * (double)v * (double)v;
    zp += f * (double)w * (double)w;
  }
  z = block_sum(z, red);
  zp = block_sum(zp, red);
  if (threadIdx.x == 0) {
    s.eig[b] = e;
    s.zansa[b] = z;
    s.zansab[b] = z;
    s.z000re[b] = z;
    s.x000re[b] = 1.0e10;
    s.eigb[b] = e;
    s.dinnerx[b] = 0.0;
    s.betk[b] = 0.0;
    s.cai[b] = zp;
    s.izcnt[b] = 0;
    s.lreset[b] = 1;
    s.iter[b] = 0;
    s.active[b] = 1;
  }
}

__global__ void k_seq_reset(SeqArgs q) {
  *q.cur = 0;
  q.pairs[0] = 0;
  q.pairs[1] = -1;
}

// h of band b before the projections (the previous h does not enter after a reset).
template <typename T>
__device__ __forceinline__ T seq_h(const T *gb, const T *hb, int i, T beta, bool reset) {
  return reset ? gb[i] : gb[i] + beta * hb[i];
}

// CTA j < b: p[j], q[j]; CTA b: p[b] = <x|h>.
constexpr int SQD_T = 512;
template <typename T>
__global__ void __launch_bounds__(SQD_T) k_seq_dots(int ne, long ldx, const T *__restrict__ snap,
                                                    const T *__restrict__ x, const T *__restrict__ g,
                                                    const T *__restrict__ h, CgState s,
                                                    const int *__restrict__ cur, int nb, double *__restrict__ p,
                                                    double *__restrict__ q) {
  __shared__ double red[2][SQD_T / 32];
  const int b = *cur, j = blockIdx.x;
  if (b >= nb || j > b) return;
  const T *xb = x + b * ldx, *gb = g + b * ldx, *hb = h + b * ldx;
  const T *v = j < b ? snap + j * ldx : xb;
  const bool reset = s.lreset[b];
  const T beta = reset ? (T)0 : (T)(s.cai[b] / s.betk[b]);
  double sh = 0.0, sx = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < ne; i += SQD_T) {
    const double f = i == 0 ? 1.0 : 2.0, a = f * (double)v[i];
    sh += a * (double)seq_h(gb, hb, i, beta, reset);
    sx += a * (double)xb[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sh += __shfl_xor_sync(0xffffffffu, sh, o);
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { red[0][warp] = sh; red[1][warp] = sx; }
  __syncthreads();
  if (warp < 2) {
    double r = lane < SQD_T / 32 ? red[warp][lane] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (lane == 0) {
      if (warp == 0) p[j] = r;
      else if (j < b) q[j] = r;
    }
  }
}

// h <- h - sum_{j<b} p_j s_j - hhx x: a CTA owns 32 consecutive rows (one per
// lane); warp w takes j = w, w + 8, ..., and the eight partial sums are added
// in a fixed order.
template <typename T>
__global__ void __launch_bounds__(256) k_seq_axpy_h(int ne, long ldx, const T *__restrict__ snap,
                                                    const T *__restrict__ x, const T *__restrict__ g,
                                                    T *__restrict__ h, CgState s, const int *__restrict__ cur,
                                                    int nb, const double *__restrict__ p,
                                                    const double *__restrict__ q) {
  __shared__ double part[8][33];
  __shared__ double pq[8];
  const int b = *cur;
  if (b >= nb) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double acc = 0.0, c = 0.0;
  if (i < ne) {
    int j = w;
    for (; j + 24 < b; j += 32) {
      const T a0 = snap[j * ldx + i], a1 = snap[(j + 8) * ldx + i];
      const T a2 = snap[(j + 16) * ldx + i], a3 = snap[(j + 24) * ldx + i];
      acc += p[j] * (double)a0;
      acc += p[j + 8] * (double)a1;
      acc += p[j + 16] * (double)a2;
      acc += p[j + 24] * (double)a3;
    }
    for (; j < b; j += 8) acc += p[j] * (double)snap[j * ldx + i];
  }
  for (int j = threadIdx.x; j < b; j += 256) c += p[j] * q[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  part[w][lane] = acc;
  if (lane == 0) pq[w] = c;
  __syncthreads();
  if (w == 0 && i < ne) {
    double t = 0.0, d = 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      t += part[u][lane];
      d += pq[u];
    }
    const bool reset = s.lreset[b];
    const T beta = reset ? (T)0 : (T)(s.cai[b] / s.betk[b]);
    T *hb = h + b * ldx;
    const double hv = (double)seq_h(g + b * ldx, (const T *)hb, i, beta, reset);
    hb[i] = (T)(hv - t - (p[b] - d) * (double)x[b * ldx + i]);
  }
}

constexpr int SQU_C = 8;   // CTAs of the update's cluster (the portable limit)

// The update of band *cur by one cluster; when the band stops, its final
// vector has become its snapshot column (cgjr(:,ib) = gdcr(:,ibb),
// eigen.f90:699, real*4 when q.ccreal4) and the next band starts.
template <typename T>
__global__ void __cluster_dims__(SQU_C, 1, 1) __launch_bounds__(CGT)
    k_seq_update(int ne, long ldx, T *__restrict__ x, T *__restrict__ hx, T *__restrict__ g, const T *__restrict__ h,
                 const T *__restrict__ gh, const double *__restrict__ dk, CgState s, CgParm pm, SeqArgs q) {
  __shared__ double red[3][32];
  __shared__ double slot[3][4];
  cg::cluster_group cl = cg::this_cluster();
  const int b = *q.cur;   // every CTA reads it before the first cluster barrier
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  if (b >= q.nb) {        // the same in every CTA
    if (first) cudaGraphSetConditional(q.handle, 0);
    return;
  }
  T *xb = x + b * ldx, *hxb = hx + b * ldx, *gb = g + b * ldx, *sb = (T *)q.snap + b * ldx;
  const T *hb = h + b * ldx, *ghb = gh + b * ldx;
  const double dinx = s.dinnerx[b], e15 = 1.5 * s.ekib[b];
  double e = s.eig[b], dtnew, alpsq;
  const int i0 = blockIdx.x * CGT + threadIdx.x, step = SQU_C * CGT;
  double v[3] = {0.0, 0.0, 0.0};
  for (int i = i0; i < ne; i += step) {
    const double f = i == 0 ? 1.0 : 2.0, hv = (double)hb[i];
    v[0] += f * hv * (double)hxb[i];
    v[1] += f * hv * (double)ghb[i];
    v[2] += f * hv * hv;
  }
  cluster_sums<3, SQU_C>(v, red, slot[0]);
  if (v[2] > 0.0) {
    bkl_step(v[0], v[1], v[2], e, dtnew, alpsq);
  } else {                // the same in every thread of the cluster
    double w[1] = {0.0};
    for (int i = i0; i < ne; i += step) w[0] += (i == 0 ? 1.0 : 2.0) * (double)hb[i] * (double)xb[i];
    __syncthreads();
    cluster_sums<1, SQU_C>(w, red, slot[1]);
    bkl_line(v[0], v[1], v[2], w[0], dinx, pm, &s.dinnerx[b], first, e, dtnew, alpsq);
  }
  const T a = (T)alpsq, dt = (T)dtnew, et = (T)e;
  double z[2] = {0.0, 0.0};
  for (int i = i0; i < ne; i += step) {
    const T xn = a * (xb[i] + dt * hb[i]);
    const T hn = a * (hxb[i] + dt * ghb[i]);
    xb[i] = xn;
    hxb[i] = hn;
    sb[i] = q.ccreal4 ? (T)(float)xn : xn;
    const T gv = et * xn - hn;
    const T gp = (T)((double)gv * prpcg(dk[i], e15));
    gb[i] = gp;
    const double f = i == 0 ? 1.0 : 2.0;
    z[0] += f * (double)gv * (double)gv;
    z[1] += f * (double)gp * (double)gp;
  }
  __syncthreads();
  cluster_sums<2, SQU_C>(z, red, slot[2]);
  if (first) {
    const int iter = s.iter[b] + 1;
    s.iter[b] = iter;
    s.lreset[b] = 0;
    s.betk[b] = s.cai[b];
    s.cai[b] = z[1];
    if (bkl_stop(s, pm, b, iter, e, z[0])) {
      const int nx = b + 1;
      *q.cur = nx;
      q.pairs[0] = nx;
      q.pairs[1] = -1;
      if (nx >= q.nb) cudaGraphSetConditional(q.handle, 0);
    }
  }
  cl.sync();   // no CTA leaves while another still reads its sums
}

// KB projections of band *cur: out[j] = scale_j (2 sum B_j y - B_j(0) y(0) -
// 2 B_j(1) y(1)), one CTA per projector j.
template <typename T>
__global__ void __launch_bounds__(256) k_seq_kb_dots(int ne, const T *__restrict__ V, long ldv,
                                                     const T *__restrict__ Y, long ldy, const int *__restrict__ cur,
                                                     const T *__restrict__ scale, double *__restrict__ out) {
  __shared__ double red[8];
  const int j = blockIdx.x;
  const T *v = V + j * ldv, *y = Y + (long)*cur * ldy;
  double sum = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < ne; i += 256) sum += (double)v[i] * (double)y[i];
  sum = block_sum(sum, red);
  if (threadIdx.x == 0)
    out[j] = (2.0 * sum - (double)v[0] * (double)y[0] - 2.0 * (double)v[1] * (double)y[1]) * (double)scale[j];
}

// Y_cur(i) = sum_j coef_j B_j(i) (rows and order as in k_seq_axpy_h).
template <typename T>
__global__ void __launch_bounds__(256) k_seq_kb_axpy(int n, int ne, const T *__restrict__ V, long ldv,
                                                     const double *__restrict__ coef, T *__restrict__ Y, long ldy,
                                                     const int *__restrict__ cur) {
  __shared__ double part[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double acc = 0.0;
  if (i < ne) {
    int j = w;
    for (; j + 24 < n; j += 32) {
      const T a0 = V[(long)j * ldv + i], a1 = V[(long)(j + 8) * ldv + i];
      const T a2 = V[(long)(j + 16) * ldv + i], a3 = V[(long)(j + 24) * ldv + i];
      acc += coef[j] * (double)a0;
      acc += coef[j + 8] * (double)a1;
      acc += coef[j + 16] * (double)a2;
      acc += coef[j + 24] * (double)a3;
    }
    for (; j < n; j += 8) acc += coef[j] * (double)V[(long)j * ldv + i];
  }
  part[w][lane] = acc;
  __syncthreads();
  if (w == 0 && i < ne) {
    double t = 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) t += part[u][lane];
    Y[(long)*cur * ldy + i] = (T)t;
  }
}

// ekinetic2 (engrad.f90:75-127): ekib(b) = 2*<c|T|c>, and sum occ*<c|T|c>
// into *ekin (one CTA per band writes its term; summed by k_sum_occ).
template <typename T>
__global__ void __launch_bounds__(CGT) k_ekin(int ne, long ldx, const T *__restrict__ x,
                                                      const double *__restrict__ dk, double *__restrict__ ekib) {
  __shared__ double red[CGT / 32];
  const int b = blockIdx.x;
  const T *xb = x + b * ldx;
  double s = 0.0;
  for (int i = threadIdx.x; i < ne; i += blockDim.x) s += dk[i] * ld(xb, i) * ld(xb, i);
  s = block_sum(s, red);
  if (threadIdx.x == 0) ekib[b] = 2.0 * (2.0 * s - dk[0] * ld(xb, 0) * ld(xb, 0));
}

// gradresnv (engrad.f90:1013-1067): per-band |eig*c - hc|^2 (Gamma metric).
template <typename T>
__global__ void __launch_bounds__(CGT) k_gradres(int ne, long ldx, const T *__restrict__ x,
                                                         const T *__restrict__ hx, const double *__restrict__ eig,
                                                         double *__restrict__ prod) {
  __shared__ double red[CGT / 32];
  const int b = blockIdx.x;
  const T *xb = x + b * ldx, *hb = hx + b * ldx;
  const double e = eig[b];
  double s = 0.0;
  for (int i = threadIdx.x; i < ne; i += blockDim.x) {
    const double r = e * ld(xb, i) - ld(hb, i);
    s += r * r;
  }
  s = block_sum(s, red);
  const double r0 = e * ld(xb, 0) - ld(hb, 0);
  if (threadIdx.x == 0) prod[b] = 2.0 * s - r0 * r0;
}

// Device-side summaries for a sync-free SCF iteration: out[0] = max_b prod,
// out[1] = sum_b occ_b prod_b (gradresnv's zmax and occupation-weighted sum).
__global__ void k_gradres_stats(const double *__restrict__ prod, const double *__restrict__ occ, int nb,
                                double *__restrict__ out) {
  const int lane = threadIdx.x;
  double m = 0.0, s = 0.0;
  for (int b = lane; b < nb; b += 32) {
    m = fmax(m, prod[b]);
    if (occ) s += occ[b] * prod[b];
  }
  for (int o = 16; o > 0; o >>= 1) {
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  if (lane == 0) { out[0] = m; out[1] = s; }
}

// *out = sum of the per-band CG iteration counts (H|psi> band applications).
__global__ void k_iter_sum(const int *__restrict__ iter, int nb, int *__restrict__ out) {
  const int lane = threadIdx.x;
  int s = 0;
  for (int b = lane; b < nb; b += 32) s += iter[b];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) *out = s;
}

// Row scaling of the projection matrix P (nproj x ncol, column-major, columns
// through colmap): P(j, n) *= v(j).
template <typename T>
__global__ void k_scale_rows(int nproj, int ncol, T *__restrict__ P, long ldp, const T *__restrict__ v,
                             const int *__restrict__ colmap, const int *__restrict__ ncol_dev) {
  const int nc = ncol_dev ? min(ncol, *ncol_dev) : ncol;
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= (long)nproj * nc) return;
  const int n = (int)(e / nproj), j = (int)(e - (long)n * nproj);
  const long cn = colmap ? colmap[n] : n;
  P[cn * ldp + j] *= v[j];
}

// ---- launchers -------------------------------------------------------------
template <typename T> void cg_init(int nb, int ne, long ldx, const T *x, const T *hx, T *g, const CgState &s, cudaStream_t st) {
  k_cg_init<T><<<nb, CGT, 0, st>>>(ne, ldx, x, hx, g, s); note_launch();
}
template <typename T> void cg_prec(int nb, int ne, long ldx, T *g, T *h, const double *dk, const CgState &s, cudaStream_t st) {
  k_cg_prec<T><<<(nb + 1) * CGC, CGB, 0, st>>>(nb, ne, ldx, g, h, dk, s); note_launch();
}
template <typename T> void cg_orth(int nb, int ne, long ldx, const T *x, T *h, const CgState &s, cudaStream_t st) {
  k_cg_orth<T><<<nb * CGC, CGB, 0, st>>>(ne, ldx, x, h, s); note_launch();
}
void gradres_stats(const double *prod, const double *occ, int nb, double *out, cudaStream_t st) {
  k_gradres_stats<<<1, 32, 0, st>>>(prod, occ, nb, out); note_launch();
}
void iter_sum(const int *iter, int nb, int *out, cudaStream_t st) { k_iter_sum<<<1, 32, 0, st>>>(iter, nb, out); note_launch(); }
template <typename T> void cg_update(int nb, int ne, long ldx, T *x, T *hx, T *g, const T *h, const T *gh,
                                     const CgState &s, const CgParm &pm, cudaStream_t st) {
  k_cg_update<T><<<nb * CGC, CGB, 0, st>>>(ne, ldx, x, hx, g, h, gh, s, pm); note_launch();
}
template <typename T> void seq_init(int nb, int ne, long ldx, const T *x, const T *hx, T *g, const double *dk,
                                    const CgState &s, const SeqArgs &q, cudaStream_t st) {
  k_seq_init<T><<<nb, CGT, 0, st>>>(ne, ldx, x, hx, g, dk, s); note_launch();
  k_seq_reset<<<1, 1, 0, st>>>(q); note_launch();
}
template <typename T> void seq_project(int ne, long ldx, const T *x, const T *g, T *h, const CgState &s,
                                       const SeqArgs &q, double *p, double *w, cudaStream_t st) {
  k_seq_dots<T><<<q.nb, SQD_T, 0, st>>>(ne, ldx, (const T *)q.snap, x, g, h, s, q.cur, q.nb, p, w); note_launch();
  k_seq_axpy_h<T><<<(ne + 31) / 32, 256, 0, st>>>(ne, ldx, (const T *)q.snap, x, g, h, s, q.cur, q.nb, p, w);
  note_launch();
}
template <typename T> void seq_kb(int np, int ne, const T *kbg, const T *scale, const T *h, T *gh, long ldx,
                                  const int *cur, double *coef, cudaStream_t st) {
  k_seq_kb_dots<T><<<np, 256, 0, st>>>(ne, kbg, ne, h, ldx, cur, scale, coef); note_launch();
  k_seq_kb_axpy<T><<<(ne + 31) / 32, 256, 0, st>>>(np, ne, kbg, ne, coef, gh, ldx, cur); note_launch();
}
template <typename T> void seq_update(int ne, long ldx, T *x, T *hx, T *g, const T *h, const T *gh, const double *dk,
                                      const CgState &s, const CgParm &pm, const SeqArgs &q, cudaStream_t st) {
  k_seq_update<T><<<SQU_C, CGT, 0, st>>>(ne, ldx, x, hx, g, h, gh, dk, s, pm, q); note_launch();
}
template <typename T> void ekin(int nb, int ne, long ldx, const T *x, const double *dk, double *ekib, cudaStream_t st) {
  k_ekin<T><<<nb, CGT, 0, st>>>(ne, ldx, x, dk, ekib); note_launch();
}
template <typename T> void gradres(int nb, int ne, long ldx, const T *x, const T *hx, const double *eig, double *prod,
                                   cudaStream_t st) {
  k_gradres<T><<<nb, CGT, 0, st>>>(ne, ldx, x, hx, eig, prod); note_launch();
}
template <typename T> void scale_rows(int nproj, int ncol, T *P, long ldp, const T *v, const int *colmap,
                                      const int *ncol_dev, cudaStream_t st) {
  const long n = (long)nproj * ncol;
  k_scale_rows<T><<<(int)((n + 255) / 256), 256, 0, st>>>(nproj, ncol, P, ldp, v, colmap, ncol_dev); note_launch();
}

#define QX_INST(T)                                                                                          \
  template void cg_init<T>(int, int, long, const T *, const T *, T *, const CgState &, cudaStream_t);        \
  template void cg_prec<T>(int, int, long, T *, T *, const double *, const CgState &, cudaStream_t);         \
  template void cg_orth<T>(int, int, long, const T *, T *, const CgState &, cudaStream_t);                   \
  template void seq_init<T>(int, int, long, const T *, const T *, T *, const double *, const CgState &,      \
                            const SeqArgs &, cudaStream_t);                                                 \
  template void seq_project<T>(int, long, const T *, const T *, T *, const CgState &, const SeqArgs &,       \
                               double *, double *, cudaStream_t);                                           \
  template void seq_kb<T>(int, int, const T *, const T *, const T *, T *, long, const int *, double *,       \
                          cudaStream_t);                                                                    \
  template void seq_update<T>(int, long, T *, T *, T *, const T *, const T *, const double *,                \
                              const CgState &, const CgParm &, const SeqArgs &, cudaStream_t);              \
  template void cg_update<T>(int, int, long, T *, T *, T *, const T *, const T *, const CgState &,            \
                             const CgParm &, cudaStream_t);                                                  \
  template void ekin<T>(int, int, long, const T *, const double *, double *, cudaStream_t);                  \
  template void gradres<T>(int, int, long, const T *, const T *, const double *, double *, cudaStream_t);    \
  template void scale_rows<T>(int, int, T *, long, const T *, const int *, const int *, cudaStream_t);
QX_INST(float)
QX_INST(double)

}  // namespace qx
