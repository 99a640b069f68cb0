// Device state and launchers of the batched CG band update and small
// per-band reductions.
#pragma once
#include <cuda_runtime.h>

namespace qx {

// Per-band CG state (device arrays of length nb) plus the active list.
struct CgState {
  double *eig, *zansa, *zansab, *z000re, *x000re, *eigb, *betk, *dinnerx, *ekib, *cai;
  int *iter, *izcnt, *lreset, *active;
  int *list;    // active band indices (nb)
  int *pairs;   // band pairs of the FFT pipeline (2 * ceil(nb/2))
  int *nact;    // number of active bands
  int *npair;   // number of pairs
};

// Convergence parameters of eigen_BKL (modules.f90:171-182 defaults).
struct CgParm {
  int itermx, iteremx, noband;
  double tolera, roughfzan, roughfeig, threinn, wdinner;
};

// Sequential (one-rank) CG: bands are updated one after another; *cur is the
// band being updated, pairs = {cur, -1} drives the H|psi> pipeline, and the
// update kernel keeps the band's snapshot column, advances cur and clears the
// while-loop condition of the enclosing graph after the last band.
struct SeqArgs {
  int *cur, *pairs;
  void *snap;
  int nb;
  int ccreal4;
  cudaGraphConditionalHandle handle;
};

template <typename T> void cg_init(int nb, int ne, long ldx, const T *x, const T *hx, T *g, const CgState &s, cudaStream_t st);
template <typename T> void cg_prec(int nb, int ne, long ldx, T *g, T *h, const double *dk, const CgState &s, cudaStream_t st);
template <typename T> void cg_orth(int nb, int ne, long ldx, const T *x, T *h, const CgState &s, cudaStream_t st);
// Entry state of every band (g preconditioned) and band 0 as the current one.
template <typename T> void seq_init(int nb, int ne, long ldx, const T *x, const T *hx, T *g, const double *dk,
                                    const CgState &s, const SeqArgs &q, cudaStream_t st);
// h of band *cur, projected on the snapshot columns below and on x (subgs3,
// subgs4); p, w: nb doubles each of scratch.
template <typename T> void seq_project(int ne, long ldx, const T *x, const T *g, T *h, const CgState &s,
                                       const SeqArgs &q, double *p, double *w, cudaStream_t st);
// gh_cur = beta D <beta|h_cur> (G-space KB; coef: np doubles of scratch).
template <typename T> void seq_kb(int np, int ne, const T *kbg, const T *scale, const T *h, T *gh, long ldx,
                                  const int *cur, double *coef, cudaStream_t st);
template <typename T> void seq_update(int ne, long ldx, T *x, T *hx, T *g, const T *h, const T *gh, const double *dk,
                                      const CgState &s, const CgParm &pm, const SeqArgs &q, cudaStream_t st);
void gradres_stats(const double *prod, const double *occ, int nb, double *out, cudaStream_t st);
void iter_sum(const int *iter, int nb, int *out, cudaStream_t st);
template <typename T> void cg_update(int nb, int ne, long ldx, T *x, T *hx, T *g, const T *h, const T *gh,
                                     const CgState &s, const CgParm &pm, cudaStream_t st);
template <typename T> void ekin(int nb, int ne, long ldx, const T *x, const double *dk, double *ekib, cudaStream_t st);
template <typename T> void gradres(int nb, int ne, long ldx, const T *x, const T *hx, const double *eig, double *prod,
                                   cudaStream_t st);
template <typename T> void scale_rows(int nproj, int ncol, T *P, long ldp, const T *v, const int *colmap,
                                      const int *ncol_dev, cudaStream_t st);

}  // namespace qx
