// Launchers of the per-step FP64 kernels (k_proj.cu) and the Krylov kernels
// (k_krylov.cu).
#pragma once

#include <cuda_runtime.h>

#include "vfs_common.cuh"

namespace vfs {

// Contravariant flux Ucont as three component arrays (SoA) on the device.
struct Ucont {
  double *x, *y, *z;
};

// ticket (of the reductions below): an unsigned that is 0 between launches; the
// launches that share one are ordered.
int launch_aos2soa(size_t n, const double* aos, double* x, double* y, double* z, cudaStream_t s);
int launch_soa2aos(size_t n, const double* x, const double* y, const double* z, double* aos, cudaStream_t s);
// comp / ncomp: labels 0..ncomp-1 of the connected fluid regions (nullptr
// when the fluid is one region): the compatibility fix and the mean removal
// then act per region.  sc holds 4 doubles for launch_rhs.
int launch_rhs(const Dims& d, const Ucont& u, const double* nvert, double dt, double st, double coeff, int meanfix,
               double* b, double* parts, double* sc, unsigned* ticket, cudaStream_t s, const uint8_t* nb8 = nullptr,
               const int* comp = nullptr, int ncomp = 1);
int launch_volume_flux(const Dims& d, int mode, const Ucont& u, const double* nvert, const double* M, double* parts,
                       double* fa4, unsigned* ticket, cudaStream_t s, const uint8_t* nb8 = nullptr);
// subtracts each region's fluid mean from x
int launch_remove_mean(const Dims& d, const double* nvert, double* x, double* parts, double* sc, unsigned* ticket,
                       cudaStream_t s, const int* comp, int ncomp);
// sum and count of x over the fluid (sc[0..1])
int launch_fluid_sum(const Dims& d, const double* nvert, const double* x, double* parts, double* sc, unsigned* ticket,
                     cudaStream_t s);
// phi of a solve: the mean of sc subtracted on the fluid (sc nullable), zero on
// boundary and solid cells, periodic ghosts
int launch_phi_finish(const Dims& d, const double* nvert, double* phi, const double* sc, cudaStream_t s);
int launch_update_pressure(const Dims& d, const double* nvert, const double* phi, double* p, cudaStream_t s);
int launch_proj_dots(const Dims& d, const double* M, double* pd, cudaStream_t s);
// nb8: nvert as bytes when every value is an integer in [0, 127] (exact
// integer pair tests), else nullptr (FP64 tests).  Projects the faces of
// planes [k0, k1) (k1 < 0: mz) and syncs their periodic ghosts.  A plane
// reads phi and the metrics alone, and the ghost sync of an interior plane
// reads that plane alone, so interior slabs may go in any order; the k ghost
// planes 0 and mz-1 (filled from planes mz-2 and 1) come after all of them.
int launch_projection(const Dims& d, const double* pd, const double* M, const double* nvert, const uint8_t* nb8,
                      const double* phi, double dt, double st, double coeff, const Ucont& u, cudaStream_t s,
                      int k0 = 0, int k1 = -1);
// The same projection on face weights and cross-term codes precomputed by
// launch_proj_weights (pw [9][N], pc [N]): FMAs, no nvert tests; equal to
// the reference's operation order to rounding (<= 1e-14 relative).
int launch_proj_weights(const Dims& d, const double* pd, const double* M, const double* nvert, double* pw, uint16_t* pc, unsigned* used,
                        cudaStream_t s);
int launch_projection_fast(const Dims& d, unsigned used, const double* pw, const uint16_t* pc, const double* phi, double dt, double st,
                           double coeff, const Ucont& u, cudaStream_t s, int k0 = 0, int k1 = -1);
// periodic ghost sync of the Ucont components on planes [k0, k1)
int launch_ucont_ghosts(const Dims& d, const Ucont& u, int k0, int k1, cudaStream_t s);
// minv: per-cell inverse of the metric matrix [csi; eta; zet] (9 doubles,
// row-major), from launch_inverse_metric.
int launch_contra2cart(const Dims& d, const double* minv, const double* nvert, const Ucont& u, double* ucat, cudaStream_t s);
int launch_inverse_metric(const Dims& d, const double* M, const double* nvert, double* minv, cudaStream_t s);
// Divergence check that needs no scratch (no allocation, nothing shared between
// calls); returns 0, 1 (argument) or 2 (CUDA) and sets *why on error.
int divergence_max_noalloc(int device, const Dims& d, const Ucont& u, const double* aj, const double* nvert, double* out,
                          cudaStream_t s, const char** why);
// out[0] = ||r||_2 over the array, out[1] = max |r| over the cells the
// divergence check keeps
int launch_norm_absmax(const Dims& d, const double* r, const double* nvert, double* parts, double* out, unsigned* ticket,
                       cudaStream_t s, const uint8_t* nb8 = nullptr);
int launch_divergence(const Dims& d, const Ucont& u, const double* aj, const double* nvert, double* parts, double* out,
                      unsigned* ticket, cudaStream_t s, const uint8_t* nb8 = nullptr);

// ---- FGMRES device state (k_krylov.cu) ----
// One flexible GMRES(m) solve keeps all of its scalars on the device so an
// iteration is a fixed sequence of launches with no host round trip; every
// kernel returns at once when the solve has converged.
struct KrylovState {
  int m;          // restart length
  int j;          // current Arnoldi column
  int done;       // 1 once converged (or broken down)
  int epoch;      // solve round, copied to the host beside done (a stale copy is recognisable)
  int it;         // preconditioner applications so far
  int reorth;     // 1 if the second Gram-Schmidt pass is needed this column
  double rtol, atol, bnorm, beta, resid;  // converged: resid <= rtol*bnorm and (atol <= 0 or resid <= atol)
  double hn, inv_hn;
  double* H;      // (m+1) x m, column-major: H[j*(m+1) + i]
  double* cs;     // m
  double* sn;     // m
  double* g;      // m+1
  double* y;      // m
  double* h;      // m+1 dots of the current pass
  double* hacc;   // m+1 accumulated dots of the column
  double* vs;     // m+1 column scales: basis vector q is vs[q] * V_q
  int orth2;      // 1: CGS2 (columns stored normalised, vs = 1)
  int f32;        // 1: FP32 directions (see column_scale)
  unsigned ticket[1];  // blocks of the running reduction that have arrived (0 between launches)
};

// The scale vs[j] of the column that opens an iteration, split as p2 m: with
// FP32 directions the product A z takes the power of two p2 into z (exact, on
// the FP32 pipe) and leaves the rest m, in [1, 2), to the few scalars that
// follow, so that it needs no FP64 multiply a cell (one of its twelve
// operations on 11 slots).  The vectors of the iteration are then 1 / m times
// their values: w = A z p2, dots times m, and the column stored from it.
struct ColumnScale {
  float p2;
  double m;
};
__device__ __forceinline__ ColumnScale column_scale(const KrylovState* st) {
  const double vs = st->vs[st->j];
  if (!st->f32) return {1.f, 1.};
  int e = (int)((__double_as_longlong(vs) >> 52) & 0x7ff) - 1023;
  e = e < -120 ? -120 : (e > 120 ? 120 : e);  // a float either way; m then takes the rest
  return {__int_as_float((e + 127) << 23), vs * __longlong_as_double((long long)(1023 - e) << 52)};
}

// parts must hold nblocks * (m + 2) doubles.
int krylov_nblocks(size_t n);
// a round's opening: bs = aj b, bnorm, and on a cold start V_0 = bs with beta
int launch_open_b(KrylovState* st, const Dims& d, const double* aj, const double* b, double* bs, double* V, bool cold,
                  double* parts, cudaStream_t s);
// beta of a warm start's or restart's residual r
int launch_beta(KrylovState* st, const double* r, size_t n, double* parts, cudaStream_t s);
// v = r / beta in place and out = T(v)
template <typename T>
int launch_open_v(const KrylovState* st, double* v, T* out, size_t n, const float* dinv, cudaStream_t s);
// The Krylov kernels take the column count from the device state, so one
// iteration is a fixed launch sequence.
// first pass: the dots of the columns with w
int launch_multidot(KrylovState* st, const double* V, const double* w, size_t n, double* parts, cudaStream_t s);
// close: the launch's last block closes the Arnoldi column (what
// launch_arnoldi_finish does as its own launch) and writes done and epoch to
// the pinned host ints hst.
int launch_gs_update(KrylovState* st, const double* V, double* w, size_t n, double* parts, int close, int* hst,
                     cudaStream_t s);
// second CGS pass fused with the first update
int launch_gs_update_dots(KrylovState* st, const double* V, double* w, size_t n, double* parts, cudaStream_t s);
template <typename T>
int launch_cgs_update(KrylovState* st, double* V, const double* w, T* out, size_t n, double* parts, int close, int* hst,
                      cudaStream_t s, const float* dinv = nullptr);
template <typename T>
int launch_vnext_in(KrylovState* st, const double* w, double* V, T* out, size_t n, const float* dinv, cudaStream_t s);
// w = A z (aj-scaled FP64 operator, z in T) and Z[st->j] = z on the interior
template <typename T>
int launch_apply64_krylov(const OpView<double>& A, const T* z, T* Z, const KrylovState* st, double* w, cudaStream_t s);
int launch_arnoldi_finish(KrylovState* st, int nparts, const double* parts, int* hst, cudaStream_t s);
int launch_lsq_update(KrylovState* st, cudaStream_t s);
template <typename T>
int launch_x_update(KrylovState* st, const T* Z, size_t n, double* x, cudaStream_t s);

}  // namespace vfs
