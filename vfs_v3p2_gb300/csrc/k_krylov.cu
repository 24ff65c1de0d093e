// Flexible GMRES(m) in FP64 with all scalars on the device.
//
// The Krylov basis V (m+1 vectors) is FP64; the preconditioned directions Z
// are in the multigrid precision T.  Basis vector q is vs[q] * V_q: with one
// classical Gram-Schmidt pass (the default) the update sweep stores the
// orthogonalised column unnormalised, together with the multigrid input of
// the next iteration and its norm partials, and the scale 1 / ||.|| follows
// from the reduction; the matrix-vector product and the solution update
// apply vs.  With CGS2 (classical with one re-orthogonalisation pass) the
// columns are stored normalised (vs = 1).  Every pass is a deterministic
// multi-dot or norm (fixed block partials summed in index order by the block
// that arrives last) or one fused update sweep.  The Hessenberg column, Givens rotations and the
// residual estimate live in a KrylovState in device memory and are updated by
// the last block of the sweep before them, so the host enqueues iterations without reading
// anything back; every kernel returns immediately once st->done is set.
#include "vfs_common.cuh"
#include "vfs_proj.h"

namespace vfs {

constexpr int KB = 256;
constexpr int MAXCOL = 64;  // largest restart length

// Blocks of the norms and update sweeps: two cells per thread (one turn of the
// update's loop) until the grid fills four blocks per SM (four cells a thread:
// 32^3 9.2 -> 11.5 us an update).
int krylov_nblocks(size_t n) {
  size_t b = (n + KB * 2 - 1) / (KB * 2);
  if (b > 152 * 4) b = 152 * 4;
  return (int)(b ? b : 1);
}

__device__ __forceinline__ bool is_done(const KrylovState* st) { return *(volatile const int*)&st->done; }
// done and epoch to pinned host memory (the host reads them after the event
// that follows the iteration).
__device__ __forceinline__ void post_status(const KrylovState* st, int* hst) {
  if (!hst) return;
  volatile int* h = hst;
  h[0] = st->done;
  h[1] = st->epoch;
  __threadfence_system();
}
__device__ __forceinline__ bool met(const KrylovState* st, double r) {
  return r <= st->rtol * st->bnorm && (st->atol <= 0. || r <= st->atol);
}

// The norm of a new round's vectors from their partials, by one block: MODE 0
// (beta alone: a restart's residual), 1 (bnorm alone: a warm start, whose
// residual follows), 2 (both: a cold start, where r0 = aj b).  Clears the
// Hessenberg matrix and g with the whole block.
template <int MODE>
__device__ __forceinline__ void norm_close(KrylovState* st, const double* parts, int nparts) {
  __shared__ double sh[32];
  double s = 0.;
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) s += __ldcg(parts + p);
  s = block_sum(s, sh);
  if (MODE != 1) {
    const int m = st->m;
    for (int q = threadIdx.x; q <= m; q += blockDim.x) st->g[q] = 0.;
    for (int q = threadIdx.x; q < (m + 1) * m; q += blockDim.x) st->H[q] = 0.;
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  const double nrm = sqrt(s);
  if (MODE != 0) {
    st->bnorm = nrm;
    st->done = (nrm == 0.) ? 1 : 0;
    st->it = 0;
    st->j = 0;
    if (nrm == 0. || MODE == 1) return;
  }
  st->beta = nrm;
  st->resid = nrm;
  st->g[0] = nrm;
  st->j = 0;
  st->inv_hn = nrm > 0. ? 1. / nrm : 0.;
  st->vs[0] = 1.;  // V_0 is stored normalised
  if (met(st, nrm)) st->done = 1;
}

// beta = ||r|| of a restart (or warm start): partials and, by the last block, the close.
__global__ void __launch_bounds__(KB) k_beta(KrylovState* st, const double* __restrict__ v, size_t n, double* parts) {
  if (is_done(st)) return;
  __shared__ double sh[32];
  double s = 0.;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const double a = v[t];
    s = fma(a, a, s);
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) parts[blockIdx.x] = s;
  if (last_block(st->ticket)) norm_close<0>(st, parts, gridDim.x);
}
int launch_beta(KrylovState* st, const double* r, size_t n, double* parts, cudaStream_t s) {
  k_beta<<<krylov_nblocks(n), KB, 0, s>>>(st, r, n, parts); ++g_launches;
  return (int)cudaGetLastError();
}

// Opening of a round: the aj-scaled right-hand side bs = aj b on the interior
// (bs's ghosts are zero), its norm, and on a cold start the residual r0 = bs
// as V_0 (scaled by launch_open_v) and its norm: one pass and one launch.
template <bool COLD>
__global__ void __launch_bounds__(KB) k_open_b(KrylovState* st, Dims d, const double* __restrict__ aj,
                                               const double* __restrict__ b, double* __restrict__ bs,
                                               double* __restrict__ V, double* parts) {
  __shared__ double sh[32];
  const int lane = threadIdx.x & 31, nw = gridDim.x * (KB / 32);
  double s = 0.;
  for (int r = blockIdx.x * (KB / 32) + (threadIdx.x >> 5); r < d.my * d.mz; r += nw) {
    const int k = r / d.my, j = r - k * d.my;
    const bool in = j > 0 && k > 0 && j < d.my - 1 && k < d.mz - 1;
    const size_t o = (size_t)r * d.mx;
    for (int i = lane; i < d.mx; i += 32) {
      double v = 0.;
      if (in && i > 0 && i < d.mx - 1) {
        v = aj[o + i] * b[o + i];
        bs[o + i] = v;
        s = fma(v, v, s);
      }
      if (COLD) V[o + i] = v;
    }
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) parts[blockIdx.x] = s;
  if (last_block(st->ticket)) norm_close<COLD ? 2 : 1>(st, parts, gridDim.x);
}
int launch_open_b(KrylovState* st, const Dims& d, const double* aj, const double* b, double* bs, double* V, bool cold,
                  double* parts, cudaStream_t s) {
  const int nb = krylov_nblocks(ncell(d));
  if (cold) k_open_b<true><<<nb, KB, 0, s>>>(st, d, aj, b, bs, V, parts);
  else k_open_b<false><<<nb, KB, 0, s>>>(st, d, aj, b, bs, V, parts);
  ++g_launches;
  return (int)cudaGetLastError();
}

// v0 = r / beta in place and the first preconditioner input T(v0) (times 1 / D
// of the FP16 normalised operator when dinv is set); r's ghosts are zero.
template <typename T>
__global__ void __launch_bounds__(KB) k_open_v(const KrylovState* st, double* v, T* __restrict__ out, size_t n,
                                               const float* __restrict__ dinv) {
  if (is_done(st)) return;
  const double f = st->inv_hn;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const double a = v[t] * f;
    v[t] = a;
    out[t] = dinv ? from_double<T>(a) * (T)dinv[t] : from_double<T>(a);
  }
}
template <typename T>
int launch_open_v(const KrylovState* st, double* v, T* out, size_t n, const float* dinv, cudaStream_t s) {
  k_open_v<T><<<krylov_nblocks(n) * 4, KB, 0, s>>>(st, v, out, n, dinv); ++g_launches;
  return (int)cudaGetLastError();
}
template int launch_open_v<float>(const KrylovState*, double*, float*, size_t, const float*, cudaStream_t);
template int launch_open_v<double>(const KrylovState*, double*, double*, size_t, const float*, cudaStream_t);

// Multi-dot partials: parts[q * nblocks + b] = sum over block b's cells of
// V_q . w for q < nv, up to DCH columns per sweep (w is re-read from L2).
// The column count nv = st->j + 1 is the device's, so that a launch can be
// replayed from a graph.
constexpr int DCH = 8;

// Sums of DCH values over a warp by halving exchanges: 4 + 2 + 1 adds leave
// one value per lane, two more finish it, 9 FP64 adds instead of 8 x 5 (the
// adds go through the FP64 pipe at 16 cycles a warp, which is what the plain
// tree cost: 640 cycles a column and block).  Lane l ends with the sum of
// value warp_sum8_index(l).
__device__ __forceinline__ double warp_sum8(const double* a, int lane) {
  constexpr unsigned FULL = 0xffffffffu;
  double t[4];
  const bool h4 = lane & 16, h2 = lane & 8, h1 = lane & 4;
#pragma unroll
  for (int q = 0; q < 4; q++) t[q] = (h4 ? a[q + 4] : a[q]) + __shfl_xor_sync(FULL, h4 ? a[q] : a[q + 4], 16);
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const double keep = h2 ? t[q + 2] : t[q], send = h2 ? t[q] : t[q + 2];
    t[q] = keep + __shfl_xor_sync(FULL, send, 8);
  }
  const double keep = h1 ? t[1] : t[0], send = h1 ? t[0] : t[1];
  double r = keep + __shfl_xor_sync(FULL, send, 4);
  r += __shfl_xor_sync(FULL, r, 2);
  r += __shfl_xor_sync(FULL, r, 1);
  return r;
}
__device__ __forceinline__ int warp_sum8_index(int lane) { return (lane & 16 ? 4 : 0) | (lane & 8 ? 2 : 0) | (lane & 4 ? 1 : 0); }

// Sum the multi-dot partials into st->h (and accumulate the column in hacc):
// one warp per dot (q = warp, warp + 8, ...), each lane summing a fixed
// stride of the block partials in four chains, then the warp tree.
__device__ __forceinline__ void dots_finish(KrylovState* st, const double* parts, int nparts, int nv, int pass) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const double m = column_scale(st).m;
  for (int q = threadIdx.x >> 5; q < nv; q += nw) {
    const double* pq = parts + (size_t)q * nparts;
    double s[4] = {0., 0., 0., 0.};
    for (int p = lane; p < nparts; p += 128) {
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (p + 32 * u < nparts) s[u] += __ldcg(pq + p + 32 * u);
    }
    const double t = warp_sum((s[0] + s[1]) + (s[2] + s[3])) * st->vs[q] * m;
    if (lane == 0) {
      st->h[q] = t;
      st->hacc[q] = (pass == 1) ? t : st->hacc[q] + t;
    }
  }
}

// NQ consecutive basis columns V0 .. V0 + (NQ-1) n against w, each thread's
// cells accumulated in increasing order, the next cell's loads issued before
// a cell's products: the SM's warps run in step, so without that the loads
// and the FP64 pipe take turns (256x128x128, 5 columns: 66 -> 59 us; 128x64x96,
// 7: 37 -> 27; the update, whose chains need two cells a turn, measured slower
// so, 72 -> 78).  OWN: w's cells were written by this thread
// (read past the non-coherent path).
template <int NQ, bool OWN>
__device__ __forceinline__ void dot_chunk(const double* __restrict__ V0, const double* w, size_t n, double* a) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  double v[2][NQ], wv[2];
  auto load = [&](int b, size_t c) {
    wv[b] = OWN ? __ldcg(w + c) : __ldg(w + c);
#pragma unroll
    for (int q = 0; q < NQ; q++) v[b][q] = __ldg(V0 + (size_t)q * n + c);
  };
  auto add = [&](int b) {
#pragma unroll
    for (int q = 0; q < NQ; q++) a[q] = fma(v[b][q], wv[b], a[q]);
  };
  if (t >= n) return;
  load(0, t);
  for (;;) {
    t += stride;
    if (t >= n) { add(0); return; }
    load(1, t);
    add(0);
    t += stride;
    if (t >= n) { add(1); return; }
    load(0, t);
    add(1);
  }
}

// The dots of the nv columns and, by the last block, their finish.
template <bool OWN>
__device__ __forceinline__ void dots(KrylovState* st, const double* __restrict__ V, int nv, const double* w, size_t n,
                                     double* parts, int pass) {
  __shared__ double red[KB / 32][MAXCOL + DCH];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  for (int q0 = 0; q0 < nv; q0 += DCH) {
    double a[DCH] = {0., 0., 0., 0., 0., 0., 0., 0.};
    const double* V0 = V + (size_t)q0 * n;
    switch (min(DCH, nv - q0)) {
      case 8: dot_chunk<8, OWN>(V0, w, n, a); break;
      case 7: dot_chunk<7, OWN>(V0, w, n, a); break;
      case 6: dot_chunk<6, OWN>(V0, w, n, a); break;
      case 5: dot_chunk<5, OWN>(V0, w, n, a); break;
      case 4: dot_chunk<4, OWN>(V0, w, n, a); break;
      case 3: dot_chunk<3, OWN>(V0, w, n, a); break;
      case 2: dot_chunk<2, OWN>(V0, w, n, a); break;
      default: dot_chunk<1, OWN>(V0, w, n, a); break;
    }
    const double r = warp_sum8(a, lane);
    if ((lane & 3) == 0) red[wp][q0 + warp_sum8_index(lane)] = r;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nv; q += blockDim.x) {
    double r = 0.;
    for (int u = 0; u < KB / 32; u++) r += red[u][q];
    parts[(size_t)q * gridDim.x + blockIdx.x] = r;
  }
  if (last_block(st->ticket)) dots_finish(st, parts, gridDim.x, nv, pass);
}
__global__ void __launch_bounds__(KB) k_multidot(KrylovState* st, const double* __restrict__ V,
                                                 const double* __restrict__ w, size_t n, double* parts) {
  if (is_done(st)) return;
  dots<false>(st, V, st->j + 1, w, n, parts, 1);
}

// Blocks of the dots: a warp's reduction of eight columns takes nine FP64 adds
// whatever its cells, so two blocks per SM until a thread has eight cells
// (104x40x72, 21 columns: 30.4 us a launch at two cells a thread, 23.6 so).
static int dots_nblocks(size_t n) {
  const size_t two = (n + KB * 2 - 1) / (KB * 2), eight = (n + KB * 8 - 1) / (KB * 8);
  const size_t full = eight / 152 * 152;  // no partial wave
  const size_t b = full > 152 * 2 ? full : (two < 152 * 2 ? two : 152 * 2);
  return (int)(b > 152 * 4 ? 152 * 4 : (b ? b : 1));
}
int launch_multidot(KrylovState* st, const double* V, const double* w, size_t n, double* parts, cudaStream_t s) {
  k_multidot<<<dots_nblocks(n), KB, 0, s>>>(st, V, w, n, parts); ++g_launches;
  return (int)cudaGetLastError();
}

// Close Arnoldi column j from the nparts partials of ||w||^2 (one block):
// ||w||, Hessenberg column, Givens rotations, residual estimate |g[j+1]|,
// convergence test, 1 / h[j+1][j] for the next basis vector, and the status
// to the host.  The column, the previous rotations and g[j] are staged in
// shared memory by the whole block first, so that the serial rotation loop
// of thread 0 reads no global memory.
__device__ __forceinline__ void arnoldi_close(KrylovState* st, const double* parts, int nparts, int* hst) {
  __shared__ double sh[32];
  __shared__ double hc[MAXCOL + 2], cq[MAXCOL + 1], sq[MAXCOL + 1];
  double s = 0.;
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) s += __ldcg(parts + p);
  const int m = st->m, j = st->j;
  for (int q = threadIdx.x; q <= j; q += blockDim.x) hc[q] = st->hacc[q];
  for (int q = threadIdx.x; q < j; q += blockDim.x) {
    cq[q] = st->cs[q];
    sq[q] = st->sn[q];
  }
  s = block_sum(s, sh);  // (its barriers also order the staging)
  if (threadIdx.x != 0) return;
  const double nw = sqrt(s), hn = nw * column_scale(st).m;  // of the stored column, and its value's
  double* Hc = st->H + (size_t)j * (m + 1);
  hc[j + 1] = hn;
  for (int q = 0; q < j; q++) {
    const double a = hc[q], b = hc[q + 1];
    hc[q] = cq[q] * a + sq[q] * b;
    hc[q + 1] = -sq[q] * a + cq[q] * b;
  }
  for (int q = 0; q < j; q++) Hc[q] = hc[q];
  const double a = hc[j], b = hc[j + 1];
  const double den = sqrt(a * a + b * b);
  const double c = den > 0. ? a / den : 1., sn = den > 0. ? b / den : 0.;
  st->cs[j] = c;
  st->sn[j] = sn;
  Hc[j] = den;
  Hc[j + 1] = 0.;
  st->g[j + 1] = -sn * st->g[j];
  st->g[j] = c * st->g[j];
  st->resid = fabs(st->g[j + 1]);
  st->hn = hn;
  st->inv_hn = nw > 0. ? 1. / nw : 0.;
  st->vs[j + 1] = st->orth2 ? 1. : st->inv_hn;  // CGS2 normalises the column in k_vnext_in
  st->j = j + 1;
  st->it += 1;
  if (met(st, st->resid) || hn == 0. || !(st->resid == st->resid)) st->done = 1;
  post_status(st, hst);
}
// The close as its own launch, for a probed iteration (which times it alone).
__global__ void __launch_bounds__(KB) k_arnoldi_finish(KrylovState* st, const double* __restrict__ parts, int nparts,
                                                       int* hst) {
  if (is_done(st)) {
    if (threadIdx.x == 0) post_status(st, hst);
    return;
  }
  arnoldi_close(st, parts, nparts, hst);
}
int launch_arnoldi_finish(KrylovState* st, int nparts, const double* parts, int* hst, cudaStream_t s) {
  k_arnoldi_finish<<<1, KB, 0, s>>>(st, parts, nparts, hst); ++g_launches;
  return (int)cudaGetLastError();
}

// h of the last dots as factors of the stored columns (in shared memory).
__device__ __forceinline__ void column_factors(const KrylovState* st, int nv, double* hs) {
  const double m = column_scale(st).m;
  for (int q = threadIdx.x; q < nv; q += blockDim.x) hs[q] = st->h[q] * st->vs[q] / m;
  __syncthreads();
}
// w -= sum_q hs[q] V_q, two cells per turn as in dot_chunk (the same cells a
// thread); returns the thread's sum of w^2 after the update.
__device__ __forceinline__ double subtract_columns(const double* __restrict__ V, int nv, double* w, size_t n,
                                                   const double* hs) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  double s = 0.;
  for (; t + stride < n; t += 2 * stride) {
    double a0 = w[t], a1 = w[t + stride];
#pragma unroll 4
    for (int q = 0; q < nv; q++) {
      const double h = hs[q];
      const double v0 = V[(size_t)q * n + t], v1 = V[(size_t)q * n + t + stride];
      a0 = fma(-h, v0, a0);
      a1 = fma(-h, v1, a1);
    }
    w[t] = a0;
    w[t + stride] = a1;
    s = fma(a0, a0, s);
    s = fma(a1, a1, s);
  }
  if (t < n) {
    double a = w[t];
#pragma unroll 4
    for (int q = 0; q < nv; q++) a = fma(-hs[q], V[(size_t)q * n + t], a);
    w[t] = a;
    s = fma(a, a, s);
  }
  return s;
}

// w -= sum_q h[q] V_q, with the partials of ||w||^2 after the update; close:
// the last block closes the Arnoldi column.
__global__ void __launch_bounds__(KB) k_gs_update(KrylovState* st, const double* __restrict__ V,
                                                  double* __restrict__ w, size_t n, double* parts, int close, int* hst) {
  if (is_done(st)) {
    if (close && blockIdx.x == 0 && threadIdx.x == 0) post_status(st, hst);
    return;
  }
  const int nv = st->j + 1;
  __shared__ double sh[32];
  __shared__ double hs[72];
  column_factors(st, nv, hs);
  const double s = block_sum(subtract_columns(V, nv, w, n, hs), sh);
  if (threadIdx.x == 0) parts[blockIdx.x] = s;
  if (close && last_block(st->ticket)) arnoldi_close(st, parts, gridDim.x, hst);
}
int launch_gs_update(KrylovState* st, const double* V, double* w, size_t n, double* parts, int close, int* hst,
                     cudaStream_t s) {
  k_gs_update<<<krylov_nblocks(n), KB, 0, s>>>(st, V, w, n, parts, close, hst); ++g_launches;
  return (int)cudaGetLastError();
}

// One-pass classical Gram-Schmidt update of column j = st->j: the
// orthogonalised vector u = w - sum_q h_q vs_q V_q is stored unnormalised as
// V_{j+1}, its multigrid-precision copy as the next preconditioner input, and
// the partials of ||u||^2 go to parts; the close of the column sets vs_{j+1}
// (close: by the last block, else k_arnoldi_finish).
// dinv (nullable): 1 / D of the FP16 normalised multigrid operator, applied
// to the multigrid copy after its rounding to T.
// Two columns of two cells a step: the loads of one step overlap the FP64
// products of another warp's, which longer steps queue behind each other
// (256x128x128 by 8 columns 92 us, 4 73, 2 60, 1 65; 512x256x256 404 -> 324;
// with the registers left free: capped for five blocks per SM 61 and 351).
template <typename T>
__global__ void __launch_bounds__(KB, 1) k_cgs_update(KrylovState* st, double* V, const double* __restrict__ w,
                                                   T* __restrict__ out, size_t n, double* parts,
                                                   const float* __restrict__ dinv, int close, int* hst) {
  if (is_done(st)) {
    if (close && blockIdx.x == 0 && threadIdx.x == 0) post_status(st, hst);
    return;
  }
  const int nv = st->j + 1;
  __shared__ double sh[32];
  __shared__ double hs[72];
  const double m = column_scale(st).m;
  for (int q = threadIdx.x; q < nv; q += blockDim.x) hs[q] = st->h[q] * st->vs[q] / m;
  __syncthreads();
  double* vn = V + (size_t)nv * n;
  double s = 0.;
  // two cells per turn (their basis loads in flight together), in cell order
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (; t + stride < n; t += 2 * stride) {
    double a0 = w[t], a1 = w[t + stride];
#pragma unroll 2
    for (int q = 0; q < nv; q++) {
      const double h = hs[q];
      const double v0 = V[(size_t)q * n + t], v1 = V[(size_t)q * n + t + stride];
      a0 = fma(-h, v0, a0);
      a1 = fma(-h, v1, a1);
    }
    vn[t] = a0;
    vn[t + stride] = a1;
    out[t] = dinv ? from_double<T>(a0) * (T)dinv[t] : from_double<T>(a0);
    out[t + stride] = dinv ? from_double<T>(a1) * (T)dinv[t + stride] : from_double<T>(a1);
    s = fma(a0, a0, s);
    s = fma(a1, a1, s);
  }
  if (t < n) {
    double a = w[t];
#pragma unroll 4
    for (int q = 0; q < nv; q++) a = fma(-hs[q], V[(size_t)q * n + t], a);
    vn[t] = a;
    out[t] = dinv ? from_double<T>(a) * (T)dinv[t] : from_double<T>(a);
    s = fma(a, a, s);
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) parts[blockIdx.x] = s;
  if (close && last_block(st->ticket)) arnoldi_close(st, parts, gridDim.x, hst);
}
template <typename T>
int launch_cgs_update(KrylovState* st, double* V, const double* w, T* out, size_t n, double* parts, int close, int* hst,
                      cudaStream_t s, const float* dinv) {
  k_cgs_update<T><<<krylov_nblocks(n), KB, 0, s>>>(st, V, w, out, n, parts, dinv, close, hst); ++g_launches;
  return (int)cudaGetLastError();
}
template int launch_cgs_update<float>(KrylovState*, double*, const double*, float*, size_t, double*, int, int*,
                                      cudaStream_t, const float*);
template int launch_cgs_update<double>(KrylovState*, double*, const double*, double*, size_t, double*, int, int*,
                                       cudaStream_t, const float*);

// CGS2 middle pass: w <- w - V h (h from the first pass) and the second
// pass's dots V_q . w.  A thread's dots take the cells that it has updated,
// in chunks of columns as k_multidot's, the columns from L2 again: one launch
// for any number of columns (five that held all columns in registers and
// summed each by a tree of its own took 83 us at 128x64x96, 13 columns).
__global__ void __launch_bounds__(KB) k_gs_update_dots(KrylovState* st, const double* __restrict__ V, double* w, size_t n,
                                                       double* parts) {
  if (is_done(st)) return;
  const int nv = st->j + 1;
  __shared__ double hs[72];
  column_factors(st, nv, hs);
  subtract_columns(V, nv, w, n, hs);
  dots<true>(st, V, nv, w, n, parts, 2);
}
int launch_gs_update_dots(KrylovState* st, const double* V, double* w, size_t n, double* parts, cudaStream_t s) {
  k_gs_update_dots<<<dots_nblocks(n), KB, 0, s>>>(st, V, w, n, parts); ++g_launches;
  return (int)cudaGetLastError();
}

// y = R^{-1} g over the st->j closed columns (runs whether or not done).
__global__ void k_lsq(KrylovState* st) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int m = st->m, J = st->j;
  for (int q = J - 1; q >= 0; q--) {
    double s = st->g[q];
    for (int p = q + 1; p < J; p++) s -= st->H[(size_t)p * (m + 1) + q] * st->y[p];
    st->y[q] = s / st->H[(size_t)q * (m + 1) + q];
  }
}
int launch_lsq_update(KrylovState* st, cudaStream_t s) {
  k_lsq<<<1, 32, 0, s>>>(st); ++g_launches;
  return (int)cudaGetLastError();
}

// x += sum_q y_q Z_q over the closed columns; the last block marks them as
// applied (a later update adds nothing).
template <typename T>
__global__ void __launch_bounds__(KB) k_x_update(KrylovState* st, const T* __restrict__ Z, size_t n, double* x) {
  __shared__ double ys[72];
  const int J = st->j;
  for (int q = threadIdx.x; q < J; q += blockDim.x) ys[q] = st->y[q] * st->vs[q];
  __syncthreads();
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const double x0 = x[t];
    double a = x0;
    bool special = false;
#pragma unroll 4
    for (int q = 0; q < J; q++) {
      const T z = Z[(size_t)q * n + t];
      if constexpr (sizeof(T) == 4) a = fma(ys[q], widen_normal(z, special), a);
      else a = fma(ys[q], z, a);
    }
    if (special) {
      a = x0;
      for (int q = 0; q < J; q++) a = fma(ys[q], to_acc<double>(Z[(size_t)q * n + t]), a);
    }
    x[t] = a;
  }
  if (last_block(st->ticket) && threadIdx.x == 0) st->j = 0;
}
template <typename T>
int launch_x_update(KrylovState* st, const T* Z, size_t n, double* x, cudaStream_t s) {
  k_x_update<T><<<krylov_nblocks(n) * 4, KB, 0, s>>>(st, Z, n, x); ++g_launches;
  return (int)cudaGetLastError();
}
template int launch_x_update<float>(KrylovState*, const float*, size_t, double*, cudaStream_t);
template int launch_x_update<double>(KrylovState*, const double*, size_t, double*, cudaStream_t);

// Next basis vector and multigrid input in one sweep: V_{j+1} = w / h_{j+1,j}
// and out = T(V_{j+1}) over the interior; ghost entries of w are zero.
// V_{j+1} is V + st->j * n (the column just opened).
template <typename T>
__global__ void __launch_bounds__(KB) k_vnext_in(const KrylovState* st, const double* __restrict__ w, double* V,
                                                  T* __restrict__ out, size_t n, const float* __restrict__ dinv) {
  if (is_done(st)) return;
  const double f = st->inv_hn;
  double* vn = V + (size_t)st->j * n;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const double v = w[t] * f;
    vn[t] = v;
    out[t] = dinv ? from_double<T>(v) * (T)dinv[t] : from_double<T>(v);
  }
}
template <typename T>
int launch_vnext_in(KrylovState* st, const double* w, double* V, T* out, size_t n, const float* dinv, cudaStream_t s) {
  k_vnext_in<T><<<krylov_nblocks(n) * 4, KB, 0, s>>>(st, w, V, out, n, dinv); ++g_launches;
  return (int)cudaGetLastError();
}
template int launch_vnext_in<float>(KrylovState*, const double*, double*, float*, size_t, const float*, cudaStream_t);
template int launch_vnext_in<double>(KrylovState*, const double*, double*, double*, size_t, const float*, cudaStream_t);

}  // namespace vfs
