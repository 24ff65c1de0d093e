// Per-step FP64 kernels around the solve: the divergence right-hand side and
// its compatibility fix, the immersed-boundary flux balance, null-space
// removal, the phi / pressure ghost fills, the contravariant velocity
// correction (Projection), Contra2Cart and the divergence check.
//
// Compiled with --fmad=false like k_setup.cu: each kernel performs the
// reference's multiplies and adds in the reference's order, so for equal
// inputs the outputs are bit-identical (reductions excepted, which sum in a
// fixed tree order instead of the reference's loop order).

#include "vfs_common.cuh"
#include "vfs_kernels.h"
#include "vfs_proj.h"

namespace vfs {

constexpr int RB = 256;  // reduction block size

#define GRID_LOOP(d)                                                                          \
  for (size_t _t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; _t < ncell(d);              \
       _t += (size_t)gridDim.x * blockDim.x)
// cells [c0, c1) of the grid, grid-stride
#define RANGE_LOOP(c0, c1)                                                                     \
  for (size_t _t = (c0) + blockIdx.x * (size_t)blockDim.x + threadIdx.x; _t < (c1);           \
       _t += (size_t)gridDim.x * blockDim.x)
// 32-bit index split (grids stay below 2^31 cells)
#define DECOMP(d, i, j, k)                          \
  const unsigned _u = (unsigned)_t;                 \
  const unsigned _q = _u / (unsigned)(d).mx;        \
  int i = (int)(_u - _q * (unsigned)(d).mx);        \
  int k = (int)(_q / (unsigned)(d).my);             \
  int j = (int)(_q - (unsigned)k * (unsigned)(d).my)

static inline int nblk(size_t n, int bs = 256) {
  size_t b = (n + bs - 1) / bs;
  if (b > 152 * 16) b = 152 * 16;
  return (int)(b ? b : 1);
}

// Rows (j, k) of the grid, a warp each: base cell o of the row, in: the row is
// interior in j and k.  One division a row instead of two a cell, and a warp
// reads consecutive cells.
#define ROW_LOOP(d)                                                                                       \
  const int _lane = threadIdx.x & 31, _rows = (d).my * (d).mz, _nw = gridDim.x * (RB / 32);             \
  for (int _r = blockIdx.x * (RB / 32) + (threadIdx.x >> 5); _r < _rows; _r += _nw)
#define ROW_DECOMP(d, j, k, o, in)                                                \
  const int k = _r / (d).my, j = _r - k * (d).my;                               \
  const size_t o = (size_t)_r * (d).mx;                                         \
  const bool in = j > 0 && k > 0 && j < (d).my - 1 && k < (d).mz - 1

// Blocks of a reduction (four per SM: a block's FP64 sums and the fence before
// its ticket cost as much as several rows; 256x128x128 divergence 84 us at 16,
// 76 at 8, 72 at 4) and of an update without one (eight).
static inline int row_blocks(const Dims& d, int per_sm = 4) {
  const int b = ((size_t)d.my * d.mz + RB / 32 - 1) / (RB / 32);
  return b < 152 * per_sm ? b : 152 * per_sm;
}

// Sums of NQ per-block partials (parts[q * nblocks + b]) in a fixed order, by
// the last block: out[q].
template <int NQ>
__device__ __forceinline__ void finish_sums(const double* parts, double* out, double* sh) {
  const int nb = gridDim.x;
  for (int q = 0; q < NQ; q++) {
    double s = 0.;
    for (int p = threadIdx.x; p < nb; p += blockDim.x) s += __ldcg(parts + (size_t)q * nb + p);
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[q] = s;
    __syncthreads();
  }
}
// Block maximum of integers that order like the values (max_abs), and the
// maximum of all blocks' by the last one.
__device__ __forceinline__ unsigned long long block_maxbits(unsigned long long v, double* sh) {
  return (unsigned long long)block_max((long long)v, (long long*)sh);
}
__device__ __forceinline__ double finish_max(const double* parts, double* sh) {
  unsigned long long m = 0ull;
  for (int p = threadIdx.x; p < (int)gridDim.x; p += blockDim.x) {
    const unsigned long long v = (unsigned long long)__double_as_longlong(__ldcg(parts + p));
    m = v > m ? v : m;
  }
  return __longlong_as_double((long long)block_maxbits(m, sh));
}

// ---- AoS (reference Cmpnts) <-> SoA device layout ----
__global__ void k_aos2soa(size_t n, const double* __restrict__ a, double* x, double* y, double* z) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    x[t] = a[3 * t];
    y[t] = a[3 * t + 1];
    z[t] = a[3 * t + 2];
  }
}
__global__ void k_soa2aos(size_t n, const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
                          double* a) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    a[3 * t] = x[t];
    a[3 * t + 1] = y[t];
    a[3 * t + 2] = z[t];
  }
}
int launch_aos2soa(size_t n, const double* aos, double* x, double* y, double* z, cudaStream_t s) {
  k_aos2soa<<<nblk(n), 256, 0, s>>>(n, aos, x, y, z); ++g_launches;
  return (int)cudaGetLastError();
}
int launch_soa2aos(size_t n, const double* x, const double* y, const double* z, double* aos, cudaStream_t s) {
  k_soa2aos<<<nblk(n), 256, 0, s>>>(n, x, y, z, aos); ++g_launches;
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// PoissonRHS2_hypre (poisson_hypre.c:342-429): b = div(U*) * st * coeff / dt
// on fluid cells, periodic wrap of the minus faces; partial sums of b and of
// the fluid count for the compatibility fix of PoissonRHS2 (poisson.c:1879-1903).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(RB) k_rhs(Dims d, Ucont u, const double* __restrict__ nvert,
                                            const uint8_t* __restrict__ nb8, double scale, double* b, double* parts,
                                            double* sc, unsigned* ticket) {
  __shared__ double sh[32];
  __shared__ unsigned shc[32];
  double lsum = 0.;
  unsigned lcnt = 0;  // fluid cells, counted on the integer pipe (exact)
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    const long long os = (j == 1 && d.jp) ? (long long)(d.my - 3) * d.mx : -(long long)d.mx;
    const long long ob = (k == 1 && d.kp) ? (long long)(d.mz - 3) * d.my * d.mx : -(long long)d.my * d.mx;
    for (int i = _lane; i < d.mx; i += 32) {
      const size_t c = o + i;
      double val = 0.;
      if (in && i > 0 && i < d.mx - 1) {  // the fluid test by select, so that no load waits for it
        const bool fluid = nb8 ? nb8[c] == 0 : !at_least(nvert[c], 0.1);
        // (0 - u_x) + u_x(i-1) is exactly the first difference
        double v = u.x[(i == 1 && d.ip) ? o + d.mx - 2 : c - 1] - u.x[c];
        v -= u.y[c];
        v += u.y[c + os];
        v -= u.z[c];
        v += u.z[c + ob];
        val = fluid ? v * scale : 0.;
        lsum += val;
        lcnt += fluid;
      }
      b[c] = val;
    }
  }
  lsum = block_sum(lsum, sh);
  lcnt = block_sum(lcnt, shc);
  if (threadIdx.x == 0) {
    parts[blockIdx.x] = lsum;
    parts[gridDim.x + blockIdx.x] = (double)lcnt;
  }
  if (last_block(ticket)) finish_sums<2>(parts, sc, sh);
}
// b += -sum / count on fluid interior cells (sc = {sum, count}).
__global__ void __launch_bounds__(RB) k_meanfix(Dims d, const double* __restrict__ nvert, const double* __restrict__ sc,
                                                double* b) {
  const double v = (sc[1] > 0.) ? -sc[0] / sc[1] : 0.;
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    if (!in) continue;
    for (int i = 1 + _lane; i < d.mx - 1; i += 32)
      if (below(nvert[o + i], 0.1)) b[o + i] += v;
  }
}
int launch_rhs(const Dims& d, const Ucont& u, const double* nvert, double dt, double st, double coeff, int meanfix,
               double* b, double* parts, double* sc, unsigned* ticket, cudaStream_t s, const uint8_t* nb8, const int* comp,
               int ncomp) {
  const int nb = row_blocks(d);
  k_rhs<<<nb, RB, 0, s>>>(d, u, nvert, nb8, -1.0 / dt * st * coeff, b, parts, sc, ticket); ++g_launches;
  if (meanfix && comp && ncomp > 1) {
    // one compatibility fix per connected fluid region (sums in sc[2..3])
    return launch_remove_mean(d, nvert, b, parts, sc + 2, ticket, s, comp, ncomp);
  }
  if (meanfix) {
    k_meanfix<<<row_blocks(d, 8), RB, 0, s>>>(d, nvert, sc, b);
    ++g_launches;
  }
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// IB flux balance.  mode 1: VolumeFlux(flg = 0), poisson.c:2898-3240
// (immersed == 1).  mode 0: VolumeFlux(lUcor), poisson.c:2634-2828 with
// immersed == 0, which zeroes every fluid / non-fluid face.
// phase 0: (mode 1) zero faces with |U| <= 1e-10 and sum flux, area;
// phase 1: apply the correction flux / area and sum the corrected faces again
// (the reference's second measuring pass, fused: same values, same order).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double nrm3(const double* v, size_t c) {
  return sqrt(v[3 * c] * v[3 * c] + v[3 * c + 1] * v[3 * c + 1] + v[3 * c + 2] * v[3 * c + 2]);
}

// nb8 (nvert as bytes, every value an integer in [0, 127]) turns the FP64
// interface tests into exact integer ones: nv < 0.1 <=> 0, nv > 0.1 <=> >= 1,
// 0.1 < nv < 1.1 <=> 1.
// Interface faces are few: a cell whose byte equals its three + neighbours'
// has none, and a warp without any skips the FP64 reductions.
__global__ void __launch_bounds__(RB) k_vflux(Dims d, int mode, int phase, Ucont u, const double* __restrict__ nv,
                                              const double* __restrict__ csi, const double* __restrict__ eta,
                                              const double* __restrict__ zet, const double* __restrict__ fa, double* parts,
                                              double* out, unsigned* ticket, const uint8_t* __restrict__ nb8) {
  __shared__ double sh[32];
  const double eps = 1.e-10, ibmval = 1.1;
  double flux = 0., area = 0.;
  double corr = 0.;
  bool any = false;
  if (phase == 1) corr = (fa[1] > 1.e-15) ? fa[0] / fa[1] : 0.;
  double* uf[3] = {u.x, u.y, u.z};
  const double* mt[3] = {csi, eta, zet};
  const int off[3] = {1, d.mx, d.mx * d.my};
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    if (!in) continue;
    for (int i = 1 + _lane; i < d.mx - 1; i += 32) {
      const size_t c = o + i;
      if (nb8) {
        const int a = nb8[c];
        // (no short circuit: the four loads go together)
        if (((a ^ nb8[c + off[0]]) | (a ^ nb8[c + off[1]]) | (a ^ nb8[c + off[2]])) == 0) continue;
      }
      const bool lim1[3] = {i < d.mx - 2, j < d.my - 2, k < d.mz - 2};
#pragma unroll
      for (int f = 0; f < 3; f++) {
        double* uu = uf[f];
        const size_t cf = c + off[f];
        bool plus, minus;
        if (mode == 1) {
          if (nb8) {
            const int a = nb8[c], b = nb8[cf];
            plus = a == 0 && b == 1 && lim1[f];
            minus = a == 1 && b == 0 && lim1[f];
          } else {
            plus = nv[c] < 0.1 && nv[cf] > 0.1 && nv[cf] < ibmval && lim1[f];
            minus = nv[c] > 0.1 && nv[c] < ibmval && nv[cf] < 0.1 && lim1[f];
          }
          if (!(plus || minus)) continue;
          any = true;
          if (phase == 0) {
            if (fabs(uu[c]) > eps) {
              flux += plus ? uu[c] : -uu[c];
              area += nrm3(mt[f], c);
            } else uu[c] = 0.;
          } else {
            // phase 1: correct, and measure the corrected face at once (the
            // same values and order as a separate measuring pass)
            const double nr = nrm3(mt[f], c);
            if (fabs(uu[c]) > eps) {
              if (plus) uu[c] -= nr * corr;
              else uu[c] += nr * corr;
            }
            flux += plus ? uu[c] : -uu[c];
            area += nr;
          }
        } else {
          if (nb8) {
            const int a = nb8[c], b = nb8[cf];
            plus = a == 0 && b != 0;
            minus = a != 0 && b == 0;
          } else {
            plus = nv[c] < VFS_THR && nv[cf] > VFS_THR;
            minus = nv[c] > VFS_THR && nv[cf] < VFS_THR;
          }
          if (!(plus || minus)) continue;
          any = true;
          if (phase == 1) uu[c] = 0.;  // and measured as such
          flux += plus ? uu[c] : -uu[c];
          area += nrm3(mt[f], c);
        }
      }
    }
  }
  if (__syncthreads_or(any)) {
    flux = block_sum(flux, sh);
    area = block_sum(area, sh);
  }
  if (threadIdx.x == 0) {
    parts[blockIdx.x] = flux;
    parts[gridDim.x + blockIdx.x] = area;
  }
  if (last_block(ticket)) finish_sums<2>(parts, out, sh);
}
int launch_volume_flux(const Dims& d, int mode, const Ucont& u, const double* nvert, const double* M, double* parts,
                       double* fa4, unsigned* ticket, cudaStream_t s, const uint8_t* nb8) {
  const size_t N = ncell(d);
  const int nb = row_blocks(d);
  const double *csi = M + N * MP_CSI, *eta = M + N * MP_ETA, *zet = M + N * MP_ZET;
  for (int phase = 0; phase < 2; phase++) {
    k_vflux<<<nb, RB, 0, s>>>(d, mode, phase, u, nvert, csi, eta, zet, fa4, parts, fa4 + 2 * phase, ticket, nb8);
    ++g_launches;
  }
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Remove_Nullspace (poisson_hypre.c:207-270): subtract the fluid mean of phi.
// With comp (labels of the connected fluid regions), only region q: a grid
// cut apart by bodies has one constant null vector per region, as in the
// reference's two-region split of PoissonNullSpaceFunction
// (poisson.c:819-873, regions from FullyBlocked, poisson.c:1918-1998).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(RB) k_fluid_sum(Dims d, const double* __restrict__ nvert, const double* __restrict__ x,
                                                  double* parts, double* sc, unsigned* ticket,
                                                  const int* __restrict__ comp, int q) {
  __shared__ double sh[32];
  __shared__ unsigned shc[32];
  double s = 0.;
  unsigned n = 0;  // counted on the integer pipe (exact)
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    if (!in) continue;
    for (int i = 1 + _lane; i < d.mx - 1; i += 32)
      if (below(nvert[o + i], 0.1) && (!comp || comp[o + i] == q)) {
        s += x[o + i];
        n += 1;
      }
  }
  s = block_sum(s, sh);
  n = block_sum(n, shc);
  if (threadIdx.x == 0) {
    parts[blockIdx.x] = s;
    parts[gridDim.x + blockIdx.x] = (double)n;
  }
  if (last_block(ticket)) finish_sums<2>(parts, sc, sh);
}
int launch_fluid_sum(const Dims& d, const double* nvert, const double* x, double* parts, double* sc, unsigned* ticket,
                     cudaStream_t s) {
  k_fluid_sum<<<row_blocks(d), RB, 0, s>>>(d, nvert, x, parts, sc, ticket, nullptr, 0); ++g_launches;
  return (int)cudaGetLastError();
}
__global__ void __launch_bounds__(RB) k_sub_mean(Dims d, const double* __restrict__ nvert, const double* __restrict__ sc,
                                                 double* x, const int* __restrict__ comp, int q) {
  const double v = (sc[1] > 0.) ? -sc[0] / sc[1] : 0.;
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    if (!in) continue;
    for (int i = 1 + _lane; i < d.mx - 1; i += 32)
      if (below(nvert[o + i], 0.1) && comp[o + i] == q) x[o + i] += v;
  }
}
int launch_remove_mean(const Dims& d, const double* nvert, double* x, double* parts, double* sc, unsigned* ticket,
                       cudaStream_t s, const int* comp, int ncomp) {
  const int nb = row_blocks(d);
  for (int q = 0; q < ncomp; q++) {
    k_fluid_sum<<<nb, RB, 0, s>>>(d, nvert, x, parts, sc, ticket, comp, q); ++g_launches;
    k_sub_mean<<<nb, RB, 0, s>>>(d, nvert, sc, x, comp, q); ++g_launches;
  }
  return (int)cudaGetLastError();
}

// v into interior cell (i, j, k) and into the ghost cells that mirror it
// through periodic axes (poisson.c:146-181, 2580-2616).  The thread of the
// source writes them, so a fill needs no launch after its update.
__device__ __forceinline__ void put_mirrored(const Dims& d, double* a, int i, int j, int k, double v) {
  a[cidx(d, i, j, k)] = v;
  const int gi = d.ip ? (i == 1 ? d.mx - 1 : i == d.mx - 2 ? 0 : -1) : -1;
  const int gj = d.jp ? (j == 1 ? d.my - 1 : j == d.my - 2 ? 0 : -1) : -1;
  const int gk = d.kp ? (k == 1 ? d.mz - 1 : k == d.mz - 2 ? 0 : -1) : -1;
  if (gi < 0 && gj < 0 && gk < 0) return;
  for (int q = 1; q < 8; q++) {
    const int x = q & 1 ? gi : i, y = q & 2 ? gj : j, z = q & 4 ? gk : k;
    if (x >= 0 && y >= 0 && z >= 0) a[cidx(d, x, y, z)] = v;
  }
}
// A ghost cell that mirrors an interior one (its value comes from there).
__device__ __forceinline__ bool mirrors(const Dims& d, int i, int j, int k) {
  return interior(d, wrapi(i, d.mx, d.ip), wrapi(j, d.my, d.jp), wrapi(k, d.mz, d.kp));
}

// Remove_Nullspace's mean (sc = {sum, count}, nullable), Convert_Phi2_Phi
// (poisson.c:97-185: zero on boundary and non-fluid cells) and the periodic
// ghosts in one pass.
__global__ void __launch_bounds__(RB) k_phi_finish(Dims d, const double* __restrict__ nvert, const double* __restrict__ sc,
                                                   double* phi) {
  const double v = (sc && sc[1] > 0.) ? -sc[0] / sc[1] : 0.;
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    for (int i = _lane; i < d.mx; i += 32) {
      if (in && i > 0 && i < d.mx - 1) {
        const double nv = nvert[o + i];
        double x = phi[o + i];
        if (below(nv, 0.1)) x += v;
        if (at_least(nv, 1.0)) x = 0.;  // (int)nv > 0.1
        put_mirrored(d, phi, i, j, k, x);
      } else if (!mirrors(d, i, j, k)) {
        phi[o + i] = 0.;
      }
    }
  }
}
int launch_phi_finish(const Dims& d, const double* nvert, double* phi, const double* sc, cudaStream_t s) {
  k_phi_finish<<<row_blocks(d, 8), RB, 0, s>>>(d, nvert, sc, phi); ++g_launches;
  return (int)cudaGetLastError();
}

// UpdatePressure (poisson.c:2522-2548, non-PRIMITIVE branch, + ghost fill): a
// ghost whose mirror is a boundary cell of another axis copies that cell,
// which the update leaves alone.
__global__ void __launch_bounds__(RB) k_update_p(Dims d, const double* __restrict__ nvert, const double* __restrict__ phi,
                                                 double* p) {
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    for (int i = _lane; i < d.mx; i += 32) {
      if (in && i > 0 && i < d.mx - 1) {
        double x = p[o + i];
        if (below(nvert[o + i], 0.1)) x += phi[o + i];
        put_mirrored(d, p, i, j, k, x);
      } else if (!mirrors(d, i, j, k)) {
        const size_t src = cidx(d, wrapi(i, d.mx, d.ip), wrapi(j, d.my, d.jp), wrapi(k, d.mz, d.kp));
        if (src != o + i) p[o + i] = p[src];
      }
    }
  }
}
int launch_update_pressure(const Dims& d, const double* nvert, const double* phi, double* p, cudaStream_t s) {
  k_update_p<<<row_blocks(d, 8), RB, 0, s>>>(d, nvert, phi, p); ++g_launches;
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Projection (poisson.c:2202-2397): U^xi -= (dpdc g11 + dpde g12 + dpdz g13)
// dt st / coeff at i faces (likewise j, k), with the LHS's one-sided /
// centred / zero regimes for the cross derivatives; faces touching nvert are
// left alone.  pd holds the nine metric dot products of each face family
// (icsi.icsi, ieta.icsi, izet.icsi, jcsi.jeta, jeta.jeta, jzet.jeta,
// kcsi.kzet, keta.kzet, kzet.kzet) and M the face Jacobians iaj, jaj, kaj,
// multiplied in the reference's order: (dpdc * dot) * iaj.
// ---------------------------------------------------------------------------
// x / coeff is skipped when coeff == 1 (x / 1.0 == x exactly), and x * st
// when st == 1 (x * 1.0 == x exactly); r1 = r2 = r3 = 1 (no level set), so
// their divisions are always exact and omitted.
__device__ __forceinline__ double div_c(double x, double coeff) { return coeff == 1.0 ? x : x / coeff; }
__device__ __forceinline__ double mul_st(double x, double st) { return st == 1.0 ? x : x * st; }

template <bool NVI>
__global__ void __launch_bounds__(128) k_projection(Dims d, size_t c0, size_t c1, const double* __restrict__ pd,
                             const double* __restrict__ iaj,
                             const double* __restrict__ jaj, const double* __restrict__ kaj, const double* __restrict__ nvert,
                             const uint8_t* __restrict__ nb8, const double* __restrict__ phi, double dt, double st,
                             double coeff, Ucont u) {
  const size_t N = ncell(d);
  const int mx = d.mx, my = d.my, mz = d.mz, ip = d.ip, jp = d.jp, kp = d.kp;
  const double THR = VFS_THR;
  auto gt2 = [&](size_t a, size_t b) -> bool {
    if (NVI) return (nb8[a] | nb8[b]) != 0;
    return nvert[a] + nvert[b] > THR;
  };
  auto lt2 = [&](size_t a, size_t b) -> bool {
    if (NVI) return (nb8[a] | nb8[b]) == 0;
    return nvert[a] + nvert[b] < THR;
  };
  RANGE_LOOP(c0, c1) {
    DECOMP(d, i, j, k);
    const size_t c = _t;
// nvert pair tests: with NVI every nvert is an integer in [0, 127] and nb8
// holds it as a byte, so a + b > 0.1 <=> (a | b) != 0 and a + b < 0.1 <=>
// (a | b) == 0 exactly (no FP64 add and compare)
#define NVX(ii, jj, kk) cidx(d, ii, jj, kk)
#define GT2(A, B) gt2(NVX A, NVX B)
#define LT2(A, B) lt2(NVX A, NVX B)
#define PH(ii, jj, kk) phi[cidx(d, ii, jj, kk)]
    double dpdc, dpde, dpdz;
    if (j > 0 && j < my - 1 && k > 0 && k < mz - 1)
      if ((i > 0 && i < mx - 2) || (ip && i == mx - 2)) {
        dpdc = PH(i + 1, j, k) - PH(i, j, k);
        if (i == mx - 2 && ip) dpdc = PH(1, j, k) - PH(i, j, k);
        dpde = 0.;
        dpdz = 0.;
        if ((j == my - 2 && !jp) || GT2((i, j + 1, k), (i + 1, j + 1, k))) {
          if (LT2((i, j - 1, k), (i + 1, j - 1, k)) && (j != 1))
            dpde = (PH(i, j, k) + PH(i + 1, j, k) - PH(i, j - 1, k) - PH(i + 1, j - 1, k)) * 0.5;
        } else if ((j == 1 && !jp) || GT2((i, j - 1, k), (i + 1, j - 1, k))) {
          if (LT2((i, j + 1, k), (i + 1, j + 1, k)))
            dpde = (PH(i, j + 1, k) + PH(i + 1, j + 1, k) - PH(i, j, k) - PH(i + 1, j, k)) * 0.5;
        } else {
          dpde = (PH(i, j + 1, k) + PH(i + 1, j + 1, k) - PH(i, j - 1, k) - PH(i + 1, j - 1, k)) * 0.25;
        }
        if ((k == mz - 2 && !kp) || GT2((i, j, k + 1), (i + 1, j, k + 1))) {
          if (LT2((i, j, k - 1), (i + 1, j, k - 1)) && (k != 1))
            dpdz = (PH(i, j, k) + PH(i + 1, j, k) - PH(i, j, k - 1) - PH(i + 1, j, k - 1)) * 0.5;
        } else if ((k == 1 && !kp) || GT2((i, j, k - 1), (i + 1, j, k - 1))) {
          if (LT2((i, j, k + 1), (i + 1, j, k + 1)))
            dpdz = (PH(i, j, k + 1) + PH(i + 1, j, k + 1) - PH(i, j, k) - PH(i + 1, j, k)) * 0.5;
        } else {
          dpdz = (PH(i, j, k + 1) + PH(i + 1, j, k + 1) - PH(i, j, k - 1) - PH(i + 1, j, k - 1)) * 0.25;
        }
        if (LT2((i, j, k), (i + 1, j, k))) {
          const double a = iaj[c];
          u.x[c] -= div_c(mul_st((dpdc * pd[0 * N + c] * a + dpde * pd[1 * N + c] * a + dpdz * pd[2 * N + c] * a) * dt, st), coeff);
        }
      }
    if (i > 0 && i < mx - 1 && k > 0 && k < mz - 1)
      if ((j > 0 && j < my - 2) || (jp && j == my - 2)) {
        dpdc = 0.;
        dpdz = 0.;
        if ((i == mx - 2 && !ip) || GT2((i + 1, j, k), (i + 1, j + 1, k))) {
          if (LT2((i - 1, j, k), (i - 1, j + 1, k)) && (i != 1))
            dpdc = (PH(i, j, k) + PH(i, j + 1, k) - PH(i - 1, j, k) - PH(i - 1, j + 1, k)) * 0.5;
        } else if ((i == 1 && !ip) || GT2((i - 1, j, k), (i - 1, j + 1, k))) {
          if (LT2((i + 1, j, k), (i + 1, j + 1, k)))
            dpdc = (PH(i + 1, j, k) + PH(i + 1, j + 1, k) - PH(i, j, k) - PH(i, j + 1, k)) * 0.5;
        } else {
          dpdc = (PH(i + 1, j, k) + PH(i + 1, j + 1, k) - PH(i - 1, j, k) - PH(i - 1, j + 1, k)) * 0.25;
        }
        if (j == my - 2 && jp) dpde = PH(i, 1, k) - PH(i, j, k);
        else dpde = PH(i, j + 1, k) - PH(i, j, k);
        if ((k == mz - 2 && !kp) || GT2((i, j, k + 1), (i, j + 1, k + 1))) {
          if (LT2((i, j, k - 1), (i, j + 1, k - 1)) && (k != 1))
            dpdz = (PH(i, j, k) + PH(i, j + 1, k) - PH(i, j, k - 1) - PH(i, j + 1, k - 1)) * 0.5;
        } else if ((k == 1 && !kp) || GT2((i, j, k - 1), (i, j + 1, k - 1))) {
          if (LT2((i, j, k + 1), (i, j + 1, k + 1)))
            dpdz = (PH(i, j, k + 1) + PH(i, j + 1, k + 1) - PH(i, j, k) - PH(i, j + 1, k)) * 0.5;
        } else {
          dpdz = (PH(i, j, k + 1) + PH(i, j + 1, k + 1) - PH(i, j, k - 1) - PH(i, j + 1, k - 1)) * 0.25;
        }
        if (LT2((i, j, k), (i, j + 1, k))) {
          const double a = jaj[c];
          u.y[c] -= div_c(mul_st((dpdc * pd[3 * N + c] * a + dpde * pd[4 * N + c] * a + dpdz * pd[5 * N + c] * a) * dt, st), coeff);
        }
      }
    if (i > 0 && i < mx - 1 && j > 0 && j < my - 1)
      if ((k > 0 && k < mz - 2) || (kp && k == mz - 2)) {
        dpdc = 0.;
        dpde = 0.;
        if ((i == mx - 2 && !ip) || GT2((i + 1, j, k), (i + 1, j, k + 1))) {
          if (LT2((i - 1, j, k), (i - 1, j, k + 1)) && (i != 1))
            dpdc = (PH(i, j, k) + PH(i, j, k + 1) - PH(i - 1, j, k) - PH(i - 1, j, k + 1)) * 0.5;
        } else if ((i == 1 && !ip) || GT2((i - 1, j, k), (i - 1, j, k + 1))) {
          if (LT2((i + 1, j, k), (i + 1, j, k + 1)))
            dpdc = (PH(i + 1, j, k) + PH(i + 1, j, k + 1) - PH(i, j, k) - PH(i, j, k + 1)) * 0.5;
        } else {
          dpdc = (PH(i + 1, j, k) + PH(i + 1, j, k + 1) - PH(i - 1, j, k) - PH(i - 1, j, k + 1)) * 0.25;
        }
        if ((j == my - 2 && !jp) || GT2((i, j + 1, k), (i, j + 1, k + 1))) {
          if (LT2((i, j - 1, k), (i, j - 1, k + 1)) && (j != 1))
            dpde = (PH(i, j, k) + PH(i, j, k + 1) - PH(i, j - 1, k) - PH(i, j - 1, k + 1)) * 0.5;
        } else if ((j == 1 && !jp) || GT2((i, j - 1, k), (i, j - 1, k + 1))) {
          if (LT2((i, j + 1, k), (i, j + 1, k + 1)))
            dpde = (PH(i, j + 1, k) + PH(i, j + 1, k + 1) - PH(i, j, k) - PH(i, j, k + 1)) * 0.5;
        } else {
          dpde = (PH(i, j + 1, k) + PH(i, j + 1, k + 1) - PH(i, j - 1, k) - PH(i, j - 1, k + 1)) * 0.25;
        }
        if (k == mz - 2 && kp) dpdz = PH(i, j, 1) - PH(i, j, k);
        else dpdz = PH(i, j, k + 1) - PH(i, j, k);
        if (LT2((i, j, k), (i, j, k + 1))) {
          const double a = kaj[c];
          u.z[c] -= div_c(mul_st((dpdc * pd[6 * N + c] * a + dpde * pd[7 * N + c] * a + dpdz * pd[8 * N + c] * a) * dt, st), coeff);
        }
      }
#undef PH
#undef NVX
#undef GT2
#undef LT2
  }
}

// ---------------------------------------------------------------------------
// Projection on precomputed face weights.  Every choice the reference's
// Projection makes per face (poisson.c:2221-2363: the face is skipped where
// nvert touches it, each cross derivative is centred, one-sided or zero by
// the nvert and wall tests) depends on the grid only, so it is made once
// (k_proj_weights, at the operator set-up): per face a normal weight
// dot * aj_face and two cross weights s * dot * aj_face (s = 0.25 centred,
// 0.5 one-sided, 0 none; all three 0 where the face is not projected), and
// per cross term two code bits choosing its upper and lower pair (the pair
// beside the face, or the face's own pair for a one-sided difference).  The
// step then applies, per face, U -= (wN dn + wA (Up_A - Lo_A) + wB (Up_B -
// Lo_B)) dt st / coeff with FMAs and no nvert loads: 9 FP64 operations per
// cell and 4 per cross term in use, at most 33, instead of about 60 (they
// bound the kernel).  The same products in a
// different order: the result differs from the reference's operation order
// by rounding (<= 1e-14 relative).  used: bit q is set where some weight
// pw[q] is not zero (grids uniform along an axis have whole arrays of zero
// cross weights, which the step does not read).
// pw: [9][N] (i face: normal, j cross, k cross | j face: normal, i cross,
// k cross | k face: normal, i cross, j cross); pc: two bits per cross term
// in that order (bit 0: the upper pair is the face's own, bit 1: the lower),
// then bits 12, 13, 14: the i, j, k face is projected (a face that is not
// keeps its flux bit for bit).
// ---------------------------------------------------------------------------
__global__ void k_proj_weights(Dims d, const double* __restrict__ pd, const double* __restrict__ iaj,
                               const double* __restrict__ jaj, const double* __restrict__ kaj,
                               const double* __restrict__ nvert, double* __restrict__ pw, uint16_t* __restrict__ pc,
                               unsigned* __restrict__ used) {
  const size_t N = ncell(d);
  unsigned mine = 0;
  const int mx = d.mx, my = d.my, mz = d.mz, ip = d.ip, jp = d.jp, kp = d.kp;
  const double THR = VFS_THR;
  GRID_LOOP(d) {
    DECOMP(d, i, j, k);
    const size_t c = _t;
#define NVX(ii, jj, kk) nvert[cidx(d, ii, jj, kk)]
#define GT2(a, b, cc, e, f, g_) (NVX(a, b, cc) + NVX(e, f, g_) > THR)
#define LT2(a, b, cc, e, f, g_) (NVX(a, b, cc) + NVX(e, f, g_) < THR)
    double w[9] = {0., 0., 0., 0., 0., 0., 0., 0., 0.};
    unsigned code = 0;
    // one cross term: up/low pairs (the face's own one where one-sided) and the scale
    auto cross = [&](bool top_blocked, bool low_ok, bool bot_blocked, bool up_ok, double& sc, unsigned& bits) {
      sc = 0.;
      bits = 0;
      if (top_blocked) {
        if (low_ok) sc = 0.5, bits = 1u;  // (own pair) - (lower pair)
      } else if (bot_blocked) {
        if (up_ok) sc = 0.5, bits = 2u;   // (upper pair) - (own pair)
      } else {
        sc = 0.25;                         // (upper pair) - (lower pair)
      }
    };
    if (j > 0 && j < my - 1 && k > 0 && k < mz - 1 && ((i > 0 && i < mx - 2) || (ip && i == mx - 2)) &&
        LT2(i, j, k, i + 1, j, k)) {  // i face, poisson.c:2221-2265
      double se, sz;
      unsigned be, bz;
      cross((j == my - 2 && !jp) || GT2(i, j + 1, k, i + 1, j + 1, k), LT2(i, j - 1, k, i + 1, j - 1, k) && j != 1,
            (j == 1 && !jp) || GT2(i, j - 1, k, i + 1, j - 1, k), LT2(i, j + 1, k, i + 1, j + 1, k), se, be);
      cross((k == mz - 2 && !kp) || GT2(i, j, k + 1, i + 1, j, k + 1), LT2(i, j, k - 1, i + 1, j, k - 1) && k != 1,
            (k == 1 && !kp) || GT2(i, j, k - 1, i + 1, j, k - 1), LT2(i, j, k + 1, i + 1, j, k + 1), sz, bz);
      const double a = iaj[c];
      w[0] = pd[0 * N + c] * a;
      w[1] = se * (pd[1 * N + c] * a);
      w[2] = sz * (pd[2 * N + c] * a);
      code |= be | (bz << 2) | (1u << 12);
    }
    if (i > 0 && i < mx - 1 && k > 0 && k < mz - 1 && ((j > 0 && j < my - 2) || (jp && j == my - 2)) &&
        LT2(i, j, k, i, j + 1, k)) {  // j face, poisson.c:2267-2314
      double sc, sz;
      unsigned bc, bz;
      cross((i == mx - 2 && !ip) || GT2(i + 1, j, k, i + 1, j + 1, k), LT2(i - 1, j, k, i - 1, j + 1, k) && i != 1,
            (i == 1 && !ip) || GT2(i - 1, j, k, i - 1, j + 1, k), LT2(i + 1, j, k, i + 1, j + 1, k), sc, bc);
      cross((k == mz - 2 && !kp) || GT2(i, j, k + 1, i, j + 1, k + 1), LT2(i, j, k - 1, i, j + 1, k - 1) && k != 1,
            (k == 1 && !kp) || GT2(i, j, k - 1, i, j + 1, k - 1), LT2(i, j, k + 1, i, j + 1, k + 1), sz, bz);
      const double a = jaj[c];
      w[3] = pd[4 * N + c] * a;
      w[4] = sc * (pd[3 * N + c] * a);
      w[5] = sz * (pd[5 * N + c] * a);
      code |= (bc << 4) | (bz << 6) | (1u << 13);
    }
    if (i > 0 && i < mx - 1 && j > 0 && j < my - 1 && ((k > 0 && k < mz - 2) || (kp && k == mz - 2)) &&
        LT2(i, j, k, i, j, k + 1)) {  // k face, poisson.c:2316-2363
      double sc, se;
      unsigned bc, be;
      cross((i == mx - 2 && !ip) || GT2(i + 1, j, k, i + 1, j, k + 1), LT2(i - 1, j, k, i - 1, j, k + 1) && i != 1,
            (i == 1 && !ip) || GT2(i - 1, j, k, i - 1, j, k + 1), LT2(i + 1, j, k, i + 1, j, k + 1), sc, bc);
      cross((j == my - 2 && !jp) || GT2(i, j + 1, k, i, j + 1, k + 1), LT2(i, j - 1, k, i, j - 1, k + 1) && j != 1,
            (j == 1 && !jp) || GT2(i, j - 1, k, i, j - 1, k + 1), LT2(i, j + 1, k, i, j + 1, k + 1), se, be);
      const double a = kaj[c];
      w[6] = pd[8 * N + c] * a;
      w[7] = sc * (pd[6 * N + c] * a);
      w[8] = se * (pd[7 * N + c] * a);
      code |= (bc << 8) | (be << 10) | (1u << 14);
    }
#undef NVX
#undef GT2
#undef LT2
#pragma unroll
    for (int q = 0; q < 9; q++) {
      pw[(size_t)q * N + c] = w[q];
      if (w[q] != 0.) mine |= 1u << q;
    }
    pc[c] = (uint16_t)code;
  }
  mine = __reduce_or_sync(0xFFFFFFFFu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicOr(used, mine);
}

int launch_proj_weights(const Dims& d, const double* pd, const double* M, const double* nvert, double* pw, uint16_t* pc,
                        unsigned* used, cudaStream_t s) {
  const size_t N = ncell(d);
  VFS_CUDA_OK(cudaMemsetAsync(used, 0, sizeof(unsigned), s));
  k_proj_weights<<<nblk(N), 256, 0, s>>>(d, pd, M + N * MP_IAJ, M + N * MP_JAJ, M + N * MP_KAJ, nvert, pw, pc, used);
  ++g_launches;
  return (int)cudaGetLastError();
}

// U -= sc (wN dn + wA (Up_A - Lo_A) + wB (Up_B - Lo_B)) on the projected
// faces of the cells [c0, c1) (interior planes; the face bits are set on
// interior cells only, and the normal difference wraps only on a periodic
// seam, where alone the last face is projected).  All loads but the cross
// terms' wait for nothing, and those only for the code; every phi read lies in
// the array: the seven points of any cell of an interior plane do, the cross
// terms' are read by interior cells.  The FP64 pipe bounds it (branches for
// the one-sided and zero terms ran 23 operations where 17 are needed):
// 256x128x128 (i-k terms only) 234 -> 164 us, 512x256x256 2361 -> 1833.
__global__ void __launch_bounds__(128) k_projection_fast(Dims d, size_t c0, size_t c1, unsigned used,
                                                         const double* __restrict__ pw,
                                                         const uint16_t* __restrict__ pc,
                                                         const double* __restrict__ phi, double sc, Ucont u) {
  const size_t N = ncell(d);
  const int mx = d.mx, my = d.my, mz = d.mz;
  const int sy = mx, sz = mx * my;
  RANGE_LOOP(c0, c1) {
    DECOMP(d, i, j, k);
    const int c = (int)_t;
    const unsigned code = pc[c];
    double w[9];
#pragma unroll
    for (int q = 0; q < 9; q++) w[q] = (used >> q) & 1u ? pw[(size_t)q * N + c] : 0.;
    const double pc0 = phi[c];
    const double pe = phi[i == mx - 2 ? c + 3 - mx : c + 1];
    const double pn = phi[j == my - 2 ? c + (3 - my) * sy : c + sy];
    const double pt = phi[k == mz - 2 ? c + (3 - mz) * sz : c + sz];
    const double ux = u.x[c], uy = u.y[c], uz = u.z[c];
    // t + weight (upper - lower pair of c and c + e along o) for cross term q;
    // a one-sided term takes the face's own pair by offset, not by branch or
    // select of sums (both cost FP64 operations), and a face that is not
    // projected or a zero weight takes none
    auto cross = [&](int q, double t, unsigned face, int e, int o, unsigned bits) -> double {
      if (!((used >> q) & 1u)) return t;
      const int up = (face && !(bits & 1u)) ? o : 0, lo = (face && !(bits & 2u)) ? -o : 0, ee = face ? e : 0;
      const double s = fma(w[q], (phi[c + up] - phi[c + lo]) + (phi[c + ee + up] - phi[c + ee + lo]), t);
      return zero_bits(w[q]) ? t : s;
    };
    const unsigned fi = code & (1u << 12), fj = code & (1u << 13), fk = code & (1u << 14);
    double tx = w[0] * (pe - pc0), ty = w[3] * (pn - pc0), tz = w[6] * (pt - pc0);
    tx = cross(1, tx, fi, 1, sy, code);
    tx = cross(2, tx, fi, 1, sz, code >> 2);
    ty = cross(4, ty, fj, sy, 1, code >> 4);
    ty = cross(5, ty, fj, sy, sz, code >> 6);
    tz = cross(7, tz, fk, sz, 1, code >> 8);
    tz = cross(8, tz, fk, sz, sy, code >> 10);
    if (fi) u.x[c] = fma(-tx, sc, ux);
    if (fj) u.y[c] = fma(-ty, sc, uy);
    if (fk) u.z[c] = fma(-tz, sc, uz);
  }
}

int launch_projection_fast(const Dims& d, unsigned used, const double* pw, const uint16_t* pc, const double* phi, double dt, double st,
                           double coeff, const Ucont& u, cudaStream_t s, int k0, int k1) {
  const size_t P = (size_t)d.mx * d.my;
  if (k1 < 0) k1 = d.mz;
  if (k0 < 0 || k0 >= k1 || k1 > d.mz) return (int)cudaErrorInvalidValue;
  const int p0 = k0 > 1 ? k0 : 1, p1 = k1 < d.mz - 1 ? k1 : d.mz - 1;
  if (p0 < p1) {
    const size_t c0 = p0 * P, c1 = p1 * P;
    const double sc = dt * st / coeff;
    k_projection_fast<<<(unsigned)((c1 - c0 + 127) / 128), 128, 0, s>>>(d, c0, c1, used, pw, pc, phi, sc, u);
    ++g_launches;
  }
  return launch_ucont_ghosts(d, u, k0, k1, s);
}

// periodic ghost sync of the flagged component (poisson.c:2398-2437) on
// planes [k0, k1): the i ghost planes of u.x, the j ghost planes of u.y and
// the k ghost planes of u.z, no other cell.  Every source is interior in all
// periodic directions, so the sync never reads a cell it writes; the source
// of a cell on an interior plane k lies on plane k.
__global__ void k_ucont_ghosts(Dims d, int k0, int k1, Ucont u) {
  const int nk = k1 - k0, nx = d.ip ? 2 * d.my * nk : 0, ny = d.jp ? 2 * d.mx * nk : 0;
  const int g0 = k0 == 0 ? 1 : 0, g1 = k1 == d.mz ? 1 : 0;  // k ghost planes in the range
  const int nz = d.kp ? (g0 + g1) * d.mx * d.my : 0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nx + ny + nz; t += gridDim.x * blockDim.x) {
    int i, j, k;
    double* a;
    if (t < nx) {
      const int q = t >> 1;
      i = t & 1 ? d.mx - 1 : 0;
      j = q % d.my;
      k = k0 + q / d.my;
      a = u.x;
    } else if (t < nx + ny) {
      const int q = t - nx, r = q / d.mx;
      i = q - r * d.mx;
      j = r & 1 ? d.my - 1 : 0;
      k = k0 + (r >> 1);
      a = u.y;
    } else {
      const int q = t - nx - ny, r = q / d.mx;
      i = q - r * d.mx;
      j = r % d.my;
      k = (r >= d.my || !g0) ? d.mz - 1 : 0;
      a = u.z;
    }
    a[cidx(d, i, j, k)] = a[cidx(d, wrapi(i, d.mx, d.ip), wrapi(j, d.my, d.jp), wrapi(k, d.mz, d.kp))];
  }
}

// The nine metric dot products of the projection (same expressions as the
// reference's Projection, poisson.c:2262-2360, without the Jacobian).
__global__ void k_proj_dots(Dims d, const double* __restrict__ M, double* pd) {
  const size_t N = ncell(d);
  GRID_LOOP(d) {
    const size_t c = _t;
    const double* A = M + N * MP_ICSI + 3 * c;
    const double* B = M + N * MP_IETA + 3 * c;
    const double* E = M + N * MP_IZET + 3 * c;
    pd[0 * N + c] = A[0] * A[0] + A[1] * A[1] + A[2] * A[2];
    pd[1 * N + c] = B[0] * A[0] + B[1] * A[1] + B[2] * A[2];
    pd[2 * N + c] = E[0] * A[0] + E[1] * A[1] + E[2] * A[2];
    A = M + N * MP_JCSI + 3 * c;
    B = M + N * MP_JETA + 3 * c;
    E = M + N * MP_JZET + 3 * c;
    pd[3 * N + c] = A[0] * B[0] + A[1] * B[1] + A[2] * B[2];
    pd[4 * N + c] = B[0] * B[0] + B[1] * B[1] + B[2] * B[2];
    pd[5 * N + c] = E[0] * B[0] + E[1] * B[1] + E[2] * B[2];
    A = M + N * MP_KCSI + 3 * c;
    B = M + N * MP_KETA + 3 * c;
    E = M + N * MP_KZET + 3 * c;
    pd[6 * N + c] = A[0] * E[0] + A[1] * E[1] + A[2] * E[2];
    pd[7 * N + c] = B[0] * E[0] + B[1] * E[1] + B[2] * E[2];
    pd[8 * N + c] = E[0] * E[0] + E[1] * E[1] + E[2] * E[2];
  }
}
int launch_proj_dots(const Dims& d, const double* M, double* pd, cudaStream_t s) {
  k_proj_dots<<<nblk(ncell(d)), 256, 0, s>>>(d, M, pd); ++g_launches;
  return (int)cudaGetLastError();
}

int launch_projection(const Dims& d, const double* pd, const double* M, const double* nvert, const uint8_t* nb8,
                      const double* phi, double dt, double st, double coeff, const Ucont& u, cudaStream_t s, int k0,
                      int k1) {
  const size_t N = ncell(d);
  const size_t P = (size_t)d.mx * d.my;
  if (k1 < 0) k1 = d.mz;
  if (k0 < 0 || k0 >= k1 || k1 > d.mz) return (int)cudaErrorInvalidValue;
  // planes 0 and mz-1 hold no projected face (every branch needs 0 < k < mz-1)
  const int p0 = k0 > 1 ? k0 : 1, p1 = k1 < d.mz - 1 ? k1 : d.mz - 1;
  if (p0 < p1) {
    const size_t c0 = p0 * P, c1 = p1 * P;
    if (nb8)
      k_projection<true><<<nblk(c1 - c0, 128), 128, 0, s>>>(d, c0, c1, pd, M + N * MP_IAJ, M + N * MP_JAJ,
                                                            M + N * MP_KAJ, nvert, nb8, phi, dt, st, coeff, u);
    else
      k_projection<false><<<nblk(c1 - c0, 128), 128, 0, s>>>(d, c0, c1, pd, M + N * MP_IAJ, M + N * MP_JAJ,
                                                             M + N * MP_KAJ, nvert, nb8, phi, dt, st, coeff, u);
    ++g_launches;
  }
  return launch_ucont_ghosts(d, u, k0, k1, s);
}

int launch_ucont_ghosts(const Dims& d, const Ucont& u, int k0, int k1, cudaStream_t s) {
  const size_t P = (size_t)d.mx * d.my;
  if (k0 < 0 || k0 >= k1 || k1 > d.mz) return (int)cudaErrorInvalidValue;
  const size_t n = (size_t)(d.ip ? 2 * d.my * (k1 - k0) : 0) + (d.jp ? 2 * d.mx * (k1 - k0) : 0) +
                   (d.kp ? ((k0 == 0) + (k1 == d.mz)) * P : 0);
  if (n == 0) return (int)cudaSuccess;
  k_ucont_ghosts<<<nblk(n), 256, 0, s>>>(d, k0, k1, u); ++g_launches;
  return (int)cudaGetLastError();
}

// Contra2Cart (rhs.c:144-183): Cartesian velocity at fluid cells, the
// solution of [csi; eta; zet] ucat = q for the cell-centred contravariant
// fluxes q.  The reference solves each cell's 3 x 3 system by Cramer's rule
// (three FP64 divisions); the metric is static, so its inverse (adjugate /
// determinant, same cofactors) is formed once per grid, with the 1/2 of the
// face average q = (U_f- + U_f+) / 2 folded in (an exact power-of-two
// scale), and the step applies it with three multiplies and six FMAs (this
// unit is built without automatic contraction; the FMAs are explicit).
// Agrees with Cramer's rule to rounding.
__global__ void k_inverse_metric(Dims d, const double* __restrict__ M, const double* __restrict__ nvert, double* minv) {
  const size_t N = ncell(d);
  GRID_LOOP(d) {
    DECOMP(d, i, j, k);
    double* o = minv + 9 * _t;
    if (!interior(d, i, j, k) || !(nvert[_t] < 0.1)) {
      for (int q = 0; q < 9; q++) o[q] = 0.;
      continue;
    }
    const size_t c = _t;
    const double* A = M + N * MP_CSI + 3 * c;
    const double* B = M + N * MP_ETA + 3 * c;
    const double* E = M + N * MP_ZET + 3 * c;
    const double det = A[0] * (B[1] * E[2] - B[2] * E[1]) - A[1] * (B[0] * E[2] - B[2] * E[0]) + A[2] * (B[0] * E[1] - B[1] * E[0]);
    const double r = 0.5 / det;
    o[0] = (B[1] * E[2] - B[2] * E[1]) * r;
    o[1] = -(A[1] * E[2] - A[2] * E[1]) * r;
    o[2] = (A[1] * B[2] - A[2] * B[1]) * r;
    o[3] = -(B[0] * E[2] - B[2] * E[0]) * r;
    o[4] = (A[0] * E[2] - A[2] * E[0]) * r;
    o[5] = -(A[0] * B[2] - A[2] * B[0]) * r;
    o[6] = (B[0] * E[1] - B[1] * E[0]) * r;
    o[7] = -(A[0] * E[1] - A[1] * E[0]) * r;
    o[8] = (A[0] * B[1] - A[1] * B[0]) * r;
  }
}
int launch_inverse_metric(const Dims& d, const double* M, const double* nvert, double* minv, cudaStream_t s) {
  k_inverse_metric<<<nblk(ncell(d)), 256, 0, s>>>(d, M, nvert, minv); ++g_launches;
  return (int)cudaGetLastError();
}

__global__ void k_contra2cart(Dims d, const double* __restrict__ minv, const double* __restrict__ nvert, Ucont u,
                              double* ucat) {
  GRID_LOOP(d) {
    DECOMP(d, i, j, k);
    if (!interior(d, i, j, k) || !(nvert[_t] < 0.1)) continue;
    const size_t c = _t;
    const double* m = minv + 9 * c;
    const double q0 = u.x[cidx(d, i - 1, j, k)] + u.x[c];  // twice the face averages
    const double q1 = u.y[cidx(d, i, j - 1, k)] + u.y[c];
    const double q2 = u.z[cidx(d, i, j, k - 1)] + u.z[c];
    ucat[3 * c] = fma(m[2], q2, fma(m[1], q1, m[0] * q0));
    ucat[3 * c + 1] = fma(m[5], q2, fma(m[4], q1, m[3] * q0));
    ucat[3 * c + 2] = fma(m[8], q2, fma(m[7], q1, m[6] * q0));
  }
}
int launch_contra2cart(const Dims& d, const double* minv, const double* nvert, const Ucont& u, double* ucat, cudaStream_t s) {
  k_contra2cart<<<nblk(ncell(d)), 256, 0, s>>>(d, minv, nvert, u, ucat); ++g_launches;
  return (int)cudaGetLastError();
}

// Divergence (main.c:1279-1349): max over cells of |div U| * aj, 0 where the
// cell or a face neighbour carries nvert.
// Cell c or one of its six face neighbours carries nvert (the reference's
// sum > 0.1 test).  With nb8 (every nvert an integer in [0, 127]) the sum of
// non-negative integers exceeds 0.1 exactly when one of them is nonzero, an
// integer or of the bytes.
__device__ __forceinline__ bool near_body(const Dims& d, const double* __restrict__ nvert,
                                          const uint8_t* __restrict__ nb8, size_t c) {
  const size_t sy = d.mx, sz = (size_t)d.mx * d.my;
  if (nb8) return (nb8[c] | nb8[c + sz] | nb8[c - sz] | nb8[c + sy] | nb8[c - sy] | nb8[c + 1] | nb8[c - 1]) != 0;
  const double n0 = nvert[c], nt = nvert[c + sz], nbk = nvert[c - sz], nn = nvert[c + sy], ns = nvert[c - sy],
               ne = nvert[c + 1], nw = nvert[c - 1];
  // all zero (bits, on the integer pipe) almost everywhere; else the reference's sum
  if (((abs_bits(n0) | abs_bits(nt) | abs_bits(nbk)) | (abs_bits(nn) | abs_bits(ns)) | (abs_bits(ne) | abs_bits(nw))) == 0ull)
    return false;
  return n0 + nt + nbk + nn + ns + ne + nw > 0.1;
}

// What bounds it: the FP64 pipe, six operations a cell (the test for bodies and
// the maximum run on the integer pipe: 256x128x128 83 -> 72 us; a caller's
// 151x67x93 arrays with doubles for nvert 44.6 -> 22.5 us a call).
// The block's maximum as max_abs bits, in every thread.
__device__ __forceinline__ unsigned long long divergence_bits(const Dims& d, const Ucont& u,
                                                              const double* __restrict__ aj,
                                                              const double* __restrict__ nvert,
                                                              const uint8_t* __restrict__ nb8, double* sh) {
  unsigned long long mxv = 0ull;
  const size_t sy = d.mx, sz = (size_t)d.mx * d.my;
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    if (!in) continue;
    for (int i = 1 + _lane; i < d.mx - 1; i += 32) {
      const size_t c = o + i;
      const double v = (u.x[c] - u.x[c - 1] + u.y[c] - u.y[c - sy] + u.z[c] - u.z[c - sz]) * aj[c];
      if (!near_body(d, nvert, nb8, c)) max_abs(mxv, v);
    }
  }
  return block_maxbits(mxv, sh);
}
__global__ void __launch_bounds__(RB) k_divergence(Dims d, Ucont u, const double* __restrict__ aj,
                                                   const double* __restrict__ nvert, double* parts, double* out,
                                                   unsigned* ticket, const uint8_t* __restrict__ nb8) {
  __shared__ double sh[32];
  const unsigned long long mxv = divergence_bits(d, u, aj, nvert, nb8, sh);
  if (threadIdx.x == 0) parts[blockIdx.x] = __longlong_as_double((long long)mxv);
  if (!last_block(ticket)) return;
  const double m = finish_max(parts, sh);
  if (threadIdx.x == 0) *out = m;
}
int launch_divergence(const Dims& d, const Ucont& u, const double* aj, const double* nvert, double* parts, double* out,
                      unsigned* ticket, cudaStream_t s, const uint8_t* nb8) {
  k_divergence<<<row_blocks(d), RB, 0, s>>>(d, u, aj, nvert, parts, out, ticket, nb8); ++g_launches;
  return (int)cudaGetLastError();
}

// ||r|| over the array and max |r| over the cells the Divergence check keeps
// (main.c:1279-1349: the cell and its six face neighbours free of nvert): with
// st = 1 the projection leaves div u = dt / coeff * r there for the aj-scaled
// residual r (whose ghosts are zero).
__global__ void __launch_bounds__(RB) k_norm_absmax(Dims d, const double* __restrict__ r, const double* __restrict__ nvert,
                                                    double* parts, double* out, unsigned* ticket,
                                                    const uint8_t* __restrict__ nb8) {
  __shared__ double sh[32];
  unsigned long long mxv = 0ull;
  double s = 0.;
  ROW_LOOP(d) {
    ROW_DECOMP(d, j, k, o, in);
    if (!in) continue;
    for (int i = 1 + _lane; i < d.mx - 1; i += 32) {
      const double v = r[o + i];
      s = fma(v, v, s);
      if (!near_body(d, nvert, nb8, o + i)) max_abs(mxv, v);
    }
  }
  s = block_sum(s, sh);
  mxv = block_maxbits(mxv, sh);
  if (threadIdx.x == 0) {
    parts[gridDim.x + blockIdx.x] = s;
    parts[blockIdx.x] = __longlong_as_double((long long)mxv);
  }
  if (!last_block(ticket)) return;
  const double m = finish_max(parts, sh);
  finish_sums<1>(parts + gridDim.x, out, sh);
  if (threadIdx.x == 0) {
    out[0] = sqrt(out[0]);
    out[1] = m;
  }
}
int launch_norm_absmax(const Dims& d, const double* r, const double* nvert, double* parts, double* out, unsigned* ticket,
                       cudaStream_t s, const uint8_t* nb8) {
  k_norm_absmax<<<row_blocks(d), RB, 0, s>>>(d, r, nvert, parts, out, ticket, nb8); ++g_launches;
  return (int)cudaGetLastError();
}

// ---- allocation-free divergence check ----
// The blocks' maxima meet in *out itself, cleared on the stream before the
// launch: the bits of |v| order like the values, and a maximum does not depend
// on the order of its blocks.  No scratch and no state outlive a call, so calls
// on different streams or threads (with an *out each) have nothing to share.
__global__ void __launch_bounds__(RB) k_divergence_into(Dims d, Ucont u, const double* __restrict__ aj,
                                                        const double* __restrict__ nvert, unsigned long long* out) {
  __shared__ double sh[32];
  const unsigned long long mxv = divergence_bits(d, u, aj, nvert, nullptr, sh);
  if (threadIdx.x == 0) atomicMax(out, mxv);
}

int divergence_max_noalloc(int device, const Dims& d, const Ucont& u, const double* aj, const double* nvert, double* out,
                           cudaStream_t s, const char** why) {
  constexpr int MAXDEV = 64;
  if (device < 0 || device >= MAXDEV) {
    *why = "device index out of range";
    return 1;
  }
  int cur = -1;
  cudaError_t e = cudaGetDevice(&cur);
  if (e == cudaSuccess && cur != device) {
    *why = "the device argument must be the calling thread's current device";
    return 1;
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(out, 0, sizeof(double), s);
  if (e == cudaSuccess) {
    k_divergence_into<<<row_blocks(d), RB, 0, s>>>(d, u, aj, nvert, (unsigned long long*)out); ++g_launches;
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    *why = cudaGetErrorString(e);
    return 2;
  }
  return 0;
}

}  // namespace vfs
