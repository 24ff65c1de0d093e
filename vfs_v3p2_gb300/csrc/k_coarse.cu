// The V-cycle below (and including) a small level in one launch.
//
// What bounds it: latency.  Run one kernel per operation, a level of 32^3
// cells or fewer takes 3 to 4 us per sweep, restriction or prolongation in a
// captured iteration whatever its size (launch, one round of dependent loads
// from L2, the column solves, the drain), 17 such launches for three levels.
// Here one cluster of up to 16 blocks keeps x, the line arrays and the coarse
// right-hand sides in shared memory for the whole descent and ascent; a
// cluster barrier (and the boundary k planes written straight into the
// neighbour blocks' halo planes) separates the operations instead of a
// launch.  A thread keeps its cells' share of the operator in registers over
// a level's sweeps.
//
// Split: block r of the cluster owns k planes 1 + r c .. of every level (c
// planes each), so a sweep needs only the planes next to its slab from other
// blocks, and the y lines and i rows stay inside a block.  The coarsest
// level's packed right-hand side and solution are kept whole in every block
// (at most 2048 values), its matrix rows are spread over the cluster's warps.
//
// Per cell the arithmetic and its order are the stand-alone kernels'
// (face_row, line_solve, resrestrict_tile, prolong_tile, gemv_tile), so the
// result is theirs bit for bit.
#include "mg_coarse.h"
#include "mg_tiles.cuh"
#include "vfs_common.cuh"

namespace vfs {

// Values between two columns of the line arrays: twice an odd number.
__host__ __device__ inline int cv_line_pitch(int nj) {
  const int p = (nj + 1) & ~1;
  return p % 4 == 0 ? p + 2 : p;
}

namespace {

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Shared-memory address of a local variable, and the same place in block r.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned remote(unsigned a, unsigned r) {
  unsigned o;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(r));
  return o;
}
__device__ __forceinline__ void st_remote(unsigned a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ float ld_remote(unsigned a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// The 128-byte lines of p .. p + bytes into L2, one a lane (whole warps; every
// line starts inside the range).
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes) {
  for (unsigned o = (threadIdx.x & 31u) * 128u; o < bytes; o += 32u * 128u)
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)p + o));
}

// One level as its block sees it.
struct Slab {
  int mx, ni, nj, nk, P, pc;  // P, pc: cells of a ghosted and of a packed k plane
  int lp;                     // pitch of a column in the line arrays
  int c, k0, cown, n;         // planes per block, first own plane, own planes and cells (0: none)
  int up, dn;                 // blocks that hold the planes after and before the slab (-1: none)
};
__device__ __forceinline__ Slab slab_of(const CvLevel& L, int rank) {
  Slab s;
  s.mx = L.d.mx;
  s.ni = L.d.mx - 2;
  s.nj = L.d.my - 2;
  s.nk = L.d.mz - 2;
  s.P = L.d.mx * L.d.my;
  s.pc = s.ni * s.nj;
  s.lp = cv_line_pitch(s.nj);
  s.c = L.c;
  s.k0 = 1 + rank * L.c;
  s.cown = max(0, min(L.c, s.nk - rank * L.c));
  s.n = s.cown * s.pc;
  const int last = (s.nk - 1) / L.c;  // last block with planes
  s.up = rank < last ? rank + 1 : (L.d.kp ? 0 : -1);
  s.dn = rank > 0 ? rank - 1 : (L.d.kp ? last : -1);
  return s;
}

// line_solve for a column stored contiguously (lp values apart from the
// next): pairs of rows move as 8-byte words at constant offsets, 20
// instructions per 8 rows where a column strided by a run-time pitch takes 56
// (one warp solves a block's columns while the others wait, so its issue is
// the time).  A pitch of twice an odd number keeps a warp's 8-byte accesses
// free of bank conflicts.  Row by row the arithmetic is line_solve's.
__device__ __forceinline__ void line_solve_packed(float* su, const float* sp, const float* sl, int nj) {
  constexpr int B = 8;
  float y = 0.f;
  int j = 0;
  for (; j + B <= nj; j += B) {
    float2 a[B / 2], r[B / 2];
#pragma unroll
    for (int u = 0; u < B / 2; u++) {
      a[u] = *(const float2*)(sp + j + 2 * u);
      r[u] = *(const float2*)(su + j + 2 * u);
    }
#pragma unroll
    for (int u = 0; u < B / 2; u++) {
      r[u].x = y = fmaf(-a[u].x, y, r[u].x);
      r[u].y = y = fmaf(-a[u].y, y, r[u].y);
      *(float2*)(su + j + 2 * u) = r[u];
    }
  }
  for (; j < nj; j++) su[j] = y = fmaf(-sp[j], y, su[j]);
  float xn = 0.f;
  for (j = nj; j % B != 0; j--) su[j - 1] = xn = fmaf(-sl[j - 1], xn, su[j - 1]);
  for (; j > 0; j -= B) {
    float2 c[B / 2], r[B / 2];
#pragma unroll
    for (int u = 0; u < B / 2; u++) {
      c[u] = *(const float2*)(sl + j - 2 - 2 * u);
      r[u] = *(const float2*)(su + j - 2 - 2 * u);
    }
#pragma unroll
    for (int u = 0; u < B / 2; u++) {
      r[u].y = xn = fmaf(-c[u].y, xn, r[u].y);
      r[u].x = xn = fmaf(-c[u].x, xn, r[u].x);
      *(float2*)(su + j - 2 - 2 * u) = r[u];
    }
  }
}

// The thread's cells of a level (packed index threadIdx.x + q CV_NT of the
// slab) with their share of the operator in registers: the sweeps then read
// x alone, 11 shared-memory loads a cell.
template <int Q>
struct Cells {
  float2 fic[Q], fiw[Q], fkc[Q], fkb[Q];  // FaceData's weights
  float gjc[Q], gjs[Q], aj[Q], inv[Q], b[Q];
  unsigned code[Q];   // its code bits: c, c-i << 4, c-k << 8
  int xo[Q];          // in a ghosted buffer of the slab (halo plane first)
  int so[Q];          // in the line arrays
  short oe[Q], ow[Q], on[Q], os[Q];  // x offsets of the i and j neighbours, periodic seams folded in
};
template <int Q>
__device__ __forceinline__ void load_cells(const CvLevel& L, const Slab& s, const float* __restrict__ b,
                                           const float* sb, Cells<Q>& C) {
  const Dims& d = L.d;
#pragma unroll
  for (int q = 0; q < Q; q++) {
    // a thread without a q-th cell reads the block's first one and drops it
    const int idx = threadIdx.x + q * CV_NT, id = idx < s.n ? idx : 0;
    const int kk = id / s.pc, t = id - kk * s.pc, jl = t / s.ni;
    const int i = 1 + t - jl * s.ni, j = 1 + jl, k = min(s.k0 + kk, s.nk);
    const int lc = j * s.mx + i, gc = k * s.P + lc;
    const int oiW = (i == 1 && d.ip) ? d.mx - 3 : -1;
    const int ojS = ((j == 1 && d.jp) ? d.my - 3 : -1) * s.mx;
    const int okB = (k == 1 && d.kp) ? (d.mz - 3) * s.P : -s.P;
    C.xo[q] = (kk + 1) * s.P + lc;
    C.so[q] = (kk * s.ni + i - 1) * s.lp + jl;
    C.oe[q] = (short)((i == d.mx - 2 && d.ip) ? 3 - d.mx : 1);
    C.ow[q] = (short)oiW;
    C.on[q] = (short)(((j == d.my - 2 && d.jp) ? 3 - d.my : 1) * s.mx);
    C.os[q] = (short)ojS;
    C.fic[q] = __ldg(L.ffi + gc);
    C.fiw[q] = __ldg(L.ffi + gc + oiW);
    C.fkc[q] = __ldg(L.ffk + gc);
    C.fkb[q] = __ldg(L.ffk + gc + okB);
    C.gjc[q] = __ldg(L.ffj + gc);
    C.gjs[q] = __ldg(L.ffj + gc + ojS);
    const float ajc = __ldg(L.faj + gc), ajw = __ldg(L.faj + gc + oiW), ajb = __ldg(L.faj + gc + okB);
    C.inv[q] = __ldg(L.lf + gc);
    C.b[q] = b ? __ldg(b + gc) : sb[id];
    C.aj[q] = face_aj(ajc);
    C.code[q] = face_code(ajc) | face_code(ajw) << 4 | face_code(ajb) << 8;
  }
}

// b - A x of the thread's q-th cell.
template <int Q>
__device__ __forceinline__ float cell_residual(const Slab& s, const Cells<Q>& C, const float* x, int q) {
  const float* p = x + C.xo[q];
  const float *pt = p + s.P, *pb = p - s.P;
  const int e = C.oe[q], w = C.ow[q];
  float xv[19];
  xv[CP] = p[0];
  xv[EP] = p[e];
  xv[WP] = p[w];
  xv[NP] = p[C.on[q]];
  xv[SP] = p[C.os[q]];
  xv[TP] = pt[0];
  xv[TE] = pt[e];
  xv[TW] = pt[w];
  xv[BP] = pb[0];
  xv[BE] = pb[e];
  xv[BW] = pb[w];
  const FaceData f{C.fic[q], C.fiw[q], C.fkc[q], C.fkb[q], C.gjc[q], C.gjs[q], C.aj[q], C.code[q], C.code[q] >> 4,
                   C.code[q] >> 8};
  return C.b[q] - face_row(f, xv);
}

// x of own cell (plane kk) at offset xo into the block's buffer x and the
// halo planes of the blocks beside it.
__device__ __forceinline__ void put_x(const Slab& s, float* x, int xo, float v) {
  x[xo] = v;
  if (xo < 2 * s.P && s.dn >= 0) {
    const int cd = min(s.c, s.nk - s.dn * s.c);  // planes of the block before
    st_remote(remote(smem_addr(x + cd * s.P + xo), s.dn), v);
  }
  if (xo >= s.cown * s.P && s.up >= 0) st_remote(remote(smem_addr(x + xo - s.cown * s.P), s.up), v);
}

// One sweep: x_new = x_old + omega delta from buffer `from` (null: a zero
// guess, whose residual is b) into `to`, or into global memory when out is
// set.
template <int Q>
__device__ __forceinline__ void sweep(const CvLevel& L, const Slab& s, const Cells<Q>& C, float* sm, const float* from,
                                      float* to, float omega, float* __restrict__ out) {
  float* su = sm + L.osu;
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const int idx = threadIdx.x + q * CV_NT;
    if (idx >= s.n) break;
    const float r = from ? cell_residual(s, C, from, q) : C.b[q];
    su[C.so[q]] = C.aj[q] != 0.f ? r * C.inv[q] : 0.f;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < s.ni * s.cown; t += CV_NT)
    line_solve_packed(su + t * s.lp, sm + L.osp + t * s.lp, sm + L.osl + t * s.lp, s.nj);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const int idx = threadIdx.x + q * CV_NT;
    if (idx >= s.n) break;
    const float v = fmaf(omega, su[C.so[q]], from ? from[C.xo[q]] : 0.f);
    if (out) out[(s.k0 - 1) * s.P + C.xo[q]] = v;
    else put_x(s, to, C.xo[q], v);
  }
  cluster_sync_all();
}

// One visit of level l.  Down: line couplings, pre-sweeps, residual
// restriction into the next coarser level's right-hand side.  Up: prolongation
// from it, post-sweeps.  (One body for both, so that the sweep's code is in
// the kernel once per instantiation: the launch runs through its
// instructions a few times only.)
template <int Q>
__device__ __forceinline__ void visit(const CvArgs& a, int l, bool up, int rank, float* sm) {
  const CvLevel& L = a.lev[l];
  const CvLevel& K = a.lev[l - 1];
  const Slab s = slab_of(L, rank);
  float* su = sm + L.osu;
  Cells<Q> C;
  load_cells<Q>(L, s, l == a.top ? a.b : nullptr, sm + L.ob, C);
  int cur = up ? (L.npre - 1) & 1 : 1;
  if (!up) {
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int idx = threadIdx.x + q * CV_NT;
      if (idx >= s.n) break;
      const int jl = (idx % s.pc) / s.ni;
      const bool live = C.aj[q] != 0.f;
      const float lo = jl > 0 ? C.aj[q] * C.gjs[q] : 0.f, hi = jl < s.nj - 1 ? C.aj[q] * C.gjc[q] : 0.f;
      sm[L.osp + C.so[q]] = live ? lo * C.inv[q] : 0.f;
      sm[L.osl + C.so[q]] = live ? hi * C.inv[q] : 0.f;
    }
  } else {
    float* xf = sm + L.ox[cur];
    const int cmx = K.d.mx, cP = K.d.mx * K.d.my, cnk = K.d.mz - 2;
    // the coarse solution: level 0 whole in this block, else the buffer its post-sweeps ended in
    const unsigned xc = smem_addr(sm + (l > 1 ? K.ox[(K.npre - 1 + K.npost) & 1] : a.ox0));
#pragma unroll 1
    for (int idx = threadIdx.x; idx < s.n; idx += CV_NT) {
      const int kk = idx / s.pc, t = idx - kk * s.pc, jl = t / s.ni;
      const int i = 1 + t - jl * s.ni, j = 1 + jl, k = s.k0 + kk;
      const int ic = (i + 1) / 2, jc = (j + 1) / 2, kc = (k + 1) / 2;
      const int xo = (kk + 1) * s.P + j * s.mx + i;
      const unsigned cd = __ldg(L.pcode + (s.k0 - 1) * s.P + xo);
      const int ia = (int)(cd & 3) - 1, ja = (int)((cd >> 2) & 3) - 1, ka = (int)((cd >> 4) & 3) - 1;
      // (jc, ic) of coarse plane z: level 0 in this block, another level's in the block that owns it
      auto plane = [&](int z) -> unsigned {
        const unsigned o = 4u * (unsigned)(jc * cmx + ic);
        if (l == 1) return remote(xc + 4u * (unsigned)(z * cP) + o, rank);
        const int r = (z - 1) / K.c;
        return remote(xc + 4u * (unsigned)((z - r * K.c) * cP) + o, r);
      };
      const bool in = l == 1 || (kc + ka >= 1 && kc + ka <= cnk);  // ghost planes hold zeros
      const unsigned p0 = plane(kc), p1 = plane(in ? kc + ka : kc);
      const unsigned di = 4u * (unsigned)ia, dj = 4u * (unsigned)(ja * cmx);
      float v1 = ld_remote(p1), vj1 = ld_remote(p1 + dj), vi1 = ld_remote(p1 + di), vij1 = ld_remote(p1 + dj + di);
      if (!in) v1 = vj1 = vi1 = vij1 = 0.f;
      const float v = prolong_value<float>(ld_remote(p0), ld_remote(p0 + dj), ld_remote(p0 + di), ld_remote(p0 + dj + di),
                                           v1, vj1, vi1, vij1);
      put_x(s, xf, xo, xf[xo] + ((cd & 0x80u) ? 0.f : v));
    }
    cluster_sync_all();
  }
  const float* w = (up ? a.wpost : a.wpre)[l == a.top ? a.topset : 0];
  const int n = up ? L.npost : L.npre;
#pragma unroll 1
  for (int q = 0; q < n; q++, cur ^= 1)
    sweep<Q>(L, s, C, sm, up || q > 0 ? sm + L.ox[cur] : nullptr, sm + L.ox[cur ^ 1], w[q],
             (up && l == a.top && q == n - 1) ? a.x : nullptr);
  if (up) return;
  // weighted residual in su
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const int idx = threadIdx.x + q * CV_NT;
    if (idx >= s.n) break;
    const float ww = __ldg(L.rw + (s.k0 - 1) * s.P + C.xo[q]);
    const float rr = cell_residual(s, C, sm + L.ox[cur], q) * ww;
    su[C.so[q]] = ww != 0.f ? rr : 0.f;
  }
  cluster_sync_all();
  // the children's sums where the coarse cells live (at most one a thread: a
  // coarse slab is a quarter of the fine one)
  const bool last = l == 1;
  const int ci = K.d.mx - 2, cj = K.d.my - 2;
  const Slab cs = slab_of(K, rank);
  const int tc = last ? threadIdx.x * a.cl + rank : threadIdx.x;
  if (tc < (last ? a.n0 : cs.n)) {
    const int kk = tc / (ci * cj), u = tc - kk * (ci * cj), J = 1 + u / ci, I = 1 + u - (J - 1) * ci;
    const int kc = last ? 1 + kk : cs.k0 + kk;
    float acc = 0.f;
    if (!(__ldg(K.nvert + (size_t)kc * K.d.mx * K.d.my + J * K.d.mx + I) > 0.1)) {
      const unsigned su0 = smem_addr(su);
      // fine planes 2 kc - 1 (p0) and 2 kc (p1); the upper child's place in the line arrays
      const int q0 = 2 * kc - 2, r0 = q0 / s.c, r1 = (q0 + 1) / s.c;
      const int h = (2 * I - 1) * s.lp + 2 * J - 1, lpl = s.ni * s.lp;
      const unsigned p0 = remote(su0 + 4u * (unsigned)((q0 - r0 * s.c) * lpl + h), r0);
      const unsigned p1 = remote(su0 + 4u * (unsigned)((q0 + 1 - r1 * s.c) * lpl + h), r1);
      const unsigned di = 4u * (unsigned)s.lp;
      const float s111 = ld_remote(p1), s110 = ld_remote(p1 - di), s101 = ld_remote(p1 - 4u), s100 = ld_remote(p1 - 4u - di);
      const float s011 = ld_remote(p0), s010 = ld_remote(p0 - di), s001 = ld_remote(p0 - 4u), s000 = ld_remote(p0 - 4u - di);
      // MyRestriction's order
      acc = (s111 + s110 + s101 + s011 + s100 + s001 + s010 + s000) * 0.125f;
    }
    // level 0's go through global memory (L2): every block needs all of them
    if (!last) sm[K.ob + tc] = acc;
    else __stcg(a.b0 + tc, acc);
  }
  if (last) {
    cluster_sync_all();
    for (int t = threadIdx.x; t < a.n0; t += CV_NT) sm[a.osb + t] = __ldcg(a.b0 + t);
  }
  __syncthreads();
}

// The instantiation a level's slab needs (cells a thread owns).
__device__ __forceinline__ void run_level(const CvArgs& a, int l, bool up, int rank, float* sm) {
  if (a.lev[l].c * (a.lev[l].d.mx - 2) * (a.lev[l].d.my - 2) <= CV_NT) visit<1>(a, l, up, rank, sm);
  else visit<CV_Q>(a, l, up, rank, sm);
}

}  // namespace

__global__ void __launch_bounds__(CV_NT, 1) k_coarse_vcycle(const __grid_constant__ CvArgs a) {
  if (skipped(a.skip)) return;  // the same in every block: no barrier is left waiting
  extern __shared__ __align__(16) float sm[];
  const int rank = (int)cluster_rank(), cl = a.cl;
  for (int t = threadIdx.x; t < a.nfloats / 4; t += CV_NT) reinterpret_cast<float4*>(sm)[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  // this block's rows of the dense inverse and its planes of the levels below
  // the top, on their way into L2 during the first sweeps: on a large grid
  // everything has left it since the last V-cycle
  {
    const int nw = CV_NT / 32;
    for (int r = threadIdx.x >> 5; r * cl + rank < a.n0; r += nw) prefetch_l2(a.Binv + (size_t)(r * cl + rank) * a.n0, a.n0 * 4u);
    for (int l = a.top - 1; l >= 1; l--) {
      const CvLevel& L = a.lev[l];
      const Slab s = slab_of(L, rank);
      if (s.cown == 0) continue;
      const size_t o = (size_t)s.k0 * s.P;
      const unsigned n = s.cown * s.P;
      const int w = threadIdx.x >> 5;
      if (w == 0) prefetch_l2(L.ffi + o, n * 8u);
      if (w == 1) prefetch_l2(L.ffk + o, n * 8u);
      if (w == 2) prefetch_l2(L.ffj + o, n * 4u);
      if (w == 3) prefetch_l2(L.faj + o, n * 4u);
      if (w == 4) prefetch_l2(L.lf + o, n * 4u);
      if (w == 5) prefetch_l2(L.rw + o, n * 4u);
      if (w == 6) prefetch_l2(L.pcode + o, n);
    }
  }
  // no block writes into another's shared memory before that one has cleared it
  cluster_sync_all();
  for (int v = 0; v <= 2 * a.top; v++) {  // down from the top, the coarsest level, up again
    if (v != a.top) {
      run_level(a, v < a.top ? a.top - v : v - a.top, v > a.top, rank, sm);
      continue;
    }
    // coarsest level: x = Binv b, a warp per row, the value sent to every block
    const CvLevel& C = a.lev[0];
    const int ci = C.d.mx - 2, cj = C.d.my - 2, n = a.n0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* sb = sm + a.osb;
    const unsigned x0 = smem_addr(sm + a.ox0);
    // R rows of a warp at a time, so that their loads are in flight together
    constexpr int R = 4;
    const int step = cl * (CV_NT / 32);
    for (int row0 = warp * cl + rank; row0 < n; row0 += R * step) {
      const float* Br[R];
      float v[R];
#pragma unroll
      for (int u = 0; u < R; u++) {
        Br[u] = a.Binv + (size_t)min(row0 + u * step, n - 1) * n;
        v[u] = 0.f;
      }
      if (n % 4 == 0) {
        const float4* sv = reinterpret_cast<const float4*>(sb);
#pragma unroll 2
        for (int q = lane; q < n / 4; q += 32) {
          const float4 y = sv[q];
          float4 m[R];
#pragma unroll
          for (int u = 0; u < R; u++) m[u] = __ldg(reinterpret_cast<const float4*>(Br[u]) + q);
#pragma unroll
          for (int u = 0; u < R; u++) {
            v[u] = fma(m[u].x, y.x, v[u]);
            v[u] = fma(m[u].y, y.y, v[u]);
            v[u] = fma(m[u].z, y.z, v[u]);
            v[u] = fma(m[u].w, y.w, v[u]);
          }
        }
      } else {
#pragma unroll 4
        for (int col = lane; col < n; col += 32) {
          const float y = sb[col];
#pragma unroll
          for (int u = 0; u < R; u++) v[u] = fma(__ldg(Br[u] + col), y, v[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < R; u++) {
        const float t = __shfl_sync(0xffffffffu, warp_sum(v[u]), 0);
        const int row = row0 + u * step;
        const int I = 1 + row % ci, J = 1 + (row / ci) % cj, K = 1 + row / (ci * cj);
        if (row < n && lane < cl) st_remote(remote(x0 + 4u * (unsigned)cidx(C.d, I, J, K), lane), t);
      }
    }
    cluster_sync_all();
  }
}

bool cv_layout(CvArgs& a, int cl) {
  a.cl = cl;
  size_t o = 0;
  a.osb = 0;
  o += ((size_t)a.n0 + 3) & ~(size_t)3;
  a.ox0 = (int)o;
  o += ncell(a.lev[0].d);
  for (int l = 0; l <= a.top; l++) {
    CvLevel& L = a.lev[l];
    const size_t nk = L.d.mz - 2, P = (size_t)L.d.mx * L.d.my, pc = (size_t)(L.d.mx - 2) * (L.d.my - 2);
    const size_t ln = (size_t)(L.d.mx - 2) * cv_line_pitch(L.d.my - 2);
    L.c = (int)((nk + cl - 1) / cl);
    if (l == 0) continue;
    for (int q = 0; q < 2; q++) {
      L.ox[q] = (int)o;
      o += (L.c + 2) * P;
    }
    o = (o + 1) & ~(size_t)1;  // the line arrays move in 8-byte words
    for (int* p : {&L.osu, &L.osp, &L.osl}) {
      *p = (int)o;
      o += L.c * ln;
    }
    L.ob = (int)o;
    if (l < a.top) o += L.c * pc;
    // a thread's cells of the level and its one cell of the level below
    const size_t cc = l > 1 ? (size_t)a.lev[l - 1].c * (a.lev[l - 1].d.mx - 2) * (a.lev[l - 1].d.my - 2) : 0;
    if (L.c * pc > (size_t)CV_NT * CV_Q || cc > CV_NT || (size_t)a.n0 > (size_t)cl * CV_NT || P > 16383 || o * sizeof(float) > CV_SMEM_MAX) return false;
  }
  a.nfloats = (int)((o + 3) & ~(size_t)3);
  return true;
}

static cudaLaunchConfig_t cv_config(const CvArgs& a, cudaStream_t s, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.cl);
  cfg.blockDim = dim3(CV_NT);
  cfg.dynamicSmemBytes = (size_t)a.nfloats * sizeof(float);
  cfg.stream = s;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = a.cl;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

int cv_cluster(CvArgs& a) {
  // both attributes cost nothing once set
  if (cudaFuncSetAttribute(k_coarse_vcycle, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CV_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(k_coarse_vcycle, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int cl : {CV_MAXBLOCKS, 8}) {
    if (!cv_layout(a, cl)) continue;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = cv_config(a, nullptr, &attr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_coarse_vcycle, &cfg) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (n > 0) return cl;
  }
  return 0;
}

int launch_coarse_vcycle(const CvArgs& a, cudaStream_t s) {
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = cv_config(a, s, &attr);
  ++g_launches;
  return (int)cudaLaunchKernelEx(&cfg, k_coarse_vcycle, a);
}

}  // namespace vfs
