// FP64 ground-state kernels: the one-by-one Gram-Schmidt, the band-by-band CG of
// the reference, and the Hermitian eigen-decomposition of the subspace
// diagonalisation (its products and the blocked Gram-Schmidt are in k_zgemm.cu).
// Every reduction is a fixed-order sum (deterministic).  Arrays:
// zu_GS(NL,NB,NK_s:NK_e) complex(8).
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include <algorithm>

#include "sgpu_internal.cuh"

namespace sgpu {

constexpr int GS_THREADS = 512;

// ------------------------------------------------------------------ groups --
// The CG and one-by-one Gram-Schmidt kernels run one thread-block cluster per
// k-point: the cluster's C CTAs split the NL points into contiguous slices, and
// every inner product is a fixed-order CTA sum followed by a sum of the C partials
// in rank order, read from each CTA's shared memory over the cluster (distributed
// shared memory); all CTAs of the cluster obtain the same value.  C = 1 is one CTA
// per k-point.
namespace cgx = cooperative_groups;

constexpr int GRP_NV = 8;    // values of one sum

struct GrpShared {
  double sh[32 * GRP_NV];
  double part[2][GRP_NV];    // this CTA's partial sums (double-buffered)
  double tot[GRP_NV];
  double2 dots[2][CGB];      // this CTA's inner products with the lower bands (double-buffered)
  double2 pdots[GS_THREADS / 32][4];  // a warp's share of four of them
  double2 d[CGB], c[CGB];
};

struct Grp {
  int k, rank, C, lo, hi;
  int parity, dparity;
  GrpShared* s;
};

__device__ __forceinline__ Grp grp_make(int NL, GrpShared* s) {
  cgx::cluster_group cl = cgx::this_cluster();
  Grp g;
  g.C = (int)cl.num_blocks();
  g.rank = (int)cl.block_rank();
  g.k = blockIdx.x / g.C;
  const int slice = (NL + g.C - 1) / g.C;
  g.lo = min(NL, g.rank * slice);
  g.hi = min(NL, g.lo + slice);
  g.parity = 0;
  g.dparity = 0;
  g.s = s;
  return g;
}

// sum of NV doubles over the k-point's cluster, valid in every thread of every CTA
template <int NV>
__device__ __forceinline__ void grp_allsum(Grp& g, double (&v)[NV]) {
  static_assert(NV <= GRP_NV, "the exchange holds GRP_NV values");
  block_allsum<NV>(v, g.s->sh);
  if (g.C == 1) return;
  cgx::cluster_group cl = cgx::this_cluster();
  if (threadIdx.x == 0)
#pragma unroll
    for (int j = 0; j < NV; ++j) g.s->part[g.parity][j] = v[j];
  cl.sync();  // every CTA's partial is in place (and every read of this slot from two sums ago is done)
  if (threadIdx.x < NV) {
    double t = 0.0;
    for (int r = 0; r < g.C; ++r) t += cl.map_shared_rank(&g.s->part[g.parity][0], r)[threadIdx.x];
    g.s->tot[threadIdx.x] = t;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] = g.s->tot[j];
  g.parity ^= 1;
}

// before a CTA of a cluster leaves: no other CTA still reads its shared memory
__device__ __forceinline__ void grp_exit(const Grp& g) {
  if (g.C > 1) cgx::this_cluster().sync();
}

// acc += (Re, Im) conj(a) b
__device__ __forceinline__ void zdot_add(double& re, double& im, double2 a, double2 b) {
  re = fma(a.x, b.x, fma(a.y, b.y, re));
  im = fma(a.x, b.y, fma(-a.y, b.x, im));
}
__device__ __forceinline__ double rdot(double2 a, double2 b, double acc) { return fma(a.x, b.x, fma(a.y, b.y, acc)); }

// <a|b> over the NL points (the cluster's sum), valid in every thread
__device__ __forceinline__ double2 grp_zdot(Grp& g, const double2* __restrict__ a, const double2* __restrict__ b) {
  double v[2] = {0.0, 0.0};
  for (int i = g.lo + threadIdx.x; i < g.hi; i += blockDim.x) zdot_add(v[0], v[1], a[i], b[i]);
  grp_allsum<2>(g, v);
  return make_double2(v[0], v[1]);
}

__device__ __forceinline__ double grp_nrm2(Grp& g, const double2* __restrict__ a) {
  double v[1] = {0.0};
  for (int i = g.lo + threadIdx.x; i < g.hi; i += blockDim.x) v[0] = rdot(a[i], a[i], v[0]);
  grp_allsum<1>(g, v);
  return v[0];
}

#define GRP_FOR(i) for (int i = g.lo + threadIdx.x; i < g.hi; i += blockDim.x)

// ------------------------------------------------------------ Gram-Schmidt --
// Gram_Schmidt_ompk (GS/Gram_Schmidt.f90:32-55) as the reference does it, for the
// bands p0 .. p0+pb-1 of the k-points the blocked form refuses (bad[k], see
// k_zgemm.cu; the bands below p0 are already projected out): for each band, subtract
// the projections on the panel's lower bands one by one, then normalise.
__global__ void __launch_bounds__(GS_THREADS) k_gram_schmidt(double2* __restrict__ zu, int NB, int NL, double Hxyz,
                                                            int p0, int pb, const int* __restrict__ bad) {
  __shared__ GrpShared sm;
  Grp g = grp_make(NL, &sm);
  if (!bad[g.k]) return;  // the whole cluster
  double2* base = zu + ((size_t)g.k * NB + p0) * NL;
  for (int ib = 0; ib < pb; ++ib) {
    double2* u = base + (size_t)ib * NL;
    for (int ibt = 0; ibt < ib; ++ibt) {
      const double2* ut = base + (size_t)ibt * NL;
      const double2 d = grp_zdot(g, ut, u);
      const double2 zov = make_double2(d.x * Hxyz, d.y * Hxyz);
      GRP_FOR(i) u[i] = csub(u[i], cmul(ut[i], zov));
    }
    const double inv = 1.0 / sqrt(grp_nrm2(g, u) * Hxyz);
    GRP_FOR(i) u[i] = make_double2(u[i].x * inv, u[i].y * inv);
  }
  grp_exit(g);
}

// ---------------------------------------------------------------------- CG --
// CG_ompk with skip_gsortho='n' (GS/CG.f90:34-139), split into kernels around
// the H applications; one cluster per k-point works on band ib of its k-point.
// Work vectors W[which][k][NL]: each kind is a contiguous batch of one vector per
// k-point for the H application.  Every CTA reads the k-point's state at the start
// of a kernel; rank 0 writes it back only after a cluster-wide sum, i.e. after every
// CTA has read it.
//
// Projections on the lower bands.  The reference subtracts them one by one, each
// inner product taken with the vector as already updated: ib dependent sums.  In
// terms of the inner products with the original vector, d_j = <u_j|x>, those
// coefficients solve the unit triangular system
//     c_j = d_j - sum_{i<j} <u_j|u_i> c_i,    c = (I + L)^-1 d,
// (modified Gram-Schmidt in its inverse compact WY form: Swirydowicz, Langou,
// Ananthan, Yang and Thomas, Numer. Linear Algebra Appl. 28 (2021) e2343), so one
// exchange gives all of them and the result is the reference's up to rounding, also
// where the bands are not orthogonal to each other (they are not: the reference
// orthogonalises a new band with the real parts of its overlaps, CG.f90:45,70).
// (I + L)^-1 grows by one row per finished band: gs_M, and gs_MR for the real parts.
// Lower bands are taken in blocks of CGB, block after block, so one row holds the
// CGB columns of its own block.
// At 32^3, two k-points, 144 bands, TPA, 4 iterations, sgpu_cg and two Gram-Schmidt: 805 ms
// with dependent sums, now 106 ms.
enum { CG_XK = 0, CG_HXK, CG_TXK, CG_GK, CG_PK, CG_PKO, CG_HT, CG_TT, CG_HK, CG_NW };

struct CGState {
  double xkHxk, gkgk;
  int done, iters;
};

__device__ __forceinline__ double2* wv(double2* W, int nkl, int k, int which, int NL) {
  return W + ((size_t)which * nkl + k) * NL;
}

// everything the CG kernels of one handle share
struct CGArgs {
  double2* zu;       // [nkl][NB][NL]
  double2* W;        // [CG_NW][nkl][NL]
  CGState* st;       // [nkl]
  double2* M;        // [nkl][NB][CGB] rows of (I + L)^-1
  double* MR;        // [nkl][NB][CGB] the same for the real parts of the overlaps
  double* tband;     // [nkl] kinetic energy of xk
  int nkl, NB, NL;
  double Hxyz;
};

__device__ __forceinline__ double warp_sum_gs(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// c = (I + L)^-1 d for the n bands of one block, one warp per row.  row: row 0 of the
// block in gs_M / gs_MR.
template <bool REAL>
__device__ __forceinline__ void cg_solve(const double2* __restrict__ M, const double* __restrict__ MR, int n,
                                         const double2* d, double2* c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int j0 = warp; j0 < n; j0 += 4 * nw) {  // four rows of the warp at a time, their loads in flight together
    double2 v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = make_double2(0.0, 0.0);
    const int jl = min(n - 1, j0 + 3 * nw);
    for (int i = lane; i <= jl; i += 32) {
      const double2 di = d[i];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int j = j0 + r * nw;
        if (j < n && i <= j) {
          if (REAL) v[r].x = fma(MR[(size_t)j * CGB + i], di.x, v[r].x);
          else v[r] = cfma(M[(size_t)j * CGB + i], di, v[r]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      v[r].x = warp_sum_gs(v[r].x);
      if (!REAL) v[r].y = warp_sum_gs(v[r].y);
      if (lane == 0 && j0 + r * nw < n) c[j0 + r * nw] = v[r];
    }
  }
}

// x <- x - sum_j c_j u_j at one point
__device__ __forceinline__ double2 cg_subtract(double2 x, const double2* __restrict__ u, int NL, int n,
                                               const double2* c) {
  int j = 0;
  for (; j + 8 <= n; j += 8) {
    double2 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = u[(size_t)(j + q) * NL];
#pragma unroll
    for (int q = 0; q < 8; ++q) x = csub(x, cmul(c[j + q], v[q]));
  }
  for (; j < n; ++j) x = csub(x, cmul(c[j], u[(size_t)j * NL]));
  return x;
}

// the same at a thread's points of the CTA's slice, four points at a time (their loads are
// in flight together)
__device__ __forceinline__ void grp_subtract(const Grp& g, double2* x, const double2* __restrict__ u, int NL, int n,
                                             const double2* c) {
  int i = g.lo + threadIdx.x;
  const int nt = blockDim.x;
  for (; i + 3 * nt < g.hi; i += 4 * nt) {
    double2 v[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) v[p] = x[i + p * nt];
#pragma unroll 2
    for (int j = 0; j < n; ++j) {
      const double2 cj = c[j];
      const double2* uj = u + (size_t)j * NL + i;
#pragma unroll
      for (int p = 0; p < 4; ++p) v[p] = csub(v[p], cmul(cj, uj[p * nt]));
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) x[i + p * nt] = v[p];
  }
  for (; i < g.hi; i += nt) x[i] = cg_subtract(x[i], u + i, NL, n, c);
}

// Hxyz <u_j|x> for n bands u_j into s.d, over the cluster (ends with a CTA barrier).  A warp
// takes four bands (sharing the loads of x); with fewer groups of four than warps, the warps
// of one group split the slice.
__device__ __forceinline__ void grp_dots(Grp& g, const double2* __restrict__ u, int NL, int n, const double2* x,
                                         double Hxyz) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ng = (n + 3) / 4, parts = max(1, nw / max(1, ng));
  double2* loc = g.s->dots[g.dparity];
  __syncthreads();  // x is written by other threads of the CTA
  for (int g0 = 0; g0 < ng; g0 += nw) {  // (parts > 1 only when one round takes all groups)
    const int gi = parts > 1 ? warp % ng : g0 + warp, part = parts > 1 ? warp / ng : 0;
    if (gi < ng && part < parts) {
      const double2* uj = u + (size_t)4 * gi * NL;
      const int nj = min(4, n - 4 * gi);
      double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
      for (int i = g.lo + lane + 32 * part; i < g.hi; i += 32 * parts) {
        const double2 xi = x[i];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < nj) zdot_add(v[2 * j], v[2 * j + 1], uj[(size_t)j * NL + i], xi);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = warp_sum_gs(v[j]) * Hxyz;
      if (lane == 0)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < nj) {
            if (parts > 1) g.s->pdots[warp][j] = make_double2(v[2 * j], v[2 * j + 1]);
            else loc[4 * gi + j] = make_double2(v[2 * j], v[2 * j + 1]);
          }
    }
  }
  if (parts > 1) {
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      double2 t = make_double2(0.0, 0.0);
      for (int p = 0; p < parts; ++p) t = cadd(t, g.s->pdots[p * ng + j / 4][j & 3]);
      loc[j] = t;
    }
  }
  if (g.C > 1) cgx::this_cluster().sync(); else __syncthreads();
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    double2 t = make_double2(0.0, 0.0);
    if (g.C > 1) {
      cgx::cluster_group cl = cgx::this_cluster();
      for (int r = 0; r < g.C; ++r) t = cadd(t, cl.map_shared_rank(loc, r)[j]);
    } else {
      t = loc[j];
    }
    g.s->d[j] = t;
  }
  __syncthreads();
  g.dparity ^= 1;
}

// x <- x minus its projections on the ib lower bands, taken one by one
template <bool REAL>
__device__ __forceinline__ void grp_project(Grp& g, const CGArgs& a, int ib, double2* x) {
  const double2* base = a.zu + (size_t)g.k * a.NB * a.NL;
  for (int b0 = 0; b0 < ib; b0 += CGB) {
    const int n = min(CGB, ib - b0);
    const double2* u = base + (size_t)b0 * a.NL;
    const size_t row = ((size_t)g.k * a.NB + b0) * CGB;
    grp_dots(g, u, a.NL, n, x, a.Hxyz);
    cg_solve<REAL>(a.M + row, a.MR + row, n, g.s->d, g.s->c);
    __syncthreads();
    grp_subtract(g, x, u, a.NL, n, g.s->c);
  }
}

// Row ib of (I + L)^-1 from the overlaps d_i = <u_i|u_ib> of the block's lower bands:
// m = -l (I + L)^-1 with l_i = <u_ib|u_i> = conj(d_i), and 1 on the diagonal.  n = ib's
// index in its block.
__device__ __forceinline__ void cg_new_row(double2* __restrict__ M, double* __restrict__ MR, int n, const double2* d) {
  __shared__ double3 ps[GS_THREADS];
  const int cols = (n + 32) / 32 * 32, parts = max(1, min(8, (int)blockDim.x / cols));  // parts of the sum per column
  const int t = threadIdx.x;
  for (int c0 = 0; c0 <= n; c0 += blockDim.x) {  // (one round wherever parts > 1)
    const int i = parts > 1 ? t % cols : c0 + t, part = parts > 1 ? t / cols : 0;
    double2 m = make_double2(0.0, 0.0);
    double mr = 0.0;
    if (i < n && part < parts) {
#pragma unroll 8
      for (int l = i + part; l < n; l += parts) {
        m = csub(m, cmul(make_double2(d[l].x, -d[l].y), M[(size_t)l * CGB + i]));
        mr = fma(-d[l].x, MR[(size_t)l * CGB + i], mr);
      }
    }
    if (parts > 1) {
      ps[t] = make_double3(m.x, m.y, mr);
      __syncthreads();
      if (part == 0)
        for (int p = 1; p < parts; ++p) {
          const double3 q = ps[p * cols + i];
          m = make_double2(m.x + q.x, m.y + q.y);
          mr += q.z;
        }
    }
    if (part == 0 && i <= n) {
      if (i == n) { m = make_double2(1.0, 0.0); mr = 1.0; }
      M[(size_t)n * CGB + i] = m;
      MR[(size_t)n * CGB + i] = mr;
    }
  }
}

// gk = hxk - xkHxk xk (xkHxk = the new Rayleigh quotient); with pre: hk's start and T_band
// are left to cg_after_gradient, once gk is orthogonal to the lower bands
__device__ __forceinline__ void cg_gradient(Grp& g, const CGArgs& a, double e) {
  const double2 *xk = wv(a.W, a.nkl, g.k, CG_XK, a.NL), *hxk = wv(a.W, a.nkl, g.k, CG_HXK, a.NL);
  double2* gk = wv(a.W, a.nkl, g.k, CG_GK, a.NL);
  GRP_FOR(i) gk[i] = make_double2(hxk[i].x - e * xk[i].x, hxk[i].y - e * xk[i].y);
}

// Conjugate direction from hk (the gradient gk itself without a preconditioner, else
// K gk after its projections on the lower bands), pko = its normalised component
// orthogonal to xk (CG.f90:92-106; with a preconditioner Payne et al., Rev. Mod. Phys.
// 64, 1045 (1992), section V.B: hk orthogonal to xk too, beta = <gk|hk> / previous).
// One exchange for every inner product (linear in the old direction), one for the norm.
__device__ __forceinline__ void cg_direction(Grp& g, const CGArgs& a, bool pre, int iter, double gkgk_old) {
  double2 *xk = wv(a.W, a.nkl, g.k, CG_XK, a.NL), *gk = wv(a.W, a.nkl, g.k, CG_GK, a.NL);
  double2 *hk = pre ? wv(a.W, a.nkl, g.k, CG_HK, a.NL) : gk;
  double2 *pk = wv(a.W, a.nkl, g.k, CG_PK, a.NL), *pko = wv(a.W, a.nkl, g.k, CG_PKO, a.NL);
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // <x|h>, Re <g|h>, <g|x>, <x|p_old>, <x|x>
  GRP_FOR(i) {
    const double2 x = xk[i], h = hk[i];
    zdot_add(v[0], v[1], x, h);
    if (pre) {
      const double2 gg = gk[i];
      v[2] = rdot(gg, h, v[2]);
      zdot_add(v[3], v[4], gg, x);
      v[7] = rdot(x, x, v[7]);
    } else {
      v[2] = rdot(h, h, v[2]);
    }
    if (iter > 1) zdot_add(v[5], v[6], x, pk[i]);
  }
  grp_allsum<8>(g, v);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] *= a.Hxyz;
  double2 zs = make_double2(v[0], v[1]);     // <x|h>
  double2 zh = make_double2(0.0, 0.0);       // the part of x taken out of h
  double s = v[2];
  if (pre) {  // h <- h - x <x|h>, s = Re <g|h>
    zh = zs;
    s -= v[3] * zh.x - v[4] * zh.y;
    zs = make_double2(zs.x * (1.0 - v[7]), zs.y * (1.0 - v[7]));
  }
  const double uk = iter > 1 ? s / gkgk_old : 0.0;
  if (iter > 1) zs = make_double2(fma(uk, v[5], zs.x), fma(uk, v[6], zs.y));
  if (g.rank == 0 && threadIdx.x == 0) a.st[g.k].gkgk = s;
  double n2[1] = {0.0};
  GRP_FOR(i) {
    const double2 x = xk[i];
    double2 p = hk[i];
    if (pre) p = csub(p, cmul(x, zh));
    if (iter > 1) {
      const double2 o = pk[i];
      p = make_double2(fma(uk, o.x, p.x), fma(uk, o.y, p.y));
    }
    pk[i] = p;
    p = csub(p, cmul(x, zs));
    pko[i] = p;
    n2[0] = rdot(p, p, n2[0]);
  }
  grp_allsum<1>(g, n2);
  const double inv = 1.0 / sqrt(n2[0] * a.Hxyz);
  GRP_FOR(i) pko[i] = make_double2(pko[i].x * inv, pko[i].y * inv);
}

// hk starts as gk (the preconditioner works in place on it)
__device__ __forceinline__ void cg_copy_gradient(Grp& g, const CGArgs& a) {
  const double2* gk = wv(a.W, a.nkl, g.k, CG_GK, a.NL);
  double2* hk = wv(a.W, a.nkl, g.k, CG_HK, a.NL);
  GRP_FOR(i) hk[i] = gk[i];
}

// In the kernels below, proj: the projections on the lower bands run inside the
// cluster; otherwise they are the separate kernels of launch_cg_project (few
// k-points: the clusters alone would leave most SMs idle), and the kernel stops, or
// starts, where they come.

// The residual of the finished band ib-1, esp_var = sqrt(||H u - <u|H u> u||^2 Hxyz) occ
// (CG.f90:124-126), then band ib orthogonalised against the lower bands with REAL
// coefficients (s is real(8) in the reference, CG.f90:45,70) and normalised into xk.
__global__ void __launch_bounds__(GS_THREADS) k_cg_open(const CGArgs a, int ib, int proj,
                                                        const double* __restrict__ occ_gs,
                                                        double* __restrict__ esp_var, double* __restrict__ res,
                                                        int* __restrict__ iters) {
  __shared__ GrpShared sm;
  Grp g = grp_make(a.NL, &sm);
  double2* xk = wv(a.W, a.nkl, g.k, CG_XK, a.NL);
  if (ib > 0) {
    const double2 *u = xk, *ht = wv(a.W, a.nkl, g.k, CG_HT, a.NL);
    double e[1] = {0.0}, v[1] = {0.0};
    GRP_FOR(i) e[0] = rdot(u[i], ht[i], e[0]);
    grp_allsum<1>(g, e);
    e[0] *= a.Hxyz;
    GRP_FOR(i) {
      const double2 r = make_double2(ht[i].x - e[0] * u[i].x, ht[i].y - e[0] * u[i].y);
      v[0] = rdot(r, r, v[0]);
    }
    grp_allsum<1>(g, v);
    if (g.rank == 0 && threadIdx.x == 0) {
      const size_t o = (size_t)g.k * a.NB + ib - 1;
      esp_var[o] = sqrt(v[0] * a.Hxyz) * occ_gs[o];
      res[o] = sqrt(v[0] * a.Hxyz);  // the residual norm itself, for convergence tests
      iters[o] = a.st[g.k].iters;
    }
  }
  if (ib < a.NB) {
    double2* u = a.zu + ((size_t)g.k * a.NB + ib) * a.NL;
    if (proj) grp_project<true>(g, a, ib, u);
    const double inv = 1.0 / sqrt(grp_nrm2(g, u) * a.Hxyz);
    GRP_FOR(i) xk[i] = make_double2(u[i].x * inv, u[i].y * inv);
    if (g.rank == 0 && threadIdx.x == 0) { a.st[g.k].done = 0; a.st[g.k].iters = 0; }
  }
  grp_exit(g);
}

// After H xk: the Rayleigh quotient, the gradient and (without a preconditioner) the
// first direction (CG.f90:80-106).
__global__ void __launch_bounds__(GS_THREADS) k_cg_first(const CGArgs a, int ib, int proj, int pre) {
  __shared__ GrpShared sm;
  Grp g = grp_make(a.NL, &sm);
  const double2 *xk = wv(a.W, a.nkl, g.k, CG_XK, a.NL), *hxk = wv(a.W, a.nkl, g.k, CG_HXK, a.NL);
  const double2* txk = wv(a.W, a.nkl, g.k, CG_TXK, a.NL);
  double v[2] = {0.0, 0.0};
  GRP_FOR(i) {
    v[0] = rdot(xk[i], hxk[i], v[0]);
    if (pre) v[1] = rdot(xk[i], txk[i], v[1]);
  }
  grp_allsum<2>(g, v);
  const double e = v[0] * a.Hxyz;
  if (g.rank == 0 && threadIdx.x == 0) {
    a.st[g.k].xkHxk = e;
    if (pre) a.tband[g.k] = v[1] * a.Hxyz;
  }
  cg_gradient(g, a, e);
  if (proj) {
    grp_project<false>(g, a, ib, wv(a.W, a.nkl, g.k, CG_GK, a.NL));
    if (pre) cg_copy_gradient(g, a);
    else cg_direction(g, a, false, 1, 0.0);
  }
  grp_exit(g);
}

// The direction of iteration iter from the projected gradient (or, with a
// preconditioner, from hk).
__global__ void __launch_bounds__(GS_THREADS) k_cg_dir(const CGArgs a, int ib, int iter, int proj, int pre) {
  __shared__ GrpShared sm;
  Grp g = grp_make(a.NL, &sm);
  const CGState st0 = a.st[g.k];
  if (st0.done) return;  // uniform over the cluster, before any cluster-wide sum
  if (pre && proj) grp_project<false>(g, a, ib, wv(a.W, a.nkl, g.k, CG_HK, a.NL));
  cg_direction(g, a, pre, iter, st0.gkgk);
  grp_exit(g);
}

// 2x2 Rayleigh-Ritz in span{xk, pko} and the update (CG.f90:108-119); then, as long as
// iterations are left, the next gradient (and direction), else the finished band:
// zu(:,ib) = xk / |xk|, also left in xk for the residual, and its row of (I + L)^-1.
__global__ void __launch_bounds__(GS_THREADS) k_cg_step(const CGArgs a, int ib, int iter, int last, int proj, int pre,
                                                        double delta_cg) {
  __shared__ GrpShared sm;
  Grp g = grp_make(a.NL, &sm);
  const int k = g.k;
  const CGState st0 = a.st[k];
  double2 *xk = wv(a.W, a.nkl, k, CG_XK, a.NL), *hxk = wv(a.W, a.nkl, k, CG_HXK, a.NL);
  double2* txk = wv(a.W, a.nkl, k, CG_TXK, a.NL);
  bool done = st0.done != 0;
  if (!done) {
    const double2 *pko = wv(a.W, a.nkl, k, CG_PKO, a.NL), *ht = wv(a.W, a.nkl, k, CG_HT, a.NL);
    const double2* tt = wv(a.W, a.nkl, k, CG_TT, a.NL);
    const double xkHxk = st0.xkHxk;
    double v[3] = {0.0, 0.0, 0.0};
    GRP_FOR(i) {
      const double2 h = ht[i];
      zdot_add(v[0], v[1], xk[i], h);
      v[2] = rdot(pko[i], h, v[2]);
    }
    grp_allsum<3>(g, v);
    const double2 xkHpk = make_double2(v[0] * a.Hxyz, v[1] * a.Hxyz);
    const double pkHpk = v[2] * a.Hxyz;
    const double ev = 0.5 * ((xkHxk + pkHpk) - sqrt((xkHxk - pkHpk) * (xkHxk - pkHpk) +
                                                   4 * (xkHpk.x * xkHpk.x + xkHpk.y * xkHpk.y)));
    double2 cx = make_double2(xkHpk.x / (ev - xkHxk), xkHpk.y / (ev - xkHxk));
    const double cp = 1.0 / sqrt(1.0 + (cx.x * cx.x + cx.y * cx.y));
    cx = make_double2(cx.x * cp, cx.y * cp);
    if (g.rank == 0 && threadIdx.x == 0) a.st[k].iters = iter;
    if (fabs(ev - xkHxk) < delta_cg) {  // delta_cg = 1e-15 in the reference (CG.f90:42,114)
      done = true;
      if (g.rank == 0 && threadIdx.x == 0) a.st[k].done = 1;
    } else {
      double w[2] = {0.0, 0.0};
      GRP_FOR(i) {
        const double2 p = pko[i], h = ht[i], t = tt[i];
        const double2 x = cfma(cx, xk[i], make_double2(cp * p.x, cp * p.y));
        const double2 hx = cfma(cx, hxk[i], make_double2(cp * h.x, cp * h.y));
        const double2 tx = cfma(cx, txk[i], make_double2(cp * t.x, cp * t.y));
        xk[i] = x;
        hxk[i] = hx;
        txk[i] = tx;
        w[0] = rdot(x, hx, w[0]);
        w[1] = rdot(x, tx, w[1]);
      }
      if (!last) {
        grp_allsum<2>(g, w);
        const double e = w[0] * a.Hxyz;
        if (g.rank == 0 && threadIdx.x == 0) {
          a.st[k].xkHxk = e;
          if (pre) a.tband[k] = w[1] * a.Hxyz;
        }
        cg_gradient(g, a, e);
        if (proj) {
          grp_project<false>(g, a, ib, wv(a.W, a.nkl, k, CG_GK, a.NL));
          if (pre) cg_copy_gradient(g, a);
          else cg_direction(g, a, false, iter + 1, st0.gkgk);
        }
      }
    }
  }
  if (last) {
    double2* u = a.zu + ((size_t)k * a.NB + ib) * a.NL;
    const double inv = 1.0 / sqrt(grp_nrm2(g, xk) * a.Hxyz);
    GRP_FOR(i) {
      const double2 x = make_double2(xk[i].x * inv, xk[i].y * inv);
      u[i] = x;
      xk[i] = x;
    }
    if (proj) {
      const int b0 = ib / CGB * CGB;
      grp_dots(g, a.zu + ((size_t)k * a.NB + b0) * a.NL, a.NL, ib - b0, u, a.Hxyz);
      const size_t row = ((size_t)k * a.NB + b0) * CGB;
      if (g.rank == 0) cg_new_row(a.M + row, a.MR + row, ib - b0, g.s->d);
    }
  }
  grp_exit(g);
}

// ------------------------------------------- projections over the whole GPU --
// Few k-points: nkl clusters of at most 16 CTAs leave most SMs idle while they read
// the lower bands twice per projection.  Here the inner products run over (k-point,
// CG_DB bands, range of points) and the subtraction over (k-point, 256 points).
constexpr int CG_DB = 4;  // bands of a CTA, sharing the loads of x

__global__ void __launch_bounds__(256) k_cg_dots(const double2* __restrict__ zu, const double2* __restrict__ x,
                                                 size_t xstride, int b0, int n, int NB, int NL, int chunk,
                                                 const CGState* __restrict__ st, double2* __restrict__ part) {
  __shared__ double sh[32 * 2 * CG_DB];
  const int k = blockIdx.z, j0 = blockIdx.x * CG_DB, sp = blockIdx.y;
  if (st && st[k].done) return;
  const double2* u = zu + ((size_t)k * NB + b0 + j0) * NL;
  const double2* xk = x + k * xstride;
  const int nj = min(CG_DB, n - j0), i1 = min(NL, (sp + 1) * chunk);
  double v[2 * CG_DB];
#pragma unroll
  for (int j = 0; j < 2 * CG_DB; ++j) v[j] = 0.0;
#pragma unroll 2
  for (int i = sp * chunk + threadIdx.x; i < i1; i += 256) {
    const double2 xi = xk[i];
#pragma unroll
    for (int j = 0; j < CG_DB; ++j)
      if (j < nj) zdot_add(v[2 * j], v[2 * j + 1], u[(size_t)j * NL + i], xi);
  }
  block_allsum<2 * CG_DB>(v, sh);
  if (threadIdx.x == 0)
#pragma unroll
    for (int j = 0; j < CG_DB; ++j)
      if (j < nj) part[((size_t)k * gridDim.y + sp) * CGB + j0 + j] = make_double2(v[2 * j], v[2 * j + 1]);
}

// d_j = Hxyz sum over the ranges, in order
__device__ __forceinline__ void cg_sum_dots(const double2* __restrict__ part, int k, int nsplit, int n, double Hxyz,
                                            double2* d) {
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    double2 t = make_double2(0.0, 0.0);
    for (int sp = 0; sp < nsplit; ++sp) t = cadd(t, part[((size_t)k * nsplit + sp) * CGB + j]);
    d[j] = make_double2(t.x * Hxyz, t.y * Hxyz);
  }
}

template <bool REAL>
__global__ void __launch_bounds__(256) k_cg_subtract(const double2* __restrict__ zu, double2* __restrict__ x,
                                                     size_t xstride, double2* __restrict__ copy, int b0, int n, int NB,
                                                     int NL, double Hxyz, const double2* __restrict__ M,
                                                     const double* __restrict__ MR, const CGState* __restrict__ st,
                                                     const double2* __restrict__ part, int nsplit) {
  __shared__ double2 d[CGB], c[CGB];
  const int k = blockIdx.y;
  if (st && st[k].done) return;
  cg_sum_dots(part, k, nsplit, n, Hxyz, d);
  __syncthreads();
  const size_t row = ((size_t)k * NB + b0) * CGB;
  cg_solve<REAL>(M + row, MR + row, n, d, c);
  __syncthreads();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= NL) return;
  const double2 v = cg_subtract(x[k * xstride + i], zu + ((size_t)k * NB + b0) * NL + i, NL, n, c);
  x[k * xstride + i] = v;
  if (copy) copy[(size_t)k * NL + i] = v;
}

__global__ void __launch_bounds__(256) k_cg_row(double2* __restrict__ M, double* __restrict__ MR, int b0, int n, int NB,
                                                double Hxyz, const double2* __restrict__ part, int nsplit) {
  __shared__ double2 d[CGB];
  const int k = blockIdx.x;
  cg_sum_dots(part, k, nsplit, n, Hxyz, d);
  __syncthreads();
  const size_t row = ((size_t)k * NB + b0) * CGB;
  cg_new_row(M + row, MR + row, n, d);
}

// ------------------------------------------------------------------ launch --
// CTAs per k-point: enough clusters to cover the SMs about once (C <= 16, a
// power of two, slices of at least 1024 points); 16 needs the non-portable
// cluster size, else 8.
static int gs_cluster_size(const System& s) {
  int C = 1;
  while (C < 16 && s.nkl * C * 2 <= s.nsm && s.NL / (C * 2) >= 1024) C *= 2;
  return C;
}

template <typename Kern, typename... Args>
static cudaError_t launch_gs(const System& s, Kern kern, Args... args) {
  int C = gs_cluster_size(s);
  for (;;) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s.nkl * C);
    cfg.blockDim = dim3(GS_THREADS);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s.launch_stream();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaSuccess;
    if (C > 8) e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kern, args...);
    if (e == cudaSuccess || C <= 8) return e;
    (void)cudaGetLastError();  // the non-portable size was refused: clear it and use 8
    --s.launches;
    C = 8;
  }
}

cudaError_t launch_gram_schmidt_panel(const System& s, double2* zu, int p0, int pb, const int* bad) {
  return launch_gs(s, k_gram_schmidt, zu, s.NB, s.NL, s.Hxyz, p0, pb, bad);
}

static CGArgs cg_args(const System& s, double2* zu) {
  CGArgs a;
  a.zu = zu;
  a.W = s.gs_W;
  a.st = (CGState*)s.gs_st;
  a.M = s.gs_M;
  a.MR = s.gs_MR;
  a.tband = s.gs_tb;
  a.nkl = s.nkl;
  a.NB = s.NB;
  a.NL = s.NL;
  a.Hxyz = s.Hxyz;
  return a;
}

// Where the lower bands are projected: inside the clusters, or, when these cover less
// than half the SMs and a CTA's share of the lower bands takes longer to read than two
// more launches, by the kernels over the whole GPU.
bool cg_wide(const System& s) {
  const int C = gs_cluster_size(s);
  return 2 * s.nkl * C < s.nsm && (size_t)s.NL / C * s.NB >= 131072;
}

static int cg_splits(const System& s, int n) {
  const int ctas = s.nkl * ((n + CG_DB - 1) / CG_DB);
  return std::max(1, std::min({CG_DOT_SPLITS, (4 * s.nsm + ctas - 1) / ctas, (s.NL + 1023) / 1024}));
}

static cudaError_t launch_cg_dots(const System& s, const double2* zu, const double2* x, size_t xstride, int b0, int n,
                                  const CGState* st, int& nsplit) {
  nsplit = cg_splits(s, n);
  const int chunk = (s.NL + nsplit - 1) / nsplit;
  k_cg_dots<<<dim3((n + CG_DB - 1) / CG_DB, nsplit, s.nkl), 256, 0, s.launch_stream()>>>(zu, x, xstride, b0, n, s.NB,
                                                                                        s.NL, chunk, st, s.gs_dots);
  return cudaGetLastError();
}

// which: the work vector (CG_GK: also copied to hk if copy_hk), or -1 for band ib of zu
// itself, with the real coefficients
cudaError_t launch_cg_project(const System& s, double2* zu, int ib, int which, bool copy_hk) {
  double2* x = which < 0 ? zu + (size_t)ib * s.NL : s.gs_W + (size_t)which * s.nkl * s.NL;
  const size_t xs = which < 0 ? (size_t)s.NB * s.NL : (size_t)s.NL;
  const CGState* st = which < 0 ? nullptr : (const CGState*)s.gs_st;
  double2* copy = copy_hk ? s.gs_W + (size_t)CG_HK * s.nkl * s.NL : nullptr;
  if (ib == 0 && copy)
    return cudaMemcpyAsync(copy, x, (size_t)s.nkl * s.NL * sizeof(double2), cudaMemcpyDeviceToDevice, s.stream);
  for (int b0 = 0; b0 < ib; b0 += CGB) {
    const int n = std::min(CGB, ib - b0);
    int ns = 1;
    cudaError_t e = launch_cg_dots(s, zu, x, xs, b0, n, st, ns);
    if (e != cudaSuccess) return e;
    const dim3 grid((s.NL + 255) / 256, s.nkl);
    double2* cp = b0 + n == ib ? copy : nullptr;
    if (which < 0)
      k_cg_subtract<true><<<grid, 256, 0, s.launch_stream()>>>(zu, x, xs, cp, b0, n, s.NB, s.NL, s.Hxyz, s.gs_M,
                                                               s.gs_MR, st, s.gs_dots, ns);
    else
      k_cg_subtract<false><<<grid, 256, 0, s.launch_stream()>>>(zu, x, xs, cp, b0, n, s.NB, s.NL, s.Hxyz, s.gs_M,
                                                                s.gs_MR, st, s.gs_dots, ns);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// the finished band's row of (I + L)^-1 (wide form; the cluster form does it in k_cg_step)
cudaError_t launch_cg_row(const System& s, double2* zu, int ib) {
  const int b0 = ib / CGB * CGB, n = ib - b0;
  int ns = 1;
  if (n > 0) {
    const cudaError_t e = launch_cg_dots(s, zu, zu + (size_t)ib * s.NL, (size_t)s.NB * s.NL, b0, n, nullptr, ns);
    if (e != cudaSuccess) return e;
  }
  k_cg_row<<<s.nkl, 256, 0, s.launch_stream()>>>(s.gs_M, s.gs_MR, b0, n, s.NB, s.Hxyz, s.gs_dots, ns);
  return cudaGetLastError();
}

cudaError_t launch_cg_open(const System& s, double2* zu, int ib, bool proj) {
  return launch_gs(s, k_cg_open, cg_args(s, zu), ib, proj ? 1 : 0, (const double*)s.occ_gs, s.gs_out, s.gs_res,
                   s.gs_iters);
}
cudaError_t launch_cg_first(const System& s, double2* zu, int ib, bool proj, bool pre) {
  return launch_gs(s, k_cg_first, cg_args(s, zu), ib, proj ? 1 : 0, pre ? 1 : 0);
}
cudaError_t launch_cg_dir(const System& s, double2* zu, int ib, int iter, bool proj, bool pre) {
  return launch_gs(s, k_cg_dir, cg_args(s, zu), ib, iter, proj ? 1 : 0, pre ? 1 : 0);
}
cudaError_t launch_cg_step(const System& s, double2* zu, int ib, int iter, bool last, bool proj, bool pre) {
  return launch_gs(s, k_cg_step, cg_args(s, zu), ib, iter, last ? 1 : 0, proj ? 1 : 0, pre ? 1 : 0, s.cg_delta);
}
size_t cg_state_bytes() { return sizeof(CGState); }
int cg_work_vectors() { return CG_NW; }

// ------------------------------------------- Hermitian Jacobi eigensolver --
// Cyclic two-sided Jacobi with the round-robin ordering: each step rotates
// n/2 disjoint index pairs at once.  For a pair (p,q) with A_pq = |b| e^{i phi},
// J = D R with D = diag(1, e^{-i phi}) (makes the pair real) and the real Jacobi
// rotation R = [[c, s], [-s, c]], t = sign(tau)/(|tau|+sqrt(1+tau^2)),
// tau = (a_qq-a_pp)/(2|b|).
//
// One CTA per k-point.  The 2x2 blocks (pair, pair) of A <- J^H A J are independent: one
// sweep over them a step, a warp per column pair.  V <- V J runs one step behind, on the
// warps that do not compute the next step's rotations.  A and V live in shared memory as
// long as both fit (JAC_SMEM), else in global memory.  Bound by the chain of FP64
// reciprocal roots of a step's rotations and the two barriers.
// At 32 k-points x 40 bands 0.53 ms; 1.05 ms with rows and columns rotated one after the
// other in global memory, 0.64 ms with square roots and divisions in the usual order.
//
// Sweeps stop when the off-diagonal norm of the upper triangle, the one the rotations
// are taken from, is below 1e-15 of the Frobenius norm, or after max_sweeps (the count
// used is written to sweeps[k]).  (Rounding leaves the lower triangle a floor of its own
// that the sweeps do not lower, at 128 bands above that threshold.)  Pairs below 1e-25 of
// the norm are not rotated: in the square of a tiny A_pq an underflow would make e^{i phi}
// a number of another modulus, and the rotation no rotation.
__device__ __forceinline__ int rr_partner(int i, int step, int n) {
  // round-robin: position 0 fixed, others rotate; returns the partner of index i
  if (i == 0) return 1 + (step % (n - 1));
  int pos = (i - 1 - step) % (n - 1);
  if (pos < 0) pos += n - 1;  // position of i in the rotating ring, 0..n-2
  // positions pair as (ring 0 <-> fixed 0), (ring r <-> ring n-1-r)
  if (pos == 0) return 0;
  const int ppos = n - 1 - pos;
  int idx = (ppos + step) % (n - 1);
  return idx + 1;
}


struct JacPair {
  int p, q;            // q = -1: the odd index out
  double c, s;
  double2 eph;         // e^{i phi}
};

constexpr size_t JAC_SMEM = 220 * 1024;

// the rotations of two steps; the eigenvalues and their order.  Beyond 3700 bands the
// rotations too are in global memory (gpr).
static size_t jac_pair_bytes(int NB) { return 2 * (size_t)((NB + 1) / 2) * sizeof(JacPair); }
static size_t jac_sort_bytes(int NB) { return (size_t)NB * (sizeof(double) + sizeof(int)) + 16; }

// GPR: the rotations are in gpr (a template parameter, so that the others are addressed as
// shared memory)
template <bool GPR>
__global__ void __launch_bounds__(1024) k_jacobi_herm(double2* __restrict__ Aall, double2* __restrict__ Vall, int NB,
                                                      int max_sweeps, int in_smem, JacPair* gpr,
                                                      double* __restrict__ w, int* __restrict__ sweeps) {
  extern __shared__ __align__(16) unsigned char jraw[];
  const int n = NB + (NB & 1), nh = n / 2;  // even count for the round-robin (index NB is a dummy)
  // [2][nh], this step's and the previous one's
  JacPair* pr2 = GPR ? gpr + (size_t)blockIdx.x * 2 * nh : reinterpret_cast<JacPair*>(jraw);
  double* ev = reinterpret_cast<double*>(jraw + (GPR ? 0 : 2 * nh * sizeof(JacPair)));  // [NB] eigenvalues
  int* rank = reinterpret_cast<int*>(ev + NB);              // [NB]
  double2* mats = reinterpret_cast<double2*>(jraw + (((size_t)((unsigned char*)(rank + NB) - jraw) + 15) & ~(size_t)15));
  __shared__ double sh[64];
  const int k = blockIdx.x, t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5, nwarp = nt >> 5;
  double2* Ag = Aall + (size_t)k * NB * NB;
  double2* Vg = Vall + (size_t)k * NB * NB;
  double2* A = in_smem ? mats : Ag;
  double2* V = in_smem ? mats + (size_t)NB * NB : Vg;
#define AE(r, c) A[(size_t)(c) * NB + (r)]
#define VE(r, c) V[(size_t)(c) * NB + (r)]
  for (int e = t; e < NB * NB; e += nt) {
    if (in_smem) A[e] = Ag[e];
    V[e] = make_double2((e % NB) == (e / NB) ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    double v[2] = {0.0, 0.0};  // squared norms: the diagonal, the upper triangle
    for (int e = t; e < NB * NB; e += nt) {
      const int r = e % NB, c = e / NB;
      const double2 x = A[e];
      if (r <= c) v[r != c] += x.x * x.x + x.y * x.y;
    }
    block_allsum<2>(v, sh);  // the same in every thread
    const double fro2 = v[0] + 2.0 * v[1];
    if (2.0 * v[1] <= 1e-30 * fro2) break;
    const double tiny2 = 1e-50 * fro2;
    for (int step = 0; step <= n - 1; ++step) {
      JacPair* pr = pr2 + (step & 1) * nh;
      const JacPair* prev = pr2 + ((step & 1) ^ 1) * nh;
      const int npw = (nh + 31) / 32;  // warps that compute rotations
      if (warp < npw && step < n - 1) {
        for (int i = t; i < nh; i += 32 * min(npw, nwarp)) {
          // ring position i pairs with n-1-i (i = 0: the fixed index)
          const int q0 = i == 0 ? 0 : 1 + (i + step) % (n - 1), q1 = rr_partner(q0, step, n);
          JacPair j;
          j.p = min(q0, q1);
          j.q = max(q0, q1) < NB ? max(q0, q1) : -1;
          j.c = 1.0;
          j.s = 0.0;
          j.eph = make_double2(1.0, 0.0);
          if (j.q >= 0) {
            const double app = AE(j.p, j.p).x, aqq = AE(j.q, j.q).x;
            const double2 b = AE(j.p, j.q);
            const double m2 = b.x * b.x + b.y * b.y;
            if (m2 > tiny2 && m2 > 1e-290) {
              // with delta = (a_qq - a_pp) / 2 and h = sqrt(delta^2 + |b|^2): c^2 = (1 + |delta| / h) / 2,
              // s = sign(delta) |b| / (2 c h), the same rotation from two reciprocal roots in a row
              const double del = 0.5 * (aqq - app);
              const double ih = rsqrt(fma(del, del, m2)), iab = rsqrt(m2);
              const double c2 = fma(0.5 * fabs(del), ih, 0.5), ic = rsqrt(c2);
              j.c = c2 * ic;
              j.s = (del >= 0 ? 0.5 : -0.5) * (m2 * iab) * ih * ic;
              j.eph = make_double2(b.x * iab, b.y * iab);
            }
          }
          pr[i] = j;
        }
      }
      if (step > 0 && (warp >= npw || step == n - 1 || npw >= nwarp)) {  // V <- V J of the previous step
        const int w0 = step == n - 1 || npw >= nwarp ? 0 : npw;
        for (int f = warp - w0; f < nh; f += nwarp - w0) {
          const JacPair b = prev[f];
          if (b.q < 0) continue;
          const double2 em = make_double2(b.eph.x, -b.eph.y);
          for (int row = lane; row < NB; row += 32) {
            const double2 xp = VE(row, b.p), ex = cmul(em, VE(row, b.q));
            VE(row, b.p) = make_double2(b.c * xp.x - b.s * ex.x, b.c * xp.y - b.s * ex.y);
            VE(row, b.q) = make_double2(b.s * xp.x + b.c * ex.x, b.s * xp.y + b.c * ex.y);
          }
        }
      }
      __syncthreads();
      if (step == n - 1) break;
      // A <- J^H A J, block by block: a warp per column pair, lanes over row pairs
      for (int jb = warp; jb < nh; jb += nwarp) {
        const JacPair b = pr[jb];
        const double2 em = make_double2(b.eph.x, -b.eph.y);
        for (int ja = lane; ja < nh; ja += 32) {
          const JacPair a = pr[ja];
          const int rows[2] = {a.p, a.q}, cols[2] = {b.p, b.q};
          double2 x[2][2];
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
              x[i][j] = rows[i] >= 0 && cols[j] >= 0 ? AE(rows[i], cols[j]) : make_double2(0.0, 0.0);
#pragma unroll
          for (int j = 0; j < 2; ++j) {  // rows: new_p = c x_p - s e^{i phi} x_q, new_q = s x_p + c e^{i phi} x_q
            const double2 ex = cmul(a.eph, x[1][j]), xp = x[0][j];
            x[0][j] = make_double2(a.c * xp.x - a.s * ex.x, a.c * xp.y - a.s * ex.y);
            x[1][j] = make_double2(a.s * xp.x + a.c * ex.x, a.s * xp.y + a.c * ex.y);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {  // columns: new_p = c x_p - s e^{-i phi} x_q, new_q = s x_p + c e^{-i phi} x_q
            const double2 ex = cmul(em, x[i][1]), xp = x[i][0];
            x[i][0] = make_double2(b.c * xp.x - b.s * ex.x, b.c * xp.y - b.s * ex.y);
            x[i][1] = make_double2(b.s * xp.x + b.c * ex.x, b.s * xp.y + b.c * ex.y);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
              if (rows[i] >= 0 && cols[j] >= 0) AE(rows[i], cols[j]) = x[i][j];
        }
      }
      __syncthreads();
    }
  }
  if (t == 0) sweeps[k] = sweep;
  // eigenvalues = diag, sorted ascending with the eigenvector columns (like zheev)
  double* wk = w + (size_t)k * NB;
  for (int i = t; i < NB; i += nt) ev[i] = AE(i, i).x;
  __syncthreads();
  for (int i = t; i < NB; i += nt) {
    int r = 0;
    for (int j2 = 0; j2 < NB; ++j2) r += (ev[j2] < ev[i]) || (ev[j2] == ev[i] && j2 < i);
    rank[i] = r;
    wk[r] = ev[i];
  }
  __syncthreads();
  // permuted eigenvectors into A (A is no longer needed)
  for (int e = t; e < NB * NB; e += nt) {
    const int row = e % NB, col = e / NB;
    Ag[(size_t)rank[col] * NB + row] = VE(row, col);
  }
#undef AE
#undef VE
}

cudaError_t launch_jacobi(const System& s, double2* A, double2* V, int max_sweeps, double* w, int* sweeps) {
  const size_t pairs = jac_pair_bytes(s.NB), sort = jac_sort_bytes(s.NB), both = 2 * (size_t)s.NB * s.NB * sizeof(double2);
  const int in_smem = pairs + sort + both <= JAC_SMEM;
  // (the split-K partials, at least nkl NB^2 values, are not in use here)
  JacPair* gpr = pairs + sort <= JAC_SMEM ? nullptr : reinterpret_cast<JacPair*>(s.gs_part);
  const size_t smem = (gpr ? 0 : pairs) + sort + (in_smem ? both : 0);
  auto kern = gpr ? k_jacobi_herm<true> : k_jacobi_herm<false>;
  const cudaError_t e = raise_smem_limit((const void*)kern, smem);
  if (e != cudaSuccess) return e;
  const int nt = 32 * std::min(32, std::max(8, (s.NB + 1) / 2 + 1));  // a warp per column pair, and one for the rotations
  kern<<<s.nkl, nt, smem, s.launch_stream()>>>(A, V, s.NB, max_sweeps, in_smem, gpr, w, sweeps);
  return cudaGetLastError();
}

}  // namespace sgpu
