// FP64 complex products of the ground state on the tensor pipe
// (mma.sync m8n8k4.f64; tcgen05 has no FP64), and the blocked Gram-Schmidt
// built on them.
//
// A complex product is two real ones over the interleaved (re, im) index: with
// k = (point, part), Re sum conj(a) b = sum_k a_k b_k and Im = sum_k a_k b'_k,
// b' = (im, -re), so one fragment of A serves both and no operand is reordered
// in shared memory.
#include <cuda_runtime.h>

#include <algorithm>

#include "sgpu_internal.cuh"

namespace sgpu {

__device__ __forceinline__ void zmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// ------------------------------------------------------------ A^H B, split K --
// part[sp][k][n][m] = sum_{i in split sp} conj(A[k][m][i]) B[k][n][i],  m < M, n < N.
// CTA: a 32 x 32 tile of one k-point and one range of points; four warps of 16 x 16;
// chunks of 8 points through a four-stage cp.async ring (rows padded to 10 values:
// the eight rows a warp reads fall in distinct banks, two wavefronts a load).
// lower: tiles above the diagonal are skipped (Hermitian products).
// Bound by the FP64 pipe: 8 MMAs per 4 shared-memory loads.  At 16x16x32, 32 k, 40 bands:
// H_sub 0.25 ms (CUDA cores, 16 x 16 tiles: 0.51), the rotation 0.14 ms (0.45).
constexpr int ZT = 32, ZK = 8, ZROW = ZK + 2, ZST = 4;

__global__ void __launch_bounds__(128) k_zgemm_hn(const double2* __restrict__ A, const double2* __restrict__ B,
                                                 size_t kstride, int M, int N, int NL, int kchunk, int tm_count,
                                                 int lower, const int* __restrict__ skip, double2* __restrict__ part) {
  __shared__ double2 sa[ZST][ZT][ZROW], sb[ZST][ZT][ZROW];
  const int k = blockIdx.x / tm_count, tm = blockIdx.x - k * tm_count, tn = blockIdx.y;
  if (lower && tm < tn) return;  // whole CTA
  if (skip && skip[k]) return;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int i0 = blockIdx.z * kchunk, i1 = min(i0 + kchunk, NL);
  const double2* Ak = A + k * kstride + (size_t)tm * ZT * NL;
  const double2* Bk = B + k * kstride + (size_t)tn * ZT * NL;
  const int mrows = min(ZT, M - tm * ZT), nrows = min(ZT, N - tn * ZT);
  const int nch = i1 > i0 ? (i1 - i0 + ZK - 1) / ZK : 0;
  const int cp = t % ZK, cr = t / ZK;  // this thread copies point cp of rows cr, cr + 16
  auto issue = [&](int c) {
    if (c < nch) {
      const int s = c % ZST, i = i0 + c * ZK + cp;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = cr + 16 * h;
        if (r < mrows && i < i1) cp_async16(&sa[s][r][cp], Ak + (size_t)r * NL + i);
        else sa[s][r][cp] = make_double2(0.0, 0.0);
        if (r < nrows && i < i1) cp_async16(&sb[s][r][cp], Bk + (size_t)r * NL + i);
        else sb[s][r][cp] = make_double2(0.0, 0.0);
      }
    }
    cp_async_commit();
  };
  const int wm = (warp & 1) * 16, wn = (warp >> 1) * 16;
  const int row = lane >> 2, pt = (lane >> 1) & 1, prt = lane & 1;
  // the warp's 8 x 8 sub-tiles with an element to compute (uniform over the warp)
  bool need[2][2];
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
      need[mi][ni] = wm + 8 * mi < mrows && wn + 8 * ni < nrows && !(lower && tm == tn && wm + 8 * mi + 7 < wn + 8 * ni);
  const bool any = need[0][0] || need[0][1] || need[1][0] || need[1][1];
  double cre[2][2][2] = {}, cim[2][2][2] = {};
  for (int c = 0; c < ZST - 1; ++c) issue(c);
  for (int c = 0; c < nch; ++c) {
    cp_async_wait<ZST - 2>();
    __syncthreads();
    issue(c + ZST - 1);
    const int s = c % ZST;
    if (!any) continue;
#pragma unroll
    for (int ks = 0; ks < ZK / 2; ++ks) {
      const int p = 2 * ks + pt;
      double a[2], br[2], bi[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        a[h] = reinterpret_cast<const double*>(&sa[s][wm + 8 * h + row][p])[prt];
        const double2 b = sb[s][wn + 8 * h + row][p];
        br[h] = prt ? b.y : b.x;
        bi[h] = prt ? -b.x : b.y;
      }
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) {
          if (need[mi][ni]) {
            zmma(cre[mi][ni], a[mi], br[ni]);
            zmma(cim[mi][ni], a[mi], bi[ni]);
          }
        }
    }
  }
  cp_async_wait<0>();
  const int nkl = gridDim.x / tm_count;
  double2* out = part + ((size_t)blockIdx.z * nkl + k) * N * M;
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int m = tm * ZT + wm + 8 * mi + row, n = tn * ZT + wn + 8 * ni + 2 * (lane & 3) + e;
        if (m < M && n < N) out[(size_t)n * M + m] = make_double2(cre[mi][ni][e], cim[mi][ni][e]);
      }
}

// ------------------------------------------------------------------- X Z ----
// out[k][n][i] = sum_m X[k][m][i] Z[k][n][m]                 (base null)
//             = base[k][n][i] - sum_m X[k][m][i] Z[k][n][m]  (base = out: in place)
// CTA: 64 points x 32 outputs, four warps of 16 points; chunks of 8 rows of X and Z
// through a three-stage ring.  Every input of the CTA's points is read before the
// first output is written, so out may be X itself when one CTA covers all outputs
// (N <= 32).  Points are contiguous in both arrays: loads and stores are 128-byte runs.
constexpr int ZP = 64, ZST2 = 3;

__global__ void __launch_bounds__(128) k_zgemm_nn(const double2* X, size_t xstride, const double2* __restrict__ Z,
                                                 size_t zstride, int ldz, int M, int N, int NL, const double2* base,
                                                 double2* out, size_t ostride, const int* __restrict__ skip) {
  __shared__ double2 sx[ZST2][ZK][ZP], sz[ZST2][ZT][ZROW];
  const int npt = (NL + ZP - 1) / ZP, k = blockIdx.x / npt, n0 = blockIdx.y * ZT, p0 = (blockIdx.x - k * npt) * ZP;
  if (skip && skip[k]) return;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const double2* Xk = X + k * xstride;
  const double2* Zk = Z + k * zstride;
  const int nch = (M + ZK - 1) / ZK;
  auto issue = [&](int c) {
    if (c < nch) {
      const int s = c % ZST2;
#pragma unroll
      for (int h = 0; h < 4; ++h) {  // 8 rows x 64 points
        const int e = t + 128 * h, r = e / ZP, p = e % ZP, m = c * ZK + r;
        if (m < M && p0 + p < NL) cp_async16(&sx[s][r][p], Xk + (size_t)m * NL + p0 + p);
        else sx[s][r][p] = make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // 32 outputs x 8 coefficients
        const int e = t + 128 * h, n = e / ZK, r = e % ZK, m = c * ZK + r;
        if (m < M && n0 + n < N) cp_async16(&sz[s][n][r], Zk + (size_t)(n0 + n) * ldz + m);
        else sz[s][n][r] = make_double2(0.0, 0.0);
      }
    }
    cp_async_commit();
  };
  const int row = lane >> 2, mm = (lane >> 1) & 1, prt = lane & 1;
  double cre[2][4][2] = {}, cim[2][4][2] = {};
  for (int c = 0; c < ZST2 - 1; ++c) issue(c);
  for (int c = 0; c < nch; ++c) {
    cp_async_wait<ZST2 - 2>();
    __syncthreads();
    issue(c + ZST2 - 1);
    const int s = c % ZST2;
#pragma unroll
    for (int ks = 0; ks < ZK / 2; ++ks) {
      const int r = 2 * ks + mm;
      double a[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) a[h] = reinterpret_cast<const double*>(&sx[s][r][16 * warp + 8 * h + row])[prt];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        if (n0 + 8 * ni >= N) continue;  // uniform
        const double2 z = sz[s][8 * ni + row][r];
        const double br = prt ? -z.y : z.x, bi = prt ? z.x : z.y;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          zmma(cre[h][ni], a[h], br);
          zmma(cim[h][ni], a[h], bi);
        }
      }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = p0 + 16 * warp + 8 * h + row;
    if (i >= NL) continue;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = n0 + 8 * ni + 2 * (lane & 3) + e;
        if (n >= N) continue;
        double2 v = make_double2(cre[h][ni][e], cim[h][ni][e]);
        if (base) {
          const double2 b = base[k * ostride + (size_t)n * NL + i];
          v = make_double2(b.x - v.x, b.y - v.y);
        }
        out[k * ostride + (size_t)n * NL + i] = v;
      }
  }
}

// ranges of points of a split product: about four CTAs per SM, at least 64 points
// each, and no more partials than gs_part holds
static int zsplit(const System& s, int tiles, size_t mn) {
  const int want = (4 * s.nsm + s.nkl * tiles - 1) / (s.nkl * tiles);
  const int most = (int)std::min<size_t>(64, s.gs_part_elems / std::max<size_t>(1, s.nkl * mn));
  return std::max(1, std::min({want, most, (s.NL + 63) / 64}));
}

static cudaError_t launch_hn(const System& s, const double2* A, int M, const double2* B, int N, bool lower,
                             double2* part, int& nsplit, const int* skip = nullptr) {
  const int tm = (M + ZT - 1) / ZT, tn = (N + ZT - 1) / ZT;
  nsplit = zsplit(s, lower ? tm * (tm + 1) / 2 : tm * tn, (size_t)M * N);
  const int kchunk = ((s.NL + nsplit - 1) / nsplit + ZK - 1) / ZK * ZK;
  k_zgemm_hn<<<dim3(s.nkl * tm, tn, nsplit), 128, 0, s.launch_stream()>>>(A, B, (size_t)s.NB * s.NL, M, N, s.NL,
                                                                         kchunk, tm, lower ? 1 : 0, skip, part);
  return cudaGetLastError();
}

static cudaError_t launch_nn(const System& s, const double2* X, int M, const double2* Z, size_t zstride, int ldz, int N,
                             const double2* base, double2* out, const int* skip = nullptr) {
  const size_t ks = (size_t)s.NB * s.NL;
  // (k-points in the first grid dimension: the others end at 65535)
  k_zgemm_nn<<<dim3(s.nkl * ((s.NL + ZP - 1) / ZP), (N + ZT - 1) / ZT), 128, 0, s.launch_stream()>>>(
      X, ks, Z, zstride, ldz, M, N, s.NL, base, out, ks, skip);
  return cudaGetLastError();
}

// ------------------------------------------------------ subspace products --
// za[k][n][m] = Hxyz * sum_sp part[sp][k][n][m]  then made Hermitian like
// diag_omp builds it (GS/diag.f90:112-116): the lower triangle (m > n) is
// computed, the upper is its conjugate, the diagonal is real.
__global__ void k_zgemm_reduce_herm(const double2* __restrict__ part, int nsplit, int nkl, int NB, double Hxyz,
                                    double2* __restrict__ za) {
  const size_t tot = (size_t)nkl * NB * NB;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < tot; e += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(e / ((size_t)NB * NB));
    const int n = (int)((e / NB) % NB), m = (int)(e % NB);
    // element (row m, column n) of za(:,:) stored at za[k][n][m] (column-major)
    const int lo_r = m > n ? m : n, lo_c = m > n ? n : m;  // lower-triangle source
    double2 s = make_double2(0, 0);
    for (int sp = 0; sp < nsplit; ++sp) {
      const double2 p = part[(((size_t)sp * nkl + k) * NB + lo_c) * NB + lo_r];
      s.x += p.x;
      s.y += p.y;
    }
    s = make_double2(s.x * Hxyz, s.y * Hxyz);
    if (m == n) s.y = 0.0;
    else if (m < n) s.y = -s.y;
    za[e] = s;
  }
}

cudaError_t launch_subspace_h(const System& s, const double2* U, const double2* HU, double2* part, double2* za) {
  int nsplit = 1;
  cudaError_t e = launch_hn(s, U, s.NB, HU, s.NB, true, part, nsplit);
  if (e != cudaSuccess) return e;
  const size_t tot = (size_t)s.nkl * s.NB * s.NB;
  k_zgemm_reduce_herm<<<(int)std::min<size_t>((tot + 255) / 256, 4096), 256, 0, s.launch_stream()>>>(
      part, nsplit, s.nkl, s.NB, s.Hxyz, za);
  return cudaGetLastError();
}

// out[k][n][i] = sum_m in[k][m][i] Z[k][n][m]   (zutmp(:,ib1) = sum_ib2 zu(:,ib2) za(ib2,ib1), diag.f90:120-126)
cudaError_t launch_rotate(const System& s, const double2* in, const double2* Z, double2* out) {
  return launch_nn(s, in, s.NB, Z, (size_t)s.NB * s.NB, s.NB, s.NB, nullptr, out);
}

// ---------------------------------------------------- blocked Gram-Schmidt --
// The reference projects each band on the lower ones one by one
// (GS/Gram_Schmidt.f90:32-55), i.e. builds the QR factorisation with a positive
// diagonal by modified Gram-Schmidt: NB (NB-1) / 2 dependent inner products.
// Here panels of up to 32 bands are orthonormalised through their Gram matrix, then
// projected out of all later bands at once (modified Gram-Schmidt by blocks):
//   S = P^H P, S = L L^H, P <- P L^-H, twice (CholeskyQR2: Yamamoto, Nakatsukasa,
//   Yanagisawa and Fukaya, ETNA 44 (2015) 306: orthogonal to working precision for
//   condition numbers up to ~1e8), then X <- X - P (P^H X) for the later bands.
// Which rounds a panel gets follows from tau = sum |(D^1/2 L^-H)_ml|^2, D the diagonal of S:
// tau bounds the largest eigenvalue of the inverse of the panel's scaled Gram matrix, whose
// trace is pb, so the squared condition number of the scaled bands is at most pb tau.  (The
// pivots bound nothing of the kind: bands that each overlap with the one before keep pivots of
// a quarter while the condition number grows like 1.7^pb.)
//   tau <= GS_ONCE pb (orthogonal bands have tau = pb): one round leaves the panel
//     orthonormal to a few eps; the bands of a running ground state are here.
//   tau <= GS_COND: two rounds, the first leaving an error of at most about 1e-16 pb tau <
//     1e-3, which the second squares away; it has to find tau <= GS_ONCE pb itself.
//   beyond, or a pivot below GS_PIVOT of its diagonal entry, a zero or a NaN: k_gram_schmidt,
//     the one-by-one form, for that k-point.
// The factorisation is unique, so the result is the reference's up to rounding.  Largest
// |<u_i|u_j> - delta_ij|, 32 bands with a sine of 0.51 / 0.6 / 0.8 to the band before: one by
// one 1e-8 / 3e-12 / 2e-15, here 1e-8 (one by one) / 6e-16 (two rounds) / 9e-16.
// One Gram-Schmidt at 16x16x32, 32 k, 40 bands: 3.56 -> 0.5 ms.
static_assert(GSP == ZT, "a panel is one output tile of k_zgemm_nn (in place)");
constexpr double GS_PIVOT = 1e-9, GS_ONCE = 2.0, GS_COND = 1e11;

// Sums the panel's Gram matrix, factors it and writes Z[k][n][m] = (L^-H)(m, n):
// one CTA per k-point, thread (i, l) owns element (i, l) of the trailing matrix and
// of L^-1 (eliminated together, one barrier a column).  bad[k]: refused, the panel must not
// be multiplied (0 times an infinity would spread it over the panel); skip[k]: no second round.
__global__ void __launch_bounds__(GSP* GSP) k_gs_chol(const double2* __restrict__ part, int nsplit, int nkl, int pb,
                                                      double Hxyz, int round, int* __restrict__ bad,
                                                      int* __restrict__ skip, double2* __restrict__ Z) {
  __shared__ double2 A[GSP][GSP + 1], W[GSP][GSP + 1];
  __shared__ double d0[GSP], inv[GSP], sh[32];
  const int k = blockIdx.x, i = threadIdx.x / GSP, l = threadIdx.x % GSP;
  if (round == 1 && skip[k]) return;  // (the products of this round return too)
  double2 a = make_double2(0.0, 0.0);
  if (i < pb && l <= i)
    for (int sp = 0; sp < nsplit; ++sp) {
      const double2 v = part[(((size_t)sp * nkl + k) * pb + l) * pb + i];
      a.x += v.x;
      a.y += v.y;
    }
  a = make_double2(a.x * Hxyz, a.y * Hxyz);
  A[i][l] = a;
  W[i][l] = make_double2(i == l ? 1.0 : 0.0, 0.0);
  if (i == l) d0[i] = a.x;
  bool ok = true;
  for (int j = 0; j < pb && ok; ++j) {
    __syncthreads();
    const double d = A[j][j].x;
    ok = d > GS_PIVOT * d0[j] && d > 0.0 && d < 1e300;  // the same for every thread; false for NaN
    if (!ok) break;
    const double r = 1.0 / sqrt(d);
    if (threadIdx.x == 0) inv[j] = r;
    if (i > j && i < pb) {
      const double2 lij = make_double2(A[i][j].x * r, A[i][j].y * r);
      if (l > j && l <= i) {
        const double2 llj = make_double2(A[l][j].x * r, -A[l][j].y * r);
        A[i][l] = csub(A[i][l], cmul(lij, llj));
      } else if (l <= j) {  // row j of L^-1 is scaled by r at the end
        W[i][l] = csub(W[i][l], cmul(lij, make_double2(W[j][l].x * r, W[j][l].y * r)));
      }
    }
  }
  __syncthreads();
  double tau[1] = {0.0};
  if (ok && i < pb && l <= i) tau[0] = (W[i][l].x * W[i][l].x + W[i][l].y * W[i][l].y) * inv[i] * inv[i] * d0[l];
  block_allsum<1>(tau, sh);
  const bool good = tau[0] <= GS_ONCE * pb;  // the same in every thread; false for NaN
  ok = ok && (good || (round == 0 && tau[0] <= GS_COND));
  if (ok && i < pb && l < pb)
    Z[((size_t)k * GSP + i) * GSP + l] =
        l <= i ? make_double2(W[i][l].x * inv[i], -W[i][l].y * inv[i]) : make_double2(0.0, 0.0);
  if (threadIdx.x == 0) {
    bad[k] = !ok;
    if (round == 0 || !ok) skip[k] = !ok || good;
  }
}

// C[k][n][m] = Hxyz sum_sp part[sp][k][n][m]
__global__ void k_part_sum(const double2* __restrict__ part, int nsplit, size_t tot, double Hxyz,
                           double2* __restrict__ C) {
  const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e >= tot) return;
  double2 s = make_double2(0.0, 0.0);
  for (int sp = 0; sp < nsplit; ++sp) {
    const double2 v = part[sp * tot + e];
    s.x += v.x;
    s.y += v.y;
  }
  C[e] = make_double2(s.x * Hxyz, s.y * Hxyz);
}

cudaError_t launch_gram_schmidt(const System& s, double2* zu) {
  cudaError_t e;
  const int npan = (s.NB + GSP - 1) / GSP, pw = (s.NB + npan - 1) / npan;  // panels of equal width
  for (int p0 = 0; p0 < s.NB; p0 += pw) {
    const int pb = std::min(pw, s.NB - p0), rest = s.NB - p0 - pb;
    double2* P = zu + (size_t)p0 * s.NL;
    int ns = 1;
    int* skip = s.gs_bad + s.nkl;
    for (int round = 0; round < 2; ++round) {
      if ((e = launch_hn(s, P, pb, P, pb, true, s.gs_part, ns, round ? skip : nullptr)) != cudaSuccess) return e;
      k_gs_chol<<<s.nkl, GSP * GSP, 0, s.launch_stream()>>>(s.gs_part, ns, s.nkl, pb, s.Hxyz, round, s.gs_bad, skip,
                                                            s.gs_R);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      if ((e = launch_nn(s, P, pb, s.gs_R, (size_t)GSP * GSP, GSP, pb, nullptr, P, round ? skip : s.gs_bad)) !=
          cudaSuccess)
        return e;
    }
    if ((e = launch_gram_schmidt_panel(s, zu, p0, pb, s.gs_bad)) != cudaSuccess) return e;
    if (rest > 0) {
      double2* X = P + (size_t)pb * s.NL;
      if ((e = launch_hn(s, P, pb, X, rest, false, s.gs_part, ns)) != cudaSuccess) return e;
      const size_t tot = (size_t)s.nkl * rest * pb;
      k_part_sum<<<(int)((tot + 255) / 256), 256, 0, s.launch_stream()>>>(s.gs_part, ns, tot, s.Hxyz, s.gs_A);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      if ((e = launch_nn(s, P, pb, s.gs_A, (size_t)rest * pb, pb, rest, X, X)) != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace sgpu
