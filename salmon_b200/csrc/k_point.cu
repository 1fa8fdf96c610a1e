// One H application of a small batch, one thread per grid point.
//
// The march of k_pass.cu gives one CTA a whole orbital (or x-slab): with few or small
// orbitals the GPU is mostly idle and a CTA's march is a chain of NLx barriers.  Here
// every point is independent: 24 neighbours through L1 / L2, the Kleinman-Bylander term
// at sphere points summed from the point's <= 4 table entries and the projections U
// (entry order, FP64, as k_kb_w), so no KB field is written and read back.  The
// arithmetic is k_pass.cu's, term by term.
//
// Bound by L1 wavefronts (25 loads a point against about 13 shared-memory values a
// point in the march), so it loses once the march fills the GPU; hpsi_point_wins has
// the line.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "sgpu_internal.cuh"
#include "stencil_ops.cuh"

namespace sgpu {

template <typename R>
struct PointArgs {
  const C2<R>* in;       // [nb][NL]
  C2<R>* out;            // [nb][NL]
  C2<R>* tt;             // [nb][NL] (mode 1)
  const R* vloc;
  const double* kAc;     // [nkl][3]
  int o_beg, nbk, NLx, NLy, NLz, NL, nblk;
  double lap0sum;
  R lapt[12], nabc[12];
  float2 cl2[12], cn2[12];
  // Kleinman-Bylander tables (nsp 0: none)
  int nsp, Nlma, Nps;
  const int* sp_off;
  const short* lqi;
  const int4* rec;
  const int* cont;
  const double2* zproj;  // [nkl][Nlma][Nps]
  const double2* U;      // [nb][Nlma]
  C2<R>* S;              // [nb][nsp] export of the output (null: none)
  C2<R> zf;              // mode 2: the Taylor stage coefficient c
};

// MODE as in k_hpsi_pass: 0 out = H in, 1 also tt = H in - V in before the nonlocal
// term, 2 out = in + c H in.
template <typename R, int MODE>
__global__ void __launch_bounds__(256) k_hpsi_point(const PointArgs<R> a) {
  using T = C2<R>;
  const int b = blockIdx.x / a.nblk, i = (blockIdx.x - b * a.nblk) * 256 + threadIdx.x;
  if (i >= a.NL) return;
  const int kl = (a.o_beg + b) / a.nbk;
  const int NLx = a.NLx, NLy = a.NLy, NLz = a.NLz, NYZ = NLy * NLz;
  const int x = i / NYZ, yz = i - x * NYZ, y = yz / NLz, z = yz - y * NLz;
  const T* E = a.in + (size_t)b * a.NL;
  // the sphere index and the table entries are loaded beside the neighbours
  const int lq = a.nsp > 0 ? (int)__ldg(a.lqi + i) : -1;
  const int q = lq >= 0 ? __ldg(a.sp_off + x) + lq : -1;
  int4 ra = make_int4(0, 0, 0, 0), rb = ra;
  if (q >= 0) {
    ra = __ldg(a.rec + 2 * (size_t)q);
    rb = __ldg(a.rec + 2 * (size_t)q + 1);
  }
  const double kxd = a.kAc[3 * kl], kyd = a.kAc[3 * kl + 1], kzd = a.kAc[3 * kl + 2];
  const R A = (R)((kxd * kxd + kyd * kyd + kzd * kzd - a.lap0sum) * 0.5);  // k2lap0_2 (hpsi.f90:120-121)
  auto CL = [&](int n) { if constexpr (std::is_same<R, float>::value) return a.cl2[n]; else return a.lapt[n]; };
  auto CN = [&](int n) { if constexpr (std::is_same<R, float>::value) return a.cn2[n]; else return a.nabc[n]; };
  T v = mk<R>(0, 0), w = mk<R>(0, 0), wa = mk<R>(0, 0);
  const T c = __ldg(E + i);
  auto axis = [&](int pos, int len, int stride, int n0, auto k) {
    T p[4], m[4];
#pragma unroll
    for (int n = 1; n <= 4; ++n) {
      int pp = pos + n, pm = pos - n;
      while (pp >= len) pp -= len;
      while (pm < 0) pm += len;
      p[n - 1] = __ldg(E + i + (pp - pos) * stride);
      m[n - 1] = __ldg(E + i + (pm - pos) * stride);
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) stencil_pair(v, wa, p[n], m[n], CL(n0 + n), CN(n0 + n));
    w = kscale(k, wa, w);
    wa = mk<R>(0, 0);
  };
  axis(z, NLz, 1, 8, kpair<R>(kzd));
  axis(y, NLy, NLz, 4, kpair<R>(kyd));
  axis(x, NLx, NYZ, 0, kpair<R>(kxd));
  const R vl = __ldg(a.vloc + i);
  // F = B E + A E - 0.5 v - zI w   (stencil/F90/hpsi.f90:190)
  T f;
  f.x = fma(vl + A, c.x, fma((R)-0.5, v.x, w.y));
  f.y = fma(vl + A, c.y, fma((R)-0.5, v.y, -w.x));
  const size_t o = (size_t)b * a.NL + i;
  if constexpr (MODE == 1) a.tt[o] = mk<R>(fma(-vl, c.x, f.x), fma(-vl, c.y, f.y));
  if (q >= 0) {  // + pseudo_pt scatter (hpsi.f90:194-206)
    const int ne = ra.y + rb.w;
    const double2* zk = a.zproj + (size_t)kl * a.Nlma * a.Nps;
    const double2* Ub = a.U + (size_t)b * a.Nlma;
    double2 acc = make_double2(0.0, 0.0);
    const int e4[4] = {ra.z, ra.w, rb.x, rb.y};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < ne) {
        const int ilma = e4[e] >> 16;
        acc = cfma(__ldg(zk + (size_t)ilma * a.Nps + (e4[e] & 0xffff)), __ldg(Ub + ilma), acc);
      }
    for (int e = 4; e < ne; ++e) {
      const int en = __ldg(a.cont + rb.z + (e - 4)), ilma = en >> 16;
      acc = cfma(__ldg(zk + (size_t)ilma * a.Nps + (en & 0xffff)), __ldg(Ub + ilma), acc);
    }
    f = cadd(f, mk<R>((R)acc.x, (R)acc.y));
  }
  if constexpr (MODE == 2) f = cfma(a.zf, f, c);
  a.out[o] = f;
  if (a.S && q >= 0) a.S[(size_t)b * a.nsp + q] = f;
}

template <typename R>
static cudaError_t launch_point_t(const System& s, int mode, const PassIO& io, int o_beg, int nb, int nbk) {
  PointArgs<R> a;
  a.in = (const C2<R>*)io.in;
  a.out = (C2<R>*)io.out;
  a.tt = (C2<R>*)io.tt;
  a.vloc = std::is_same<R, float>::value ? (const R*)s.vloc32 : (const R*)s.vloc64;
  a.kAc = s.kAc_d;
  a.o_beg = o_beg;
  a.nbk = nbk;
  a.NLx = s.NLx; a.NLy = s.NLy; a.NLz = s.NLz; a.NL = s.NL;
  a.nblk = (s.NL + 255) / 256;
  a.lap0sum = s.lap[0][0] + s.lap[1][0] + s.lap[2][0];
  for (int n = 0; n < 4; ++n)
    for (int d = 0; d < 3; ++d) {
      a.lapt[4 * d + n] = (R)s.lap[d][n + 1];
      a.nabc[4 * d + n] = (R)s.nab[d][n + 1];
      a.cl2[4 * d + n] = make_float2((float)s.lap[d][n + 1], (float)s.lap[d][n + 1]);
      a.cn2[4 * d + n] = make_float2((float)s.nab[d][n + 1], (float)s.nab[d][n + 1]);
    }
  a.nsp = s.nsp;
  a.Nlma = s.Nlma;
  a.Nps = s.Nps;
  a.sp_off = s.sp_off;
  a.lqi = s.lqi;
  a.rec = s.rec;
  a.cont = s.cont;
  a.zproj = s.zproj64;
  a.U = s.U;
  a.S = (C2<R>*)io.S;
  a.zf = mk<R>((R)io.zc[0], (R)io.zc[1]);
  const int grid = nb * a.nblk;
  switch (mode) {
    case 0: k_hpsi_point<R, 0><<<grid, 256, 0, s.launch_stream()>>>(a); break;
    case 1: k_hpsi_point<R, 1><<<grid, 256, 0, s.launch_stream()>>>(a); break;
    default: k_hpsi_point<R, 2><<<grid, 256, 0, s.launch_stream()>>>(a);
  }
  return cudaGetLastError();
}

// The point form's time grows with the points and, through k_uvpsi, with the points of an
// atom; the march's stays at the latency of its NLx steps until the CTAs fill the GPU.  Both
// therefore compare as the points of one step of the march, nb x plane.  Four stages with the
// KB term, point form against march, us:
//   one-row planes  complex(4) 8^3 x 128 orbitals 54 / 66, x 512 78 / 66; 20^3 x 32 95 / 119, x 64
//                   130 / 123; 24^3 x 32 138 / 156, x 64 193 / 156; 36^3 x 16 241 / 242;
//                   complex(8) 8^3 x 256 70 / 78, x 512 99 / 78; 12^3 x 64 71 / 90, x 128 98 / 90;
//                   20^3 x 64 167 / 180; 24^3 x 32 168 / 230; 36^3 x 16 306 / 394, x 32 467 / 402
//   two-row planes  (123 points an atom unless said) complex(4) 16x16x32 x 32 80 / 90, x 64 115 / 90;
//                   32^3 x 16 115 / 131, x 32 185 / 131, with 1020 points x 4 128 / 146, x 12 172 / 148;
//                   48^3 x 8 160 / 222, x 16 279 / 227; complex(8) 16x16x32 x 32 103 / 123, x 64
//                   152 / 131; 32^3 x 16 158 / 189, x 32 270 / 189, with 1020 points x 8 173 / 185,
//                   x 12 206 / 185; 48^3 x 8 238 / 284, x 12 328 / 284
// CG's vectors (slabs > 0: the x-slabs their march would have, which shorten it; complex(8), no
// export to S) compare by their points.  sgpu_cg, 6 bands x 4 iterations, ms, point form against
// march: two-row planes 16x16x32 x 48 3.07 / 3.22, x 64 3.62 / 3.58; 32^3 x 12 3.01 / 3.20, x 24
// 5.40 / 5.17, with 1020 points an atom x 1 2.25 / 2.02; 48^3 (no slabs) x 12 9.34 / 9.64, x 16 14.6 /
// 14.1; one-row planes 24^3 with 57 points an atom x 16 2.70 / 2.83, x 32 3.28 / 3.03, with 437 points
// x 32 3.36 / 3.42, x 48 4.91 / 4.75; 18x24x27 x 64 5.37 / 5.71.
// The lines below lie near the crossings, where both forms take the same time to a few percent.
// Only with every launch choice left to the library: a KB kernel, pass form, table staging,
// x-slab count or Taylor form set through sgpu_set_param keeps its kernels.
bool hpsi_point_wins(const System& s, int nb, int prec, int slabs) {
  if (s.kb_kernel != 0 || s.taylor_kernel != 0 || !s.pass_fixed || !s.pass_tab || s.nslab != 1) return false;
  const long plane = (long)s.NLy * s.NLz, mps = s.max_mps;
  const int pr = prec < 0 ? s.prec : prec;
  const bool f = pr == SGPU_PREC_C64, two_row = s.p2_rows[pr] > 0;
  if (slabs > 0) {
    long most = 240000 + 700 * plane;
    if (slabs > 1 && two_row) most = 500000 - 480 * mps;
    else if (slabs > 1 && s.NLz % 2 == 0) most = std::min(most, 240000 + 600 * mps);
    return (long)nb * s.NL <= most;
  }
  if (two_row) return nb * plane <= (f ? std::min(18500L, 22000 - 14 * mps) : std::min(19000L, 20000 - 10 * mps));
  return nb * plane <= (f ? 20000L : std::min(28000L, 14000 + 30 * plane));
}

// the projections of the batch must be in s.U (launch_uvpsi / launch_uvpsi_from_S)
cudaError_t launch_hpsi_point(const System& s, int mode, const PassIO& io, int o_beg, int nb, int nbk, int prec) {
  if (nb == 0) return cudaSuccess;
  return (prec < 0 ? s.prec : prec) == SGPU_PREC_C64 ? launch_point_t<float>(s, mode, io, o_beg, nb, nbk)
                                                     : launch_point_t<double>(s, mode, io, o_beg, nb, nbk);
}

}  // namespace sgpu
