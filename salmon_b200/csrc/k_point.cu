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

// The point form's time grows with the points; the march's stays at the latency of its
// NLx steps until the CTAs fill the GPU, later the larger the plane.  Four stages with
// the KB term, point form against march, us: complex(4) 8^3 x 256 orbitals 62 / 90, x 1024
// 123 / 82; 20^3 x 64 131 / 123; 32^3 x 16 188 / 188; 48^3 x 4 107 / 262, x 16 279 / 246;
// complex(8) 8^3 x 256 70 / 105, x 1024 158 / 131; 20^3 x 64 168 / 180; 32^3 x 16 237 / 423,
// x 64 581 / 434; 48^3 x 16 427 / 583.  The lines below lie under the crossings.
// Only with every launch choice left to the library: a KB kernel, pass form, table
// staging, x-slab count or Taylor form set through sgpu_set_param keeps its kernels.
bool hpsi_point_wins(const System& s, int nb, int prec) {
  if (s.kb_kernel != 0 || s.taylor_kernel != 0 || !s.pass_fixed || !s.pass_tab || s.nslab != 1) return false;
  const long plane = (long)s.NLy * s.NLz;
  const bool f = (prec < 0 ? s.prec : prec) == SGPU_PREC_C64;
  return (long)nb * s.NL <= (f ? 200000 + 300 * plane : 240000 + 700 * plane);
}

// the projections of the batch must be in s.U (launch_uvpsi / launch_uvpsi_from_S)
cudaError_t launch_hpsi_point(const System& s, int mode, const PassIO& io, int o_beg, int nb, int nbk, int prec) {
  if (nb == 0) return cudaSuccess;
  return (prec < 0 ? s.prec : prec) == SGPU_PREC_C64 ? launch_point_t<float>(s, mode, io, o_beg, nb, nbk)
                                                     : launch_point_t<double>(s, mode, io, o_beg, nb, nbk);
}

}  // namespace sgpu
