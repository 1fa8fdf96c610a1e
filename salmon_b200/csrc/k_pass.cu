// One Hamiltonian application (and the fused last Taylor pass) for sm_100a.
//
// H psi = (k2lap0_2 + Vloc) psi - 1/2 sum lapt (psi(+n)+psi(-n)) - i sum nabt (psi(+n)-psi(-n))
//         + W,   W = sum_ilma zproj(:,ilma) U(ilma) at the sphere points
// restates hpsi_omp_KB_base (common/hpsi.f90:98-208): the stencil of
// stencil/F90/hpsi.f90:190 plus the Kleinman-Bylander scatter of pseudo_pt
// (:194-206).  W is computed beforehand by k_kbfield (k_hpsi.cu) in a compact
// per-orbital array over the sphere points, ordered by grid index.
//
// Layout: one CTA per (orbital, x-slab).  A y-z plane of one orbital is a
// contiguous NLy*NLz run in HBM (z unit stride).  Each thread owns RZ
// consecutive z points of one y row and marches along x:
//   * planes stream into a shared-memory ring with cp.async, NR-5 planes ahead
//     of use, together with each plane's contiguous chunk of W, so HBM latency
//     is off the critical path;
//   * the thread's own 9 x-neighbours sit in a register queue;
//   * y and z neighbours come from the shared-memory plane;
//   * a point's local sphere index (int16 table, loaded one plane ahead) tells
//     whether to add W and whether to export the output value to S, the
//     compact sphere-value array the next pass's projections read.
// Each input element is read from HBM once per pass (the 8 halo planes of a
// slab come from L2), each output element written once.
#include <cuda_runtime.h>

#include <type_traits>

#include "sgpu_internal.cuh"
#include "stencil_ops.cuh"

namespace sgpu {

template <typename R>
struct PassArgs {
  const C2<R>* in;       // [nb][NL]
  C2<R>* out;            // [nb][NL]
  C2<R>* tt;             // [nb][NL]   (mode 1)
  const R* vloc;
  const double* kAc;     // [nkl][3]
  int o_beg, NBocc;
  int NLx, NLy, NLz, NL, SX;
  double lap0sum;        // lapx(0)+lapy(0)+lapz(0)
  R lapt[12];            // lapx(1:4), lapy(1:4), lapz(1:4)
  R nabc[12];            // nabx(1:4), naby(1:4), nabz(1:4)
  float2 cl2[12], cn2[12];  // complex(4): lapt and nabc as broadcast pairs for the packed FP32 arithmetic
  // Kleinman-Bylander term by plane: plane x's sphere points are
  // sp_off[x] .. sp_off[x+1]-1 (at most maxpts); lqi[i] is the index of grid
  // point i among its plane's sphere points, or -1.
  const int* sp_off;
  // y-blocks (YB form, planes wider than one CTA): each orbital plane is split
  // into nyblk CTAs of NYB rows; sp_blk[x*(nyblk+1) + yb] is the first sphere
  // point of plane x in rows >= yb*NYB (sp_blk[x*(nyblk+1)] = sp_off[x]).
  int NYB, nyblk;
  const int* sp_blk;
  const short* lqi;
  const C2<R>* W;        // [nb][nsp] KB term at the sphere points (null: none)
  C2<R>* S;              // [nb][nsp] export of the output (null: none)
  int nsp, maxpts;
  C2<R> zf;              // mode 2: the Taylor stage coefficient c
};

template <typename R> struct PassGeom {
  static constexpr int NR = std::is_same<R, float>::value ? 8 : 6;  // ring planes
};

size_t pass_smem_bytes(int prec, int NLy, int NLz, int maxpts, bool with_w, int NLx, int nyblk, int NYB,
                       bool tables, int nr) {
  const size_t e = prec == SGPU_PREC_C64 ? sizeof(float2) : sizeof(double2);
  const int NR = nr > 0 ? nr : (prec == SGPU_PREC_C64 ? PassGeom<float>::NR : PassGeom<double>::NR);
  const size_t ryz = nyblk > 1 ? (size_t)(NYB + 8) * NLz : (size_t)NLy * NLz;
  const size_t tyz = nyblk > 1 ? (size_t)NYB * NLz : (size_t)NLy * NLz;
  return e * (size_t)NR * (ryz + (with_w ? (size_t)maxpts : 0)) +
         (tables ? (size_t)NR * tyz * (e / 2 + sizeof(short)) : 0) + sizeof(int) * (size_t)NLx * (nyblk + 1) +
         sizeof(int);
}

// MODE 0: out = H in.   MODE 1: also tt = H in - V in before the nonlocal term.
// MODE 2: out = in + c H in, one linear factor of the Taylor polynomial
// (RT/hamiltonian.f90:46-49, :99-122 evaluated as the product of its four
// linear factors; see enqueue_taylor_step).
//
// YB (planes of more than 512 threads' points): the plane is split over nyblk
// CTAs of NYB rows; each CTA's ring holds its rows and 4 halo rows on each side.
// TB (two-point form): Vloc and the local sphere indices of each owned plane
// travel with the plane through the ring (copy group of the plane) instead of
// being loaded from global memory one plane ahead; this takes the dependent
// global loads off each march step.
//
// GY, GZ (non-zero: the plane shape NLy x NLz at compile time, complex(4), two-point
// table form): the ring then has one slot per
// unrolled phase (NR = 9), so every ring, table and neighbour offset is a
// compile-time constant and the per-step address arithmetic drops to a few adds.
template <typename R, int RZ, int MODE, bool YB, bool TB, int GY = 0, int GZ = 0>
__global__ void __launch_bounds__(512) k_hpsi_pass(const PassArgs<R> a) {
  static_assert(!TB || RZ == 2, "table staging copies the two points' entries as one run");
  static_assert(GZ == 0 || (std::is_same<R, float>::value && TB && !YB), "fixed shapes: complex(4) table form, no y-blocks");
  using T = C2<R>;
  constexpr bool FIXED = GZ > 0;
  constexpr int NR = FIXED ? 9 : PassGeom<R>::NR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NLy = FIXED ? GY : a.NLy, NLz = FIXED ? GZ : a.NLz, NYZ = NLy * NLz;
  const bool with_w = a.W != nullptr;
  const bool do_export = a.S != nullptr;
  const int NYBc = YB ? a.NYB : NLy;  // rows of a y-block
  const int nyblk = YB ? a.nyblk : 1;
  const int RYZ = YB ? (NYBc + 8) * NLz : NYZ;  // ring plane size
  T* ring = reinterpret_cast<T*>(smem_raw);
  T* wring = ring + (size_t)NR * RYZ;  // [NR][maxpts] W chunks of the ring's planes
  constexpr bool tab = TB;
  const int TYZ = YB ? NYBc * NLz : NYZ;  // table plane size (owned rows)
  R* vtab = reinterpret_cast<R*>(wring + (with_w ? (size_t)NR * a.maxpts : 0));  // [NR][TYZ] (tab)
  short* lqtab = reinterpret_cast<short*>(vtab + (tab ? (size_t)NR * TYZ : 0));    // [NR][TYZ] (tab)
  // sp_off[0..NLx] (or sp_blk in the YB form)
  int* spo = reinterpret_cast<int*>(lqtab + (tab ? (size_t)NR * TYZ : 0));
  if constexpr (YB) {
    for (int i = threadIdx.x; i < a.NLx * (nyblk + 1); i += blockDim.x) spo[i] = a.sp_blk[i];
  } else {
    for (int i = threadIdx.x; i <= a.NLx; i += blockDim.x) spo[i] = a.sp_off[i];
  }
  __syncthreads();

  const int b = YB ? blockIdx.x / nyblk : blockIdx.x;
  const int yb = YB ? blockIdx.x - b * nyblk : 0;
  const int y0 = YB ? yb * NYBc : 0;
  const int o = a.o_beg + b;
  const int kl = o / a.NBocc;
  const double kxd = a.kAc[3 * kl], kyd = a.kAc[3 * kl + 1], kzd = a.kAc[3 * kl + 2];
  const R A = (R)((kxd * kxd + kyd * kyd + kzd * kzd - a.lap0sum) * 0.5);  // k2lap0_2 (hpsi.f90:120-121)
  // nabt = k_d nab_d (hpsi.f90:122-124), applied once per axis:
  // w = sum_d k_d sum_n nab_d,n (psi(+n) - psi(-n))
  using KT = typename std::conditional<std::is_same<R, float>::value, float2, double>::type;
  const KT kx = kpair<R>(kxd), ky = kpair<R>(kyd), kz = kpair<R>(kzd);
  // FD coefficients: broadcast pairs for complex(4), scalars for complex(8)
  auto CL = [&](int i) -> KT {
    if constexpr (std::is_same<R, float>::value) return a.cl2[i]; else return a.lapt[i];
  };
  auto CN = [&](int i) -> KT {
    if constexpr (std::is_same<R, float>::value) return a.cn2[i]; else return a.nabc[i];
  };

  const int NZG = NLz / RZ;
  const int t = threadIdx.x;
  const int bd = blockDim.x;
  const int ny_own = YB ? min(NYBc, NLy - y0) : NLy;
  const bool act = t < ny_own * NZG;
  const int yl = act ? t / NZG : 0;  // row in the block
  const int y = y0 + yl;             // row in the plane
  const int z0 = act ? (t - yl * NZG) * RZ : 0;
  const int own = y * NLz + z0;                       // in the plane
  const int own_r = YB ? (4 + yl) * NLz + z0 : own;   // in the ring
  const int own_t = YB ? yl * NLz + z0 : own;         // in the table planes

  const int x_beg = blockIdx.y * a.SX;
  const int x_end = min(x_beg + a.SX, a.NLx);
  if (x_beg >= x_end) return;  // whole CTA leaves together
  const int nplanes = x_end - x_beg + 4;  // planes the ring delivers: x_beg .. x_end+3
  const int nown = x_end - x_beg;         // planes that need W
  const T* inb = a.in + (size_t)b * a.NL;
  const T* Wb = with_w ? a.W + (size_t)b * a.nsp : nullptr;
  T* Sb = do_export ? a.S + (size_t)b * a.nsp : nullptr;

  // plane jn (relative to x_beg) into ring slot sl (= jn modulo the ring), with its W chunk
  auto refill = [&](int jn, int sl) {
    int p = x_beg + jn;
    while (p >= a.NLx) p -= a.NLx;
    if constexpr (YB) {
      if (jn < nplanes) {  // the block's rows and the halo rows, periodic in y
        T* dst = ring + (size_t)sl * RYZ;
        const T* src = inb + (size_t)p * NYZ;
        for (int idx = t; idx < (NYBc + 8) * NZG; idx += bd) {
          const int r = idx / NZG, zz = (idx - r * NZG) * RZ;
          int gy = y0 - 4 + r;
          gy += gy < 0 ? NLy : 0;
          gy -= gy >= NLy ? NLy : 0;
          cp_run<R, RZ>(dst + r * NLz + zz, src + gy * NLz + zz);
        }
      }
    } else {
      if (act && jn < nplanes) cp_run<R, RZ>(ring + (size_t)sl * NYZ + own, inb + (size_t)p * NYZ + own);
    }
    if constexpr (TB) {
      if (act && jn < nown) {
        const size_t g = (size_t)p * NYZ + own;
        R* vd = vtab + (size_t)sl * TYZ + own_t;
        if constexpr (sizeof(R) == 4) cp_async8(vd, a.vloc + g); else cp_async16(vd, a.vloc + g);
        if (with_w || do_export) cp_async4(lqtab + (size_t)sl * TYZ + own_t, a.lqi + g);
      }
    }
    if (with_w && jn < nown) {
      const int q0 = YB ? spo[p * (nyblk + 1) + yb] : spo[p];
      const int q1 = YB ? spo[p * (nyblk + 1) + yb + 1] : spo[p + 1];
      T* dst = wring + (size_t)sl * a.maxpts;
      for (int qq = q0 + t; qq < q1; qq += bd) cp_run<R, 1>(dst + (qq - q0), Wb + qq);
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int n = 0; n < NR - 1; ++n) refill(n, n);

  int yo[8];  // ring offsets of the y neighbours
#pragma unroll
  for (int n = 1; n <= 4; ++n) {
    yo[n - 1] = (YB ? 4 + yl + n : wrapi(y + n, NLy)) * NLz + z0;
    yo[3 + n] = (YB ? 4 + yl - n : wrapi(y - n, NLy)) * NLz + z0;
  }
  constexpr int NZZ = RZ + 8;  // z runs start at z0-4, z0-4+RZ, ..., z0+4
  int zoff[NZZ / RZ];
#pragma unroll
  for (int m = 0; m < NZZ / RZ; ++m) zoff[m] = (YB ? 4 + yl : y) * NLz + wrapi(z0 + m * RZ - 4, NLz);

  // register queue: in the march step of phase P (plane x = x_beg + 9i + P),
  // plane x-4+m sits in q[(P+m) % 9]; the march is unrolled nine times so the
  // queue rotates by renaming, without register moves.
  T q[9][RZ];
  if (act) {
#pragma unroll
    for (int n = 0; n < 4; ++n) ld_run<R, RZ>(q[n], inb + (size_t)wrapi(x_beg - 4 + n, a.NLx) * NYZ + own);
  }
  R vl[RZ];    // Vloc of the current plane, loaded one plane ahead
  int lq[RZ];  // local sphere indices of the current plane, loaded one plane ahead
#pragma unroll
  for (int r = 0; r < RZ; ++r) { vl[r] = (R)0; lq[r] = -1; }
  if (act && !TB) {
#pragma unroll
    for (int r = 0; r < RZ; ++r) vl[r] = __ldg(a.vloc + (size_t)x_beg * NYZ + own + r);
    if (with_w || do_export) ld_lq<RZ>(lq, a.lqi + (size_t)x_beg * NYZ + own);
  }

  int x = x_beg;
  auto step = [&](auto phase) -> bool {
    constexpr int P = decltype(phase)::value;
    const int j = x - x_beg;
    // ring slot of plane j+k: with one slot per phase (j modulo 9 is P) a constant
    auto slot = [&](int k) -> int { return FIXED ? (P + k) % NR : (j + k) % NR; };
    const int s0 = slot(0);
    cp_async_wait<NR - 6>();  // this thread's copies of planes <= x+4 have landed
    __syncthreads();          // ... and everyone's; the slot of plane x-1 is free
    refill(j + NR - 1, slot(NR - 1));
    const T* pl = ring + (size_t)s0 * RYZ;
    if (act) {
      if constexpr (P == 0) {
        if (j == 0) {
#pragma unroll
          for (int n = 4; n < 8; ++n) lds_run<R, RZ>(q[n], ring + (size_t)(n - 4) * RYZ + own_r);
        }
      }
      lds_run<R, RZ>(q[(P + 8) % 9], ring + (size_t)slot(4) * RYZ + own_r);
      const size_t pbase = (size_t)x * NYZ + own;
      R vln[RZ];
      int lqn[RZ];
#pragma unroll
      for (int r = 0; r < RZ; ++r) { vln[r] = (R)0; lqn[r] = -1; }
      if constexpr (TB) {  // this plane's tables arrived with it (copy group j)
        const R* vs = vtab + (size_t)s0 * TYZ + own_t;
#pragma unroll
        for (int r = 0; r < RZ; ++r) vl[r] = vs[r];
        if (with_w || do_export) {
          const int v2 = *reinterpret_cast<const int*>(lqtab + (size_t)s0 * TYZ + own_t);
          lq[0] = (int)(short)(v2 & 0xffff);
          lq[RZ - 1] = v2 >> 16;
        }
      } else if (x + 1 < x_end) {
#pragma unroll
        for (int r = 0; r < RZ; ++r) vln[r] = __ldg(a.vloc + pbase + NYZ + r);
        if (with_w || do_export) ld_lq<RZ>(lqn, a.lqi + pbase + NYZ);
      }
      T v[RZ], w[RZ], wa[RZ];
#pragma unroll
      for (int r = 0; r < RZ; ++r) { v[r] = mk<R>(0, 0); wa[r] = mk<R>(0, 0); }
      if constexpr (std::is_same<R, float>::value) {
        // z: the values z0-4 .. z0+RZ+3 of plane x (the centre run from the queue), as pairs
        T zv[NZZ];
#pragma unroll
        for (int m = 0; m < NZZ / RZ; ++m) {
          T run[RZ];
          if (m * RZ == 4) {
#pragma unroll
            for (int s2 = 0; s2 < RZ; ++s2) run[s2] = q[(P + 4) % 9][s2];
          } else {
            lds_run<R, RZ>(run, pl + zoff[m]);
          }
#pragma unroll
          for (int s2 = 0; s2 < RZ; ++s2) zv[m * RZ + s2] = run[s2];
        }
#pragma unroll
        for (int n = 1; n <= 4; ++n)
#pragma unroll
          for (int r = 0; r < RZ; ++r) stencil_pair(v[r], wa[r], zv[4 + r + n], zv[4 + r - n], CL(8 + n - 1), CN(8 + n - 1));
      } else {
#pragma unroll
        for (int m = 0; m < NZZ / RZ; ++m) {  // z: each value feeds every point it neighbours, as it arrives
          T run[RZ];
          if (m * RZ == 4) {
#pragma unroll
            for (int s2 = 0; s2 < RZ; ++s2) run[s2] = q[(P + 4) % 9][s2];
          } else {
            lds_run<R, RZ>(run, pl + zoff[m]);
          }
#pragma unroll
          for (int s2 = 0; s2 < RZ; ++s2)
#pragma unroll
            for (int r = 0; r < RZ; ++r) {
              const int k = m * RZ + s2 - 4 - r;
              if (k != 0 && k >= -4 && k <= 4) {
                const int n = k > 0 ? k : -k;
                const R cl = a.lapt[7 + n];
                const R cn = k > 0 ? a.nabc[7 + n] : -a.nabc[7 + n];
                v[r].x = fma(cl, run[s2].x, v[r].x);
                v[r].y = fma(cl, run[s2].y, v[r].y);
                wa[r].x = fma(cn, run[s2].x, wa[r].x);
                wa[r].y = fma(cn, run[s2].y, wa[r].y);
              }
            }
        }
      }
#pragma unroll
      for (int r = 0; r < RZ; ++r) { w[r] = kscale(kz, wa[r], mk<R>(0, 0)); wa[r] = mk<R>(0, 0); }
      // the y terms go to a second accumulator (fixed shapes): two shorter FMA
      // chains (0.469 -> 0.438 ms at 32^3)
      constexpr bool SPLITV = FIXED;
      T vy[RZ];
#pragma unroll
      for (int r = 0; r < RZ; ++r) vy[r] = mk<R>(0, 0);
#pragma unroll
      for (int n = 1; n <= 4; ++n) {  // y
        T rp[RZ], rm[RZ];
        lds_run<R, RZ>(rp, pl + yo[n - 1]);
        lds_run<R, RZ>(rm, pl + yo[3 + n]);
#pragma unroll
        for (int r = 0; r < RZ; ++r) stencil_pair(SPLITV ? vy[r] : v[r], wa[r], rp[r], rm[r], CL(4 + n - 1), CN(4 + n - 1));
      }
#pragma unroll
      for (int r = 0; r < RZ; ++r) { w[r] = kscale(ky, wa[r], w[r]); wa[r] = mk<R>(0, 0); }
#pragma unroll
      for (int n = 1; n <= 4; ++n)  // x: the register queue
#pragma unroll
        for (int r = 0; r < RZ; ++r)
          stencil_pair(v[r], wa[r], q[(P + 4 + n) % 9][r], q[(P + 4 - n) % 9][r], CL(n - 1), CN(n - 1));
#pragma unroll
      for (int r = 0; r < RZ; ++r) w[r] = kscale(kx, wa[r], w[r]);
      if constexpr (SPLITV) {
#pragma unroll
        for (int r = 0; r < RZ; ++r) v[r] = cadd(v[r], vy[r]);
      }

      // plane-relative sphere index lq -> this block's W chunk
      const T* wpl = wring + (size_t)s0 * a.maxpts -
                     (YB ? spo[x * (nyblk + 1) + yb] - spo[x * (nyblk + 1)] : 0);
      T res[RZ];
#pragma unroll
      for (int r = 0; r < RZ; ++r) {
        const T c = q[(P + 4) % 9][r];
        // F = B E + A E - 0.5 v - zI w   (stencil/F90/hpsi.f90:190)
        T f;
        f.x = fma(vl[r] + A, c.x, fma((R)-0.5, v[r].x, w[r].y));
        f.y = fma(vl[r] + A, c.y, fma((R)-0.5, v[r].y, -w[r].x));
        if constexpr (MODE == 1) {  // ttpsi = H tpsi - Vloc tpsi before pseudo_pt (hpsi.f90:131-133)
          a.tt[(size_t)b * a.NL + pbase + r] = mk<R>(fma(-vl[r], c.x, f.x), fma(-vl[r], c.y, f.y));
        }
        if (with_w && lq[r] >= 0) f = cadd(f, wpl[lq[r]]);  // + pseudo_pt scatter (hpsi.f90:203-206)
        res[r] = f;
      }
      if constexpr (MODE == 2) {  // one Taylor stage: out = in + c H in
#pragma unroll
        for (int r = 0; r < RZ; ++r) res[r] = cfma(a.zf, res[r], q[(P + 4) % 9][r]);
      }
      st_run<R, RZ>(a.out + (size_t)b * a.NL + pbase, res);
      if (do_export) {  // the output at the sphere points, for the next projections
        const int q0 = YB ? spo[x * (nyblk + 1)] : spo[x];
#pragma unroll
        for (int r = 0; r < RZ; ++r)
          if (lq[r] >= 0) Sb[q0 + lq[r]] = res[r];
      }
      if constexpr (!TB) {
#pragma unroll
        for (int r = 0; r < RZ; ++r) { vl[r] = vln[r]; lq[r] = lqn[r]; }
      }
    }
    ++x;
    return x < x_end;
  };
  for (;;) {
    if (!step(std::integral_constant<int, 0>{})) break;
    if (!step(std::integral_constant<int, 1>{})) break;
    if (!step(std::integral_constant<int, 2>{})) break;
    if (!step(std::integral_constant<int, 3>{})) break;
    if (!step(std::integral_constant<int, 4>{})) break;
    if (!step(std::integral_constant<int, 5>{})) break;
    if (!step(std::integral_constant<int, 6>{})) break;
    if (!step(std::integral_constant<int, 7>{})) break;
    if (!step(std::integral_constant<int, 8>{})) break;
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------- two rows a thread --
// The pass at compile-time plane shapes, one CTA per (orbital, block of GB rows): a thread
// owns the points of two consecutive y rows, at two z points (complex(4)) or one
// (complex(8)).
//
// k_hpsi_pass at these shapes is held by shared-memory wavefronts and latency, not by one
// peak: it reads 13 values of shared memory a point (8 rows of y neighbours for two points,
// the plane four ahead for the queue; in complex(8) its two z points lie 32 bytes apart, so
// half of the wavefronts are bank conflicts) from a ring that, with its tables, leaves room
// for one CTA per SM.  Here
//   * the ten rows y0-4 .. y0+5 serve both of the thread's rows, two of them from its own
//     registers, and the step's address arithmetic, table loads and barrier are shared by
//     the rows; complex(8) lanes read consecutive 16-byte values;
//   * the thread's own column comes from global memory straight into the register queue
//     (plane x+5 while plane x is worked on, into the slot of plane x-4, whose last use, the
//     x terms, comes first; hinted into L2 three planes earlier) and goes from there to
//     shared memory when its plane is due, so shared memory holds three planes instead of
//     nine: several small CTAs per SM, whose barriers fall at different times;
//   * the halo rows of a block, the plane's V_loc, sphere indices and W chunk are copied by
//     cp.async two planes ahead;
//   * the march is unrolled three times only, with the queue moved down by three planes in
//     the third step: nine renamed phases are 67 KB of code, and waits for instructions were
//     the second largest stall.
// The x terms are added first, and the sum starts at the centre term (see m2A).  One second
// derivative accumulator per point: a second one for y, as in k_hpsi_pass, spills at three
// CTAs per SM (0.412 against 0.377 ms at 32^3).  Complex(8) adds the small terms first and
// starts the first derivatives by a product, complex(4) neither: whichever spilled least (no
// complex(4) instance spills; ten of the sixteen complex(8) ones do, 4 to 24 bytes, of the
// Taylor stages with KB the 16x16 one).  KB: W and S are both given (a Taylor stage).  Measured times: see pass2_rows.
constexpr int P2_NS = 3;  // planes in shared memory = phases of the unrolled march

template <typename R> struct P2Geom { static constexpr int RZ = std::is_same<R, float>::value ? 2 : 1; };

template <typename R, int MODE, bool KB, int GY, int GZ, int GB, int MB>
__global__ void __launch_bounds__(((GB / 2 * (GZ / P2Geom<R>::RZ) + 31) / 32) * 32, MB) k_hpsi_pass2(const PassArgs<R> a) {
  using T = C2<R>;
  constexpr bool F = std::is_same<R, float>::value;
  constexpr int RZ = P2Geom<R>::RZ;
  constexpr bool YB = GB < GY;
  constexpr int NYZ = GY * GZ, NZG = GZ / RZ, nyblk = GY / GB, NTA = GB / 2 * NZG, NT = ((NTA + 31) / 32) * 32;
  constexpr int RYZ = (YB ? GB + 8 : GY) * GZ, TYZ = GB * GZ;  // shared plane and table sizes
  static_assert(GY % GB == 0 && GB % 2 == 0 && GZ % 2 == 0 && GY >= 8 && GZ >= 8, "whole row pairs, no double wrap");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const bool with_w = KB || a.W != nullptr;
  const bool do_export = KB || a.S != nullptr;
  T* planes = reinterpret_cast<T*>(smem_raw);                       // [NS][RYZ]
  T* wtab = planes + P2_NS * RYZ;                                   // [NS][maxpts] W chunks
  R* vtab = reinterpret_cast<R*>(wtab + (with_w ? P2_NS * a.maxpts : 0));  // [NS][TYZ]
  short* lqtab = reinterpret_cast<short*>(vtab + P2_NS * TYZ);      // [NS][TYZ]
  int* spo = reinterpret_cast<int*>(lqtab + P2_NS * TYZ);           // [NLx][nyblk+1] sphere points
  const int t = threadIdx.x;
  for (int i = t; i < a.NLx * (nyblk + 1); i += NT) spo[i] = a.sp_blk[i];
  __syncthreads();

  const int b = blockIdx.x / nyblk, yb = blockIdx.x - b * nyblk;
  const int kl = (a.o_beg + b) / a.NBocc;
  const double kxd = a.kAc[3 * kl], kyd = a.kAc[3 * kl + 1], kzd = a.kAc[3 * kl + 2];
  // the sum v starts at -2 k2lap0_2 psi (hpsi.f90:120-121), so that it shrinks as the
  // neighbours come in and the large terms cancel inside it, not after it: in complex(4) a
  // step's error against 64 bits is below that of a sum from zero
  using KT = typename std::conditional<F, float2, double>::type;
  const KT m2A = kpair<R>(a.lap0sum - (kxd * kxd + kyd * kyd + kzd * kzd));
  const KT kx = kpair<R>(kxd), ky = kpair<R>(kyd), kz = kpair<R>(kzd);
  auto CL = [&](int n) -> KT { if constexpr (F) return a.cl2[n]; else return a.lapt[n]; };
  auto CN = [&](int n) -> KT { if constexpr (F) return a.cn2[n]; else return a.nabc[n]; };

  const bool act = NT == NTA || t < NTA;
  const int yl = act ? 2 * (t / NZG) : 0;      // first row in the block
  const int z0 = act ? RZ * (t % NZG) : 0;
  const int own = (yb * GB + yl) * GZ + z0;    // in the plane; the second row is own + GZ
  const int own_r = ((YB ? 4 : 0) + yl) * GZ + z0;
  const int own_t = yl * GZ + z0;

  const int x_beg = blockIdx.y * a.SX, x_end = min(x_beg + a.SX, a.NLx);
  if (x_beg >= x_end) return;  // whole CTA leaves together
  const T* inb = a.in + (size_t)b * a.NL;
  const T* Wb = with_w ? a.W + (size_t)b * a.nsp : nullptr;
  T* Sb = do_export ? a.S + (size_t)b * a.nsp : nullptr;

  // halo rows, tables and W chunk of plane p (x_beg <= p < x_end) into slot sl
  auto fetch = [&](int p, int sl) {
    if (p < x_end) {
      if constexpr (YB) {
        for (int idx = t; idx < 8 * NZG; idx += NT) {
          const int r = idx / NZG, zz = (idx - r * NZG) * RZ;
          int gy = yb * GB + (r < 4 ? r - 4 : GB + r - 4);
          gy += gy < 0 ? GY : 0;
          gy -= gy >= GY ? GY : 0;
          cp_async16(planes + sl * RYZ + (r < 4 ? r : GB + r) * GZ + zz, inb + (size_t)p * NYZ + gy * GZ + zz);
        }
      }
      if (act) {
        const size_t g = (size_t)p * NYZ + own;
        R* vd = vtab + sl * TYZ + own_t;
        cp_async8(vd, a.vloc + g);
        cp_async8(vd + GZ, a.vloc + g + GZ);
        if ((with_w || do_export) && (RZ == 2 || z0 % 2 == 0)) {  // (a pair of points per copy)
          short* ld = lqtab + sl * TYZ + own_t;
          cp_async4(ld, a.lqi + g);
          cp_async4(ld + GZ, a.lqi + g + GZ);
        }
      }
      if (with_w) {
        const int q0 = spo[p * (nyblk + 1) + yb], q1 = spo[p * (nyblk + 1) + yb + 1];
        T* dst = wtab + sl * a.maxpts;
        for (int qq = q0 + t; qq < q1; qq += NT) cp_run<R, 1>(dst + (qq - q0), Wb + qq);
      }
    }
    cp_async_commit();
  };
  fetch(x_beg, 0);
  fetch(x_beg + 1, 1);

  // shared-plane offsets of the rows yl-4 .. yl-1 and yl+2 .. yl+5, and of the runs of RZ
  // points around z0
  int yo[8];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int rm = yl - 4 + n, rp = yl + 2 + n;
    yo[n] = (YB ? 4 + rm : (rm < 0 ? rm + GY : rm)) * GZ + z0;
    yo[4 + n] = (YB ? 4 + rp : (rp >= GY ? rp - GY : rp)) * GZ + z0;
  }
  constexpr int NZR = 8 / RZ;  // runs z0-4, .., z0-RZ and z0+RZ, .., z0+4
  int zo[NZR];
#pragma unroll
  for (int m = 0; m < NZR; ++m) {
    int zz = z0 + (m < NZR / 2 ? RZ * m - 4 : RZ * (m - NZR / 2 + 1));
    zz += zz < 0 ? GZ : 0;
    zz -= zz >= GZ ? GZ : 0;
    zo[m] = own_r - z0 + zz;
  }

  T q[9][2][RZ];  // in step P: plane x-4+m at [P+m] before the x terms (moved down after the third step's)
  const T* col = inb + own;
  if (act) {
#pragma unroll
    for (int n = 0; n < 9; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) ld_run<R, RZ>(q[n][r], col + (size_t)wrapi(x_beg - 4 + n, a.NLx) * NYZ + r * GZ);
  }
  T qn[2][2][RZ];  // planes x+5 of the first two steps: q[9], q[10]
  auto Q = [&](int m) -> T(&)[2][RZ] { return m < 9 ? q[m] : qn[m - 9]; };
  int x = x_beg;
  int xq = wrapi(x_beg + 5, a.NLx);  // the plane that enters the queue in this step
  int xp = wrapi(x_beg + 8, a.NLx);  // the plane hinted into L2
  auto step = [&](auto phase) -> bool {
    constexpr int P = decltype(phase)::value;
    constexpr int sl = P, sl2 = (P + 2) % P2_NS;
    T* pl = planes + sl * RYZ;
    T c[2][RZ], v[2][RZ], w[2][RZ], wa[2][RZ];
    if (act) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int s = 0; s < RZ; ++s) {
          c[r][s] = Q(P + 4)[r][s];
          v[r][s] = kscale(m2A, c[r][s], mk<R>(0, 0));
          if constexpr (F) wa[r][s] = mk<R>(0, 0);
        }
        st_run<R, RZ>(pl + own_r + r * GZ, c[r]);
      }
#pragma unroll
      for (int m = 1; m <= 4; ++m) {  // x: the register queue
        const int n = F ? m : 5 - m;  // (constant after unrolling)
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int s = 0; s < RZ; ++s)
            if (!F && m == 1) stencil_pair_first<false, true>(v[r][s], wa[r][s], Q(P + 8)[r][s], Q(P)[r][s], CL(3), CN(3));
            else stencil_pair(v[r][s], wa[r][s], Q(P + 4 + n)[r][s], Q(P + 4 - n)[r][s], CL(n - 1), CN(n - 1));
      }
      if constexpr (P == 2) {  // planes x-3 .. x+4 to the front; plane x+5 arrives behind them
#pragma unroll
        for (int m = 0; m < 8; ++m)
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int s = 0; s < RZ; ++s) q[m][r][s] = Q(m + 3)[r][s];
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (x + 1 < x_end) ld_run<R, RZ>(P < 2 ? qn[P < 2 ? P : 0][r] : q[8][r], col + (size_t)xq * NYZ + r * GZ);
#pragma unroll
        for (int s = 0; s < RZ; ++s) {
          w[r][s] = kscale(kx, wa[r][s], mk<R>(0, 0));
          if constexpr (F) wa[r][s] = mk<R>(0, 0);
        }
      }
    }
    if (t == 0) prefetch_l2_bulk(inb + (size_t)xp * NYZ + (YB ? yb * GB * GZ : 0), TYZ * sizeof(T));
    xq = xq + 1 < a.NLx ? xq + 1 : 0;
    xp = xp + 1 < a.NLx ? xp + 1 : 0;
    cp_async_wait<1>();  // this thread's copies of plane x have landed
    __syncthreads();     // ... everyone's, and every column's values; plane x-1 is no longer read
    fetch(x + 2, sl2);
    if (act) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {  // z
        T zv[RZ + 8];
#pragma unroll
        for (int m = 0; m < NZR; ++m) {
          T run[RZ];
          lds_run<R, RZ>(run, pl + zo[m] + r * GZ);
#pragma unroll
          for (int s = 0; s < RZ; ++s) zv[RZ * (m < NZR / 2 ? m : m + 1) + s] = run[s];
        }
#pragma unroll
        for (int s = 0; s < RZ; ++s) zv[4 + s] = c[r][s];
#pragma unroll
        for (int m = 1; m <= 4; ++m) {
          const int n = F ? m : 5 - m;  // (constant after unrolling)
#pragma unroll
          for (int s = 0; s < RZ; ++s)
            if (!F && m == 1) stencil_pair_first<false, true>(v[r][s], wa[r][s], zv[8 + s], zv[s], CL(11), CN(11));
            else stencil_pair(v[r][s], wa[r][s], zv[4 + s + n], zv[4 + s - n], CL(7 + n), CN(7 + n));
        }
#pragma unroll
        for (int s = 0; s < RZ; ++s) {
          w[r][s] = kscale(kz, wa[r][s], w[r][s]);
          if constexpr (F) wa[r][s] = mk<R>(0, 0);
        }
      }
      {  // y: rows yl-4 .. yl+5, the thread's own two from the queue
        T yv[10][RZ];
#pragma unroll
        for (int n = 0; n < 4; ++n) lds_run<R, RZ>(yv[n], pl + yo[n]);
#pragma unroll
        for (int s = 0; s < RZ; ++s) { yv[4][s] = c[0][s]; yv[5][s] = c[1][s]; }
#pragma unroll
        for (int n = 0; n < 4; ++n) lds_run<R, RZ>(yv[6 + n], pl + yo[4 + n]);
#pragma unroll
        for (int m = 1; m <= 4; ++m) {
          const int n = F ? m : 5 - m;  // (constant after unrolling)
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int s = 0; s < RZ; ++s)
              if (!F && m == 1) stencil_pair_first<false, true>(v[r][s], wa[r][s], yv[8 + r][s], yv[r][s], CL(7), CN(7));
              else stencil_pair(v[r][s], wa[r][s], yv[4 + r + n][s], yv[4 + r - n][s], CL(3 + n), CN(3 + n));
        }
      }
      const size_t pbase = (size_t)b * a.NL + (size_t)x * NYZ + own;
      const int qp = spo[x * (nyblk + 1)];  // the plane's first sphere point
      // plane-relative sphere index lq -> this block's W chunk
      const T* wpl = wtab + sl * a.maxpts - (YB ? spo[x * (nyblk + 1) + yb] - qp : 0);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        R vl[RZ];
#pragma unroll
        for (int s = 0; s < RZ; ++s) vl[s] = vtab[sl * TYZ + own_t + r * GZ + s];
        int lq[RZ];
#pragma unroll
        for (int s = 0; s < RZ; ++s) lq[s] = -1;
        if (with_w || do_export) {
          const short* ls = lqtab + sl * TYZ + own_t + r * GZ;
          if constexpr (RZ == 2) {
            const int v2 = *reinterpret_cast<const int*>(ls);
            lq[0] = (int)(short)(v2 & 0xffff);
            lq[RZ - 1] = v2 >> 16;
          } else {
            lq[0] = ls[0];
          }
        }
        T res[RZ];
#pragma unroll
        for (int s = 0; s < RZ; ++s) {
          const T ww = kscale(ky, wa[r][s], w[r][s]), vv = v[r][s], cc = c[r][s];
          // F = B E + A E - 0.5 v - zI w   (stencil/F90/hpsi.f90:190), A E inside v
          T f;
          f.x = fma(vl[s], cc.x, fma((R)-0.5, vv.x, ww.y));
          f.y = fma(vl[s], cc.y, fma((R)-0.5, vv.y, -ww.x));
          if constexpr (MODE == 1)  // ttpsi = H tpsi - Vloc tpsi before pseudo_pt (hpsi.f90:131-133)
            a.tt[pbase + r * GZ + s] = mk<R>(fma(-vl[s], cc.x, f.x), fma(-vl[s], cc.y, f.y));
          if (with_w && lq[s] >= 0) f = cadd(f, wpl[lq[s]]);  // + pseudo_pt scatter (hpsi.f90:203-206)
          res[s] = MODE == 2 ? cfma(a.zf, f, cc) : f;         // mode 2: one Taylor stage
        }
        st_run<R, RZ>(a.out + pbase + r * GZ, res);
        if (do_export) {
#pragma unroll
          for (int s = 0; s < RZ; ++s)
            if (lq[s] >= 0) Sb[qp + lq[s]] = res[s];
        }
      }
    }
    ++x;
    return x < x_end;
  };
  for (;;) {
    if (!step(std::integral_constant<int, 0>{})) break;
    if (!step(std::integral_constant<int, 1>{})) break;
    if (!step(std::integral_constant<int, 2>{})) break;
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------- launch ---
// Vloc and sphere-index tables through the ring: two-point form, when both
// precisions' rings still fit in shared memory with them
static bool pass_tables(const System& s, int RZ) {
  if (RZ != 2 || !s.pass_tab) return false;
  const int NYB = s.nyblk > 1 ? s.NYB : s.NLy;
  for (int pr = 0; pr < 2; ++pr)
    if (pass_smem_bytes(pr, s.NLy, s.NLz, s.maxpts, true, s.NLx, s.nyblk, NYB, true) > 227 * 1024) return false;
  return true;
}

// plane shapes with a compile-time form of k_hpsi_pass (complex(4), table form, without
// y-blocks): 16x16 and 20x20.  (The larger ones have the two-row pass.)
static int fixed_shape(int NLy, int NLz, int nyblk) {
  if (nyblk > 1) return 0;
  if (NLy == 16 && NLz == 16) return 1;
  if (NLy == 20 && NLz == 20) return 2;
  return 0;
}

template <typename R, int RZ, int MODE>
static void (*pass_kernel(bool yb, bool tb, int shape))(const PassArgs<R>) {
  if constexpr (RZ == 2 && std::is_same<R, float>::value) {
    if (tb && !yb) {
      switch (shape) {
        case 1: return k_hpsi_pass<R, RZ, MODE, false, true, 16, 16>;
        case 2: return k_hpsi_pass<R, RZ, MODE, false, true, 20, 20>;
        default: break;
      }
    }
  }
  if constexpr (RZ == 2) {
    if (tb) return yb ? k_hpsi_pass<R, RZ, MODE, true, true> : k_hpsi_pass<R, RZ, MODE, false, true>;
  }
  return yb ? k_hpsi_pass<R, RZ, MODE, true, false> : k_hpsi_pass<R, RZ, MODE, false, false>;
}

// the compile-time shape the pass uses for this system and precision (0: none);
// its 9-plane ring must fit in shared memory
template <typename R, int RZ>
static int pass_shape(const System& s, bool tb) {
  if (!std::is_same<R, float>::value || RZ != 2 || !tb || !s.pass_fixed) return 0;
  const int sh = fixed_shape(s.NLy, s.NLz, s.nyblk);
  const int nyb = s.nyblk > 1 ? s.NYB : s.NLy;
  if (sh && pass_smem_bytes(SGPU_PREC_C64, s.NLy, s.NLz, s.maxpts, true, s.NLx, s.nyblk, nyb, true, 9) > 227 * 1024)
    return 0;
  return sh;
}

// Rows of a block of the two-row pass (0: no such form for this plane shape).  One Taylor
// stage, two-row form against k_hpsi_pass, ms: complex(4) 32^3 x 2048 orbitals 0.385 / 0.454
// (blocks of 8 rows: 0.419), 48^3 x 1728 1.12 / 1.60 (8 rows: 1.18), 16x16x32 x 1024
// 0.055 / 0.067; slower on 16x16 (0.041 / 0.034) and 20x20 planes (0.29 / 0.15: 100 points'
// threads in four warps), which keep k_hpsi_pass.  Complex(8) 32^3 x 2048 0.907 / 1.248 (16
// rows: 1.05), 48^3 x 800 1.17 / 1.98, 16x16x32 x 1024 0.125 / 0.172 (16 rows: 0.145), 16^3 x
// 1024 0.069 / 0.087; 20^3 x 2048 0.39 / 0.32, not taken.
int pass2_rows(int prec, int NLy, int NLz) {
  if (NLy == 32 && NLz == 32) return prec == SGPU_PREC_C64 ? 16 : 8;
  if (NLy == 48 && NLz == 48) return prec == SGPU_PREC_C64 ? 16 : 8;
  if (NLy == 16 && NLz == 32) return prec == SGPU_PREC_C64 ? 16 : 8;
  if (NLy == 16 && NLz == 16) return prec == SGPU_PREC_C64 ? 0 : 16;
  return 0;
}
template <typename R, int MODE, bool KB>
static void (*pass2_kernel(int NLy, int NLz))(const PassArgs<R>) {
  if constexpr (std::is_same<R, float>::value) {
    if (NLy == 32) return k_hpsi_pass2<R, MODE, KB, 32, 32, 16, 3>;
    if (NLy == 48) return k_hpsi_pass2<R, MODE, KB, 48, 48, 16, 2>;
    return k_hpsi_pass2<R, MODE, KB, 16, 32, 16, 3>;
  } else {
    if (NLy == 32) return k_hpsi_pass2<R, MODE, KB, 32, 32, 8, 3>;
    if (NLy == 48) return k_hpsi_pass2<R, MODE, KB, 48, 48, 8, 2>;
    if (NLz == 32) return k_hpsi_pass2<R, MODE, KB, 16, 32, 8, 3>;
    return k_hpsi_pass2<R, MODE, KB, 16, 16, 16, 3>;
  }
}
template <typename R>
static size_t pass2_smem(const System& s, bool with_w) {
  constexpr int pr = std::is_same<R, float>::value ? SGPU_PREC_C64 : SGPU_PREC_C128;
  const int rows = s.p2_rows[pr], nblk = s.NLy / rows;
  const size_t ryz = (size_t)(nblk > 1 ? rows + 8 : s.NLy) * s.NLz, tyz = (size_t)rows * s.NLz;
  return P2_NS * (ryz * sizeof(C2<R>) + tyz * (sizeof(R) + sizeof(short)) +
                  (with_w ? (size_t)s.p2_maxpts[pr] * sizeof(C2<R>) : 0)) +
         sizeof(int) * (size_t)s.NLx * (nblk + 1);
}
template <typename R>
static bool pass2_fits(const System& s) {
  constexpr int pr = std::is_same<R, float>::value ? SGPU_PREC_C64 : SGPU_PREC_C128;
  return s.p2_rows[pr] > 0 && s.pass_fixed && s.pass_tab && pass2_smem<R>(s, true) <= 227 * 1024;
}

template <typename R, int RZ, int MODE>
static cudaError_t launch_pass_t(const System& s, const PassIO& io, int o_beg, int nb, int nbk) {
  PassArgs<R> a;
  a.in = (const C2<R>*)io.in;
  a.out = (C2<R>*)io.out;
  a.tt = (C2<R>*)io.tt;
  a.vloc = std::is_same<R, float>::value ? (const R*)s.vloc32 : (const R*)s.vloc64;
  a.kAc = s.kAc_d;
  a.o_beg = o_beg;
  a.NBocc = nbk;
  a.NLx = s.NLx; a.NLy = s.NLy; a.NLz = s.NLz; a.NL = s.NL;
  const int nslab = s.nslab < 1 ? 1 : (s.nslab > s.NLx ? s.NLx : s.nslab);
  a.SX = (s.NLx + nslab - 1) / nslab;
  a.lap0sum = s.lap[0][0] + s.lap[1][0] + s.lap[2][0];
  for (int n = 0; n < 4; ++n)
    for (int d = 0; d < 3; ++d) {
      a.lapt[4 * d + n] = (R)s.lap[d][n + 1];
      a.nabc[4 * d + n] = (R)s.nab[d][n + 1];
      a.cl2[4 * d + n] = make_float2((float)s.lap[d][n + 1], (float)s.lap[d][n + 1]);
      a.cn2[4 * d + n] = make_float2((float)s.nab[d][n + 1], (float)s.nab[d][n + 1]);
    }
  a.sp_off = s.sp_off;
  a.nyblk = s.nyblk;
  a.NYB = s.nyblk > 1 ? s.NYB : s.NLy;
  a.sp_blk = s.sp_blk;
  a.lqi = s.lqi;
  a.W = (const C2<R>*)io.W;
  a.S = (C2<R>*)io.S;
  a.nsp = s.nsp;
  a.maxpts = s.maxpts;
  a.zf = mk<R>((R)io.zc[0], (R)io.zc[1]);
  if constexpr (RZ == 2) {
    if (pass2_fits<R>(s)) {
      constexpr int pr = std::is_same<R, float>::value ? SGPU_PREC_C64 : SGPU_PREC_C128;
      const int rows = s.p2_rows[pr], nblk = s.NLy / rows;
      a.sp_blk = s.p2_blk[pr];
      a.maxpts = s.p2_maxpts[pr];
      const int bt = ((rows / 2 * (s.NLz / P2Geom<R>::RZ) + 31) / 32) * 32;
      auto kern = MODE == 2 && io.W && io.S ? pass2_kernel<R, MODE, MODE == 2>(s.NLy, s.NLz)
                                            : pass2_kernel<R, MODE, false>(s.NLy, s.NLz);
      const size_t smem = pass2_smem<R>(s, io.W != nullptr);
      if (smem > 48 * 1024) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaError_t e = cudaStreamIsCapturing(s.stream, &cs);
        if (e != cudaSuccess) return e;
        if (cs == cudaStreamCaptureStatusNone && (e = raise_smem_limit((const void*)kern, smem)) != cudaSuccess) return e;
      }
      kern<<<dim3(nb * nblk, (s.NLx + a.SX - 1) / a.SX), bt, smem, s.launch_stream()>>>(a);
      return cudaGetLastError();
    }
  }
  const int nthr = a.NYB * (s.NLz / RZ);
  const int block = ((nthr + 31) / 32) * 32;
  const bool tb = pass_tables(s, RZ);
  const int shape = pass_shape<R, RZ>(s, tb);
  const size_t smem = pass_smem_bytes(std::is_same<R, float>::value ? SGPU_PREC_C64 : SGPU_PREC_C128, s.NLy, s.NLz,
                                      s.maxpts, io.W != nullptr, s.NLx, s.nyblk, a.NYB, tb, shape ? 9 : 0);
  auto kern = pass_kernel<R, RZ, MODE>(s.nyblk > 1, tb, shape);
  if (smem > 48 * 1024) {
    // set outside stream capture (prepare_pass sets it before a capture)
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s.stream, &cs);
    if (e != cudaSuccess) return e;
    if (cs == cudaStreamCaptureStatusNone) {
      e = raise_smem_limit((const void*)kern, smem);
      if (e != cudaSuccess) return e;
    }
  }
  dim3 grid(nb * s.nyblk, (s.NLx + a.SX - 1) / a.SX);
  kern<<<grid, block, smem, s.launch_stream()>>>(a);
  return cudaGetLastError();
}

template <typename R, int RZ>
static cudaError_t launch_pass_rz(const System& s, int mode, const PassIO& io, int o_beg, int nb, int nbk) {
  switch (mode) {
    case 0: return launch_pass_t<R, RZ, 0>(s, io, o_beg, nb, nbk);
    case 1: return launch_pass_t<R, RZ, 1>(s, io, o_beg, nb, nbk);
    default: return launch_pass_t<R, RZ, 2>(s, io, o_beg, nb, nbk);
  }
}

cudaError_t launch_hpsi_pass(const System& s, int mode, const PassIO& io, int o_beg, int nb, int nbk, int prec) {
  if (nb == 0) return cudaSuccess;
  const bool rz2 = (s.NLz % 2) == 0;
  if ((prec < 0 ? s.prec : prec) == SGPU_PREC_C64)
    return rz2 ? launch_pass_rz<float, 2>(s, mode, io, o_beg, nb, nbk)
               : launch_pass_rz<float, 1>(s, mode, io, o_beg, nb, nbk);
  return rz2 ? launch_pass_rz<double, 2>(s, mode, io, o_beg, nb, nbk)
             : launch_pass_rz<double, 1>(s, mode, io, o_beg, nb, nbk);
}

template <typename R, int RZ>
static cudaError_t prepare_pass_rz(const System& s) {
  if constexpr (RZ == 2) {
    if (pass2_fits<R>(s)) {
      const size_t smem = pass2_smem<R>(s, true);
      const int y = s.NLy, z = s.NLz;
      cudaError_t e = cudaSuccess;
      for (const void* k : {(const void*)pass2_kernel<R, 0, false>(y, z), (const void*)pass2_kernel<R, 1, false>(y, z),
                            (const void*)pass2_kernel<R, 2, false>(y, z), (const void*)pass2_kernel<R, 2, true>(y, z)})
        if (e == cudaSuccess) e = raise_smem_limit(k, smem);
      return e;
    }
  }
  const bool yb = s.nyblk > 1, tb = pass_tables(s, RZ);
  const int shape = pass_shape<R, RZ>(s, tb);
  const size_t smem = pass_smem_bytes(std::is_same<R, float>::value ? SGPU_PREC_C64 : SGPU_PREC_C128, s.NLy, s.NLz,
                                      s.maxpts, true, s.NLx, s.nyblk, yb ? s.NYB : s.NLy, tb, shape ? 9 : 0);
  if (smem <= 48 * 1024) return cudaSuccess;
  cudaError_t e;
  if ((e = raise_smem_limit((const void*)pass_kernel<R, RZ, 0>(yb, tb, shape), smem)))
    return e;
  if ((e = raise_smem_limit((const void*)pass_kernel<R, RZ, 1>(yb, tb, shape), smem)))
    return e;
  return raise_smem_limit((const void*)pass_kernel<R, RZ, 2>(yb, tb, shape), smem);
}

cudaError_t prepare_pass(const System& s) {
  const bool rz2 = (s.NLz % 2) == 0;
  cudaError_t e = rz2 ? prepare_pass_rz<float, 2>(s) : prepare_pass_rz<float, 1>(s);
  if (e != cudaSuccess) return e;
  return rz2 ? prepare_pass_rz<double, 2>(s) : prepare_pass_rz<double, 1>(s);
}

int pass_block_threads(int NLy, int NLz) {  // without y-blocks
  const int rz = (NLz % 2) == 0 ? 2 : 1;
  return ((NLy * (NLz / rz) + 31) / 32) * 32;
}

}  // namespace sgpu
