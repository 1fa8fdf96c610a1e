// FP64 reductions over the resident orbitals: density, current, energy terms.
// Orbitals may be complex(8) or complex(4); every sum is accumulated in FP64
// in a fixed order (no atomics), so results are reproducible run to run.
#include <cuda_runtime.h>

#include <algorithm>

#include <type_traits>

#include "sgpu_internal.cuh"

namespace sgpu {

// ------------------------------------------------------------- psi_rho ---
// rho(i) = sum_{k,b} occ(b,k) |zu(i,b,k)|^2   (common/psi_rho.f90:93-146, sym1)
// Orbitals are split into chunks; each chunk writes a partial density, and the
// partials are summed in chunk order.
constexpr int RHO_CHUNK = 64;

template <typename R>
__global__ void k_rho_partial(const C2<R>* __restrict__ zu, const double* __restrict__ occ_o, int norb, int NL,
                              int chunk, double* __restrict__ part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NL) return;
  const int o0 = blockIdx.y * chunk;
  const int o1 = min(o0 + chunk, norb);
  double acc = 0.0;
  int o = o0;
  // 16 loads in flight: on small grids (few CTAs) the chunk is a chain of load latencies
  constexpr int UN = 16;
  for (; o + UN <= o1; o += UN) {
    C2<R> z[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) z[u] = zu[(size_t)(o + u) * NL + i];
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const double2 v = to_d2(z[u]);
      acc += occ_o[o + u] * (v.x * v.x + v.y * v.y);
    }
  }
  for (; o < o1; ++o) {
    const double2 z = to_d2(zu[(size_t)o * NL + i]);
    acc += occ_o[o] * (z.x * z.x + z.y * z.y);
  }
  part[(size_t)blockIdx.y * NL + i] = acc;
}

__global__ void k_rho_final(const double* __restrict__ part, int nchunk, int NL, double* __restrict__ rho) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NL) return;
  double acc = 0.0;
#pragma unroll 16
  for (int c = 0; c < nchunk; ++c) acc += part[(size_t)c * NL + i];
  rho[i] = acc;
}

cudaError_t launch_psi_rho(System& s, double* rho_dev) {
  // chunks of 64 orbitals, of 16 (one round of loads) where those leave SMs without two CTAs
  // and the partial densities fit
  const int nblk = (s.NL + 255) / 256;
  int chunk = RHO_CHUNK;
  if (nblk * ((s.norb + RHO_CHUNK - 1) / RHO_CHUNK) < 2 * s.nsm && (size_t)((s.norb + 15) / 16) * s.NL <= s.red_elems)
    chunk = 16;
  const int nchunk = (s.norb + chunk - 1) / chunk;
  if ((size_t)nchunk * s.NL > s.red_elems) return cudaErrorInvalidValue;
  dim3 grid(nblk, nchunk);
  if (s.prec == SGPU_PREC_C64)
    k_rho_partial<float><<<grid, 256, 0, s.launch_stream()>>>((const float2*)s.zu, s.occ_o, s.norb, s.NL, chunk, s.red);
  else
    k_rho_partial<double><<<grid, 256, 0, s.launch_stream()>>>((const double2*)s.zu, s.occ_o, s.norb, s.NL, chunk, s.red);
  k_rho_final<<<(s.NL + 255) / 256, 256, 0, s.launch_stream()>>>(s.red, nchunk, s.NL, rho_dev);
  return cudaGetLastError();
}

// ------------------------------------------------------ block reduction ---
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* sh /*[32*NV]*/) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[warp * NV + k] = v[k];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = lane < nw ? sh[lane * NV + k] : 0.0;
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
  }
}

// ------------------------------------------------------------- current ---
// Per orbital: jt = sum |psi|^2 (current.f90:182-186) and the current_stencil
// sums F,G,H = 2 sum Im(conj(psi) sum_n nab_n psi(+n)) (stencil/F90/current.f90),
// with forward neighbours only (n = 1..4), as the reference's stencil has them.
//
// The orbital's planes are marched along x, the planes ahead in a register queue (FP64,
// converted once on load), the current plane staged in FP64 in shared memory for the y and
// z neighbours.  Sums are FP64, per thread in plane order, then a fixed-order block sum.
struct Nab12 {
  double v[12];  // nabx(1:4), naby(1:4), nabz(1:4): kernel parameters, read from the parameter bank
};

// The march for any plane shape, two rows per thread: the plane is split into blocks of GB
// rows (even; the last may be shorter), one CTA per (orbital, block); thread (r, z) owns the
// points of rows 2r and 2r+1, so row 2r+1 is a y neighbour in registers and the four rows
// after it are read once for both.  A CTA stages its rows and the four rows after them.
//
// EKIN: the kinetic energy instead of the current.  Summed over the periodic grid, the
// backward neighbours give the same products as the forward ones,
//   sum_i conj(e_i) (e_{i+n} + e_{i-n}) = 2 sum_i Re(conj(e_i) e_{i+n}),
//   sum_i conj(e_i) (e_{i+n} - e_{i-n}) = 2i sum_i Im(conj(e_i) e_{i+n}),
// so tpsum = sum conj(e) (lap0_2 e - 0.5 v - i w) (stencil/F90/total_energy.f90:93-180) needs
// the forward neighbours only: half of the arithmetic and of the shared-memory reads.  With
// one CTA per plane and 24 neighbours through L1, 20^3 x 2048 orbitals, complex(8), took
// 1.14 ms; now 0.17 (sgpu_energy_terms: see launch_energy).  The norm, Laplacian and k parts are
// summed over the block and subtracted at the end, so the large terms cancel in the sums and
// not point by point; the rounding is the same, that of the products.  Restated on the host
// against extended precision, 20^3: a smooth orbital 7.0e-15 (point by point 8.6e-15), one
// that is constant to 1e-2 1.5e-11 (2.6e-11), to 1e-4 3.0e-7 (2.5e-7).  The current with this
// form: see current_stencil.
// Few orbitals leave SMs idle behind a chain of NLx steps: the march is then cut into slabs
// of SX planes, one CTA each (see march_slabs).
// out[o][block][slab][4] = {sum |e|^2, F/2, G/2, H/2}, or [o][block][slab][2] = {Re tpsum, 0}.
struct FwdCoef {
  double lap0_2;    // EKIN: -(lapx(0)+lapy(0)+lapz(0))/2
  double lap[12];   // EKIN: lapx(1:4), lapy(1:4), lapz(1:4)
  double nab[12];   // nabx(1:4), naby(1:4), nabz(1:4)
};

template <typename R, bool EKIN, bool SLABS>
__global__ void __launch_bounds__(256, 2) k_fwd_march(const C2<R>* __restrict__ zu, int NLx, int NLy, int NLz, int GB,
                                                      int nblk, int SX, int NBocc, const double* __restrict__ kAc,
                                                      const FwdCoef c, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[32 * 4];
  double2* buf = reinterpret_cast<double2*>(smem_raw);  // [2][(GB+4)*NLz]
  const int RB = (GB + 4) * NLz;
  const int o = blockIdx.x / nblk, h = blockIdx.x - o * nblk, t = threadIdx.x, nt = blockDim.x;
  const int NYZ = NLy * NLz, rows = min(GB, NLy - h * GB);
  const int x_beg = SLABS ? blockIdx.y * SX : 0, x_end = SLABS ? min(x_beg + SX, NLx) : NLx;  // (never empty)
  const C2<R>* E = zu + (size_t)o * NLx * NYZ;
  const int y0 = 2 * (t / NLz), z = t - (t / NLz) * NLz;
  const bool act = y0 < rows, two = y0 + 1 < rows;
  const int own = act ? (h * GB + y0) * NLz + z : 0;
  const int own_b = two ? own + NLz : own;
  int zo[4];
#pragma unroll
  for (int n = 1; n <= 4; ++n) {
    int zz = z + n;
    while (zz >= NLz) zz -= NLz;
    zo[n - 1] = zz - z;
  }
  double k[3] = {0, 0, 0};
  if (EKIN) {
    const int kl = o / NBocc;
#pragma unroll
    for (int d = 0; d < 3; ++d) k[d] = kAc[3 * kl + d];
  }
  auto load = [&](int x, int i, bool ok) -> double2 {
    return ok ? to_d2(__ldg(E + (size_t)x * NYZ + i)) : make_double2(0, 0);
  };
  // register queues: at phase P (plane x = x_beg + 5i + P) plane x+m sits in slot (P+m) % 5
  double2 qa[5], qb[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const int xm = (x_beg + m) % NLx;
    qa[m] = load(xm, own, act);
    qb[m] = load(xm, own_b, two);
  }
  int xn = (x_beg + 5) % NLx;
  C2<R> na = __ldg(E + (size_t)xn * NYZ + own), nb = __ldg(E + (size_t)xn * NYZ + own_b);  // in flight
  xn = xn + 1 < NLx ? xn + 1 : 0;
  double v[4] = {0, 0, 0, 0};
  int x = x_beg, left = x_end - x_beg;
  auto step = [&](auto phase) -> bool {
    constexpr int P = decltype(phase)::value;
    double2* pl = buf + (x & 1) * RB;
    const double2 ea = qa[P % 5], eb = qb[P % 5];
    double2* pa = pl + y0 * NLz + z;
    if (act) pa[0] = ea;
    if (two) pa[NLz] = eb;
    for (int i = t; i < 4 * NLz; i += nt) {
      int hr = h * GB + rows + i / NLz;
      while (hr >= NLy) hr -= NLy;
      pl[rows * NLz + i] = to_d2(__ldg(E + (size_t)x * NYZ + hr * NLz + i % NLz));
    }
    __syncthreads();
    if (act) {
      double2 r[5];  // rows y0 + 1 .. y0 + 5 at column z
      r[0] = two ? eb : pa[NLz];
#pragma unroll
      for (int m = 1; m < 4; ++m) r[m] = pa[(m + 1) * NLz];
      r[4] = two ? pa[5 * NLz] : make_double2(0, 0);
      const double2 zero = make_double2(0, 0);
      if constexpr (EKIN) {
        double2 la = zero, lb = zero, ta = zero, tb = zero;  // sum lap e(+n), sum k nab e(+n)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          double2 wa = zero, wb = zero;
#pragma unroll
          for (int n = 1; n <= 4; ++n) {
            const double2 fa = d == 0 ? qa[(P + n) % 5] : (d == 1 ? r[n - 1] : pa[zo[n - 1]]);
            const double2 fb = d == 0 ? qb[(P + n) % 5] : (d == 1 ? r[n] : (two ? pa[NLz + zo[n - 1]] : zero));
            const double cl = c.lap[4 * d + n - 1], cn = c.nab[4 * d + n - 1];
            la.x = fma(cl, fa.x, la.x); la.y = fma(cl, fa.y, la.y);
            lb.x = fma(cl, fb.x, lb.x); lb.y = fma(cl, fb.y, lb.y);
            wa.x = fma(cn, fa.x, wa.x); wa.y = fma(cn, fa.y, wa.y);
            wb.x = fma(cn, fb.x, wb.x); wb.y = fma(cn, fb.y, wb.y);
          }
          ta.x = fma(k[d], wa.x, ta.x); ta.y = fma(k[d], wa.y, ta.y);
          tb.x = fma(k[d], wb.x, tb.x); tb.y = fma(k[d], wb.y, tb.y);
        }
        v[0] = fma(ea.x, ea.x, fma(ea.y, ea.y, fma(eb.x, eb.x, fma(eb.y, eb.y, v[0]))));
        v[1] += fma(ea.x, la.x, ea.y * la.y) + fma(eb.x, lb.x, eb.y * lb.y);  // Re(conj(e) l)
        v[2] += fma(ea.x, ta.y, -ea.y * ta.x) + fma(eb.x, tb.y, -eb.y * tb.x);  // Im(conj(e) t)
      } else {
        v[0] = fma(ea.x, ea.x, fma(ea.y, ea.y, fma(eb.x, eb.x, fma(eb.y, eb.y, v[0]))));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          double2 wa = zero, wb = zero;
#pragma unroll
          for (int n = 1; n <= 4; ++n) {
            const double2 fa = d == 0 ? qa[(P + n) % 5] : (d == 1 ? r[n - 1] : pa[zo[n - 1]]);
            const double2 fb = d == 0 ? qb[(P + n) % 5] : (d == 1 ? r[n] : (two ? pa[NLz + zo[n - 1]] : zero));
            const double cn = c.nab[4 * d + n - 1];
            wa.x = fma(cn, fa.x, wa.x); wa.y = fma(cn, fa.y, wa.y);
            wb.x = fma(cn, fb.x, wb.x); wb.y = fma(cn, fb.y, wb.y);
          }
          // aimag(conjg(e) s) = e.x s.y - e.y s.x, point a then point b
          v[1 + d] = fma(eb.x, wb.y, fma(-eb.y, wb.x, fma(ea.x, wa.y, fma(-ea.y, wa.x, v[1 + d]))));
        }
      }
    }
    qa[P % 5] = act ? to_d2(na) : make_double2(0, 0);  // plane x+5 takes the slot of plane x
    qb[P % 5] = two ? to_d2(nb) : make_double2(0, 0);
    na = __ldg(E + (size_t)xn * NYZ + own);
    nb = __ldg(E + (size_t)xn * NYZ + own_b);
    xn = xn + 1 < NLx ? xn + 1 : 0;
    ++x;
    return --left > 0;
  };
  for (;;) {
    if (!step(std::integral_constant<int, 0>{})) break;
    if (!step(std::integral_constant<int, 1>{})) break;
    if (!step(std::integral_constant<int, 2>{})) break;
    if (!step(std::integral_constant<int, 3>{})) break;
    if (!step(std::integral_constant<int, 4>{})) break;
  }
  block_sum<4>(v, sh);
  if (t == 0) {
    const size_t row = SLABS ? (size_t)blockIdx.x * gridDim.y + blockIdx.y : blockIdx.x;
    if (EKIN) {
      out[2 * row] = c.lap0_2 * v[0] - v[1] + 2.0 * v[2];
      out[2 * row + 1] = 0.0;
    } else {
#pragma unroll
      for (int m = 0; m < 4; ++m) out[4 * row + m] = v[m];
    }
  }
}

// rows of a block: the largest even number whose row pairs' points fit 256 threads, the
// blocks of a plane as equal as that allows
int march_rows(int NLy, int NLz) {
  const int most = std::max(2, 2 * (256 / NLz)), nblk = (NLy + most - 1) / most;
  return ((NLy + nblk - 1) / nblk + 1) / 2 * 2;
}
static int march_blocks(int NLy, int NLz) {
  const int GB = march_rows(NLy, NLz);
  return (NLy + GB - 1) / GB;
}
// Slabs of the march, each of at least four planes (a slab reads five planes before its first
// step): as many as two CTAs per SM take for the energy, one for the current, which runs
// beside a step's density and potential: two delay those (step at 24x8x48, complex(8), 98
// orbitals 283 us without slabs, 282 with one, 289 with two).
// Without slabs and with them, complex(4), us: sgpu_energy_terms 18x24x27 x 16 orbitals 64 / 55,
// 40^3 x 1 107 / 80, x 64 123 / 119; sgpu_current 36^3 x 4 90 / 66.
static int march_slabs(const System& s, int ctas_per_sm) {
  const int ctas = s.norb * march_blocks(s.NLy, s.NLz);
  const int most = std::max(1, std::min(ctas_per_sm * s.nsm / ctas, s.NLx / 4)), SX = (s.NLx + most - 1) / most;
  return (s.NLx + SX - 1) / SX;
}
int march_parts(const System& s) {
  return march_blocks(s.NLy, s.NLz) * std::max(march_slabs(s, 1), march_slabs(s, 2));
}

template <typename R, bool EKIN>
static cudaError_t fwd_march(System& s, double* out, int& nx) {
  FwdCoef c;
  c.lap0_2 = -(s.lap[0][0] + s.lap[1][0] + s.lap[2][0]) * 0.5;
  for (int n = 0; n < 4; ++n)
    for (int d = 0; d < 3; ++d) {
      c.lap[4 * d + n] = s.lap[d][n + 1];
      c.nab[4 * d + n] = s.nab[d][n + 1];
    }
  const int GB = march_rows(s.NLy, s.NLz);
  const int nblk = march_blocks(s.NLy, s.NLz), nslab = march_slabs(s, EKIN ? 2 : 1);
  nx = nblk * nslab;
  const int nt = (GB / 2 * s.NLz + 31) / 32 * 32;
  const size_t smem = 2 * (size_t)(GB + 4) * s.NLz * sizeof(double2);
  // (bounds known at compile time without slabs: 172.5 against 173.4 us at 20^3 x 2048)
  auto kern = nslab > 1 ? k_fwd_march<R, EKIN, true> : k_fwd_march<R, EKIN, false>;
  const cudaError_t e = raise_smem_limit((const void*)kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<dim3(s.norb * nblk, nslab), nt, smem, s.launch_stream()>>>(
      (const C2<R>*)s.zu, s.NLx, s.NLy, s.NLz, GB, nblk, (s.NLx + nslab - 1) / nslab, s.NBocc, s.kAc_d, c, out);
  return cudaGetLastError();
}

// The x-march with each GY x GZ plane split over NP CTAs of GY/NP rows (one
// point per thread, (GY/NP)*GZ threads): a CTA stages its rows and the four rows
// after them (the forward y-neighbours, read from L2 each step) in FP64 in
// shared memory.  Small CTAs at few registers let several orbitals' marches
// share an SM, so one CTA's barrier waits overlap another's arithmetic.
// out[o][h][4], h = the part.
template <typename R, int GY, int GZ, int NP>
__global__ void __launch_bounds__(GY / NP * GZ) k_current_march_yh(const C2<R>* __restrict__ zu, int NLx,
                                                                  const Nab12 nab, double* __restrict__ out) {
  constexpr int NYH = GY / NP, NT = NYH * GZ, NYZ = GY * GZ, RB = (NYH + 4) * GZ;
  static_assert(NT % 32 == 0 && NT <= 1024 && 4 * GZ <= NT, "one point per thread, halo loaded by the first rows");
  __shared__ double2 buf[2][RB];
  __shared__ double sh[32 * 4];
  const int o = blockIdx.x / NP, h = blockIdx.x - (blockIdx.x / NP) * NP, t = threadIdx.x;
  const C2<R>* E = zu + (size_t)o * NLx * NYZ;
  const double* nb = nab.v;
  const int yl = t / GZ, z = t - (t / GZ) * GZ;
  const int own = (h * NYH + yl) * GZ + z;                           // in the plane
  const int hrow = ((h + 1) * NYH + (t / GZ)) % GY;                   // halo row of threads t < 4 GZ
  const int hsrc = hrow * GZ + z;
  int zo[4];                                                          // z neighbours in the staged rows
#pragma unroll
  for (int n = 1; n <= 4; ++n) zo[n - 1] = yl * GZ + ((z + n) % GZ);
  // register queue: at phase P (plane x = 5i + P) plane x+m sits in q[(P+m) % 5];
  // the march is unrolled five times so the queue rotates by renaming (NLx >= 5)
  double2 q[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) q[m] = to_d2(__ldg(E + (size_t)m * NYZ + own));
  C2<R> nxt = __ldg(E + (size_t)(5 % NLx) * NYZ + own);
  int xn = 6 < NLx ? 6 : 6 - NLx;                                     // the plane loaded next
  double v[4] = {0, 0, 0, 0};
  int x = 0;
  auto step = [&](auto phase) -> bool {
    constexpr int P = decltype(phase)::value;
    double2* pl = buf[x & 1];
    const double2 e = q[P % 5];
    pl[t] = e;
    if (t < 4 * GZ) pl[NT + t] = to_d2(__ldg(E + (size_t)x * NYZ + hsrc));
    __syncthreads();
    v[0] = fma(e.x, e.x, fma(e.y, e.y, v[0]));
    double2 sx = make_double2(0, 0), sy = make_double2(0, 0), sz = make_double2(0, 0);
#pragma unroll
    for (int n = 1; n <= 4; ++n) {
      const double2 ex = q[(P + n) % 5];
      const double2 ey = pl[(yl + n) * GZ + z];
      const double2 ez = pl[zo[n - 1]];
      sx.x = fma(nb[n - 1], ex.x, sx.x); sx.y = fma(nb[n - 1], ex.y, sx.y);
      sy.x = fma(nb[3 + n], ey.x, sy.x); sy.y = fma(nb[3 + n], ey.y, sy.y);
      sz.x = fma(nb[7 + n], ez.x, sz.x); sz.y = fma(nb[7 + n], ez.y, sz.y);
    }
    // aimag(conjg(e) s) = e.x s.y - e.y s.x
    v[1] = fma(e.x, sx.y, fma(-e.y, sx.x, v[1]));
    v[2] = fma(e.x, sy.y, fma(-e.y, sy.x, v[2]));
    v[3] = fma(e.x, sz.y, fma(-e.y, sz.x, v[3]));
    q[P % 5] = to_d2(nxt);  // plane x+5 takes the slot of plane x
    nxt = __ldg(E + (size_t)xn * NYZ + own);
    xn = xn + 1 < NLx ? xn + 1 : 0;
    ++x;
    return x < NLx;
  };
  for (;;) {
    if (!step(std::integral_constant<int, 0>{})) break;
    if (!step(std::integral_constant<int, 1>{})) break;
    if (!step(std::integral_constant<int, 2>{})) break;
    if (!step(std::integral_constant<int, 3>{})) break;
    if (!step(std::integral_constant<int, 4>{})) break;
  }
  block_sum<4>(v, sh);
  if (t == 0) {
    double* d = out + 4 * (size_t)blockIdx.x;
    d[0] = v[0];
    d[1] = v[1];
    d[2] = v[2];
    d[3] = v[3];
  }
}
// The same march with two rows per thread: thread (r, z) owns the points of rows
// 2r and 2r+1, so row 2r+1 is a y-neighbour in registers and the four rows above
// it are read once for both points (six shared-memory loads a point instead of
// eight; the march is bound by shared-memory wavefronts).  Each GY x GZ plane is
// split over NP CTAs of GY/NP rows ((GY/NP/2)*GZ threads) plus four halo rows.
template <typename R, int GY, int GZ, int NP, int MB = 1>
__global__ void __launch_bounds__(GY / NP / 2 * GZ, MB) k_current_march_y2(const C2<R>* __restrict__ zu, int NLx,
                                                                      const Nab12 nab, double* __restrict__ out) {
  constexpr int NYH = GY / NP, NT = NYH / 2 * GZ, NYZ = GY * GZ, RB = (NYH + 4) * GZ;
  static_assert(NYH % 2 == 0 && NT % 32 == 0 && NT <= 1024 && 4 * GZ <= NT, "two rows per thread, halo by the first");
  __shared__ double2 buf[2][RB];
  __shared__ double sh[32 * 4];
  const int o = blockIdx.x / NP, h = blockIdx.x - (blockIdx.x / NP) * NP, t = threadIdx.x;
  const C2<R>* E = zu + (size_t)o * NLx * NYZ;
  const double* nb = nab.v;
  const int y0 = 2 * (t / GZ), z = t - (t / GZ) * GZ;                 // local rows y0, y0 + 1
  const int own = (h * NYH + y0) * GZ + z;                            // row y0 in the plane; y0 + 1 is own + GZ
  const int hsrc = (((h + 1) * NYH + t / GZ) % GY) * GZ + z;          // halo row of threads t < 4 GZ
  int zo[4];                                                          // z + n in a staged row
#pragma unroll
  for (int n = 1; n <= 4; ++n) zo[n - 1] = (z + n) % GZ;
  // register queues as in k_current_march_yh (plane x + m in slot (P + m) % 5)
  double2 qa[5], qb[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    qa[m] = to_d2(__ldg(E + (size_t)m * NYZ + own));
    qb[m] = to_d2(__ldg(E + (size_t)m * NYZ + own + GZ));
  }
  C2<R> na = __ldg(E + (size_t)(5 % NLx) * NYZ + own), nb_ = __ldg(E + (size_t)(5 % NLx) * NYZ + own + GZ);
  int xn = 6 < NLx ? 6 : 6 - NLx;
  double v[4] = {0, 0, 0, 0};
  int x = 0;
  auto step = [&](auto phase) -> bool {
    constexpr int P = decltype(phase)::value;
    double2* pl = buf[x & 1];
    const double2 ea = qa[P % 5], eb = qb[P % 5];
    pl[y0 * GZ + z] = ea;
    pl[(y0 + 1) * GZ + z] = eb;
    if (t < 4 * GZ) pl[NYH * GZ + t] = to_d2(__ldg(E + (size_t)x * NYZ + hsrc));
    __syncthreads();
    v[0] = fma(ea.x, ea.x, fma(ea.y, ea.y, fma(eb.x, eb.x, fma(eb.y, eb.y, v[0]))));
    double2 r[5];  // rows y0 + 1 .. y0 + 5 at column z
    r[0] = eb;
#pragma unroll
    for (int k = 1; k < 5; ++k) r[k] = pl[(y0 + 1 + k) * GZ + z];
    double2 sxa = make_double2(0, 0), sya = sxa, sza = sxa, sxb = sxa, syb = sxa, szb = sxa;
#pragma unroll
    for (int n = 1; n <= 4; ++n) {
      const double2 xa = qa[(P + n) % 5], xb = qb[(P + n) % 5];
      const double2 ya = r[n - 1], yb = r[n];
      const double2 za = pl[y0 * GZ + zo[n - 1]], zb = pl[(y0 + 1) * GZ + zo[n - 1]];
      sxa.x = fma(nb[n - 1], xa.x, sxa.x); sxa.y = fma(nb[n - 1], xa.y, sxa.y);
      sxb.x = fma(nb[n - 1], xb.x, sxb.x); sxb.y = fma(nb[n - 1], xb.y, sxb.y);
      sya.x = fma(nb[3 + n], ya.x, sya.x); sya.y = fma(nb[3 + n], ya.y, sya.y);
      syb.x = fma(nb[3 + n], yb.x, syb.x); syb.y = fma(nb[3 + n], yb.y, syb.y);
      sza.x = fma(nb[7 + n], za.x, sza.x); sza.y = fma(nb[7 + n], za.y, sza.y);
      szb.x = fma(nb[7 + n], zb.x, szb.x); szb.y = fma(nb[7 + n], zb.y, szb.y);
    }
    // aimag(conjg(e) s) = e.x s.y - e.y s.x, point a then point b
    v[1] = fma(eb.x, sxb.y, fma(-eb.y, sxb.x, fma(ea.x, sxa.y, fma(-ea.y, sxa.x, v[1]))));
    v[2] = fma(eb.x, syb.y, fma(-eb.y, syb.x, fma(ea.x, sya.y, fma(-ea.y, sya.x, v[2]))));
    v[3] = fma(eb.x, szb.y, fma(-eb.y, szb.x, fma(ea.x, sza.y, fma(-ea.y, sza.x, v[3]))));
    qa[P % 5] = to_d2(na);  // plane x+5 takes the slot of plane x
    qb[P % 5] = to_d2(nb_);
    na = __ldg(E + (size_t)xn * NYZ + own);
    nb_ = __ldg(E + (size_t)xn * NYZ + own + GZ);
    xn = xn + 1 < NLx ? xn + 1 : 0;
    ++x;
    return x < NLx;
  };
  for (;;) {
    if (!step(std::integral_constant<int, 0>{})) break;
    if (!step(std::integral_constant<int, 1>{})) break;
    if (!step(std::integral_constant<int, 2>{})) break;
    if (!step(std::integral_constant<int, 3>{})) break;
    if (!step(std::integral_constant<int, 4>{})) break;
  }
  block_sum<4>(v, sh);
  if (t == 0) {
    double* d = out + 4 * (size_t)blockIdx.x;
    d[0] = v[0];
    d[1] = v[1];
    d[2] = v[2];
    d[3] = v[3];
  }
}
template <typename R, int GY, int GZ, int NP, int MB = 1>
static cudaError_t current_march_y2(System& s, const Nab12& nab, double* out) {
  k_current_march_y2<R, GY, GZ, NP, MB><<<NP * s.norb, GY / NP / 2 * GZ, 0, s.launch_stream()>>>((const C2<R>*)s.zu,
                                                                                             s.NLx, nab, out);
  return cudaGetLastError();
}

template <typename R, int GY, int GZ, int NP>
static cudaError_t current_march_yh(System& s, const Nab12& nab, double* out) {
  k_current_march_yh<R, GY, GZ, NP><<<NP * s.norb, GY / NP * GZ, 0, s.launch_stream()>>>((const C2<R>*)s.zu, s.NLx,
                                                                                          nab, out);
  return cudaGetLastError();
}

// Weighted projections for the nonlocal current (current.f90:247-265):
// Uw[o][ilma][w] = sum_j conj(zproj(j,ilma,k)) r_w(j) psi(J(j)), r = (1, x, y, z).
// psi(J(j)) is read from src[o*ld + idx[j]]: the compact sphere values S with
// the sphere-point map qmap when they are current, else the orbitals with the
// grid index idx_proj.
// One CTA per (projector item, k-point, group of up to 32 bands of that k-point,
// part of the item's points): the points are split into nsplit contiguous ranges
// of UVW_CH-point chunks so that the grid fills the GPU, and each range writes its
// own partial Uw[part][o][ilma][w] (k_current_comb adds the parts in order).  Per
// chunk, conj(zproj) of the item's projectors, the weights r and the bands' values
// are staged in shared memory (band rows padded by one element: the eight band
// rows a warp reads at one point fall in distinct banks).  Thread (lane, warp)
// takes bands bg, bg+8, bg+16, bg+24 (bg = lane & 7) of projector lane >> 3 over
// every eighth point of the chunk: t = conj(zproj) psi once, then
// Uw[., 0] += t, Uw[., w] += r_w t (12 FP64 operations a band and point instead
// of the 16 of four complex products), and the eight warps' sums are added in
// a fixed order.
constexpr int UVW_CH = 128;
template <typename R> struct UvwGeom {
  static constexpr int SROW = UVW_CH + 1;  // padded band row
  static constexpr size_t stage = sizeof(C2<R>) * 32 * SROW + sizeof(double2) * 4 * UVW_CH +
                                  sizeof(double) * 3 * UVW_CH + sizeof(int) * UVW_CH;
  static constexpr size_t red = sizeof(double2) * 8 * 32 * 9;  // the part sums, eight entries (+1 pad) at a time
  static constexpr size_t smem = stage > red ? stage : red;
};

template <typename R>
__global__ void __launch_bounds__(256, 2) k_uvpsi_w(const C2<R>* __restrict__ src, int ld, int NBocc,
                                                     const double2* __restrict__ zproj, int Nlma, int Nps,
                                                     const int* __restrict__ idx, const int* __restrict__ atom_off,
                                                     const double* __restrict__ rpos, const int4* __restrict__ items,
                                                     const int* __restrict__ lma_list, int nsplit, int norb,
                                                     double2* __restrict__ Uw) {
  constexpr int CH = UVW_CH, SROW = UvwGeom<R>::SROW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<R>* ps = reinterpret_cast<C2<R>*>(smem_raw);                          // [32][SROW] band values
  double2* cz = reinterpret_cast<double2*>(ps + 32 * SROW);                // [4][CH] conj(zproj)
  double* rw = reinterpret_cast<double*>(cz + 4 * CH);                     // [CH][3] weights x, y, z
  int* is = reinterpret_cast<int*>(rw + 3 * CH);                           // [CH] gather index
  double2* red = reinterpret_cast<double2*>(smem_raw);                     // [8][32][9] after the sums
  const int t = threadIdx.x, lane = t & 31, part = t >> 5;
  const int bg = lane & 7, pg = lane >> 3;  // bands bg + 8i, projector pg (its 4 weights)
  const int4 item = items[blockIdx.x];
  const int kl = blockIdx.y, b0 = (blockIdx.z / nsplit) * 32, split = blockIdx.z - (blockIdx.z / nsplit) * nsplit;
  const int a = item.x, l0 = item.y, np = item.z;
  const int p0 = atom_off[a], mps = atom_off[a + 1] - p0;
  const int nbr = min(32, NBocc - b0);
  if (nbr <= 0) return;  // whole CTA leaves together
  const int nch = (mps + CH - 1) / CH, cps = (nch + nsplit - 1) / nsplit;
  const int cbeg = min(nch, split * cps), cend = min(nch, cbeg + cps);  // may be empty: zeros are written
  double2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int w = 0; w < 4; ++w) acc[i][w] = make_double2(0.0, 0.0);
  for (int c = cbeg; c < cend; ++c) {
    const int c0 = c * CH, len = min(CH, mps - c0);
    __syncthreads();  // the previous chunk is no longer read
    for (int q = t; q < 4 * CH; q += 256) {  // conj(zproj) of point j, projector p
      const int p = q / CH, j = q - p * CH;
      double2 z = make_double2(0.0, 0.0);
      if (j < len && p < np) z = zproj[((size_t)kl * Nlma + lma_list[l0 + p]) * Nps + c0 + j];
      cz[p * CH + j] = make_double2(z.x, -z.y);
      if (p == 0) {
        const double* r = rpos + 3 * (size_t)(p0 + c0 + j);
        rw[3 * j] = j < len ? r[0] : 0.0;
        rw[3 * j + 1] = j < len ? r[1] : 0.0;
        rw[3 * j + 2] = j < len ? r[2] : 0.0;
        is[j] = j < len ? idx[p0 + c0 + j] : 0;
      }
    }
    __syncthreads();
    const int tot = 32 * len;
    for (int q0 = t; q0 < tot; q0 += 8 * 256) {
      C2<R> vals[8];
      int slot[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int q = q0 + u * 256;
        slot[u] = -1;
        if (q < tot) {
          const int bb = q / len, j = q - bb * len;
          slot[u] = bb * SROW + j;
          vals[u] = bb < nbr ? __ldg(src + (size_t)(kl * NBocc + b0 + bb) * ld + is[j]) : C2<R>{};
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (slot[u] >= 0) ps[slot[u]] = vals[u];
    }
    __syncthreads();
    for (int j = part; j < len; j += 8) {
      const double2 zc = cz[pg * CH + j];
      const double r1 = rw[3 * j], r2 = rw[3 * j + 1], r3 = rw[3 * j + 2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double2 e = to_d2(ps[(bg + 8 * i) * SROW + j]);
        const double tx = fma(zc.x, e.x, -zc.y * e.y), ty = fma(zc.x, e.y, zc.y * e.x);
        acc[i][0].x += tx;
        acc[i][0].y += ty;
        acc[i][1].x = fma(r1, tx, acc[i][1].x);
        acc[i][1].y = fma(r1, ty, acc[i][1].y);
        acc[i][2].x = fma(r2, tx, acc[i][2].x);
        acc[i][2].y = fma(r2, ty, acc[i][2].y);
        acc[i][3].x = fma(r3, tx, acc[i][3].x);
        acc[i][3].y = fma(r3, ty, acc[i][3].y);
      }
    }
  }
  // the eight warps' sums, eight of a thread's sixteen entries at a time
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    __syncthreads();  // the staging buffers (or the previous half) are no longer read
#pragma unroll
    for (int k = 0; k < 8; ++k) red[(part * 32 + lane) * 9 + k] = acc[2 * half + k / 4][k % 4];
    __syncthreads();
    {  // thread (lane', k): entry k of lane' summed over the parts in order
      const int ln = t >> 3, k = t & 7;
      double2 sum = make_double2(0.0, 0.0);
#pragma unroll
      for (int pp = 0; pp < 8; ++pp) {
        const double2 v = red[(pp * 32 + ln) * 9 + k];
        sum.x += v.x;
        sum.y += v.y;
      }
      const int tb = ln & 7, tp = ln >> 3, i = 2 * half + k / 4, w = k & 3;
      const int b = tb + 8 * i;
      if (tp < np && b < nbr)
        Uw[(((size_t)split * norb + kl * NBocc + b0 + b) * Nlma + lma_list[l0 + tp]) * 4 + w] = sum;
    }
  }
}

// Per orbital, combines the plane sums and the weighted projections exactly as
// current() does (current.f90:182-273): jo[o][d].
// One warp per orbital: lane l takes projectors l, l+32, ... in order, the lanes'
// nonlocal sums are added by a fixed butterfly, and lane 0 adds the plane sums.
constexpr int COMB_T = 256;
__global__ void __launch_bounds__(COMB_T) k_current_comb(const double* __restrict__ part, int nx,
                                                        const double2* __restrict__ Uw, int nsplit,
                                                        const double* __restrict__ occ_o,
                                                        const double* __restrict__ kAc, const int* __restrict__ iuV,
                                                        int norb, int NBocc, int Nlma, double Hxyz, double IaLxyz,
                                                        double* __restrict__ jo) {
  const int o = blockIdx.x * (COMB_T / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (o >= norb) return;  // whole warp
  const double occ = occ_o[o];
  double jn[3] = {0, 0, 0};
  for (int l = lane; l < Nlma; l += 32) {
    double2 u[4];  // the point-range parts of k_uvpsi_w, added in order
#pragma unroll
    for (int w = 0; w < 4; ++w) u[w] = Uw[((size_t)o * Nlma + l) * 4 + w];
    for (int sp = 1; sp < nsplit; ++sp)
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const double2 v = Uw[(((size_t)sp * norb + o) * Nlma + l) * 4 + w];
        u[w].x += v.x;
        u[w].y += v.y;
      }
    const double f = Hxyz * (double)iuV[l];
    const double2 u0 = make_double2(u[0].x * f, u[0].y * f);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double2 ud = make_double2(u[1 + d].x * Hxyz, u[1 + d].y * Hxyz);
      // aimag(conjg(ud) * u0)
      jn[d] += occ * IaLxyz * 2.0 * (ud.x * u0.y - ud.y * u0.x);
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) jn[d] += __shfl_xor_sync(0xffffffffu, jn[d], off);
  if (lane == 0) {
    double v[4] = {0, 0, 0, 0};
    for (int x = 0; x < nx; ++x) {  // per-orbital rows of partial sums, in order
      const double* d = part + ((size_t)o * nx + x) * 4;
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] += d[k];
    }
    const int kl = o / NBocc;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double j = occ * kAc[3 * kl + d] * v[0] + 2.0 * v[1 + d] * occ;
      jo[3 * (size_t)o + d] = j * Hxyz * IaLxyz + jn[d];
    }
  }
}

// sum over orbitals in a fixed order
__global__ void k_current_sum(const double* __restrict__ jo, int norb, double* __restrict__ jav) {
  __shared__ double sh[32 * 3];
  double v[3] = {0, 0, 0};
  for (int o = threadIdx.x; o < norb; o += blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] += jo[3 * (size_t)o + d];
  }
  block_sum<3>(v, sh);
  if (threadIdx.x == 0) {
    jav[0] = v[0];
    jav[1] = v[1];
    jav[2] = v[2];
  }
}


// scratch of launch_current (part [norb][rows][4], jo [norb][3]) and of launch_energy
// (part [norb][rows][2], eo [norb][2])
size_t current_red_elems(int norb, int rows) { return (size_t)norb * rows * 4 + 3 * (size_t)norb + 32; }

template <typename R>
static cudaError_t current_stencil(System& s, const Nab12& nab, double* part, int& nx) {
  nx = 1;
  // 32x32 planes: two CTAs of 16 rows per orbital plane, two rows per thread at
  // three CTAs per SM (value 2: four CTAs of 8 rows, one row per thread).
  // At 32^3 x 2048 orbitals, complex(4): 0.328 against 0.388 ms; two rows per
  // thread at 118 registers (two CTAs per SM) 0.709 ms, one CTA per plane 0.344 ms
  // (complex(8): 0.394 / 0.403 / 0.642 / 0.423 ms)
  // Both fixed forms fill their queue with planes 0 .. 4 as they lie in memory; grids of
  // fewer planes take the march for any shape, which wraps them.
  const bool fixed = s.cur_fixed && s.NLx >= 5;
  if (fixed && s.NLy == 32 && s.NLz == 32) {
    if (s.cur_fixed == 2) {
      nx = 4;
      return current_march_yh<R, 32, 32, 4>(s, nab, part);
    }
    nx = 2;
    return current_march_y2<R, 32, 32, 2, 3>(s, nab, part);
  }
  // 48x48 planes (the 48^3 grid): six CTAs of 8 rows per orbital plane (two rows per
  // thread, 192 threads; value 2: one row per thread, 384 threads): 0.284 against
  // 0.313 ms at 432 orbitals, complex(4); 0.298 against 0.328 ms complex(8)
  if (fixed && s.NLy == 48 && s.NLz == 48) {
    nx = 6;
    return s.cur_fixed == 2 ? current_march_yh<R, 48, 48, 6>(s, nab, part) : current_march_y2<R, 48, 48, 6>(s, nab, part);
  }
  // other planes: row blocks of any shape.  Whole planes per CTA (to 1024 points) and one CTA
  // per plane beyond, in brackets, ms: 16x16x32 x 1024 orbitals, complex(4) 0.061 (0.088), 20^3 x
  // 2048 0.143 (0.217), 8^3 x 1024 0.008 (0.021).  At 32^3 and 48^3 it is slower than the fixed
  // forms above: 0.49 / 0.33 and, 800 orbitals, 0.75 / 0.52.
  return fwd_march<R, false>(s, part, nx);
}

// The stencil sums {jt, F, G, H} of the resident orbitals into part[o][nx][4].
cudaError_t launch_current_stencil(System& s, double* part, int& nx) {
  Nab12 nab;
  for (int n = 0; n < 4; ++n)
    for (int d = 0; d < 3; ++d) nab.v[4 * d + n] = s.nab[d][n + 1];
  nx = 1;
  return s.prec == SGPU_PREC_C64 ? current_stencil<float>(s, nab, part, nx) : current_stencil<double>(s, nab, part, nx);
}

// The weighted projections of the nonlocal current, Uw[o][ilma][w]
// (current.f90:225-273), from the sphere values when they are current.
cudaError_t launch_current_proj(System& s) {
  if (!s.Nlma || !s.nitems) return cudaSuccess;
  cudaError_t e;
  const size_t smem = s.prec == SGPU_PREC_C64 ? UvwGeom<float>::smem : UvwGeom<double>::smem;
  if (smem > 48 * 1024) {  // set on every call: the attribute is per device
    e = s.prec == SGPU_PREC_C64
            ? cudaFuncSetAttribute(k_uvpsi_w<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
            : cudaFuncSetAttribute(k_uvpsi_w<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 gu(s.nitems, s.nkl, (s.NBocc + 31) / 32 * s.uvw_split);
  // the compact sphere values are current after every Taylor step: 4x fewer bytes than gathering from zu
  const bool fromS = s.S_valid && s.Sbuf;
  const int ld = fromS ? s.nsp : s.NL;
  const int* idx = fromS ? s.qmap : s.idx_proj;
  if (s.prec == SGPU_PREC_C64)
    k_uvpsi_w<float><<<gu, 256, smem, s.launch_stream()>>>(fromS ? (const float2*)s.Sbuf : (const float2*)s.zu, ld,
                                                            s.NBocc, s.zproj64, s.Nlma, s.Nps, idx, s.atom_off,
                                                            s.rpos, s.items, s.lma_list, s.uvw_split, s.norb,
                                                            s.Uw);
  else
    k_uvpsi_w<double><<<gu, 256, smem, s.launch_stream()>>>(fromS ? (const double2*)s.Sbuf : (const double2*)s.zu,
                                                             ld, s.NBocc, s.zproj64, s.Nlma, s.Nps, idx, s.atom_off,
                                                             s.rpos, s.items, s.lma_list, s.uvw_split, s.norb,
                                                            s.Uw);
  return cudaGetLastError();
}

cudaError_t launch_current(System& s, double* jav_dev) {
  double* part = s.red;                              // [norb][nx][4], nx <= part_rows
  double* jo = part + (size_t)s.norb * s.part_rows * 4;  // [norb][3]
  if ((size_t)s.norb * s.part_rows * 4 + 3 * (size_t)s.norb + 12 > s.red_elems) return cudaErrorInvalidValue;
  int nx = 1;
  cudaError_t e;
  if (!s.cur_valid) {
    e = launch_current_stencil(s, part, nx);
    if (e != cudaSuccess) return e;
  }
  if ((e = launch_current_proj(s)) != cudaSuccess) return e;
  if (s.cur_valid) {  // computed by the Taylor step that produced these orbitals (flag_current),
    // on the second stream: the projections above overlap them; the sums wait here
    e = s.aux_join();
    if (e != cudaSuccess) return e;
    part = s.cur_part;
    nx = s.cur_nx;
  }
  k_current_comb<<<(s.norb + COMB_T / 32 - 1) / (COMB_T / 32), COMB_T, 0, s.launch_stream()>>>(part, nx, s.Uw, s.uvw_split, s.occ_o, s.kAc_d, s.iuV_d,
                                                                     s.norb, s.NBocc, s.Nlma, s.Hxyz, 1.0 / s.aLxyz,
                                                                     jo);
  k_current_sum<<<1, 256, 0, s.launch_stream()>>>(jo, s.norb, jav_dev);
  return cudaGetLastError();
}

// -------------------------------------------------------------- energy ---
// per orbital: occ Re(tpsum) Hxyz + occ |k|^2/2 and occ sum |U|^2 iuV
__global__ void k_energy_comb(const double* __restrict__ part, int nx, const double2* __restrict__ U,
                              const double* __restrict__ occ_o, const double* __restrict__ kAc,
                              const int* __restrict__ iuV, int norb, int NBocc, int Nlma, double Hxyz,
                              double* __restrict__ eo) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= norb) return;
  double tr = 0;
  for (int x = 0; x < nx; ++x) tr += part[((size_t)o * nx + x) * 2];  // per-orbital rows, in order
  const int kl = o / NBocc;
  const double occ = occ_o[o];
  const double k2 = kAc[3 * kl] * kAc[3 * kl] + kAc[3 * kl + 1] * kAc[3 * kl + 1] + kAc[3 * kl + 2] * kAc[3 * kl + 2];
  double en = 0;
  for (int l = 0; l < Nlma; ++l) {
    const double2 u = U[(size_t)o * Nlma + l];      // Hxyz * sum uV ekr psi
    en += occ * (u.x * u.x + u.y * u.y) * (double)iuV[l];
  }
  eo[2 * (size_t)o] = occ * tr * Hxyz + occ * k2 / 2.0;   // real part of occ*tpsum*Hxyz + occ*|k|^2/2
  eo[2 * (size_t)o + 1] = en;
}

__global__ void k_energy_sum(const double* __restrict__ eo, int norb, double* __restrict__ e) {
  __shared__ double sh[32 * 2];
  double v[2] = {0, 0};
  for (int o = threadIdx.x; o < norb; o += blockDim.x) {
    v[0] += eo[2 * (size_t)o];
    v[1] += eo[2 * (size_t)o + 1];
  }
  block_sum<2>(v, sh);
  if (threadIdx.x == 0) {
    e[0] = v[0];
    e[1] = v[1];
  }
}

// sgpu_energy_terms, before (one CTA per plane; 32x32 and 48x48 planes a nine-plane march) and
// with the forward march, ms: 20^3 x 2048 orbitals complex(8) 1.24 / 0.26, 32^3 x 2048
// complex(4) 1.08 / 0.74, 48^3 x 800 1.97 / 1.34, 16^3 x 1024 0.37 / 0.09.
cudaError_t launch_energy(System& s, double* e_dev) {
  double* part = s.red;                                // [norb][nx][2], nx <= part_rows
  double* eo = part + 2 * (size_t)s.norb * s.part_rows;  // [norb][2]
  if (2 * (size_t)s.norb * s.part_rows + 2 * (size_t)s.norb + 32 > s.red_elems) return cudaErrorInvalidValue;
  int nx = 1;
  cudaError_t err = s.prec == SGPU_PREC_C64 ? fwd_march<float, true>(s, part, nx) : fwd_march<double, true>(s, part, nx);
  if (err != cudaSuccess) return err;
  // U = Hxyz * sum conj(zproj) psi = Hxyz * sum uV ekr psi  (total_energy.f90:191-197), FP64 projectors
  if (s.Nlma) {
    err = launch_uvpsi(s, s.zu, 0, s.norb, s.NBocc, false);
    if (err != cudaSuccess) return err;
  }
  k_energy_comb<<<(s.norb + 127) / 128, 128, 0, s.launch_stream()>>>(part, nx, s.U, s.occ_o, s.kAc_d, s.iuV_d,
                                                                    s.norb, s.NBocc, s.Nlma, s.Hxyz, eo);
  k_energy_sum<<<1, 256, 0, s.launch_stream()>>>(eo, s.norb, e_dev);
  return cudaGetLastError();
}

}  // namespace sgpu
