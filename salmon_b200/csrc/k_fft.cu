// Batched 3D FFTs of grid functions and the Teter-Payne-Allan kinetic-energy
// preconditioner applied with them (ground-state CG).
//
// The FFT is a mixed-radix (2, 3) Stockham autosort transform of every line
// along one axis, in shared memory, FP64; a 3D transform is three axis passes.
// Grid sizes must be of the form 2^a 3^b (16, 24, 32, 48, 64, ...), at most
// FFT_NMAX points per axis.
//
// Teter, Payne and Allan, Phys. Rev. B 40, 12255 (1989): the residual is
// multiplied in reciprocal space by
//     K(x) = (27 + 18x + 12x^2 + 8x^3) / (27 + 18x + 12x^2 + 8x^3 + 16x^4),
// x = T(G) / T_band, with T(G) the kinetic energy of the plane wave G at k and
// T_band the kinetic energy of the band being optimised.  T(G) is taken as the
// symbol of the finite-difference kinetic operator of hpsi (the Nd=4
// Laplacian and the k.nabla term on this grid), so that K is consistent with
// the H that CG minimises.
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "sgpu_internal.cuh"

namespace sgpu {

constexpr int FFT_NMAX = 96;  // 2 x 16 lines x 96 x 16 B = 48 KB of shared memory
constexpr int FFT_TL = 16;       // lines per CTA
constexpr int FFT_THREADS = 256;

bool fft_size_ok(int n) {
  if (n < 1 || n > FFT_NMAX) return false;
  while (n % 2 == 0) n /= 2;
  while (n % 3 == 0) n /= 3;
  return n == 1;
}

// Lines of one axis: line L of vector v = (lo, li) with L = lo*ninner + li;
// element t sits at v*NL + lo*lo_stride + li + t*stride.
struct FftAxis {
  int n, nlines, ninner, lo_stride, stride;
  bool rows;  // the axis is the contiguous one (load whole rows)
};

__global__ void __launch_bounds__(FFT_THREADS) k_fft_lines(double2* __restrict__ data, int NL, FftAxis ax, int sign,
                                                            double scale) {
  extern __shared__ double2 fsm[];
  const int n = ax.n;
  double2* x = fsm;
  double2* y = fsm + FFT_TL * n;
  const int v = blockIdx.y;
  const int L0 = blockIdx.x * FFT_TL;
  const int nl = min(FFT_TL, ax.nlines - L0);
  double2* base = data + (size_t)v * NL;
  auto addr = [&](int l, int t) -> size_t {
    const int L = L0 + l;
    const int lo = L / ax.ninner, li = L - lo * ax.ninner;
    return (size_t)lo * ax.lo_stride + li + (size_t)t * ax.stride;
  };
  // load: coalesced along the contiguous direction of memory
  for (int e = threadIdx.x; e < nl * n; e += blockDim.x) {
    int l, t;
    if (ax.rows) { l = e / n; t = e - l * n; } else { t = e / nl; l = e - t * nl; }
    x[l * n + t] = base[addr(l, t)];
  }
  __syncthreads();
  int Ns = 1;
  int m = n;
  while (m > 1) {
    const int R = (m % 2 == 0) ? 2 : 3;
    m /= R;
    const int nR = n / R;
    for (int e = threadIdx.x; e < nl * nR; e += blockDim.x) {
      const int l = e / nR, j = e - l * nR;
      const int k = j % Ns;
      const double2* xl = x + l * n;
      double2* yl = y + l * n;
      // twiddle exp(sign * 2 pi i k r / (Ns R)) for r = 1..R-1
      double s1, c1;
      sincospi(2.0 * sign * k / (double)(Ns * R), &s1, &c1);
      const int idx = (j / Ns) * Ns * R + k;
      if (R == 2) {
        const double2 a = xl[j];
        const double2 b0 = xl[j + nR];
        const double2 b = make_double2(b0.x * c1 - b0.y * s1, b0.x * s1 + b0.y * c1);
        yl[idx] = make_double2(a.x + b.x, a.y + b.y);
        yl[idx + Ns] = make_double2(a.x - b.x, a.y - b.y);
      } else {
        const double c2 = c1 * c1 - s1 * s1, s2 = 2.0 * s1 * c1;
        const double2 a = xl[j];
        const double2 b0 = xl[j + nR], d0 = xl[j + 2 * nR];
        const double2 b = make_double2(b0.x * c1 - b0.y * s1, b0.x * s1 + b0.y * c1);
        const double2 d = make_double2(d0.x * c2 - d0.y * s2, d0.x * s2 + d0.y * c2);
        // size-3 DFT: w = exp(sign 2 pi i / 3) = -1/2 + sign i sqrt(3)/2
        const double h = 0.86602540378443864676 * sign;
        const double2 sp = make_double2(b.x + d.x, b.y + d.y), sm = make_double2(b.x - d.x, b.y - d.y);
        yl[idx] = make_double2(a.x + sp.x, a.y + sp.y);
        const double2 mid = make_double2(a.x - 0.5 * sp.x, a.y - 0.5 * sp.y);
        yl[idx + Ns] = make_double2(mid.x - h * sm.y, mid.y + h * sm.x);
        yl[idx + 2 * Ns] = make_double2(mid.x + h * sm.y, mid.y - h * sm.x);
      }
    }
    __syncthreads();
    double2* t = x;
    x = y;
    y = t;
    Ns *= R;
  }
  for (int e = threadIdx.x; e < nl * n; e += blockDim.x) {
    int l, t;
    if (ax.rows) { l = e / n; t = e - l * n; } else { t = e / nl; l = e - t * nl; }
    const double2 w = x[l * n + t];
    base[addr(l, t)] = make_double2(w.x * scale, w.y * scale);
  }
}

static FftAxis axis_of(const System& s, int d) {
  FftAxis a;
  if (d == 2) {  // z: rows of NLz
    a.n = s.NLz; a.nlines = s.NLx * s.NLy; a.ninner = 1; a.lo_stride = s.NLz; a.stride = 1; a.rows = true;
  } else if (d == 1) {  // y: lines (x, z), stride NLz
    a.n = s.NLy; a.nlines = s.NLx * s.NLz; a.ninner = s.NLz; a.lo_stride = s.NLy * s.NLz; a.stride = s.NLz;
    a.rows = false;
  } else {  // x: lines (y, z), stride NLy*NLz
    a.n = s.NLx; a.nlines = s.NLy * s.NLz; a.ninner = s.NLy * s.NLz; a.lo_stride = 0; a.stride = s.NLy * s.NLz;
    a.rows = false;
  }
  return a;
}

cudaError_t launch_fft3d(const System& s, double2* data, int nvec, int sign, bool normalise) {
  if (!fft_size_ok(s.NLx) || !fft_size_ok(s.NLy) || !fft_size_ok(s.NLz)) return cudaErrorInvalidValue;
  for (int d = 2; d >= 0; --d) {
    const FftAxis a = axis_of(s, d);
    const size_t smem = 2 * (size_t)FFT_TL * a.n * sizeof(double2);
    dim3 grid((a.nlines + FFT_TL - 1) / FFT_TL, nvec);
    k_fft_lines<<<grid, FFT_THREADS, smem, s.launch_stream()>>>(data, s.NL, a, sign, normalise ? 1.0 / a.n : 1.0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Kinetic symbol of the FD operator along one axis for the phase th = 2 pi m / n
// per grid step: -1/2 (lap0 + 2 sum lap_n cos(n th)) + 2 k sum nab_n sin(n th)
__device__ __forceinline__ double fd_symbol(const double* lap, const double* nab, double k, double th) {
  double t = lap[0];
  double g = 0.0;
#pragma unroll
  for (int n = 1; n <= 4; ++n) {
    double sn, cs;
    sincos(n * th, &sn, &cs);
    t += 2.0 * lap[n] * cs;
    g += nab[n] * sn;
  }
  return -0.5 * t + 2.0 * k * g;
}

struct TpaArgs {
  int NLx, NLy, NLz, NL;
  double lap[3][5], nab[3][5];
};

// data[v] (reciprocal space) *= K(T(G)/T_band[v]) with the k-point of vector v
__global__ void k_tpa_scale(double2* __restrict__ data, TpaArgs a, const double* __restrict__ kAc,
                            const double* __restrict__ tband, int kl_of_vec_stride, const int* __restrict__ kidx) {
  const int v = blockIdx.y;
  const int kl = kidx ? kidx[v] : v / kl_of_vec_stride;
  const double kx = kAc[3 * kl], ky = kAc[3 * kl + 1], kz = kAc[3 * kl + 2];
  const double tb = fmax(tband[v], 1e-6);
  const double pi2 = 6.28318530717958647692;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.NL; i += gridDim.x * blockDim.x) {
    const int ix = i / (a.NLy * a.NLz), iy = (i / a.NLz) % a.NLy, iz = i % a.NLz;
    const int mx = ix <= a.NLx / 2 ? ix : ix - a.NLx;
    const int my = iy <= a.NLy / 2 ? iy : iy - a.NLy;
    const int mz = iz <= a.NLz / 2 ? iz : iz - a.NLz;
    const double T = 0.5 * (kx * kx + ky * ky + kz * kz) + fd_symbol(a.lap[0], a.nab[0], kx, pi2 * mx / a.NLx) +
                     fd_symbol(a.lap[1], a.nab[1], ky, pi2 * my / a.NLy) +
                     fd_symbol(a.lap[2], a.nab[2], kz, pi2 * mz / a.NLz);
    const double x = fmax(T, 0.0) / tb;
    const double p = 27.0 + x * (18.0 + x * (12.0 + 8.0 * x));
    const double K = p / (p + 16.0 * x * x * x * x);
    double2* d = data + (size_t)v * a.NL + i;
    *d = make_double2(d->x * K, d->y * K);
  }
}

// ------------------------------------------------------- fused transforms --
// A factor in reciprocal space costs six axis transforms.  One launch each (plus the
// factor, the conversion of a real input and the epilogue) is ten launches of a few us on
// grids of a few thousand points, all latency.  Here a CTA transforms a whole x-plane
// along z and y in shared memory, and the x lines run forward, through the factor and
// backward in one kernel: three launches.  Radix 4, 2 and 3 Stockham passes with the
// twiddles of a line length tabulated once per CTA.
// The potential update's kernels (cold caches): 8^3 52 -> 22 us, 18x24x27 63 -> 29 us.
__device__ __forceinline__ double2 tw_mul(double2 b, double2 w) {
  return make_double2(b.x * w.x - b.y * w.y, b.x * w.y + b.y * w.x);
}

// tw[t] = exp(sign 2 pi i t / n)
__device__ __forceinline__ void fft_twiddles(double2* tw, int n, int sign) {
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    double sn, cs;
    sincospi(2.0 * sign * t / (double)n, &sn, &cs);
    tw[t] = make_double2(cs, sn);
  }
}

// nl lines of n points, element t of line l at l * ls + t * es, from x through y and back;
// returns the buffer that holds the result.  Starts and ends with a CTA barrier.
__device__ double2* fft_lines_smem(double2* x, double2* y, int nl, int n, int ls, int es, int sign, const double2* tw) {
  int Ns = 1, m = n;
  __syncthreads();
  while (m > 1) {
    const int R = m % 4 == 0 ? 4 : (m % 2 == 0 ? 2 : 3);
    m /= R;
    const int nR = n / R, ts = n / (Ns * R);
    for (int e = threadIdx.x; e < nl * nR; e += blockDim.x) {
      // neighbouring threads on neighbouring addresses: along the line, or across lines
      const int l = es == 1 ? e / nR : e % nl, j = es == 1 ? e - l * nR : e / nl;
      const int k = j % Ns, t = k * ts, idx = (j / Ns) * Ns * R + k;
      const double2* xl = x + l * ls;
      double2* yl = y + l * ls;
      const double2 a = xl[j * es];
      if (R == 4) {
        const double2 b = tw_mul(xl[(j + nR) * es], tw[t]), c = tw_mul(xl[(j + 2 * nR) * es], tw[2 * t]),
                      d = tw_mul(xl[(j + 3 * nR) * es], tw[3 * t]);
        const double2 s0 = cadd(a, c), s1 = csub(a, c), s2 = cadd(b, d), s3 = csub(b, d);
        const double2 i3 = sign < 0 ? make_double2(s3.y, -s3.x) : make_double2(-s3.y, s3.x);  // sign i s3
        yl[idx * es] = cadd(s0, s2);
        yl[(idx + Ns) * es] = cadd(s1, i3);
        yl[(idx + 2 * Ns) * es] = csub(s0, s2);
        yl[(idx + 3 * Ns) * es] = csub(s1, i3);
      } else if (R == 2) {
        const double2 b = tw_mul(xl[(j + nR) * es], tw[t]);
        yl[idx * es] = cadd(a, b);
        yl[(idx + Ns) * es] = csub(a, b);
      } else {
        const double2 b = tw_mul(xl[(j + nR) * es], tw[t]), d = tw_mul(xl[(j + 2 * nR) * es], tw[2 * t]);
        // size-3 DFT: w = exp(sign 2 pi i / 3) = -1/2 + sign i sqrt(3)/2
        const double h = 0.86602540378443864676 * sign;
        const double2 sp = cadd(b, d), sm = csub(b, d);
        const double2 mid = make_double2(a.x - 0.5 * sp.x, a.y - 0.5 * sp.y);
        yl[idx * es] = cadd(a, sp);
        yl[(idx + Ns) * es] = make_double2(mid.x - h * sm.y, mid.y + h * sm.x);
        yl[(idx + 2 * Ns) * es] = make_double2(mid.x + h * sm.y, mid.y - h * sm.x);
      }
    }
    __syncthreads();
    double2* sw = x;
    x = y;
    y = sw;
    Ns *= R;
  }
  return x;
}

constexpr int FFP_THREADS = 512;
constexpr int FFX_TL = 8;  // x lines per CTA of the middle kernel

// rows padded by one value: the y lines of neighbouring z fall in distinct banks, and so do
// the rows of the z lines
static size_t fft_plane_smem(const System& s) {
  return (2 * (size_t)s.NLy * (s.NLz + 1) + s.NLy + s.NLz) * sizeof(double2);
}
bool fft_fused_ok(const System& s) {
  return fft_size_ok(s.NLx) && fft_size_ok(s.NLy) && fft_size_ok(s.NLz) && fft_plane_smem(s) <= 220 * 1024;
}

// One x-plane of vector blockIdx.y along z and y (forward: z first; backward: y first), from
// real (or null) or from z, in place or, with EPI, into the epilogue f(index, value).
template <bool REAL_IN, typename Epi>
__device__ __forceinline__ void fft_plane(const double* real, const double2* zin, int NLx, int NLy, int NLz, int sign,
                                          Epi&& out) {
  extern __shared__ double2 fsm[];
  const int ld = NLz + 1, NYZ = NLy * NLz, pl = NLy * ld;
  double2 *x = fsm, *y = fsm + pl, *twy = fsm + 2 * pl, *twz = twy + NLy;
  const size_t off = (size_t)blockIdx.y * NLx * NYZ + (size_t)blockIdx.x * NYZ;
  fft_twiddles(twy, NLy, sign);
  fft_twiddles(twz, NLz, sign);
  for (int i = threadIdx.x; i < NYZ; i += blockDim.x)
    x[(i / NLz) * ld + i % NLz] = REAL_IN ? make_double2(real[off + i], 0.0) : zin[off + i];
  double2* r = fft_lines_smem(x, y, NLy, NLz, ld, 1, sign, twz);
  r = fft_lines_smem(r, r == x ? y : x, NLz, NLy, 1, ld, sign, twy);
  for (int i = threadIdx.x; i < NYZ; i += blockDim.x) out(off + i, r[(i / NLz) * ld + i % NLz]);
}

template <bool REAL_IN>
__global__ void __launch_bounds__(FFP_THREADS) k_fft_planes(const double* __restrict__ real, double2* z, int NLx, int NLy,
                                                           int NLz, int sign, double scale) {
  fft_plane<REAL_IN>(real, z, NLx, NLy, NLz, sign,
                     [&](size_t i, double2 v) { z[i] = make_double2(v.x * scale, v.y * scale); });
}

// x lines forward, the factor fac(v, ix, iy, iz), backward
template <typename Fac>
__device__ __forceinline__ void fft_mid(double2* z, int NLx, int NYZ, Fac&& fac) {
  extern __shared__ double2 fsm[];
  const int n = NLx, l0 = blockIdx.x * FFX_TL, nl = min(FFX_TL, NYZ - l0), v = blockIdx.y;
  double2 *x = fsm, *y = fsm + FFX_TL * n, *twf = fsm + 2 * FFX_TL * n, *twb = twf + n;
  double2* base = z + (size_t)v * n * NYZ + l0;
  fft_twiddles(twf, n, -1);
  fft_twiddles(twb, n, +1);
  for (int e = threadIdx.x; e < nl * n; e += blockDim.x) {
    const int t = e / nl, l = e - t * nl;
    x[t * FFX_TL + l] = base[(size_t)t * NYZ + l];
  }
  double2* r = fft_lines_smem(x, y, nl, n, 1, FFX_TL, -1, twf);
  for (int e = threadIdx.x; e < nl * n; e += blockDim.x) {
    const int t = e / nl, l = e - t * nl;
    const double f = fac(v, t, l0 + l);
    const double2 w = r[t * FFX_TL + l];
    r[t * FFX_TL + l] = make_double2(w.x * f, w.y * f);
  }
  r = fft_lines_smem(r, r == x ? y : x, nl, n, 1, FFX_TL, +1, twb);
  for (int e = threadIdx.x; e < nl * n; e += blockDim.x) {
    const int t = e / nl, l = e - t * nl;
    base[(size_t)t * NYZ + l] = r[t * FFX_TL + l];
  }
}

// rho(G) -> Vh(G) = 4 pi rho(G) / |G|^2 / NL, Vh(0) = 0 (Hartree.f90:71-80); |G| from
// the cell (G_d = 2 pi m_d / aL_d with m_d in [-N/2, N/2), Hartree.f90:38-62 and init.f90:52)
__global__ void __launch_bounds__(FFT_THREADS) k_fft_mid_poisson(double2* z, int NLx, int NLy, int NLz, double bx,
                                                                double by, double bz) {
  const double NL = (double)NLx * NLy * NLz;
  fft_mid(z, NLx, NLy * NLz, [&](int, int ix, int yz) -> double {
    const int iy = yz / NLz, iz = yz - iy * NLz;
    const int mx = ix < NLx - NLx / 2 ? ix : ix - NLx;
    const int my = iy < NLy - NLy / 2 ? iy : iy - NLy;
    const int mz = iz < NLz - NLz / 2 ? iz : iz - NLz;
    const double gx = mx * bx, gy = my * by, gz = mz * bz;
    const double G2 = gx * gx + gy * gy + gz * gz;
    return ix + yz == 0 ? 0.0 : 4.0 * 3.14159265358979323846 / G2 / NL;
  });
}

// the TPA factor of vector v (see k_tpa_scale) over NL; the axes' symbols are tabulated
__global__ void __launch_bounds__(FFT_THREADS) k_fft_mid_tpa(double2* z, TpaArgs a, const double* __restrict__ kAc,
                                                            const double* __restrict__ tband, int kl_of_vec_stride,
                                                            const int* __restrict__ kidx) {
  __shared__ double tx[FFT_NMAX], tyz[FFX_TL];
  const int v = blockIdx.y, kl = kidx ? kidx[v] : v / kl_of_vec_stride;
  const double kx = kAc[3 * kl], ky = kAc[3 * kl + 1], kz = kAc[3 * kl + 2];
  const double tb = fmax(tband[v], 1e-6), pi2 = 6.28318530717958647692;
  const int NYZ = a.NLy * a.NLz, l0 = blockIdx.x * FFX_TL;
  for (int i = threadIdx.x; i < a.NLx + FFX_TL; i += blockDim.x) {
    if (i < a.NLx) {
      const int mx = i <= a.NLx / 2 ? i : i - a.NLx;
      tx[i] = 0.5 * (kx * kx + ky * ky + kz * kz) + fd_symbol(a.lap[0], a.nab[0], kx, pi2 * mx / a.NLx);
    } else if (l0 + i - a.NLx < NYZ) {
      const int yz = l0 + i - a.NLx, iy = yz / a.NLz, iz = yz - iy * a.NLz;
      const int my = iy <= a.NLy / 2 ? iy : iy - a.NLy, mz = iz <= a.NLz / 2 ? iz : iz - a.NLz;
      tyz[i - a.NLx] = fd_symbol(a.lap[1], a.nab[1], ky, pi2 * my / a.NLy) +
                       fd_symbol(a.lap[2], a.nab[2], kz, pi2 * mz / a.NLz);
    }
  }
  const double inv = 1.0 / a.NL;
  fft_mid(z, a.NLx, NYZ, [&](int, int ix, int yz) -> double {  // (barriers lie between the tables and here)
    const double x = fmax(tx[ix] + tyz[yz - l0], 0.0) / tb;
    const double p = 27.0 + x * (18.0 + x * (12.0 + 8.0 * x));
    return inv * p / (p + 16.0 * x * x * x * x);
  });
}

static cudaError_t launch_fft_planes(const System& s, const double* real, double2* z, int nvec, int sign) {
  const size_t smem = fft_plane_smem(s);
  const cudaError_t e = raise_smem_limit(real ? (const void*)k_fft_planes<true> : (const void*)k_fft_planes<false>, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid(s.NLx, nvec);
  if (real) k_fft_planes<true><<<grid, FFP_THREADS, smem, s.launch_stream()>>>(real, z, s.NLx, s.NLy, s.NLz, sign, 1.0);
  else k_fft_planes<false><<<grid, FFP_THREADS, smem, s.launch_stream()>>>(nullptr, z, s.NLx, s.NLy, s.NLz, sign, 1.0);
  return cudaGetLastError();
}

static dim3 fft_mid_grid(const System& s, int nvec) { return dim3((s.NLy * s.NLz + FFX_TL - 1) / FFX_TL, nvec); }
static size_t fft_mid_smem(const System& s) { return (2 * (size_t)FFX_TL + 2) * s.NLx * sizeof(double2); }

cudaError_t launch_fft_planes_real(const System& s, const double* rho, double2* z) {
  return launch_fft_planes(s, rho, z, 1, -1);
}

cudaError_t launch_fft_mid_poisson(const System& s, double2* z) {
  const double pi2 = 6.28318530717958647692;
  k_fft_mid_poisson<<<fft_mid_grid(s, 1), FFT_THREADS, fft_mid_smem(s), s.launch_stream()>>>(
      z, s.NLx, s.NLy, s.NLz, pi2 / s.aL[0], pi2 / s.aL[1], pi2 / s.aL[2]);
  return cudaGetLastError();
}

// Perdew and Zunger, Phys. Rev. B 23, 5048 (1981), unpolarised: the exchange
// energy per electron -(3/4)(3/(2 pi))^(2/3)/rs plus the correlation fit
// (gamma/(1 + beta1 sqrt(rs) + beta2 rs) for rs >= 1, A ln rs + B + C rs ln rs + D rs
// below), as PZxc evaluates it (xc/builtin_pz.f90:45-76); vxc = exc + rho dexc/drho.
__device__ __forceinline__ void pz(double rho, double& exc, double& vxc) {  // rho: total density
  const double pi = 3.14159265358979323846;
  const double gammaU = -0.1423, beta1U = 1.0529, beta2U = 0.3334;
  const double AU = 0.0311, BU = -0.048, CU = 0.002, DU = -0.0116;
  const double cx = 0.75 * cbrt((3.0 / (2.0 * pi)) * (3.0 / (2.0 * pi)));
  const double tr = rho + 1e-10;
  const double rs = cbrt(3.0 / (4.0 * pi * tr));
  double e = -cx / rs;
  double de = e / (3.0 * tr);
  if (rs > 1.0) {
    const double sq = sqrt(rs);
    const double den = 1.0 + beta1U * sq + beta2U * rs;
    e += gammaU / den;
    de += gammaU * (0.5 * beta1U * sq + beta2U * rs) / (3.0 * tr) / (den * den);
  } else {
    const double ln = log(rs);
    e += AU * ln + BU + CU * rs * ln + DU * rs;
    de -= rs / (3.0 * tr) * (AU / rs + CU * (ln + 1.0) + DU);
  }
  exc = e;
  vxc = e + rho * de;
}

__device__ __forceinline__ double vloc_point(double vh, double rho, double vpsl, double (&acc)[2]) {
  double exc, vxc;
  pz(rho, exc, vxc);
  acc[0] = fma(0.5 * vh, rho, acc[0]);
  acc[1] = fma(exc, rho, acc[1]);
  return vh + vpsl + vxc;
}

// The CTA's energies into part; the last CTA to arrive adds all parts in CTA order, so the
// sum does not depend on which one it is.
__device__ __forceinline__ void vloc_energies(double (&acc)[2], double* part, double Hxyz, unsigned* count,
                                              double* energies) {
  __shared__ double sh[64];
  __shared__ unsigned arrived;
  block_allsum<2>(acc, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = acc[0];
    part[2 * blockIdx.x + 1] = acc[1];
    __threadfence();
    arrived = atomicAdd(count, 1u);
  }
  __syncthreads();
  if (arrived != gridDim.x - 1) return;  // whole CTA
  __threadfence();
  double v[2] = {0.0, 0.0};
  for (int i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
    v[0] += __ldcg(part + 2 * i);
    v[1] += __ldcg(part + 2 * i + 1);
  }
  block_allsum<2>(v, sh);
  if (threadIdx.x == 0) {
    energies[0] = v[0] * Hxyz;
    energies[1] = v[1] * Hxyz;
    *count = 0u;
  }
}

// the backward planes with Vloc = Re Vh + Vpsl + Vxc and its energies as the epilogue
__global__ void __launch_bounds__(FFP_THREADS) k_fft_planes_vloc(const double2* __restrict__ z, int NLx, int NLy, int NLz,
                                                                const double* __restrict__ rho,
                                                                const double* __restrict__ vpsl,
                                                                double* __restrict__ v64, float* __restrict__ v32,
                                                                double* part, double Hxyz, unsigned* count,
                                                                double* energies) {
  double acc[2] = {0.0, 0.0};
  fft_plane<false>(nullptr, z, NLx, NLy, NLz, +1, [&](size_t i, double2 vh) {
    const double v = vloc_point(vh.x, rho[i], vpsl[i], acc);
    v64[i] = v;
    v32[i] = (float)v;
  });
  vloc_energies(acc, part, Hxyz, count, energies);
}

cudaError_t launch_fft_planes_vloc(const System& s, const double2* z, const double* rho, double* part,
                                   double* energies_dev) {
  const size_t smem = fft_plane_smem(s);
  const cudaError_t e = raise_smem_limit((const void*)k_fft_planes_vloc, smem);
  if (e != cudaSuccess) return e;
  k_fft_planes_vloc<<<s.NLx, FFP_THREADS, smem, s.launch_stream()>>>(z, s.NLx, s.NLy, s.NLz, rho, s.vpsl, s.vloc64,
                                                                     s.vloc32, part, s.Hxyz, s.xc_count, energies_dev);
  return cudaGetLastError();
}

// Vloc from the transformed potential where the planes do not fit in shared memory
__global__ void __launch_bounds__(256) k_vloc(const double2* __restrict__ vh, const double* __restrict__ rho,
                                              const double* __restrict__ vpsl, int NL, double* __restrict__ v64,
                                              float* __restrict__ v32, double* part, double Hxyz, unsigned* count,
                                              double* energies) {
  double acc[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NL; i += gridDim.x * blockDim.x) {
    const double v = vloc_point(vh[i].x, rho[i], vpsl[i], acc);
    v64[i] = v;
    v32[i] = (float)v;
  }
  vloc_energies(acc, part, Hxyz, count, energies);
}

cudaError_t launch_vloc(const System& s, const double2* z, const double* rho, double* part, double* energies_dev) {
  k_vloc<<<148, 256, 0, s.launch_stream()>>>(z, rho, s.vpsl, s.NL, s.vloc64, s.vloc32, part, s.Hxyz, s.xc_count,
                                             energies_dev);
  return cudaGetLastError();
}

cudaError_t launch_tpa(const System& s, double2* data, int nvec, const double* tband_dev, int vecs_per_k,
                       const int* kidx_dev) {
  cudaError_t e;
  if (fft_fused_ok(s)) {
    TpaArgs a;
    a.NLx = s.NLx; a.NLy = s.NLy; a.NLz = s.NLz; a.NL = s.NL;
    for (int d = 0; d < 3; ++d)
      for (int n = 0; n < 5; ++n) { a.lap[d][n] = s.lap[d][n]; a.nab[d][n] = s.nab[d][n]; }
    if ((e = launch_fft_planes(s, nullptr, data, nvec, -1)) != cudaSuccess) return e;
    k_fft_mid_tpa<<<fft_mid_grid(s, nvec), FFT_THREADS, fft_mid_smem(s), s.launch_stream()>>>(
        data, a, s.kAc_d, tband_dev, vecs_per_k, kidx_dev);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return launch_fft_planes(s, nullptr, data, nvec, +1);
  }
  if ((e = launch_fft3d(s, data, nvec, -1, false)) != cudaSuccess) return e;
  TpaArgs a;
  a.NLx = s.NLx; a.NLy = s.NLy; a.NLz = s.NLz; a.NL = s.NL;
  for (int d = 0; d < 3; ++d)
    for (int n = 0; n < 5; ++n) { a.lap[d][n] = s.lap[d][n]; a.nab[d][n] = s.nab[d][n]; }
  dim3 grid((s.NL + 255) / 256 < 1024 ? (s.NL + 255) / 256 : 1024, nvec);
  k_tpa_scale<<<grid, 256, 0, s.launch_stream()>>>(data, a, s.kAc_d, tband_dev, vecs_per_k, kidx_dev);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return launch_fft3d(s, data, nvec, +1, true);
}

}  // namespace sgpu

extern "C" int sgpu_tpa_apply(sgpu_handle h, const void* in_dev, void* out_dev, int nvec, const int* kidx,
                              const double* tband) {
  using sgpu::System;
  if (!h || !in_dev || !out_dev || !tband || nvec < 1) {
    sgpu::set_last_error("sgpu_tpa_apply: bad argument");
    return SGPU_ERR_ARG;
  }
  System* s = h;
  std::vector<int> kv(nvec);
  for (int v = 0; v < nvec; ++v) {
    kv[v] = kidx ? kidx[v] : v;
    if (kv[v] < 0 || kv[v] >= s->nkl) {
      sgpu::set_last_error("sgpu_tpa_apply: k-point index outside the handle's k range");
      return SGPU_ERR_ARG;
    }
  }
  if (!(sgpu::fft_size_ok(s->NLx) && sgpu::fft_size_ok(s->NLy) && sgpu::fft_size_ok(s->NLz))) {
    sgpu::set_last_error("sgpu_tpa_apply: grid sizes must be 2^a 3^b <= 96");
    return SGPU_ERR_UNSUPPORTED;
  }
  double* tb = nullptr;
  int* kd = nullptr;
  cudaError_t e = cudaMalloc(&tb, (size_t)nvec * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&kd, (size_t)nvec * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyAsync(tb, tband, (size_t)nvec * sizeof(double), cudaMemcpyHostToDevice, s->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(kd, kv.data(), (size_t)nvec * sizeof(int), cudaMemcpyHostToDevice, s->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(out_dev, in_dev, (size_t)nvec * s->NL * sizeof(double2), cudaMemcpyDeviceToDevice, s->stream);
  if (e == cudaSuccess) e = sgpu::launch_tpa(*s, (double2*)out_dev, nvec, tb, 1, kd);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  cudaFree(tb);
  cudaFree(kd);
  if (e != cudaSuccess) {
    sgpu::set_last_error(std::string("sgpu_tpa_apply: ") + cudaGetErrorString(e));
    return SGPU_ERR_CUDA;
  }
  return 0;
}
