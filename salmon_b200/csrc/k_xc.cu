// Self-consistent local potential on the device: Hartree potential by FFT,
// Perdew-Zunger LDA exchange-correlation, and Vloc = Vh + Vpsl + Vexc
// (RT/dt_evolve.f90:190-207 with common/Hartree.f90 and xc/builtin_pz.f90).
#include <cuda_runtime.h>

#include "sgpu_internal.cuh"

namespace sgpu {

// rho (real) -> complex work array
__global__ void k_real_to_complex(const double* __restrict__ r, double2* __restrict__ z, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) z[i] = make_double2(r[i], 0.0);
}

// rho(G) -> Vh(G) = 4 pi rho(G) / |G|^2 / NL, Vh(0) = 0 (Hartree.f90:71-80); |G| from
// the cell (G_d = 2 pi m_d / aL_d with m_d in [-N/2, N/2), Hartree.f90:38-62 and init.f90:52)
__global__ void k_poisson(double2* __restrict__ z, int NLx, int NLy, int NLz, double bx, double by, double bz) {
  const int NL = NLx * NLy * NLz;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NL) return;
  const int ix = i / (NLy * NLz), iy = (i / NLz) % NLy, iz = i % NLz;
  const int mx = ix < NLx - NLx / 2 ? ix : ix - NLx;
  const int my = iy < NLy - NLy / 2 ? iy : iy - NLy;
  const int mz = iz < NLz - NLz / 2 ? iz : iz - NLz;
  const double gx = mx * bx, gy = my * by, gz = mz * bz;
  const double G2 = gx * gx + gy * gy + gz * gz;
  const double f = (i == 0) ? 0.0 : 4.0 * 3.14159265358979323846 / G2 / NL;
  z[i] = make_double2(z[i].x * f, z[i].y * f);
}

cudaError_t launch_update_vloc(const System& s, const double* rho_dev, double* energies_dev) {
  if (!fft_size_ok(s.NLx) || !fft_size_ok(s.NLy) || !fft_size_ok(s.NLz)) return cudaErrorInvalidValue;
  double2* z = s.stage;                               // NL complex work values
  double* part = s.xc_part;                           // 2 x XC_PARTS partial energies
  cudaError_t e;
  if (fft_fused_ok(s)) {
    if ((e = launch_fft_planes_real(s, rho_dev, z)) != cudaSuccess) return e;
    if ((e = launch_fft_mid_poisson(s, z)) != cudaSuccess) return e;
    return launch_fft_planes_vloc(s, z, rho_dev, part, energies_dev);
  }
  const int nb = (s.NL + 255) / 256;
  k_real_to_complex<<<nb, 256, 0, s.launch_stream()>>>(rho_dev, z, s.NL);
  if ((e = launch_fft3d(s, z, 1, -1, false)) != cudaSuccess) return e;
  const double pi2 = 6.28318530717958647692;
  k_poisson<<<nb, 256, 0, s.launch_stream()>>>(z, s.NLx, s.NLy, s.NLz, pi2 / s.aL[0], pi2 / s.aL[1], pi2 / s.aL[2]);
  if ((e = launch_fft3d(s, z, 1, +1, false)) != cudaSuccess) return e;
  return launch_vloc(s, z, rho_dev, part, energies_dev);
}

// The etrs potential history (RT/dt_evolve.f90:248-252, control/control_sc.f90:82):
// reset: hist1 = hist2 = Vloc;
// extrapolate: Vnew = 3 Vloc - 3 hist1 + hist2, hist2 = hist1, hist1 = Vloc, Vloc = Vnew
// (in FP64, with the FP32 copy of Vloc refreshed).
__global__ void k_vloc_history(double* __restrict__ v64, float* __restrict__ v32, double* __restrict__ h1,
                               double* __restrict__ h2, int NL, int extrapolate) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NL; i += gridDim.x * blockDim.x) {
    const double v = v64[i];
    if (extrapolate) {
      const double vn = 3.0 * v - 3.0 * h1[i] + h2[i];
      h2[i] = h1[i];
      h1[i] = v;
      v64[i] = vn;
      v32[i] = (float)vn;
    } else {
      h1[i] = v;
      h2[i] = v;
    }
  }
}

cudaError_t launch_vloc_history(const System& s, bool extrapolate) {
  if (!s.vloc_hist) return cudaErrorInvalidValue;
  k_vloc_history<<<(s.NL + 255) / 256, 256, 0, s.launch_stream()>>>(s.vloc64, s.vloc32, s.vloc_hist,
                                                                     s.vloc_hist + s.NL, s.NL, extrapolate ? 1 : 0);
  return cudaGetLastError();
}

}  // namespace sgpu
