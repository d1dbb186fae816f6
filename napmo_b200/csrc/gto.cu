// Contracted Cartesian Gaussian basis functions (and their gradients) on grid
// points: phi_mu(r) = N_c sum_k c_k N_k (x-Ax)^lx (y-Ay)^ly (z-Az)^lz
// exp(-zeta_k |r-A|^2), nAPMO src/system/gto.cpp:41-51,182-192.
//
// The exponentials of a shell are evaluated once and shared by its Cartesian
// components.  Shells whose
// smallest exponent gives zeta_min r^2 > 746 are skipped: exp() of any
// argument below -745.2 is exactly zero in double precision, so the skip does
// not change a single value.  Output is basis-major phi[mu * ld + p] so that
// consecutive threads write consecutive addresses.
#include "common.h"
#include "kernels.cuh"

namespace napmo {

namespace {

constexpr int kGtoThreads = 128;
constexpr int kMaxComp = 15;  // Cartesian components up to L = 4

__device__ __forceinline__ double ipow(double x, int n) {
  double r = 1.0;
  for (int i = 0; i < n; ++i) r *= x;
  return r;
}

// Values alone.  A full shell of angular momentum L, with everything about it
// known at compile time but the order of its components: powers of dx, dy, dz in
// registers, the component's by selection.  Sums and products run in the order of
// gto_grad_kernel.
template <int L>
__device__ __forceinline__ void shell_values(const DeviceBasis &b, const int *info, double zmin,
                                             double dx, double dy, double dz, double *phi,
                                             long ld) {
  constexpr int N = (L + 1) * (L + 2) / 2;
  const int f0 = __ldg(info + 0), p0 = __ldg(info + 2), np = __ldg(info + 3),
            c0 = __ldg(info + 4);
  double r2 = 0.0;
  r2 += dx * dx;
  r2 += dy * dy;
  r2 += dz * dz;
  double acc[N];
#pragma unroll
  for (int c = 0; c < N; ++c) acc[c] = 0.0;
  if (zmin * r2 <= 746.0) {
    for (int k = 0; k < np; ++k) {
      const double a = __ldg(b.prim_zeta + p0 + k) * r2;
      if (a > 746.0) continue;  // exp(-a) is zero (see the file's comment)
      const double e = exp(-a);
#pragma unroll
      for (int c = 0; c < N; ++c) acc[c] += __ldg(b.coef + c0 + c * np + k) * e;
    }
  }
  double px[L + 1], py[L + 1], pz[L + 1];
  px[0] = py[0] = pz[0] = 1.0;
#pragma unroll
  for (int k = 1; k <= L; ++k) {
    px[k] = px[k - 1] * dx;
    py[k] = py[k - 1] * dy;
    pz[k] = pz[k - 1] * dz;
  }
  auto power = [](const double(&w)[L + 1], int l) {
    double v = w[0];
#pragma unroll
    for (int k = 1; k <= L; ++k) v = l == k ? w[k] : v;
    return v;
  };
#pragma unroll
  for (int c = 0; c < N; ++c) {
    const int *l = b.func_l + 3 * (f0 + c);
    phi[(long)(f0 + c) * ld] =
        power(px, __ldg(l)) * power(py, __ldg(l + 1)) * power(pz, __ldg(l + 2)) * acc[c];
  }
}

// A shell whose components are not all present (any l).
__device__ __noinline__ void partial_shell_values(const DeviceBasis &b, const int *info,
                                                  double zmin, double dx, double dy, double dz,
                                                  double *phi, long ld) {
  const int f0 = info[0], ncomp = info[1], p0 = info[2], np = info[3], c0 = info[4];
  double r2 = 0.0;
  r2 += dx * dx;
  r2 += dy * dy;
  r2 += dz * dz;
  for (int c = 0; c < ncomp; ++c) {
    double acc = 0.0;
    if (zmin * r2 <= 746.0)
      for (int k = 0; k < np; ++k) acc += b.coef[c0 + c * np + k] * exp(-b.prim_zeta[p0 + k] * r2);
    const int *l = b.func_l + 3 * (f0 + c);
    phi[(long)(f0 + c) * ld] = ipow(dx, l[0]) * ipow(dy, l[1]) * ipow(dz, l[2]) * acc;
  }
}

// CTA = (128 points, kGtoShells shells), thread = point.  Bound by the
// exponentials of the occupied neighbourhood and by writing phi; one thread per
// point over all shells, with components and powers in run-time loops, left
// both far off (C4H10 75 x 194, 179 MB of phi: 291 us; this 100, of which
// writing takes 27).
constexpr int kGtoShells = 8;
__global__ void __launch_bounds__(kGtoThreads, 8)
gto_values_kernel(DeviceBasis b, int npoint, const double *__restrict__ gx,
                  const double *__restrict__ gy, const double *__restrict__ gz,
                  double *__restrict__ phi, long ld) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npoint) return;
  const double px = gx[p], py = gy[p], pz = gz[p];
  const int s1 = min(b.nshell, (int)(blockIdx.y + 1) * kGtoShells);
  for (int s = blockIdx.y * kGtoShells; s < s1; ++s) {
    const int *info = b.shell_info + 6 * s;
    const double *cen = b.shell_center + 4 * s;
    const double dx = px - __ldg(cen + 0);
    const double dy = py - __ldg(cen + 1);
    const double dz = pz - __ldg(cen + 2);
    const double zmin = __ldg(cen + 3);
    const int L = __ldg(info + 5), ncomp = __ldg(info + 1);
    switch (2 * ncomp == (L + 1) * (L + 2) ? L : -1) {
      case 0: shell_values<0>(b, info, zmin, dx, dy, dz, phi + p, ld); break;
      case 1: shell_values<1>(b, info, zmin, dx, dy, dz, phi + p, ld); break;
      case 2: shell_values<2>(b, info, zmin, dx, dy, dz, phi + p, ld); break;
      case 3: shell_values<3>(b, info, zmin, dx, dy, dz, phi + p, ld); break;
      case 4: shell_values<4>(b, info, zmin, dx, dy, dz, phi + p, ld); break;
      default: partial_shell_values(b, info, zmin, dx, dy, dz, phi + p, ld);
    }
  }
}

// Values and gradients: one thread per point walks all shells.
__global__ void __launch_bounds__(kGtoThreads)
gto_grad_kernel(DeviceBasis b, int npoint, const double *__restrict__ gx,
           const double *__restrict__ gy, const double *__restrict__ gz,
           double *__restrict__ phi, long ld, double *__restrict__ grad) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npoint) return;
  const double px = gx[p], py = gy[p], pz = gz[p];
  const long plane = (long)b.nfunc * ld;
  for (int s = 0; s < b.nshell; ++s) {
    const int *info = b.shell_info + 6 * s;
    const int f0 = __ldg(info + 0), ncomp = __ldg(info + 1), p0 = __ldg(info + 2),
              np = __ldg(info + 3), c0 = __ldg(info + 4);
    const double *cen = b.shell_center + 4 * s;
    const double dx = px - __ldg(cen + 0);
    const double dy = py - __ldg(cen + 1);
    const double dz = pz - __ldg(cen + 2);
    double r2 = 0.0;
    r2 += dx * dx;
    r2 += dy * dy;
    r2 += dz * dz;
    double acc[kMaxComp], accz[kMaxComp];
#pragma unroll
    for (int c = 0; c < kMaxComp; ++c) {
      acc[c] = 0.0;
      accz[c] = 0.0;
    }
    if (__ldg(cen + 3) * r2 <= 746.0) {
      for (int k = 0; k < np; ++k) {
        const double zeta = __ldg(b.prim_zeta + p0 + k);
        const double e = exp(-zeta * r2);
#pragma unroll
        for (int c = 0; c < kMaxComp; ++c) {
          if (c < ncomp) {
            const double t = __ldg(b.coef + c0 + c * np + k) * e;
            acc[c] += t;
            accz[c] += t * zeta;
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < kMaxComp; ++c) {
      if (c < ncomp) {
        const int f = f0 + c;
        const int lx = __ldg(b.func_l + 3 * f), ly = __ldg(b.func_l + 3 * f + 1),
                  lz = __ldg(b.func_l + 3 * f + 2);
        const double px_ = ipow(dx, lx), py_ = ipow(dy, ly), pz_ = ipow(dz, lz);
        phi[(long)f * ld + p] = px_ * py_ * pz_ * acc[c];
        // d/dx [x^lx e^{-zeta r^2}] = lx x^(lx-1) - 2 zeta x^(lx+1)
        const double gxv = (lx ? lx * ipow(dx, lx - 1) * acc[c] : 0.0) -
                           2.0 * ipow(dx, lx + 1) * accz[c];
        const double gyv = (ly ? ly * ipow(dy, ly - 1) * acc[c] : 0.0) -
                           2.0 * ipow(dy, ly + 1) * accz[c];
        const double gzv = (lz ? lz * ipow(dz, lz - 1) * acc[c] : 0.0) -
                           2.0 * ipow(dz, lz + 1) * accz[c];
        grad[(long)f * ld + p] = gxv * py_ * pz_;
        grad[plane + (long)f * ld + p] = px_ * gyv * pz_;
        grad[2 * plane + (long)f * ld + p] = px_ * py_ * gzv;
      }
    }
  }
}

}  // namespace

cudaError_t launch_basis_values(const DeviceBasis &b, int npoint, const double *x,
                                const double *y, const double *z, double *phi,
                                long ld, double *grad, cudaStream_t s) {
  if (npoint <= 0 || b.nfunc == 0) return cudaSuccess;
  const int blocks = (npoint + kGtoThreads - 1) / kGtoThreads;
  if (grad)
    gto_grad_kernel<<<blocks, kGtoThreads, 0, s>>>(b, npoint, x, y, z, phi, ld, grad);
  else
    gto_values_kernel<<<dim3(blocks, (b.nshell + kGtoShells - 1) / kGtoShells), kGtoThreads, 0,
                        s>>>(b, npoint, x, y, z, phi, ld);
  return cudaGetLastError();
}

}  // namespace napmo
