// ch3d_step.cu -- the pressure Poisson pipeline (src/CFD_2nd/m_Poisson.f90:1078-
// 1201), the diagnostics and the 2nd-order statistics, and the solve without
// allocations.  FP64 and FP32 (mixed) instances.
//
// Per substep the device runs:
//   substep_setup  PMcoeUpdate + bulk-velocity reduction (ch3d_substep.cu)
//   ustar          right-hand sides and Crank-Nicolson solves (ch3d_march.cu, or
//                  ch3d_rhs.cu and ch3d_sweep.cu)
//   prsrc_xfft     clcPrSrcOther fused with the forward x R2C FFT
//   spectral       z FFT, y tridiagonal per (kx,kz) with the (0,0) pin, z iFFT
//   xifft          x C2R FFT * normfft -> phi
//   proj           FluidVelUpdate + the pressure update + next bulk partial sums,
//                  in the last substep the step's diagnostics
// and per step: step_end (limit checks).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>
#include "ch3d_ctx.h"
#include "ch3d_dev.cuh"
#include "ch3d_fft.cuh"

namespace ch3d {

// ---------------------------------------------------------------------------
// y tridiagonal per (kx,kz) (src/CFD_2nd/m_Poisson.f90:1114-1156):
// [am2Pr, ac2Pr + WaveNumX + WaveNumZ, ap2Pr], with the (kx,kz)=(0,0) system's
// first row replaced by the identity and zero right-hand side.  Solved in FP64
// in shared memory (also in the mixed path), partitioned over the block's threads
// but with per-system factors.  Block = TS consecutive kx at one kz.
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256) k_ysolve(Geo<T> g, Metrics<double> m, const double* __restrict__ wave,
                                                typename CplxOf<T>::type* __restrict__ spec, int TS, int P,
                                                const DevScalars* __restrict__ sc) {
  typedef typename CplxOf<T>::type CT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (sc->status) return;
  const int nx = g.nx, ny = g.ny, nxh = g.nxh;
  const int kx0 = blockIdx.x * TS, kz = blockIdx.y;
  const int Q = P - 1;
  double2* F = (double2*)smem_raw;               // ny * TS
  double* CP = (double*)(F + (size_t)ny * TS);   // ny * TS  (cp, later beta)
  double* AL = CP + (size_t)ny * TS;             // ny * TS
  double2* IFc = (double2*)(AL + (size_t)ny * TS); // TS * Q * 2
  double* RED = (double*)(IFc + (size_t)TS * (Q > 0 ? Q : 1) * 2);  // TS * Q * 5 : Minv(4), v
  const long long zs = (long long)nxh * ny;
  for (int t = threadIdx.x; t < ny * TS; t += blockDim.x) {
    const int s = t % TS, j = t / TS;
    const int kx = kx0 + s;
    double2 v = make_double2(0.0, 0.0);
    if (kx < nxh) {
      CT c = spec[kx + (long long)nxh * j + zs * kz];
      v = make_double2((double)c.x, (double)c.y);
    }
    F[t] = v;
  }
  __syncthreads();
  const double wz = wave[nx + kz];
  for (int t = threadIdx.x; t < TS * P; t += blockDim.x) {
    const int s = t % TS, p = t / TS;
    const int kx = kx0 + s;
    const double lam = wave[kx < nxh ? kx : 0] + wz;
    const bool pin = (kx == 0 && kz == 0);
    const int jlo = chunk_lo(p, ny, P), jhi = chunk_hi(p, ny, P);
    double cpp = 0.0, dal = 0.0;
    double2 d = make_double2(0.0, 0.0);
    for (int j = jlo; j <= jhi; ++j) {
      const int jc = j + 1;
      double a = m.am2Pr[jc], c = m.ap2Pr[jc], b = m.ac2Pr[jc] + lam;
      double2 f = F[j * TS + s];
      if (pin && j == 0) { a = 0.0; b = 1.0; c = 0.0; f = make_double2(0.0, 0.0); }
      const double mm = (j == jlo) ? b : b - a * cpp;
      const double rm = 1.0 / mm;
      const double cp = c * rm;
      if (j == jlo) { d.x = f.x * rm; d.y = f.y * rm; dal = -a * rm; }
      else { d.x = (f.x - a * d.x) * rm; d.y = (f.y - a * d.y) * rm; dal = -a * dal * rm; }
      F[j * TS + s] = d;
      CP[j * TS + s] = cp;
      AL[j * TS + s] = (p == 0) ? 0.0 : dal;
      cpp = cp;
    }
    double be = (p == P - 1) ? 0.0 : -CP[jhi * TS + s];
    double al = AL[jhi * TS + s];
    double2 y = F[jhi * TS + s];
    CP[jhi * TS + s] = be;
    for (int j = jhi - 1; j >= jlo; --j) {
      const double cp = CP[j * TS + s];
      const double2 dj = F[j * TS + s];
      y.x = dj.x - cp * y.x; y.y = dj.y - cp * y.y;
      al = AL[j * TS + s] - cp * al;
      be = -cp * be;
      F[j * TS + s] = y;
      AL[j * TS + s] = al;
      CP[j * TS + s] = be;
    }
  }
  __syncthreads();
  if (threadIdx.x < TS && Q > 0) {
    const int s = threadIdx.x;
    double* R = RED + (size_t)s * Q * 5;
    double2* G = IFc + (size_t)s * Q * 2;
    double m01p = 0.0, vprev = 0.0;
    double2 gu = make_double2(0.0, 0.0), gw;
    for (int q = 0; q < Q; ++q) {
      const int eq = chunk_hi(q, ny, P), sq1 = chunk_lo(q + 1, ny, P);
      const double l = -AL[eq * TS + s], v = -CP[sq1 * TS + s];
      double d00 = 1.0, d01 = -CP[eq * TS + s], d10 = -AL[sq1 * TS + s], d11 = 1.0;
      if (q > 0) d01 -= l * m01p * vprev;  // (L_q Minv_{q-1} U_{q-1}) has only a (0,1) entry
      const double r = 1.0 / (d00 * d11 - d01 * d10);
      const double M00 = d11 * r, M01 = -d01 * r, M10 = -d10 * r, M11 = d00 * r;
      double2 ru = F[eq * TS + s];
      if (q > 0) { ru.x -= l * gu.x; ru.y -= l * gu.y; }
      const double2 rw = F[sq1 * TS + s];
      gu = make_double2(M00 * ru.x + M01 * rw.x, M00 * ru.y + M01 * rw.y);
      gw = make_double2(M10 * ru.x + M11 * rw.x, M10 * ru.y + M11 * rw.y);
      G[2 * q] = gu; G[2 * q + 1] = gw;
      R[5 * q + 0] = M00; R[5 * q + 1] = M01; R[5 * q + 2] = M10; R[5 * q + 3] = M11; R[5 * q + 4] = v;
      m01p = M01; vprev = v;
    }
    double2 zw = G[2 * (Q - 1) + 1];
    for (int q = Q - 2; q >= 0; --q) {
      const double* Rq = R + 5 * q;
      const double fx = Rq[4] * zw.x, fy = Rq[4] * zw.y;
      double2 zu = G[2 * q], zwn = G[2 * q + 1];
      zu.x -= Rq[1] * fx; zu.y -= Rq[1] * fy;
      zwn.x -= Rq[3] * fx; zwn.y -= Rq[3] * fy;
      G[2 * q] = zu; G[2 * q + 1] = zwn;
      zw = zwn;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ny * TS; t += blockDim.x) {
    const int s = t % TS, j = t / TS;
    const int kx = kx0 + s;
    if (kx >= nxh) continue;
    const int p = chunk_of(j, ny, P);
    double2 x = F[t];
    const double2* G = IFc + (size_t)s * Q * 2;
    if (p > 0) { const double al = AL[t]; x.x += al * G[2 * (p - 1)].x; x.y += al * G[2 * (p - 1)].y; }
    if (p < P - 1) { const double be = CP[t]; x.x += be * G[2 * p + 1].x; x.y += be * G[2 * p + 1].y; }
    spec[kx + (long long)nxh * j + zs * kz] = mk((T)x.x, (T)x.y);
  }
}

// CheckDivergence, CalcVmax, CalcMaxCFL of the next step, CalcUxAver partials
// (src/CFD_2nd/m_Tools.f90:21-104,250-270).  A thread walks `rows` rows of
// one (i, k) column (uy(j+1) carried to the next row), a block of 32 x 4
// columns reduces its maxima and sum and issues one atomic per quantity
// (per-cell blocks made the same-address atomics the bottleneck).
template <class T>
__global__ void __launch_bounds__(128) k_diag(Geo<T> g, Metrics<T> m, const T* __restrict__ ux,
                                              const T* __restrict__ uy, const T* __restrict__ uz,
                                              double* __restrict__ part, DevScalars* __restrict__ sc, int rows) {
  __shared__ double red[6][4];
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), k = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int j0 = blockIdx.z * rows, j1 = min(j0 + rows, ny);
  double dv = 0, v0 = 0, v1 = 0, v2 = 0, cf = 0, s = 0;
  if (i < nx && k < nz) {
    const long long plane = (long long)nx * ny;
    const long long col = i + plane * k;
    const long long dxp = i + 1 == nx ? 1 - nx : 1;
    const long long dzp = k + 1 == nz ? -(long long)(nz - 1) * plane : plane;
    const double rdx = g.rdx, rdz = g.rdz;
    double b = uy[col + (long long)j0 * nx];
    const C4<T> c4(g);
    Nbr n4 = make_nbr(g, i, j0, k);  // the 4th-order divergence's neighbourhood, moved up row by row
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      if (j > j0) nbr_next_row(n4, g, j);
      const long long idx = col + (long long)j * nx;
      const int jc = j + 1;
      const double a = ux[idx], c = uz[idx];
      const double aip = ux[idx + dxp], ckp = uz[idx + dzp];
      const double bjp = j + 1 < ny ? (double)uy[idx + nx]
                                    : (g.bc.hi == 0 ? (double)uy[col] : (double)(T)g.bc.uy_hi);  // periodic: row 0
      const double rdyp = m.rdyp[jc];
      double d = fabs((aip - a) * rdx + (bjp - b) * rdyp + (ckp - c) * rdz);
      if (g.order == 4) d = fabs((double)div4_at(g, c4, m.rdyp[jc], ux, uy, uz, n4));
      // fmax(NaN, x) = x on the device, so NaN is folded into +inf first: a NaN
      // field still trips the limit checks of the step
      if (!(d == d)) d = INFINITY;
      dv = fmax(dv, d);
      v0 = fmax(v0, a == a ? fabs(a) : INFINITY);
      v1 = fmax(v1, b == b ? fabs(b) : INFINITY);
      v2 = fmax(v2, c == c ? fabs(c) : INFINITY);
      cf = fmax(cf, fabs(a + aip) * rdx + fabs(b + bjp) * rdyp + fabs(c + ckp) * rdz);
      s += a * (double)m.dyp[jc];
      b = bjp;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    dv = fmax(dv, __shfl_xor_sync(0xffffffffu, dv, o));
    v0 = fmax(v0, __shfl_xor_sync(0xffffffffu, v0, o));
    v1 = fmax(v1, __shfl_xor_sync(0xffffffffu, v1, o));
    v2 = fmax(v2, __shfl_xor_sync(0xffffffffu, v2, o));
    cf = fmax(cf, __shfl_xor_sync(0xffffffffu, cf, o));
    s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = cf; red[1][w] = dv; red[2][w] = v0; red[3][w] = v1; red[4][w] = v2; red[5][w] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r[6];
    for (int q = 0; q < 5; ++q) r[q] = fmax(fmax(red[q][0], red[q][1]), fmax(red[q][2], red[q][3]));
    r[5] = (red[5][0] + red[5][1]) + (red[5][2] + red[5][3]);
    atomic_max_nonneg(&sc->uddx, r[0] * 0.5);
    atomic_max_nonneg(&sc->divmax2, r[1]);
    atomic_max_nonneg(&sc->vmax[0], r[2]);
    atomic_max_nonneg(&sc->vmax[1], r[3]);
    atomic_max_nonneg(&sc->vmax[2], r[4]);
    part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = r[5];
  }
}

// max |div u| of the current field into *slot (for ch3d_project)
template <class T>
__global__ void __launch_bounds__(256) k_divmax(Geo<T> g, Metrics<T> m, const T* __restrict__ ux,
                                                const T* __restrict__ uy, const T* __restrict__ uz,
                                                unsigned long long* slot) {
  __shared__ double red[256];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  const int tl = threadIdx.x + blockDim.x * threadIdx.y;
  double dv = 0;
  if (i < g.nx && j < g.ny) {
    const int ip = wrapp(i, g.nx), kp = wrapp(k, g.nz);
    const long long idx = i + (long long)g.nx * (j + (long long)g.ny * k);
    dv = fabs(((double)ux[ip + (long long)g.nx * (j + (long long)g.ny * k)] - ux[idx]) * g.rdx +
              ((double)fld(uy, g, 1, i, j + 1, k) - uy[idx]) * m.rdyp[j + 1] +
              ((double)uz[i + (long long)g.nx * (j + (long long)g.ny * kp)] - uz[idx]) * g.rdz);
    if (g.order == 4) dv = fabs((double)div4_cell(g, C4<T>(g), m.rdyp[j + 1], ux, uy, uz, i, j, k));
  }
  red[tl] = dv;
  __syncthreads();
  for (int w = blockDim.x * blockDim.y / 2; w > 0; w >>= 1) {
    if (tl < w) red[tl] = fmax(red[tl], red[tl + w]);
    __syncthreads();
  }
  if (tl == 0) atomic_max_nonneg(slot, red[0]);
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
static dim3 cell_grid(const ch3d_ctx* c) { return dim3((c->nx + 31) / 32, (c->ny + 7) / 8, c->nz); }
static dim3 cell_block() { return dim3(32, 8, 1); }


// clcU1/2/3Hat_FEXP (src/CFD_2nd/m_TSchemeFEXP_inc.f90:391-488): u* = u + Rhs,
// every cell; between walls the uy row on the lower wall then takes uy_ym,
// as SetBC_and_UpdateHaloForPrSrc (src/CFD_2nd/m_BC_and_Halo.f90:349-405)
// sets it before the divergence.  blockIdx.y = component.
template <class T>
__global__ void __launch_bounds__(256) k_uhat_fexp(Geo<T> g, const T* __restrict__ ux, const T* __restrict__ uy,
                                                   const T* __restrict__ uz, const T* __restrict__ rx,
                                                   const T* __restrict__ ry, const T* __restrict__ rz,
                                                   T* __restrict__ sx, T* __restrict__ sy, T* __restrict__ sz,
                                                   const DevScalars* __restrict__ sc) {
  if (sc->status) return;
  const int comp = blockIdx.y;
  const T* u = comp == 0 ? ux : (comp == 1 ? uy : uz);
  const T* r = comp == 0 ? rx : (comp == 1 ? ry : rz);
  T* us = comp == 0 ? sx : (comp == 1 ? sy : sz);
  const long long plane = (long long)g.nx * g.ny;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < g.N; q += (long long)gridDim.x * blockDim.x) {
    T v = u[q] + r[q];
    if (comp == 1 && g.bc.lo != 0 && q % plane < g.nx) v = (T)g.bc.uy_lo;
    us[q] = v;
  }
}
template <class T> static cudaError_t uhat_fexp_t(ch3d_ctx* c) {
  T** f = (T**)c->f;
  const long long nb = (c->N + 255) / 256;
  const unsigned gx = (unsigned)(nb < 148LL * 16 ? nb : 148LL * 16);
  k_uhat_fexp<T><<<dim3(gx, 3), 256, 0, c->stream>>>(make_geo<T>(c), f[0], f[1], f[2], f[7], f[8], f[9], f[12], f[13],
                                                     f[14], c->sc);
  return cudaGetLastError();
}
cudaError_t launch_uhat_fexp(ch3d_ctx* c) { return c->fp32 ? uhat_fexp_t<float>(c) : uhat_fexp_t<double>(c); }



// The register-resident transforms where the length has a plan, else the generic ones (ch3d_fft.cu).
template <class T> static cudaError_t prsrc_t(ch3d_ctx* c, int mode) {
  typedef typename CplxOf<T>::type CT;
  cudaError_t e;
  if (launch_prsrc_xfft_r(c, mode, &e)) return e;
  if ((e = fft_generic_setup(c->device, c->fp32, c->planz)) != cudaSuccess) return e;
  T** f = (T**)c->f;
  const T* a = mode >= 2 ? f[10] : (mode == 1 ? f[0] : f[12]);
  return xfft_generic<T>(make_geo<T>(c), metrics_of<T>(c), a, mode == 1 ? f[1] : f[13], mode == 1 ? f[2] : f[14],
                         (CT*)c->spec, c->planx, (const CT*)c->twx, (const CT*)c->twr, mode, c->sc, f[3], c->stream);
}
cudaError_t launch_prsrc_xfft(ch3d_ctx* c, int mode) { return c->fp32 ? prsrc_t<float>(c, mode) : prsrc_t<double>(c, mode); }

template <class T> static cudaError_t zfft_t(ch3d_ctx* c, int inverse) {
  typedef typename CplxOf<T>::type CT;
  cudaError_t e;
  if (launch_zfft_r(c, inverse, &e)) return e;
  if ((e = fft_generic_setup(c->device, c->fp32, c->planz)) != cudaSuccess) return e;
  return zfft_generic<T>(make_geo<T>(c), (CT*)c->spec, c->planz, (const CT*)c->twz, inverse, c->sc, c->stream);
}
static cudaError_t zfft(ch3d_ctx* c, int inverse) { return c->fp32 ? zfft_t<float>(c, inverse) : zfft_t<double>(c, inverse); }
// forward z transform of the spectrum alone (the first step of the spectral solve)
cudaError_t launch_zfft_forward(ch3d_ctx* c) { return zfft(c, 0); }

cudaError_t launch_poisson_spectral(ch3d_ctx* c) {
  cudaError_t e = zfft(c, 0);
  if (e == cudaSuccess) e = launch_ysolve(c);
  return e == cudaSuccess ? zfft(c, 1) : e;
}

template <class T> static cudaError_t xifft_t(ch3d_ctx* c) {
  typedef typename CplxOf<T>::type CT;
  cudaError_t e;
  if (launch_xifft_r(c, &e)) return e;
  if ((e = fft_generic_setup(c->device, c->fp32, c->planz)) != cudaSuccess) return e;
  return xifft_generic<T>(make_geo<T>(c), (const CT*)c->spec, (T*)c->f[10], c->planx, (const CT*)c->twx,
                          (const CT*)c->twr, (T)c->normfft, c->sc, c->stream);
}
cudaError_t launch_xifft(ch3d_ctx* c) { return c->fp32 ? xifft_t<float>(c) : xifft_t<double>(c); }

cudaError_t launch_proj(ch3d_ctx* c, int mode) { return launch_proj_march(c, mode, false); }
cudaError_t launch_proj_diag(ch3d_ctx* c) { return launch_proj_march(c, 0, true); }
cudaError_t launch_bulk_partials(ch3d_ctx* c) { return launch_bulk_march(c); }

// rows per k_diag block: whole columns when the x-z plane alone gives about
// eight blocks per SM, shorter chunks on small grids
static int diag_rows(const ch3d_ctx* c) {
  const long long cols = (long long)((c->nx + 31) / 32) * ((c->nz + 3) / 4);
  const long long chunks = (148LL * 8 + cols - 1) / cols;
  const int rows = (int)((c->ny + chunks - 1) / chunks);
  return rows < 8 ? 8 : rows;
}
static dim3 diag_grid(const ch3d_ctx* c) {
  const int rows = diag_rows(c);
  return dim3((c->nx + 31) / 32, (c->nz + 3) / 4, (c->ny + rows - 1) / rows);
}
int diag_npart(const ch3d_ctx* c) {
  const dim3 g = diag_grid(c);
  return (int)(g.x * g.y * g.z);
}

template <class T> static cudaError_t diag_t(ch3d_ctx* c) {
  T** f = (T**)c->f;
  k_diag<T><<<diag_grid(c), 128, 0, c->stream>>>(make_geo<T>(c), metrics_of<T>(c), f[0], f[1], f[2], c->part2, c->sc,
                                                 diag_rows(c));
  return cudaGetLastError();
}
cudaError_t launch_diag(ch3d_ctx* c) { return c->fp32 ? diag_t<float>(c) : diag_t<double>(c); }

template <class T> static cudaError_t divmax_t(ch3d_ctx* c, unsigned long long* slot) {
  T** f = (T**)c->f;
  k_divmax<T><<<cell_grid(c), cell_block(), 0, c->stream>>>(make_geo<T>(c), metrics_of<T>(c), f[0], f[1], f[2], slot);
  return cudaGetLastError();
}
template <class T> __global__ void k_fill_row0(T* __restrict__ a, int nx, int ny, int nz, T v) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nx * nz) return;
  const int i = (int)(t % nx), k = (int)(t / nx);
  a[i + (long long)nx * ny * k] = v;
}
// FP64 <-> FP32 conversion of n values (mixed-precision upload/download)
__global__ void k_f64_to_f32(const double* __restrict__ a, float* __restrict__ b, long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    b[t] = (float)a[t];
}
__global__ void k_f32_to_f64(const float* __restrict__ a, double* __restrict__ b, long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    b[t] = (double)a[t];
}
cudaError_t launch_convert(ch3d_ctx* c, const void* src, void* dst, long long n, int to_f32) {
  const long long nb = (n + 255) / 256;
  const unsigned g = (unsigned)(nb < 148LL * 32 ? nb : 148LL * 32);
  if (n <= 0) return cudaSuccess;
  if (to_f32) k_f64_to_f32<<<g, 256, 0, c->stream>>>((const double*)src, (float*)dst, n);
  else k_f32_to_f64<<<g, 256, 0, c->stream>>>((const float*)src, (double*)dst, n);
  return cudaGetLastError();
}

cudaError_t launch_fill_row0(ch3d_ctx* c, int q, double v) {
  const unsigned nb = (unsigned)(((long long)c->nx * c->nz + 255) / 256);
  if (c->fp32) k_fill_row0<float><<<nb, 256, 0, c->stream>>>((float*)c->f[q], c->nx, c->ny, c->nz, (float)v);
  else k_fill_row0<double><<<nb, 256, 0, c->stream>>>((double*)c->f[q], c->nx, c->ny, c->nz, v);
  return cudaGetLastError();
}

cudaError_t launch_divmax(ch3d_ctx* c, unsigned long long* slot) {
  return c->fp32 ? divmax_t<float>(c, slot) : divmax_t<double>(c, slot);
}

// ---------------------------------------------------------------------------
// clcStat_CH moment sums (src/CFD_2nd/m_FlowType_Channel.f90:175-330), FP64
// accumulation in both precision modes.  Block (j, k-chunk); blockIdx.x == ny
// is the nyp row (:296-316).  Partials are summed in a fixed order by
// k_stats_finalize, so the statistics are deterministic.
// ---------------------------------------------------------------------------
#define CH3D_NSTAT 35

template <class T>
__device__ __forceinline__ double fd(const T* a, const Geo<T>& g, int comp, int i, int j, int k) {
  return (double)fld(a, g, comp, i, j, k);
}

template <class T>
__global__ void __launch_bounds__(256) k_stats(Geo<T> g, Metrics<double> m, const T* __restrict__ ux,
                                               const T* __restrict__ uy, const T* __restrict__ uz,
                                               const T* __restrict__ pr, double* __restrict__ part, int kch) {
  __shared__ double wred[CH3D_NSTAT][8];
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int j = blockIdx.x;  // 0..ny-1 interior rows (jc = j+1); ny: the nyp row
  const int k0 = blockIdx.y * kch, k1 = min(nz, k0 + kch);
  double S[CH3D_NSTAT];
#pragma unroll
  for (int q = 0; q < CH3D_NSTAT; ++q) S[q] = 0.0;
  const double rdx = (double)g.rdx, rdz = (double)g.rdz, rdx2 = (double)g.rdx2, rdz2 = (double)g.rdz2;
  const double rdxh = rdx * 0.5;
  if (j < ny) {
    const int jc = j + 1;
    const double InterpY1 = 0.5 * m.yinterp[jc], InterpY2 = 0.5 - InterpY1;
    const double cac = m.rdyc[jc], cacU = m.rdyc[jc + 1], caj = m.rdyp[jc];
    for (int k = k0; k < k1; ++k) {
      const int km = wrapm(k, nz), kp = wrapp(k, nz);
      for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        const int im = wrapm(i, nx), ip = wrapp(i, nx);
        const double uxloc = fd(ux, g, 0, i, j, k), uyloc = fd(uy, g, 1, i, j, k), uzloc = fd(uz, g, 2, i, j, k);
        const double prloc = fd(pr, g, 3, i, j, k);
        const double ux_ip = fd(ux, g, 0, ip, j, k), ux_im = fd(ux, g, 0, im, j, k);
        const double ux_jm = fd(ux, g, 0, i, j - 1, k), ux_jp = fd(ux, g, 0, i, j + 1, k);
        const double ux_km = fd(ux, g, 0, i, j, km), ux_kp = fd(ux, g, 0, i, j, kp);
        const double uy_jp = fd(uy, g, 1, i, j + 1, k), uy_im = fd(uy, g, 1, im, j, k), uy_ip = fd(uy, g, 1, ip, j, k);
        const double uy_jm = fd(uy, g, 1, i, j - 1, k), uy_km = fd(uy, g, 1, i, j, km), uy_kp = fd(uy, g, 1, i, j, kp);
        const double uy_im_jp = fd(uy, g, 1, im, j + 1, k);
        const double uz_kp = fd(uz, g, 2, i, j, kp), uz_km = fd(uz, g, 2, i, j, km);
        const double uz_im = fd(uz, g, 2, im, j, k), uz_ip = fd(uz, g, 2, ip, j, k);
        const double uz_jm = fd(uz, g, 2, i, j - 1, k), uz_jp = fd(uz, g, 2, i, j + 1, k);
        const double uxCell = 0.5 * (uxloc + ux_ip);
        const double uyCell = 0.5 * (uyloc + uy_jp);
        const double uzCell = 0.5 * (uzloc + uz_kp);
        const double prloc2 = InterpY1 * (fd(pr, g, 3, im, j - 1, k) + fd(pr, g, 3, i, j - 1, k)) +
                              InterpY2 * (fd(pr, g, 3, im, j, k) + prloc);
        const double dudx = (ux_ip - uxloc) * rdx, dudy = (uxloc - ux_jm) * cac, dudz = (uxloc - ux_km) * rdz;
        const double dvdx = (uyloc - uy_im) * rdx, dvdy = (uy_jp - uyloc) * caj, dvdz = (uyloc - uy_km) * rdz;
        const double dwdx = (uzloc - uz_im) * rdx, dwdy = (uzloc - uz_jm) * cac, dwdz = (uz_kp - uzloc) * rdz;
        const double dudxx = (ux_ip - 2.0 * uxloc + ux_im) * rdx2;
        const double dudyy = m.ap2c[jc] * ux_jp + m.ac2c[jc] * uxloc + m.am2c[jc] * ux_jm;
        const double dudzz = (ux_kp - 2.0 * uxloc + ux_km) * rdz2;
        const double dvdxx = (uy_ip - 2.0 * uyloc + uy_im) * rdx2;
        const double dvdyy = m.ap2p[jc] * uy_jp + m.ac2p[jc] * uyloc + m.am2p[jc] * uy_jm;
        const double dvdzz = (uy_kp - 2.0 * uyloc + uy_km) * rdz2;
        const double dwdxx = (uz_ip - 2.0 * uzloc + uz_im) * rdx2;
        const double dwdyy = m.ap2c[jc] * uz_jp + m.ac2c[jc] * uzloc + m.am2c[jc] * uz_jm;
        const double dwdzz = (uz_kp - 2.0 * uzloc + uz_km) * rdz2;
        const double vor_x = dwdy - dvdz, vor_y = dudz - dwdx, vor_z = dvdx - dudy;
        const double dudxC = (ux_ip - ux_im) * rdxh;
        const double dvdxU = (uy_jp - uy_im_jp) * rdx;
        const double dudyU = (ux_jp - uxloc) * cacU;
        const double dvdyM = (uy_im_jp - uy_im) * caj;
        const double dudzC = (InterpY1 * (fd(ux, g, 0, i, j - 1, kp) - fd(ux, g, 0, i, j - 1, km)) +
                              InterpY2 * (ux_kp - ux_km)) * rdz;
        const double dvdzC = (fd(uy, g, 1, im, j, kp) - fd(uy, g, 1, im, j, km) + uy_kp - uy_km) * rdz * 0.25;
        S[0] += uxloc; S[1] += uyloc; S[2] += uzloc; S[3] += prloc;
        S[4] += uxloc * uxloc; S[5] += uyloc * uyloc; S[6] += uzloc * uzloc; S[7] += prloc * prloc;
        S[8] += uxCell * uyCell; S[9] += uyCell * uzCell; S[10] += uxCell * uzCell;
        S[11] += uxCell * prloc; S[12] += uyCell * prloc; S[13] += uzCell * prloc;
        S[14] += uxCell * uxCell * uyCell; S[15] += uyloc * uyloc * uyloc; S[16] += uzCell * uzCell * uyCell;
        S[17] += uxCell * uyCell * uyCell; S[18] += uxloc * uxloc * uxloc; S[19] += uzloc * uzloc * uzloc;
        S[20] += uxloc * uxloc * uxloc * uxloc; S[21] += uyloc * uyloc * uyloc * uyloc;
        S[22] += uzloc * uzloc * uzloc * uzloc;
        S[23] += prloc * dudx; S[24] += prloc * dvdy; S[25] += prloc * dwdz;
        S[26] += prloc2 * (dudy + dvdx);
        S[27] += uxloc * (dudxx + dudyy + dudzz); S[28] += uyloc * (dvdxx + dvdyy + dvdzz);
        S[29] += uzloc * (dwdxx + dwdyy + dwdzz);
        S[30] += dudxC * (dvdxU + dvdx) * 0.5 + (dudyU + dudy) * (dvdyM + dvdy) * 0.25;
        S[31] += dudzC * dvdzC;
        S[32] += vor_x * vor_x; S[33] += vor_y * vor_y; S[34] += vor_z * vor_z;
      }
    }
  } else {
    // jc = nyp: ghost row above the last cell (SetBC_and_UpdateHalo values)
    const int jc = ny + 1, jm = ny - 1;
    const double cac = m.rdyc[jc];
    const double InterpY1 = 0.5 * m.yinterp[jc], InterpY2 = 0.5 - InterpY1;
    for (int k = k0; k < k1; ++k)
      for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        const int im = wrapm(i, nx);
        const double prloc2 = InterpY1 * (fd(pr, g, 3, im, jm, k) + fd(pr, g, 3, i, jm, k)) +
                              InterpY2 * (fd(pr, g, 3, im, ny, k) + fd(pr, g, 3, i, ny, k));
        const double dudy = (fd(ux, g, 0, i, ny, k) - fd(ux, g, 0, i, jm, k)) * cac;
        const double dwdy = (fd(uz, g, 2, i, ny, k) - fd(uz, g, 2, i, jm, k)) * cac;
        const double vor_x = dwdy, vor_z = -dudy;
        S[26] += prloc2 * (dudy + 0.0);
        S[32] += vor_x * vor_x;
        S[34] += vor_z * vor_z;
      }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < CH3D_NSTAT; ++q) {
    double v = S[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) wred[q][w] = v;
  }
  __syncthreads();
  if (threadIdx.x < CH3D_NSTAT) {
    double v = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) v += wred[threadIdx.x][q];
    part[((size_t)j * gridDim.y + blockIdx.y) * CH3D_NSTAT + threadIdx.x] = v;
  }
}

// SumStat(:,jc) += sum of the partials * inxz (m_FlowType_Channel.f90:290-293);
// PrGradsum += PrGradAver (:318).
__global__ void k_stats_finalize(const double* __restrict__ part, int nch, double inxz, double* __restrict__ sumstat,
                                 DevScalars* sc, double* prgradsum) {
  const int j = blockIdx.x, q = threadIdx.x;
  if (q < CH3D_NSTAT) {
    double v = 0.0;
    for (int c = 0; c < nch; ++c) v += part[((size_t)j * nch + c) * CH3D_NSTAT + q];
    sumstat[(size_t)j * CH3D_NSTAT + q] += v * inxz;
  }
  if (j == 0 && q == 0) *prgradsum += sc->PrGradAver;
}

template <class T> static cudaError_t stats_t(ch3d_ctx* c) {
  T** f = (T**)c->f;
  const int kch = (c->nz + 7) / 8;
  const int nch = (c->nz + kch - 1) / kch;
  k_stats<T><<<dim3(c->ny + 1, nch), 256, 0, c->stream>>>(make_geo<T>(c), c->m64full, f[0], f[1], f[2], f[3],
                                                           c->statpart, kch);
  k_stats_finalize<<<c->ny + 1, 64, 0, c->stream>>>(c->statpart, nch, 1.0 / ((double)c->nx * (double)c->nz), c->stat,
                                                   c->sc, c->stat + (size_t)CH3D_NSTAT * (c->ny + 1));
  return cudaGetLastError();
}
cudaError_t launch_stats(ch3d_ctx* c) { return c->fp32 ? stats_t<float>(c) : stats_t<double>(c); }

// ---------------------------------------------------------------------------
// Allocation-free Poisson solve (ch3d_poisson_noalloc in include/ch3d.h).
// Its working memory is this file-scope device array, present on every GPU
// that loads the library until the process exits.  In host code the name
// g_noalloc_scratch is only a host-side stand-in for the symbol; the device
// address is obtained once per device with cudaGetSymbolAddress (with that
// device current) and cached.  All calls share the array.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_noalloc_scratch[CH3D_NOALLOC_SCRATCH_BYTES];

namespace {
// per device: the scratch array's device address and the kernels' shared-memory limits set
PerDevice g_noalloc_site;
void* g_noalloc_addr[kMaxDevices] = {nullptr};
constexpr int kNoallocSmemLimit = 200 * 1024;

size_t align256(size_t b) { return (b + 255) / 256 * 256; }
}  // namespace

// Once per device (that device current): looks up the array's device address
// and sets the dynamic shared-memory limits of the kernels the solve runs.
cudaError_t noalloc_scratch_address(int dev, void** out) {
  cudaError_t e = once_per_device(g_noalloc_site, dev, [&] {
    void* p = nullptr;
    cudaError_t r = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (r != cudaSuccess) return r;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    FFTPlanDev p9 = {}, p16 = {};  // both radix sets of z plans
    p16.npass = 1;
    p16.radix[0] = 16;
    if ((r = fft_generic_setup(dev, false, p9)) != cudaSuccess) return r;
    if ((r = fft_generic_setup(dev, false, p16)) != cudaSuccess) return r;
    if ((r = cudaFuncSetAttribute(k_ysolve<double>, a, kNoallocSmemLimit)) != cudaSuccess) return r;
    g_noalloc_addr[dev] = p;
    return cudaSuccess;
  });
  if (e == cudaSuccess) *out = g_noalloc_addr[dev];
  return e;
}

// Launch shape of the allocation-free solve's y kernel: threads per system,
// systems per block and its dynamic shared memory.
struct NoallocShape {
  int P, TS;
  size_t smy;
};
static NoallocShape noalloc_shape(int ny) {
  NoallocShape s;
  int P = 16;
  while (P > 1 && ny < 2 * P) P >>= 1;
  s.P = P;
  s.TS = 8;
  const int Q = P - 1;
  s.smy = (size_t)ny * s.TS * (sizeof(double2) + 2 * sizeof(double)) +
          (size_t)s.TS * (Q > 0 ? Q : 1) * (2 * sizeof(double2) + 5 * sizeof(double)) + 16;
  return s;
}

// Largest dynamic shared memory (bytes) one kernel of the solve asks for; the
// solve runs only where it is within noalloc_smem_limit().
size_t noalloc_smem(int ny, const FFTPlanDev& planx, const FFTPlanDev& planz) {
  const size_t f = fft_generic_smem(planx, planz), y = noalloc_shape(ny).smy;
  return f > y ? f : y;
}
size_t noalloc_smem_limit() { return (size_t)kNoallocSmemLimit; }

// Bytes of scratch the solve of an nx x ny x nz grid needs.
size_t noalloc_bytes(int nx, int ny, int nz) {
  const int nxh = nx / 2 + 1, M = nx / 2;
  size_t b = align256((size_t)nxh * ny * nz * sizeof(double2));
  b += align256((size_t)4 * (ny + 3) * sizeof(double));     // rdyp, am2Pr, ac2Pr, ap2Pr
  b += align256((size_t)(nx + nz) * sizeof(double));        // WaveNumX | WaveNumZ
  b += align256((size_t)(M + M + 1 + nz) * sizeof(double2)); // twiddles
  b += align256(sizeof(DevScalars));
  return b;
}

cudaError_t poisson_noalloc(int nx, int ny, int nz, double xlx, double zlz, const double* yp, int bclo, int bchi,
                            const double* d_src, double* d_phi, cudaStream_t st, const FFTPlanDev& planx,
                            const FFTPlanDev& planz) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  void* base = nullptr;
  e = noalloc_scratch_address(dev, &base);
  if (e != cudaSuccess) return e;
  const int nxh = nx / 2 + 1, M = nx / 2, L = ny + 3;
  unsigned char* p = (unsigned char*)base;
  double2* spec = (double2*)p;
  p += align256((size_t)nxh * ny * nz * sizeof(double2));
  double* met = (double*)p;
  p += align256((size_t)4 * L * sizeof(double));
  double* wave = (double*)p;
  p += align256((size_t)(nx + nz) * sizeof(double));
  double2* tw = (double2*)p;
  p += align256((size_t)(M + M + 1 + nz) * sizeof(double2));
  DevScalars* sc = (DevScalars*)p;

  // host tables: the Poisson metrics of InitMeshAndMetries (m_MeshAndMetries.f90:186-240),
  // the modified wavenumbers (m_Poisson.f90:38-66) and the FFT twiddles
  std::vector<double> h(4 * (size_t)L, 0.0), dyp(L, 0.0), dyc(L, 0.0), yc(L, 0.0), rdyc(L, 0.0);
  const int nyp = ny + 1;
  auto Y = [&](int j) { return yp[j - 1]; };
  for (int j = 1; j <= ny; ++j) { yc[j] = 0.5 * (Y(j) + Y(j + 1)); dyp[j] = Y(j + 1) - Y(j); }
  dyp[0] = dyp[1]; dyp[nyp] = dyp[ny];
  for (int j = 2; j <= ny; ++j) dyc[j] = yc[j] - yc[j - 1];
  dyc[1] = dyp[1]; dyc[nyp] = dyp[ny];
  double* rdyp = h.data();
  double *am = h.data() + L, *ac = h.data() + 2 * L, *ap = h.data() + 3 * L;
  for (int j = 0; j <= nyp; ++j) rdyp[j] = 1.0 / dyp[j];
  for (int j = 1; j <= nyp; ++j) rdyc[j] = 1.0 / dyc[j];
  for (int j = 1; j <= ny; ++j) { am[j] = rdyp[j] * rdyc[j]; ap[j] = rdyp[j] * rdyc[j + 1]; }
  if (bclo != 0) { am[1] = 0.0; ap[1] = rdyp[1] * rdyc[2]; }
  if (bchi != 0) { am[ny] = rdyp[ny] * rdyc[ny]; ap[ny] = 0.0; }
  for (int j = 1; j <= ny; ++j) ac[j] = -(am[j] + ap[j]);
  const double PIv = 3.141592653589793238462643383279502884;
  const double rdx = (double)nx / xlx, rdz = (double)nz / zlz;
  std::vector<double> w(nx + nz);
  for (int i = 0; i < nx; ++i) w[i] = 2.0 * rdx * rdx * (std::cos(2.0 * PIv * (double)i / (double)nx) - 1.0);
  for (int k = 0; k < nz; ++k) w[nx + k] = 2.0 * rdz * rdz * (std::cos(2.0 * PIv * (double)k / (double)nz) - 1.0);
  std::vector<double2> t(M + M + 1 + nz);
  auto fill = [&](double2* o, int n, int cnt) {
    for (int q = 0; q < cnt; ++q) {
      long double ang = -2.0L * 3.141592653589793238462643383279502884L * (long double)q / (long double)n;
      o[q] = make_double2((double)cosl(ang), (double)sinl(ang));
    }
  };
  fill(t.data(), M, M);
  fill(t.data() + M, nx, M + 1);
  fill(t.data() + 2 * M + 1, nz, nz);
  if ((e = cudaMemcpyAsync(met, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(wave, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(tw, t.data(), t.size() * sizeof(double2), cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
  // what must start at zero: the status word and the divergence maximum
  if ((e = cudaMemsetAsync(sc, 0, sizeof(DevScalars), st)) != cudaSuccess) return e;

  Geo<double> g;
  std::memset(&g, 0, sizeof(g));
  g.nx = nx; g.ny = ny; g.nz = nz; g.nxh = nxh; g.N = (long long)nx * ny * nz;
  g.rdx = rdx; g.rdz = rdz; g.rdx2 = rdx * rdx; g.rdz2 = rdz * rdz;
  g.bc.lo = bclo; g.bc.hi = bchi;
  g.bc.dyp1 = dyp[1]; g.bc.dypN = dyp[nyp];
  Metrics<double> m;
  std::memset(&m, 0, sizeof(m));
  m.rdyp = met; m.am2Pr = met + L; m.ac2Pr = met + 2 * L; m.ap2Pr = met + 3 * L;
  const double2* twx = tw;
  const double2* twr = tw + M;
  const double2* twz = tw + 2 * M + 1;

  // forward x transform of the source (mode 2: the source is read as is)
  const NoallocShape sh = noalloc_shape(ny);
  if ((e = xfft_generic<double>(g, m, d_src, d_src, d_src, spec, planx, twx, twr, 2, sc, nullptr, st)) != cudaSuccess ||
      (e = zfft_generic<double>(g, spec, planz, twz, 0, sc, st)) != cudaSuccess)
    return e;
  k_ysolve<double><<<dim3((nxh + sh.TS - 1) / sh.TS, nz), sh.TS * sh.P < 64 ? 64 : sh.TS * sh.P, sh.smy, st>>>(
      g, m, wave, spec, sh.TS, sh.P, sc);
  if ((e = cudaGetLastError()) != cudaSuccess ||
      (e = zfft_generic<double>(g, spec, planz, twz, 1, sc, st)) != cudaSuccess ||
      (e = xifft_generic<double>(g, spec, d_phi, planx, twx, twr, 1.0 / ((double)nx * (double)nz), sc, st)) != cudaSuccess)
    return e;
  // the host tables above are pageable and local to this call
  return cudaStreamSynchronize(st);
}

}  // namespace ch3d
