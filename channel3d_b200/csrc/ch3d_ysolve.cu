// ch3d_ysolve.cu -- the y systems of the pressure Poisson solve, one complex
// tridiagonal system per (kx, kz) column of the (kx, j, kz) spectrum:
// [am2Pr, ac2Pr + WaveNumX + WaveNumZ, ap2Pr] between walls
// (src/CFD_2nd/m_Poisson.f90:1114-1156), cyclic when y is periodic (:954-1073).
//
// The elimination factors depend on the mode only and are computed once per
// run.  With them, the forward elimination and the back substitution are
// first-order linear recurrences with known coefficients, so a column is cut
// into chunks of rows that stay in registers: each chunk runs its recurrence
// from zero, the chunks' (coefficient product, end value) pairs are combined
// by a scan over the chunks, and the chunk repeats the recurrence from its
// true start value.
#include "ch3d_ctx.h"
#include "ch3d_dev.cuh"

namespace ch3d {

// The kz of block row y: kz and nz-kz next to each other, because their
// systems share the factors (WaveNumZ is even in kz): the second read hits L2.
__device__ __forceinline__ int kz_of_block(int y, int nz) {
  return y == 0 ? 0 : ((y & 1) ? (y + 1) / 2 : nz - y / 2);
}

// Factors of the Thomas elimination (InverseTridiagonal, m_Tools.f90:224-251),
// one thread per (kx, |kz|) column: rm_j = 1 / (b_j - a_j cp_{j-1}), cp_j =
// c_j rm_j (formed where it is used); row 1 of the (0,0) system is replaced by
// phi = 0 (m_Poisson.f90:1136-1140).  In FP64, stored in precision R, layout
// ((kzh * ny) + j) * ldx + kx.
template <class R>
__global__ void __launch_bounds__(128) k_ythomas_factors(Metrics<double> m, const double* __restrict__ wave, int nx,
                                                         int ny, R* __restrict__ RMf, int ldx, int kxn) {
  const int kx = blockIdx.x * blockDim.x + threadIdx.x, kzh = blockIdx.y;
  if (kx >= kxn) return;
  const double lam = wave[kx] + wave[nx + kzh];
  const bool pin = (kx == 0 && kzh == 0);
  double cp = 0.0;
  for (int j = 0; j < ny; ++j) {
    const int jc = j + 1;
    double a = m.am2Pr[jc], c = m.ap2Pr[jc], b = m.ac2Pr[jc] + lam;
    if (pin && j == 0) { a = 0.0; b = 1.0; c = 0.0; }
    const double rm = 1.0 / (j == 0 ? b : b - a * cp);
    cp = c * rm;
    RMf[((size_t)kzh * ny + j) * ldx + kx] = (R)rm;
  }
}

// Factors of the cyclic systems (InversePeriodicTridiagonal,
// src/CFD_2nd/m_Tools.f90:109-162; row 1 of the (0,0) system replaced by
// phi = 0, m_Poisson.f90:1012-1029), one thread per (kx, |kz|), FP64, layout
// ((kzh * ny) + j) * nxh + kx:
//   PP_0 = b_1 (row 1 divides), PP_j = 1 / (b + a arrmn1_{j-1}) (ppj),
//   A1_j = arrmn1_j, A1_{n-1} = the closing denominator,
//   A2_j = arrmn2_j after the backward pass.
__global__ void __launch_bounds__(128) k_ycyclic_factors(Metrics<double> m, const double* __restrict__ wave, int nx,
                                                         int ny, int nxh, double* __restrict__ PP,
                                                         double* __restrict__ A1, double* __restrict__ A2) {
  const int kx = blockIdx.x * blockDim.x + threadIdx.x, kzh = blockIdx.y;
  if (kx >= nxh) return;
  const double lam = wave[kx] + wave[nx + kzh];
  const bool pin = (kx == 0 && kzh == 0);
  const size_t st = (size_t)nxh, o = (size_t)kzh * ny * st + kx;
  auto coef = [&](int j, double& a, double& b, double& c) {
    a = m.am2Pr[j + 1]; c = m.ap2Pr[j + 1]; b = m.ac2Pr[j + 1] + lam;
    if (pin && j == 0) { a = 0.0; b = 1.0; c = 0.0; }
  };
  double a, b, c;
  coef(0, a, b, c);
  double v1 = -c / b, v2 = -a / b;
  PP[o] = b; A1[o] = v1; A2[o] = v2;
  for (int j = 1; j <= ny - 2; ++j) {
    coef(j, a, b, c);
    const double ppj = 1.0 / (b + a * v1);
    v1 = -c * ppj;
    v2 = -a * v2 * ppj;
    PP[o + st * j] = ppj; A1[o + st * j] = v1; A2[o + st * j] = v2;
  }
  // backward pass: arrmn2_n = 1, arrmn2_j += arrmn1_j arrmn2_{j+1}
  double w = 1.0;
  A2[o + st * (ny - 1)] = w;
  for (int j = ny - 2; j >= 0; --j) {
    w = A2[o + st * j] + A1[o + st * j] * w;
    A2[o + st * j] = w;
  }
  coef(ny - 1, a, b, c);
  A1[o + st * (ny - 1)] = c * A2[o] + a * A2[o + st * (ny - 2)] + b;
}

template <class T> struct Vec2Of;
template <> struct Vec2Of<double> { typedef double2 type; };
template <> struct Vec2Of<float> { typedef float2 type; };

// ---------------------------------------------------------------------------
// Chunked solve.  A block owns C columns; thread (column c, chunk p) holds RPT
// consecutive rows in registers.  Composition of two maps d -> A d + B:
// (A2, B2) after (A1, B1) = (A2 A1, B2 + A2 B1); the products of the
// elimination coefficients are at most 1 in magnitude.
// ---------------------------------------------------------------------------
template <class R> struct Aff { R A, x, y; };
template <class R> __device__ __forceinline__ Aff<R> after(const Aff<R>& f2, const Aff<R>& f1) {
  return {f2.A * f1.A, f2.x + f2.A * f1.x, f2.y + f2.A * f1.y};
}

// Exclusive scan over the chunks of a column (UP: from chunk 0 upwards, else
// from the last chunk downwards) of the chunks' maps; returns the value the
// recurrence enters this thread's chunk with, starting from zero.
// agg: [warps][C] in shared memory.
template <class R, int C, bool UP>
__device__ __forceinline__ void chunk_scan(Aff<R> f, Aff<R>* agg, int lane, int warp, int nwarps, int c, R& dx, R& dy) {
  constexpr int CW = 32 / C;  // chunks per warp
  const int q = UP ? lane / C : CW - 1 - lane / C;  // position of the chunk within its warp, in scan order
#pragma unroll
  for (int o = 1; o < CW; o <<= 1) {
    Aff<R> g;
    if (UP) {
      g.A = __shfl_up_sync(0xffffffffu, f.A, o * C);
      g.x = __shfl_up_sync(0xffffffffu, f.x, o * C);
      g.y = __shfl_up_sync(0xffffffffu, f.y, o * C);
    } else {
      g.A = __shfl_down_sync(0xffffffffu, f.A, o * C);
      g.x = __shfl_down_sync(0xffffffffu, f.x, o * C);
      g.y = __shfl_down_sync(0xffffffffu, f.y, o * C);
    }
    if (q >= o) f = after(f, g);
  }
  if (q == CW - 1) agg[warp * C + c] = f;
  __syncthreads();
  dx = (R)0; dy = (R)0;
  for (int w = 0; w < nwarps - 1; ++w) {  // the warps before this one, in scan order
    const int wq = UP ? w : nwarps - 1 - w;
    if (UP ? wq >= warp : wq <= warp) break;
    const Aff<R> g = agg[wq * C + c];
    dx = g.x + g.A * dx;
    dy = g.y + g.A * dy;
  }
  Aff<R> e;
  if (UP) {
    e.A = __shfl_up_sync(0xffffffffu, f.A, C % 32);
    e.x = __shfl_up_sync(0xffffffffu, f.x, C % 32);
    e.y = __shfl_up_sync(0xffffffffu, f.y, C % 32);
  } else {
    e.A = __shfl_down_sync(0xffffffffu, f.A, C % 32);
    e.x = __shfl_down_sync(0xffffffffu, f.x, C % 32);
    e.y = __shfl_down_sync(0xffffffffu, f.y, C % 32);
  }
  if (q > 0) {
    dx = e.x + e.A * dx;
    dy = e.y + e.A * dy;
  }
}

// One block: `col` is this thread's column (row stride st) and rm its factors
// (row stride fst); `valid` false: the column does not exist (the thread takes
// part in the scans with zeros).  CYC: the cyclic systems, rm = PP, with the
// closing vector a2 (row stride fst) and denominator den.
template <class T, class R, int C, int RPT, bool CYC>
__device__ __forceinline__ void ysolve_block(int ny, bool valid, bool pin, typename CplxOf<T>::type* col, size_t st,
                                             const R* __restrict__ rm, size_t fst, const double* __restrict__ a2,
                                             const double* __restrict__ den, const double* __restrict__ am,
                                             const double* __restrict__ ap, unsigned char* smem) {
  typedef typename CplxOf<T>::type CT;
  typedef typename Vec2Of<R>::type R2;
  const int c = threadIdx.x % C, p = threadIdx.x / C, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  Aff<R>* agg = reinterpret_cast<Aff<R>*>(smem);  // [2][nwarps][C]
  const int n = CYC ? ny - 1 : ny;                // rows of the recurrences
  const int j0 = p * RPT;
  R2 v[RPT];
  R r[RPT], w[CYC ? RPT : 1];
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    const bool ok = valid && j0 + u < n;
    CT f = mk((T)0, (T)0);
    r[u] = (R)0;
    if (ok) {
      f = col[st * (j0 + u)];
      r[u] = __ldg(rm + fst * (j0 + u));
    }
    v[u].x = (R)f.x; v[u].y = (R)f.y;
    if (CYC) w[u] = ok ? (R)__ldg(a2 + fst * (j0 + u)) : (R)0;
  }
  CT last = mk((T)0, (T)0);
  if (CYC && valid) last = col[st * (ny - 1)];
  if (p == 0) {
    if (pin) { v[0].x = (R)0; v[0].y = (R)0; }
    if (CYC && valid) r[0] = (R)1 / r[0];  // row 1 divides by b_1
  }
  // forward elimination d_j = (f_j - a_j d_{j-1}) rm_j, the row's product f_j rm_j formed first
  R s[RPT];
  Aff<R> f = {(R)1, (R)0, (R)0};
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    const int jc = j0 + u < n ? j0 + u + 1 : n;
    s[u] = j0 + u == 0 ? (R)0 : (R)__ldg(am + jc) * r[u];
    v[u].x *= r[u]; v[u].y *= r[u];
    f.x = v[u].x - s[u] * f.x;
    f.y = v[u].y - s[u] * f.y;
    f.A *= -s[u];
  }
  R dx, dy;
  chunk_scan<R, C, true>(f, agg, lane, warp, nwarps, c, dx, dy);
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    dx = v[u].x - s[u] * dx;
    dy = v[u].y - s[u] * dy;
    v[u].x = dx; v[u].y = dy;
  }
  // back substitution x_j = d_j - cp_j x_{j+1}, cp_j = c_j rm_j
  f = {(R)1, (R)0, (R)0};
#pragma unroll
  for (int u = RPT - 1; u >= 0; --u) {
    const int jc = j0 + u < n ? j0 + u + 1 : n;
    s[u] = pin && j0 + u == 0 ? (R)0 : (R)__ldg(ap + jc) * r[u];
    f.x = v[u].x - s[u] * f.x;
    f.y = v[u].y - s[u] * f.y;
    f.A *= -s[u];
  }
  chunk_scan<R, C, false>(f, agg + nwarps * C, lane, warp, nwarps, c, dx, dy);
#pragma unroll
  for (int u = RPT - 1; u >= 0; --u) {
    dx = v[u].x - s[u] * dx;
    dy = v[u].y - s[u] * dy;
    v[u].x = dx; v[u].y = dy;
  }
  if constexpr (CYC) {  // closure of row n, then f_j = f_n arrmn2_j + arrmn3_j
    R2* ends = reinterpret_cast<R2*>(agg + 2 * nwarps * C);  // [2][C]: arrmn3 of rows 1 and n-1
    if (p == 0) ends[c] = v[0];
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (j0 + u == ny - 2) ends[C + c] = v[u];
    __syncthreads();
    if (!valid) return;
    const R2 e0 = ends[c], el = ends[C + c];
    const R an = am[ny], cn = ap[ny], rd = (R)1 / (R)*den;
    const R fx = ((R)last.x - cn * e0.x - an * el.x) * rd, fy = ((R)last.y - cn * e0.y - an * el.y) * rd;
    if (p == 0) col[st * (ny - 1)] = mk((T)fx, (T)fy);
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (j0 + u < n) col[st * (j0 + u)] = mk((T)(v[u].x + fx * w[u]), (T)(v[u].y + fy * w[u]));
  } else {
    if (!valid) return;
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (j0 + u < n) col[st * (j0 + u)] = mk((T)v[u].x, (T)v[u].y);
  }
}

// Columns per block: 128-byte row segments (8 FP64 or 16 FP32 columns).  A
// column tile is read once and written once with its factors in between:
// 2.25 spectrum-sized arrays of traffic, against 5.5 for one thread per column
// (forward values stored and read back, two factor arrays).
//   RPT rows per thread by ny: enough chunks for the loads of a whole column to
//   be in flight at once, few enough rows for the registers (6 per FP64 row).
//   Mixed path (T float): the blocks from nhi on solve the low modes kx < KX,
//   |kz| <= KL in FP64 with half the columns and half the rows per thread.
template <class T, int RPT, int MAXT, int MINB, bool CYC>
__global__ void __launch_bounds__(MAXT, MINB) k_yscan(Geo<T> g, const double* __restrict__ am,
                                                      const double* __restrict__ ap, const T* __restrict__ RM,
                                                      const double* __restrict__ A1, const double* __restrict__ A2,
                                                      typename CplxOf<T>::type* __restrict__ spec, int nhi,
                                                      const double* __restrict__ RM64, int KL, int KX,
                                                      const DevScalars* __restrict__ sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (sc->status) return;
  constexpr int C = 128 / (2 * (int)sizeof(T));
  const int nxh = g.nxh, ny = g.ny, nz = g.nz;
  const size_t st = (size_t)nxh;
  if (sizeof(T) == 8 || (int)blockIdx.x < nhi) {
    const long long q = (long long)blockIdx.x * C + threadIdx.x % C;
    const int kx = (int)(q % nxh), ky = (int)(q / nxh);
    bool valid = ky < nz;
    const int kz = valid ? kz_of_block(ky, nz) : 0;
    const int kzh = kz <= nz - kz ? kz : nz - kz;
    if (sizeof(T) == 4 && kx < KX && kzh <= KL) valid = false;
    const size_t o = (size_t)kzh * ny * st + kx;
    ysolve_block<T, T, C, RPT, CYC>(ny, valid, kx == 0 && kz == 0, spec + kx + st * ny * kz, st, RM + o, st,
                                    CYC ? A2 + o : nullptr, CYC ? A1 + o + st * (ny - 1) : nullptr, am, ap, smem_raw);
  } else if constexpr (sizeof(T) == 4) {
    constexpr int CL = C / 2;
    const int q = ((int)blockIdx.x - nhi) * CL + (int)threadIdx.x % CL;
    const int zi = q / KX, kx = q - zi * KX;
    const int kz = zi <= KL ? zi : nz - (zi - KL);
    const bool valid = zi <= 2 * KL && kx < nxh && (zi <= KL || kz > KL);
    const int kzh = valid ? (kz <= nz - kz ? kz : nz - kz) : 0;
    ysolve_block<T, double, CL, RPT / 2, false>(ny, valid, kx == 0 && kz == 0, spec + kx + st * ny * (valid ? kz : 0), st,
                                                RM64 + (size_t)kzh * ny * KX + kx, (size_t)KX, nullptr, nullptr, am, ap,
                                                smem_raw);
  }
}

// ---------------------------------------------------------------------------
// One thread per column, for columns too long for the chunked kernel's
// registers.  The forward sweep keeps d_j in place in the spectrum (the FP64
// low modes of the mixed path in an FP64 scratch array, layout [j][low
// column]), the backward sweep overwrites it with the solution.  Rows are
// processed in batches of YB whose loads are all issued before the dependent
// recurrence.
// ---------------------------------------------------------------------------
template <class R, class CT, int YB, class LD, class ST, class STD, class LDD>
__device__ __forceinline__ void thomas_column(int ny, bool pin, const R* __restrict__ rm, size_t fst,
                                              const double* __restrict__ am, const double* __restrict__ ap, LD load,
                                              ST store, STD store_d, LDD load_d) {
  R dx = (R)0, dy = (R)0;
  for (int j0 = 0; j0 < ny; j0 += YB) {
    R fx[YB], fy[YB], r[YB], a[YB];
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j0 + u;
      if (j < ny) {
        const CT f = load(j);
        fx[u] = (R)f.x; fy[u] = (R)f.y;
        r[u] = __ldg(rm + fst * j);
        a[u] = (R)__ldg(am + j + 1);
      }
    }
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j0 + u;
      if (j < ny) {
        if (j == 0) {
          dx = pin ? (R)0 : fx[u] * r[u];
          dy = pin ? (R)0 : fy[u] * r[u];
        } else {
          dx = (fx[u] - a[u] * dx) * r[u];
          dy = (fy[u] - a[u] * dy) * r[u];
        }
        store_d(j, dx, dy);
      }
    }
  }
  store(ny - 1, dx, dy);
  for (int j1 = ny - 2; j1 >= 0; j1 -= YB) {
    R ex[YB], ey[YB], r[YB], c[YB];
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j1 - u;
      if (j >= 0) {
        const CT v = load_d(j);
        ex[u] = (R)v.x; ey[u] = (R)v.y;
        r[u] = __ldg(rm + fst * j);  // multiplied below: the product here waits for each row's loads (32x1024x32 397 us, 228)
        c[u] = (R)__ldg(ap + j + 1);
      }
    }
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j1 - u;
      if (j >= 0) {
        const R cp = pin && j == 0 ? (R)0 : c[u] * r[u];
        dx = ex[u] - cp * dx;
        dy = ey[u] - cp * dy;
        store(j, dx, dy);
      }
    }
  }
}

// All columns in the precision of the field; in the mixed path the blocks from nhi on
// solve the low modes kx < KX, |kz| <= KL (column zi = kz for kz <= KL, KL + nz - kz
// above) in FP64 beside the FP32 columns, their forward sweep kept in the FP64 scratch
// scr, [j][low column].  With both z transforms 384 us for 32x800x32 mixed, 857 with the
// low modes in a launch before the others.
template <class T>
__global__ void __launch_bounds__(128) k_ythomas(Geo<T> g, Metrics<double> m, const T* __restrict__ RMf,
                                                 typename CplxOf<T>::type* __restrict__ spec, int nhi,
                                                 const double* __restrict__ RM64, double2* __restrict__ scr, int KL,
                                                 int KX, const DevScalars* __restrict__ sc) {
  typedef typename CplxOf<T>::type CT;
  if (sc->status) return;
  const int nxh = g.nxh, ny = g.ny, nz = g.nz;
  const size_t st = (size_t)nxh;
  if (sizeof(T) == 8 || (int)blockIdx.x < nhi) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nxh * nz) return;
    const int kx = (int)(t % nxh), kz = (int)(t / nxh);
    const int kzh = kz <= nz - kz ? kz : nz - kz;
    if (sizeof(T) == 4 && kx < KX && kzh <= KL) return;
    CT* col = spec + kx + st * ny * kz;
    auto load = [&](int j) { return col[st * j]; };
    auto store = [&](int j, T x, T y) { col[st * j] = mk(x, y); };
    thomas_column<T, CT, 16>(ny, kx == 0 && kz == 0, RMf + (size_t)kzh * ny * st + kx, st, m.am2Pr, m.ap2Pr, load,
                             store, store, load);
  } else if constexpr (sizeof(T) == 4) {
    const int q = ((int)blockIdx.x - nhi) * blockDim.x + threadIdx.x;
    if (q >= (2 * KL + 1) * KX) return;
    const int zi = q / KX, kx = q - zi * KX;
    const int kz = zi <= KL ? zi : nz - (zi - KL);
    if (kx >= nxh || (zi > KL && kz <= KL)) return;
    const int kzh = kz <= nz - kz ? kz : nz - kz;
    CT* col = spec + kx + st * ny * kz;
    const size_t nlow = (size_t)(2 * KL + 1) * KX;
    double2* w = scr + (size_t)zi * KX + kx;  // [j][low column]
    auto load = [&](int j) { const CT v = col[st * j]; return make_double2(v.x, v.y); };
    auto store = [&](int j, double x, double y) { col[st * j] = mk((T)x, (T)y); };
    auto store_d = [&](int j, double x, double y) { w[nlow * j] = make_double2(x, y); };
    auto load_d = [&](int j) { return w[nlow * j]; };
    thomas_column<double, double2, 16>(ny, kx == 0 && kz == 0, RM64 + (size_t)kzh * ny * KX + kx, (size_t)KX, m.am2Pr,
                                       m.ap2Pr, load, store, store_d, load_d);
  }
}

// One thread per (kx, kz) column of the (kx, j, kz) spectrum (kx fastest, so
// a warp reads 32 consecutive kx of one row), FP64, in place: forward
// elimination, the backward pass of the right-hand side (arrmn3), the closure
// of row n, and the back substitution f_j = f_n arrmn2_j + arrmn3_j.  Each
// pass loads YB rows (and their factors) before its dependent recurrence, so
// YB loads of every column are in flight at once.
template <class T, int YB>
__global__ void __launch_bounds__(128) k_ycyclic(Geo<T> g, Metrics<double> m, const double* __restrict__ PP,
                                                 const double* __restrict__ A1, const double* __restrict__ A2,
                                                 typename CplxOf<T>::type* __restrict__ spec,
                                                 const DevScalars* __restrict__ sc) {
  typedef typename CplxOf<T>::type CT;
  if (sc->status) return;
  const int nxh = g.nxh, ny = g.ny, nz = g.nz;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nxh * nz) return;
  const int kx = (int)(t % nxh), kz = (int)(t / nxh);
  const int kzh = kz <= nz - kz ? kz : nz - kz;
  const size_t st = (size_t)nxh;
  CT* col = spec + kx + st * ny * kz;
  const size_t o = (size_t)kzh * ny * st + kx;
  const bool pin = (kx == 0 && kz == 0);
  // forward elimination, rows 1..n-1 (0-based 0..ny-2); row 1 divides by b_1
  double dx = 0.0, dy = 0.0;
  for (int j0 = 0; j0 <= ny - 2; j0 += YB) {
    double fx[YB], fy[YB], pp[YB], am[YB];
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j0 + u;
      if (j <= ny - 2) {
        const CT f = col[st * j];
        fx[u] = (double)f.x; fy[u] = (double)f.y;
        pp[u] = PP[o + st * j];
        am[u] = m.am2Pr[j + 1];
      }
    }
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j0 + u;
      if (j <= ny - 2) {
        if (j == 0) {
          dx = pin ? 0.0 : fx[u] / pp[u];
          dy = pin ? 0.0 : fy[u] / pp[u];
        } else {
          dx = (fx[u] - am[u] * dx) * pp[u];
          dy = (fy[u] - am[u] * dy) * pp[u];
        }
        col[st * j] = mk((T)dx, (T)dy);
      }
    }
  }
  // backward pass: arrmn3_n = 0, arrmn3_j = f_j + arrmn1_j arrmn3_{j+1}
  double ex = 0.0, ey = 0.0, lx = 0.0, ly = 0.0;
  for (int j1 = ny - 2; j1 >= 0; j1 -= YB) {
    double vx[YB], vy[YB], a1[YB];
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j1 - u;
      if (j >= 0) {
        const CT f = col[st * j];
        vx[u] = (double)f.x; vy[u] = (double)f.y;
        a1[u] = A1[o + st * j];
      }
    }
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j1 - u;
      if (j >= 0) {
        ex = vx[u] + a1[u] * ex;
        ey = vy[u] + a1[u] * ey;
        col[st * j] = mk((T)ex, (T)ey);
        if (j == ny - 2) { lx = ex; ly = ey; }
      }
    }
  }
  // closure of row n, then f_j = f_n arrmn2_j + arrmn3_j
  const double an = m.am2Pr[ny], cn = m.ap2Pr[ny], den = A1[o + st * (ny - 1)];
  const CT fl = col[st * (ny - 1)];
  const double fnx = ((double)fl.x - cn * ex - an * lx) / den, fny = ((double)fl.y - cn * ey - an * ly) / den;
  col[st * (ny - 1)] = mk((T)fnx, (T)fny);
  for (int j0 = 0; j0 <= ny - 2; j0 += YB) {
    double vx[YB], vy[YB], a2[YB];
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j0 + u;
      if (j <= ny - 2) {
        const CT f = col[st * j];
        vx[u] = (double)f.x; vy[u] = (double)f.y;
        a2[u] = A2[o + st * j];
      }
    }
#pragma unroll
    for (int u = 0; u < YB; ++u) {
      const int j = j0 + u;
      if (j <= ny - 2) col[st * j] = mk((T)(fnx * a2[u] + vx[u]), (T)(fny * a2[u] + vy[u]));
    }
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// Rows the chunked kernel takes: 32 chunks of 24 rows.
constexpr int kScanMaxRows = 768;
bool ysolve_chunked(int ny) { return ny <= kScanMaxRows; }

template <class T, int RPT, int MINB, bool CYC> static cudaError_t yscan_launch(ch3d_ctx* c) {
  typedef typename CplxOf<T>::type CT;
  constexpr int C = 128 / (2 * (int)sizeof(T)), CW = 32 / C;
  const int P = ((c->ny + RPT - 1) / RPT + CW - 1) / CW * CW;  // chunks, whole warps
  const int threads = C * P, nwarps = threads / 32;
  const long long ncol = (long long)c->nxh * c->nz;
  const int nhi = (int)((ncol + C - 1) / C);
  const int nlo = sizeof(T) == 4 ? ((2 * c->KL + 1) * c->TSy + C / 2 - 1) / (C / 2) : 0;
  // the scans' warp aggregates (FP64 for the low modes, half the columns) and the cyclic closure's two rows
  const size_t smem = (size_t)2 * nwarps * 8 * sizeof(Aff<double>) + 2 * 8 * sizeof(double2);
  k_yscan<T, RPT, 32 * C, MINB, CYC><<<nhi + nlo, threads, smem, c->stream>>>(
      make_geo<T>(c), c->m64full.am2Pr, c->m64full.ap2Pr, (const T*)c->yRM, (const double*)c->yCP, c->yA2,
      (CT*)c->spec, nhi, c->yRM64, c->KL, c->TSy, c->sc);
  return cudaGetLastError();
}
// 32 chunks of 4, 8, 12 or 24 rows, registers for 4, 3, 2 and 1 blocks of 256 (FP64) or 2, 2, 2, 1 of 512 threads
template <class T, bool CYC> static cudaError_t yscan_t(ch3d_ctx* c) {
  constexpr bool D = sizeof(T) == 8;
  if (c->ny <= 128) return yscan_launch<T, 4, D ? 4 : 2, CYC>(c);
  if (c->ny <= 256) return yscan_launch<T, 8, D ? 3 : 2, CYC>(c);
  if (c->ny <= 384) return yscan_launch<T, 12, 2, CYC>(c);
  return yscan_launch<T, 24, 1, CYC>(c);
}

cudaError_t launch_ysolve(ch3d_ctx* c) {
  if (ysolve_chunked(c->ny)) {
    if (y_periodic(c)) return yscan_t<double, true>(c);  // periodic y: FP64 only
    return c->fp32 ? yscan_t<float, false>(c) : yscan_t<double, false>(c);
  }
  const unsigned gy = (unsigned)(((long long)c->nxh * c->nz + 127) / 128);
  if (y_periodic(c)) {
    k_ycyclic<double, 16><<<gy, 128, 0, c->stream>>>(make_geo<double>(c), c->m64full, (const double*)c->yRM,
                                                     (const double*)c->yCP, c->yA2, (double2*)c->spec, c->sc);
  } else if (!c->fp32) {
    k_ythomas<double><<<gy, 128, 0, c->stream>>>(make_geo<double>(c), c->m64full, (const double*)c->yRM,
                                                 (double2*)c->spec, (int)gy, nullptr, nullptr, 0, 0, c->sc);
  } else {
    const int nlow = (2 * c->KL + 1) * c->TSy;
    k_ythomas<float><<<gy + (nlow + 127) / 128, 128, 0, c->stream>>>(
        make_geo<float>(c), c->m64full, (const float*)c->yRM, (float2*)c->spec, (int)gy, c->yRM64, (double2*)c->ylow,
        c->KL, c->TSy, c->sc);
  }
  return cudaGetLastError();
}

cudaError_t launch_ysolve_factors(ch3d_ctx* c) {
  const dim3 g((c->nxh + 127) / 128, c->nz / 2 + 1);
  if (y_periodic(c)) {
    k_ycyclic_factors<<<g, 128, 0, c->stream>>>(c->m64full, c->wave, c->nx, c->ny, c->nxh, (double*)c->yRM,
                                                (double*)c->yCP, c->yA2);
  } else if (!c->fp32) {
    k_ythomas_factors<double><<<g, 128, 0, c->stream>>>(c->m64full, c->wave, c->nx, c->ny, (double*)c->yRM, c->nxh,
                                                        c->nxh);
  } else {
    k_ythomas_factors<float><<<g, 128, 0, c->stream>>>(c->m64full, c->wave, c->nx, c->ny, (float*)c->yRM, c->nxh,
                                                       c->nxh);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_ythomas_factors<double><<<dim3(1, c->KL + 1), 128, 0, c->stream>>>(c->m64full, c->wave, c->nx, c->ny, c->yRM64,
                                                                        c->TSy, c->nxh < c->TSy ? c->nxh : c->TSy);
  }
  return cudaGetLastError();
}

}  // namespace ch3d
