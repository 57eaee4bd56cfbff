// ch3d_march.cuh -- shared by the right-hand-side kernels (ch3d_march.cu,
// ch3d_rhs.cu) and the line solves (ch3d_sweep.cu): the coefficient tables of
// the substeps (filled by ch3d_substep.cu) and the 2nd-order right-hand sides
// at one cell.
#pragma once
#include "ch3d_dev.cuh"

namespace ch3d {

// Row table (precision T, MT_W values per row j = 0..ny-1): the y metrics at
// jc = j + 1 and the Thomas factors a, 1/m, c/m of the two Helmholtz sets (set
// 0: ux and uz, set 1: uy; m_TSchemePIMP_inc.f90:392-430, 542-589, 702-740).
// cp of the last row is stored as 0 (it has no upper neighbour).
enum {
  MT_IY1, MT_IY3, MT_RDYP, MT_RDYC, MT_AP2C, MT_AC2C, MT_AM2C, MT_AP2P, MT_AC2P, MT_AM2P,
  MT_A0, MT_RM0, MT_CP0, MT_A1, MT_RM1, MT_CP1, MT_W
};

// Second table for the twisted march (lower half eliminated upwards, upper half
// downwards): the downward factors c, 1/m', a/m' of both sets, with
// m'_{ny-1} = b, m'_j = b_j - c_j aq_{j+1}; rows of MD_W values.
enum { MD_C0, MD_RQ0, MD_AQ0, MD_C1, MD_RQ1, MD_AQ1, MD_W = 8 };

// Layout of the table buffer (values of precision T at the start of a buffer
// sized for FP64): the row tables of the RK substeps ns = 1..3 (ny * MT_W values
// each), their downward tables (ny * MD_W each), then per substep the pmBeta its
// factors were computed for (FP64 bit patterns; all ones = not yet computed).
constexpr int kMarchTables = 3;
inline unsigned long long* march_beta_slots(void* mtab, int ny) {
  return (unsigned long long*)((char*)mtab + (size_t)kMarchTables * ny * (MT_W + MD_W) * sizeof(double));
}
template <class T> inline T* march_down_tables(void* mtab, int ny) { return (T*)mtab + (size_t)kMarchTables * ny * MT_W; }

// Factor block of one periodic direction (Fortran index 1..n): ppj | vecn1 |
// vecn2 (n+1 each), then a, b, c, denominator (InversePTriFixedCoe,
// src/CFD_2nd/m_Tools.f90:167-219); the x, z and y blocks of a substep follow
// each other, kMarchTables substeps.
__host__ __device__ inline int ptri_stride(int n) { return 3 * (n + 1) + 4; }
__host__ __device__ inline size_t ptri_doubles(int nx, int ny, int nz) {
  return (size_t)ptri_stride(nx) + ptri_stride(nz) + ptri_stride(ny);
}
// block of direction d (0 x, 1 z, 2 y) of the first substep
inline const double* ptri_block(const ch3d_ctx* c, int d) {
  return c->pfac + (d > 0 ? ptri_stride(c->nx) : 0) + (d > 1 ? ptri_stride(c->nz) : 0);
}

// Stencil values of one cell: c centre, ip/im i+1/i-1, jp/jm j+1/j-1, kp/km k+1/k-1.
template <class T> struct Sten2 {
  T ux_c, ux_ip, ux_im, ux_jp, ux_jm, ux_kp, ux_km, ux_ip_jm, ux_ip_km;
  T uy_c, uy_ip, uy_im, uy_jp, uy_jm, uy_kp, uy_km, uy_im_jp, uy_jp_km;
  T uz_c, uz_ip, uz_im, uz_jp, uz_jm, uz_kp, uz_km, uz_im_kp, uz_jm_kp;
  T p_c, p_im, p_jm, p_km;
};

// Viscous treatment of the right-hand sides: Crank-Nicolson in y (PIMP), in all
// directions (FIMP), none (FEXP), or the LES form with a constant viscosity.
enum { RHS_PIMP, RHS_FIMP, RHS_FEXP, RHS_LESC };

template <class T> struct RhsCoef { T gamma, theta, alpha, beta; };

// clcRhsX/Y/Z of one cell without the mean pressure gradient: right-hand sides
// r and new Hist values h; tr: the row's table entries, ho: the old Hist.
// PIMP: m_TSchemePIMP_inc.f90:7-75, 161-209, 277-325; FIMP: m_TSchemeFIMP_inc.f90:
// 6-177; FEXP: m_TSchemeFEXP_inc.f90:6-324.
template <int SCH, class T>
__device__ __forceinline__ void rhs2_cell(const Geo<T>& g, const T* tr, const Sten2<T>& s, const T (&ho)[3],
                                          const RhsCoef<T>& pm, T (&r)[3], T (&h)[3]) {
  const T two = (T)2, half = (T)0.5, quarter = (T)0.25, one = (T)1;
  const T rdx = g.rdx, rdz = g.rdz, rdx2 = g.rdx2, rdz2 = g.rdz2, xnu = g.xnu;
  const T IY1 = tr[MT_IY1], IY2 = one - IY1;
  const T IY3 = tr[MT_IY3], IY4 = one - IY3;
  // conv + the terms each scheme takes explicitly; dc: x and z viscous terms, d2: the y one
  auto close = [&](int c, T conv, T dc, T d2, T gradp) {
    if (SCH == RHS_FIMP) {
      h[c] = conv;
      r[c] = pm.gamma * h[c] + pm.theta * ho[c] - pm.alpha * gradp + two * pm.beta * (dc + d2);
    } else if (SCH == RHS_FEXP) {
      h[c] = conv + xnu * (dc + d2);
      r[c] = pm.gamma * h[c] + pm.theta * ho[c] - pm.alpha * gradp;
    } else {
      h[c] = conv + xnu * dc;
      r[c] = pm.gamma * h[c] + pm.theta * ho[c] - pm.alpha * gradp + two * pm.beta * d2;
    }
  };
  {  // RhsX
    const T qdx1 = quarter * rdx, qdx3 = quarter * rdz;
    const T sucaj = half * tr[MT_RDYP];
    T h11 = ((s.ux_ip + s.ux_c) * (s.ux_ip + s.ux_c) - (s.ux_c + s.ux_im) * (s.ux_c + s.ux_im)) * qdx1;
    T h12 = ((s.uy_jp + s.uy_im_jp) * (IY3 * s.ux_c + IY4 * s.ux_jp) - (s.uy_c + s.uy_im) * (IY1 * s.ux_jm + IY2 * s.ux_c)) * sucaj;
    T h13 = ((s.uz_kp + s.uz_im_kp) * (s.ux_kp + s.ux_c) - (s.uz_c + s.uz_im) * (s.ux_c + s.ux_km)) * qdx3;
    T d11q1 = (s.ux_ip - two * s.ux_c + s.ux_im) * rdx2;
    T d22q1 = tr[MT_AP2C] * s.ux_jp + tr[MT_AC2C] * s.ux_c + tr[MT_AM2C] * s.ux_jm;
    T d33q1 = g.ap3c * s.ux_kp + g.ac3c * s.ux_c + g.am3c * s.ux_km;
    close(0, -h11 - h12 - h13 + g.g1, d11q1 + d33q1, d22q1, (s.p_c - s.p_im) * rdx);
  }
  {  // RhsY
    const T hdx1 = half * rdx, hdx3 = half * rdz;
    const T sucac = tr[MT_RDYC], qsucac = quarter * sucac;
    T h21 = ((IY1 * s.ux_ip_jm + IY2 * s.ux_ip) * (s.uy_ip + s.uy_c) - (IY1 * s.ux_jm + IY2 * s.ux_c) * (s.uy_c + s.uy_im)) * hdx1;
    T h22 = ((s.uy_jp + s.uy_c) * (s.uy_jp + s.uy_c) - (s.uy_c + s.uy_jm) * (s.uy_c + s.uy_jm)) * qsucac;
    T h23 = ((IY1 * s.uz_jm_kp + IY2 * s.uz_kp) * (s.uy_kp + s.uy_c) - (IY1 * s.uz_jm + IY2 * s.uz_c) * (s.uy_c + s.uy_km)) * hdx3;
    T d11q2 = g.ap1c * s.uy_ip + g.ac1c * s.uy_c + g.am1c * s.uy_im;
    T d22q2 = tr[MT_AP2P] * s.uy_jp + tr[MT_AC2P] * s.uy_c + tr[MT_AM2P] * s.uy_jm;
    T d33q2 = g.ap3c * s.uy_kp + g.ac3c * s.uy_c + g.am3c * s.uy_km;
    close(1, -h21 - h22 - h23 + g.g2, d11q2 + d33q2, d22q2, (s.p_c - s.p_jm) * sucac);
  }
  {  // RhsZ
    const T qdx1 = quarter * rdx, qdx3 = quarter * rdz;
    const T sucaj = half * tr[MT_RDYP];
    T h31 = ((s.ux_ip + s.ux_ip_km) * (s.uz_ip + s.uz_c) - (s.ux_c + s.ux_km) * (s.uz_c + s.uz_im)) * qdx1;
    T h32 = ((s.uy_jp + s.uy_jp_km) * (IY3 * s.uz_c + IY4 * s.uz_jp) - (s.uy_c + s.uy_km) * (IY1 * s.uz_jm + IY2 * s.uz_c)) * sucaj;
    T h33 = ((s.uz_kp + s.uz_c) * (s.uz_kp + s.uz_c) - (s.uz_c + s.uz_km) * (s.uz_c + s.uz_km)) * qdx3;
    T d11q3 = g.ap1c * s.uz_ip + g.ac1c * s.uz_c + g.am1c * s.uz_im;
    T d22q3 = tr[MT_AP2C] * s.uz_jp + tr[MT_AC2C] * s.uz_c + tr[MT_AM2C] * s.uz_jm;
    T d33q3 = (s.uz_kp - two * s.uz_c + s.uz_km) * rdz2;
    close(2, -h31 - h32 - h33 + g.g3, d11q3 + d33q3, d22q3, (s.p_c - s.p_km) * rdz);
  }
}

// clcRhsX/Y/Z_PIMP_LES (m_TSchemePIMP_inc.f90:80-156, 214-272, 330-387) with the
// total viscosity xnu everywhere and the explicit force f (the learned closure):
// the averages over y without weights, the full stress divergence explicitly.
template <class T>
__device__ __forceinline__ void rhs2_les_const(const Geo<T>& g, const T* tr, const Sten2<T>& s, const T (&ho)[3],
                                               const T (&f)[3], const RhsCoef<T>& pm, T (&r)[3], T (&h)[3]) {
  const T rdx = g.rdx, rdz = g.rdz, rdx2 = g.rdx2, rdz2 = g.rdz2, nu = g.xnu;
  const T qdx1 = (T)0.25 * rdx, qdx3 = (T)0.25 * rdz, rdyp = tr[MT_RDYP], sucaj = (T)0.25 * rdyp;
  {
    const T h11 = ((s.ux_ip + s.ux_c) * (s.ux_ip + s.ux_c) - (s.ux_c + s.ux_im) * (s.ux_c + s.ux_im)) * qdx1;
    const T h12 = ((s.uy_jp + s.uy_im_jp) * (s.ux_jp + s.ux_c) - (s.uy_c + s.uy_im) * (s.ux_c + s.ux_jm)) * sucaj;
    const T h13 = ((s.uz_kp + s.uz_im_kp) * (s.ux_kp + s.ux_c) - (s.uz_c + s.uz_im) * (s.ux_c + s.ux_km)) * qdx3;
    const T sgs1 = rdx2 * nu * ((s.ux_ip - s.ux_c) - (s.ux_c - s.ux_im));
    const T sgs2 = rdx * rdyp * nu * ((s.uy_jp - s.uy_im_jp) - (s.uy_c - s.uy_im));
    const T sgs3 = rdx * rdz * nu * ((s.uz_kp - s.uz_im_kp) - (s.uz_c - s.uz_im));
    const T d22 = nu * (tr[MT_AP2C] * (s.ux_jp - s.ux_c) - tr[MT_AM2C] * (s.ux_c - s.ux_jm));
    const T d33 = nu * (g.ap3c * (s.ux_kp - s.ux_c) - g.am3c * (s.ux_c - s.ux_km));
    h[0] = -h11 - h12 - h13 + sgs1 + sgs2 + sgs3 + (sgs1 + d33) + g.g1 + f[0];
    r[0] = pm.gamma * h[0] + pm.theta * ho[0] - pm.alpha * ((s.p_c - s.p_im) * rdx) + (T)2 * pm.beta * d22;
  }
  {
    const T sucac = tr[MT_RDYC], qsucac = (T)0.25 * sucac;
    const T h21 = ((s.ux_ip + s.ux_ip_jm) * (s.uy_ip + s.uy_c) - (s.ux_c + s.ux_jm) * (s.uy_c + s.uy_im)) * qdx1;
    const T h22 = ((s.uy_jp + s.uy_c) * (s.uy_jp + s.uy_c) - (s.uy_c + s.uy_jm) * (s.uy_c + s.uy_jm)) * qsucac;
    const T h23 = ((s.uz_kp + s.uz_jm_kp) * (s.uy_kp + s.uy_c) - (s.uz_c + s.uz_jm) * (s.uy_c + s.uy_km)) * qdx3;
    const T sgs1 = rdx * sucac * nu * ((s.ux_ip - s.ux_ip_jm) - (s.ux_c - s.ux_jm));
    const T sgs2 = nu * (tr[MT_AP2P] * (s.uy_jp - s.uy_c) - tr[MT_AM2P] * (s.uy_c - s.uy_jm));
    const T sgs3 = rdz * sucac * nu * ((s.uz_kp - s.uz_jm_kp) - (s.uz_c - s.uz_jm));
    const T d11 = nu * (g.ap1c * (s.uy_ip - s.uy_c) - g.am1c * (s.uy_c - s.uy_im));
    const T d33 = nu * (g.ap3c * (s.uy_kp - s.uy_c) - g.am3c * (s.uy_c - s.uy_km));
    h[1] = -h21 - h22 - h23 + sgs1 + sgs2 + sgs3 + (d11 + d33) + g.g2 + f[1];
    r[1] = pm.gamma * h[1] + pm.theta * ho[1] - pm.alpha * ((s.p_c - s.p_jm) * sucac) + (T)2 * pm.beta * sgs2;
  }
  {
    const T h31 = ((s.ux_ip + s.ux_ip_km) * (s.uz_ip + s.uz_c) - (s.ux_c + s.ux_km) * (s.uz_c + s.uz_im)) * qdx1;
    const T h32 = ((s.uy_jp + s.uy_jp_km) * (s.uz_jp + s.uz_c) - (s.uy_c + s.uy_km) * (s.uz_c + s.uz_jm)) * sucaj;
    const T h33 = ((s.uz_kp + s.uz_c) * (s.uz_kp + s.uz_c) - (s.uz_c + s.uz_km) * (s.uz_c + s.uz_km)) * qdx3;
    const T sgs1 = rdx * rdz * nu * ((s.ux_ip - s.ux_ip_km) - (s.ux_c - s.ux_km));
    const T sgs2 = rdz * rdyp * nu * ((s.uy_jp - s.uy_jp_km) - (s.uy_c - s.uy_km));
    const T sgs3 = rdz2 * nu * ((s.uz_kp - s.uz_c) - (s.uz_c - s.uz_km));
    const T d11 = nu * (g.ap1c * (s.uz_ip - s.uz_c) - g.am1c * (s.uz_c - s.uz_im));
    const T d22 = nu * (tr[MT_AP2C] * (s.uz_jp - s.uz_c) - tr[MT_AM2C] * (s.uz_c - s.uz_jm));
    h[2] = -h31 - h32 - h33 + sgs1 + sgs2 + sgs3 + (d11 + sgs3) + g.g3 + f[2];
    r[2] = pm.gamma * h[2] + pm.theta * ho[2] - pm.alpha * ((s.p_c - s.p_km) * rdz) + (T)2 * pm.beta * d22;
  }
}

}  // namespace ch3d
