// ch3d_rhs.cu -- the 2nd-order right-hand sides as a march over chunks of rows:
// clcRhsX/Y/Z_PIMP, _FIMP and _FEXP (src/CFD_2nd/m_TSchemePIMP_inc.f90:7-325,
// m_TSchemeFIMP_inc.f90:6-177, m_TSchemeFEXP_inc.f90:6-324) and the constant-
// viscosity LES form of the learned closure.  The line solves (ch3d_sweep.cu)
// follow; large PIMP grids run ch3d_march.cu instead, which eliminates as it
// marches.
//
// A block of 32 x 4 columns marches up its chunk of rows through a ring of
// rows staged in shared memory (ux, uy, uz, p with a one-cell x/z halo and the
// row's table entries), copied two (FP64) or four (FP32) rows ahead; each thread
// forms the three right-hand sides of its cell from rows j-1, j, j+1 of the ring.
// One thread per cell and component, with the stencil read from global memory,
// was bound by its loads: 157 us at 128^3 (87 with a warm L2).  Now 50 us there for
// 0.22 GB (ADI; 44% of the DRAM bandwidth) and 9 us at 64^3, bound by the latency of a
// row with 16 warps per SM: the registers allow four blocks of 128 threads.
#include "ch3d_march.cuh"

namespace ch3d {

constexpr int kRhsBZ = 4, kRhsSX = 34, kRhsPL = kRhsSX * (kRhsBZ + 2);  // staged points per row and field
template <class T> struct RhsRing {
  static constexpr int D = sizeof(T) == 8 ? 2 : 4, RS = D + 4;  // rows in flight, row slots
};

// FUSE (FEXP only): writes u* = u + r in place of the right-hand sides; between
// walls the uy row on the lower wall takes uy_ym (see k_uhat_fexp).
// T: the fields; R: the arithmetic and the row table.
template <class T, class R, int SCH, bool PER, bool FUSE>
__global__ void __launch_bounds__(32 * kRhsBZ, sizeof(R) == 8 ? 4 : 5)
    k_rhs_rows(Geo<R> g, const R* __restrict__ tab, const T* __restrict__ ux, const T* __restrict__ uy,
               const T* __restrict__ uz, const T* __restrict__ pr, T* __restrict__ hx, T* __restrict__ hy,
               T* __restrict__ hz, T* __restrict__ rx, T* __restrict__ ry, T* __restrict__ rz,
               const double* __restrict__ force, int rows, const DevScalars* __restrict__ sc) {
  constexpr int BZ = kRhsBZ, SX = kRhsSX, PL = kRhsPL, D = RhsRing<T>::D, RS = RhsRing<T>::RS;
  constexpr int NT = 32 * BZ, NS = (PL + NT - 1) / NT;
  __shared__ __align__(16) T ring[4][RS][PL];
  __shared__ __align__(16) R trs[RS][MT_W];
  if (sc->status) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long plane = (long long)nx * ny;
  tab += (size_t)(sc->ns - 1) * ny * MT_W;  // this substep's table
  const int tid = threadIdx.x, tx = tid & 31, tz = tid >> 5;
  const int ntx = (nx + 31) / 32;
  const int i0 = (blockIdx.x % ntx) * 32, k0 = (blockIdx.x / ntx) * BZ;
  const int j0 = blockIdx.y * rows, j1 = min(j0 + rows, ny);
  const int i = i0 + tx, k = k0 + tz;
  const bool act = i < nx && k < nz;
  long long so[NS];  // staging slot offsets: s = tid + q NT -> halo-tile position (s % SX, s / SX), periodic in x and z
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const int s = tid + q * NT;
    int ig = (i0 - 1 + s % SX) % nx, kg = (k0 - 1 + s / SX) % nz;
    if (ig < 0) ig += nx;
    if (kg < 0) kg += nz;
    so[q] = s < PL ? ig + plane * kg : 0;
  }
  auto slot = [&](int r) { return (r - j0 + 1) % RS; };  // r >= j0 - 1
  // row r of the march; periodic in y it wraps, between walls rows -1 and ny are ghosts
  auto issue_row = [&](int r) {
    const int rr = r < 0 ? ny - 1 : (r == ny ? 0 : r);
    if (!PER && rr != r) return;
    const long long ro = (long long)rr * nx;
    const int sl = slot(r);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const int s = tid + q * NT;
      if (s < PL) {
        cp_async_el(&ring[0][sl][s], ux + so[q] + ro);
        cp_async_el(&ring[1][sl][s], uy + so[q] + ro);
        cp_async_el(&ring[2][sl][s], uz + so[q] + ro);
        cp_async_el(&ring[3][sl][s], pr + so[q] + ro);
      }
    }
    constexpr int TV = MT_W * (int)sizeof(R) / 16;
    if (tid < TV)
      cp_async_el(reinterpret_cast<float4*>(&trs[sl][0]) + tid, reinterpret_cast<const float4*>(tab + (size_t)rr * MT_W) + tid);
  };
  // wall ghost rows from the thread's own staged slots (SetBC_and_UpdateHalo, m_BC_and_Halo.f90:241-282)
  auto ghost_row = [&](int r) {
    const int sl = slot(r);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const int s = tid + q * NT;
      if (s >= PL) continue;
      if (r < 0) {
        const T u = ring[0][slot(0)][s], w = ring[2][slot(0)][s], v1 = ring[1][slot(1)][s];
        ring[0][sl][s] = g.bc.lo == -1 ? (T)(g.bc.ux_lo * 2.0) - u : u - (T)(g.bc.ux_lo * g.bc.dyp1);
        ring[1][sl][s] = (T)(g.bc.uy_lo * 2.0) - v1;
        ring[2][sl][s] = g.bc.lo == -1 ? (T)(g.bc.uz_lo * 2.0) - w : w - (T)(g.bc.uz_lo * g.bc.dyp1);
        ring[3][sl][s] = ring[3][slot(0)][s];
      } else {
        const int sn = slot(ny - 1);
        const T u = ring[0][sn][s], w = ring[2][sn][s];
        ring[0][sl][s] = g.bc.hi == -1 ? (T)(g.bc.ux_hi * 2.0) - u : (T)(g.bc.ux_hi * g.bc.dypN) + u;
        ring[1][sl][s] = (T)g.bc.uy_hi;
        ring[2][sl][s] = g.bc.hi == -1 ? (T)(g.bc.uz_hi * 2.0) - w : (T)(g.bc.uz_hi * g.bc.dypN) + w;
        ring[3][sl][s] = ring[3][sn][s];
      }
    }
  };
  // prologue: rows j0-1 and j0 as one copy group, then a row per group
  issue_row(j0 - 1);
#pragma unroll
  for (int r = 0; r <= D + 1; ++r) {
    if (j0 + r <= j1) issue_row(j0 + r);
    cp_async_commit();
  }
  const RhsCoef<R> pm = {(R)sc->pmGamma, (R)sc->pmTheta, (R)sc->pmAlpha,
                         SCH == RHS_LESC ? (R)sc->pmBetaT : (R)sc->pmBeta};
  // the partially implicit RhsX gets the mean pressure gradient in the y solve (clcRhsX_PIMP :61-74)
  const R dpm = SCH == RHS_PIMP ? (R)0 : (R)sc->dpmdxns;
  const bool hread = act && pm.theta != (R)0;  // pmTheta = 0 (first RK3 substep): the old Hist does not enter
  const int c0 = (tz + 1) * SX + tx + 1;
  long long idx = act ? i + plane * k + (long long)j0 * nx : 0;
  T hc[3] = {(T)0, (T)0, (T)0}, h1[3] = {(T)0, (T)0, (T)0};  // Hist of rows j and j+1
  if (hread) {
    hc[0] = hx[idx]; hc[1] = hy[idx]; hc[2] = hz[idx];
    if (j0 + 1 < j1) { h1[0] = hx[idx + nx]; h1[1] = hy[idx + nx]; h1[2] = hz[idx + nx]; }
  }
  for (int j = j0; j < j1; ++j, idx += nx) {
    cp_async_wait<D>();  // this thread's copies of rows <= j+1 are done
    if (!PER && j + 1 == ny) ghost_row(ny);
    if (!PER && j == 0) ghost_row(-1);
    __syncthreads();
    // written after the barrier: slot (j+D+2) differs from those of rows j-1, j, j+1 that others still read
    if (j + D + 2 <= j1) issue_row(j + D + 2);
    cp_async_commit();
    T hn[3] = {(T)0, (T)0, (T)0};
    if (hread && j + 2 < j1) { hn[0] = hx[idx + 2 * nx]; hn[1] = hy[idx + 2 * nx]; hn[2] = hz[idx + 2 * nx]; }
    if (act) {
      const int s0 = slot(j - 1), s1 = slot(j), s2 = slot(j + 1);
      const T *X0 = &ring[0][s0][c0], *X1 = &ring[0][s1][c0], *X2 = &ring[0][s2][c0];
      const T *Y0 = &ring[1][s0][c0], *Y1 = &ring[1][s1][c0], *Y2 = &ring[1][s2][c0];
      const T *Z0 = &ring[2][s0][c0], *Z1 = &ring[2][s1][c0], *Z2 = &ring[2][s2][c0];
      const T *P0 = &ring[3][s0][c0], *P1 = &ring[3][s1][c0];
      const Sten2<R> s = {(R)X1[0], (R)X1[1], (R)X1[-1], (R)X2[0], (R)X0[0], (R)X1[SX], (R)X1[-SX], (R)X0[1], (R)X1[1 - SX],
                          (R)Y1[0], (R)Y1[1], (R)Y1[-1], (R)Y2[0], (R)Y0[0], (R)Y1[SX], (R)Y1[-SX], (R)Y2[-1], (R)Y2[-SX],
                          (R)Z1[0], (R)Z1[1], (R)Z1[-1], (R)Z2[0], (R)Z0[0], (R)Z1[SX], (R)Z1[-SX], (R)Z1[SX - 1], (R)Z0[SX],
                          (R)P1[0], (R)P1[-1], (R)P0[0], (R)P1[-SX]};
      const R ho[3] = {(R)hc[0], (R)hc[1], (R)hc[2]};
      R r[3], h[3];
      if constexpr (SCH == RHS_LESC) {
        const R f[3] = {force[idx], force[g.N + idx], force[2 * g.N + idx]};
        rhs2_les_const(g, trs[s1], s, ho, f, pm, r, h);
      } else {
        rhs2_cell<SCH>(g, trs[s1], s, ho, pm, r, h);
      }
      r[0] += dpm;
      hx[idx] = (T)h[0]; hy[idx] = (T)h[1]; hz[idx] = (T)h[2];
      if (FUSE) {
        rx[idx] = (T)(s.ux_c + r[0]);
        ry[idx] = !PER && j == 0 ? (T)g.bc.uy_lo : (T)(s.uy_c + r[1]);
        rz[idx] = (T)(s.uz_c + r[2]);
      } else {
        rx[idx] = (T)r[0]; ry[idx] = (T)r[1]; rz[idx] = (T)r[2];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) { hc[c] = h1[c]; h1[c] = hn[c]; }
  }
}

// Rows per block: 32 where that gives four blocks per SM, else 16 or 8 (each
// chunk reads two rows of its neighbours again).
static int rhs_rows(const ch3d_ctx* c) {
  const long long tiles = (long long)((c->nx + 31) / 32) * ((c->nz + kRhsBZ - 1) / kRhsBZ);
  int rows = 32;
  while (rows > 8 && tiles * ((c->ny + rows - 1) / rows) < 4LL * sm_count(c->device)) rows >>= 1;
  return rows;
}

template <class T, class R, int SCH, bool PER, bool FUSE> static cudaError_t rhs_launch(ch3d_ctx* c, const double* force) {
  T** f = (T**)c->f;
  const int rows = rhs_rows(c), o = FUSE ? 12 : 7;
  const dim3 grid((unsigned)(((c->nx + 31) / 32) * ((c->nz + kRhsBZ - 1) / kRhsBZ)), (c->ny + rows - 1) / rows);
  k_rhs_rows<T, R, SCH, PER, FUSE><<<grid, 32 * kRhsBZ, 0, c->stream>>>(make_geo<R>(c), (const R*)c->mtab, f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[o], f[o + 1], f[o + 2], force, rows, c->sc);
  return cudaGetLastError();
}

// clcRhsX/Y/Z of the context's scheme -> RhsX/Y/Z
template <class T> static cudaError_t rhs_t(ch3d_ctx* c) {
  const bool per = y_periodic(c);
  switch (c->cfg.IsImplicit) {
    case 0: return per ? rhs_launch<T, T, RHS_FEXP, true, false>(c, nullptr) : rhs_launch<T, T, RHS_FEXP, false, false>(c, nullptr);
    case 1: return per ? rhs_launch<T, T, RHS_PIMP, true, false>(c, nullptr) : rhs_launch<T, T, RHS_PIMP, false, false>(c, nullptr);
    default: return per ? rhs_launch<T, T, RHS_FIMP, true, false>(c, nullptr) : rhs_launch<T, T, RHS_FIMP, false, false>(c, nullptr);
  }
}
cudaError_t launch_rhs(ch3d_ctx* c) { return c->fp32 ? rhs_t<float>(c) : rhs_t<double>(c); }

// explicit scheme: right-hand sides and u* = u + Rhs in one pass
template <class T> static cudaError_t fexp_t(ch3d_ctx* c) {
  return y_periodic(c) ? rhs_launch<T, T, RHS_FEXP, true, true>(c, nullptr)
                       : rhs_launch<T, T, RHS_FEXP, false, true>(c, nullptr);
}
cudaError_t launch_ustar_fexp(ch3d_ctx* c) { return c->fp32 ? fexp_t<float>(c) : fexp_t<double>(c); }

// learned closure (partially implicit): constant viscosity, explicit force, FP64 arithmetic on either field type
cudaError_t launch_rhs_les_const(ch3d_ctx* c) {
  return c->fp32 ? rhs_launch<float, double, RHS_LESC, false, false>(c, c->sgs_f)
                 : rhs_launch<double, double, RHS_LESC, false, false>(c, c->sgs_f);
}

}  // namespace ch3d
