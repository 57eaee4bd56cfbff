// ch3d_march.cu -- the 2nd-order partially implicit substep's right-hand
// sides fused with its y Crank-Nicolson solves, as a column march:
// clcRhsX/Y/Z_PIMP (src/CFD_2nd/m_TSchemePIMP_inc.f90:7-75, 161-209, 277-325)
// followed by clcU1/2/3Hat_PIMP (:392-430, 542-589, 702-740), u -> u*.
//
// One thread owns one (i, k) column and all three velocity components.  A
// block of 32 x BZ columns marches j upwards through a ring of staged rows in
// shared memory (ux, uy, uz, p of the block's columns plus a one-cell halo in
// x and z, and the row's table entries; rows -1 and ny are the wall ghosts of
// SetBC_and_UpdateHalo, src/CFD_2nd/m_BC_and_Halo.f90:241-282).  At row j the
// thread evaluates the three right-hand sides from rows j-1, j, j+1 of the
// ring, updates Hist, and eliminates row j of the three tridiagonal systems
// (Thomas; the factors are the same for every column and come from a per-row
// table).  Instead of the eliminated right-hand side d_j it stores
//     g_j = u_j + d_j + cp_j u_{j+1}
// in the u* array; the back substitution x_j = d_j - cp_j x_{j+1} of
// u*_j = u_j + x_j then reads only g:  u*_j = g_j - cp_j u*_{j+1}.
// On grids with few column tiles the march runs from both walls (twisted); on
// large grids it stops at g and the divergence and projection marches of this
// file substitute u* themselves (13 values of global traffic per cell: ux uy
// uz p, Hist x3 read + written, g x3 written).  Where the march substitutes
// itself, g is read back and u* written as well (19 values).
#include "ch3d_march.cuh"

namespace ch3d {

// Staging geometry: x halo H rounded up to whole copy vectors of VW points, and
// points per staged row of a 32 x BZ tile.
constexpr int march_hx(int H, int VW) { return (H + VW - 1) / VW * VW; }
constexpr int march_pl(int H, int VW, int BZ) { return (32 + 2 * march_hx(H, VW)) * (BZ + 2 * H); }

// Shared memory of one thread group of the march: RS row slots of the four
// staged fields (PL points each) and of the row table (MT_W values).
template <class T> constexpr size_t march_group_smem(int RS, int PL) {
  return (size_t)4 * RS * PL * sizeof(T) + (size_t)RS * MT_W * sizeof(T);
}

// Ring of RS row slots (row r in slot (r + 1) % RS); rows j+2 .. j+D+1 are in
// flight while row j is computed.  Slot (j+D+2), written after the barrier of
// iteration j, must differ from the slots of rows j-1, j, j+1 that other
// threads still read: RS >= D + 4.
//
// O4: the 4th-order right-hand sides (clcRhsXYZ, src/CFD_4th/m_TScheme.f90:
// 189-377) with a 3-cell x/z halo; their x- and z-interpolated velocities
// (:209-227) are formed from the staged rows instead of being stored.
//
// TW (twisted, for grids with too few column tiles to fill the GPU): the block
// has two thread groups per tile; the lower marches rows 0..m-1 upwards with the
// upward elimination, the upper rows ny-1..m downwards with the downward one,
// each with its own row ring; they meet at rows m-1, m (a 2x2 solve) and
// substitute outwards.  Same right-hand sides, half the march length.
//
// BS = false: the march stops at g; k_div_bsub and k_proj_bsub substitute
// u* = g - cp u*_{j+1} themselves while they walk each column downwards, so u*
// is never stored and g is never read back here (6 arrays less traffic).
//
// VW: rows staged in copy vectors of VW elements, 4 (16-byte copies of FP32 rows, the
// x halo rounded up to 4 points) where the FP32 march stops at g, which takes lines of
// whole vectors only, else 1.  That march is bound by instruction issue, so a quarter of
// the copy instructions and a sixth block per SM count: 2.08 ms per launch at 768x384x576
// and 194 us at 256x192x256, element by element with five blocks 2.28 ms and 201 us (the
// same bits).
template <class T, bool O4, bool TW, bool BS, int VW, int BZ, int D, int RS>
__global__ void __launch_bounds__(32 * BZ * (TW ? 2 : 1),
                                  VW == 4 ? 6 : (O4 ? 384 : (sizeof(T) == 4 ? 640 : 512)) / (32 * BZ * (TW ? 2 : 1)))
    k_rhs_march(Geo<T> g, const T* __restrict__ tab, const T* __restrict__ dtab, const T* __restrict__ ux, const T* __restrict__ uy,
                const T* __restrict__ uz, const T* __restrict__ pr, T* __restrict__ hx, T* __restrict__ hy,
                T* __restrict__ hz, T* __restrict__ uxs, T* __restrict__ uys, T* __restrict__ uzs,
                const DevScalars* __restrict__ sc) {
  constexpr int H = O4 ? 3 : 1;  // x/z halo
  constexpr int HX = march_hx(H, VW);  // staged x halo
  constexpr int BX = 32, NT = BX * BZ, SX = BX + 2 * HX, PL = march_pl(H, VW, BZ);
  constexpr int NS = (PL / VW + NT - 1) / NT;  // staging vectors per thread and array
  static_assert(VW == 1 || (VW == 4 && sizeof(T) == 4), "16-byte vectors of FP32 rows only");
  typedef typename std::conditional<VW == 4, float4, T>::type VT;
  static_assert(RS >= D + 4, "ring too small for the prefetch distance");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int hf = TW ? (int)threadIdx.x / NT : 0;  // thread group: 0 lower (or the only one), 1 upper
  // per thread group: the field rows [4][RS][PL], then the table rows [RS][MT_W]
  unsigned char* const grp_smem = smem_raw + (size_t)hf * march_group_smem<T>(RS, PL);
  T (*ring)[RS][PL] = reinterpret_cast<T (*)[RS][PL]>(grp_smem);
  T (*trs)[MT_W] = reinterpret_cast<T (*)[MT_W]>(grp_smem + (size_t)4 * RS * PL * sizeof(T));
  if (sc->status) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long plane = (long long)nx * ny;
  tab += (size_t)(sc->ns - 1) * ny * MT_W;  // this substep's tables
  dtab += (size_t)(sc->ns - 1) * ny * MD_W;
  const int tid = TW ? (int)threadIdx.x - hf * NT : (int)threadIdx.x, tx = tid & 31, tz = tid >> 5;
  const int mh = TW ? ny / 2 : ny;          // rows of the lower group (all rows without TW)
  const int nrow = TW && hf ? ny - mh : mh;  // rows this group marches
  const int dj = hf ? -1 : 1;                // march direction
  auto in_group = [&](int r) { return TW ? (hf ? r >= mh - 1 && r < ny : r >= 0 && r <= mh) : r >= 0 && r < ny; };
  auto slot = [](int r) { return (r + 1) % RS; };  // r >= -1
  // the groups march different numbers of rows (ny odd): each syncs on its own named barrier
  auto group_sync = [&]() {
    if constexpr (TW) {
      if (hf) asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
      else asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
    } else {
      __syncthreads();
    }
  };
  long long so[NS];  // staging slot offsets of the current tile
  auto issue_row = [&](int r) {  // r < ny
    const long long ro = (long long)r * nx;
    const int sl = slot(r);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const int s = (tid + q * NT) * VW;
      if (s < PL) {
        cp_async_el(reinterpret_cast<VT*>(&ring[0][sl][s]), reinterpret_cast<const VT*>(ux + so[q] + ro));
        cp_async_el(reinterpret_cast<VT*>(&ring[1][sl][s]), reinterpret_cast<const VT*>(uy + so[q] + ro));
        cp_async_el(reinterpret_cast<VT*>(&ring[2][sl][s]), reinterpret_cast<const VT*>(uz + so[q] + ro));
        cp_async_el(reinterpret_cast<VT*>(&ring[3][sl][s]), reinterpret_cast<const VT*>(pr + so[q] + ro));
      }
    }
    // the row's table entries (MT_W values, 16-byte copies) in the same copy group
    constexpr int TV = MT_W * (int)sizeof(T) / 16;
    if (tid < TV)
      cp_async_el(reinterpret_cast<float4*>(&trs[sl][0]) + tid, reinterpret_cast<const float4*>(tab + (size_t)r * MT_W) + tid);
  };
  // wall ghost rows from the thread's own staged slots next to them (at_jm / at_jp of ch3d_dev.cuh)
  auto ghost_row = [&](int r) {
    const int sl = slot(r);
#pragma unroll
    for (int qv = 0; qv < NS * VW; ++qv) {  // the elements of this thread's staging vectors
      const int s = (tid + (qv / VW) * NT) * VW + qv % VW;
      if (s >= PL) continue;
      if (r < 0) {
        const T u = ring[0][slot(0)][s], w = ring[2][slot(0)][s], v1 = ring[1][slot(1)][s];
        ring[0][sl][s] = g.bc.lo == -1 ? (T)(g.bc.ux_lo * 2.0) - u : u - (T)(g.bc.ux_lo * g.bc.dyp1);
        // uy(ic,0,kc) = 2 uy_ym - uy(ic,2,kc); never set (zero) in the 4th-order solver
        ring[1][sl][s] = O4 ? (T)0 : (T)(g.bc.uy_lo * 2.0) - v1;
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

  const T two = (T)2, half = (T)0.5, quarter = (T)0.25, one = (T)1;
  const T rdx = g.rdx, rdz = g.rdz, rdx2 = g.rdx2, rdz2 = g.rdz2, xnu = g.xnu;
  const T pmGamma = (T)sc->pmGamma, pmTheta = (T)sc->pmTheta, pmAlpha = (T)sc->pmAlpha, pmBeta = (T)sc->pmBeta;
  const T dpm = (T)sc->dpmdxns;
  const int c0 = (tz + H) * SX + tx + HX;
  const int ntx = (nx + BX - 1) / BX, ntiles = ntx * ((nz + BZ - 1) / BZ);

  // Persistent blocks walk tiles of 32 x BZ columns.  The back substitution of
  // a tile (HBM-bound) runs one row per forward row of the block's next tile
  // (latency-bound), so the two overlap instead of alternating in waves.
  bool pact = false;          // this thread's column of the previous tile is inside the grid
  long long pidx = 0;         // its row ny-1
  T p0 = (T)0, p1 = (T)0, p2 = (T)0;  // u* of the row above the next one to substitute
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
  const int i0 = (tile % ntx) * BX, k0 = (tile / ntx) * BZ;
  const int i = i0 + tx, k = k0 + tz;
  const bool act = i < nx && k < nz;
  // staging slots: s = tid + q NT -> halo-tile position (s % SX, s / SX), periodic in x and z
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const int s = (tid + q * NT) * VW;  // a vector never wraps: nx and i0 - HX are multiples of VW
    int ig = (i0 - HX + s % SX) % nx, kg = (k0 - H + s / SX) % nz;
    if (ig < 0) ig += nx;
    if (kg < 0) kg += nz;
    so[q] = s < PL ? ig + plane * kg : 0;
  }
  // prologue: the first D+2 rows of the march in flight, one copy group per row
#pragma unroll
  for (int r = 0; r <= D + 1; ++r) {
    const int row = hf ? ny - 1 - r : r;
    if (in_group(row)) issue_row(row);
    cp_async_commit();
  }
  const int jstart = hf ? ny - 1 : 0;
  long long idx = act ? i + plane * k + (long long)jstart * nx : 0;
  T d0 = (T)0, d1 = (T)0, d2 = (T)0;       // eliminated right-hand sides of the previous row
  T g0 = (T)0, g1 = (T)0, g2 = (T)0;       // g of the last row (= u* of row ny-1)
  T hxo = (T)0, hyo = (T)0, hzo = (T)0;    // Hist of row j
  T hx1 = (T)0, hy1 = (T)0, hz1 = (T)0;    // Hist of row j+1
  // pmTheta = 0 (first RK3 substep): the old Hist does not enter, so it is not read
  const bool hread = act && pmTheta != (T)0;
  const long long hstep = (long long)dj * nx;
  if (hread) {
    hxo = hx[idx]; hyo = hy[idx]; hzo = hz[idx];
    if (nrow > 1) { hx1 = hx[idx + hstep]; hy1 = hy[idx + hstep]; hz1 = hz[idx + hstep]; }
  }
  T lu0 = (T)0, lu1 = (T)0, lu2 = (T)0;  // u at the group's last row (TW meeting)

  // previous tile: row rb = ny-2-j of its back substitution at forward row j, its g
  // loaded two rows ahead
  T n0 = (T)0, n1 = (T)0, n2 = (T)0, m0 = (T)0, m1 = (T)0, m2 = (T)0;
  if (pact && ny >= 2) { n0 = uxs[pidx - nx]; n1 = uys[pidx - nx]; n2 = uzs[pidx - nx]; }
  if (pact && ny >= 3) { m0 = uxs[pidx - 2 * nx]; m1 = uys[pidx - 2 * nx]; m2 = uzs[pidx - 2 * nx]; }
  for (int sj = 0; sj < nrow; ++sj) {
    const int j = jstart + dj * sj;
    const int rb = ny - 2 - j;
    const bool bsub = pact && rb >= 0;
    const long long ob = pidx - (long long)(j + 1) * nx;
    const T b0 = n0, b1 = n1, b2 = n2;
    n0 = m0; n1 = m1; n2 = m2;
    if (pact && rb >= 2) { m0 = uxs[ob - 2 * nx]; m1 = uys[ob - 2 * nx]; m2 = uzs[ob - 2 * nx]; }
    cp_async_wait<D>();  // this thread's copies of rows <= j+1 are done
    if (j + 1 == ny) ghost_row(ny);
    if (j == 0) ghost_row(-1);
    group_sync();
    if (in_group(j + dj * (D + 2))) issue_row(j + dj * (D + 2));
    cp_async_commit();
    T hxn = (T)0, hyn = (T)0, hzn = (T)0;
    if (hread && sj + 2 < nrow) { hxn = hx[idx + 2 * hstep]; hyn = hy[idx + 2 * hstep]; hzn = hz[idx + 2 * hstep]; }
    if (act) {
      T rx, ry, rz, ux_c, uy_c, uz_c, ux_jp, uy_jp, uz_jp, ux_jm, uy_jm, uz_jm;
      const T* tr = trs[slot(j)];  // row j of the table, staged with the row
      if constexpr (!O4) {
      const T* X0 = &ring[0][slot(j - 1)][c0];
      const T* X1 = &ring[0][slot(j)][c0];
      const T* X2 = &ring[0][slot(j + 1)][c0];
      const T* Y0 = &ring[1][slot(j - 1)][c0];
      const T* Y1 = &ring[1][slot(j)][c0];
      const T* Y2 = &ring[1][slot(j + 1)][c0];
      const T* Z0 = &ring[2][slot(j - 1)][c0];
      const T* Z1 = &ring[2][slot(j)][c0];
      const T* Z2 = &ring[2][slot(j + 1)][c0];
      const T* P0 = &ring[3][slot(j - 1)][c0];
      const T* P1 = &ring[3][slot(j)][c0];

      const Sten2<T> s = {X1[0], X1[1], X1[-1], X2[0], X0[0], X1[SX], X1[-SX], X0[1], X1[1 - SX],
                          Y1[0], Y1[1], Y1[-1], Y2[0], Y0[0], Y1[SX], Y1[-SX], Y2[-1], Y2[-SX],
                          Z1[0], Z1[1], Z1[-1], Z2[0], Z0[0], Z1[SX], Z1[-SX], Z1[SX - 1], Z0[SX],
                          P1[0], P1[-1], P0[0], P1[-SX]};
      ux_c = s.ux_c; ux_jp = s.ux_jp; ux_jm = s.ux_jm;
      uy_c = s.uy_c; uy_jp = s.uy_jp; uy_jm = s.uy_jm;
      uz_c = s.uz_c; uz_jp = s.uz_jp; uz_jm = s.uz_jm;
      const T ho[3] = {hxo, hyo, hzo};
      const RhsCoef<T> pm = {pmGamma, pmTheta, pmAlpha, pmBeta};
      T r[3], h[3];
      rhs2_cell<RHS_PIMP>(g, tr, s, ho, pm, r, h);
      rx = r[0]; ry = r[1]; rz = r[2];
      hx[idx] = h[0]; hy[idx] = h[1]; hz[idx] = h[2];
      } else {
        // 4th order: row r, x offset dx, z offset dz of staged array a
        auto V = [&](int a, int r, int dx, int dz) -> T { return ring[a][slot(r)][c0 + dx + dz * SX]; };
        const C4<T> q(g);
        // interpolated velocities (k_interp4 pattern): x for ux (i'-1..i'+2), uy, uz (i'-2..i'+1);
        // z for ux, uy (k'-2..k'+1), uz (k'-1..k'+2)
        auto uxhx = [&](int r, int o, int dz) {
          return q.in1 * V(0, r, o - 1, dz) + q.in2 * V(0, r, o, dz) + q.in3 * V(0, r, o + 1, dz) + q.in4 * V(0, r, o + 2, dz);
        };
        auto hxa = [&](int a, int r, int o, int dz) {
          return q.in1 * V(a, r, o - 2, dz) + q.in2 * V(a, r, o - 1, dz) + q.in3 * V(a, r, o, dz) + q.in4 * V(a, r, o + 1, dz);
        };
        auto hza = [&](int a, int r, int dx, int o) {
          return q.in1 * V(a, r, dx, o - 2) + q.in2 * V(a, r, dx, o - 1) + q.in3 * V(a, r, dx, o) + q.in4 * V(a, r, dx, o + 1);
        };
        auto uzhz = [&](int r, int o) {
          return q.in1 * V(2, r, 0, o - 1) + q.in2 * V(2, r, 0, o) + q.in3 * V(2, r, 0, o + 1) + q.in4 * V(2, r, 0, o + 2);
        };
        const bool top = j + 1 == ny;  // uyhx, uyhz vanish on the jc = nyp row (:223-226)
        const T IY1 = tr[MT_IY1], IY2 = one - IY1;
        const T IY3 = tr[MT_IY3], IY4 = one - IY3;
        const T sucaj = tr[MT_RDYP];
        ux_c = V(0, j, 0, 0); ux_jp = V(0, j + 1, 0, 0); ux_jm = V(0, j - 1, 0, 0);
        uy_c = V(1, j, 0, 0); uy_jp = V(1, j + 1, 0, 0); uy_jm = V(1, j - 1, 0, 0);
        uz_c = V(2, j, 0, 0); uz_jp = V(2, j + 1, 0, 0); uz_jm = V(2, j - 1, 0, 0);
        {  // RhsX (:235-268)
          const T uxhyc = IY1 * ux_jm + IY2 * ux_c;
          const T uxhyp = IY3 * ux_c + IY4 * ux_jp;
          const T a1 = uxhx(j, -2, 0), a2 = uxhx(j, -1, 0), a3 = uxhx(j, 0, 0), a4 = uxhx(j, 1, 0);
          const T h11 = q.dx1 * a1 * a1 + q.dx2 * a2 * a2 + q.dx3 * a3 * a3 + q.dx4 * a4 * a4;
          const T h12 = ((top ? (T)0 : hxa(1, j + 1, 0, 0)) * uxhyp - hxa(1, j, 0, 0) * uxhyc) * sucaj;
          const T h13 = q.dz1 * hza(0, j, 0, -1) * hxa(2, j, 0, -1) + q.dz2 * hza(0, j, 0, 0) * hxa(2, j, 0, 0) +
                        q.dz3 * hza(0, j, 0, 1) * hxa(2, j, 0, 1) + q.dz4 * hza(0, j, 0, 2) * hxa(2, j, 0, 2);
          const T d11 = q.dxx1 * V(0, j, -2, 0) + q.dxx2 * V(0, j, -1, 0) + q.dxx3 * ux_c + q.dxx4 * V(0, j, 1, 0) +
                        q.dxx5 * V(0, j, 2, 0);
          const T d22 = tr[MT_AP2C] * ux_jp + tr[MT_AC2C] * ux_c + tr[MT_AM2C] * ux_jm;
          const T d33 = q.dzz1 * V(0, j, 0, -2) + q.dzz2 * V(0, j, 0, -1) + q.dzz3 * ux_c + q.dzz4 * V(0, j, 0, 1) +
                        q.dzz5 * V(0, j, 0, 2);
          const T conv = -h11 - h12 - h13 + xnu * (d11 + d33) + g.g1;
          const T gradp = q.dx1 * V(3, j, -2, 0) + q.dx2 * V(3, j, -1, 0) + q.dx3 * V(3, j, 0, 0) + q.dx4 * V(3, j, 1, 0);
          rx = pmGamma * conv + pmTheta * hxo - pmAlpha * gradp + two * pmBeta * d22;
          hx[idx] = conv;
        }
        {  // RhsY (:270-305)
          const T sucac = tr[MT_RDYC], qsucac = quarter * sucac;
          const T uxhym = IY1 * V(0, j - 1, -1, 0) + IY2 * V(0, j, -1, 0);
          const T uxhyc = IY1 * V(0, j - 1, 0, 0) + IY2 * V(0, j, 0, 0);
          const T uxhyp = IY1 * V(0, j - 1, 1, 0) + IY2 * V(0, j, 1, 0);
          const T uxhyu = IY1 * V(0, j - 1, 2, 0) + IY2 * V(0, j, 2, 0);
          const T uzhym = IY1 * V(2, j - 1, 0, -1) + IY2 * V(2, j, 0, -1);
          const T uzhyc = IY1 * V(2, j - 1, 0, 0) + IY2 * V(2, j, 0, 0);
          const T uzhyp = IY1 * V(2, j - 1, 0, 1) + IY2 * V(2, j, 0, 1);
          const T uzhyu = IY1 * V(2, j - 1, 0, 2) + IY2 * V(2, j, 0, 2);
          const T h21 = q.dx1 * hxa(1, j, -1, 0) * uxhym + q.dx2 * hxa(1, j, 0, 0) * uxhyc +
                        q.dx3 * hxa(1, j, 1, 0) * uxhyp + q.dx4 * hxa(1, j, 2, 0) * uxhyu;
          const T h22 = ((uy_jp + uy_c) * (uy_jp + uy_c) - (uy_c + uy_jm) * (uy_c + uy_jm)) * qsucac;
          const T h23 = q.dz1 * hza(1, j, 0, -1) * uzhym + q.dz2 * hza(1, j, 0, 0) * uzhyc +
                        q.dz3 * hza(1, j, 0, 1) * uzhyp + q.dz4 * hza(1, j, 0, 2) * uzhyu;
          const T d11 = q.dxx1 * V(1, j, -2, 0) + q.dxx2 * V(1, j, -1, 0) + q.dxx3 * uy_c + q.dxx4 * V(1, j, 1, 0) +
                        q.dxx5 * V(1, j, 2, 0);
          const T d22 = tr[MT_AP2P] * uy_jp + tr[MT_AC2P] * uy_c + tr[MT_AM2P] * uy_jm;
          const T d33 = q.dzz1 * V(1, j, 0, -2) + q.dzz2 * V(1, j, 0, -1) + q.dzz3 * uy_c + q.dzz4 * V(1, j, 0, 1) +
                        q.dzz5 * V(1, j, 0, 2);
          const T conv = -h21 - h22 - h23 + xnu * (d11 + d33) + g.g2;
          const T gradp = (V(3, j, 0, 0) - V(3, j - 1, 0, 0)) * sucac;
          ry = pmGamma * conv + pmTheta * hyo - pmAlpha * gradp + two * pmBeta * d22;
          hy[idx] = conv;
        }
        {  // RhsZ (:307-343)
          const T uzhyc = IY1 * uz_jm + IY2 * uz_c;
          const T uzhyp = IY3 * uz_c + IY4 * uz_jp;
          const T h31 = q.dx1 * hxa(2, j, -1, 0) * hza(0, j, -1, 0) + q.dx2 * hxa(2, j, 0, 0) * hza(0, j, 0, 0) +
                        q.dx3 * hxa(2, j, 1, 0) * hza(0, j, 1, 0) + q.dx4 * hxa(2, j, 2, 0) * hza(0, j, 2, 0);
          const T h32 = ((top ? (T)0 : hza(1, j + 1, 0, 0)) * uzhyp - hza(1, j, 0, 0) * uzhyc) * sucaj;
          const T b1 = uzhz(j, -2), b2 = uzhz(j, -1), b3 = uzhz(j, 0), b4 = uzhz(j, 1);
          const T h33 = q.dz1 * b1 * b1 + q.dz2 * b2 * b2 + q.dz3 * b3 * b3 + q.dz4 * b4 * b4;
          const T d11 = q.dxx1 * V(2, j, -2, 0) + q.dxx2 * V(2, j, -1, 0) + q.dxx3 * uz_c + q.dxx4 * V(2, j, 1, 0) +
                        q.dxx5 * V(2, j, 2, 0);
          const T d22 = tr[MT_AP2C] * uz_jp + tr[MT_AC2C] * uz_c + tr[MT_AM2C] * uz_jm;
          const T d33 = q.dzz1 * V(2, j, 0, -2) + q.dzz2 * V(2, j, 0, -1) + q.dzz3 * uz_c + q.dzz4 * V(2, j, 0, 1) +
                        q.dzz5 * V(2, j, 0, 2);
          const T conv = -h31 - h32 - h33 + xnu * (d11 + d33) + g.g3;
          const T gradp = q.dz1 * V(3, j, 0, -2) + q.dz2 * V(3, j, 0, -1) + q.dz3 * V(3, j, 0, 0) + q.dz4 * V(3, j, 0, 1);
          rz = pmGamma * conv + pmTheta * hzo - pmAlpha * gradp + two * pmBeta * d22;
          hz[idx] = conv;
        }
      }
      rx += dpm;                     // mean pressure gradient (clcRhsX_PIMP :61-74)
      if (j == 0) ry = (T)0;         // duy_ym: uy_ym is constant (Update_uy_ym_CH)
      if (!TW || hf == 0) {  // upward elimination; g = u + d + cp u_{j+1}
        d0 = (rx - tr[MT_A0] * d0) * tr[MT_RM0];
        d1 = (ry - tr[MT_A1] * d1) * tr[MT_RM1];
        d2 = (rz - tr[MT_A0] * d2) * tr[MT_RM0];
        g0 = ux_c + d0 + tr[MT_CP0] * ux_jp;
        g1 = uy_c + d1 + tr[MT_CP1] * uy_jp;
        g2 = uz_c + d2 + tr[MT_CP0] * uz_jp;
      } else {               // downward elimination; g = u + e + aq u_{j-1}
        const T* td = dtab + (size_t)j * MD_W;
        d0 = (rx - __ldg(td + MD_C0) * d0) * __ldg(td + MD_RQ0);
        d1 = (ry - __ldg(td + MD_C1) * d1) * __ldg(td + MD_RQ1);
        d2 = (rz - __ldg(td + MD_C0) * d2) * __ldg(td + MD_RQ0);
        g0 = ux_c + d0 + __ldg(td + MD_AQ0) * ux_jm;
        g1 = uy_c + d1 + __ldg(td + MD_AQ1) * uy_jm;
        g2 = uz_c + d2 + __ldg(td + MD_AQ0) * uz_jm;
      }
      uxs[idx] = g0; uys[idx] = g1; uzs[idx] = g2;
      lu0 = ux_c; lu1 = uy_c; lu2 = uz_c;
    }
    if (bsub) {  // u*_rb = g_rb - cp_rb u*_{rb+1}
      const T* tb = tab + (size_t)rb * MT_W;
      const T cb0 = __ldg(tb + MT_CP0), cb1 = __ldg(tb + MT_CP1);
      p0 = b0 - cb0 * p0; p1 = b1 - cb1 * p1; p2 = b2 - cb0 * p2;
      uxs[ob] = p0; uys[ob] = p1; uzs[ob] = p2;
    }
    idx += hstep;
    hxo = hx1; hyo = hy1; hzo = hz1;
    hx1 = hxn; hy1 = hyn; hz1 = hzn;
  }
  cp_async_wait<0>();
  __syncthreads();  // the ring is refilled by the next tile's prologue (or reused below)
  if constexpr (TW) {
    // meeting of the groups at rows m-1 (lower: x = d - cp x_m) and m (upper: x = e - aq x_{m-1})
    T* xch = reinterpret_cast<T*>(smem_raw);  // [2][NT][6]
    if (act) {
      T* o = xch + ((size_t)hf * NT + tid) * 6;
      o[0] = d0; o[1] = d1; o[2] = d2; o[3] = lu0; o[4] = lu1; o[5] = lu2;
    }
    __syncthreads();
    if (!act) return;
    const T* lo = xch + (size_t)tid * 6;
    const T* up = xch + ((size_t)NT + tid) * 6;
    const T* tl = tab + (size_t)(mh - 1) * MT_W;
    const T* tu = dtab + (size_t)mh * MD_W;
    T xl[3], xu[3];
    const T cpl[3] = {__ldg(tl + MT_CP0), __ldg(tl + MT_CP1), __ldg(tl + MT_CP0)};
    const T aqu[3] = {__ldg(tu + MD_AQ0), __ldg(tu + MD_AQ1), __ldg(tu + MD_AQ0)};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      xl[q] = (lo[q] - cpl[q] * up[q]) / ((T)1 - cpl[q] * aqu[q]);
      xu[q] = up[q] - aqu[q] * xl[q];
    }
    // this group's boundary row, then outwards: u*_j = g_j - f_j u*_{j -+ 1}
    const int jb = hf ? mh : mh - 1;
    const T* uu = hf ? up : lo;
    const T* xx = hf ? xu : xl;
    long long o = i + plane * k + (long long)jb * nx;
    T c0v = uu[3] + xx[0], c1v = uu[4] + xx[1], c2v = uu[5] + xx[2];
    uxs[o] = c0v; uys[o] = c1v; uzs[o] = c2v;
    const T* ft = hf ? dtab : tab;  // substitution factors: aq (upper group) or cp (lower)
    const int fw = hf ? MD_W : MT_W, fo0 = hf ? MD_AQ0 : MT_CP0, fo1 = hf ? MD_AQ1 : MT_CP1;
    const int nout = hf ? ny - 1 - jb : jb;  // rows still to substitute
    constexpr int B = 8;
    for (int r0 = 0; r0 < nout; r0 += B) {
      T a0[B], a1[B], a2[B];
#pragma unroll
      for (int b = 0; b < B; ++b) {
        if (r0 + b < nout) {
          const long long ob = o - (long long)dj * (r0 + b + 1) * nx;
          a0[b] = uxs[ob]; a1[b] = uys[ob]; a2[b] = uzs[ob];
        }
      }
#pragma unroll
      for (int b = 0; b < B; ++b) {
        if (r0 + b < nout) {
          const int jr = jb - dj * (r0 + b + 1);
          const T* tb = ft + (size_t)jr * fw;
          const T f0 = __ldg(tb + fo0), f1 = __ldg(tb + fo1);
          c0v = a0[b] - f0 * c0v; c1v = a1[b] - f1 * c1v; c2v = a2[b] - f0 * c2v;
          const long long ob = o - (long long)dj * (r0 + b + 1) * nx;
          uxs[ob] = c0v; uys[ob] = c1v; uzs[ob] = c2v;
        }
      }
    }
    return;
  }
  pact = BS && act; pidx = idx - nx; p0 = g0; p1 = g1; p2 = g2;
  }  // tiles
  if (!pact) return;

  // back substitution of the block's last tile, rows loaded in batches of 8
  constexpr int B = 8;
  long long idx = pidx;  // row ny-1 (u* = g there)
  T g0 = p0, g1 = p1, g2 = p2;
  for (int j = ny - 2; j >= 0; j -= B) {
    T a0[B], a1[B], a2[B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      if (j - b >= 0) {
        const long long o = idx - (long long)(b + 1) * nx;
        a0[b] = uxs[o]; a1[b] = uys[o]; a2[b] = uzs[o];
      }
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      if (j - b >= 0) {
        const T* tr = tab + (size_t)(j - b) * MT_W;
        const T cp0 = __ldg(tr + MT_CP0), cp1 = __ldg(tr + MT_CP1);
        g0 = a0[b] - cp0 * g0; g1 = a1[b] - cp1 * g1; g2 = a2[b] - cp0 * g2;
        const long long o = idx - (long long)(b + 1) * nx;
        uxs[o] = g0; uys[o] = g1; uzs[o] = g2;
      }
    }
    idx -= (long long)B * nx;
  }
}

// ---------------------------------------------------------------------------
// FluidVelUpdate (src/CFD_2nd/m_TScheme.f90:281-306; 4th order
// src/CFD_4th/m_TScheme.f90:148-173) + the pressure update as a march: a thread
// owns one (i, k) column over a chunk of `rows` rows and keeps phi at j-1, j, j+1
// in registers (Neumann ghosts of SetBC_and_UpdateHalo_pr at the walls, periodic
// rows without).  The block's sum of ux * s1coe (the next substep's bulk
// constraint, clcRhsX_PIMP m_TSchemePIMP_inc.f90:60-74, or mean viscous stress)
// goes to part[block].  mode 1: projection only (pmAlpha = 1, p kept).
// KIND: 0 PressureUpdate_PIMP (src/CFD_2nd/m_TSchemePIMP_inc.f90:852-873), 1 _FIMP and
// _FEXP (m_TSchemeFIMP_inc.f90:1371-1386, m_TSchemeFEXP_inc.f90:513-548), 2 the 4th
// order (PIMP), 3 PressureUpdate_PIMP_LES (m_TSchemePIMP_inc.f90:878-904).
// ---------------------------------------------------------------------------
// Rows per block of the march projection: 32 where the grid fills the GPU anyway,
// else as few as give about four blocks per SM (at least 4: a block's first and
// last row read phi of the rows next to them).  64^3: 17.2 us with 32 rows (64
// blocks), 9.4 us with 4.
static int proj_rows(const ch3d_ctx* c) {
  const long long cols = (long long)((c->nx + 31) / 32) * ((c->nz + 3) / 4);
  int rows = 32;
  while (rows > 4 && cols * ((c->ny + rows - 1) / rows) < 4LL * sm_count(c->device)) rows >>= 1;
  return rows;
}

__device__ __forceinline__ double block_sum128(double v, double* sh /* 4 */) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  return threadIdx.x == 0 ? (sh[0] + sh[1]) + (sh[2] + sh[3]) : 0.0;
}

// DIAG (last substep of a step, 2nd order): CheckDivergence, CalcVmax, the next step's CalcMaxCFL and the
// CalcUxAver partials (src/CFD_2nd/m_Tools.f90:21-104,250-270) of the new
// velocity, fused in.  The i+1, j+1 and k+1 neighbours of the new velocity
// are recomputed from u* and phi with the same expressions their own threads
// use, so they equal the stored values bit for bit.
template <class T, bool DIAG, int KIND>
__global__ void __launch_bounds__(128) k_proj_march(Geo<T> g, Metrics<T> m, const T* uxs, const T* uys,
                                                    const T* uzs, T* ux, T* uy, T* uz, T* __restrict__ pr,
                                                    const T* __restrict__ phi, const T* __restrict__ nut,
                                                    double* __restrict__ part,
                                                    double* __restrict__ part2, int mode, int rows,
                                                    DevScalars* __restrict__ sc) {
  __shared__ double red[7][4];
  if (sc->status) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long plane = (long long)nx * ny;
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), k = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int j0 = blockIdx.z * rows, j1 = min(j0 + rows, ny);
  double s = 0.0, s2 = 0.0, dv = 0.0, v0 = 0.0, v1 = 0.0, v2 = 0.0, cf = 0.0;
  if (i < nx && k < nz) {
    const long long col = i + plane * k;
    const long long dxm = i == 0 ? nx - 1 : -1;                           // offset to i-1
    const long long dzm = k == 0 ? (long long)(nz - 1) * plane : -plane;  // offset to k-1
    const long long dxp = i + 1 == nx ? 1 - nx : 1;                       // offset to i+1
    const long long dzp = k + 1 == nz ? -(long long)(nz - 1) * plane : plane;  // offset to k+1
    const T pmAlpha = mode == 0 ? (T)sc->pmAlpha : (T)1;
    const T pmBeta = (T)sc->pmBeta;
    const T rdxEta2 = g.rdx * pmAlpha, rdzEta2 = g.rdz * pmAlpha;
    const double rdx = g.rdx, rdz = g.rdz;
    const bool per = g.bc.lo == 0;  // periodic in y
    const T pmBetaT = KIND == 3 ? (T)sc->pmBetaT : (T)0;
    const long long dx2 = i >= 2 ? -2 : nx - 2;
    const long long dz2 = k >= 2 ? -2 * plane : (long long)(nz - 2) * plane;
    const C4<T> c4(g);
    T pm = __ldg(phi + col + (long long)(j0 > 0 ? j0 - 1 : (per ? ny - 1 : 0)) * nx);
    T pc = __ldg(phi + col + (long long)j0 * nx);
    // rows in batches of PB: all loads of a batch before its stores (u* and u may
    // be the same arrays, mode 1, so the compiler cannot reorder them itself)
    constexpr int PB = DIAG || KIND >= 2 ? 2 : 4;
    for (int jb = j0; jb < j1; jb += PB) {
      T vpp[PB], vpx[PB], vpz[PB], vu[PB], vv[PB], vw[PB], vp[PB], mr[PB], mp[PB], mc[PB], mm[PB], ms[PB];
      T ex[4][PB];  // KIND 2: phi at i-2, i+1, k-2, k+1; KIND 3: nut at j, j+1, j-1
      T qux[PB], qpx[PB], quz[PB], qpz[PB], quy[PB], qr[PB], qrp[PB], qdy[PB];  // DIAG neighbours, metrics
#pragma unroll
      for (int b = 0; b < PB; ++b) {
        const int j = jb + b < j1 ? jb + b : j1 - 1;
        const long long idx = col + (long long)j * nx;
        const int jn = j + 1 < ny ? j + 1 : (per ? 0 : ny - 1);
        vpp[b] = __ldg(phi + col + (long long)jn * nx);
        vpx[b] = __ldg(phi + idx + dxm);
        vpz[b] = __ldg(phi + idx + dzm);
        vu[b] = uxs[idx]; vv[b] = uys[idx]; vw[b] = uzs[idx];
        vp[b] = mode == 0 ? pr[idx] : (T)0;
        mr[b] = m.rdyc[j + 1]; mp[b] = m.ap2Pr[j + 1]; mc[b] = m.ac2Pr[j + 1]; mm[b] = m.am2Pr[j + 1];
        ms[b] = m.s1coe[j + 1];
        if (KIND == 2) {
          ex[0][b] = __ldg(phi + idx + dx2);
          ex[1][b] = __ldg(phi + idx + dxp);
          ex[2][b] = __ldg(phi + idx + dz2);
          ex[3][b] = __ldg(phi + idx + dzp);
        }
        if (KIND == 3 && mode == 0) {
          ex[0][b] = __ldg(nut + idx);
          ex[1][b] = j < ny - 1 ? __ldg(nut + idx + nx) : (T)0;
          ex[2][b] = j > 0 ? __ldg(nut + idx - nx) : (T)0;
          ex[3][b] = m.rdyc[j + 2];
        }
        if (DIAG) {
          qux[b] = uxs[idx + dxp]; qpx[b] = __ldg(phi + idx + dxp);
          quz[b] = uzs[idx + dzp]; qpz[b] = __ldg(phi + idx + dzp);
          quy[b] = uys[col + (long long)jn * nx];
          qr[b] = m.rdyc[jn + 1]; qrp[b] = m.rdyp[j + 1]; qdy[b] = m.dyp[j + 1];
        }
      }
#pragma unroll
      for (int b = 0; b < PB; ++b) {
        const int j = jb + b;
        if (j >= j1) break;
        const long long idx = col + (long long)j * nx;
        const T pp = vpp[b];
        const T sucacEta2 = mr[b] * pmAlpha;
        T uxn = vu[b] - (pc - vpx[b]) * rdxEta2;
        T uyn = vv[b] - (pc - pm) * sucacEta2;
        T uzn = vw[b] - (pc - vpz[b]) * rdzEta2;
        if (KIND == 2) {
          uxn = vu[b] - pmAlpha * (c4.dx1 * ex[0][b] + c4.dx2 * vpx[b] + c4.dx3 * pc + c4.dx4 * ex[1][b]);
          uyn = vv[b] - pmAlpha * ((pc - pm) * mr[b]);
          uzn = vw[b] - pmAlpha * (c4.dz1 * ex[2][b] + c4.dz2 * vpz[b] + c4.dz3 * pc + c4.dz4 * ex[3][b]);
        }
        ux[idx] = uxn; uy[idx] = uyn; uz[idx] = uzn;
        if (KIND == 1) {
          if (mode == 0) pr[idx] = vp[b] + pc;
        } else if (KIND == 3) {
          if (mode == 0) {
            const T nc = ex[0][b];
            const T njp = j < ny - 1 ? ex[1][b] : (g.bc.hi == -1 ? (T)2 * g.xnu - nc : nc);
            const T njm = j > 0 ? ex[2][b] : (g.bc.lo == -1 ? (T)2 * g.xnu - nc : nc);
            const T rdyp = m.rdyp[j + 1];
            const T pmBetap = -pmBetaT * (rdyp * ex[3][b]) * ((T)0.5 * (njp + nc));
            const T pmBetam = -pmBetaT * (rdyp * mr[b]) * ((T)0.5 * (nc + njm));
            pr[idx] = vp[b] + pmBetap * pp + (-(pmBetap + pmBetam) + (T)1) * pc + pmBetam * pm;
          }
        } else if (mode == 0) {
          const T pmBetap = -pmBeta * mp[b];
          const T pmBetac = -pmBeta * mc[b] + (T)1;
          const T pmBetam = -pmBeta * mm[b];
          pr[idx] = vp[b] + pmBetap * pp + pmBetac * pc + pmBetam * pm;
        }
        s += (double)uxn * (double)ms[b];
        if (DIAG) {
          // the new velocity at i+1, k+1 and j+1, as the threads that own them compute it
          const T uxp = qux[b] - (qpx[b] - pc) * rdxEta2;
          const T uzp = quz[b] - (qpz[b] - pc) * rdzEta2;
          const T uyp = j + 1 < ny || per ? quy[b] - (pp - pc) * (qr[b] * pmAlpha) : (T)g.bc.uy_hi;
          const double a = uxn, bb = uyn, c = uzn, aip = uxp, bjp = uyp, ckp = uzp, rdyp = qrp[b];
          double d = fabs((aip - a) * rdx + (bjp - bb) * rdyp + (ckp - c) * rdz);
          if (!(d == d)) d = INFINITY;  // NaN folded into +inf: a NaN field trips the limits
          dv = fmax(dv, d);
          v0 = fmax(v0, a == a ? fabs(a) : INFINITY);
          v1 = fmax(v1, bb == bb ? fabs(bb) : INFINITY);
          v2 = fmax(v2, c == c ? fabs(c) : INFINITY);
          cf = fmax(cf, fabs(a + aip) * rdx + fabs(bb + bjp) * rdyp + fabs(c + ckp) * rdz);
          s2 += a * (double)qdy[b];
        }
        pm = pc; pc = pp;
      }
    }
  }
  if constexpr (!DIAG) {
    const double bs = block_sum128(s, red[0]);
    if (threadIdx.x == 0) part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = bs;
  } else {
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    dv = fmax(dv, __shfl_xor_sync(0xffffffffu, dv, o));
    v0 = fmax(v0, __shfl_xor_sync(0xffffffffu, v0, o));
    v1 = fmax(v1, __shfl_xor_sync(0xffffffffu, v1, o));
    v2 = fmax(v2, __shfl_xor_sync(0xffffffffu, v2, o));
    cf = fmax(cf, __shfl_xor_sync(0xffffffffu, cf, o));
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = s; red[1][w] = s2; red[2][w] = cf; red[3][w] = dv; red[4][w] = v0; red[5][w] = v1; red[6][w] = v2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r[7];
    for (int q = 0; q < 2; ++q) r[q] = (red[q][0] + red[q][1]) + (red[q][2] + red[q][3]);
    for (int q = 2; q < 7; ++q) r[q] = fmax(fmax(red[q][0], red[q][1]), fmax(red[q][2], red[q][3]));
    const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    part[bid] = r[0];
    part2[bid] = r[1];
    atomic_max_nonneg(&sc->uddx, r[2] * 0.5);
    atomic_max_nonneg(&sc->divmax2, r[3]);
    atomic_max_nonneg(&sc->vmax[0], r[4]);
    atomic_max_nonneg(&sc->vmax[1], r[5]);
    atomic_max_nonneg(&sc->vmax[2], r[6]);
  }
  }
}

// the same partial sums of ux * s1coe for a freshly uploaded field
template <class T>
__global__ void __launch_bounds__(128) k_bulk_march(Geo<T> g, Metrics<T> m, const T* __restrict__ ux,
                                                    double* __restrict__ part, int rows) {
  __shared__ double red[4];
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), k = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int j0 = blockIdx.z * rows, j1 = min(j0 + rows, ny);
  double s = 0.0;
  if (i < nx && k < nz) {
    const long long col = i + (long long)nx * ny * k;
    for (int j = j0; j < j1; ++j) s += (double)ux[col + (long long)j * nx] * (double)m.s1coe[j + 1];
  }
  const double bs = block_sum128(s, red);
  if (threadIdx.x == 0) part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = bs;
}

// ---------------------------------------------------------------------------
// Marches that substitute the march's g themselves (BS = false above): one
// thread per (i, k) column, 32 x 4 columns per block, walking j downwards with
// u*_j = g_j - cp_j u*_{j+1} (cp of the substep's row table; u*_{ny-1} = g_{ny-1}
// since cp_{ny-1} = 0) for its own column and, where a stencil needs them, for
// the columns at i+1 (ux) and k+1 (uz), with the same expressions as the
// threads that own them.  All loads of a batch of PB rows are issued before its
// recurrence steps.
// ---------------------------------------------------------------------------

// clcPrSrcOther (src/CFD_2nd/m_TScheme.f90:213-241): div(u*) per cell into dv
// (scaled by 1/pmAlpha and transformed by the x kernel, mode 3), its maximum
// |div| into divmax1 (CheckDivergence before the projection).  PB rows of loads
// in flight: 8 (168 registers, three blocks per SM) where the grid runs many
// waves anyway, 4 (100 registers) where the column blocks fit in one wave at five.
template <class T, int PB, bool BND>
__global__ void __launch_bounds__(128) k_div_bsub(Geo<T> g, Metrics<T> m, const T* __restrict__ tab,
                                                  const T* __restrict__ gx, const T* __restrict__ gy,
                                                  const T* __restrict__ gz, T* __restrict__ dv, T* __restrict__ bnd,
                                                  int rows, DevScalars* __restrict__ sc) {
  __shared__ double red[4];
  if (sc->status) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long plane = (long long)nx * ny;
  tab += (size_t)(sc->ns - 1) * ny * MT_W;
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), k = blockIdx.y * 4 + (threadIdx.x >> 5);
  double dmax = 0.0;
  if (i < nx && k < nz) {
    const long long col = i + plane * k;
    const long long dxp = i + 1 == nx ? 1 - nx : 1;                            // offset to i+1
    const long long dzp = k + 1 == nz ? -(long long)(nz - 1) * plane : plane;  // offset to k+1
    const T rdx = g.rdx, rdz = g.rdz;
    T ax = (T)0, axp = (T)0, ay = (T)0, az = (T)0, azp = (T)0;  // u* of row j+1
    T ayn = (T)g.bc.uy_hi;  // uy at j+1: the wall value above the top row
    // rows ny-1-b, ny-1-b-PB, ... pass through register slot b; a slot is refilled
    // with the row PB below as soon as it is consumed
    T vx[PB], vxp[PB], vy[PB], vz[PB], vzp[PB], c0[PB], c1[PB], sy[PB];
    auto load = [&](int b, int j) {
      const long long idx = col + (long long)j * nx;
      vx[b] = gx[idx]; vxp[b] = gx[idx + dxp]; vy[b] = gy[idx];
      vz[b] = gz[idx]; vzp[b] = gz[idx + dzp];
      c0[b] = __ldg(tab + (size_t)j * MT_W + MT_CP0);
      c1[b] = __ldg(tab + (size_t)j * MT_W + MT_CP1);
      sy[b] = m.rdyp[j + 1];
    };
#pragma unroll
    for (int b = 0; b < PB; ++b) load(b, ny - 1 - b >= 0 ? ny - 1 - b : 0);
    for (int jb = ny - 1; jb >= 0; jb -= PB) {
#pragma unroll
      for (int b = 0; b < PB; ++b) {
        const int j = jb - b;
        if (j < 0) break;
        ax = vx[b] - c0[b] * ax;
        axp = vxp[b] - c0[b] * axp;
        ay = vy[b] - c1[b] * ay;
        az = vz[b] - c0[b] * az;
        azp = vzp[b] - c0[b] * azp;
        const T r = (axp - ax) * rdx + (ayn - ay) * sy[b] + (azp - az) * rdz;
        if (j >= PB) load(b, j - PB);
        dv[col + (long long)j * nx] = r;
        if (BND && (j & (rows - 1)) == 0 && j > 0) {  // u* above the chunk of rows that ends here
          const long long n2 = (long long)nx * nz;
          T* const q = bnd + 3 * n2 * (j / rows - 1) + i + (long long)nx * k;
          q[0] = ax; q[n2] = ay; q[2 * n2] = az;
        }
        dmax = fmax(dmax, fabs((double)r));
        ayn = ay;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dmax;
  __syncthreads();
  if (threadIdx.x == 0) atomic_max_nonneg(&sc->divmax1, fmax(fmax(red[0], red[1]), fmax(red[2], red[3])));
}

// FluidVelUpdate + PressureUpdate_PIMP (m_TScheme.f90:281-306, m_TSchemePIMP_inc.f90:
// 852-873) from g, as k_proj_march in mode 0; DIAG: the step diagnostics of the
// last substep (CheckDivergence, CalcVmax, CalcMaxCFL, CalcUxAver).  A block walks
// the whole column where the tiles alone fill the GPU (rows = ny), else the chunk
// blockIdx.z of `rows` rows from the u* that k_div_bsub left above it (bnd).  Partial
// sums go to the slots of the chunked projection grid (npz row chunks), the unused
// chunk slots of each block set to zero.
template <class T, bool DIAG>
__global__ void __launch_bounds__(128) k_proj_bsub(Geo<T> g, Metrics<T> m, const T* __restrict__ tab,
                                                   const T* __restrict__ gx, const T* __restrict__ gy,
                                                   const T* __restrict__ gz, T* __restrict__ ux, T* __restrict__ uy,
                                                   T* __restrict__ uz, T* __restrict__ pr, const T* __restrict__ phi,
                                                   const T* __restrict__ bnd, double* __restrict__ part,
                                                   double* __restrict__ part2, int npz, int rows,
                                                   DevScalars* __restrict__ sc) {
  __shared__ double red[7][4];
  if (sc->status) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long plane = (long long)nx * ny;
  tab += (size_t)(sc->ns - 1) * ny * MT_W;
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), k = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int j0 = blockIdx.z * rows, j1 = min(j0 + rows, ny);
  double s = 0.0, s2 = 0.0, dvm = 0.0, v0 = 0.0, v1 = 0.0, v2 = 0.0, cf = 0.0;
  if (i < nx && k < nz) {
    const long long col = i + plane * k;
    const long long dxm = i == 0 ? nx - 1 : -1;                                // offset to i-1
    const long long dzm = k == 0 ? (long long)(nz - 1) * plane : -plane;       // offset to k-1
    const long long dxp = i + 1 == nx ? 1 - nx : 1;                            // offset to i+1
    const long long dzp = k + 1 == nz ? -(long long)(nz - 1) * plane : plane;  // offset to k+1
    const T pmAlpha = (T)sc->pmAlpha, pmBeta = (T)sc->pmBeta;
    const T rdxEta2 = g.rdx * pmAlpha, rdzEta2 = g.rdz * pmAlpha;
    const double rdx = g.rdx, rdz = g.rdz;
    T ax = (T)0, ay = (T)0, az = (T)0, axp = (T)0, azp = (T)0;  // u* of row j+1
    T pc = __ldg(phi + col + (long long)(j1 - 1) * nx);         // phi(j)
    T pp = pc;                                                   // phi(j+1), clamped at the top row
    T uyp = (T)g.bc.uy_hi;                                       // new uy at j+1 (DIAG)
    if (j1 < ny) {
      const long long n2 = (long long)nx * nz;
      const T* const q = bnd + 3 * n2 * blockIdx.z;
      const long long cc = i + (long long)nx * k, ck = i + (long long)nx * (k + 1 == nz ? 0 : k + 1);
      ax = __ldg(q + cc); ay = __ldg(q + n2 + cc); az = __ldg(q + 2 * n2 + cc);
      pp = __ldg(phi + col + (long long)j1 * nx);
      if (DIAG) {
        axp = __ldg(q + cc + dxp);
        azp = __ldg(q + 2 * n2 + ck);
        uyp = ay - (pp - pc) * (m.rdyc[j1 + 1] * pmAlpha);
      }
    }
    // rows pass through PB register slots, each refilled with the row PB below once consumed
    constexpr int PB = DIAG ? 2 : 4;
    T vx[PB], vy[PB], vz[PB], vp[PB], vpm[PB], vpx[PB], vpz[PB], c0[PB], c1[PB];
    T mr[PB], mp[PB], mc[PB], mm[PB], ms[PB];
    T qx[PB], qz[PB], qpx[PB], qpz[PB], qrp[PB], qdy[PB];  // DIAG neighbours, metrics
    auto load = [&](int b, int j) {
      const long long idx = col + (long long)j * nx;
      const int jm = j > 0 ? j - 1 : 0;
      vx[b] = gx[idx]; vy[b] = gy[idx]; vz[b] = gz[idx]; vp[b] = pr[idx];
      vpm[b] = __ldg(phi + col + (long long)jm * nx);
      vpx[b] = __ldg(phi + idx + dxm);
      vpz[b] = __ldg(phi + idx + dzm);
      c0[b] = __ldg(tab + (size_t)j * MT_W + MT_CP0);
      c1[b] = __ldg(tab + (size_t)j * MT_W + MT_CP1);
      mr[b] = m.rdyc[j + 1]; mp[b] = m.ap2Pr[j + 1]; mc[b] = m.ac2Pr[j + 1]; mm[b] = m.am2Pr[j + 1];
      ms[b] = m.s1coe[j + 1];
      if (DIAG) {
        qx[b] = gx[idx + dxp]; qpx[b] = __ldg(phi + idx + dxp);
        qz[b] = gz[idx + dzp]; qpz[b] = __ldg(phi + idx + dzp);
        qrp[b] = m.rdyp[j + 1]; qdy[b] = m.dyp[j + 1];
      }
    };
#pragma unroll
    for (int b = 0; b < PB; ++b) load(b, j1 - 1 - b >= j0 ? j1 - 1 - b : j0);
    for (int jb = j1 - 1; jb >= j0; jb -= PB) {
#pragma unroll
      for (int b = 0; b < PB; ++b) {
        const int j = jb - b;
        if (j < j0) break;
        const long long idx = col + (long long)j * nx;
        ax = vx[b] - c0[b] * ax;
        ay = vy[b] - c1[b] * ay;
        az = vz[b] - c0[b] * az;
        const T pm = vpm[b];
        const T sucacEta2 = mr[b] * pmAlpha;
        const T uxn = ax - (pc - vpx[b]) * rdxEta2;
        const T uyn = ay - (pc - pm) * sucacEta2;
        const T uzn = az - (pc - vpz[b]) * rdzEta2;
        ux[idx] = uxn; uy[idx] = uyn; uz[idx] = uzn;
        const T pmBetap = -pmBeta * mp[b];
        const T pmBetac = -pmBeta * mc[b] + (T)1;
        const T pmBetam = -pmBeta * mm[b];
        pr[idx] = vp[b] + pmBetap * pp + pmBetac * pc + pmBetam * pm;
        s += (double)uxn * (double)ms[b];
        if (DIAG) {
          // the new velocity at i+1, k+1 and j+1, as the threads that own them compute it
          axp = qx[b] - c0[b] * axp;
          azp = qz[b] - c0[b] * azp;
          const T uxp = axp - (qpx[b] - pc) * rdxEta2;
          const T uzp = azp - (qpz[b] - pc) * rdzEta2;
          const double a = uxn, bb = uyn, c = uzn, aip = uxp, bjp = uyp, ckp = uzp, rdyp = qrp[b];
          double d = fabs((aip - a) * rdx + (bjp - bb) * rdyp + (ckp - c) * rdz);
          if (!(d == d)) d = INFINITY;  // NaN folded into +inf: a NaN field trips the limits
          dvm = fmax(dvm, d);
          v0 = fmax(v0, a == a ? fabs(a) : INFINITY);
          v1 = fmax(v1, bb == bb ? fabs(bb) : INFINITY);
          v2 = fmax(v2, c == c ? fabs(c) : INFINITY);
          cf = fmax(cf, fabs(a + aip) * rdx + fabs(bb + bjp) * rdyp + fabs(c + ckp) * rdz);
          s2 += a * (double)qdy[b];
          uyp = uyn;
        }
        pp = pc; pc = pm;
        if (j >= j0 + PB) load(b, j - PB);
      }
    }
  }
  const int nb = gridDim.x * gridDim.y, bid = blockIdx.x + gridDim.x * blockIdx.y + nb * blockIdx.z;
  if (gridDim.z == 1)
    for (int z = 1 + threadIdx.x; z < npz; z += blockDim.x) {  // the chunk slots this grid leaves empty
      part[bid + (long long)nb * z] = 0.0;
      if (DIAG) part2[bid + (long long)nb * z] = 0.0;
    }
  if constexpr (!DIAG) {
    const double bs = block_sum128(s, red[0]);
    if (threadIdx.x == 0) part[bid] = bs;
  } else {
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      dvm = fmax(dvm, __shfl_xor_sync(0xffffffffu, dvm, o));
      v0 = fmax(v0, __shfl_xor_sync(0xffffffffu, v0, o));
      v1 = fmax(v1, __shfl_xor_sync(0xffffffffu, v1, o));
      v2 = fmax(v2, __shfl_xor_sync(0xffffffffu, v2, o));
      cf = fmax(cf, __shfl_xor_sync(0xffffffffu, cf, o));
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
      red[0][w] = s; red[1][w] = s2; red[2][w] = cf; red[3][w] = dvm; red[4][w] = v0; red[5][w] = v1; red[6][w] = v2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double r[7];
      for (int q = 0; q < 2; ++q) r[q] = (red[q][0] + red[q][1]) + (red[q][2] + red[q][3]);
      for (int q = 2; q < 7; ++q) r[q] = fmax(fmax(red[q][0], red[q][1]), fmax(red[q][2], red[q][3]));
      part[bid] = r[0];
      part2[bid] = r[1];
      atomic_max_nonneg(&sc->uddx, r[2] * 0.5);
      atomic_max_nonneg(&sc->divmax2, r[3]);
      atomic_max_nonneg(&sc->vmax[0], r[4]);
      atomic_max_nonneg(&sc->vmax[1], r[5]);
      atomic_max_nonneg(&sc->vmax[2], r[6]);
    }
  }
}

static dim3 march_proj_grid(const ch3d_ctx* c) {
  const int rows = proj_rows(c);
  return dim3((c->nx + 31) / 32, (c->nz + 3) / 4, (c->ny + rows - 1) / rows);
}
int march_npart(const ch3d_ctx* c) {
  const dim3 g = march_proj_grid(c);
  return (int)(g.x * g.y * g.z);
}

bool march_diag_fusable(const ch3d_ctx* c) {
  // the substituting projection carries them for full tiles only
  return c->cfg.order == 2 && (!c->gsub || (c->nx % 32 == 0 && c->nz % 4 == 0));
}

template <class T> static cudaError_t proj_march_t(ch3d_ctx* c, int mode, bool diag) {
  T** f = (T**)c->f;
  T* in[3] = {mode == 1 ? f[0] : f[12], mode == 1 ? f[1] : f[13], mode == 1 ? f[2] : f[14]};
  auto go = [&](auto kern) {
    kern<<<march_proj_grid(c), 128, 0, c->stream>>>(make_geo<T>(c), metrics_of<T>(c), in[0], in[1], in[2], f[0], f[1],
                                                   f[2], f[3], f[10], f[11], c->part, c->part2, mode, proj_rows(c), c->sc);
    return cudaGetLastError();
  };
  const ch3d_config& q = c->cfg;
  if (q.order == 4) return go(k_proj_march<T, false, 2>);
  if (q.IsImplicit != 1) return diag ? go(k_proj_march<T, true, 1>) : go(k_proj_march<T, false, 1>);
  if (q.LES_type > 0) return diag ? go(k_proj_march<T, true, 3>) : go(k_proj_march<T, false, 3>);
  return diag ? go(k_proj_march<T, true, 0>) : go(k_proj_march<T, false, 0>);
}
cudaError_t launch_proj_march(ch3d_ctx* c, int mode, bool diag) {
  return c->fp32 ? proj_march_t<float>(c, mode, diag) : proj_march_t<double>(c, mode, diag);
}
template <class T> static cudaError_t bulk_march_t(ch3d_ctx* c) {
  T** f = (T**)c->f;
  k_bulk_march<T><<<march_proj_grid(c), 128, 0, c->stream>>>(make_geo<T>(c), metrics_of<T>(c), f[0], c->part,
                                                          proj_rows(c));
  return cudaGetLastError();
}
cudaError_t launch_bulk_march(ch3d_ctx* c) { return c->fp32 ? bulk_march_t<float>(c) : bulk_march_t<double>(c); }

// Rows per block of the substituting projection: the whole column, or, in FP64, chunks
// where the tiles, three blocks per SM, leave more than a fifth of their waves' slots
// empty (on 148 SMs below 356 tiles, 445 to 710, 889 to 1065 and 1333 to 1420).  Steps of
// 192 rows, whole columns / chunks of 32: 384 tiles 1794 / 1833 us, 512 2419 / 2277, 648
// 3418 / 3367, 768 3606 / 3620, 864 4095 / 4143, 1024 4821 / 4718, 1152 5486 / 5461, 1296
// 6070 / 6241.  Mixed, the launch: 512 tiles 115 / 121 us, 3456 1343 / 1436.
static int bsub_rows(const ch3d_ctx* c) {
  const long long tiles = (long long)((c->nx + 31) / 32) * ((c->nz + 3) / 4);
  const long long slots = 3LL * sm_count(c->device), waves = (tiles + slots - 1) / slots;
  return c->fp32 || 5 * tiles >= 4 * waves * slots ? c->ny : proj_rows(c);
}
template <class T> static cudaError_t div_bsub_t(ch3d_ctx* c) {
  T** f = (T**)c->f;
  const dim3 grid((c->nx + 31) / 32, (c->nz + 3) / 4);
  const int rows = bsub_rows(c);
  T* const bnd = rows < c->ny ? f[7] : nullptr;
  auto go = [&](auto kern) {
    kern<<<grid, 128, 0, c->stream>>>(make_geo<T>(c), metrics_of<T>(c), (const T*)c->mtab, f[12], f[13], f[14], f[10],
                                      bnd, rows, c->sc);
    return cudaGetLastError();
  };
  // 256x192x256 (512 blocks): 74 us with 4 rows, 93 with 8; 768x384x576 (3456 blocks):
  // 0.84 ms with 8 rows against 0.88 with 4
  if constexpr (sizeof(T) == 8)
    if (bnd) return go(k_div_bsub<T, 4, true>);
  // FP32: 8 rows always (256x192x256 with the x transform 93 / 86 us, 768x384x576 the same)
  if constexpr (sizeof(T) == 4) return go(k_div_bsub<T, 8, false>);
  else return (long long)grid.x * grid.y > 6LL * sm_count(c->device) ? go(k_div_bsub<T, 8, false>) : go(k_div_bsub<T, 4, false>);
}
cudaError_t launch_div_bsub(ch3d_ctx* c) { return c->fp32 ? div_bsub_t<float>(c) : div_bsub_t<double>(c); }

template <class T> static cudaError_t proj_bsub_t(ch3d_ctx* c, bool diag) {
  T** f = (T**)c->f;
  const int rows = bsub_rows(c), npz = (int)march_proj_grid(c).z;
  const dim3 grid((c->nx + 31) / 32, (c->nz + 3) / 4, (c->ny + rows - 1) / rows);
  auto go = [&](auto kern) {
    kern<<<grid, 128, 0, c->stream>>>(make_geo<T>(c), metrics_of<T>(c), (const T*)c->mtab, f[12], f[13], f[14], f[0],
                                      f[1], f[2], f[3], f[10], f[7], c->part, c->part2, npz, rows, c->sc);
    return cudaGetLastError();
  };
  return diag ? go(k_proj_bsub<T, true>) : go(k_proj_bsub<T, false>);
}
cudaError_t launch_proj_bsub(ch3d_ctx* c, bool diag) {
  return c->fp32 ? proj_bsub_t<float>(c, diag) : proj_bsub_t<double>(c, diag);
}

// The march runs twisted when all column tiles fit on the GPU at once as
// two-group blocks.
template <class T, bool O4> struct MarchShape {
  static constexpr int BZ = 4, D = sizeof(T) == 8 ? 2 : 4, RS = D + 4;
  // resident blocks per SM of the 2nd-order kernel
  static constexpr int bps(bool stops_at_g) { return sizeof(T) == 8 ? 4 : (stops_at_g ? 6 : 5); }
  static constexpr int H = O4 ? 3 : 1;
  static constexpr size_t smem = march_group_smem<T>(RS, march_pl(H, 1, BZ));
  // the march that stops at g (lines of multiples of 128 points): copy vectors
  static constexpr int GW = sizeof(T) == 4 ? 4 : 1;
  static constexpr size_t smem_g = march_group_smem<T>(RS, march_pl(H, GW, BZ));
};
template <class T, bool O4> static bool march_twisted_t(const ch3d_ctx* c) {
  typedef MarchShape<T, O4> S;
  static PerDevice site;                  // per instance: the twisted kernel's limit and occupancy
  static int occ_dev[kMaxDevices] = {};   // twisted blocks per SM, written once per device under the set-up lock
  auto kern_tw = k_rhs_march<T, O4, true, true, 1, S::BZ, S::D, S::RS>;
  const cudaError_t e = once_per_device(site, c->device, [&] {
    cudaError_t r = cudaFuncSetAttribute(kern_tw, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * S::smem));
    if (r != cudaSuccess) return r;
    int occ = 0;
    if ((r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern_tw, 64 * S::BZ, 2 * S::smem)) != cudaSuccess)
      return r;
    occ_dev[c->device] = occ;
    return cudaSuccess;
  });
  if (e != cudaSuccess) return false;  // the one-directional march has no such requirement
  const long long ntiles = (long long)((c->nx + 31) / 32) * ((c->nz + S::BZ - 1) / S::BZ);
  return c->ny >= 2 && ntiles <= (long long)sm_count(c->device) * occ_dev[c->device];
}
bool march_twisted(const ch3d_ctx* c) {
  if (c->cfg.order == 4) return c->fp32 ? march_twisted_t<float, true>(c) : march_twisted_t<double, true>(c);
  return c->fp32 ? march_twisted_t<float, false>(c) : march_twisted_t<double, false>(c);
}

template <class T, bool O4> static cudaError_t rhs_march_t(ch3d_ctx* c) {
  typedef MarchShape<T, O4> S;
  constexpr int BZ = S::BZ, D = S::D, RS = S::RS;
  const size_t smem = S::smem;
  T** f = (T**)c->f;
  auto kern = k_rhs_march<T, O4, false, true, 1, BZ, D, RS>;
  auto kern_tw = k_rhs_march<T, O4, true, true, 1, BZ, D, RS>;
  const bool tw = march_twisted_t<T, O4>(c);  // also sets the twisted kernel's shared-memory limit
  static PerDevice site;  // per instance: the one-directional kernels' limits
  cudaError_t e = once_per_device(site, c->device, [&] {
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t r = cudaFuncSetAttribute(kern, a, (int)smem);
    if constexpr (!O4) {
      if (r == cudaSuccess) r = cudaFuncSetAttribute(k_rhs_march<T, O4, false, false, S::GW, BZ, D, RS>, a, (int)S::smem_g);
    }
    return r;
  });
  if (e != cudaSuccess) return e;
  const int nsm = sm_count(c->device);
  const long long ntiles = (long long)((c->nx + 31) / 32) * ((c->nz + BZ - 1) / BZ);
  auto args = [&](auto k, unsigned grid, int threads, size_t sm) {
    k<<<grid, threads, sm, c->stream>>>(make_geo<T>(c), (const T*)c->mtab, march_down_tables<T>(c->mtab, c->ny), f[0],
                                        f[1], f[2], f[3], f[4], f[5], f[6], f[12], f[13], f[14], c->sc);
  };
  if (tw) {
    // few column tiles: all fit at once as two-group (twisted) blocks, half the march length
    args(kern_tw, (unsigned)ntiles, 64 * BZ, 2 * smem);
  } else {
    // 2nd order: persistent blocks (back substitution, if any, overlapped with the next
    // tile's march); 4th order: one tile per block
    const long long cap = !O4 ? (long long)nsm * S::bps(c->gsub) : ntiles;
    const unsigned grid = (unsigned)(ntiles < cap ? ntiles : cap);
    bool done = false;
    if constexpr (!O4) {
      if (c->gsub) {  // stops at g: the divergence and projection marches substitute
        args(k_rhs_march<T, O4, false, false, S::GW, BZ, D, RS>, grid, 32 * BZ, S::smem_g);
        done = true;
      }
    }
    if (!done) args(kern, grid, 32 * BZ, smem);
  }
  return cudaGetLastError();
}
// Grids with few columns: a column march's time is set by its dependent rows per
// thread, however few columns there are; the right-hand sides by chunks of rows
// and the y sweep as its own pass cost 6 more arrays of (L2) traffic instead.
// 64^3 (4096 columns): 50 us against 19; 192^3 (36864): 224 us against 335.  Steps of 128
// rows, rows / march: 16384 columns 535 / 587 us, 18432 706 / 740, 24576 813 / 810, 31104
// 1054 / 993; mixed 376 / 421, 466 / 520, 611 / 589, 760 / 695.  With 48 rows they meet
// near 14000 (16384: 251 / 251, mixed 177 / 172), with 256 near 25000.
bool march_rows_path(const ch3d_ctx* c) {
  return c->march && (long long)c->nx * c->nz <= 120LL * sm_count(c->device);
}
cudaError_t launch_rhs_march(ch3d_ctx* c) {
  if (c->cfg.order == 4) return c->fp32 ? rhs_march_t<float, true>(c) : rhs_march_t<double, true>(c);
  return c->fp32 ? rhs_march_t<float, false>(c) : rhs_march_t<double, false>(c);
}

}  // namespace ch3d
